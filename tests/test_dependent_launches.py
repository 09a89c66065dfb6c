"""Kernels launched with programmatic stream serialization are resident while the previous kernel of
the stream still runs, and may read what that kernel writes only after griddepcontrol.wait.  A
non-coherent load (__ldg, or any load the compiler may make one of through a __restrict__ pointer to
const) requires data that nothing writes for the kernel's whole lifetime, and a "memory" clobber does not
keep it behind the wait: these kernels use such loads for constant tables only."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bridct_b200" / "csrc"

# What may be loaded with __ldg, by file: tables written when they are created and never by a kernel,
# and the operands of kernels that are launched ordinarily (after the previous kernel has ended).
CONSTANT = {
    "sj_kernels.cuh": {"l.offs + b"},                                     # offset table of a ragged class
    "tc_pass.cuh": {"src + i"},                                           # coefficient images ...
    "tc_blocks8.cuh": {"bimage + i"},
    "tc_fused64.cuh": {"bimage + i"},
    "tc_fp8.cuh": {"src + i", "sc + (size_t)(2 * nblk) * F::kKT + i",
                   "reinterpret_cast<const float4*>(rows + (row0 + (i >> ql)) * L + col0 "
                   "+ ((i & ((1 << ql) - 1)) << 2))"},                    # k_quant8: launched with <<< >>>
    "ragged.cuh": {"reinterpret_cast<const float2*>(x + (long long)i * ld) + p"},   # k_ragged: likewise
}


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _call_arguments(code, name):
    for m in re.finditer(name + r"\s*\(", code):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(code[i], 0)
            i += 1
        yield " ".join(code[m.end():i - 1].split())


def test_non_coherent_loads_read_constant_tables_only():
    for path in sorted(CSRC.glob("*.cu*")):
        extra = set(_call_arguments(_code(path), "__ldg")) - CONSTANT.get(path.name, set())
        assert not extra, (path.name, extra)
    for name in ("k_quant8", "k_ragged"):     # the exceptions above are ordinary launches
        launches = [c for p in CSRC.glob("*.cu") for c in re.findall(r"launch_pdl\([^;]*", _code(p))]
        assert not [c for c in launches if name in c]


def test_dependent_kernels_take_no_restrict_pointers_to_data():
    constant = {"bimage", "sc"}
    for path in sorted(CSRC.glob("*.cu*")):
        code = _code(path)
        for m in re.finditer(r"__global__[^{;]*\{", code):
            end = code.find("__global__", m.end())
            if "griddep" not in code[m.end():end if end > 0 else len(code)]:
                continue
            for p in re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", m.group(0)):
                assert p in constant, (path.name, p)


# Calls back to back on one stream, each reading what the one before it wrote, against the same calls
# with a synchronization between them: shapes whose column pass loads straight to registers (32- and
# 64-point columns of two-pass shapes), 8x8 batches of both kernels, and the FP8 form.
@pytest.mark.gpu
@pytest.mark.parametrize("form,shape,batch", [("sj", (32, 1024), 40), ("sj", (64, 512), 40), ("sj", (64, 512), 3),
                                              ("sj", (64, 1024), 20), ("sj", (8, 8), 20000), ("sj", (8, 8), 500000),
                                              ("tc_fp8", (64, 64), 64)])
def test_chained_calls_equal_synchronized_ones(form, shape, batch):
    import torch

    from bridct_b200 import torch_api

    g = torch.Generator(device="cuda")
    g.manual_seed(batch)
    x = torch.randn((batch, *shape), generator=g, device="cuda")

    def chain(wait):
        bufs = [torch.empty_like(x) for _ in range(2)]
        src = x
        torch.cuda.synchronize()
        for k in range(12):
            src = torch_api.apply(src, k % 2, out=bufs[k % 2], form=form)
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return src

    want = chain(True)
    for _ in range(3):
        assert torch.equal(chain(False), want)
