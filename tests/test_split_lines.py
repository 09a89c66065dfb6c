"""Split lines (csrc/sj_split.cuh): the generated packed programs on the CPU, and on the GPU the unit
geometries a batch size selects, at the sizes where one takes over from the other."""
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "bridct_b200" / "csrc"))
import gen_sj  # noqa: E402


def test_packed_header_is_current():
    assert (ROOT / "bridct_b200" / "csrc" / "sj_packed.cuh").read_text() == gen_sj.generate_packed() + "\n"


@pytest.mark.parametrize("n", gen_sj.PACKED_STAGE2)
def test_real_columns_program_and_its_transpose(n):
    (g, outs), (gt, back) = gen_sj.build_special(n)
    rng = np.random.default_rng(n)
    r = rng.standard_normal((2 * n, 1))
    got = g.evaluate(outs, r)[:, 0]
    r0, r1 = r[0::2, 0], r[1::2, 0]
    b, h = np.arange(n), n // 2
    v0 = np.fft.fft(r0)
    v1 = [np.sum(r1 * np.exp(-2j * np.pi * b * (d + 0.5) / n)) for d in range(n)]
    want = [v0[0].real, v0[h].real / gen_sj.sj_scale(n, h)]
    for j in range(1, h):
        want += [v0[j].real / gen_sj.sj_scale(n, j), v0[j].imag / gen_sj.sj_scale(n, j)]
    for m in range(h):
        want += [v1[2 * m].real / gen_sj.sj_scale(h, m), v1[2 * m].imag / gen_sj.sj_scale(h, m)]
    assert np.abs(got - np.array(want)).max() < 1e-11
    adj = rng.standard_normal((2 * n, 1))
    at = gt.evaluate(back, np.concatenate([adj, np.zeros((2 * n, 1))]))
    assert abs(got @ adj[:, 0] - r[:, 0] @ at[:, 0]) < 1e-9


# Batches below and above the lines of the launch rules: 64 wide strips, one wide row block per SM
# (148), for every line length on both axes.
@pytest.mark.gpu
@pytest.mark.parametrize("shape,few,many", [((128, 256), 8, 40), ((256, 128), 16, 40), ((256, 256), 8, 19),
                                            ((512, 128), 8, 10), ((1024, 128), 8, 9), ((512, 512), 2, 5),
                                            ((256, 1024), 2, 10), ((1024, 1024), 1, 3)])
def test_unit_geometries_agree_bitwise_and_with_float64(shape, few, many):
    import torch

    from bridct_b200 import torch_api
    from oracle import oracle as O

    h, w = shape
    x = np.random.default_rng(h * 3 + w).standard_normal((many, h, w)).astype(np.float32)
    xd = torch.from_numpy(x).cuda()
    for mode in range(3):
        y = torch_api.apply(xd, mode)
        assert torch.equal(torch_api.apply(xd[:few].contiguous(), mode), y[:few]), mode
        ref = O.fp64_apply(x, mode)
        # the suite's bound for float32 lines: 2e-6 of the larger of the input and output maxima
        err = np.abs(y.cpu().numpy() - ref).max() / max(np.abs(x).max(), np.abs(ref).max())
        assert err <= 2e-6, (mode, err)
