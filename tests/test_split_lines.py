"""Line pairs (csrc/sj_split.cuh): the generated packed programs on the CPU, and on the GPU the
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


# Whole-array tiles: one shape per configuration, a batch too small to fill the GPU (the smaller tiles)
# and one of more than a wave of full tiles that ends in a partial one.
@pytest.mark.gpu
@pytest.mark.parametrize("shape,many", [((8, 16), 30001), ((16, 8), 30001), ((16, 16), 15001), ((16, 32), 13001),
                                        ((32, 32), 6501), ((64, 8), 15001), ((8, 64), 15001), ((64, 64), 1901),
                                        ((8, 128), 5001), ((32, 128), 1601), ((64, 128), 901), ((128, 8), 6201),
                                        ((128, 16), 2501), ((128, 32), 1601), ((8, 256), 3101), ((32, 256), 801),
                                        ((64, 256), 451), ((256, 8), 3101), ((256, 16), 1601), ((256, 64), 451),
                                        ((8, 512), 1601), ((32, 512), 451), ((512, 8), 1201), ((512, 32), 301),
                                        ((8, 1024), 901), ((16, 1024), 451), ((1024, 8), 451), ((1024, 16), 451)])
def test_tiles_agree_bitwise_and_with_float64(shape, many):
    import torch

    from bridct_b200 import torch_api
    from oracle import oracle as O

    h, w = shape
    g = torch.Generator(device="cuda")
    g.manual_seed(h * 3 + w)
    x = torch.randn((many, h, w), generator=g, device="cuda")
    guard = torch.full((many + 1, h, w), 7.0, device="cuda")
    for mode in range(3):
        y = torch_api.apply(x, mode, out=guard[:many])
        assert torch.equal(guard[many], torch.full_like(guard[many], 7.0)), mode
        for n in (1, 3):
            assert torch.equal(torch_api.apply(x[:n].contiguous(), mode), y[:n]), (mode, n)
        tail = x[-5:].cpu().numpy()
        ref = O.fp64_apply(tail, mode)
        err = np.abs(y[-5:].cpu().numpy() - ref).max() / max(np.abs(tail).max(), np.abs(ref).max())
        assert err <= 2e-6, (mode, err)


# The ragged batch's kernels over every shape and mode once: the queue with its default and its
# smallest units, the merged passes with all modes in one launch, and (two arrays of each class, more
# than 2^24 elements) a launch per mode.
@pytest.mark.gpu
@pytest.mark.parametrize("schedule,copies,unit", [("queue", 1, 16384), ("queue", 1, 1024), ("merged", 1, 16384),
                                                  ("merged", 2, 16384)])
def test_ragged_kernels_on_every_shape_and_mode(schedule, copies, unit):
    import torch

    from bridct_b200.ragged import RaggedBatch, two_pass
    from oracle import oracle as O

    sizes = (8, 16, 32, 64, 128, 256, 512, 1024)
    items = [(h, w, m) for h in sizes for w in sizes for m in range(3) for _ in range(copies)]
    total = sum(h * w for h, w, m in items if two_pass(h, w, m))
    assert (total > 1 << 24) == (copies == 2)
    classes = {f"{h}x{w}/{m}": "merged" for h, w, m in items if two_pass(h, w, m)}
    batch = RaggedBatch(items, tuning=dict(tile_floats=unit, strip_floats=unit, row_floats=unit),
                        schedule={"classes": classes, "streams": 2} if schedule == "merged" else None)
    rng = np.random.default_rng(copies)
    x = torch.from_numpy(rng.standard_normal(batch.span).astype(np.float32)).cuda()
    y = batch.apply(x)
    torch.cuda.synchronize()
    assert not batch.timed_out()
    for (h, w, m), xi, yi in zip(items, batch.unpack(x.cpu()), batch.unpack(y.cpu())):
        xi, ref = xi.numpy(), O.fp64_apply(xi.numpy(), m)
        err = np.abs(yi.numpy() - ref).max() / max(np.abs(xi).max(), np.abs(ref).max())
        assert err <= 2e-6, (h, w, m, err)
