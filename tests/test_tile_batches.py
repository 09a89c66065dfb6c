"""Whole-array tiles across the lines of their dispatch (plain_launch.cuh, tile_cfg_few and few_tiles): small
tiles of single lines, half tiles and full tiles give an array the same bits, contiguous and strided."""
import pytest

pytestmark = pytest.mark.gpu

# Elements of a batch: on either side of two tiles per SM, half a wave, a wave and 1.3 waves of the tiles of
# 1024 to 4096 floats; the last one takes full tiles for every shape and ends in a partial one.
SIZES = (1, 1 << 19, 3 << 19, 1 << 21, 3 << 20, 1 << 22, 5 << 21)


@pytest.mark.parametrize("shape", [(8, 16), (16, 8), (16, 16), (8, 32), (32, 8), (16, 32), (32, 16), (32, 32), (8, 64),
                                   (64, 8), (16, 64), (64, 16), (32, 64), (64, 32), (64, 64), (32, 128), (64, 128),
                                   (128, 64), (128, 8), (16, 512), (512, 8), (1024, 8)])
def test_an_array_has_the_same_bits_in_tiles_of_every_batch_size(shape):
    import torch

    from bridct_b200 import torch_api

    h, w = shape
    batches = [max(1, s // (h * w)) for s in SIZES]
    batches[-1] += 1
    g = torch.Generator(device="cuda")
    g.manual_seed(h * 7 + w)
    wide = torch.randn((batches[-1], h, w + 8), generator=g, device="cuda")
    view, x = wide[:, :, 4:4 + w], wide[:, :, 4:4 + w].contiguous()
    for mode in range(3):
        y = torch_api.apply(x, mode)
        for n in batches[:-1]:
            assert torch.equal(torch_api.apply(x[:n].contiguous(), mode), y[:n]), (mode, n)
        for n in batches:
            assert torch.equal(torch_api.apply(view[:n], mode), y[:n]), (mode, n, "strided")
