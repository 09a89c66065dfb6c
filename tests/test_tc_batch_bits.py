"""An array's tensor-core results have the same bits whatever shares its call: the row passes take narrow
or wide N-blocks by the number of rows (half of the 148 SMs is the line), and both sum the same products in
the same order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["tc_bf16x3", "tc_tf32x3"])
@pytest.mark.parametrize("shape,batches", [((128, 128), (1, 74, 75)), ((256, 256), (1, 9, 10, 18, 19)),
                                           ((512, 512), (1, 4, 5)), ((1024, 1024), (1, 2)), ((8, 256), (1, 17, 591, 593)),
                                           ((256, 8), (1, 295, 297)), ((128, 8), (1, 15, 17)), ((64, 1024), (1, 36, 38))])
def test_a_row_has_the_same_bits_in_a_call_of_any_size(form, shape, batches):
    import torch

    from bridct_b200 import torch_api

    g = torch.Generator(device="cuda")
    g.manual_seed(shape[0] * 5 + shape[1])
    many = 40 * batches[-1] if shape[0] * shape[1] <= 2048 else 3 * batches[-1] + 1
    x = torch.randn((many, *shape), generator=g, device="cuda")
    for mode in (0, 1, 2):
        y = torch_api.apply(x, mode, form=form)
        for n in batches:
            assert torch.equal(torch_api.apply(x[:n].contiguous(), mode, form=form), y[:n]), (mode, n)
