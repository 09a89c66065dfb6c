"""Row passes of the tensor-core forms: batch sizes on both sides of the line between the unfolded and
the folded inverse pass (CTAs of the folded one = half of the 148 SMs), and whole, partial and single
M-tiles of 128 rows in the folded forward pass."""
import numpy as np
import pytest

from tests.helpers import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["tc_bf16x3", "tc_tf32x3"])
@pytest.mark.parametrize("shape,batches", [((128, 128), (1, 74, 75)), ((256, 256), (1, 18, 19)),
                                           ((512, 512), (1, 4, 5)), ((1024, 1024), (1, 2)),
                                           ((8, 256), (1, 17, 591, 593)), ((128, 8), (1, 15, 17))])
def test_row_passes_at_the_lines_of_their_batch_sizes(form, shape, batches):
    import torch

    from bridct_b200 import torch_api
    from oracle import oracle as O

    x = np.random.default_rng(shape[0] + shape[1]).standard_normal((max(batches), *shape)).astype(np.float32)
    for mode in (0, 1):
        ref = O.fp64_apply(x, mode)
        for n in batches:
            y = torch_api.apply(torch.from_numpy(x[:n]).cuda(), mode, form=form)
            # the suite's bound for every form and direction
            assert O.rel_max_error(y.cpu().numpy(), ref[:n], x[:n], output_scaled=True) <= TOL, (mode, n)
