"""The tensor-core forms over the whole range of float32: samples above half of it whose mirrored sums
leave the range while the transform does not."""
import numpy as np
import pytest

from tests.helpers import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["tc_bf16x3", "tc_tf32x3"])
@pytest.mark.parametrize("shape", [(8, 128), (128, 8), (8, 256), (256, 8), (256, 256), (512, 64), (64, 512),
                                   (1024, 16), (16, 1024)])
def test_forward_takes_samples_near_the_largest_float(form, shape):
    import torch

    from bridct_b200 import torch_api
    from oracle import oracle as O

    h, w = shape
    x = np.zeros((4, h, w), np.float32)
    x[0, 1, 3] = x[0, 1, w - 4] = 3e38                      # equal at mirrored places of a row
    x[1, 1, 3], x[1, 1, w - 4] = 3e38, -3e38                # opposite
    x[2, 2] = x[2, h - 3] = 3e38 / np.sqrt(w)               # rows whose first coefficient is 3e38, mirrored
    x[3, 2], x[3, h - 3] = 3e38 / np.sqrt(w), -3e38 / np.sqrt(w)
    ref = O.fp64_apply(x, 0)
    assert np.abs(ref).max() < 3.4e38
    y = torch_api.apply(torch.from_numpy(x).cuda(), 0, form=form).cpu().numpy()
    assert np.isfinite(y).all()
    assert O.rel_max_error(y, ref, x, output_scaled=True) <= TOL     # the suite's bound
