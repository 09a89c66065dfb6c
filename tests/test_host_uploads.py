"""Tables that kernels read are on the device when the call that made them returns: a copy from pageable
memory may return early, and the kernels run on streams that do not wait for the default stream."""
import ctypes as C

import pytest

from bridct_b200 import _lib
from tests import fake_cuda


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


def test_every_table_has_arrived_when_its_call_returns(library, monkeypatch):
    L = fake_cuda.load(library, monkeypatch)
    x, y, ws = 1 << 20, 1 << 24, 1 << 28      # recorded, not run
    for h, w in ((64, 64), (256, 512), (1024, 8)):
        p = L.bridct_plan_create(h, w)
        assert p and L.fake_unfinished() == 0
        for form in (_lib.FORM_TC_BF16X3, _lib.FORM_TC_TF32X3, _lib.FORM_TC_FP8):
            for mode in range(2 if form == _lib.FORM_TC_FP8 else 3):   # its round trip copies
                need = L.bridct_plan_form_workspace_bytes(p, form, 1)
                assert L.bridct_plan_apply_form_device_ws(p, mode, form, x, y, 1, ws, need, 4096) == _lib.OK
                assert L.fake_unfinished() == 0, (h, w, form, mode)
    items = (_lib.RaggedItem * 3)(_lib.RaggedItem(64, 64, 0, 0, 0), _lib.RaggedItem(256, 1024, 1, 0, 4096),
                                  _lib.RaggedItem(512, 512, 2, 0, 4096 + 256 * 1024))
    b = L.bridct_ragged_create(items, 3)
    assert b and L.fake_unfinished() == 0
    assert L.bridct_ragged_set_schedule(b, (C.c_int * 3)(3, 3, 0), 3, 2) == _lib.OK
    assert L.fake_unfinished() == 0
    assert L.bridct_ragged_apply_device(b, x, y, None) == _lib.OK and L.fake_unfinished() == 0
    n = 64 * 64 + 256 * 1024 + 512 * 512
    data = (C.c_float * (2 * n + 8))()
    at = (C.addressof(data) + 15) // 16 * 16
    assert L.bridct_ragged_apply_noalloc(items, 3, at, at + 4 * n, None) == _lib.OK and L.fake_unfinished() == 0
