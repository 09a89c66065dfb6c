"""bridct_ragged_set_schedule either takes effect whole or leaves the batch as it was: whichever of its
device allocations fails, every array stays in the queue or the passes that ran it before."""
import ctypes as C

import pytest

from bridct_b200 import _lib
from tests import fake_cuda

QUEUE, MERGED = 0, 3
# 40 x 256x256 may be merged; the 128x128 arrays no sub-block of the queue holds, so they join the merged
# passes (more than 2^21 elements come together); the 64x64 ones stay in the queue.
ITEMS = [(256, 256, 0)] * 40 + [(128, 128, 1)] * 6 + [(64, 64, 2)] * 5


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


def _batch(L):
    arr, at = (_lib.RaggedItem * len(ITEMS))(), 0
    for i, (h, w, m) in enumerate(ITEMS):
        arr[i] = _lib.RaggedItem(h, w, m, 0, at)
        at += h * w
    return L.bridct_ragged_create(arr, len(ITEMS)), at


def _state(L, b, n):
    """What a caller sees of the batch, and the launches of one call."""
    classes = []
    for i in range(L.bridct_ragged_class_count(b)):
        h, w, m, s = (C.c_int() for _ in range(4))
        k = C.c_size_t()
        assert L.bridct_ragged_class_info(b, i, h, w, m, k, s) == _lib.OK
        classes.append((h.value, w.value, m.value, k.value, s.value))
    L.fake_reset()
    assert L.bridct_ragged_apply_device(b, 1 << 20, (1 << 20) + 4 * n, None) == _lib.OK   # recorded, not run
    return classes, L.bridct_ragged_units(b), L.bridct_ragged_launch_count(b), fake_cuda.launched(L)


def _set(L, b, merged):
    n = L.bridct_ragged_class_count(b)
    want = []
    for i in range(n):
        h, w = C.c_int(), C.c_int()
        assert L.bridct_ragged_class_info(b, i, h, w, None, None, None) == _lib.OK
        want.append(MERGED if merged and (h.value, w.value) == (256, 256) else QUEUE)
    return L.bridct_ragged_set_schedule(b, (C.c_int * n)(*want), n, 2)


@pytest.mark.parametrize("merged_first", [False, True])
def test_a_failed_schedule_leaves_the_batch_as_it_was(library, monkeypatch, merged_first):
    L = fake_cuda.load(library, monkeypatch)
    b, n = _batch(L)
    assert b
    assert _set(L, b, merged_first) == _lib.OK
    before, live = _state(L, b, n), L.fake_live_allocations()
    failures = 0
    while True:
        L.fake_fail_malloc(failures)
        st = _set(L, b, not merged_first)
        L.fake_fail_malloc(-1)
        if st == _lib.OK:
            break
        assert st == _lib.DEVICE_ERROR
        assert _state(L, b, n) == before, failures
        assert L.fake_live_allocations() == live, failures
        failures += 1
    assert failures == (2 if merged_first else 4)      # arrays and queue, then a table of strips and one of blocks
    after = _state(L, b, n)
    assert after != before
    merged = [name for name, _ in after[3] if "k_merged" in name]
    assert bool(merged) is not merged_first
    L.bridct_ragged_destroy(b)
