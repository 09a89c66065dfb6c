"""bridct_ragged_apply_noalloc builds its tables in static buffers, on the host as well: a first call
requests nothing of the heap but the launch bookkeeping (a map node), so no allocation failure can leave
half a table behind or cross the C boundary."""
import ctypes as C

import pytest

from bridct_b200 import _lib
from tests import fake_cuda


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    return fake_cuda.build(tmp_path_factory.mktemp("fake"))


def test_first_call_takes_no_table_from_the_heap(library, monkeypatch):
    L = fake_cuda.load(library, monkeypatch)
    L.fake_largest_new.restype = C.c_size_t
    items = (_lib.RaggedItem * 2)(_lib.RaggedItem(64, 64, 0, 0, 0), _lib.RaggedItem(256, 1024, 1, 0, 4096))
    n = 4096 + 256 * 1024
    x, y = (C.c_float * (n + 4))(), (C.c_float * (n + 4))()
    align = lambda b: (C.addressof(b) + 15) // 16 * 16
    L.fake_largest_new()
    assert L.bridct_ragged_apply_noalloc(items, 2, align(x), align(y), None) == _lib.OK, _lib.last_error()
    assert L.fake_largest_new() <= 256
    assert [n for n, _ in fake_cuda.launched(L) if "k_ragged" in n]


def test_static_device_memory_stays_below_a_megabyte(library, monkeypatch):
    L = fake_cuda.load(library, monkeypatch)
    L.fake_symbol_bytes.restype = C.c_size_t
    assert 0 < L.fake_symbol_bytes() < 1000000
