"""Keys out of range leave the caller's result untouched: their check on the
device ends before anything is written, wherever the first of them lies."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAD_ARG = 1


@pytest.mark.parametrize("bad", [-1, 1 << 30, -(1 << 31)])
@pytest.mark.parametrize("n, at", [(1, 0), (5000, 0), (5000, 4095), (5000, 4096), (5000, 4999), (300_001, 150_000)])
def test_a_refused_call_writes_nothing(fb, bad, n, at):
    keys = np.random.default_rng(n).integers(0, 1024, n).astype(np.int32)
    keys[at] = bad
    perm = np.full(n, -12345, np.int64)
    fn = fb._lib.felis_sort_by_slice
    st = fn(keys.ctypes.data_as(C.POINTER(C.c_int32)), n, perm.ctypes.data_as(C.POINTER(C.c_int64)))
    assert st == BAD_ARG and (perm == -12345).all()
