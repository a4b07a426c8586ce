"""The staged copies between device and host (HostStage) on the CPU: the source
file compiled against a host stand-in for the few runtime calls it makes, with
two devices, streams and events that belong to one of them, and page-locked
memory that can run out."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DOWN, WIDEN, UP = 0, 1, 2
MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    fake = os.path.join(ROOT, "tests", "host_cuda")
    src = os.path.join(ROOT, "felis_b200", "csrc", "lib")
    out = str(tmp_path_factory.mktemp("transfer") / "transfer_host.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", f"-I{fake}", f"-I{src}", "-x", "c++",
                    os.path.join(src, "transfer.cu"), os.path.join(fake, "transfer_calls.cpp"), "-o", out], check=True)
    so = C.CDLL(out)
    so.stage_new.restype = C.c_void_p
    so.stage_free.argtypes = [C.c_void_p]
    p, n = C.c_void_p, C.c_size_t
    so.stage_copy.argtypes = [p, C.c_int, C.c_int, C.c_int, p, p, n, p, p, n, C.POINTER(C.c_int)]
    return so


def _copy(lib, stage, how, words, device=0, current=0, split=0.3):
    """One call over `words` 32-bit values in two parts: (status, device
    afterwards, whether every value arrived)."""
    a = np.random.default_rng(words).standard_normal(words).astype(np.float32)
    b = np.zeros(words, np.float64 if how == WIDEN else np.float32)
    k, after = int(words * split), C.c_int(-1)
    st = lib.stage_copy(stage, how, device, current, a.ctypes.data, b.ctypes.data, 4 * k, a[k:].ctypes.data,
                        b[k:].ctypes.data, 4 * (words - k), C.byref(after))
    return st, after.value, np.array_equal(a, b)


@pytest.fixture
def stage(lib):
    s = lib.stage_new()
    yield s
    lib.stage_free(s)
    assert lib.host_live() == 0


@pytest.mark.parametrize("how", [DOWN, WIDEN, UP])
@pytest.mark.parametrize("words", [100, 100_001, 5 * MB, 20 * MB + 3])
def test_a_handle_of_another_device(lib, stage, how, words):
    """Copies work, and leave the caller's device, whichever is current."""
    for device, current in ((1, 0), (1, 1), (0, 1), (1, 0)):
        s = lib.stage_new()
        for _ in range(2):
            assert _copy(lib, s, how, words, device, current) == (0, current, True)
        lib.stage_free(s)
    assert _copy(lib, stage, how, words, 1, 0) == (0, 0, True)


@pytest.mark.parametrize("how", [DOWN, WIDEN, UP])
def test_small_copies_lock_no_pages(lib, stage, how):
    """Slots cost milliseconds to make: an object has them only once its copies
    have come to 64 MB at the destination, in one call or in many."""
    per = MB // (2 if how == WIDEN else 1)  # 4 MB at the destination
    before = lib.host_allocations()
    for _ in range(15):
        assert _copy(lib, stage, how, per) == (0, 0, True)
    assert lib.host_allocations() == before and lib.host_live() == 0
    for _ in range(3):
        assert _copy(lib, stage, how, per) == (0, 0, True)
    assert lib.host_live() == 1
    one = lib.stage_new()
    assert _copy(lib, one, how, 16 * per) == (0, 0, True)
    assert lib.host_live() == 2
    lib.stage_free(one)


@pytest.mark.parametrize("how", [DOWN, WIDEN, UP])
def test_copies_go_without_slots_where_there_are_none(lib, stage, how):
    """A machine without page-locked memory left still copies, and takes slots
    again when it can."""
    words = 20 * MB
    lib.fail_host_allocations(1)
    try:
        for _ in range(2):
            assert _copy(lib, stage, how, words) == (0, 0, True)
        assert lib.host_live() == 0
    finally:
        lib.fail_host_allocations(0)
    assert _copy(lib, stage, how, words) == (0, 0, True)
    assert lib.host_live() == 1
    # more slots than it has: those it had are given up, the copies go on
    lib.fail_host_allocations(1)
    try:
        assert _copy(lib, stage, how, 36 * MB) == (0, 0, True)
    finally:
        lib.fail_host_allocations(0)


@pytest.mark.parametrize("how", [DOWN, UP])
def test_small_calls_never_lock_pages(lib, stage, how):
    """A call of less than a chunk gains nothing from slots, after any number of them."""
    for _ in range(90):
        assert _copy(lib, stage, how, MB // 4 - 5) == (0, 0, True)
    assert lib.host_live() == 0
    assert _copy(lib, stage, how, MB) == (0, 0, True)
    assert lib.host_live() == 1
