"""The slice sort against a stable CPU sort at the edges of its tiles (4096),
warps' shares (256) and digits (8 bits), for keys in order, scattered, equal
and few; keys out of range are refused and leave the result alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 4095, 4096, 4097, 8193, 300_001, 1_050_000])
@pytest.mark.parametrize("kmax", [0, 1, 255, 256, 65_535, 65_536, (1 << 24), (1 << 30) - 1])
def test_sort_is_the_stable_sort(fb, n, kmax):
    rng = np.random.default_rng(n + kmax)
    near = np.clip(np.arange(n) * (kmax + 1) // n + rng.integers(-3, 4, n), 0, kmax)
    for keys in (rng.integers(0, kmax + 1, n), near, np.full(n, kmax)):
        keys = keys.astype(np.int32)
        keys[n // 2] = kmax  # the number of passes
        assert np.array_equal(fb.sort_by_slice(keys), np.argsort(keys, kind="stable"))


@pytest.mark.parametrize("bad", [-1, 1 << 30, -(1 << 31)])
def test_keys_out_of_range_are_refused(fb, bad):
    keys = np.zeros(5000, np.int32)
    keys[4999] = bad
    with pytest.raises(fb.FelisError):
        fb.sort_by_slice(keys)
