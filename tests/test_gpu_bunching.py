"""The FP64 bunching factors of phases that nothing has wrapped: as accurate far
from zero as near it, on both sides of 2^20 where the sine changes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")


@pytest.mark.parametrize("size", [10.0, 1.0e6, 2.0**20, 2.0e6, 1.0e9, 1.0e15])
def test_bunching_of_far_phases(fb, tmp_path, size):
    from felis_b200 import workloads

    harmonics = (1, 2, 3)
    cfg = fb.Config(workloads.write_input(str(tmp_path / "b.inp"), kind="sase", slices=3, beamlets=100, nx=33,
                                          total_length=0.3, harmonics=harmonics, abc_n=6))
    beam = cfg.load_beam(0, seed=4)
    n = len(beam["theta"])
    rng = np.random.default_rng(int(size) % 1000)
    beam["theta"] = size * rng.uniform(-1.1, 1.1, n)
    h = fb.Handle(cfg.params)
    h.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    got = h.bfactor()
    w = np.repeat(beam["weights"], np.diff(beam["offsets"]))
    want = []
    for H in harmonics:
        a = H * beam["theta"]
        want += [np.sum(np.cos(a) * w) / np.sum(w), np.sum(np.sin(a) * w) / np.sum(w)]
    # terms: 2 ulp of the sines on either side and the products; sums of n terms on either side
    np.testing.assert_allclose(got, want, rtol=0, atol=(2 * n + 8) * 2.0**-53)
