"""The FP64 ADI at the edges of its parts and tiles: the smallest grids, the
largest plane in shared memory and the smallest beyond it, bands of one line,
the widest grid; bit-identical to the CPU restatement.
"""
import numpy as np
import pytest

from conftest import assert_bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [7, 33, 112, 113, 129, 130, 161, 255])
def test_adi_equals_the_restatement(fb, oracle_mod, tmp_path, nx):
    from felis_b200 import workloads

    path = workloads.write_input(str(tmp_path / "a.inp"), kind="sase", slices=4, beamlets=40, nx=nx, total_length=0.3,
                                 seed_power=2e6, harmonics=(1, 3), undulator="QuadPolar", polarity=0.5,
                                 abc_n=min(10, nx // 3))
    cfg = fb.Config(path)
    p = cfg.params
    beam = cfg.load_beam(0, seed=4)
    g, o = fb.Handle(p), oracle_mod.Oracle(p, threads=4)
    keys = ("x", "y", "px", "py", "theta", "gamma")
    g.upload_particles(0, *(beam[k] for k in keys), beam["offsets"], beam["weights"])
    o.set_particles(0, *(beam[k] for k in keys), beam["offsets"], beam["weights"])
    rng = np.random.default_rng(nx)
    shape = (p.slice_n + 2, p.ny, p.nx)
    for h in range(p.num_harmony):
        for pol in (0, 1):  # edge cells included: the ADI keeps them and reads their rows
            u = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
            u *= 1e-5
            u[0] = u[-1] = 0  # the ghost planes
            g.upload_field(h, pol, u)
            o.set_field(h, pol, u)
    g.run(0, 3)
    e, _, _ = o.run(0, 3)
    for h in range(p.num_harmony):
        for pol in (0, 1):
            assert_bits(g.download_field(h, pol)[1:-1], o.get_field(h, pol)[1:-1], f"field h{h} pol{pol}")
    np.testing.assert_allclose(g.diagnostics(0, 3)[0], e, rtol=1e-12)
