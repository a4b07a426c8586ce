"""The FP64 particle kernel's instances (harmonics, space-charge modes, even
harmonics) and the window of its shared reciprocals: phase-space coordinates
inside, at the ends of and outside the window give the CPU restatement's bits.
"""
import numpy as np
import pytest

from conftest import assert_bits

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")
# zeros, subnormals, the window's lower end (2^-400) from both sides, ordinary sizes
EDGE = np.array([0.0, -0.0, 5e-324, 1e-310, 2.0**-401, 2.0**-400, -(2.0**-399), 1e-100, 1e-18, -3e-7, 2e-5])

CASES = {
    "planar": dict(),
    "elliptical": dict(undulator="QuadPolar", polarity=0.5),
    "h13": dict(harmonics=(1, 3), undulator="QuadPolar", polarity=0.5),
    "h2": dict(harmonics=(2,), undulator="QuadPolar", polarity=0.5),
    "h1234": dict(harmonics=(1, 2, 3, 4), undulator="QuadPolar", polarity=0.3),
    "h13579": dict(harmonics=(1, 3, 5, 7, 9)),
    "h12345": dict(harmonics=(1, 2, 3, 4, 5), undulator="QuadPolar", polarity=0.3),
    "modes": dict(modes=(3, 2)),
    "modes_h13": dict(modes=(2, 1), harmonics=(1, 3)),
}


@pytest.mark.parametrize("name", CASES)
def test_particle_step_equals_the_restatement(fb, oracle_mod, tmp_path, name):
    from felis_b200 import workloads

    kw = dict(CASES[name])
    modes = kw.pop("modes", (1, 1))
    text = workloads.input_text("sase", slices=2, beamlets=80, nx=41, total_length=0.3, seed_power=2e6, quads=True, **kw)
    path = tmp_path / "p.inp"
    path.write_text(text.replace(" ABC_N=", f" number_longitudinal_mode={modes[0]}\n number_azimuthal_mode={modes[1]}\n ABC_N="))
    cfg = fb.Config(str(path))
    p = cfg.params
    beam = cfg.load_beam(0, seed=5)
    n, m = beam["x"].size, EDGE.size
    for i, k in enumerate(("x", "y", "px", "py")):
        scale = 1.0 if k in ("x", "y") else 1e3
        beam[k][i * m:(i + 1) * m] = EDGE * np.where(np.abs(EDGE) > 1e-200, scale, 1.0)
        beam[k][n // 2 + i::37] = np.resize(EDGE, beam[k][n // 2 + i::37].size)
    g, o = fb.Handle(p), oracle_mod.Oracle(p, threads=4)
    g.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    o.set_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    for h in range(p.num_harmony):
        for pol, u in enumerate(cfg.load_seed(h)):
            g.upload_field(h, pol, u)
            o.set_field(h, pol, u)
    steps = 3
    g.run(0, steps)
    o.run(0, steps)
    a, b = g.download_particles(0), o.get_particles(0)
    for k in KEYS:
        assert_bits(a[k], b[k], k)
    for h in range(p.num_harmony):
        for pol in (0, 1):
            assert_bits(g.download_field(h, pol)[1:-1], o.get_field(h, pol)[1:-1], f"field h{h} pol{pol}")
