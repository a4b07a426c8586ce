"""The mixed engine's fixed-point deposit with an even harmonic: the quantum is
set by the largest term that a particle of the slice can add, not by the largest
numerator over the least gamma of different particles, so two particles far from
the beam, one with a large transverse momentum and one of a low energy, cost no
more precision than the larger of their own terms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")


@pytest.mark.parametrize("others", [0, 1100])  # wide and narrow CTAs
def test_far_particles_cost_their_own_terms(fb, tmp_path, others):
    from felis_b200 import workloads

    def config(name, kind, **kw):
        return fb.Config(workloads.write_input(str(tmp_path / name), kind=kind, nx=61, total_length=0.3, seed_power=0.0,
                                               harmonics=(1, 2), abc_n=6, undulator="QuadPolar", polarity=0.5, **kw))

    cfg = config("q.inp", "static", slices=1, beamlets=4)
    p = cfg.params
    n, a, b = 10, 5, 2  # particles; the one of large momentum; the one of low energy
    rng = np.random.default_rng(3)
    beam = {k: np.zeros(n) for k in KEYS}
    # eight particles about the middle of one cell, at one phase
    beam["x"][:] = p.min_x + (30.5 + 0.1 * rng.uniform(-1, 1, n)) * p.dx
    beam["y"][:] = p.min_y + (30.5 + 0.1 * rng.uniform(-1, 1, n)) * p.dy
    beam["theta"][:] = 0.3 + 0.01 * rng.uniform(-1, 1, n)
    beam["gamma"][:] = p.gam_r
    # the two sit in the grid's last column: counted for the bound, outside the
    # push and without an interior cell to add to
    for q in (a, b):
        beam["x"][q] = p.min_x + (p.nx - 0.5) * p.dx
    beam["py"][a] = 50.0
    beam["gamma"][b] = p.gam_r / 64.0
    weights = np.full(1, 1.0e5)
    offsets = np.array([0, n], np.int64)

    g = fb.Handle(p)
    g.upload_particles(0, *(beam[k] for k in KEYS), offsets, weights)
    g.run(0, 2)
    insts = [(cfg, beam, offsets, weights)]
    if others:
        c = config("f.inp", "sase", slices=others, beamlets=8)
        f = c.load_beam(0, seed=4)
        insts.append((c, f, f["offsets"], f["weights"]))
    m = fb.Batch([i[0].params for i in insts])
    for k, (_, u, o, w) in enumerate(insts):
        m.upload_particles(k, *(u[q] for q in KEYS), o, w)
    m.run(0, 2)

    # a term of the middle particles is H w / gamma in the units of the bound, and
    # at least 0.2 of it reaches each of its four cells; the far one's own term
    # bounds it by 2 xi2 Hmax / gamma
    K0, ue, Hmax = p.K0_init, p.ue_init, 2.0
    xi2 = np.sqrt(2.0) * K0 / (1.0 + 0.5 * K0 * K0 * (1.0 + ue * ue)) * np.sqrt(2.0) * ue * 50.0
    own, apart = max(2.0 * xi2 * Hmax, 64.0), 2.0 * xi2 * Hmax * 64.0
    quantum = 1.0625 * Hmax * own * 2.0**-21  # of a middle particle's term; term / quantum < 2^22 decides
    assert apart > 50.0 * own
    # half a quantum in either component of every term, and FP32 beside it
    tol = np.sqrt(2.0) * 0.5 * quantum / 0.2 + 3.0e-5
    for pol in (0, 1):
        want, got = g.download_field(0, pol)[1], m.download_field(0, 0, pol)[1]
        scale = np.abs(want).max()
        assert scale > 0
        assert np.abs(got - want).max() <= tol * scale, (pol, np.abs(got - want).max() / scale, tol)
