"""The ADI leaves out field planes that are known to be zero and receive no
source: a planar undulator's second polarisation.  Every way a value can come
into such a plane -- an upload into some slices, the first planes a neighbour
hands over, the slippage that moves them along -- against the CPU restatement
(FP64, bit for bit) and, for the mixed-precision engine, against FP64.
"""
import numpy as np
import pytest

from conftest import assert_bits

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")


def _case(fb, tmp_path, nx=33, harmonics=(1, 3), **kw):
    from felis_b200 import workloads

    path = workloads.write_input(str(tmp_path / "z.inp"), kind="sase", slices=6, beamlets=40, nx=nx, total_length=0.6,
                                 seed_power=2e6, harmonics=harmonics, abc_n=6, **kw)
    cfg = fb.Config(path)
    return cfg, cfg.params, cfg.load_beam(0, seed=4)


def _fields(p, rng, lit):
    """Noise in the x planes of every slice, in the y planes of slices `lit`."""
    out = {}
    for h in range(p.num_harmony):
        for pol in (0, 1):
            u = 1e-5 * (rng.standard_normal((p.slice_n + 2, p.ny, p.nx))
                        + 1j * rng.standard_normal((p.slice_n + 2, p.ny, p.nx)))
            u[0] = u[-1] = 0
            if pol:
                for s in range(p.slice_n):
                    if s not in lit:
                        u[s + 1] = 0
            out[h, pol] = u
    return out


@pytest.mark.parametrize("nx,harmonics,lit", [(33, (1, 3), ()), (33, (1, 2), (2,)), (130, (1, 3), (0, 5))])
def test_handle_equals_the_restatement(fb, oracle_mod, tmp_path, nx, harmonics, lit):
    cfg, p, beam = _case(fb, tmp_path, nx, harmonics)
    g, o = fb.Handle(p), oracle_mod.Oracle(p, threads=4)
    g.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    o.set_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    rng = np.random.default_rng(nx)
    n = 0
    for again in range(2):  # the second upload goes into planes known to be zero
        for (h, pol), u in _fields(p, rng, lit if again else ()).items():
            g.upload_field(h, pol, u)
            o.set_field(h, pol, u)
        g.run(n, 4)
        e, _, _ = o.run(n, 4)
        n += 4
        for h in range(p.num_harmony):
            for pol in (0, 1):
                assert_bits(g.download_field(h, pol)[1:-1], o.get_field(h, pol)[1:-1], f"field h{h} pol{pol}")


def test_first_planes_light_a_dark_plane(fb, tmp_path):
    """set_first_planes and an upload of the same planes continue alike."""
    cfg, p, beam = _case(fb, tmp_path)
    out = []
    for direct in (True, False):
        g = fb.Handle(p)
        g.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
        g.run(0, 3)
        rng = np.random.default_rng(1)
        first = 1e-5 * (rng.standard_normal((p.num_harmony * 2, p.ny, p.nx)) + 1j)
        if direct:
            g.set_first_planes(np.ascontiguousarray(first).reshape(g.first_planes().shape).view(g.first_planes().dtype))
        else:
            for h in range(p.num_harmony):
                for pol in (0, 1):
                    u = g.download_field(h, pol)
                    u[1] = first[h * 2 + pol]
                    g.upload_field(h, pol, u)
        g.run(3, 3)
        out.append([g.download_field(h, pol) for h in range(p.num_harmony) for pol in (0, 1)])
    for a, b in zip(*out):
        assert_bits(a[1:-1], b[1:-1], "field")
        assert np.abs(a).max() > 0


@pytest.mark.parametrize("lit", [(), (1, 4)])
def test_batch_follows_fp64(fb, tmp_path, lit):
    """The y planes evolve without a source: six FP32 solves of five roundings
    per recurrence step against FP64, 1e-5 of the largest value; dark planes
    that nothing reaches stay exactly zero."""
    cfg, p, beam = _case(fb, tmp_path)
    g, b = fb.Handle(p), fb.Batch([p])
    g.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    b.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    rng = np.random.default_rng(3)
    n = 0
    for again in range(2):
        fields = _fields(p, rng, lit if again else ())
        for (h, pol), u in fields.items():
            g.upload_field(h, pol, u)
            b.upload_field(0, h, pol, u)
        g.run(n, 3)
        b.run(n, 3)
        n += 3
    for h in range(p.num_harmony):
        y, ref = b.download_field(0, h, 1), g.download_field(h, 1)
        assert np.abs(y - ref).max() <= 1e-5 * np.abs(ref).max()
        assert (np.abs(ref).max() > 0) == bool(lit)
