"""The FP64 source deposit just around its chunks (1024 particles) and its warps'
parts of them (64 consecutive particles), and over several bands of radial bins
(512 to a band): source, field and Ez equal the CPU restatement bit for bit."""
import numpy as np
import pytest

from conftest import assert_bits

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")


def _compare(fb, oracle_mod, tmp_path, beamlets, modes=(1, 1), radial_grids=None, move=None):
    from felis_b200 import workloads

    text = workloads.input_text("sase", slices=3, total_length=0.5, seed_power=2e6, nx=41, beamlets=beamlets)
    extra = f" number_longitudinal_mode={modes[0]}\n number_azimuthal_mode={modes[1]}\n"
    if radial_grids:
        extra += f" radial_grids={radial_grids}\n"
    path = tmp_path / "d.inp"
    path.write_text(text.replace(" ABC_N=", extra + " ABC_N="))
    cfg = fb.Config(str(path))
    p = cfg.params
    beam = cfg.load_beam(0, seed=7)
    assert (np.diff(beam["offsets"]) == 4 * beamlets).all()
    if move:
        move(p, beam)
    g, o = fb.Handle(p), oracle_mod.Oracle(p, threads=4)
    g.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    o.set_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
    for pol, u in enumerate(cfg.load_seed(0)):
        g.upload_field(0, pol, u)
        o.set_field(0, pol, u)
    for it in range(2):
        for e, arg in ((g, (it,)), (o, ())):
            e.update_lattice(it, 0.5)
            e.solve_field(*arg)
            e.transverse_push(*arg)
    for pol in (0, 1):
        assert_bits(g.download_source(0, pol)[1:-1, 1:-1, 1:-1], o.get_field(0, 2 + pol)[1:-1, 1:-1, 1:-1],
                    f"source pol{pol}")
        assert_bits(g.download_field(0, pol)[1:-1], o.get_field(0, pol)[1:-1], f"field pol{pol}")
    assert_bits(g.download_ez()[:, 1:-1], o.get_ez().reshape(g.download_ez().shape)[:, 1:-1], "Ez")
    assert np.any(g.download_source(0, 0) != 0) and np.any(g.download_ez() != 0)


@pytest.mark.parametrize("beamlets", [16, 17, 255, 256, 257, 513])  # 64, 68, 1020, 1024, 1028, 2052 a slice
@pytest.mark.parametrize("modes", [(1, 1), (2, 2)])
def test_around_a_chunk_and_a_warps_part(fb, oracle_mod, tmp_path, beamlets, modes):
    _compare(fb, oracle_mod, tmp_path, beamlets, modes)


@pytest.mark.parametrize("nr, modes", [(513, (1, 1)), (700, (1, 1)), (1100, (1, 1)), (1100, (1, 2)), (600, (2, 2))])
def test_radial_bins_of_several_bands(fb, oracle_mod, tmp_path, nr, modes):
    """Particles by hand in every bin about the ends of the bands and in the
    outermost bins, beside the beam's; they lie beyond the transverse grid."""

    def move(p, beam):
        edges = [k for e in (511, 512, 1023, 1024, nr - 2) for k in range(e - 4, e + 4) if 0 < k < nr - 1]
        rng = np.random.default_rng(nr)
        n = len(beam["x"])
        who = rng.permutation(n)[:8 * len(edges)]
        r = (np.repeat(edges, 8) + rng.uniform(-0.5, 0.5, len(who))) * p.dr
        phi = rng.uniform(0, 2 * np.pi, len(who))
        beam["x"][who], beam["y"][who] = r * np.cos(phi), r * np.sin(phi)
        bins = (np.hypot(beam["x"], beam["y"]) / p.dr + 0.5).astype(int)
        assert p.nr == nr and bins.max() >= min(nr - 2, 512) and (bins <= nr - 2).all()
        assert nr == 513 or ((bins == 511).any() and (bins == 512).any())

    _compare(fb, oracle_mod, tmp_path, 200, modes, nr, move)
