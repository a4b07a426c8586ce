"""The FP64 source deposit at the edges of its chunks, warps and bands: every
cell and every radial bin is the sequential sum in particle order, so source
and Ez equal the CPU restatement bit for bit.
"""
import numpy as np
import pytest

from conftest import assert_bits

pytestmark = pytest.mark.gpu

# particles per slice around the chunk (2048) and its warps' parts (256); a
# 1 GeV beam on a fine grid spreads over several bands of target rows; modes
# (L, F) fill the radial chains' terms and shorten their chunks; more radial
# bins than one band of the radial tables
CASES = {
    "one_beamlet": dict(beamlets=1, nx=41),
    "one_warp_and_one": dict(beamlets=65, nx=41),
    "chunk": dict(beamlets=512, nx=41),
    "chunk_and_four": dict(beamlets=513, nx=42),
    "bands": dict(beamlets=700, nx=151, energy_mev=1000.0),
    "harmonics": dict(beamlets=300, nx=61, harmonics=(1, 2, 3), undulator="QuadPolar", polarity=0.5),
    "modes": dict(beamlets=300, nx=41, modes=(2, 2)),
    "many_modes": dict(beamlets=130, nx=41, modes=(4, 4)),
    "radial_bands": dict(beamlets=200, nx=41, radial_grids=1100),
    "narrow_radial": dict(beamlets=200, nx=41, radial_grids=30, modes=(1, 2)),
}


@pytest.mark.parametrize("name", CASES)
def test_deposit_equals_the_sequential_sums(fb, oracle_mod, tmp_path, name):
    from felis_b200 import workloads

    kw = dict(CASES[name])
    modes, nr = kw.pop("modes", (1, 1)), kw.pop("radial_grids", None)
    text = workloads.input_text("sase", slices=3, total_length=0.5, seed_power=2e6, **kw)
    extra = f" number_longitudinal_mode={modes[0]}\n number_azimuthal_mode={modes[1]}\n"
    if nr:
        extra += f" radial_grids={nr}\n"
    path = tmp_path / "d.inp"
    path.write_text(text.replace(" ABC_N=", extra + " ABC_N="))
    cfg = fb.Config(str(path))
    p = cfg.params
    assert (p.scl_mode, p.scf_mode) == modes
    beam = cfg.load_beam(0, seed=7)
    g, o = fb.Handle(p), oracle_mod.Oracle(p, threads=4)
    g.upload_particles(0, *(beam[k] for k in ("x", "y", "px", "py", "theta", "gamma")), beam["offsets"], beam["weights"])
    o.set_particles(0, *(beam[k] for k in ("x", "y", "px", "py", "theta", "gamma")), beam["offsets"], beam["weights"])
    for h in range(p.num_harmony):
        for pol, u in enumerate(cfg.load_seed(h)):
            g.upload_field(h, pol, u)
            o.set_field(h, pol, u)
    for it in range(2):
        for e, arg in ((g, (it,)), (o, ())):
            e.update_lattice(it, 0.5)
            e.solve_field(*arg)
            e.transverse_push(*arg)
    for h in range(p.num_harmony):
        for pol in (0, 1):
            assert_bits(g.download_source(h, pol)[1:-1, 1:-1, 1:-1], o.get_field(h, 2 + pol)[1:-1, 1:-1, 1:-1],
                        f"source h{h} pol{pol}")
            assert_bits(g.download_field(h, pol)[1:-1], o.get_field(h, pol)[1:-1], f"field h{h} pol{pol}")
    assert_bits(g.download_ez()[:, 1:-1], o.get_ez().reshape(g.download_ez().shape)[:, 1:-1], "Ez")
    assert np.any(g.download_source(0, 0) != 0)
