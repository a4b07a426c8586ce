"""Handles of different grids and mode counts live side by side: the shared
memory that a kernel's launches may take is a limit of the kernel, and a handle
made later, of a smaller grid, takes nothing from one made before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")


def _case(fb, tmp_path, name, nx, modes=(1, 1), radial_grids=None):
    from felis_b200 import workloads

    text = workloads.input_text("sase", slices=3, beamlets=40, nx=nx, total_length=0.3, seed_power=2e6)
    extra = f" number_longitudinal_mode={modes[0]}\n number_azimuthal_mode={modes[1]}\n"
    if radial_grids:
        extra += f" radial_grids={radial_grids}\n"
    path = tmp_path / name
    path.write_text(text.replace(" ABC_N=", extra + " ABC_N="))
    cfg = fb.Config(str(path))
    beam = cfg.load_beam(0, seed=4)

    def handle():
        h = fb.Handle(cfg.params)
        h.upload_particles(0, *(beam[k] for k in KEYS), beam["offsets"], beam["weights"])
        for pol, u in enumerate(cfg.load_seed(0)):
            h.upload_field(0, pol, u)
        return h

    return cfg, handle


def _state(h):
    p = h.download_particles(0)
    return [h.download_field(0, 0), h.download_field(0, 1), h.download_ez()] + [p[k] for k in KEYS]


# planes beyond shared memory (256 and 152 points), within it (102 and 66), and
# radial accumulators of many modes beside those of one
@pytest.mark.parametrize("first, second", [
    (dict(nx=255), dict(nx=151)),
    (dict(nx=101), dict(nx=65)),
    (dict(nx=41, modes=(4, 4), radial_grids=300), dict(nx=41)),
])
def test_a_second_handle_leaves_the_first_running(fb, tmp_path, first, second):
    made = [_case(fb, tmp_path, n, **kw) for n, kw in (("a.inp", first), ("b.inp", second))]
    alone = []
    for _, handle in made:
        h = handle()
        h.run(0, 4)
        alone.append(_state(h))
        h.close()
    a = made[0][1]()
    a.run(0, 2)
    b = made[1][1]()
    b.run(0, 2)
    a.run(2, 4)
    b.run(2, 4)
    for h, want in ((a, alone[0]), (b, alone[1])):
        for x, y in zip(_state(h), want):
            assert np.array_equal(x, y)
