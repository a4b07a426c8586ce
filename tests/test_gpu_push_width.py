"""The push launch gives the slices of a small ensemble wider CTAs: the same
instance alone (896, 640 or 512 threads per slice by harmonic count) and beside
others that leave it a half, a third and the smallest share of an SM gives the
same bits -- particles, fields, and the sums behind the diagnostics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")
STEPS = 4


def _load(fb, tmp_path, name, harmonics, slices, beamlets):
    from felis_b200 import workloads

    path = workloads.write_input(str(tmp_path / name), kind="sase", slices=slices, beamlets=beamlets, per_beamlet=4,
                                 nx=33, total_length=0.3, seed_power=2e6, harmonics=harmonics, abc_n=6,
                                 undulator="QuadPolar", polarity=0.5)
    cfg = fb.Config(path)
    return cfg, cfg.load_beam(0, seed=4)


@pytest.mark.parametrize("beamlets", [20, 300, 1031])  # 80 to 4124 particles a slice, odd counts over 128
@pytest.mark.parametrize("harmonics", [(1,), (1, 2), (1, 2, 3), (1, 2, 3, 4, 5)])
def test_the_width_of_a_slice_changes_nothing(fb, tmp_path, harmonics, beamlets):
    first = None
    case = _load(fb, tmp_path, "a.inp", harmonics, 5, beamlets)
    for others in (0, 200, 400, 1100):
        insts = [case] + ([_load(fb, tmp_path, "f.inp", harmonics, others, 8)] if others else [])
        b = fb.Batch([c.params for c, _ in insts])
        for k, (c, beam) in enumerate(insts):
            b.upload_particles(k, *(beam[q] for q in KEYS), beam["offsets"], beam["weights"])
        b.run(0, STEPS)
        out = [b.download_particles(0)[q] for q in KEYS]
        out += [b.download_field(0, h, pol) for h in range(len(harmonics)) for pol in (0, 1)]
        out += list(b.diagnostics(0, 0, STEPS + 1))
        if first is None:
            first = out
        for k, (x, y) in enumerate(zip(first, out)):
            assert np.array_equal(x, y), (others, k)
    assert all(np.isfinite(x).all() for x in first) and np.abs(first[6]).max() > 0
