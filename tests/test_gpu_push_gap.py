"""The beam's sums of a drift step (an in-air gap of the undulator line), which
the push launch takes without a deposit: a slice alone (wide CTAs, whose sums
are taken by some of the threads that pushed) and beside so many others that it
gets 128 threads gives the same bits, for slices of fewer particles than a wide
CTA has threads, of about as many and of more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "px", "py", "theta", "gamma")
STEPS = 12  # of one period: units of five periods with gaps of two


def _load(fb, tmp_path, name, harmonics, slices, beamlets):
    from felis_b200 import workloads

    path = workloads.write_input(str(tmp_path / name), kind="sase", slices=slices, beamlets=beamlets, per_beamlet=4,
                                 nx=33, total_length=0.5, units=10, unit_len=0.13, und_len=0.078, seed_power=2e6,
                                 harmonics=harmonics, abc_n=6, undulator="QuadPolar", polarity=0.5)
    cfg = fb.Config(path)
    return cfg, cfg.load_beam(0, seed=4)


@pytest.mark.parametrize("beamlets", [26, 32, 128, 160, 224, 225, 275, 1031])  # 104 to 4124 particles a slice
@pytest.mark.parametrize("harmonics", [(1,), (1, 2), (1, 2, 3)])
def test_sums_in_a_gap_are_those_of_the_pushed_beam(fb, tmp_path, harmonics, beamlets):
    case = _load(fb, tmp_path, "a.inp", harmonics, 5, beamlets)
    h = fb.Handle(case[0].params)
    drift = []
    for it in range(STEPS):
        h.update_lattice(it, 0.5)
        drift.append(h.lattice().drift_flag)
    assert sum(drift) >= 3 and np.abs(np.diff(drift)).sum() >= 3, drift  # several gaps, entered and left
    out = []
    for others in (0, 1100):
        insts = [case] + ([_load(fb, tmp_path, "f.inp", harmonics, others, 8)] if others else [])
        b = fb.Batch([c.params for c, _ in insts])
        for k, (c, beam) in enumerate(insts):
            b.upload_particles(k, *(beam[q] for q in KEYS), beam["offsets"], beam["weights"])
        b.run(0, STEPS)
        out.append(list(b.diagnostics(0, 0, STEPS + 1)) + [b.download_particles(0)[q] for q in KEYS])
    for k, (x, y) in enumerate(zip(*out)):
        assert np.isfinite(x).all() and np.array_equal(x, y), k
