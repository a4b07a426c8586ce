"""Gradients of the taper-surrogate network over the sizes at which the GEMMs
change their tiles: column tiles of 32, 64 or the whole width by the number of
128-row tiles, ragged last tiles in both directions, fewer rows of dz^T than a
tile, inputs wider than the hidden layers.

The CPU side rounds to BF16 where the GPU does.  Accumulation order and the
hardware tanh can move a value by one rounding (2^-8 of it) at each of the
three layers that dz crosses and once more in the forward pass it is computed
from: 4 x 2^-8 = 1.6e-2 of the norm for a block of one row, where nothing
averages.
"""
import numpy as np
import pytest
from test_gpu_mlp import cpu_gradients, random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_in,width,n_out,rows", [
    (38, 256, 33, 1), (38, 256, 33, 129), (38, 256, 33, 1153), (38, 256, 33, 2433),
    (250, 128, 1, 130), (17, 128, 128, 1281), (256, 256, 256, 515), (1, 256, 129, 2305)])
def test_gradients_over_the_tile_rules(fb, n_in, width, n_out, rows):
    rng = np.random.default_rng(rows + n_in)
    m = fb.MLP(n_in, width, n_out, seed=3)
    p = random_params(m, rng)
    m.set_params(p)
    x = rng.normal(0, 1, (rows, n_in)).astype(np.float32)
    t = rng.normal(0, 1, (rows, n_out)).astype(np.float32)
    g, loss = m.gradients(x, t)
    ref, ref_loss, _ = cpu_gradients(m.unflatten(p), x, t)
    np.testing.assert_allclose(loss, ref_loss, rtol=1.6e-2)
    for k, ((gW, gb), (rW, rb)) in enumerate(zip(m.unflatten(g), ref)):
        assert np.linalg.norm(gW - rW) < 1.6e-2 * np.linalg.norm(rW), (k, "W")
        assert np.linalg.norm(gb - rb) < 1.6e-2 * np.linalg.norm(rb), (k, "b")
    m.close()


def test_an_epoch_reads_every_row_once(fb):
    """300 rows in batches of 128 (the last holds 44): with a step of zero the
    epoch's loss is the mean squared error over all rows."""
    rng = np.random.default_rng(9)
    m = fb.MLP(38, 256, 33, seed=3)
    x = rng.normal(0, 1, (300, 38)).astype(np.float32)
    t = rng.normal(0, 1, (300, 33)).astype(np.float32)
    want = np.mean((m.forward(x).astype(np.float64) - t) ** 2)
    m.set_data(x, t)
    hist = m.train(epochs=2, batch=128, lr=0.0, weight_decay=0.0)
    np.testing.assert_allclose(hist, [want, want], rtol=1e-5)
    m.close()
