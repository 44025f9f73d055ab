"""The fused backward kernel at the edges of its row tiles and of its grid."""
import numpy as np
import pytest

from ermod_openacc_b200 import proposal as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 9471, 9505])
def test_gradients_at_tile_edges(engine_lib, n):
    """A CTA takes 32 samples and the grid at most 296 CTAs, whose later tiles add to their first:
    one sample, a tile less one, a tile, a tile and one, and around 296 x 32 = 9472.  Against the
    FP64 chain rule at the device's own activations.  An element is a sum of FP32 products over up
    to 32 rows and 296 CTAs with inner sums of 128 and 128 terms, so its rounding error is below
    (32 + 296 + 256) 2^-24 = 3.5e-5 of the sum of its terms' magnitudes, which here stays under
    five times the largest element of its layer."""
    import mlp_oracle as M
    rng = np.random.default_rng(100 + n)
    p = P.init_params(6)
    L = P.layout()
    for k in ("b1", "b2", "b3", "b4"):
        off, m = L[k]
        p[off:off + m] = rng.normal(0.0, 0.1, m)
    x = rng.uniform(0.0, 3.0, size=(n, 64)).astype(np.float32)
    y = (rng.uniform(size=n) < 0.3).astype(np.float32)
    tr = P.Trainer(p, max_batch=n)
    g, loss = tr.gradients(x, y)
    h = tr.activations(n).astype(np.float64)
    want_loss, want = M.loss_and_grad(p, x, y, tf32_inputs=True, acts=h)
    assert loss == pytest.approx(want_loss, rel=1e-5)
    for k in ("W1", "b1", "W2", "b2", "W3", "b3", "w4", "b4"):
        off, m = L[k]
        a, b = g[off:off + m], want[off:off + m]
        assert np.max(np.abs(a - b)) <= 2e-4 * np.max(np.abs(b)) + 1e-7, k
    again, _ = tr.gradients(x, y)
    assert np.array_equal(g, again)
    tr.close()
