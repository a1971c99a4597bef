"""The cost model's tiled training kernel at the edges of its tiles (32 rows,
one block per SM before blocks take several tiles; 1..32 features), against
the float64 restatement.  The tolerance is an a-priori bound: every value is
a chain of at most c fused multiply-adds in float32, so it is off by at most
c * 2**-24 times the same expression over absolute values (first order; a
factor 2 covers the rest), and a unit whose pre-activation is smaller than
its own bound may be on either side of the ReLU."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def _bounds(p, X, t):
    """Per-parameter bound on the float32 gradient's error."""
    n, nin = X.shape
    W1, b1, W2, b2, W3, b3 = mlp_ref.unpack(p.astype(np.float64), nin)
    _, (a1, h1, a2, h2) = mlp_ref.forward(p, X)
    y = h2 @ W3 + b3
    Xa = np.abs(X.astype(np.float64))
    # chains: features, two hidden layers, output, loss, both layers back,
    # a block's rows, the final rounding
    c = 2.0 * (nin + 64 + 64 + 8 + 64 + 64 + 32 * -(-n // (32 * 148)) + 8) * 2.0 ** -24
    A1 = Xa @ np.abs(W1).T + np.abs(b1)
    A2 = A1 @ np.abs(W2).T + np.abs(b2)
    Ay = A2 @ np.abs(W3) + abs(b3) + np.abs(t)
    flip2, flip1 = np.abs(a2) <= c * A2, np.abs(a1) <= c * A1
    dy = 2 * np.abs(y - t) / n
    Ady = 2 * Ay / n                       # c * Ady bounds dy's error
    d2 = dy[:, None] * np.abs(W3) * (a2 > 0)
    e2 = c * Ady[:, None] * np.abs(W3) + flip2 * dy[:, None] * np.abs(W3)
    d1 = (d2 @ np.abs(W2)) * (a1 > 0)
    e1 = e2 @ np.abs(W2) + c * (Ady[:, None] * np.abs(W3)) @ np.abs(W2) + flip1 * (d2 @ np.abs(W2))
    gW3 = (c * Ady[:, None] * A2 + dy[:, None] * c * A2).sum(0) + c * (dy[:, None] * A2).sum(0)
    gb3 = np.array([(c * Ady).sum() + c * dy.sum()])
    gW2 = e2.T @ A1 + (d2 + e2).T @ (c * A1) + c * d2.T @ A1
    gb2 = e2.sum(0) + c * d2.sum(0)
    gW1 = e1.T @ Xa + c * d1.T @ Xa
    gb1 = e1.sum(0) + c * d1.sum(0)
    return np.concatenate([gW1.ravel(), gb1, gW2.ravel(), gb2, gW3, gb3])


@pytest.mark.parametrize("nin", [1, 15, 16, 17, 32])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 32 * 148, 32 * 148 + 1])
def test_gradient_at_tile_edges(nin, n):
    rng = np.random.default_rng(100 * nin + n)
    X = rng.normal(size=(n, nin)).astype(np.float32)
    t = rng.normal(size=n).astype(np.float32)
    m = cb.Mlp(nin, seed=nin)
    p = m.get_params()
    loss, g = m.loss_grad(X, t)
    wl, wg = mlp_ref.loss_grad(p, X, t)
    assert abs(loss - wl) <= 1e-5 * wl + 1e-7
    assert np.all(np.abs(g - wg) <= _bounds(p, X, t) + 1e-12)
    # the same rows twice: nothing is left over, and sums have a fixed order
    loss2, g2 = m.loss_grad(X, t)
    assert loss2 == loss and np.array_equal(g, g2)
