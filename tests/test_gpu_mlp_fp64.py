"""The order model's sums are in FP64: its gradient and loss are within one
rounding to FP32 of the float64 restatement's, plus both sides' float64 rounding
(test_gpu_mlp_tiles' bound of a float32 chain, 2^-29 of it for each side)."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import mlp_ref
from tests.test_gpu_mlp_tiles import _bounds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nin,n", [(1, 33), (16, 1), (16, 4096), (17, 32 * 148 + 1), (32, 5000)])
def test_gradient_within_one_rounding(nin, n):
    rng = np.random.default_rng(1000 * nin + n)
    X = rng.normal(size=(n, nin)).astype(np.float32)
    t = rng.normal(size=n).astype(np.float32)
    m = cb.Mlp(nin, seed=nin)
    p = m.get_params()
    loss, g = m.loss_grad(X, t)
    wl, wg = mlp_ref.loss_grad(p, X, t)
    assert abs(loss - wl) <= 2.0 ** -24 * wl * (1 + 1e-6)
    assert np.all(np.abs(g - wg) <= 2.0 ** -24 * np.abs(wg) + 2.0 ** -28 * _bounds(p, X, t) + 2.0 ** -149)
