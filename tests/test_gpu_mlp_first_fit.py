"""The first fit of a model allocates device memory once (samples and partial
gradients in one buffer) and the buffer grows whichever of the two outgrows it:
a fit, a prediction and a gradient of other sizes in between leave the results
what they are for a model that only does the one call."""
import numpy as np
import pytest

import cuts_b200 as cb

pytestmark = pytest.mark.gpu


def _data(n, nin, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(n, nin)).astype(np.float32), rng.normal(size=n).astype(np.float32)


def test_sizes_in_any_order():
    nin = 9
    sizes = [40, 700, 33, 5000, 1, 6000]
    p = cb.Mlp(nin, seed=4).get_params()
    m = cb.Mlp(nin, seed=1)
    for n, n_pred in zip(sizes, [2 * s for s in reversed(sizes)]):
        X, t = _data(n, nin, n)
        Xp, _ = _data(n_pred, nin, 7 + n)
        calls = [lambda mdl: np.concatenate([np.ravel(v) for v in mdl.loss_grad(X, t)]), lambda mdl: mdl.predict(Xp),
                 lambda mdl: np.array([mdl.train(X, t, epochs=2, batch=max(1, n // 2), lr=1e-3)])]
        for call in calls:
            fresh = cb.Mlp(nin, seed=2)
            m.set_params(p)
            fresh.set_params(p)
            assert np.array_equal(call(m), call(fresh)), n
            assert np.array_equal(m.get_params(), fresh.get_params()), n


def test_first_fit_allocates_once():
    from torch.profiler import ProfilerActivity, profile
    X, t = _data(4096, 16, 1)
    cb.Mlp(16, seed=0).train(X, t, epochs=1, batch=4096, lr=1e-3)
    m = cb.Mlp(16, seed=1)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        m.train(X, t, epochs=1, batch=4096, lr=1e-3)
    calls = {e.key: e.count for e in prof.key_averages()}
    if not any("LaunchKernel" in key for key in calls):
        pytest.skip("no runtime calls recorded")
    assert sum(c for key, c in calls.items() if key.startswith(("cudaMalloc", "cuMemAlloc"))) == 1, calls
