"""Samples and partial gradients grow each by themselves: a prediction over more
rows than the fit had leaves the partials where they are (no memory is given
back, one small block is taken), and a fit of more blocks after it works on
both, with the results of a model that does only that call."""
import numpy as np
import pytest

import cuts_b200 as cb

pytestmark = pytest.mark.gpu


def _data(n, nin, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(n, nin)).astype(np.float32), rng.normal(size=n).astype(np.float32)


@pytest.mark.parametrize("rows,held", [(672, 937), (4096, 6000), (33, 24001)])
def test_prediction_of_more_rows_keeps_the_partials(rows, held):
    from torch.profiler import ProfilerActivity, profile
    X, t = _data(rows, 16, 1)
    Xp, _ = _data(held, 16, 2)
    cb.Mlp(16, seed=0).train(X, t, epochs=1, batch=rows, lr=1e-3)
    m = cb.Mlp(16, seed=1)
    m.train(X, t, epochs=1, batch=rows, lr=1e-3)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        m.predict(Xp)
    calls = {e.key: e.count for e in prof.key_averages()}
    if not any("LaunchKernel" in key for key in calls):
        pytest.skip("no runtime calls recorded")
    assert sum(c for key, c in calls.items() if key.startswith(("cudaMalloc", "cuMemAlloc"))) == 1, calls
    assert not any(key.startswith(("cudaFree", "cuMemFree")) for key in calls), calls


# (rows, batch) of a fit or (rows, 0) of a prediction, in turn
@pytest.mark.parametrize("order", [
    [(500, 0), (500, 500), (900, 0), (400, 400), (4000, 4000), (9000, 0), (9000, 9000)],
    [(5000, 64), (300, 0), (5000, 5000), (5001, 0), (5002, 5002), (1, 1)],
    [(9000, 0), (40, 40), (700, 700), (9001, 0), (4700, 4700), (9001, 0)],
])
def test_growth_in_turn(order):
    nin = 12
    p = cb.Mlp(nin, seed=4).get_params()
    m = cb.Mlp(nin, seed=1)
    for n, batch in order:
        X, t = _data(n, nin, n)
        fresh = cb.Mlp(nin, seed=2)
        got = []
        for mdl in (m, fresh):
            mdl.set_params(p)
            if batch:
                got.append(mdl.train(X, t, epochs=1, batch=batch, lr=1e-3))
                got[-1] = np.concatenate([[got[-1]], mdl.get_params()])
            else:
                got.append(mdl.predict(X))
        assert np.array_equal(got[0], got[1]), (n, batch)
