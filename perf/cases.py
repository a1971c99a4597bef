"""Performance cases: the engine's public calls over the sizes it is used at.

A case is a dict of plain values.  ``listed()`` gives the fixed cases,
``draw(rng)`` more of the same ranges, ``prepare(case, seed)`` what a program
holds before the call (graph resident on the GPU, query, batch, model, host
arrays), ``run(state)`` one pass through the public entry points,
``work(case)`` the bytes and operations a pass cannot do without and
``exact(case, seed)`` the 64-bit value of floating-point outputs.

Kinds of case:

* count    -- one exact count on a resident graph (``Graph.count``).
* log      -- counts with level sizes of several small queries, one call each
              (what training data for the learned order are made of).
* batch    -- many queries in one call (``Batch.run``).
* noalloc  -- many queries on caller-owned device buffers, plain counting
              (``count_noalloc``).
* load     -- a host CSR made resident, counted once, released
              (``Graph.from_csr`` + ``Graph.count``).
* mlp      -- the order model: training from given weights, then prediction.

Graphs are drawn on the GPU from the seed: "er" (every pair equally likely),
"cl" (Chung-Lu power law: endpoints by weight) or "dcl" (the same, arcs kept
one-way).
"""
import math

import numpy as np
import torch

import cuts_b200 as cb

# directed four-vertex query: two sources feeding a common chain
FEED = (4, [(0, 2), (1, 2), (0, 3), (2, 3)])
# directed triangle with one mutual edge
MUTUAL3 = (3, [(0, 1), (1, 0), (1, 2), (0, 2)])


def listed():
    return [
        # smallest: a quick exact count on a small uniform graph, where
        # latency and launches are what a caller waits for
        {"name": "er_4cycle", "kind": "count", "graph": "er", "n": 10000, "m": 40000, "gamma": 0.0, "cap": 0.0,
         "query": "4-cycle", "flags": 0, "chunks": 1, "levels": True},
        # level-size logging for the learned order: one small query after another
        {"name": "order_log", "kind": "log", "graph": "cl", "n": 3000, "m": 12000, "gamma": 2.2, "cap": 60.0,
         "kmin": 4, "kmax": 6, "nq": 12, "p": 0.3, "qseed": 1, "flags": 0},
        # the mid power-law graph, every embedding enumerated, root slices
        {"name": "triangle_plain", "kind": "count", "graph": "cl", "n": 1000000, "m": 10000000, "gamma": 2.1,
         "cap": 20000.0, "query": "triangle", "flags": 0, "chunks": 4, "levels": True},
        # the headline benchmark's second query, symmetry breaking
        {"name": "clique4_pendant_sym", "kind": "count", "graph": "cl", "n": 1000000, "m": 10000000, "gamma": 2.1,
         "cap": 20000.0, "query": "4-clique+pendant", "flags": 1, "chunks": 4, "levels": False},
        # the largest graph of the batched workload: beyond the L2 cache
        {"name": "triangle_sym_4m", "kind": "count", "graph": "cl", "n": 4000000, "m": 40000000, "gamma": 2.2,
         "cap": 20000.0, "query": "triangle", "flags": 1, "chunks": 4, "levels": False},
        # cycles: no level contains the one before, tries held in memory
        {"name": "5cycle_sym", "kind": "count", "graph": "cl", "n": 200003, "m": 1000000, "gamma": 2.3, "cap": 400.0,
         "query": "5-cycle", "flags": 1, "chunks": 1, "levels": False},
        # house, plain: a two-list join below the last level
        {"name": "house_plain", "kind": "count", "graph": "cl", "n": 100000, "m": 500000, "gamma": 2.3, "cap": 300.0,
         "query": "house", "flags": 0, "chunks": 1, "levels": True},
        # directed data and query: both list directions, signatures tested
        {"name": "feed_directed", "kind": "count", "graph": "dcl", "n": 150001, "m": 1500000, "gamma": 2.2,
         "cap": 1500.0, "query": "feed", "flags": 0, "chunks": 1, "levels": True},
        # a mixed batch against one resident graph
        {"name": "batch_mixed", "kind": "batch", "graph": "cl", "n": 200000, "m": 1600000, "gamma": 2.2, "cap": 1000.0,
         "kmin": 3, "kmax": 4, "nq": 64, "p": 0.4, "qseed": 2, "flags": 1},
        # caller-owned buffers, nothing allocated
        {"name": "noalloc_mixed", "kind": "noalloc", "graph": "cl", "n": 50001, "m": 300000, "gamma": 2.2,
         "cap": 400.0, "kmin": 2, "kmax": 4, "nq": 16, "p": 0.4, "qseed": 3, "flags": 0},
        # from host arrays to a count: copy, layout, count, release
        {"name": "load_triangle", "kind": "load", "graph": "cl", "n": 1000000, "m": 10000000, "gamma": 2.1,
         "cap": 20000.0, "query": "triangle", "flags": 1, "chunks": 1, "levels": False},
        # the order model: mini-batch training on logged level sizes, then
        # prediction of held-out rows
        {"name": "mlp_fit_predict", "kind": "mlp", "rows": 24000, "held": 6000, "epochs": 8, "batch": 4096, "lr": 2e-3},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["count", "count", "count", "count", "log", "batch", "noalloc", "load", "mlp"])
    if kind == "mlp":
        return {"kind": "mlp", "rows": _log_uniform(rng, 500, 24000), "held": _log_uniform(rng, 100, 6000),
                "epochs": rng.randint(2, 8), "batch": rng.choice([1024, 2048, 4096]), "lr": 2e-3}
    gamma = round(rng.uniform(2.1, 2.4), 2)
    if kind == "log":
        n = _log_uniform(rng, 1000, 6000)
        return {"kind": "log", "graph": "cl", "n": n, "m": 4 * n, "gamma": gamma, "cap": 60.0, "kmin": 4, "kmax": 6,
                "nq": rng.randint(4, 12), "p": 0.3, "qseed": rng.getrandbits(20), "flags": rng.choice([0, 1])}
    if kind == "batch":
        n = _log_uniform(rng, 20000, 200000)
        return {"kind": "batch", "graph": "cl", "n": n, "m": int(n * rng.uniform(3, 8)), "gamma": gamma,
                "cap": 600.0, "kmin": 3, "kmax": 4, "nq": rng.randint(8, 64), "p": round(rng.uniform(0.2, 0.6), 2),
                "qseed": rng.getrandbits(20), "flags": 1}
    if kind == "noalloc":
        n = _log_uniform(rng, 5000, 50000)
        return {"kind": "noalloc", "graph": rng.choice(["cl", "er", "dcl"]), "n": n, "m": int(n * rng.uniform(3, 6)),
                "gamma": gamma, "cap": 400.0, "kmin": 2, "kmax": 4, "nq": rng.randint(4, 16), "p": 0.4,
                "qseed": rng.getrandbits(20), "flags": 0}
    if kind == "load":
        n = _log_uniform(rng, 50000, 1000000)
        return {"kind": "load", "graph": "cl", "n": n, "m": int(n * rng.uniform(3, 10)), "gamma": gamma,
                "cap": 5000.0, "query": "triangle", "flags": 1, "chunks": 1, "levels": False}
    flags = rng.choice([0, 1])
    form = rng.choice(["er", "tri", "clique", "five", "directed"])
    if form == "er":
        n = _log_uniform(rng, 5000, 200000)
        return {"kind": "count", "graph": "er", "n": n, "m": int(n * rng.uniform(2, 6)), "gamma": 0.0, "cap": 0.0,
                "query": rng.choice(["triangle", "4-cycle", "5-cycle", "house", "3-star", "4-path"]), "flags": flags,
                "chunks": rng.choice([1, 4]), "levels": True}
    if form == "directed":
        n = _log_uniform(rng, 5000, 150000)
        return {"kind": "count", "graph": "dcl", "n": n, "m": int(n * rng.uniform(3, 10)), "gamma": gamma,
                "cap": 600.0, "query": rng.choice(["feed", "mutual3"]), "flags": 0, "chunks": 1, "levels": True}
    if form == "five":
        n = _log_uniform(rng, 5000, 200000)
        return {"kind": "count", "graph": "cl", "n": n, "m": int(n * rng.uniform(2, 5)), "gamma": round(gamma + 0.1, 2),
                "cap": 200.0, "query": rng.choice(["5-cycle", "house", "4-cycle"]), "flags": flags,
                "chunks": rng.choice([1, 4]), "levels": bool(rng.getrandbits(1))}
    n = _log_uniform(rng, 20000, 1000000)
    return {"kind": "count", "graph": "cl", "n": n, "m": int(n * rng.uniform(3, 10)), "gamma": gamma, "cap": 5000.0,
            "query": "triangle" if form == "tri" else "4-clique+pendant", "flags": flags if form == "tri" else 1,
            "chunks": rng.choice([1, 4]), "levels": bool(rng.getrandbits(1))}


# ---- inputs -----------------------------------------------------------------

def _csr(n, src, dst):
    """CSR (int64 offsets, int64 sorted lists) of distinct arcs, on the GPU."""
    key = torch.unique(src * n + dst)
    off = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return off, key % n


def _pairs(case, seed):
    """m distinct ordered pairs (a != b), unordered ones for "er" and "cl"."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n, m = case["n"], case["m"]
    t = m + m // 4 + 1024
    if case["graph"] == "er":
        a = torch.randint(n, (t,), device="cuda", generator=gen)
        b = torch.randint(n, (t,), device="cuda", generator=gen)
    else:
        u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen).clamp_(min=1e-12)
        w = (2.0 * u ** (-1.0 / (case["gamma"] - 1.0))).clamp_(max=case["cap"])
        cum = torch.cumsum(w, 0)

        def end():
            r = torch.rand(t, dtype=torch.float64, device="cuda", generator=gen) * cum[-1]
            return torch.searchsorted(cum, r).clamp_(max=n - 1)

        a, b = end(), end()
    if case["graph"] != "dcl":
        a, b = torch.minimum(a, b), torch.maximum(a, b)
    key = torch.unique((a * n + b)[a != b])
    if key.numel() > m:
        key = key[torch.randperm(key.numel(), device="cuda", generator=gen)[:m]]
    return key // n, key % n


def _graph_arrays(case, seed):
    """(out CSR, in CSR or None) on the GPU."""
    a, b = _pairs(case, seed)
    n = case["n"]
    if case["graph"] == "dcl":
        return _csr(n, a, b), _csr(n, b, a)
    return _csr(n, torch.cat([a, b]), torch.cat([b, a])), None


def _host(csr):
    if csr is None:
        return None, None
    off, adj = csr
    return off.cpu().numpy().astype(np.uint64), adj.to(torch.int32).cpu().numpy().view(np.uint32)


def _resident(case, seed):
    out, inn = _graph_arrays(case, seed)
    oo, oa = _host(out)
    io, ia = _host(inn)
    return cb.Graph.from_csr(case["n"], oo, oa, io, ia)


def _query(name):
    k, arcs = {"feed": FEED, "mutual3": MUTUAL3}.get(name) or cb.named_query_arcs(name)
    return cb.Query.from_arcs(k, arcs)


def _queries(case):
    """The case's random connected queries; on directed data, some of their
    arcs one-way.  A program asks the same questions of another graph, so they
    do not change with the inputs' seed."""
    rng = np.random.default_rng(case["qseed"])
    qs = []
    for i in range(case["nq"]):
        k = int(rng.integers(case["kmin"], case["kmax"] + 1))
        arcs = cb.random_query_arcs(k, case["p"], int(rng.integers(1 << 30)))
        if case["graph"] == "dcl":
            arcs = [x for x in arcs if x[0] < x[1] or rng.random() < 0.6]
        qs.append(cb.Query.from_arcs(k, arcs))
    return qs


_HIDDEN, _IN = 64, 16


def _mlp_inputs(case, seed):
    """Initial weights (He uniform) and rows as the order logger makes them:
    small counts, fractions and logarithms; targets are log table sizes."""
    rng = np.random.default_rng(seed)

    def uni(fan, *shape):
        lim = math.sqrt(6.0 / fan)
        return rng.uniform(-lim, lim, shape).astype(np.float32)

    p = np.concatenate([uni(_IN, _HIDDEN * _IN), np.zeros(_HIDDEN, np.float32), uni(_HIDDEN, _HIDDEN * _HIDDEN),
                        np.zeros(_HIDDEN, np.float32), uni(_HIDDEN, _HIDDEN), np.zeros(1, np.float32)])

    def rows(n):
        x = np.concatenate([rng.integers(1, 6, (n, 4)) / 4.0, rng.random((n, 8)), rng.uniform(0, 3, (n, 4))], 1)
        y = 6 * x[:, 12] - 2 * x[:, 0] + 3 * x[:, 5] * x[:, 13] + rng.normal(0, 0.3, n)
        return x.astype(np.float32), np.log1p(np.exp(y)).astype(np.float32)

    x, y = rows(case["rows"])
    return p, x, y, rows(case["held"])[0]


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "mlp":
        st["p"], st["x"], st["y"], st["held"] = _mlp_inputs(case, seed)
        st["model"] = cb.Mlp(_IN, seed=0)
    elif kind == "load":
        out, _ = _graph_arrays(case, seed)
        off, adj = out[0].cpu().pin_memory(), out[1].to(torch.int32).cpu().pin_memory()
        st["keep"] = (off, adj)  # the pinned buffers behind the arrays
        st["off"], st["adj"] = off.numpy().view(np.uint64), adj.numpy().view(np.uint32)
        st["query"] = _query(case["query"])
    elif kind == "noalloc":
        out, inn = _graph_arrays(case, seed)
        base = out[1].numel()

        def info(off, shift):
            return torch.stack([off[:-1] + shift, off[1:] - off[:-1]], 1).to(torch.int32).contiguous()

        st["info_out"] = info(out[0], 0)
        st["info_in"] = info(inn[0], base) if inn else None
        st["adj"] = (torch.cat([out[1], inn[1]]) if inn else out[1]).to(torch.int32).contiguous()
        st["queries"] = _queries(case)
        st["counts"] = torch.empty(case["nq"], dtype=torch.int64, device="cuda")
    else:
        st["graph"] = _resident(case, seed)
        if kind == "count":
            st["query"] = _query(case["query"])
        else:
            st["queries"] = _queries(case)
            if kind == "batch":
                st["batch"] = st["graph"].batch(st["queries"], flags=case["flags"])
    return st


# ---- one pass ---------------------------------------------------------------

def _result(r, levels):
    return [r.count, np.array(r.level_sizes, np.int64)] if levels else [r.count]


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "count":
        return _result(st["graph"].count(st["query"], chunks=case["chunks"], flags=case["flags"],
                                         stats=case["levels"]), case["levels"])
    if kind == "log":
        rs = [st["graph"].count(q, flags=case["flags"], stats=True) for q in st["queries"]]
        levels = np.zeros((len(rs), case["kmax"]), np.int64)
        for row, r in zip(levels, rs):
            row[:len(r.level_sizes)] = r.level_sizes
        return [np.array([r.count for r in rs], np.int64), levels]
    if kind == "batch":
        counts, status, _ = st["batch"].run()
        return [np.array(counts, np.int64), np.array(status, np.int64)]
    if kind == "noalloc":
        info_in = st["info_in"]
        cb.count_noalloc(st["info_out"].data_ptr(), info_in.data_ptr() if info_in is not None else None,
                         st["adj"].data_ptr(), case["n"], st["queries"], st["counts"].data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
        return st["counts"]
    if kind == "load":
        g = cb.Graph.from_csr(case["n"], st["off"], st["adj"])
        r = g.count(st["query"], chunks=case["chunks"], flags=case["flags"])
        info = g.info()
        g.close()
        return [int(x) for x in info] + [r.count]
    m = st["model"]
    m.set_params(st["p"])
    loss = m.train(st["x"], st["y"], epochs=case["epochs"], batch=case["batch"], lr=case["lr"])
    return {"loss": loss, "params": m.get_params(), "held": m.predict(st["held"])}


# ---- what a pass cannot do without -------------------------------------------

def work(case):
    if case["kind"] == "mlp":
        rows = case["rows"] * case["epochs"]
        macs = _IN * _HIDDEN + _HIDDEN * _HIDDEN + _HIDDEN
        return {"bytes": 4.0 * (_IN + 1) * rows + 4.0 * (_IN + 1) * case["held"],
                "flops": 6.0 * macs * rows + 2.0 * macs * (case["rows"] + case["held"])}
    arcs = case["m"] * (1 if case["graph"] == "dcl" else 2)
    dirs = 2 if case["graph"] == "dcl" else 1
    # the lists once and each vertex's place and length once, for each query;
    # made resident: the host arrays read and the device's written as well
    graph = dirs * (4.0 * arcs + 8.0 * case["n"])
    if case["kind"] == "load":
        return {"bytes": 3.0 * graph, "flops": 0.0}
    return {"bytes": graph * case.get("nq", 1), "flops": 0.0}


# ---- 64-bit results ------------------------------------------------------------

def exact(case, seed):
    """The model's weights, final loss and predictions in 64 bits; counts are
    whole numbers and have no such value."""
    if case["kind"] != "mlp":
        return None
    p32, x32, y32, held32 = _mlp_inputs(case, seed)
    p = torch.from_numpy(p32).double()
    x, y, held = (torch.from_numpy(a).double() for a in (x32, y32, held32))
    h, d = _HIDDEN, _IN
    cuts = [h * d, h, h * h, h, h, 1]

    def forward(w, v):
        w1, b1, w2, b2, w3, b3 = torch.split(w, cuts)
        z = torch.relu(v @ w1.view(h, d).T + b1)
        z = torch.relu(z @ w2.view(h, h).T + b2)
        return z @ w3 + b3

    lr, b1, b2, eps = (float(np.float32(v)) for v in (case["lr"], 0.9, 0.999, 1e-8))
    m, v, step = torch.zeros_like(p), torch.zeros_like(p), 0
    batch = case["batch"] if 0 < case["batch"] <= len(x) else len(x)
    for _ in range(case["epochs"]):
        for s in range(0, len(x), batch):
            w = p.clone().requires_grad_(True)
            loss = torch.mean((forward(w, x[s:s + batch]) - y[s:s + batch]) ** 2)
            (g,) = torch.autograd.grad(loss, w)
            step += 1
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p - lr * (m / (1 - b1 ** step)) / (torch.sqrt(v / (1 - b2 ** step)) + eps)
    return {"loss": float(torch.mean((forward(p, x) - y) ** 2)), "params": p, "held": forward(p, held)}
