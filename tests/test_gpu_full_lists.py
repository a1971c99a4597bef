"""Lists of deferred parents that are full, by the number of their pieces
(CUTS_FUSE_PIECES) or of their places (an arena so small that it has 64): the
parents beyond are counted where they are found.  Counts and level sizes of the
fused pairs and of the edge count (with and without rows of the dense core)
equal the oracle's."""
import functools

import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs

pytestmark = pytest.mark.gpu

EDGES = {n: cb.named_query_arcs(n) for n in ("4-cycle", "5-cycle", "house")}
PAIRS = {n: cb.named_query_arcs(n) for n in ("triangle", "4-clique+pendant")}
PAIRS["4-clique"] = (4, [(a, b) for a in range(4) for b in range(4) if a != b])
PAIRS["triangle+pendant"] = (4, cb.named_query_arcs("triangle")[1] + [(0, 3), (3, 0)])


def _hubs(hubs, deg, n, ring, seed):
    """`hubs` vertices, joined to one another and to `deg` of n others each,
    which form a ring joined at distances 1..ring."""
    rng = np.random.default_rng(seed)
    a, b = np.triu_indices(hubs, 1)
    src, dst = [a], [b]
    for h in range(hubs):
        src.append(np.full(deg, h))
        dst.append(hubs + rng.choice(n, deg, replace=False))
    for d in range(1, ring + 1):
        src.append(hubs + np.arange(n))
        dst.append(hubs + (np.arange(n) + d) % n)
    src, dst = np.concatenate(src), np.concatenate(dst)
    src, dst = np.concatenate([src, dst]).astype(np.uint32), np.concatenate([dst, src]).astype(np.uint32)
    oo, oa, io, ia, s, d = csr_from_arcs(hubs + n, src, dst)
    return hubs + n, oo, oa, s, d


@functools.lru_cache(None)
def _case(shape):
    n, oo, oa, s, d = _hubs(*shape, seed=3)
    od = O.Graph.from_arrays(n, s, d)
    want = {}
    for name, (k, arcs) in {**PAIRS, **EDGES}.items():
        if shape[0] == 40 and name in ("5-cycle", "house"):
            continue  # many seconds in the oracle
        q = cb.Query.from_arcs(k, arcs)
        want[name] = q, O.count(od, O.Graph.from_arcs(k, arcs), q.order)[:2]
    return n, oo, oa, want


@pytest.mark.parametrize("limit", ["pieces 0", "pieces 7", "pieces 90", "places"])
@pytest.mark.parametrize("shape", [(40, 150, 400, 2), (4, 1100, 1300, 1)])  # core rows in k_edges: from 1,024 neighbours on
def test_full_lists(shape, limit, monkeypatch):
    n, oo, oa, want = _case(shape)
    g = cb.Graph.from_csr(n, oo, oa)
    if limit == "places":
        g.set_arena_bytes(1 << 20)
    else:
        monkeypatch.setenv("CUTS_FUSE_PIECES", limit.split()[1])
    for name, (q, (cnt, lv)) in want.items():
        assert cnt > 0
        for split in (None, "3") if name in PAIRS else (None,):
            if split:
                monkeypatch.setenv("CUTS_FUSE_SPLIT", split)
            r = g.count(q, stats=True)
            assert (r.count, r.level_sizes) == (cnt, lv), (name, split)
            assert g.count(q, flags=cb.FLAG_SYMMETRY_BREAK).count == cnt, (name, split)
            monkeypatch.delenv("CUTS_FUSE_SPLIT", raising=False)
    g.close()
