"""Fused pairs on symmetric graphs with self-loops: a vertex's own entry in its
list is no neighbour -- not as a partner, not in the rows of the dense core, not
in a folded pendant's list.  Against the oracle, over plain and orbit folds,
rows (sets of 32 and more of the 1,024 highest ids), sets below the core and
deferred parents; loops on every vertex, on some, on the hubs only."""
import functools

import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs

pytestmark = pytest.mark.gpu


def _sym(edges):
    return [a for e in edges for a in (e, e[::-1])]


def _clique(k):
    return _sym([(a, b) for a in range(k) for b in range(a)])


QUERIES = {
    "triangle": (3, _clique(3)),
    "triangle+pendant": (4, _clique(3) + _sym([(0, 3)])),
    "4-clique": (4, _clique(4)),
    "4-clique+pendant": (5, _clique(4) + _sym([(0, 4)])),
    "diamond+pendant": (5, _sym([(0, 1), (1, 2), (2, 3), (3, 0), (0, 2), (0, 4)])),
    # the pendant on a vertex matched before the pair, in an orbit of its own
    "tailed": (5, _clique(3) + _sym([(0, 3), (3, 4)])),
    "5-clique": (5, _clique(5)),
}


@functools.lru_cache(None)
def _graph(shape, loops):
    rng = np.random.default_rng(11)
    if shape == "dense":  # all in the core
        n = 90
        a, b = np.triu_indices(n, 1)
        keep = rng.random(len(a)) < 0.5
        a, b = a[keep], b[keep]
    else:  # a dense part of high degree over sparse vertices below the core
        n = 1500
        a, b = np.triu_indices(60, 1)
        keep = rng.random(len(a)) < 0.7
        a, b = a[keep], b[keep]
        s = rng.integers(0, n, (2, 3000))
        a, b = np.concatenate([a, s[0]]), np.concatenate([b, s[1]])
        a, b = a[a != b], b[a != b]
    at = {"all": np.arange(n), "some": rng.choice(n, n // 3, replace=False), "hubs": np.arange(20)}[loops]
    perm = rng.permutation(n)
    src, dst = np.concatenate([a, b, at]), np.concatenate([b, a, at])
    oo, oa, _, _, s, d = csr_from_arcs(n, perm[src].astype(np.uint32), perm[dst].astype(np.uint32))
    od = O.Graph.from_arrays(n, s, d)
    want = {}
    for name, (k, arcs) in QUERIES.items():
        q = cb.Query.from_arcs(k, arcs)
        want[name] = O.count(od, O.Graph.from_arcs(k, arcs), q.order)[:2]
    return n, oo, oa, want


@pytest.mark.parametrize("split", [None, "0", "7"])
@pytest.mark.parametrize("loops", ["all", "some", "hubs"])
@pytest.mark.parametrize("shape", ["dense", "mixed"])
def test_counts_with_loops(shape, loops, split, monkeypatch):
    n, oo, oa, want = _graph(shape, loops)
    if split:
        monkeypatch.setenv("CUTS_FUSE_SPLIT", split)
    g = cb.Graph.from_csr(n, oo, oa)
    for name, (k, arcs) in QUERIES.items():
        q = cb.Query.from_arcs(k, arcs)
        cnt, lv = want[name]
        assert cnt > 0
        for flags in (0, cb.FLAG_SYMMETRY_BREAK, cb.FLAG_SYMMETRY_BREAK | cb.FLAG_NO_ORBIT_FOLD, cb.FLAG_NO_CLOSED_FORM):
            r = g.count(q, flags=flags, stats=True, alg_bytes=True)
            assert r.count == cnt, (name, flags)
            if not flags & cb.FLAG_SYMMETRY_BREAK:
                assert r.level_sizes == lv, (name, flags)
    g.close()
