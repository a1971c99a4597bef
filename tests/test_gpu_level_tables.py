"""Level kernels with membership tables, at the lengths where a table or the
candidate walk changes shape: lists of one bucket and of one entry more (4, 5,
8, 9), one and two steps of 64 candidates, the split between the tables' two
build kernels (512, 513), empty lists, self-loops; ids degree-ranked or kept
(the signature is then a compare of ids or a gather), one to three joined
lists.  Counts and level sizes equal the oracle's."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs

pytestmark = pytest.mark.gpu

HUBS = [1, 3, 4, 5, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 129, 511, 512, 513, 600]
QUERIES = {
    "4-cycle": cb.named_query_arcs("4-cycle"),
    "house": cb.named_query_arcs("house"),
    "diamond": (4, [a for e in [(0, 1), (1, 2), (2, 3), (3, 0), (0, 2)] for a in (e, e[::-1])]),
    # the last vertex joins three lists, none of them nested in the level before
    "wheel4": (5, [a for e in [(0, 1), (1, 2), (2, 3), (3, 0), (4, 0), (4, 1), (4, 2)] for a in (e, e[::-1])]),
}
DIRECTED = {
    "feed": (4, [(0, 2), (1, 2), (0, 3), (2, 3)]),
    "3-cycle+out": (4, [(0, 1), (1, 2), (2, 0), (2, 3)]),
    "mutual": (3, [(0, 1), (1, 0), (1, 2), (0, 2)]),
    "loop": (3, [(0, 0), (0, 1), (1, 2), (0, 2)]),
}


def _graph(directed, seed):
    """Vertices of the degrees in HUBS over a sparse random part."""
    rng = np.random.default_rng(seed)
    n = 700
    src, dst = [], []
    for i, d in enumerate(HUBS):
        to = rng.choice(np.arange(len(HUBS), n), d, replace=False)
        src += [i] * d
        dst += list(to)
    src += list(rng.integers(len(HUBS), n - 20, 500))  # the last 20 stay out: empty lists
    dst += list(rng.integers(len(HUBS), n - 20, 500))
    src, dst = np.array(src, np.uint32), np.array(dst, np.uint32)
    if directed:
        flip = rng.random(len(src)) < 0.5
        src, dst = np.where(flip, dst, src), np.where(flip, src, dst)
    else:
        keep = src != dst
        src, dst = np.concatenate([src[keep], dst[keep]]), np.concatenate([dst[keep], src[keep]])
    return n, src.astype(np.uint32), dst.astype(np.uint32)


@pytest.mark.parametrize("ranked", [True, False])
@pytest.mark.parametrize("directed", [False, True])
def test_tables_match_oracle(directed, ranked, monkeypatch):
    if not ranked:
        monkeypatch.setenv("CUTS_NO_RELABEL", "1")
    n, src, dst = _graph(directed, 7 + directed)
    oo, oa, io, ia, s, d = csr_from_arcs(n, src, dst)
    g = cb.Graph.from_csr(n, oo, oa, io, ia)
    od = O.Graph.from_arrays(n, s, d)
    for name, (k, arcs) in (DIRECTED if directed else QUERIES).items():
        q = cb.Query.from_arcs(k, arcs)
        cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
        for flags in (0, cb.FLAG_NO_FUSE | cb.FLAG_NO_CLOSED_FORM):
            r = g.count(q, flags=flags, stats=True)
            assert (r.count, r.level_sizes) == (cnt, lv), (name, flags)
        assert g.count(q, flags=cb.FLAG_SYMMETRY_BREAK).count == cnt, name
    g.close()


@pytest.mark.parametrize("ranked", [True, False])
@pytest.mark.parametrize("directed", [False, True])
def test_hub_tables(directed, ranked, monkeypatch):
    """Lists at the lengths where the tables' build changes kernel (one run in
    shared memory, one block, one large block, in place): hubs over a ring, so
    every triangle tests a hub's table."""
    if not ranked:
        monkeypatch.setenv("CUTS_NO_RELABEL", "1")
    degs = [1020, 1023, 1024, 1025, 4095, 4096, 4097, 24574, 24576, 24577, 26000]
    h, ring = len(degs), 26100
    n = h + ring
    rng = np.random.default_rng(3)
    src, dst = [np.arange(ring) + h], [(np.arange(ring) + 1) % ring + h]
    for i, d in enumerate(degs):  # d ring vertices each, so d or d + 10 entries
        to = rng.choice(ring, d, replace=False) + h
        src.append(np.full(d, i))
        dst.append(to)
    a, b = np.triu_indices(h, 1)
    if not directed:
        src.append(a)
        dst.append(b)
    src, dst = np.concatenate(src), np.concatenate(dst)
    if not directed:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    oo, oa, io, ia, s, d = csr_from_arcs(n, src.astype(np.uint32), dst.astype(np.uint32))
    g = cb.Graph.from_csr(n, oo, oa, io, ia)
    od = O.Graph.from_arrays(n, s, d)
    k, arcs = (3, [(0, 1), (1, 2), (0, 2)]) if directed else cb.named_query_arcs("triangle")
    q = cb.Query.from_arcs(k, arcs)
    cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
    assert cnt > 0
    for flags in (0, cb.FLAG_NO_FUSE, cb.FLAG_NO_FUSE | cb.FLAG_SYMMETRY_BREAK):
        r = g.count(q, flags=flags, stats=True)
        assert r.count == cnt, flags
        if not flags & cb.FLAG_SYMMETRY_BREAK:
            assert r.level_sizes == lv, flags
    g.close()
