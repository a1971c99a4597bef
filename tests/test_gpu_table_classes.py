"""Membership tables on both sides of the lengths where their build changes
kernel on graphs of degree-ranked ids -- 128, 1,024, 4,096 and 24,576 entries;
of directed graphs, where the classes go by out- plus in-degree, also lists of
half of it -- with the lists' lengths exact.  Every triangle tests a hub."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs

pytestmark = pytest.mark.gpu

LENGTHS = [126, 127, 128, 129, 130, 1023, 1024, 1025, 4095, 4096, 4097, 24575, 24576, 24577]


@pytest.mark.parametrize("directed", [False, True])
def test_exact_lengths(directed):
    hubs = [(d, d) for d in LENGTHS]
    if directed:  # (out, in): all of one kind, and sums on either side
        hubs = [(d, 0) for d in LENGTHS] + [(0, d) for d in LENGTHS]
        hubs += [(d // 2 + x, d - d // 2) for d in (128, 1024, 4096) for x in (-1, 0, 1)]
    h, ring = len(hubs), 24700
    n = h + ring
    rng = np.random.default_rng(8)
    src, dst = [np.arange(ring) + h], [(np.arange(ring) + 1) % ring + h]
    for i, (a, b) in enumerate(hubs):
        to = rng.choice(ring, a, replace=False) + h
        src.append(np.full(a, i))
        dst.append(to)
        if directed:
            src.append(rng.choice(ring, b, replace=False) + h)
            dst.append(np.full(b, i))
    src, dst = np.concatenate(src), np.concatenate(dst)
    if not directed:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
    oo, oa, io, ia, s, d = csr_from_arcs(n, src.astype(np.uint32), dst.astype(np.uint32))
    assert [int(x) for x in np.diff(oo.astype(np.int64))[:h]] == [a for a, _ in hubs]
    assert not directed or [int(x) for x in np.diff(io.astype(np.int64))[:h]] == [b for _, b in hubs]
    g = cb.Graph.from_csr(n, oo, oa, io, ia)
    od = O.Graph.from_arrays(n, s, d)
    queries = [cb.named_query_arcs("triangle")]
    if directed:
        queries = [(3, [(0, 1), (1, 2), (0, 2)]), (3, [(0, 1), (1, 2), (2, 0)])]
    for k, arcs in queries:
        q = cb.Query.from_arcs(k, arcs)
        cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
        assert cnt > 0
        for flags in (0, cb.FLAG_NO_FUSE):
            r = g.count(q, flags=flags, stats=True)
            assert (r.count, r.level_sizes) == (cnt, lv), (arcs, flags)
    g.close()
