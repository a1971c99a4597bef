"""Twins: last two query vertices with the same two or more neighbours, counted
together from each parent's number of candidates, and the fused, folded and
plain tails of small queries through the batched kernels, whose frontiers are
counted at once.  Counts (and level sizes) equal the oracle's on uniform,
power-law, self-loop and directed graphs."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs, directed_er, oracle_graph_from_host

pytestmark = pytest.mark.gpu


def _und(edges):
    return [a for e in edges for a in (e, e[::-1])]


UNDIRECTED = {
    "diamond": (4, _und([(0, 1), (0, 2), (0, 3), (1, 2), (1, 3)])),
    "K23": (5, _und([(0, 2), (0, 3), (0, 4), (1, 2), (1, 3), (1, 4)])),
    "5-clique-edge": (5, _und([(a, b) for a in range(5) for b in range(a + 1, 5) if (a, b) != (3, 4)])),
    "diamond+tail": (5, _und([(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (1, 4)])),
    "4-cycle": cb.named_query_arcs("4-cycle"),
    "3-path": cb.named_query_arcs("3-path"),
    "4-path": cb.named_query_arcs("4-path"),
    "triangle": cb.named_query_arcs("triangle"),
    "edge": (2, _und([(0, 1)])),
}
DIRECTED = {
    "out-twins": (4, [(0, 1), (0, 2), (1, 2), (0, 3), (1, 3)]),
    "in-out-twins": (4, [(0, 1), (0, 2), (2, 1), (0, 3), (3, 1)]),
    "both-arcs": (3, [(0, 1), (1, 0), (0, 2), (2, 0)]),
    "not-twins": (4, [(0, 1), (0, 2), (1, 2), (0, 3), (3, 1)]),
    "feed": (4, [(0, 2), (1, 2), (0, 3), (2, 3)]),
}


def _cases():
    h = cb.HostGraph.erdos_renyi(900, 14.0 / 899, seed=5)
    yield "er", h.upload(0), oracle_graph_from_host(h), UNDIRECTED
    h = cb.HostGraph.chung_lu(1500, 6000, 2.2, 2.0, 90.0, seed=6)
    yield "cl", h.upload(0), oracle_graph_from_host(h), UNDIRECTED
    oo, oa, _, _ = cb.HostGraph.erdos_renyi(150, 0.12, seed=4).csr()
    src = np.concatenate([np.repeat(np.arange(150, dtype=np.uint32), np.diff(oo.astype(np.int64))),
                          np.arange(0, 150, 3, dtype=np.uint32)])
    dst = np.concatenate([oa, np.arange(0, 150, 3, dtype=np.uint32)])
    oo, oa, io, ia, s, d = csr_from_arcs(150, src, dst)
    yield "loops", cb.Graph.from_csr(150, oo, oa, io, ia), O.Graph.from_arrays(150, s, d), UNDIRECTED
    n, src, dst = directed_er(700, 20.0, seed=9)
    oo, oa, io, ia, s, d = csr_from_arcs(n, src, dst)
    yield "directed", cb.Graph.from_csr(n, oo, oa, io, ia), O.Graph.from_arrays(n, s, d), DIRECTED


@pytest.mark.parametrize("ranked", [True, False])
def test_twins_and_frontiers(ranked, monkeypatch):
    if not ranked:
        monkeypatch.setenv("CUTS_NO_RELABEL", "1")
    monkeypatch.setenv("CUTS_BATCH_ROUTE", "0")  # every query in the batched kernel
    for gname, g, od, queries in _cases():
        qs, want = [], []
        for name, (k, arcs) in queries.items():
            q = cb.Query.from_arcs(k, arcs)
            cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
            for flags in (0, cb.FLAG_NO_CLOSED_FORM):
                r = g.count(q, flags=flags, stats=True)
                assert (r.count, r.level_sizes) == (cnt, lv), (gname, name, flags)
            assert g.count(q, flags=cb.FLAG_SYMMETRY_BREAK).count == cnt, (gname, name)
            assert sum(g.count_sharded(q, s, 3, chunks=2, flags=cb.FLAG_SYMMETRY_BREAK).count for s in range(3)) == cnt
            qs.append(q)
            want.append(cnt)
        for flags in (0, cb.FLAG_SYMMETRY_BREAK):
            for grain in (0, 4):
                counts, status, _ = g.batch(qs, flags=flags, grain=grain).run()
                assert status == [0] * len(qs) and counts == want, (gname, flags, grain)
            parts = np.zeros(len(qs), np.int64)
            b = g.batch(qs, flags=flags)
            for s in range(3):
                b.set_shard(s, 3)
                parts += np.array(b.run()[0], np.int64)
            assert list(parts) == want, (gname, flags)
        g.close()
