"""Counts queued as one chain of launches (each reads its parents' number on
the device): root slices that do not divide the root level, more slices than
roots, chains longer than one group of slices, a level that does not fit and
is continued in chunks, empty levels.  Counts and level sizes equal the
oracle's for every plan form (fused, folded, pendant pair, closed form, plain
join)."""
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import oracle_graph_from_host

pytestmark = pytest.mark.gpu

QUERIES = {name: cb.named_query_arcs(name) for name in ("triangle", "4-cycle", "house", "4-clique+pendant", "3-star",
                                                        "4-path")}
QUERIES["6-clique"] = (6, [(a, b) for a in range(6) for b in range(6) if a != b])  # empty last levels
QUERIES["edge"] = (2, [(0, 1), (1, 0)])


@pytest.fixture(scope="module")
def graph():
    h = cb.HostGraph.chung_lu(1201, 4000, 2.3, 2.0, 60.0, seed=12)
    return h.upload(0), oracle_graph_from_host(h)


@pytest.mark.parametrize("cap", [0, 4096])
@pytest.mark.parametrize("name", sorted(QUERIES))
def test_slices_and_levels(graph, name, cap):
    g, od = graph
    k, arcs = QUERIES[name]
    q = cb.Query.from_arcs(k, arcs)
    cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
    g.set_level_cap(cap)
    try:
        for chunks in (1, 2, 3, 7, 16, 17, 40, 5000):
            r = g.count(q, chunks=chunks, stats=True)
            assert (r.count, r.level_sizes) == (cnt, lv), chunks
            assert g.count(q, chunks=chunks, flags=cb.FLAG_SYMMETRY_BREAK).count == cnt, chunks
            parts = [g.count_sharded(q, s, 3, chunks=chunks) for s in range(3)]
            assert sum(p.count for p in parts) == cnt, chunks
    finally:
        g.set_level_cap(0)
