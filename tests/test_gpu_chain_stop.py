"""A chain of launches that stops because a level does not fit goes on without
queueing the slices behind it again: the number of launches stays within what
the chunks need, whatever the number of slices (empty ones included), and the
counts are the oracle's."""
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import oracle_graph_from_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap", [256, 1024, 4096, 12000])
@pytest.mark.parametrize("name", ["4-cycle", "house", "4-path", "5-cycle"])
def test_launches_of_a_stopped_chain(name, cap):
    h = cb.HostGraph.chung_lu(1201, 4000, 2.3, 2.0, 60.0, seed=12)
    g, od = h.upload(0), oracle_graph_from_host(h)
    k, arcs = cb.named_query_arcs(name)
    q = cb.Query.from_arcs(k, arcs)
    cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
    g.set_level_cap(cap)
    for chunks in (1, 5, 40, 1000, 100000):
        r = g.count(q, chunks=chunks, stats=True)
        assert (r.count, r.level_sizes) == (cnt, lv), chunks
        # the roots; one attempt to queue 16 slices; then for each slice and each
        # chunk at most two planning launches and four that count, and the chunks
        assert r.launches <= 1 + 16 * (k + 4) + 6 * (min(chunks, lv[0]) + r.chunks) + r.chunks, chunks
    g.close()
