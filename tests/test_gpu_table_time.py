"""The device time of the count that builds a graph's membership tables includes
their build: on 20M list entries it takes some 0.3 ms, many times what a few
roots' triangles do."""
import pytest

import cuts_b200 as cb

pytestmark = pytest.mark.gpu


def test_first_count_reports_the_build():
    q = cb.Query.from_arcs(*cb.named_query_arcs("triangle"))
    h = cb.HostGraph.chung_lu(1000000, 10000000, 2.5, 2.0, 500.0, seed=4)
    warm = h.upload(0)
    warm.count_sharded(q, 7, 100000)
    warm.close()
    g = h.upload(0)
    first = g.count_sharded(q, 7, 100000)
    later = min((g.count_sharded(q, 7, 100000) for _ in range(5)), key=lambda r: r.ms)
    assert first.count == later.count
    # 80 MB read and 160 MB written take 0.037 ms at the card's copy bandwidth
    assert first.ms >= later.ms + 0.037
    g.close()
