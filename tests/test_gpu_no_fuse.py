"""FLAG_NO_FUSE materialises the level before the counted one, also where the
last two levels could be counted as edges between two sets (one expansion more,
seen in the number of chunks): the plain two-list join, against the oracle."""
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import oracle_graph_from_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["triangle", "4-cycle", "5-cycle", "house"])
def test_level_is_materialised(name, monkeypatch):
    h = cb.HostGraph.chung_lu(900, 3000, 2.3, 2.0, 60.0, seed=3)
    g, od = h.upload(0), oracle_graph_from_host(h)
    k, arcs = cb.named_query_arcs(name)
    q = cb.Query.from_arcs(k, arcs)
    cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
    for flags in (0, cb.FLAG_SYMMETRY_BREAK):
        res = {}
        for how in ("fused", "flag", "env"):
            if how == "env":
                monkeypatch.setenv("CUTS_NO_FUSE", "1")
            r = g.count(q, flags=flags | (cb.FLAG_NO_FUSE if how == "flag" else 0), stats=True)
            monkeypatch.delenv("CUTS_NO_FUSE", raising=False)
            assert r.count == cnt, how
            assert flags or r.level_sizes == lv, how
            res[how] = r.chunks
        assert res["flag"] == res["env"] == k - 2  # levels 1 .. k-2 stored
        assert res["fused"] == k - 3
    b = g.batch([q], flags=cb.FLAG_NO_FUSE)
    assert b.run()[:2] == ([cnt], [0])
    g.close()
