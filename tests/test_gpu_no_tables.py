"""Counts on a graph without membership tables.  Edges, stars and paths of
three vertices look nothing up, so they leave them unbuilt (seen in the pool's
memory: the tables take twice the adjacency); and where the tables find no
memory, every kind of count searches the lists instead.  Against the oracle."""
import os
import subprocess
import sys

import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

USED = """
import sys
import cuts_b200 as cb
from cuda.bindings import runtime as rt
h = cb.HostGraph.chung_lu(200000, 2000000, 2.3, 2.0, 500.0, seed=4)
g = h.upload(0)
g.set_arena_bytes(64 << 20)
def used():
    _, pool = rt.cudaDeviceGetDefaultMemPool(0)
    _, v = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    return int(v)
out = []
for name in sys.argv[1].split(","):
    k, arcs = (2, [(0, 1), (1, 0)]) if name == "edge" else cb.named_query_arcs(name)
    q = cb.Query.from_arcs(k, arcs)
    for flags in (0, cb.FLAG_SYMMETRY_BREAK):
        g.count(q, flags=flags)
    out.append(str(used()))
print(" ".join(out))
"""


def test_counts_that_look_nothing_up_build_no_tables():
    out = subprocess.run([sys.executable, "-c", USED, "edge,3-path,3-star,triangle"], cwd=ROOT, capture_output=True,
                         text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-800:]
    edge, path, star, tri = (int(x) for x in out.stdout.split())
    assert edge == path == star
    assert tri - star >= 2 * 4 * 4000000  # twice the 4M list entries


QUERIES = {n: cb.named_query_arcs(n) for n in ("triangle", "4-cycle", "house", "4-clique+pendant", "3-star", "4-path")}
QUERIES["diamond"] = (4, [a for e in [(0, 1), (1, 2), (2, 3), (3, 0), (0, 2)] for a in (e, e[::-1])])
QUERIES["edge"] = (2, [(0, 1), (1, 0)])


@pytest.mark.parametrize("loops", [False, True])
def test_without_memory_for_tables(loops, monkeypatch):
    monkeypatch.setenv("CUTS_TABLES", "0")
    h = cb.HostGraph.chung_lu(1500, 6000, 2.2, 2.0, 80.0, seed=9)
    oo, oa, _, _ = h.csr()
    src = np.repeat(np.arange(h.n, dtype=np.uint32), np.diff(oo.astype(np.int64)))
    at = np.arange(0, h.n if loops else 0, 5, dtype=np.uint32)
    oo, oa, _, _, s, d = csr_from_arcs(h.n, np.concatenate([src, at]), np.concatenate([oa, at]))
    g = cb.Graph.from_csr(h.n, oo, oa)
    od = O.Graph.from_arrays(h.n, s, d)
    want = []
    for name, (k, arcs) in QUERIES.items():
        q = cb.Query.from_arcs(k, arcs)
        cnt, lv, _ = O.count(od, O.Graph.from_arcs(k, arcs), q.order)
        want.append(cnt)
        for flags in (0, cb.FLAG_SYMMETRY_BREAK, cb.FLAG_NO_FUSE):
            r = g.count(q, flags=flags, stats=True)
            assert r.count == cnt, (name, flags)
            assert flags & cb.FLAG_SYMMETRY_BREAK or r.level_sizes == lv, (name, flags)
    qs = [cb.Query.from_arcs(k, arcs) for k, arcs in QUERIES.values()]
    for flags in (0, cb.FLAG_SYMMETRY_BREAK):
        counts, status, _ = g.batch(qs, flags=flags).run()
        assert (counts, status) == (want, [0] * len(qs))
    # in two shards, one of a graph with tables: the routing is the same
    g.close()
    gs = [cb.Graph.from_csr(h.n, oo, oa)]
    monkeypatch.delenv("CUTS_TABLES")
    gs.append(cb.Graph.from_csr(h.n, oo, oa))
    total = [0] * len(qs)
    for r, gr in enumerate(gs):
        b = gr.batch(qs)
        b.set_shard(r, 2)
        counts, status, _ = b.run()
        assert status == [0] * len(qs)
        total = [x + y for x, y in zip(total, counts)]
        b.close()
        gr.close()
    assert total == want
