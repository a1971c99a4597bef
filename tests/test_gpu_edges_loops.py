"""Edge counts (cycles, house) on symmetric graphs with self-loops, in the
instance with rows of the dense core (lists of 1,024 entries and more) and in
the one without: a vertex's own entry is no edge between the two sets.  Counts
and level sizes equal the oracle's."""
import functools

import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs
from tests.test_gpu_full_lists import _hubs

pytestmark = pytest.mark.gpu

QUERIES = {n: cb.named_query_arcs(n) for n in ("4-cycle", "house", "5-cycle")}


@functools.lru_cache(None)
def _case(shape, every):
    n, oo, oa, s, d = _hubs(*shape, seed=6)
    at = np.arange(0, n, every, dtype=np.uint32)
    oo, oa, _, _, s, d = csr_from_arcs(n, np.concatenate([s, at]), np.concatenate([d, at]))
    od = O.Graph.from_arrays(n, s, d)
    want = {}
    for name, (k, arcs) in QUERIES.items():
        q = cb.Query.from_arcs(k, arcs)
        want[name] = q, O.count(od, O.Graph.from_arcs(k, arcs), q.order)[:2]
    return n, oo, oa, want


@pytest.mark.parametrize("every", [1, 3])
@pytest.mark.parametrize("shape", [(3, 1030, 1100, 1), (12, 60, 200, 2)])
def test_edges_with_loops(shape, every):
    n, oo, oa, want = _case(shape, every)
    g = cb.Graph.from_csr(n, oo, oa)
    assert (g.info()[3] >= 1024) == (shape[1] >= 1024)
    for name, (q, (cnt, lv)) in want.items():
        assert cnt > 0
        for chunks in (1, 3):
            r = g.count(q, chunks=chunks, stats=True)
            assert (r.count, r.level_sizes) == (cnt, lv), name
            assert g.count(q, chunks=chunks, flags=cb.FLAG_SYMMETRY_BREAK).count == cnt, name
    g.close()
