"""The allocation-free count at the sizes where its task space changes shape:
longest lists around one, two and sixteen slices of 32 candidates, vertex counts
around a block of 32 roots, few and many (query, root) pairs (blocks of one root
up to 32), queries deep enough for smaller blocks.  Against the oracle."""
import numpy as np
import pytest

import cuts_b200 as cb
from oracle import oracle as O
from tests.helpers import csr_from_arcs
from tests.test_zz_no_alloc import _device_layout, _run_twice

pytestmark = pytest.mark.gpu

SMALL = [(2, [(0, 1), (1, 0)])] + [cb.named_query_arcs(n) for n in ("3-path", "triangle")]
DEEP = SMALL + [cb.named_query_arcs(n) for n in ("5-path", "house")]


def _hub(n, deg):
    """A ring over n vertices and one hub whose list has `deg` entries."""
    i = np.arange(n)
    hub, others = n // 2, np.setdiff1d(np.arange(n), [n // 2])
    ring = np.setdiff1d(others[(others != hub + 1) & (others != hub - 1)], [0, n - 1])
    to = ring[: deg - 2]
    src = np.concatenate([i, np.full(len(to), hub)])
    dst = np.concatenate([(i + 1) % n, to])
    keep = src != dst
    src, dst = src[keep], dst[keep]
    return np.concatenate([src, dst]).astype(np.uint32), np.concatenate([dst, src]).astype(np.uint32)


@pytest.mark.parametrize("queries", ["small", "deep", "many"])
@pytest.mark.parametrize("n,deg", [(3, 2), (31, 2), (32, 2), (33, 2), (33, 30)] +
                         [(1025, d) for d in (31, 32, 33, 64, 65, 480, 481, 512, 513, 900)])
def test_counts_at_block_and_slice_edges(n, deg, queries):
    src, dst = _hub(n, deg)
    oo, oa, _, _, s, d = csr_from_arcs(n, src, dst)
    assert int(np.diff(oo.astype(np.int64)).max()) == deg
    od = O.Graph.from_arrays(n, s, d)
    defs = {"small": SMALL, "deep": DEEP, "many": SMALL * 21}[queries]
    qs, want, seen = [], [], {}
    for i, (k, arcs) in enumerate(defs):
        q = cb.Query.from_arcs(k, arcs)
        key = (k, tuple(arcs))
        if key not in seen:
            seen[key] = O.count(od, O.Graph.from_arcs(k, arcs), q.order)[0]
        qs.append(q)
        want.append(seen[key])
    info_out, _, adj = _device_layout(oo, oa)
    _run_twice(n, info_out, None, adj, qs, want)


def test_blocks_of_32_roots():
    n = 20011
    src, dst = _hub(n, 700)
    oo, oa, _, _, s, d = csr_from_arcs(n, src, dst)
    od = O.Graph.from_arrays(n, s, d)
    qs = [cb.Query.from_arcs(*SMALL[i % 3]) for i in range(64)]
    want = [O.count(od, O.Graph.from_arcs(*SMALL[i]), qs[i].order)[0] for i in range(3)]
    info_out, _, adj = _device_layout(oo, oa)
    _run_twice(n, info_out, None, adj, qs, [want[i % 3] for i in range(64)])
