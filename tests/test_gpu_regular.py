"""Fused pairs on graphs of bounded degree with enough roots that a warp takes
up to 32 of them a turn: the parents that its first launch leaves to the second
are counted there whatever the largest degree (40, 60, 64 and 65), and so are
windows dealt out in pieces because the longest list is long enough for it (192
and 193 entries, 256 and 257 with an order).

The graphs are circulants, vertex i joined to i +- 1 .. i +- r, whose counts
are known: r (r - 1) / 2 triangles per vertex.  Labels are permuted, so the
windows under symmetry breaking differ in length."""
import numpy as np
import pytest

import cuts_b200 as cb

pytestmark = pytest.mark.gpu

TRI = cb.named_query_arcs("triangle")
TAIL = (4, TRI[1] + [(0, 3), (3, 0)])  # triangle and a pendant vertex


def _circulant(n, r, extra=False):
    """CSR of the circulant under a fixed permutation; `extra`: one more edge
    between the vertices at places 0 and n // 2 (no triangle through it)."""
    perm = np.random.default_rng(5).permutation(n).astype(np.int64)
    steps = np.concatenate([np.arange(-r, 0), np.arange(1, r + 1)])
    place = np.empty(n, np.int64)
    place[perm] = np.arange(n)
    adj = np.sort(perm[(place[:, None] + steps[None, :]) % n], axis=1).astype(np.uint32)
    off = np.arange(n + 1, dtype=np.uint64) * np.uint64(2 * r)
    if not extra:
        return off, adj.ravel()
    a, b = int(perm[0]), int(perm[n // 2])
    out = adj.ravel()
    for v, w in sorted([(a, b), (b, a)], reverse=True):
        at = int(off[v]) + int(np.searchsorted(adj[v], w))
        out = np.insert(out, at, np.uint32(w))
        off = off + (np.arange(n + 1) > v).astype(np.uint64)
    return off, out


@pytest.mark.parametrize("n,r,extra", [(700003, 20, False), (700003, 30, False), (400009, 32, False), (400009, 32, True)] +
                         [(20011, 96, x) for x in (False, True)] + [(9001, 128, x) for x in (False, True)])
def test_all_deferred_parents_counted(n, r, extra):
    off, adj = _circulant(n, r, extra)
    g = cb.Graph.from_csr(n, off, adj)
    assert g.info()[3] == 2 * r + extra
    per = 6 * n * (r * (r - 1) // 2)  # ordered triangles
    arcs = 2 * r * n + 2 * extra
    # a triangle's vertices have 2 r - 2 further neighbours; the two with the
    # extra edge lie in 3 r (r - 1) / 2 triangles each, twice as ordered ones
    # with the vertex at a given place
    tail = per * (2 * r - 2) + extra * 2 * (2 * (3 * r * (r - 1) // 2))
    tri, tt = cb.Query.from_arcs(*TRI), cb.Query.from_arcs(*TAIL)
    want = {0: [n, arcs, per], cb.FLAG_SYMMETRY_BREAK: [n, arcs // 2, per // 6]}
    for flags, lv in want.items():
        for chunks in (1, 2, 16):
            for nf in (0, cb.FLAG_NO_FUSE):
                res = g.count(tri, chunks=chunks, flags=flags | nf, stats=True)
                assert (res.count, res.level_sizes) == (per, lv), (flags, chunks, nf)
    for flags in want:
        for chunks in (1, 2, 16):
            for nf in (0, cb.FLAG_NO_FUSE):
                res = g.count(tt, chunks=chunks, flags=flags | nf, stats=True)
                assert res.count == tail, (flags, chunks, nf)
    g.close()
