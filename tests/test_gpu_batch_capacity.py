"""Batches whose cycle-like queries the level engine counts: where it has no
room for a level (a capacity below twice the largest degree, an arena of a few
bytes), they run in the persistent launch instead, which stores no level.  So
also for some shards of a sharded batch only: the parts still add up."""
import pytest

import cuts_b200 as cb

pytestmark = pytest.mark.gpu

NAMES = ["triangle", "4-cycle", "3-star", "5-cycle", "house", "4-path"]


@pytest.mark.parametrize("flags", [0, cb.FLAG_SYMMETRY_BREAK])
@pytest.mark.parametrize("room", ["cap", "arena"])
def test_no_room_for_a_level(room, flags):
    h = cb.HostGraph.chung_lu(2000, 7000, 2.3, 2.0, 60.0, seed=8)
    g = h.upload(0)
    qs = [cb.Query.from_arcs(*cb.named_query_arcs(nm)) for nm in NAMES]
    want = [g.count(q, flags=flags).count for q in qs]
    cycles = [1, 3, 4]

    def squeeze(on):
        if room == "cap":
            g.set_level_cap(64 if on else 0)
        else:
            g.set_arena_bytes(20000 if on else 0)

    b = g.batch(qs, flags=flags)
    assert b.run()[0] == want
    for _ in range(2):
        squeeze(True)
        counts, status, _ = b.run()
        assert [status[i] for i in cycles] == [0] * 3
        assert [counts[i] for i in cycles] == [want[i] for i in cycles]
        squeeze(False)
        assert b.run()[:2] == (want, [0] * len(qs))
    # shards: the odd ones without room
    for nshards in (2, 3):
        total = [0] * len(qs)
        for r in range(nshards):
            squeeze(r % 2 == 1)
            b.set_shard(r, nshards)
            counts, status, _ = b.run()
            for i in cycles:
                assert status[i] == 0
                total[i] += counts[i]
        squeeze(False)
        assert [total[i] for i in cycles] == [want[i] for i in cycles]
    b.close()
    g.close()
