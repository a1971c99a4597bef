"""The count autotuner tries the kernels' default split and keeps it where it is
the fastest (a stand-in graph records what it is set to; no GPU)."""
import cuts_b200 as cb
from cuts_b200 import autotune


class FakeGraph:
    def __init__(self, best):
        self.best, self.split, self.cap = best, 0, 0

    def set_fuse_split(self, split):
        self.split = split

    def set_level_cap(self, cap):
        self.cap = cap

    def count(self, q, chunks=1, flags=0):
        return cb.CountResult(7, 1.0 if self.split == self.best else 2.0)


def test_default_split_is_tried_and_kept():
    for best in autotune.SPLITS:
        g = FakeGraph(best)
        (_, split, _), times = autotune.tune_count(g, None)
        assert split == best and g.split == best
        assert len(times) == len(autotune.CHUNKS) * len(autotune.SPLITS)
    assert 0 in autotune.SPLITS
