"""Statistics of a count: the pairs whose separation was evaluated, and the
kernels launched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_candidates_are_the_pairs_evaluated(precision):
    """Points of A 10 apart on a line through cells 83.3 wide, tested by fours
    that begin at each cell's first point; a clump of A's, far off, makes the
    catalogue large enough for whole blocks.  One point of B: next to the first
    four of a cell; between two cells, at the one point of a four and the next
    cell's first four."""
    import fcfc_gb300 as fg
    line = np.full((20, 3), 41.0)
    line[:, 0] = np.arange(20) * 10.0
    clump = 600.0 + 20.0 * np.random.default_rng(1).random((20000, 3))
    pc = fg.PairCounter("box", fg.BIN_ISO, box=1000.0, smin=0, smax=20, ds=2)
    pc.load(0, np.concatenate([line, clump]))
    for x, want in ((5.0, 4), (95.0, 1 + 4)):
        pc.load(1, np.array([[x, 41.0, 41.0]]))
        pc.count_pairs(0, 1, precision=precision)
        st = pc.stats()
        assert list(st["ncell"]) == [12, 12, 12]
        assert st["candidates"] == want, (x, st["candidates"])
        assert st["in_range"] <= want


def test_launches_are_those_made():
    """The sort of a small catalogue (cells, one scan, keys, runs) or of one with
    more counters than a scan's eight tiles (two), the count, its recheck
    (none without a queue) and the fold of FP64 sums."""
    import fcfc_gb300 as fg
    pc = fg.PairCounter("box", fg.BIN_ISO, box=200.0, smin=0, smax=20, ds=2)
    rng = np.random.default_rng(1)

    def launches(call):
        before = pc.stats()["launches"]
        call()
        return pc.stats()["launches"] - before
    pc.load(0, rng.random((3000, 3)) * 200.0)
    pc.count_pairs(0)
    assert launches(lambda: pc.count_pairs(0)) == 2
    pc.set_queue_capacity(0)
    assert launches(lambda: pc.count_pairs(0)) == 1
    assert launches(lambda: pc.count_pairs(0, weighted=True,
                                           precision=fg.PREC_FP64)) == 2
    pc.load(1, rng.random((3000, 3)) * 200.0)
    assert launches(lambda: pc.count_pairs(1)) == 1 + 4 + 1     # load, sort
    pc.load(1, rng.random((100000, 3)) * 200.0)
    assert launches(lambda: pc.count_pairs(1)) == 1 + 5 + 1
