"""Batches of very many and very few items of work: from one catalogue of one
point to more small catalogues than blocks of the launch, and one large among
them; every catalogue's counts equal the oracle's."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [0, 1, 2], [33] * 5, [7] * 700,
                                   [400] * 90 + [20000] + [31] * 90])
def test_runs_cover_every_item(sizes):
    import fcfc_gb300 as fg
    pc = fg.PairCounter("box", fg.BIN_SMU, box=100.0, smin=0, smax=20, ds=2,
                        nmu=5)
    sides = [60.0 + 0.01 * i for i in range(len(sizes))]
    cats = [np.random.default_rng(i).random((n, 3)) * side
            for i, (n, side) in enumerate(zip(sizes, sides))]
    cnt, status, _ = pc.count_batch(cats, sides)
    assert not any(status)
    for x, side, got in zip(cats, sides, cnt):
        ob = fo.Bins(False, 1, smin=0, ds=2, ns=10, nmu=5, box=side)
        np.testing.assert_array_equal(got, ob.count(x, mode=1))
