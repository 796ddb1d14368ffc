"""Batches of boxes of very different size with bins that start far out, at
finer grids (two and three cells per outer range): the boxes' cells differ in
width, and the one stencil has to hold every offset that any of them needs."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu

SHELLS = {
    "iso": dict(bintype=0, smin=180, smax=200, ds=5),
    "smu": dict(bintype=1, smin=180, smax=200, ds=5, nmu=7),
    "spi_s": dict(bintype=2, smin=150, smax=200, ds=5, pmin=0, pmax=40, dpi=4),
    "spi_p": dict(bintype=2, smin=0, smax=200, ds=20, pmin=52, pmax=100, dpi=8),
}


@pytest.mark.parametrize("k", [0, 2, 3])
@pytest.mark.parametrize("name", sorted(SHELLS))
def test_shells_of_different_boxes(name, k):
    import fcfc_gb300 as fg
    kw = SHELLS[name]
    pc = fg.PairCounter("box", box=5000.0, **kw)
    if k:
        pc.set_cells_per_smax(k)
    sides = [480.0, 5000.0, 700.0]
    cats = [np.random.default_rng(i).random((2000, 3)) * s
            for i, s in enumerate(sides)]
    cnt, status, _ = pc.count_batch(cats, sides)
    assert status == [0, 0, 0]
    for x, side, got in zip(cats, sides, cnt):
        ok = dict(smin=kw["smin"], ds=kw["ds"], box=side,
                  ns=(kw["smax"] - kw["smin"]) // kw["ds"])
        if "nmu" in kw:
            ok["nmu"] = kw["nmu"]
        if "pmin" in kw:
            ok.update(pmin=kw["pmin"], dpi=kw["dpi"],
                      np_=(kw["pmax"] - kw["pmin"]) // kw["dpi"])
        want = fo.Bins(False, kw["bintype"], **ok).count(x, mode=1)
        np.testing.assert_array_equal(got, want)
