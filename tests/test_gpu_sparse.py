"""Catalogues with far fewer points than cells of the outer range would fit in the
volume: no more cells than points (or 32768), and the oracle's counts."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geom", ["box", "survey"])
@pytest.mark.parametrize("n", [3000, 50000])
def test_sparse_catalogues(geom, n):
    import fcfc_gb300 as fg
    kw = dict(smin=0, smax=20, ds=2, nmu=7)
    side = 20000.0
    rng = np.random.default_rng(n)
    x = rng.random((n, 3)) * side
    y = rng.random((n // 3, 3)) * side
    # pairs to count: every tenth point of y next to one of x, some across
    # the box's faces
    y[::10] = x[:len(y[::10])] + rng.uniform(-15, 15, (len(y[::10]), 3))
    if geom == "box":
        y %= side
        kw["box"] = side
    else:
        x, y = x - 7000.0, y - 7000.0
    pc = fg.PairCounter(geom, fg.BIN_SMU, **kw)
    ob = fo.Bins(geom == "survey", 1, smin=0, ds=2, ns=10, nmu=7,
                 **({"box": side} if geom == "box" else {}))
    pc.load(0, x)
    pc.load(1, y)
    want = ob.count(x, y, mode=1)
    assert want.sum() > len(y) // 25
    np.testing.assert_array_equal(pc.count_pairs(0, 1), want)
    st = pc.stats()
    assert np.prod(st["ncell"]) <= max(32768, n)
    np.testing.assert_array_equal(pc.count_pairs(0), ob.count(x, mode=1))


def test_sparse_against_dense():
    """300 points against 1e5: cells for a density between the two (2 per side;
    the 300 alone would get one of the box), in either order of the catalogues."""
    import fcfc_gb300 as fg
    rng = np.random.default_rng(8)
    a, b = rng.random((300, 3)) * 400.0, rng.random((100000, 3)) * 400.0
    pc = fg.PairCounter("box", fg.BIN_SMU, box=400.0, smin=0, smax=100, ds=5,
                        nmu=10)
    want = fo.Bins(False, 1, smin=0, ds=5, ns=20, nmu=10, box=400.0).count(
        a, b, mode=1)
    pc.load(0, a)
    pc.load(1, b)
    np.testing.assert_array_equal(pc.count_pairs(0, 1), want)
    assert list(pc.stats()["ncell"]) == [2, 2, 2]
    np.testing.assert_array_equal(pc.count_pairs(1, 0), want)
