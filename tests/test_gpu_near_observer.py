"""Survey (s_perp, pi) counts of pairs on either side of the observer, whose line
of sight m = x_a + x_b is short and whose pi lies just below pi_max: FP32 cannot
tell their pi, so that each of them has to be rechecked and none left out.
Counts equal the oracle's, weighted sums and gradients to rounding."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu
PMAX, SMAX = 27.0, 40.0


def _antipodal(n, lengths, seed, below=1e-3):
    """x_a, x_b with |m| = lengths, pi in (PMAX - below, PMAX)."""
    rng = np.random.default_rng(seed)
    u, v = rng.normal(size=(2, n, 3))
    u /= np.linalg.norm(u, axis=1)[:, None]
    v -= (v * u).sum(1)[:, None] * u
    v /= np.linalg.norm(v, axis=1)[:, None]
    d = u * (PMAX - below * rng.random(n))[:, None] + \
        v * rng.uniform(1.0, SMAX - 1.0, n)[:, None]
    m = u * np.broadcast_to(lengths, n)[:, None]
    return (m + d) / 2, (m - d) / 2


def _counters(ns, dpi):
    import fcfc_gb300 as fg
    pc = fg.PairCounter("survey", fg.BIN_SPI, smin=0, smax=SMAX, ds=SMAX / ns,
                        pmin=0, pmax=PMAX, dpi=dpi)
    return pc, fo.Bins(True, 2, smin=0, ds=SMAX / ns, ns=ns, pmin=0, dpi=dpi,
                       np_=round(PMAX / dpi))


@pytest.mark.parametrize("ns,dpi", [(10, 3.0), (40, 0.025)],
                         ids=["shared", "global"])
@pytest.mark.parametrize("length", [1e-5, 0.003, 0.1, 1.0])
def test_pairs_across_the_observer(length, ns, dpi):
    pc, ob = _counters(ns, dpi)
    a, b = _antipodal(2000, length, 1)
    far = np.random.default_rng(2).uniform(-200.0, 150.0, (300, 3))
    a, b = np.concatenate([a, far[:200]]), np.concatenate([b, far[200:]])
    w = np.random.default_rng(3).normal(1.0, 0.6, len(a))
    pc.load(0, a, w)
    pc.load(1, b)
    both = np.concatenate([a, b])
    pc.load(2, both)
    np.testing.assert_array_equal(pc.count_pairs(0, 1), ob.count(a, b, mode=1))
    assert pc.stats()["precision_used"] == 0
    np.testing.assert_array_equal(pc.count_pairs(2), ob.count(both, mode=1))
    np.testing.assert_allclose(pc.count_pairs(0, 1, weighted=True),
                               ob.count(a, b, wa=w, mode=1), rtol=1e-10,
                               atol=1e-10)
    g = np.random.default_rng(4).normal(size=pc.ntot)
    da, db = pc.adjoint(0, 1, g)
    wda, wdb = ob.adjoint(a, g, b=b, wa=w)
    np.testing.assert_allclose(da, wda, rtol=1e-10, atol=1e-9)
    np.testing.assert_allclose(db, wdb, rtol=1e-10, atol=1e-9)


@pytest.mark.parametrize("length", [1e-4, 3e-4, 1e-3])
def test_single_pairs_across_the_observer(length):
    """One pair at a time: boxes of single points have no extent, and their
    line of sight is as short as the pair's.  A far third point widens the cells,
    so that the coordinates are not taken from the pair's own middle."""
    pc, ob = _counters(10, 3.0)
    a, b = _antipodal(300, length, 5)
    rng = np.random.default_rng(6)
    for i in range(len(a)):
        far = rng.uniform([400.0, 40.0, 40.0], [450.0, 90.0, 90.0])
        x, y = a[i:i + 1], np.stack([b[i], far])
        pc.load(0, x)
        pc.load(1, y)
        np.testing.assert_array_equal(pc.count_pairs(0, 1),
                                      ob.count(x, y, mode=1))


@pytest.mark.parametrize("bintype", [1, 2])
@pytest.mark.parametrize("cap", [0, 37, 5000, None])
def test_tiles_of_rechecks(bintype, cap):
    """Catalogues around the observer, whose tiles leave hundreds of pairs each to
    the recheck queue: with room for all, some or none."""
    import fcfc_gb300 as fg
    kw, ok = dict(smin=0, smax=40, ds=4), dict(smin=0, ds=4, ns=10)
    if bintype == 1:
        kw["nmu"] = ok["nmu"] = 12
    else:
        kw.update(pmin=0, pmax=30, dpi=2)
        ok.update(pmin=0, dpi=2, np_=15)
    pc, ob = fg.PairCounter("survey", bintype, **kw), fo.Bins(True, bintype, **ok)
    rng = np.random.default_rng(7)
    a, b = 20.0 * rng.normal(size=(1500, 3)), 20.0 * rng.normal(size=(700, 3))
    w = rng.integers(1, 4, len(a)).astype(float)
    if cap is not None:
        pc.set_queue_capacity(cap)
    pc.load(0, a, w)
    pc.load(1, b)
    for other in (None, 1):
        y = None if other is None else b
        np.testing.assert_array_equal(pc.count_pairs(0, other), ob.count(a, y, mode=1))
        st = pc.stats()
        assert st["in_range"] == ob.count(a, y, mode=1).sum()
        assert st["rechecked"] > st["in_range"] // 2
        assert st["recheck_inline"] == (0 if cap is None else st["rechecked"] - cap)
        # (integer weights: exact sums)
        np.testing.assert_array_equal(pc.count_pairs(0, other, weighted=True),
                                      ob.count(a, y, wa=w, mode=1))
    g = rng.integers(-3, 4, pc.ntot).astype(float)
    got, want = pc.adjoint(0, 1, g), ob.adjoint(a, g, b=b, wa=w)
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)
