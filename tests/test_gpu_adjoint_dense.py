"""Gradients of dense clumps: unit weights and a cotangent of 1, -1 or both in
sign, every pair in range, so that a point's gradient is its number of
neighbours, times that: sums of the largest terms there are, over hundreds of
blocks of 32 points of one cell.  Integers below 2^53: equal, not close."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clump(n, centre, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    x *= (rng.random(n) ** (1 / 3) / np.linalg.norm(x, axis=1))[:, None]
    return x + centre


@pytest.mark.parametrize("g", [1.0, -1.0, 0.5])
@pytest.mark.parametrize("geom,bintype", [("box", 0), ("box", 1), ("survey", 0),
                                          ("survey", 1)])
def test_dense_clump_gradients(geom, bintype, g):
    import fcfc_gb300 as fg
    kw = dict(smin=0, smax=20, ds=20)
    if bintype == 1:
        kw.update(nmu=2, with_mu_one=True)
    if geom == "box":
        kw["box"] = 200.0
    centre = [70.0, 70.0, 70.0] if geom == "box" else [900.0, 200.0, -300.0]
    pc = fg.PairCounter(geom, bintype, **kw)
    # (a block of A is dealt in up to 16 parts: 5 groups of 32 blocks each)
    n, m = 3000, 80000 + 37
    pc.load(0, _clump(n, centre, 1))
    pc.load(1, _clump(m, centre, 2))
    cot = np.full(pc.ntot, g)
    dw, _ = pc.adjoint(1, None, cot)
    assert pc.stats()["precision_used"] == fg.PREC_FP32_RECHECK
    np.testing.assert_array_equal(dw, np.full(m, g * (m - 1)))
    da, db = pc.adjoint(0, 1, cot)
    np.testing.assert_array_equal(da, np.full(n, g * m))
    np.testing.assert_array_equal(db, np.full(m, g * n))
