"""The products of the adjoint one by one: isolated pairs, each alone in its bin,
with weights and cotangent entries whose remainders below 2^-30 are the
largest.  The documented bound per product is 1.5 2^-52 of the scales
(powers of two not below the largest weight and the largest entry, here 1)."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("geom", ["box", "survey"])
def test_products_within_a_unit(geom):
    import fcfc_gb300 as fg
    n = 1000
    kw = {"box": 450.0} if geom == "box" else {}
    pc = fg.PairCounter(geom, fg.BIN_ISO, smin=0, smax=20, ds=0.02, **kw)
    # pair i: separation in the middle of bin i, 45 from the next pair
    at = np.stack(np.meshgrid(*[np.arange(10) * 45.0] * 3), -1).reshape(n, 3)
    at += [10.0, 12.0, 12.0] if geom == "box" else [500.0, 12.0, 12.0]
    sep = np.zeros((n, 3))
    sep[:, 0] = 0.02 * (np.arange(n) + 0.5)
    worst = Fraction(0)
    for seed in range(8):
        rng = np.random.default_rng(seed)
        wa, wb, g = (np.floor((1 - 0.01 * rng.random((3, n))) * 2 ** 30) - 0.5 +
                     1e-3 * rng.random((3, n))) / 2 ** 30
        g *= rng.choice([-1.0, 1.0], n)
        pc.load(0, at, wa)
        pc.load(1, at + sep, wb)
        da, db = pc.adjoint(0, 1, g)
        st = pc.stats()
        assert st["precision_used"] == fg.PREC_FP32_RECHECK
        assert st["in_range"] == n and st["rechecked"] == 0
        for w, got in ((wb, da), (wa, db)):
            for i in range(n):
                exact = Fraction(w[i]) * Fraction(g[i])
                worst = max(worst, abs(Fraction(got[i]) - exact))
    assert worst * 2 ** 52 <= 1.5, float(worst * 2 ** 52)


def test_products_of_unit_weights_have_no_bias():
    """Unweighted catalogues: the mean error of 4000 products of a weight of 1
    and a random entry.  A product is rounded by at most 2^-53 either way; the mean
    error of rounding without a bias is below that over the root of their number,
    times 4 here."""
    import fcfc_gb300 as fg
    n = 4000
    pc = fg.PairCounter("box", fg.BIN_ISO, box=2000.0, smin=0, smax=20, ds=0.005)
    at = np.stack(np.meshgrid(*[np.arange(16) * 100.0] * 3), -1).reshape(-1, 3)[:n]
    at += 50.0
    sep = np.zeros((n, 3))
    sep[:, 0] = 0.005 * (np.arange(n) + 0.5)
    g = np.random.default_rng(3).uniform(0.5, 1.0, pc.ntot)
    pc.load(0, at)
    pc.load(1, at + sep)
    da, db = pc.adjoint(0, 1, g)
    assert pc.stats()["in_range"] == n
    assert 4 * pc.stats()["rechecked"] < n
    for got in (da, db):
        err = np.array([float(Fraction(x) - Fraction(y)) for x, y in zip(got, g)])
        assert abs(err.mean()) <= 4 * 2.0 ** -53 / n ** 0.5, err.mean() * 2 ** 52
