"""Gradients of counts with more bins than the shared cotangent table holds, and
with more than 2^22 (the words a float numbers exactly), against the oracle.
Tolerance: a term is within 2^-49 max|w| max|g| of the product, and the
oracle's sum of n products in FP64 within n^2 2^-53 max|w| max|g| of theirs."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,dpi", [(20, 0.015), (419, 0.003), (600, 0.003)])
@pytest.mark.parametrize("geom", ["box", "survey"])
def test_gradients_of_many_bins(geom, ns, dpi):
    import fcfc_gb300 as fg
    edges = np.geomspace(10.0, 40.0, ns + 1)
    kw = {"box": 130.0} if geom == "box" else {}
    pc = fg.PairCounter(geom, fg.BIN_SPI, sedges=edges, pmin=0, pmax=30,
                        dpi=dpi, **kw)
    npi = round(30 / dpi)
    ob = fo.Bins(geom == "survey", 2, ns=ns, sedges=edges, np_=npi, pmin=0,
                 dpi=dpi, **kw)
    rng = np.random.default_rng(ns)
    a, b = (rng.random((n, 3)) * 110.0 for n in (400, 300))
    if geom == "survey":
        a, b = a + [400.0, -50.0, -50.0], b + [400.0, -50.0, -50.0]
    wa, wb = rng.normal(1.0, 0.6, len(a)), rng.normal(1.0, 0.6, len(b))
    g = rng.normal(size=pc.ntot)
    pc.load(0, a, wa)
    pc.load(1, b, wb)
    wm, gm = max(np.abs(wa).max(), np.abs(wb).max()), np.abs(g).max()
    tol = len(a) * (2.0 ** -49 + len(a) * 2.0 ** -53) * wm * gm
    got, _ = pc.adjoint(0, None, g)
    st = pc.stats()
    assert st["precision_used"] == fg.PREC_FP32_RECHECK
    assert 2 * st["rechecked"] < st["in_range"]      # most by the table
    want, _ = ob.adjoint(a, g, wa=wa)
    assert np.abs(want).max() > 1.0
    np.testing.assert_allclose(got, want, rtol=0, atol=tol)
    da, db = pc.adjoint(0, 1, g)
    wda, wdb = ob.adjoint(a, g, b=b, wa=wa, wb=wb)
    np.testing.assert_allclose(da, wda, rtol=0, atol=tol)
    np.testing.assert_allclose(db, wdb, rtol=0, atol=tol)
