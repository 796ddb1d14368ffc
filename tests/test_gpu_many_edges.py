"""Axes of hundreds to thousands of bins by edge tables: logarithmic s, linear
and logarithmic s_perp, irregular edges close together.  Counts equal the
oracle's, and the FP32 tables decide most pairs (few are left to the recheck)."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu

CLOSE = np.sort(np.concatenate([np.geomspace(0.5, 100.0, 300),
                                np.geomspace(0.5, 100.0, 300)[1:] * (1 - 2e-4)]))
AXES = {
    "iso_log": (0, dict(sedges=np.geomspace(0.5, 100.0, 3001)), 0.02),
    "iso_close": (0, dict(sedges=CLOSE), 0.6),
    "smu_log": (1, dict(sedges=np.geomspace(0.5, 100.0, 801), nmu=5), 0.02),
    "spi_lin": (2, dict(smin=0.0, ds=0.2, ns=500, pmin=0.0, dpi=5.0, np_=8), 0.05),
    "spi_lin_4000": (2, dict(smin=0.0, ds=0.025, ns=4000, pmin=0.0, dpi=10.0,
                             np_=4), 0.3),
    "spi_log": (2, dict(sedges=np.geomspace(0.1, 100.0, 1501), pmin=0.0, dpi=5.0,
                        np_=8), 0.05),
    "spi_plog": (2, dict(smin=0.0, ds=5.0, ns=20,
                         pedges=np.geomspace(0.05, 40.0, 801)), 0.05),
}


@pytest.mark.parametrize("name", sorted(AXES))
@pytest.mark.parametrize("geom", ["box", "survey"])
def test_many_edges(geom, name):
    import fcfc_gb300 as fg
    bt, ax, share = AXES[name]
    kw, ok = {}, dict(ax)
    for q, e, n in (("s", "sedges", "ns"), ("p", "pedges", "np_")):
        if e in ax:
            kw[e] = ax[e]
            ok[n] = len(ax[e]) - 1
        elif q + "min" in ax:
            d = "ds" if q == "s" else "dpi"
            kw.update({q + "min": ax[q + "min"], d: ax[d],
                       q + "max": ax[q + "min"] + ax[d] * ax[n]})
    if bt == 1:
        kw["nmu"] = ax["nmu"]
    rng = np.random.default_rng(3)
    a, b = rng.random((3000, 3)) * 300.0, rng.random((1500, 3)) * 300.0
    if geom == "box":
        kw["box"] = ok["box"] = 300.0
    else:
        a, b = a + [800.0, -100.0, -100.0], b + [800.0, -100.0, -100.0]
    pc, ob = fg.PairCounter(geom, bt, **kw), fo.Bins(geom == "survey", bt, **ok)
    pc.load(0, a)
    pc.load(1, b)
    for other in (None, 1):
        want = ob.count(a, b if other else None, mode=1)
        np.testing.assert_array_equal(pc.count_pairs(0, other), want)
        st = pc.stats()
        assert st["precision_used"] == fg.PREC_FP32_RECHECK
        assert st["in_range"] == want.sum()
        assert st["rechecked"] <= share * want.sum(), st["rechecked"] / want.sum()
    if geom == "box":
        cnt, status, _ = pc.count_batch([a, b], [300.0, 300.0])
        assert status == [0, 0]
        np.testing.assert_array_equal(cnt[0], ob.count(a, mode=1))
