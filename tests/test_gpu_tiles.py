"""The FP32 tile kernel at its edges: catalogues around multiples of a block
of 32 points, bins that start away from zero (columns and rows around the
bins), linear, logarithmic and irregular axes, dense cells and one cell, auto
and cross counts, against the oracle; the in-range statistic against the
unweighted counts; and histograms that do not fit in shared memory."""
import numpy as np
import pytest

from oracle import fcfc_oracle as fo

pytestmark = pytest.mark.gpu

SMU = dict(bintype=1, smin=0.0, ds=5.0, ns=8, nmu=13)
BINS = {
    "smu": SMU,
    "smu_smin": dict(SMU, smin=7.5),
    "iso": dict(bintype=0, smin=0.0, ds=2.0, ns=20),
    "iso_smin": dict(bintype=0, smin=3.0, ds=2.0, ns=18),
    "iso_log": dict(bintype=0, sedges=np.geomspace(0.3, 40.0, 12)),
    "iso_odd": dict(bintype=0, sedges=np.array([0.0, 1.3, 7.7, 7.9, 31.0, 40.0])),
    "smu_log": dict(bintype=1, sedges=np.geomspace(0.5, 40.0, 9), nmu=7),
    "spi": dict(bintype=2, smin=0.0, ds=4.0, ns=10, pmin=0.0, dpi=3.0, np_=9),
    "spi_min": dict(bintype=2, smin=2.0, ds=4.0, ns=9, pmin=4.5, dpi=3.0, np_=8),
    "spi_log": dict(bintype=2, sedges=np.geomspace(0.2, 40.0, 11), pmin=0.0,
                    dpi=2.5, np_=12),
    "spi_odd": dict(bintype=2, sedges=np.geomspace(0.2, 40.0, 11),
                    pedges=np.array([0.5, 1.0, 4.0, 4.1, 17.0, 30.0])),
}


def _pair(geom, kw, box=None):
    import fcfc_gb300 as fg
    kw = dict(kw)
    bt = kw.pop("bintype")
    args = {}
    if "sedges" in kw:
        args["sedges"] = kw["sedges"]
    else:
        args.update(smin=kw["smin"], ds=kw["ds"],
                    smax=kw["smin"] + kw["ds"] * kw["ns"])
    if bt == 1:
        args["nmu"] = kw["nmu"]
    if bt == 2:
        if "pedges" in kw:
            args["pedges"] = kw["pedges"]
        else:
            args.update(pmin=kw["pmin"], dpi=kw["dpi"],
                        pmax=kw["pmin"] + kw["dpi"] * kw["np_"])
    pc = fg.PairCounter(geom, bt, box=box, **args)
    ok = {k: v for k, v in kw.items() if k in ("sedges", "pedges", "ns", "smin", "ds",
                                               "nmu", "pmin", "dpi")}
    if bt == 2:
        ok["np_"] = len(kw["pedges"]) - 1 if "pedges" in kw else kw["np_"]
    if "sedges" in kw:
        ok["ns"] = len(kw["sedges"]) - 1
    if box is not None:
        ok["box"] = box
    return pc, fo.Bins(geom == "survey", bt, **ok)


def _points(geom, n, box, seed):
    rng = np.random.default_rng(seed)
    if geom == "box":
        x = rng.random((n, 3)) * box
        x[: n // 3] = np.mod(x[0] + rng.normal(0, 4.0, (n // 3, 3)), box)
        return x
    x = rng.random((n, 3)) * 120.0 + np.array([400.0, -60.0, -60.0])
    x[: n // 4] = rng.normal(0, 30.0, (n // 4, 3))    # around the observer
    return x


@pytest.mark.parametrize("name", sorted(BINS))
@pytest.mark.parametrize("geom", ["box", "survey"])
def test_tile_edges(geom, name):
    box = 130.0 if geom == "box" else None
    pc, ob = _pair(geom, BINS[name], box)
    for n, m in ((1, 1), (31, 33), (32, 64), (65, 1), (97, 700), (2049, 130)):
        a, b = _points(geom, n, box, n), _points(geom, m, box, 1000 + m)
        w = np.random.default_rng(5).normal(1.0, 0.6, n)     # some negative
        pc.load(0, a, w)
        pc.load(1, b)
        for other, want, wantw in (
                (None, ob.count(a, mode=1), ob.count(a, wa=w, mode=1)),
                (1, ob.count(a, b, mode=1), ob.count(a, b, wa=w, mode=1))):
            np.testing.assert_array_equal(pc.count_pairs(0, other), want)
            st = pc.stats()
            assert st["precision_used"] == 0 and st["in_range"] == want.sum()
            got = pc.count_pairs(0, other, weighted=True)
            np.testing.assert_allclose(got, wantw, rtol=1e-10, atol=1e-10)
            assert pc.stats()["in_range"] == want.sum()


def test_one_cell_and_global_histogram():
    """A dense box of one coarse cell, with histograms within and beyond
    shared memory (bins counted in global memory), batched and single."""
    box = 60.0
    x = _points("box", 3000, box, 3)
    w = np.random.default_rng(4).lognormal(0, 0.3, len(x))
    for ns, nmu in ((20, 10), (800, 100)):
        kw = dict(bintype=1, smin=0.0, ds=20.0 / ns, ns=ns, nmu=nmu)
        pc, ob = _pair("box", kw, box)
        want, wantw = ob.count(x, mode=1), ob.count(x, wa=w, mode=1)
        pc.load(0, x, w)
        np.testing.assert_array_equal(pc.count_pairs(0), want)
        assert pc.stats()["in_range"] == want.sum()
        np.testing.assert_allclose(pc.count_pairs(0, weighted=True), wantw,
                                   rtol=1e-10, atol=1e-10)
        assert pc.stats()["in_range"] == want.sum()
        cnt, status, _ = pc.count_batch([x, x[:40], x[:0]], [box, box, box])
        assert status == [0, 0, 0]
        np.testing.assert_array_equal(cnt[0], want)
        np.testing.assert_array_equal(cnt[1], ob.count(x[:40], mode=1))
        assert cnt[2].sum() == 0


@pytest.mark.parametrize("name", sorted(BINS))
@pytest.mark.parametrize("geom", ["box", "survey"])
def test_tile_fp64(geom, name):
    """The tiles with every pair in FP64: catalogues around a block, integer
    coordinates (separations and mu on the bin edges), and lengths whose
    squares FP32 does not hold.  Weighted sums: FP64 additions in any order,
    at most 2e6 terms of at most 10 each, of which a bin's sum loses less
    than 2e6 eps = 4.4e-10 of their absolute sum."""
    import fcfc_gb300 as fg
    for n, m, scale in ((1, 1, 1.0), (31, 33, 1.0), (97, 700, 1.0),
                        (2049, 130, 1.0), (300, 65, 1e20)):
        if scale != 1.0 and (geom == "survey" or name not in ("smu", "iso_smin")):
            continue
        kw = dict(BINS[name])
        if scale != 1.0:
            kw.update(smin=kw["smin"] * scale, ds=kw["ds"] * scale)
        box = 130.0 * scale if geom == "box" else None
        pc, ob = _pair(geom, kw, box)
        for whole in (False, True):
            a, b = _points(geom, n, 130.0, n), _points(geom, m, 130.0, 1000 + m)
            if whole:
                a, b = np.floor(a), np.floor(b)
            a, b = a * scale, b * scale
            w = np.random.default_rng(5).normal(1.0, 0.6, n)
            pc.load(0, a, w)
            pc.load(1, b)
            for other, want, wantw, tot in (
                    (None, ob.count(a, mode=1), ob.count(a, wa=w, mode=1),
                     ob.count(a, wa=np.abs(w), mode=1)),
                    (1, ob.count(a, b, mode=1), ob.count(a, b, wa=w, mode=1),
                     ob.count(a, b, wa=np.abs(w), mode=1))):
                got = pc.count_pairs(0, other, precision=fg.PREC_FP64)
                np.testing.assert_array_equal(got, want)
                st = pc.stats()
                assert st["precision_used"] == fg.PREC_FP64
                assert st["in_range"] == want.sum()
                got = pc.count_pairs(0, other, weighted=True,
                                     precision=fg.PREC_FP64)
                assert (np.abs(got - wantw) <= 4.4e-10 * tot).all()
                assert pc.stats()["in_range"] == want.sum()


@pytest.mark.parametrize("ns", [1, 20, 190, 191, 500, 3000, 6000])
def test_weighted_s_histogram_copies(ns):
    """Weighted s bins: 32 copies of the shared histogram down to one, and
    none in shared memory, in a box and in a batch."""
    box = 130.0
    kw = dict(bintype=0, smin=0.0, ds=40.0 / ns, ns=ns)
    pc, ob = _pair("box", kw, box)
    x = _points("box", 2100, box, ns)
    w = np.random.default_rng(6).normal(1.0, 0.6, len(x))
    want, tot = ob.count(x, wa=w, mode=1), ob.count(x, wa=np.abs(w), mode=1)
    pc.load(0, x, w)
    for _ in range(2):
        got = pc.count_pairs(0, weighted=True)
        assert (np.abs(got - want) <= 1e-10 * tot + 1e-300).all()
    cnt, status, _ = pc.count_batch([x, x[:70]], [box, box],
                                    weights=[w, w[:70]], weighted=True)
    assert status == [0, 0]
    assert (np.abs(cnt[0] - want) <= 1e-10 * tot + 1e-300).all()
