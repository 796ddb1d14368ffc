"""Weighted sums whose shared words overflow many times, on either side: clumps
whose pairs all fall into one s bin, with products of -1 and -1/4 of the weights'
scales and of both signs.  Every product is a multiple of 2^-2 and every sum
below 2^53 of them, so that the engine's exact sums equal the closed forms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 1 << 16


def _clump(n, centre, seed):
    """n points in a ball of radius 1, and one out of range of all others."""
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    x *= (rng.random(n) ** (1 / 3) / np.linalg.norm(x, axis=1))[:, None]
    x += centre
    return np.concatenate([x, [np.asarray(centre) + 60.0]])


def _weights(kind, n, seed):
    if kind == "minus_1":
        return np.ones(n), -np.ones(n)
    if kind == "minus_quarter":          # (the far points' weight of 1 is the scale)
        return np.full(n, 0.5), np.full(n, -0.5)
    rng = np.random.default_rng(seed)    # 52 % of +1, 48 % of -1
    return np.ones(n), np.where(rng.random(n) < 0.52, 1.0, -1.0)


@pytest.mark.parametrize("kind", ["minus_1", "minus_quarter", "mixed"])
@pytest.mark.parametrize("geom,bintype", [("box", 0), ("box", 1), ("survey", 0),
                                          ("survey", 1)])
def test_negative_products(geom, bintype, kind):
    import fcfc_gb300 as fg
    kw = dict(smin=0, smax=20, ds=20)
    if bintype == 1:
        kw.update(nmu=2, with_mu_one=True)   # (a mu that rounds to 1 counts)
    if geom == "box":
        kw["box"] = 200.0
    centre = [70.0, 70.0, 70.0] if geom == "box" else [900.0, 200.0, -300.0]
    pc = fg.PairCounter(geom, bintype, **kw)
    wa, wb = _weights(kind, N, 3)
    # the far points coincide with nothing: one on either side of the clump
    a, b = _clump(N, centre, 1), _clump(N, centre, 2)
    a[-1] -= 120.0
    pc.load(0, a, np.append(wa, 1.0))
    pc.load(1, b, np.append(wb, 1.0))
    got = pc.count_pairs(0, 1, weighted=True)
    assert got.sum() == wa.sum() * wb.sum()


@pytest.mark.parametrize("bintype", [0, 1])
def test_mixed_signs_auto_and_batch(bintype):
    """Auto counts: sum over i < j of w_i w_j = ((sum w)^2 - sum w^2) / 2."""
    import fcfc_gb300 as fg
    kw = dict(smin=0, smax=20, ds=20)
    if bintype == 1:
        kw.update(nmu=2, with_mu_one=True)   # (a mu that rounds to 1 counts)
    pc = fg.PairCounter("box", bintype, box=200.0, **kw)
    cats, ws, want = [], [], []
    for k, share in enumerate((0.75, 0.9)):
        x = _clump(N, [70.0, 70.0, 70.0], 10 + k)
        w = np.where(np.random.default_rng(20 + k).random(N) < share, 1.0, -1.0)
        cats.append(x)
        ws.append(np.append(w, 1.0))
        want.append((w.sum() ** 2 - N) / 2)
    for x, w, t in zip(cats, ws, want):
        pc.load(0, x, w)
        assert pc.count_pairs(0, weighted=True).sum() == t
    cnt, status, _ = pc.count_batch(cats, [200.0, 200.0], weights=ws,
                                    weighted=True)
    assert status == [0, 0]
    assert [c.sum() for c in cnt] == want
