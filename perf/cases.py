"""Performance cases of the pair-counting engine.

Each case is one pass a user's program makes through the public Python entry
points: catalogues are loaded (device pointers, host arrays, or RA/Dec/z
converted on the device) and counted, so a pass holds the catalogue
preparation and the grid sort as well as the counting.  The binning set-up
(``PairCounter``) and, where a program would keep one, the count graph are
made once in ``prepare``.

Catalogues are those of the repository's own workloads: uniform and
Neyman-Scott periodic boxes (Poisson(100) children, sigma = 5 Mpc/h), boxes
of log-uniform size at a fixed density, and a survey footprint (RA 100-260
deg, sin(Dec) uniform over 0-60 deg, z a normal truncated to 0.4-0.7, FKP
weights).
"""
import math

import numpy as np
import torch

import fcfc_gb300 as fg

BINTYPE = {"iso": fg.BIN_ISO, "smu": fg.BIN_SMU, "spi": fg.BIN_SPI}
DENSITY = 2.5e-4                 # (h/Mpc)^3, the mock boxes' number density
SIGMA = 5.0                      # Mpc/h, offset of a child from its parent
CHILDREN = 100                   # mean children per parent
OMEGA_M = 0.31
C01 = 2997.92458                 # c / (100 km/s), Mpc/h
ZMU, ZSIG, ZLO, ZHI = 0.55, 0.10, 0.4, 0.7
SKY = math.radians(160.0) * math.sin(math.radians(60.0))   # steradians


def listed():
    box = {"kind": "box", "bins": "smu", "linear": True, "smin": 0.0,
           "smax": 200.0, "ns": 40, "nmu": 100, "pimax": 0.0,
           "weighted": False, "clustered": True, "float32": False,
           "host": False, "cross": 0, "fp64": False}
    sv = {"kind": "survey", "bins": "smu", "smax": 200.0, "ns": 40,
          "nmu": 100, "pimax": 0.0, "weighted": True, "graph": True}
    return [
        # a quick look at a small catalogue: latency and launches
        dict(box, name="box_small", n=2003, box=200.0, smax=40.0, ns=8,
             nmu=20),
        # a simulation snapshot with an analytic RR, xi(s, mu)
        dict(box, name="box_smu_1e5", n=100000, box=1000.0, clustered=False),
        # a large clustered galaxy mock with weights, xi(s, mu)
        dict(box, name="box_smu_wt_2e6", n=2000000, box=2000.0,
             weighted=True),
        # the same mock, projected correlation: log s_perp bins
        dict(box, name="box_spi_wt_2e6", n=2000000, box=2000.0, bins="spi",
             linear=False, smin=0.1, smax=100.0, pimax=40.0, nmu=1,
             weighted=True),
        # xi(r) in log bins of a catalogue the program holds in host memory
        dict(box, name="box_iso_log_host", n=400009, box=1170.0, bins="iso",
             linear=False, smin=0.5, smax=150.0, ns=30, nmu=1, float32=True,
             host=True),
        # two tracers of one box (sparse against dense), small scales left out
        dict(box, name="box_cross_smu", n=60000, cross=600000, box=1340.0,
             smin=5.0, smax=155.0, ns=30, nmu=60),
        # a check of the default against the all-FP64 counter
        dict(box, name="box_fp64_wt", n=30011, box=500.0, smax=120.0, ns=24,
             nmu=50, weighted=True, fp64=True),
        # many small mocks in one call
        {"kind": "batch", "name": "mocks_small", "mocks": 48, "nmin": 20000,
         "nmax": 60000, "smax": 150.0, "ns": 30, "nmu": 100,
         "weighted": False},
        # a covariance run: 256 mocks of very different size in one call
        {"kind": "batch", "name": "mocks_256", "mocks": 256, "nmin": 10000,
         "nmax": 1000000, "smax": 200.0, "ns": 40, "nmu": 100,
         "weighted": False},
        # Landy-Szalay counts of a survey from RA/Dec/z, xi(s, mu)
        dict(sv, name="survey_ls_smu", nd=400000, nr=4000000),
        # the same for w_p: log s_perp bins, pi_max = 40
        dict(sv, name="survey_ls_spi", nd=200003, nr=2000003, bins="spi",
             smax=100.0, nmu=1, pimax=40.0),
        # gradients of weighted survey counts with respect to the weights
        {"kind": "adjoint", "name": "survey_adjoint", "nd": 50000,
         "nr": 500000, "smax": 200.0, "ns": 40, "nmu": 100},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["box"] * 6 + ["batch"] * 2 + ["survey"] * 3 +
                      ["adjoint"] * 2 + ["fp64"])
    if kind in ("box", "fp64"):
        fp64 = kind == "fp64"
        n = int(_log(rng, 1000, 40000 if fp64 else 2000000))
        side = round((n / _log(rng, 1e-4, 4e-4)) ** (1 / 3), 2)
        bins = rng.choice(["iso", "smu", "smu", "spi"])
        linear = rng.random() < 0.65
        ns = rng.randint(8, 40)
        top = min(200.0, 0.45 * side)
        if linear:
            ds = max(1, math.floor(top * rng.uniform(0.5, 1.0) / ns))
            ns = max(4, min(ns, int(top // ds)))
            smin = float(rng.choice([0, 0, 0, ds]))
            smax = smin + ds * ns
            if smax > top:
                ns -= 1
                smax -= ds
        else:
            smin = round(_log(rng, 0.1, 2.0), 3)
            smax = round(top * rng.uniform(0.5, 1.0), 2)
        return {"kind": "box", "bins": bins, "linear": linear, "smin": smin,
                "smax": smax, "ns": ns,
                "nmu": rng.randint(10, 120) if bins == "smu" else 1,
                "pimax": float(rng.randint(10, int(min(60, 0.45 * side))))
                if bins == "spi" else 0.0,
                "weighted": rng.random() < 0.5,
                "clustered": rng.random() < 0.7,
                "float32": rng.random() < 0.3, "host": rng.random() < 0.3,
                "n": n, "box": side,
                "cross": 0 if fp64 or rng.random() < 0.75
                else int(_log(rng, 1000, 600000)),
                "fp64": fp64}
    if kind == "batch":
        nmin = int(_log(rng, 17000, 100000))
        nmax = int(nmin * rng.uniform(1.5, 8))
        return {"kind": "batch", "mocks": int(_log(rng, 2, 96)),
                "nmin": nmin, "nmax": nmax,
                "smax": float(5 * rng.randint(10, 40)), "ns": 0,
                "nmu": rng.randint(20, 120), "weighted": rng.random() < 0.3}
    nd = int(_log(rng, 5000, 300000 if kind == "survey" else 60000))
    nr = int(nd * rng.uniform(2, 10))
    if kind == "adjoint":
        return {"kind": "adjoint", "nd": nd, "nr": nr,
                "smax": float(5 * rng.randint(16, 40)), "ns": 0,
                "nmu": rng.randint(10, 120)}
    bins = rng.choice(["smu", "smu", "spi", "iso"])
    return {"kind": "survey", "bins": bins, "nd": nd, "nr": nr,
            "smax": float(5 * rng.randint(10, 40)), "ns": rng.randint(10, 40)
            if bins == "spi" else 0,
            "nmu": rng.randint(10, 120) if bins == "smu" else 1,
            "pimax": float(rng.randint(20, 80)) if bins == "spi" else 0.0,
            "weighted": rng.random() < 0.8, "graph": rng.random() < 0.5}


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + 17)
    return g


def _f64(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _box_points(g, n, side, clustered, float32):
    """n points of a periodic box, three FP64 columns."""
    if clustered:
        npar = max(1, round(n / CHILDREN))
        par = _f64(g, 3, npar) * side
        at = torch.randint(npar, (n,), generator=g, device="cuda")
        x = par[:, at] + SIGMA * torch.randn(3, n, generator=g, device="cuda",
                                             dtype=torch.float64)
        x = torch.remainder(x, side)
    else:
        x = _f64(g, 3, n) * side
    if float32:
        x = x.float().double()
    x = torch.where(x >= side, torch.zeros_like(x), x)
    return [c.contiguous() for c in x]


def _lognormal(g, n, sigma=0.3):
    return torch.exp(sigma * torch.randn(n, generator=g, device="cuda",
                                         dtype=torch.float64))


def _hz(z):
    return torch.sqrt(OMEGA_M * (1 + z) ** 3 + (1 - OMEGA_M))


def _comoving(z, order=40):
    """Flat LCDM comoving distance, Gauss-Legendre in FP64."""
    x, w = np.polynomial.legendre.leggauss(order)
    d = torch.zeros_like(z)
    for xi, wi in zip(x, w):
        d += wi / _hz(0.5 * z * (1 + xi))
    return d * (0.5 * C01) * z


def _survey_points(g, n):
    """RA, Dec (degrees) and redshift of n objects."""
    ra = 100.0 + 160.0 * _f64(g, n)
    dec = torch.rad2deg(torch.asin(_f64(g, n) *
                                   math.sin(math.radians(60.0))))
    lo, hi = (math.erf((v - ZMU) / ZSIG / math.sqrt(2)) for v in (ZLO, ZHI))
    u = lo + (hi - lo) * _f64(g, n)
    z = ZMU + ZSIG * math.sqrt(2) * torch.erfinv(u)
    return [ra, dec, z.clamp(ZLO, ZHI)]


def _fkp(z, n, p0=1e4):
    """FKP weights 1 / (1 + n(z) P0) for n objects over the footprint."""
    nrm = 0.5 * (math.erf((ZHI - ZMU) / ZSIG / math.sqrt(2)) -
                 math.erf((ZLO - ZMU) / ZSIG / math.sqrt(2)))
    pdf = torch.exp(-0.5 * ((z - ZMU) / ZSIG) ** 2) / (
        ZSIG * math.sqrt(2 * math.pi) * nrm)
    vol = SKY * _comoving(z, 16) ** 2 * C01 / _hz(z)
    return 1.0 / (1.0 + p0 * n * pdf / vol)


def _xyz(rdz):
    ra, dec, z = rdz
    d = _comoving(z)
    a, b = torch.deg2rad(ra), torch.deg2rad(dec)
    return [d * torch.cos(b) * torch.cos(a), d * torch.cos(b) * torch.sin(a),
            d * torch.sin(b)]


def _ns(case):
    return case["ns"] or int(case["smax"] // 5)


def _counter(case):
    kind = case["kind"]
    kw = {}
    bins = case.get("bins", "smu")
    if bins == "smu":
        kw["nmu"] = case["nmu"]
    if bins == "spi":
        kw.update(pmin=0, pmax=case["pimax"], dpi=1)
    if kind == "box" and not case["linear"] or \
            kind == "survey" and bins == "spi":
        kw["sedges"] = np.geomspace(case.get("smin", 0.1), case["smax"],
                                    case["ns"] + 1)
    else:
        smin = case.get("smin", 0.0)
        kw.update(smin=smin, smax=case["smax"],
                  ds=(case["smax"] - smin) / _ns(case))
    if kind in ("box", "batch"):
        return fg.PairCounter("box", BINTYPE[bins],
                              box=case["box"] if kind == "box" else 1e4, **kw)
    return fg.PairCounter("survey", BINTYPE[bins], **kw)


def _inputs(case, seed):
    """The catalogues of a case: columns and weights on the GPU."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "box":
        cats = []
        for n in (case["n"], case["cross"]):
            if n:
                cats.append((_box_points(g, n, case["box"], case["clustered"],
                                         case["float32"]),
                             _lognormal(g, n) if case["weighted"] else None))
        return cats
    if kind == "batch":
        # log-uniform sizes at evenly spaced quantiles, in a fixed order
        m = case["mocks"]
        order = np.random.default_rng(7).permutation(m)
        cats = []
        for k in order:
            n = round(case["nmin"] * (case["nmax"] / case["nmin"]) **
                      ((k + 0.5) / m))
            side = float(np.float32((n / DENSITY) ** (1 / 3)))
            cats.append((_box_points(g, n, side, True, False),
                         _lognormal(g, n) if case["weighted"] else None,
                         side))
        return cats
    d, r = _survey_points(g, case["nd"]), _survey_points(g, case["nr"])
    if kind == "adjoint":
        return [(_xyz(d), _lognormal(g, case["nd"])), (_xyz(r), None)]
    w = case["weighted"]
    return [(d, _fkp(d[2], case["nd"]) if w else None),
            (r, _fkp(r[2], case["nd"]) if w else None)]


def _cotangent(case, seed):
    return np.random.default_rng(seed).normal(size=_ns(case) * case["nmu"])


def _load(pc, slot, cat, radecz=False):
    x, w = cat
    p = [c.data_ptr() for c in x]
    (pc.load_radecz_device if radecz else pc.load_device)(
        slot, *p, len(x[0]), None if w is None else w.data_ptr())


LS = ((0, None), (0, 1), (1, None))        # DD, DR, RR


def prepare(case, seed):
    cats = _inputs(case, seed)
    pc = _counter(case)
    st = {"case": case, "pc": pc, "cats": cats}
    if case["kind"] == "box" and case["host"]:
        st["host"] = [(tuple(c.cpu().numpy() for c in x),
                       None if w is None else w.cpu().numpy())
                      for x, w in cats]
    if case["kind"] == "batch":
        st["ptrs"] = [tuple(c.data_ptr() for c in x) + (len(x[0]),)
                      for x, _, _ in cats]
        st["sides"] = [s for _, _, s in cats]
        st["wptrs"] = [w.data_ptr() for _, w, _ in cats] \
            if case["weighted"] else None
    if case["kind"] == "survey" and case["graph"]:
        torch.cuda.synchronize()
        for slot, cat in enumerate(cats):
            _load(pc, slot, cat, True)
        st["graph"] = pc.count_graph([(a, b, case["weighted"])
                                      for a, b in LS])
    if case["kind"] == "adjoint":
        st["g"] = _cotangent(case, seed)
    return st


def run(state):
    case, pc, cats = state["case"], state["pc"], state["cats"]
    kind = case["kind"]
    if kind == "box":
        if case["host"]:
            for slot, (x, w) in enumerate(state["host"]):
                pc.load(slot, x, w)
        else:
            for slot, cat in enumerate(cats):
                _load(pc, slot, cat)
        return pc.count_pairs(
            0, 1 if case["cross"] else None, weighted=case["weighted"],
            precision=fg.PREC_FP64 if case["fp64"] else fg.PREC_FP32_RECHECK)
    if kind == "batch":
        cnt, status, sumw = pc.count_batch(
            state["ptrs"], state["sides"], weights=state["wptrs"],
            weighted=case["weighted"], on_device=True)
        return {"counts": np.stack(cnt), "status": np.array(status),
                "sumw": np.array(sumw)}
    if kind == "survey":
        for slot, cat in enumerate(cats):
            _load(pc, slot, cat, True)
        if case["graph"]:
            return state["graph"].run()
        return [pc.count_pairs(a, b, weighted=case["weighted"])
                for a, b in LS]
    for slot, cat in enumerate(cats):
        _load(pc, slot, cat)
    dd = pc.count_pairs(0, weighted=True)
    dr = pc.count_pairs(0, 1, weighted=True)
    gdd, _ = pc.adjoint(0, None, state["g"])
    gdr_d, gdr_r = pc.adjoint(0, 1, state["g"])
    return [dd, dr, gdd, gdr_d, gdr_r]


# ------------------------------------------------------------------ work

def _volume(case):
    """Volume of pairs that count (a ball, a shell or a cylinder)."""
    if case.get("bins") == "spi":
        return math.pi * case["smax"] ** 2 * 2 * case["pimax"]
    smin = case.get("smin", 0.0)
    return 4 / 3 * math.pi * (case["smax"] ** 3 - smin ** 3)


def _box_pairs(case, n, side, cross=0, clustered=True):
    v = _volume(case) / side ** 3
    if cross:
        return n * cross * v
    return 0.5 * n * n * v + (0.5 * n * CHILDREN if clustered else 0)


def work(case):
    """bytes: the catalogues read once, the histograms or gradients written
    once.  flops: 10 FP32 operations per in-range pair (8 without mu): the
    separation, its square and the bin; pairs expected from the mean
    densities (surveys: the footprint's, edges neglected)."""
    kind = case["kind"]
    col = 32 if case.get("weighted", True) else 24
    per = 10 if case.get("bins", "smu") == "smu" else 8
    out = 8 * _ns(case) * max(case["nmu"], int(case.get("pimax", 0)) or 1)
    if kind == "box":
        return {"bytes": col * (case["n"] + case["cross"]) + out,
                "flops": per * _box_pairs(case, case["n"], case["box"],
                                          case["cross"], case["clustered"])}
    if kind == "batch":
        b = f = 0
        for k in range(case["mocks"]):
            n = case["nmin"] * (case["nmax"] / case["nmin"]) ** (
                (k + 0.5) / case["mocks"])
            side = (n / DENSITY) ** (1 / 3)
            if side > 2 * case["smax"]:
                b += col * n + out
                f += per * _box_pairs(case, n, side)
        return {"bytes": b, "flops": f}
    z = torch.tensor([ZLO, ZHI], dtype=torch.float64)
    r = _comoving(z)
    v = _volume(case) / (SKY / 3 * float(r[1] ** 3 - r[0] ** 3))
    nd, nr = case["nd"], case["nr"]
    if kind == "survey":
        return {"bytes": col * (nd + nr) + 3 * out,
                "flops": per * v * (0.5 * nd * nd + nd * nr + 0.5 * nr * nr)}
    return {"bytes": 32 * nd + 24 * nr + 2 * out + 8 * (2 * nd + nr),
            "flops": 2 * per * v * (0.5 * nd * nd + nd * nr)}


# ------------------------------------------------------------ 64-bit values

PAIRS_MOST = 3e10      # pairs a 64-bit brute-force pass may visit


def _edges2(case):
    if case["kind"] == "box" and not case["linear"] or \
            case.get("bins") == "spi":
        e = np.geomspace(case.get("smin", 0.1), case["smax"], case["ns"] + 1)
    else:
        smin, ns = case.get("smin", 0.0), _ns(case)
        e = smin + (case["smax"] - smin) / ns * np.arange(ns + 1)
    return torch.from_numpy(e * e).cuda()


def _brute(case, a, b, g=None):
    """Weighted counts of catalogues a and b (b None: pairs of a, once) in
    64 bits, or with a cotangent g the gradients (of a's and of b's weights)
    of the sum of g times the counts."""
    auto = b is None
    xa, wa = a
    xb, wb = a if auto else b
    na, nb = len(xa[0]), len(xb[0])
    wa = torch.ones_like(xa[0]) if wa is None else wa
    wb = torch.ones_like(xb[0]) if wb is None else wb
    e2 = _edges2(case)
    ns = len(e2) - 1
    bins = case.get("bins", "smu")
    nq = case["nmu"] if bins == "smu" else (int(case["pimax"])
                                            if bins == "spi" else 1)
    box = case["box"] if case["kind"] == "box" else None
    cnt = torch.zeros(ns * nq + 1, dtype=torch.float64, device="cuda")
    if g is not None:
        gx = torch.cat([torch.from_numpy(g).cuda(), cnt.new_zeros(1)])
        da, db = torch.zeros_like(wa), torch.zeros_like(wb)
    step = max(1, int(2 ** 25 // nb))
    for i in range(0, na, step):
        j = min(na, i + step)
        d, m = [], []
        for k in range(3):
            dk = xa[k][i:j, None] - xb[k][None, :]
            if box:
                dk -= box * torch.round(dk / box)
            d.append(dk)
        s2 = d[0] * d[0] + d[1] * d[1]
        if box:
            pi2 = d[2] * d[2]
        else:
            m = [xa[k][i:j, None] + xb[k][None, :] for k in range(3)]
            dm = d[0] * m[0] + d[1] * m[1] + d[2] * m[2]
            pi2 = dm * dm / (m[0] * m[0] + m[1] * m[1] + m[2] * m[2])
        if not (box and bins == "spi"):
            s2 = s2 + d[2] * d[2]
        ok = torch.ones_like(s2, dtype=torch.bool)
        q = torch.zeros_like(s2, dtype=torch.int64)
        if bins == "spi":
            if not box:
                s2 = s2 - pi2
            q = torch.sqrt(pi2).long()
        elif bins == "smu":
            q = torch.nan_to_num(torch.sqrt(pi2 / s2) * nq).long()
        k = torch.bucketize(s2, e2, right=True) - 1
        ok = (q < nq) & (k >= 0) & (k < ns)
        if auto:
            ok[torch.arange(j - i), torch.arange(i, j)] = False
        idx = torch.where(ok, k + q * ns, ns * nq)
        if g is None:
            cnt += torch.bincount(idx.reshape(-1), minlength=ns * nq + 1,
                                  weights=(wa[i:j, None] *
                                           wb[None, :]).reshape(-1))
        else:
            G = gx[idx]
            da[i:j] = G @ wb
            db += wa[i:j] @ G
    if g is None:
        return (cnt[:-1] * (0.5 if auto else 1)).cpu().numpy()
    return da.cpu().numpy(), db.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch" or kind != "adjoint" and not case["weighted"]:
        return None

    def most(na, nb):
        return na * nb <= PAIRS_MOST
    if kind == "box":
        n, m = case["n"], case["cross"]
        if not most(n, m or n):
            return None
        cats = _inputs(case, seed)
        return _brute(case, cats[0], cats[1] if m else None)
    nd, nr = case["nd"], case["nr"]
    if not most(nd, nd):
        return None
    cats = _inputs(case, seed)
    if kind == "survey":
        cats = [(_xyz(x), w) for x, w in cats]
        return [_brute(case, cats[0], None),
                _brute(case, cats[0], cats[1]) if most(nd, nr) else None,
                _brute(case, cats[1], None) if most(nr, nr) else None]
    g = _cotangent(case, seed)
    far = most(nd, nr)
    gdr = _brute(case, *cats, g) if far else (None, None)
    return [_brute(case, cats[0], None),
            _brute(case, *cats) if far else None,
            _brute(case, cats[0], None, g)[0], gdr[0], gdr[1]]
