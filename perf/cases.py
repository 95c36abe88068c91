"""The workloads that this framework's speed is measured on.

Every case goes through the public Python entry points (`desi_b200.api`): one
pass grids its catalogs (unless the case says `resident`: a service that keeps
gridded catalogs and counts them again) and counts the histograms of one
correlation function, on the host as the caller reads them.

Kinds of case:

* `pairs`     DD, RR and DR of a data and a random catalog, isotropic,
              anisotropic or both in one call;
* `rd`        one data catalog against several random catalogs of uneven
              sizes in one batched call (the `-rd` directory mode);
* `triplets`  DDD, RRR, DDR and DRR: isotropic (bins^3), anisotropic (bins^5),
              or isotropic through the reference program's node gates (what
              `PCF.out 3iso -bpc` writes);
* `analytic`  periodic DDD counted, DDR and RRR in closed form
              (`PCF.out 3iso -bpc -a`).

Data catalogs are clustered (Neyman-Scott, 64 Gaussian children of sigma 5 per
parent), random catalogs uniform; weights are 1 or drawn from U(0.5, 1.5).
"""
import math

import numpy as np
import torch

from desi_b200 import api

CHILDREN, SIGMA = 64, 5.0


def listed():
    return [
        # the smallest call: 1000 + 1000 points from numpy arrays, a notebook's or a
        # mock's quick look; launches, copies and host work are what it costs
        dict(name="2iso small", kind="pairs", ani="iso", nd=1000, nr=1000, box=250.0, bins=30, dmax=80.0,
             bpc=False, weighted=False, source="host"),
        # the headline workload: weighted periodic 2iso + 2ani of 32768 + 32768 points
        dict(name="2iso+2ani step", kind="pairs", ani="both", nd=32768, nr=32768, box=250.0, bins=30,
             dmax=80.0, bpc=True, weighted=True, source="device"),
        # a service's request on catalogs that stay gridded on the device, at odd sizes
        dict(name="2iso resident", kind="pairs", ani="iso", nd=83511, nr=150007, box=500.0, bins=37,
             dmax=97.5, bpc=False, weighted=True, source="device", resident=True),
        # large catalogs, anisotropic counts with unit weights
        dict(name="2ani large", kind="pairs", ani="ani", nd=700001, nr=1000000, box=1000.0, bins=50,
             dmax=100.0, bpc=True, weighted=False, source="device"),
        # survey-size catalogs at small separations: gridding the points is half the work
        dict(name="2iso sparse", kind="pairs", ani="iso", nd=6000000, nr=9000001, box=2000.0, bins=20,
             dmax=20.0, bpc=True, weighted=True, source="device"),
        # one data catalog against a directory of random catalogs of uneven sizes
        dict(name="rd 2ani", kind="rd", ani="ani", nd=100003, nrand=12, lo=25000, hi=200000, box=1000.0,
             bins=40, dmax=120.0, bpc=False, weighted=True, source="device"),
        # the smallest 3-point call
        dict(name="3iso small", kind="triplets", form="iso", nd=1000, nr=1000, box=250.0, bins=20, dmax=60.0,
             bpc=False, weighted=False, source="host"),
        # the 3-point workload: periodic 3iso, 30^3 bins, dmax 80 in a box of 250
        dict(name="3iso large", kind="triplets", form="iso", nd=24001, nr=24576, box=250.0, bins=30, dmax=80.0,
             bpc=True, weighted=False, source="device"),
        # the same with weights, at an ordinary size
        dict(name="3iso weighted", kind="triplets", form="iso", nd=4099, nr=4096, box=250.0, bins=25, dmax=70.0,
             bpc=False, weighted=True, source="device"),
        # what the command line's `3iso -bpc` runs: the reference's node gates, 35 nodes per side
        dict(name="3iso gated", kind="triplets", form="gated", nd=4096, nr=4100, box=250.0, bins=30, dmax=80.0,
             bpc=True, weighted=False, source="host", partitions=35),
        # anisotropic 3-point counts (bins^5)
        dict(name="3ani", kind="triplets", form="ani", nd=3000, nr=3001, box=250.0, bins=12, dmax=60.0,
             bpc=False, weighted=False, source="host"),
        # periodic 3iso with the closed-form DDR and RRR
        dict(name="3iso analytic", kind="analytic", nd=10007, nr=0, box=250.0, bins=20, dmax=60.0, bpc=True,
             weighted=False, source="device"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    form = rng.choice(["pairs", "pairs", "pairs", "rd", "iso", "iso", "gated", "ani", "analytic"])
    box = rng.choice([250.0, 500.0, 1000.0])
    c = dict(box=box, weighted=rng.random() < 0.5, bpc=rng.random() < 0.5, source=rng.choice(["host", "device"]))
    dmax = round(rng.uniform(40.0, 80.0 if box == 250.0 else 120.0), 1)
    if form == "pairs":
        if rng.random() < 0.25:  # survey size, small separations
            c.update(box=2000.0, source="device")
            dmax, hi = round(rng.uniform(10.0, 25.0), 1), 9000000
        else:
            hi = 1000000
        cap = 700000 * _neighbours(1000000, 1000.0, 100.0)
        n = log(1000, hi)
        while n * _neighbours(n, c["box"], dmax) > cap:
            n = int(n * 0.8)
        c.update(kind="pairs", ani=rng.choice(["iso", "ani", "both"]), nd=max(500, int(n * rng.uniform(0.6, 1.0))),
                 nr=n, bins=rng.randint(20, 50), dmax=dmax, resident=rng.random() < 0.25)
    elif form == "rd":
        hi = log(4000, 200000)
        while hi * _neighbours(hi, box, dmax) > 200000 * _neighbours(200000, 1000.0, 120.0):
            hi = int(hi * 0.8)
        c.update(kind="rd", ani=rng.choice(["iso", "ani"]), nd=max(500, int(hi * rng.uniform(0.3, 1.0))),
                 nrand=rng.randint(3, 12), lo=max(250, hi // 8), hi=hi, bins=rng.randint(20, 40), dmax=dmax)
    elif form == "analytic":
        n = log(2000, 10000)
        c.update(kind="analytic", nd=n, nr=0, box=250.0, bins=rng.randint(15, 20), dmax=round(rng.uniform(40.0, 60.0), 1),
                 bpc=True, weighted=False)
    else:
        top = {"iso": 3000 if c["weighted"] else 16000, "gated": 3000, "ani": 3000}[form]
        n = log(1000, top)
        c.update(kind="triplets", form=form, box=250.0, nd=max(500, int(n * rng.uniform(0.7, 1.0))), nr=n,
                 dmax=round(rng.uniform(40.0, 60.0 if form == "ani" or c["weighted"] else 80.0), 1),
                 bins=rng.randint(8, 12) if form == "ani" else rng.randint(15, 30))
        if form == "gated":
            c.update(bpc=True, partitions=rng.choice([20, 25, 35]))
        if form != "iso":
            c["weighted"] = c["weighted"] and rng.random() < 0.3
    return c


# --- inputs -----------------------------------------------------------------

def _points(n, box, seed, clustered, weighted):
    """(n, 4) float32 points x, y, z, w on the GPU, coordinates in [0, box)."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if clustered:
        parents = torch.rand(-(-n // CHILDREN), 3, generator=g, device="cuda", dtype=torch.float64) * box
        xyz = parents.repeat_interleave(CHILDREN, 0)[:n]
        xyz = torch.remainder(xyz + SIGMA * torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64), box)
    else:
        xyz = torch.rand(n, 3, generator=g, device="cuda", dtype=torch.float64) * box
    p = torch.ones(n, 4, device="cuda")
    p[:, :3] = xyz.float()
    p[:, :3][p[:, :3] >= box] = 0.0  # rounding to float32 may reach the box's face
    if weighted:
        p[:, 3] = torch.rand(n, generator=g, device="cuda") + 0.5
    # a file's rows are in no spatial order
    return p[torch.randperm(n, generator=g, device="cuda")].contiguous()


def _sizes(case, seed):
    """Sizes of the random catalogs: one, or for `rd` log-uniform in [lo, hi]."""
    if case["kind"] == "rd":
        u = np.random.RandomState(seed % (1 << 31)).rand(case["nrand"])
        return [int(round(case["lo"] * (case["hi"] / case["lo"]) ** v)) for v in u]
    return [case["nr"]] if case["nr"] else []


def _catalogs(case, seed):
    d = _points(case["nd"], case["box"], 1000 * seed + 1, True, case["weighted"])
    r = [_points(n, case["box"], 1000 * seed + 2 + i, False, case["weighted"])
         for i, n in enumerate(_sizes(case, seed))]
    return d, r


_context = None


def _ctx():
    """The program's one library context."""
    global _context
    if _context is None:
        _context = api.Context(0)
    return _context


class _State:
    pass


def _grid(s, pts):
    c = s.case
    part = c.get("partitions", 0)
    if isinstance(pts, np.ndarray):
        return s.ctx.grid(pts, c["box"], partitions=part)
    return s.ctx.grid(None, c["box"], partitions=part, device_ptr=pts.data_ptr(), n=len(pts))


def prepare(case, seed):
    s = _State()
    s.case, s.ctx = case, _ctx()
    s.d, s.r = _catalogs(case, seed)
    if case["source"] == "host":
        s.d, s.r = s.d.cpu().numpy(), [r.cpu().numpy() for r in s.r]
    torch.cuda.synchronize()  # the library reads the points on a stream of its own
    s.grids = None
    if case.get("resident"):
        s.grids = _grid(s, s.d), [_grid(s, r) for r in s.r]
    return s


def run(s):
    c = s.case
    gd, gr = s.grids or (_grid(s, s.d), [_grid(s, r) for r in s.r])
    kw = dict(bins=c["bins"], dmax=c["dmax"], bpc=c["bpc"])
    if c["kind"] == "pairs":
        kw["ani"] = {"iso": False, "ani": True, "both": "both"}[c["ani"]]
        return {"DD": s.ctx.count_pairs(gd, **kw), "RR": s.ctx.count_pairs(gr[0], **kw),
                "DR": s.ctx.count_pairs(gd, gr[0], **kw)}
    if c["kind"] == "rd":
        dd, rr, dr = s.ctx.batch_pairs(gd, gr, ani=c["ani"] == "ani", **kw)
        return {"DD": dd, "RR": rr, "DR": dr}
    if c["kind"] == "analytic":
        ddd, ddr, rrr = s.ctx.analytic_3iso(gd, bins=c["bins"], dmax=c["dmax"])
        return {"DDD": ddd, "DDR": ddr, "RRR": rrr}
    kw.update(ani=c["form"] == "ani", ref_gates=c["form"] == "gated")
    return {"DDD": s.ctx.count_triplets(gd, **kw), "RRR": s.ctx.count_triplets(gr[0], **kw),
            "DDR": s.ctx.count_triplets(gd, gr[0], **kw), "DRR": s.ctx.count_triplets(gr[0], gd, **kw)}


# --- what a pass cannot do without --------------------------------------------

def _neighbours(n, box, dmax, ani=False):
    """Mean points of a uniform catalog within reach of a point."""
    v = 2.0 * math.pi * dmax ** 3 if ani else 4.0 / 3.0 * math.pi * dmax ** 3
    return n * min(1.0, v / box ** 3)


def work(case):
    """Each point read once, each histogram written once; 8 flops per pair (or
    third side of a triangle) in range, for uniform catalogs."""
    nd, bins, dmax, box = case["nd"], case["bins"], case["dmax"], case["box"]
    if case["kind"] == "rd":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]) if case["hi"] > case["lo"] else case["hi"]
        rs = [mean] * case["nrand"]
    else:
        rs = [case["nr"]] if case["nr"] else []
    points = nd + sum(rs)
    if case["kind"] in ("pairs", "rd"):
        kinds = {"iso": [False], "ani": [True], "both": [False, True]}[case["ani"]]
        units = out = 0.0
        for ani in kinds:
            nb = lambda n: _neighbours(n, box, dmax, ani)  # noqa: E731
            units += nd * nb(nd) / 2 + sum(r * nb(r) / 2 + nd * nb(r) for r in rs)
            out += (1 + 2 * len(rs)) * (bins * bins if ani else bins)
    else:
        tri = lambda a, b, c: a * _neighbours(b, box, dmax) * _neighbours(c, box, dmax) * 15 / 32  # noqa: E731
        out = bins ** (5 if case.get("form") == "ani" else 3)
        if case["kind"] == "analytic":
            units, out = tri(nd, nd, nd) / 6, 3 * out
        else:
            r = rs[0]
            units, out = (tri(nd, nd, nd) + tri(r, r, r)) / 6 + (tri(nd, nd, r) + tri(r, r, nd)) / 2, 4 * out
    return {"bytes": 16.0 * points + 8.0 * out, "flops": 8.0 * units}


# --- the same in 64 bits -------------------------------------------------------
# The counting rules of include/pcf.h: separations of the float32 coordinates in
# 64 bits (minimum image in a periodic box), d^2 summed (x, y), z; in range below
# dmax^2 (rounded to float32), bin = int(sqrt(d^2) * floor(bins / dmax * 1e6) / 1e6).

def _rule(case):
    f = np.float32(case["dmax"])
    return math.floor(case["bins"] / float(f) * 1e6) / 1e6, float(f * f)


def _sep(case, a, b):
    """Components of b - a for all pairs of rows of a and b."""
    v = b[None, :, :3] - a[:, None, :3]
    if case["bpc"]:
        L = case["box"]
        v = torch.where(v > 0.5 * L, v - L, torch.where(v < -0.5 * L, v + L, v))
    return v.unbind(-1)


def _bins(case, d2, excl, le=False):
    """Bin of each squared separation, and which are counted."""
    ds, dd = _rule(case)
    b = (d2.sqrt() * ds).long()
    ok = ((d2 <= dd) if le else (d2 < dd)) & (b < case["bins"])
    return b, ok & (d2 > 0) if excl else ok


def _exact_pairs(case, x, y, ani):
    cross, bins, bpc = y is not None, case["bins"], case["bpc"]
    y = x if y is None else y
    h = torch.zeros(bins * bins if ani else bins, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 24) // len(y))
    for i in range(0, len(x), step):
        dx, dy, dz = _sep(case, x[i:i + step], y)
        if ani:
            excl = not (bpc and cross)
            bz, kz = _bins(case, dz * dz, excl, bpc)
            bp, kp = _bins(case, dx * dx + dy * dy, excl, bpc)
            b, k = bz * bins + bp, kz & kp
        else:
            b, k = _bins(case, (dx * dx + dy * dy) + dz * dz, not cross)
        w = x[i:i + step, 3, None] * y[None, :, 3]
        h += torch.bincount(b[k], weights=w[k], minlength=len(h))
    return h.reshape(bins, bins) if ani else h


def _exact_triplets(case, x, y, ani):
    """Ordered triangles: points 1 and 2 from x, point 3 from y (or x), the
    third side between the images of 2 and 3 nearest to 1."""
    mixed, bins, bpc = y is not None, case["bins"], case["bpc"]
    y = x if y is None else y
    h = torch.zeros(bins ** (5 if ani else 3), dtype=torch.float64, device="cuda")
    excl3 = bpc if mixed else True

    def side(a, c, excl):
        v = torch.stack(_sep(case, a[None], c))[:, 0]
        d2 = (v[0] * v[0] + v[1] * v[1]) + v[2] * v[2]
        b, k = _bins(case, d2, excl)
        if not ani:
            return v[:, k], b[k], None, c[k, 3]
        dz = v[2]
        if bpc:
            raw = (c[:, 2] - a[2]).abs()
            dz = torch.where(raw > 0.5 * case["box"], raw - case["box"], raw)
        t = ((1.0 + dz / d2.sqrt()) * (bins / 2.0)).nan_to_num(nan=-1.0)
        k &= (t >= 0) & (t.long() < bins)
        return v[:, k], b[k], t.long()[k], c[k, 3]

    for a in x:
        vj, bj, tj, wj = side(a, x, True)
        vk, bk, tk, wk = side(a, y, excl3) if mixed else (vj, bj, tj, wj)
        e = vk[:, None, :] - vj[:, :, None]
        d2 = (e[0] * e[0] + e[1] * e[1]) + e[2] * e[2]
        b, k = _bins(case, d2, excl3)
        if not mixed:
            k.fill_diagonal_(False)
        if ani:
            s = ((((bj[:, None] * bins + bk[None]) * bins + b) * bins + tj[:, None]) * bins) + tk[None]
        else:
            s = (bj[:, None] * bins + b) * bins + bk[None]
        w = a[3] * wj[:, None] * wk[None]
        h += torch.bincount(s[k], weights=w[k], minlength=len(h))
    return h.reshape((bins,) * (5 if ani else 3))


def exact(case, seed):
    c = case
    if c["kind"] in ("pairs", "rd"):
        sizes = _sizes(c, seed)
        tests = (c["nd"] ** 2 + sum(n * n + n * c["nd"] for n in sizes)) * (2 if c["ani"] == "both" else 1)
        if tests > 6e10:
            return None
    elif c["kind"] == "analytic" or c["form"] == "gated" or max(c["nd"], c["nr"]) > 4200:
        return None
    d, r = _catalogs(c, seed)
    d, r = d.double(), [p.double() for p in r]
    if c["kind"] == "triplets":
        ani = c["form"] == "ani"
        return {"DDD": _exact_triplets(c, d, None, ani), "RRR": _exact_triplets(c, r[0], None, ani),
                "DDR": _exact_triplets(c, d, r[0], ani), "DRR": _exact_triplets(c, r[0], d, ani)}
    kinds = {"iso": [False], "ani": [True], "both": [False, True]}[c["ani"]]

    def pairs(x, y=None):
        h = [_exact_pairs(c, x, y, ani) for ani in kinds]
        return tuple(h) if len(h) > 1 else h[0]

    if c["kind"] == "rd":
        return {"DD": pairs(d), "RR": torch.stack([pairs(p) for p in r]), "DR": torch.stack([pairs(d, p) for p in r])}
    return {"DD": pairs(d), "RR": pairs(r[0]), "DR": pairs(d, r[0])}
