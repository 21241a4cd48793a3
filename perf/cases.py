"""The measured work of this library: pair counts as a user's program runs them.

A case is one pass through the public Python binding of the C ABI: a cross
count (one corels2 call), an auto count (one corels1 call), a batch of boxes,
or the four terms of a sky run, on catalogues of the shapes and distributions
that this repository's benchmark, configurations and tests use.  Unless a case
says `upload`, its catalogues are in the context's slots before the pass, as a
program keeps them that counts several terms of one run.

Everything below is seeded; `exact` restates the counts and accumulators in
64-bit torch without this library's code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from corr_pc_gb300 import _lib, synth

C_KMS = 299792.458
BOX = dict(kind="box", which=0, n_s=20000, n_d=0, L=250.0, clustered=False, sigma=2.0, f32=False,
           weights=False, jk_side=2, nrp=10, npi=20, rmin=0.1, rmax=20.0, pmax=100.0, lin=False,
           upload=False)
SKY = dict(kind="sky", which=1, n_s=2000, n_r=20000, jk_side=10, nrp=15, npi=30, rmin=0.3,
           rmax=60.0, pmax=60.0, chi_min=500.0, chi_max=1500.0)


def listed():
    return [
        # one small sub-volume or test catalogue: the call is latency, launches
        # and the host path; linear bins and no jackknife, as quick looks use
        dict(BOX, name="box_wgg_2k_linear", n_s=2000, L=100.0, jk_side=0, lin=True, nrp=20,
             npi=10, rmin=0.0, rmax=25.0, pmax=40.0),
        # the 20,000-point uniform box: wgg with 8 cubes
        dict(BOX, name="box_wgg_20k", f32=False),
        # the 200k clustered box, wg+ with 64 cubes, catalogues resident
        dict(BOX, name="box_wgp_200k", which=1, n_s=200003, L=500.0, clustered=True, f32=True,
             jk_side=4, nrp=20, npi=40, rmax=60.0),
        # the same survey box end to end: both uploads and the count, from host
        # arrays, as one run of the command line does after reading its files
        dict(BOX, name="box_wgp_200k_from_host", which=1, n_s=200003, L=500.0, clustered=True,
             f32=True, jk_side=4, nrp=20, npi=40, rmax=60.0, upload=True),
        # the 20M-point w++ box's density, clustering and binning at a tenth of
        # the points: the heaviest single count (S and D read the same files)
        dict(BOX, name="box_wpp_2M", which=2, n_s=2000000, L=1000.0, clustered=True, sigma=3.0,
             f32=True, jk_side=5, nrp=25, npi=50, rmax=100.0),
        # w++ of a weighted shape sample against a larger weighted density
        # sample, positions of double precision, 27 cubes, odd sizes
        dict(BOX, name="box_wpp_cross_weighted", which=2, n_s=60001, n_d=151003, L=400.0,
             clustered=True, weights=True, jk_side=3, nrp=15, npi=25, rmin=0.2, rmax=50.0,
             pmax=75.0),
        # a galaxy size or mass field against density (kappa)
        dict(BOX, name="box_kappa_200k", which=3, n_s=200003, L=500.0, clustered=True, f32=True,
             jk_side=4, nrp=20, npi=40, rmax=60.0),
        # 3-D orientation against density in (r, mu)
        dict(BOX, name="box_ed_rmu_200k", which=5, n_s=200003, L=500.0, clustered=True, f32=True,
             jk_side=4, nrp=20, npi=10, rmax=60.0, pmax=1.0),
        # auto pairs of one shape sample (estimators 1 to 3)
        dict(BOX, name="box_auto_100k", kind="auto", which=1, n_s=100003, L=400.0, clustered=True,
             f32=True, jk_side=3, nrp=20, npi=40, rmax=60.0),
        # several uneven sub-boxes in one batch, w++ with 27 cubes each
        dict(BOX, name="box_batch_wpp_12", kind="batch", which=2, n_s=60000, boxes=12, L=200.0,
             jk_side=3, nrp=20, npi=40, rmax=60.0),
        # a small survey: wgg of 5,000 galaxies and 12,000 randoms
        dict(SKY, name="sky_wgg_5k_12k", which=0, n_s=5003, n_r=12007, jk_side=4, nrp=10, npi=20),
        # a survey patch: wg+ with ten times as many randoms, 100 regions
        dict(SKY, name="sky_wgp_20k_200k", n_s=20011, n_r=200017),
    ]


def _pairs(case):
    """Expected binned pairs of a pass (a smooth estimate, for sizes only)."""
    c = case
    if c["kind"] == "sky":
        # RsRd, SRd, DRs, SD: (n_s + n_r)^2 ordered pairs in all, of which the
        # patch (10 x 10 degrees) keeps its window's share
        chi = 0.75 * c["chi_max"] + 0.25 * c["chi_min"]
        f = min(1.0, math.pi * (c["rmax"] / chi) ** 2 / math.radians(10.0) ** 2)
        return (c["n_s"] + c["n_r"]) ** 2 * f * min(1.0, 2.5 * c["pmax"] / (c["chi_max"] - c["chi_min"]))
    depth = 2.0 * c["pmax"] if c["which"] != 5 else 2.0 * c["rmax"]
    f = math.pi * c["rmax"] ** 2 * depth / c["L"] ** 3
    n2 = c["n_d"] or c["n_s"]
    if c["kind"] == "batch":
        # sizes log-uniform on [n/10, n]: mean square 0.215 n^2
        return 0.215 * c["boxes"] * c["n_s"] ** 2 * f
    return c["n_s"] * n2 * f * (0.5 if c["kind"] == "auto" else 1.0)


def _fields(case):
    return {0: 1, 1: 8, 2: 12, 3: 2, 5: 4}[case["which"]]


def draw(rng):
    logu = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    kind = rng.choice(["box", "box", "box", "box", "auto", "batch", "sky", "sky"])
    if kind == "sky":
        c = dict(SKY, which=rng.choice([0, 1, 1, 2]), n_s=int(logu(1500, 20000)),
                 jk_side=rng.choice([3, 5, 10]), nrp=rng.randint(8, 18), npi=rng.randint(10, 34),
                 rmax=rng.choice([40.0, 60.0]))
        c["n_r"] = int(c["n_s"] * logu(2.0, 10.0)) + 1
        cap = 1.5e9
    else:
        which = rng.choice([0, 1, 1, 2, 2, 3, 5]) if kind == "box" else rng.choice([1, 2])
        n = int(logu(2000, 400000))
        L = rng.choice([250.0, 400.0, 500.0, 800.0])
        c = dict(BOX, kind=kind, which=which, n_s=n, L=L, clustered=rng.random() < 0.6,
                 sigma=rng.uniform(1.5, 3.5), f32=rng.random() < 0.6, weights=rng.random() < 0.3,
                 jk_side=rng.choice([0, 2, 3, 4]), nrp=rng.randint(8, 25), npi=rng.randint(10, 50),
                 rmin=rng.choice([0.1, 0.3, 1.0]), rmax=rng.uniform(20.0, 0.2 * L),
                 pmax=rng.choice([60.0, 75.0, 100.0]), lin=rng.random() < 0.2,
                 upload=kind == "box" and rng.random() < 0.25)
        if kind == "box" and which == 2 and rng.random() < 0.5 or kind == "box" and rng.random() < 0.2:
            c["n_d"] = int(n * logu(0.4, 3.0)) + 1
        if which == 5:
            c.update(pmax=1.0, npi=rng.randint(5, 20), rmin=max(c["rmin"], 0.1))
        if kind == "batch":
            c.update(boxes=rng.randint(3, 12), n_s=int(logu(8000, 80000)), clustered=False,
                     upload=False, L=rng.choice([200.0, 250.0]), rmax=rng.uniform(20.0, 60.0))
        cap = 8e9
    while _pairs(c) > cap:
        for k in ("n_s", "n_d", "n_r"):
            if c.get(k):
                c[k] = int(c[k] * 0.8) | 1
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


class _Cat:
    """The arrays that a catalogue upload reads (unset ones are absent)."""

    def __init__(self, **kw):
        for k in ("x", "y", "z", "w", "e1", "e2", "phi", "jk", "jk_prob", "dc", "da", "e3"):
            setattr(self, k, kw.get(k))


class _Table:
    """Flat LCDM distance table on z = k dz (the distances file of a sky run)."""

    def __init__(self, z_max, dz, omega_m=0.3, h0=100.0):
        n = int(math.ceil((z_max + 1.0) / dz)) + 21
        self.z = np.arange(n) * dz
        self.H = h0 * np.sqrt(omega_m * (1.0 + self.z) ** 3 + 1.0 - omega_m)
        inv = C_KMS / self.H
        self.DC = np.concatenate(([0.0], np.cumsum(0.5 * (inv[1:] + inv[:-1]) * dz)))
        self.DA = self.DC / (1.0 + self.z)
        self.transverse = self.DC


def _box_params(c):
    ed = c["which"] == 5
    return synth.InpParams(
        which_corr=c["which"], coordinates=7 if ed else 6, estimator=0, data_sorted=1,
        do_jk=1 if c["jk_side"] else 0, n_jk_regions=c["jk_side"] ** 3, bin_r_min=c["rmin"],
        bin_r_max=c["rmax"], n_bins=c["nrp"], lin_bin=int(c["lin"]), n_p_bin=c["npi"],
        p_min=-c["pmax"], p_max=c["pmax"], z_min=0.0, z_max=c["L"], periodic_box=1,
        periodic_box_size=c["L"])


def _sky_params(c):
    return synth.InpParams(
        which_corr=c["which"], coordinates=0, estimator=0, data_sorted=1, use_comoving=1,
        do_jk=1 if c["jk_side"] else 0, n_jk_regions=c["jk_side"] ** 2, bin_r_min=c["rmin"],
        bin_r_max=c["rmax"], n_bins=c["nrp"], lin_bin=0, n_p_bin=c["npi"], p_min=-c["pmax"],
        p_max=c["pmax"], z_min=0.0, z_max=1.0, dz=0.0001, z_sep_min=0.0, z_sep_max=0.0,
        periodic_box=0, periodic_box_size=0.0)


def _shapes(rng, n):
    r = 0.95 * np.sqrt(-2.0 * 0.25 * np.log1p(-rng.random(n) * (1.0 - math.exp(-2.0))))
    t = rng.uniform(0.0, 2.0 * math.pi, n)
    return r * np.cos(t), r * np.sin(t)


def _points(rng, c, n):
    """n points of the box, sorted by z: uniform, or Neyman-Scott clusters of
    100 with Gaussian offsets, wrapped."""
    L = c["L"]
    if c["clustered"]:
        par = rng.uniform(0.0, L, (max(1, n // 100), 3))
        x = par[rng.integers(0, par.shape[0], n)] + rng.normal(0.0, c["sigma"], (n, 3))
        x = np.mod(x, L)
    else:
        x = rng.uniform(0.0, L, (n, 3))
    if c["f32"]:
        x = x.astype(np.float32).astype(np.float64)
    x[x >= L] = 0.0
    x = x[np.argsort(x[:, 2], kind="stable")]
    return [np.ascontiguousarray(x[:, k]) for k in range(3)]


def _box_sample(rng, c, n):
    x, y, z = _points(rng, c, n)
    k = dict(x=x, y=y, z=z, w=rng.uniform(0.5, 1.5, n) if c["weights"] else np.ones(n))
    if c["jk_side"]:
        s = c["jk_side"]
        i = [np.minimum((v * (s / c["L"])).astype(np.int64), s - 1) for v in (x, y, z)]
        k["jk"] = ((i[0] * s + i[1]) * s + i[2]).astype(np.int32)
    return k


def _box_e(rng, c, n, role):
    """The shape columns that the read path gives the sample in this role."""
    w = c["which"]
    if w in (1, 2) and role == "S" or w == 2:
        e1, e2 = _shapes(rng, n)
        return dict(e1=e1, e2=e2, phi=0.5 * np.arctan2(-e2, e1))
    if w == 3 and role == "S":
        k = rng.normal(0.0, 0.43, n)
        return dict(e1=k - k.mean(), phi=np.full(n, -10.0))
    if w == 5 and role == "S":
        v = rng.normal(size=(3, n))
        v /= np.sqrt((v * v).sum(0))
        return dict(e1=v[0].copy(), e2=v[1].copy(), e3=v[2].copy(), phi=np.full(n, -10.0))
    return dict(phi=np.full(n, -10.0))


def _box_cats(c, seed):
    """(D, S): the density and the shape sample (the same galaxies when the case
    gives no n_d); each has its own jackknife draws, as each read has."""
    rng = np.random.default_rng([20240, int(seed)])
    s = _box_sample(rng, c, c["n_s"])
    es = _box_e(rng, c, c["n_s"], "S")
    if c["n_d"]:
        d = _box_sample(rng, c, c["n_d"])
        ed = _box_e(rng, c, c["n_d"], "D")
    else:
        d = s
        ed = es if c["which"] == 2 else dict(phi=np.full(c["n_s"], -10.0))
    S = _Cat(**s, **es, jk_prob=rng.random(c["n_s"]))
    D = _Cat(**d, **ed, jk_prob=rng.random(c["n_d"] or c["n_s"]))
    return D, S


def _batch_cases(c, seed):
    rng = np.random.default_rng([77, c["boxes"], c["n_s"]])  # the sizes belong to the case
    n = np.exp(rng.uniform(math.log(c["n_s"] / 10.0), math.log(c["n_s"]), c["boxes"]))
    return [(dict(c, kind="box", n_s=int(v)), 1000 * int(seed) + b) for b, v in enumerate(n)]


def _sky_cats(c, seed):
    """Samples S, D (the same galaxies), Rs, Rd (the same randoms) on a 10 x 10
    degree patch, uniform in volume; weights on the data, shapes on S (and on D
    for w++)."""
    rng = np.random.default_rng([555, int(seed)])
    p = _sky_params(c)
    t = _Table(p.z_max, p.dz)
    out = []
    for n in (c["n_s"], c["n_r"]):
        ra = rng.uniform(0.0, 10.0, n)
        de = np.degrees(np.arcsin(rng.uniform(0.0, math.sin(math.radians(10.0)), n)))
        chi = np.cbrt(rng.uniform(c["chi_min"] ** 3, c["chi_max"] ** 3, n))
        z = np.interp(chi, t.DC, t.z)
        o = np.argsort(z, kind="stable")
        ra, de, z = ra[o], de[o], z[o]
        k = np.floor(z / p.dz).astype(np.int64)
        g = c["jk_side"]
        jk = (np.minimum((ra * g / 10.0).astype(np.int64), g - 1) * g
              + np.clip((de * g / 10.0).astype(np.int64), 0, g - 1)).astype(np.int32)
        out.append(dict(x=ra, y=de, z=z, dc=t.DC[k].copy(), da=t.transverse[k].copy(), jk=jk,
                        jk_prob=np.ones(n)))
    data, rand = out
    data["w"] = rng.uniform(0.5, 1.5, c["n_s"])
    rand["w"] = np.ones(c["n_r"])
    none = dict(phi=np.full(c["n_s"], -10.0))
    e = none
    if c["which"]:
        e1, e2 = _shapes(rng, c["n_s"])
        e = dict(e1=e1, e2=e2, phi=0.5 * np.arctan2(-e2, e1))
    S = _Cat(**data, **e)
    D = _Cat(**data, **(e if c["which"] == 2 else none))
    R = _Cat(**rand, phi=np.full(c["n_r"], -10.0))
    return p, t, {"S": S, "D": D, "Rs": R, "Rd": R}


SKY_TERMS = (("SRd", "Rd", "S"), ("RsRd", "Rd", "Rs"), ("SD", "D", "S"), ("DRs", "Rs", "D"))


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    if case["kind"] == "sky":
        p, t, cats = _sky_cats(case, seed)
        st.ctx = _lib.Context(p, table=t)
        slot = {}
        for k, r in enumerate(("S", "D", "Rs", "Rd")):
            st.ctx.upload(k, cats[r])
            slot[r] = k
        st.jobs = [(st.ctx, term, slot[a], slot[b]) for term, a, b in SKY_TERMS]
        return st
    if case["kind"] == "batch":
        st.jobs = []
        for c, s in _batch_cases(case, seed):
            D, S = _box_cats(c, s)
            ctx = _lib.Context(_box_params(c))
            ctx.upload(0, D)
            ctx.upload(1, S)
            st.jobs.append((ctx, "SD", 0, 1))
        return st
    st.cats = _box_cats(case, seed)
    st.ctx = _lib.Context(_box_params(case))
    if not case["upload"]:
        if case["kind"] != "auto":
            st.ctx.upload(0, st.cats[0])
        st.ctx.upload(1, st.cats[1])
        st.cats = None
    return st


def _result(r):
    return {k: r[k] for k in ("num", "sums", "n_window", "n_binned")}


def run(state):
    kind = state.case["kind"]
    if kind in ("sky", "batch"):
        return [_result(r) for r in _lib.count_batch(state.jobs)]
    if kind == "auto":
        return _result(state.ctx.count_auto("SS", 1))
    if state.case["upload"]:
        state.ctx.upload(0, state.cats[0])
        state.ctx.upload(1, state.cats[1])
    return _result(state.ctx.count("SD", 0, 1))


def work(case):
    """Bytes: the catalogue columns (8 doubles and a label per galaxy) read once
    and the histogram blocks (14 words per bin) written once.  Operations: the
    separation, the bin and each accumulated field of every binned pair, the
    rotations for the shape correlations."""
    c = case
    flops_pair = 10 + 2 * _fields(c) + {0: 0, 1: 20, 2: 40, 3: 0, 5: 12}[c["which"]]
    hist = (1 + (c["jk_side"] ** (2 if c["kind"] == "sky" else 3))) * c["nrp"] * c["npi"] * 14 * 8
    if c["kind"] == "sky":
        n, jobs = 2 * (c["n_s"] + c["n_r"]), 4
        flops_pair = 12 if c["which"] == 0 else 16  # nine pairs in ten are counts (RsRd)
    elif c["kind"] == "batch":
        n, jobs = 2 * sum(b["n_s"] for b, _ in _batch_cases(c, 0)), c["boxes"]
    else:
        n, jobs = c["n_s"] + (0 if c["kind"] == "auto" else c["n_d"] or c["n_s"]), 1
    return {"bytes": float(n * 68 + jobs * hist), "flops": float(flops_pair * _pairs(c))}


# ---------------------------------------------------------------------------
# 64-bit restatement (torch)
# ---------------------------------------------------------------------------

_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_CHUNK = 24_000_000


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_DEV)


class _Gal:
    def __init__(self, cat):
        n = len(cat.x)
        zero = np.zeros(n)
        f = lambda v, d: _t(d if v is None else np.asarray(v, dtype=np.float64))  # noqa: E731
        self.n = n
        self.x, self.y, self.z = f(cat.x, zero), f(cat.y, zero), f(cat.z, zero)
        self.w = f(cat.w, np.ones(n))
        self.e1, self.e2, self.e3 = f(cat.e1, zero), f(cat.e2, zero), f(cat.e3, zero)
        self.phi = f(cat.phi, np.full(n, -10.0))
        self.jk = _t(np.zeros(n, np.int64) if cat.jk is None else cat.jk.astype(np.int64))
        self.keep = _t((np.zeros(n) if cat.jk_prob is None else cat.jk_prob) >= 0.5)
        self.idx = torch.arange(n, device=_DEV)
        if cat.dc is not None:
            self.dc, self.da = _t(cat.dc), _t(cat.da)


class _Hist:
    def __init__(self, p, n_hist):
        self.p, self.nh, self.nc = p, n_hist, p.n_bins * p.n_p_bin
        self.num = torch.zeros(n_hist * self.nc, dtype=torch.int64, device=_DEV)
        self.sums = torch.zeros((13, n_hist * self.nc), dtype=torch.float64, device=_DEV)
        self.window = 0

    def bins(self, r, pi):
        p = self.p
        k2 = torch.floor((pi - p.p_min) / ((p.p_max - p.p_min) / p.n_p_bin))
        if p.lin_bin:
            k1 = torch.floor((r - p.bin_r_min) / ((p.bin_r_max - p.bin_r_min) / p.n_bins))
        else:
            size = (math.log10(p.bin_r_max) - math.log10(p.bin_r_min)) / p.n_bins
            k1 = torch.floor(torch.log10(r / p.bin_r_min) / size)
        ok = (k1 >= 0) & (k1 < p.n_bins) & (k2 >= 0) & (k2 < p.n_p_bin)
        return ok, k1, k2

    def add(self, cell, f, regions):
        """f: {field: values}; regions: list of (mask, region) attributions."""
        rep = max(1, 200000 // self.nc)  # copies: fewer additions meet in one place
        wide = cell + self.nc * (torch.arange(cell.numel(), device=_DEV) % rep)
        fold = lambda b: b.reshape(rep, self.nc).sum(0)  # noqa: E731
        self.num[:self.nc] += fold(torch.bincount(wide, minlength=rep * self.nc))
        for q, v in f.items():
            self.sums[q, :self.nc] += fold(torch.bincount(wide, weights=v, minlength=rep * self.nc))
        for m, reg in regions:
            h = (1 + reg[m]) * self.nc + cell[m]
            self.num += torch.bincount(h, minlength=self.nh * self.nc)
            for q, v in f.items():
                if q == 0 or (q % 2 == 1 and self.p.which_corr != 0):
                    self.sums[q] += torch.bincount(h, weights=v[m], minlength=self.nh * self.nc)

    def result(self):
        shape = (self.nh, self.p.n_bins, self.p.n_p_bin)
        return {"num": self.num.reshape(shape).cpu().numpy(),
                "sums": self.sums.t().reshape(shape + (13,)).contiguous().cpu().numpy(),
                "n_window": self.window, "n_binned": int(self.num[:self.nc].sum())}


def _values(corel, gws, g1, i, g2, j, theta, sep):
    wt = g1.w[i] * g2.w[j]
    f = {0: wt}
    if corel == "dd":
        return f
    hold, h = (g2, j) if gws == 2 else (g1, i)
    if corel == "dk":
        f[1] = wt * hold.e1[h]
        return f
    if corel == "ed":
        norm = torch.sqrt(sep[0] * sep[0] + sep[1] * sep[1] + sep[2] * sep[2])
        ca = (hold.e1[h] * sep[0] + hold.e2[h] * sep[1] + hold.e3[h] * sep[2]) / norm
        f[11] = ca * ca
        f[12] = f[11] * f[11]
        return f
    c, s = torch.cos(2.0 * theta), torch.sin(2.0 * theta)
    rot = lambda g, k: (c * g.e1[k] - s * g.e2[k], s * g.e1[k] + c * g.e2[k])  # noqa: E731

    def ephi(phi):
        a = (phi - theta).abs()
        return torch.where(a > math.pi / 2.0, math.pi - a, a)

    if corel == "sd":
        ep, ex = rot(hold, h)
        f[1], f[3], f[11] = wt * ep, wt * ex, ephi(g1.phi[i])
        f[2], f[4], f[12] = f[1] * f[1], f[3] * f[3], f[11] * f[11]
        return f
    a, b = rot(g1, i), rot(g2, j)
    if gws:
        f[1] = wt * (b[0] if gws == 2 else a[0])
        f[11] = ephi(hold.phi[h])
        f[2], f[12] = f[1] * f[1], f[11] * f[11]
    f[5], f[7] = wt * (a[0] * b[0]), wt * (a[1] * b[1])
    f[9] = wt * (a[1] * b[0] + a[0] * b[1]) / 2.0
    f[6], f[8] = f[5] * f[5], f[7] * f[7]
    f[10] = (wt * a[1] * b[0] / 2.0) ** 2 + (wt * a[0] * b[1] / 2.0) ** 2
    return f


def _rule(which, kind, n1, n2):
    """(corel, shape holder, swapped) of a cross count."""
    gws = 2 if kind in ("SD", "SRd") else 0
    if which == 0 or kind == "RsRd":
        corel = "dd"
    elif which == 2 and kind == "SD":
        corel = "ss"
    else:
        corel = {1: "sd", 2: "sd", 3: "dk", 5: "ed"}[which]
    if n2 > n1:
        return corel, {2: 1, 1: 2, 0: 0}[gws], True
    return corel, gws, False


def _box_exact(p, g1, g2, corel, gws, auto=False):
    """Every periodic image of every pair, windowed and binned in 64 bits.  Auto
    counts: row i with rows j > i, and with every row in the +1 z image (input
    sorted by z)."""
    L, rm = p.periodic_box_size, p.bin_r_max
    rmu = p.coordinates == 7
    lo_z, hi_z = (-rm, rm) if rmu else (p.p_min, p.p_max)
    H = _Hist(p, 1 + (p.n_jk_regions if p.do_jk else 0))
    first_m = torch.zeros(g1.n, dtype=torch.bool, device=_DEV)
    first_m[:-1] = g1.z[1:] - L >= g1.z[:-1] + lo_z
    for s in (-1, 0, 1):
        for sy in (-1, 0, 1):
            for sx in (-1, 0, 1):
                rows = torch.ones(g1.n, dtype=torch.bool, device=_DEV)
                cand = torch.ones(g2.n, dtype=torch.bool, device=_DEV)
                for v1, v2, sh, a, b in ((g1.z, g2.z, s, lo_z, hi_z), (g1.x, g2.x, sx, -rm, rm),
                                         (g1.y, g2.y, sy, -rm, rm)):
                    if sh == 1:
                        rows &= v1 + b > L
                        cand &= v2 + L <= L + b
                    elif sh == -1:
                        rows &= v1 + a < 0
                        cand &= v2 - L >= a
                if auto and s == -1:
                    rows &= first_m
                ri, cj = rows.nonzero()[:, 0], cand.nonzero()[:, 0]
                if not ri.numel() or not cj.numel():
                    continue
                z2 = g2.z[cj] + L * s
                z1 = g1.z[ri]
                b0 = 0
                while b0 < ri.numel():  # rows are z-sorted: blocks against a z range
                    b1 = min(ri.numel(), b0 + 256)
                    a = int(torch.searchsorted(z2, z1[b0] + (lo_z - 1e-6)))
                    e = int(torch.searchsorted(z2, z1[b1 - 1] + (hi_z + 1e-6), right=True))
                    if e <= a:
                        b0 = b1
                        continue
                    b1 = min(b1, b0 + max(1, _CHUNK // (e - a)))
                    i0, j0 = ri[b0:b1], cj[a:e]
                    b0 = b1
                    x1, y1, zz1 = g1.x[i0][:, None], g1.y[i0][:, None], g1.z[i0][:, None]
                    x2, y2 = (g2.x[j0] + L * sx)[None], (g2.y[j0] + L * sy)[None]
                    zz2 = z2[a:e][None]
                    m = (zz2 <= zz1 + hi_z) & (zz2 >= zz1 + lo_z)
                    m &= (y2 <= y1 + rm) & (y2 >= y1 - rm) & (x2 <= x1 + rm) & (x2 >= x1 - rm)
                    if auto and s != 1:
                        m &= j0[None] > i0[:, None]
                    k = m.nonzero()
                    del m
                    H.window += k.shape[0]
                    i, j = i0[k[:, 0]], j0[k[:, 1]]
                    del k
                    dx = g1.x[i] - (g2.x[j] + L * sx)
                    dy = g1.y[i] - (g2.y[j] + L * sy)
                    pi = (g2.z[j] + L * s) - g1.z[i]
                    r = torch.sqrt(dx * dx + dy * dy)
                    if rmu:
                        r = torch.sqrt(r * r + pi * pi)
                        ok, k1, k2 = H.bins(r, pi / r)
                    else:
                        ok, k1, k2 = H.bins(r, pi)
                    i, j = i[ok], j[ok]
                    cell = (k1[ok] * p.n_p_bin + k2[ok]).to(torch.int64)
                    theta = torch.atan((g2.y[j] - g1.y[i]) / (g2.x[j] - g1.x[i])) \
                        if corel in ("sd", "ss") else None
                    sep = (dx[ok], dy[ok], g1.z[i] - (g2.z[j] + L * s)) if corel == "ed" else None
                    f = _values(corel, gws, g1, i, g2, j, theta, sep)
                    regs = []
                    if p.do_jk:
                        same = g1.jk[i] == g2.jk[j]
                        regs = [(same | g1.keep[i], g1.jk[i]), (~same & g2.keep[j], g2.jk[j])]
                    H.add(cell, f, regs)
    return H.result()


def _sky_windows(p, t, cat):
    """Per-row redshift, RA and Dec windows from the distance table."""
    r2d = 180.0 / math.pi
    row = lambda v, z: (lambda k: v[k] + (v[k + 1] - v[k]) * (z - p.dz * k) / p.dz)(  # noqa: E731
        np.floor(z / p.dz).astype(np.int64))
    ks = int(math.ceil(p.z_max / p.dz))
    z_sep = p.p_max * t.H[ks] / 300000.0 + 0.001
    z, ra, dec = cat.z, cat.x, cat.y
    z_max = z + p.p_max * row(t.H, z + z_sep) / 300000.0
    z_min = np.maximum(z + p.p_min * row(t.H, z) / 300000.0, 0.001)
    da = p.bin_r_max / row(t.transverse, z_min)
    dr = dec / r2d
    lim = np.arccos((np.cos(da) - np.sin(dr) ** 2) / np.cos(dr) ** 2) * 1.02 * r2d
    ra_max, ra_min = ra + lim, ra - lim
    ra_min = np.where(ra_max > 360, 0.0, ra_min)
    ra_max = np.where(ra_min < 0, 360.0, ra_max)
    return [_t(v) for v in (z_min, z_max, ra_min, ra_max, dec - da * r2d * 1.05,
                            dec + da * r2d * 1.05)]


def _sky_exact(p, t, c1, c2, corel, gws):
    r2d = 180.0 / math.pi
    g1, g2 = _Gal(c1), _Gal(c2)
    win = _sky_windows(p, t, c1)
    for g in (g1, g2):
        g.a, g.d = g.x / r2d, g.y / r2d
        g.sd, g.cd = torch.sin(g.d), torch.cos(g.d)
    H = _Hist(p, 1 + (p.n_jk_regions if p.do_jk else 0))
    lo = torch.searchsorted(g2.z, win[0].contiguous())
    hi = torch.searchsorted(g2.z, win[1].contiguous(), right=True)
    b0 = 0
    while b0 < g1.n:
        b1 = min(g1.n, b0 + 256)
        a, e = int(lo[b0:b1].min()), int(hi[b0:b1].max())
        b1 = min(b1, b0 + max(1, _CHUNK // max(1, e - a)))
        i0 = torch.arange(b0, b1, device=_DEV)
        j0 = torch.arange(a, e, device=_DEV)
        b0 = b1
        if e <= a:
            continue
        w = [v[i0][:, None] for v in win]
        z2, x2, y2 = g2.z[j0][None], g2.x[j0][None], g2.y[j0][None]
        k = (~((z2 < w[0]) | (z2 > w[1]) | (y2 > w[5]) | (y2 < w[4]) | (x2 < w[2]) | (x2 > w[3]))).nonzero()
        H.window += k.shape[0]
        i, j = i0[k[:, 0]], j0[k[:, 1]]
        s = g1.sd[i] * g2.sd[j] + g1.cd[i] * g2.cd[j] * torch.cos(g1.a[i] - g2.a[j])
        th = torch.where(s > 0.9999999999, torch.zeros_like(s), torch.acos(s.clamp(max=1.0)))
        r = th * (g1.da[i] + g2.da[j]) / 2.0
        ok, k1, k2 = H.bins(r, g2.dc[j] - g1.dc[i])
        i, j = i[ok], j[ok]
        cell = (k1[ok] * p.n_p_bin + k2[ok]).to(torch.int64)
        theta = torch.atan((g2.y[j] - g1.y[i]) / ((g2.x[j] - g1.x[i])
                                                  * torch.cos((g1.d[i] + g2.d[j]) / 2.0))) \
            if corel != "dd" else None
        f = _values(corel, gws, g1, i, g2, j, theta, None)
        regs = []
        if p.do_jk:
            same = g1.jk[i] == g2.jk[j]
            regs = [(g1.keep[i], g1.jk[i]), (~same & g2.keep[j], g2.jk[j])]
        H.add(cell, f, regs)
    return H.result()


def exact(case, seed):
    per_pair = 3 if case["kind"] == "sky" else 1 + _fields(case)
    if _pairs(case) * per_pair > 8e9 or (_DEV == "cpu" and _pairs(case) > 2e7):
        return None
    if case["kind"] == "sky":
        p, t, cats = _sky_cats(case, seed)
        out = []
        for term, a, b in SKY_TERMS:
            corel, gws, swap = _rule(case["which"], term, len(cats[a].x), len(cats[b].x))
            c1, c2 = (cats[b], cats[a]) if swap else (cats[a], cats[b])
            out.append(_sky_exact(p, t, c1, c2, corel, gws))
        return out
    if case["kind"] == "batch":
        return [exact(c, s) for c, s in _batch_cases(case, seed)]
    D, S = _box_cats(case, seed)
    p = _box_params(case)
    if case["kind"] == "auto":
        g = _Gal(S)
        return _box_exact(p, g, g, "ss", 1, auto=True)
    corel, gws, swap = _rule(case["which"], "SD", len(D.x), len(S.x))
    a, b = (S, D) if swap else (D, S)
    return _box_exact(p, _Gal(a), _Gal(b), corel, gws)
