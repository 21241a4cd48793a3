"""The box pair kernel against the plain FP64 kernel where its tiles, queues,
histograms and bin maps change form: counts and window pairs identical, sums
within the accuracy bar."""
import numpy as np
import pytest

from corr_pc_gb300 import _lib, host, synth

pytestmark = pytest.mark.gpu


# Tolerance of a bin of n pairs: the kernel adds each pair's term as a multiple of
# 2^-29 of the next power of two above the field's bound (half of it per pair,
# whatever the sum), and a term itself is within 1e-6 of its bin's largest.
def _quanta(S, D):
    w = np.prod([1.0 if c.w is None else np.abs(c.w).max() for c in (S, D)])
    e = max(np.sqrt(sum(v ** 2 for v in (c.e1, c.e2, c.e3) if v is not None)).max()
            if c.e1 is not None else 0.0 for c in (S, D))
    t = max(2 * (10.0 + np.pi), 3 * e * e)
    b = np.array([w] + [w * e, (w * e) ** 2] * 2 + [w * e * e, (w * e * e) ** 2] * 3
                 + [t, max(2 * t * t, 9 * e ** 4)])
    return 2.0 ** np.ceil(np.log2(np.maximum(b, 1e-30) * 1.001)) * 2.0 ** -29


def _same(a, b, S, D, label=""):
    assert (a["n_binned"], a["n_window"]) == (b["n_binned"], b["n_window"]), label
    assert np.array_equal(a["num"], b["num"]), label
    ref = np.nan_to_num(b["sums"])
    tol = 1e-6 * np.abs(ref).max(axis=(0, 1, 2)) + b["num"][..., None] * _quanta(S, D)
    assert (np.abs(np.nan_to_num(a["sums"]) - ref) <= tol).all(), label


def _params(which, n, *, L=60.0, rmin=0.3, rmax=12.0, nrp=7, npi=13, pmax=20.0, side=2, **kw):
    p = synth._box_params(which_corr=which, L=L, rmin=rmin, rmax=rmax, nrp=nrp, npi=npi, pmax=pmax,
                          njk=side ** 3, n=n)
    for k, v in kw.items():
        setattr(p, k, v)
    return p


def _context(p, cats):
    prep = host.prepare(p, cats)
    ctx = _lib.Context(p)
    for k, (name, _) in enumerate(cats):
        ctx.upload(k, prep[name])
    return ctx


def _cat(n, seed, L=60.0, side=2, which=1, weights=False):
    c = synth.uniform_box(n, L, seed, nside_jk=side, with_shapes=which in (1, 2))
    if which in (3, 4):
        c = synth.with_kappa(c, seed + 1)
    if which == 5:
        c = synth.with_orientation(c, seed + 1)
    if weights:
        c.w = np.random.default_rng(seed).uniform(0.5, 1.99, n)
    return c


@pytest.mark.parametrize("n_s,n_d", [(1, 1), (8, 40), (16, 33), (17, 500), (33, 129), (129, 2000),
                                     (2100, 257)])
@pytest.mark.parametrize("which", [0, 1, 2, 3, 5])
def test_row_counts(which, n_s, n_d):
    """Tiles of fewer rows than lanes, whole warps and one row more, g1/g2 swap;
    the boxes differ in every option the kernel is compiled or branched for."""
    S = _cat(n_s, 3 * n_s, which=which, weights=n_s % 2 == 1)
    D = _cat(n_d, n_d, which=which)
    for kw in (dict(), dict(lin_bin=1, bin_r_min=0.0), dict(p_min=-6.0, z_sep_min=-6.0),
               dict(do_jk=0), dict(coordinates=7, p_min=-1.0, p_max=1.0)):
        p = _params(which, n_s, **kw)
        p.n_density = n_d
        ctx = _context(p, [("S", S), ("D", D)])
        _same(ctx.count("SD", 1, 0), ctx.count("SD", 1, 0, engine="fp64"), S, D, str(kw))
        ctx.close()


@pytest.mark.parametrize("window", [0, 5, 8, 21, 40, 64])
@pytest.mark.parametrize("which,twin", [(1, False), (2, False), (2, True), (3, True)])
def test_windows_and_blocks(which, twin, window):
    """Every block size (a wider window takes larger blocks), units repeated over
    windows, both orders of a twin job with exact ties (a lattice)."""
    S = _cat(1500, 11, which=which)
    if twin:
        g = (np.arange(12) + 0.5) * 5.0
        x, y, z = (v.ravel() for v in np.meshgrid(g, g, g, indexing="ij"))
        e1, e2 = synth.shapes(np.random.default_rng(5), x.size)
        S = synth.Catalog(x, y, z, None, e1, e2 if which == 2 else None,
                          synth.jk_cubes(x, y, z, 60.0, 2)).sorted_by_z()
    D = S if twin else _cat(2500, 12, which=which)
    p = _params(which, S.n, npi=64, nrp=9, rmax=15.0, pmax=25.0)
    p.n_density = D.n
    ctx = _context(p, [("S", S), ("D", D)])
    ctx.set_tuning(0, window)
    _same(ctx.count("SD", 1, 0), ctx.count("SD", 1, 0, engine="fp64"), S, D)
    ctx.close()


@pytest.mark.parametrize("corr", [0, 2, 3])
def test_a_bin_past_its_words(corr):
    """A clump over eight jackknife regions whose tiles put more than 2^17 pairs in one
    bin, each term near its bound: the block's histogram is flushed inside a unit;
    and the auto pairs."""
    rng = np.random.default_rng(9)
    n = 3000
    x, y, z = 30.0 + rng.uniform(-0.4, 0.4, (3, n))
    e1, e2 = synth.shapes(rng, n)
    c = synth.Catalog(x, y, z, np.full(n, 1.99), e1 if corr else None, e2 if corr == 2 else None,
                      synth.jk_cubes(x, y, z, 60.0, 2)).sorted_by_z()
    p = _params(corr, n, rmin=0.0, rmax=2.0, nrp=2, npi=1, pmax=2.0, lin_bin=1)
    ctx = _context(p, [("S", c), ("D", c)])
    ref = ctx.count("SD", 1, 0, engine="fp64")
    assert ref["num"].max() > n * n / 2
    for w in (0, 1):
        ctx.set_tuning(0, w)
        _same(ctx.count("SD", 1, 0), ref, c, c)
    ctx.close()
    p.estimator = 1
    ctx = _context(p, [("S", c)])
    _same(ctx.count_auto("SS", 0), ctx.count_auto("SS", 0, engine="fp64"), c, c)
    ctx.close()


def test_cell_width_follows_the_largest_catalogue():
    """The automatic cell width depends on the catalogue's size: a count after a
    larger upload rebuilds the smaller one, and keeps its result."""
    L = 250.0
    cats = [_cat(900, 1, L), _cat(12000, 2, L), _cat(150000, 3, L)]
    p = _params(1, 900, L=L, rmax=20.0, npi=20, pmax=100.0)
    p.n_density = 12000
    prep = host.prepare(p, [("S", cats[0]), ("D", cats[1])])
    ctx = _lib.Context(p)
    ctx.upload(0, prep["S"])
    ctx.upload(1, prep["D"])
    first = ctx.count("SD", 1, 0)
    _same(first, ctx.count("SD", 1, 0, engine="fp64"), cats[0], cats[1])
    p3 = _params(1, 900, L=L, rmax=20.0, npi=20, pmax=100.0)
    p3.n_density = 150000
    ctx.upload(2, host.prepare(p3, [("S", cats[0]), ("D", cats[2])])["D"])
    _same(ctx.count("SD", 2, 0), ctx.count("SD", 2, 0, engine="fp64"), cats[0], cats[2])
    _same(ctx.count("SD", 1, 0), first, cats[0], cats[1])
    ctx.close()
