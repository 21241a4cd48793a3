"""The fast sky kernel against the plain FP64 sky kernel at the sizes and options
where its tiles, queues and histograms change form: counts and window pairs
identical, sums within the accuracy bar."""
import numpy as np
import pytest

from corr_pc_gb300 import _lib, host, synth

pytestmark = pytest.mark.gpu


def _run(n_s, n_r, *, which=1, side=3, keep=False, dec0=0.0, nrp=12, npi=16, lin=False,
         weights=True, seed=5):
    p = synth._sky_params(which_corr=which, rmin=0.0 if lin else 0.3, rmax=40.0, nrp=nrp, npi=npi,
                          pmax=40.0, njk=side * side)
    p.lin_bin = int(lin)
    if lin:
        p.bin_r_min = 1.0
    t = synth.flat_lcdm_table(p.z_max, p.dz)
    s = synth.sky_patch(n_s, seed, t, nside_jk=side, with_shapes=True, weights=weights)
    r = synth.sky_patch(n_r, seed + 1, t, nside_jk=side)
    s.y += dec0
    r.y += dec0
    cats = host.prepare(p, [("S", s), ("Rs", r), ("D", s), ("Rd", r)], table=t)
    rng = np.random.default_rng(seed)
    if keep:  # galaxies that leave their region's sample
        for c in cats.values():
            c.jk_prob = rng.random(c.n)
    ctx = _lib.Context(p, table=t)
    for k, name in enumerate(("S", "Rs", "D", "Rd")):
        ctx.upload(k, cats[name])
    return ctx, [("SRd", 3, 0), ("RsRd", 3, 1), ("SD", 2, 0), ("DRs", 1, 2)]


# Tolerance of a bin of n pairs: the kernel adds each pair's term as a multiple of
# 2^-30 of the next power of two above the field's bound (half of it per pair,
# whatever the sum), and a term itself is within 1e-6 of its bin's largest.
def _quanta(wmax, emax):
    w, e, t = wmax * wmax, emax, 10.0 + np.pi
    b = np.array([w] + [w * e, (w * e) ** 2] * 2 + [w * e * e, (w * e * e) ** 2] * 3
                 + [t, 2 * t * t])
    return 2.0 ** np.ceil(np.log2(b * 1.001)) * 2.0 ** -30


def _same(a, b, label):
    assert (a["n_binned"], a["n_window"]) == (b["n_binned"], b["n_window"]), label
    assert np.array_equal(a["num"], b["num"]), label
    _close(a["sums"], b["sums"], b["num"], label)


def _close(got, ref, num, label):
    tol = 1e-6 * np.abs(ref).max(axis=(0, 1, 2)) + num[..., None] * _quanta(1.5, 1.0)
    assert (np.abs(got - ref) <= tol).all(), label


@pytest.mark.parametrize("case", [
    dict(n_s=1, n_r=1), dict(n_s=7, n_r=31), dict(n_s=33, n_r=97), dict(n_s=129, n_r=2000),
    dict(n_s=900, n_r=1500, keep=True), dict(n_s=900, n_r=4001, which=2, keep=True),
    dict(n_s=800, n_r=3000, side=0), dict(n_s=800, n_r=3000, side=20),
    # the acos of the RA window leaves its range near the pole
    dict(n_s=800, n_r=3000, dec0=79.9), dict(n_s=800, n_r=3000, lin=True, which=0),
    # histograms too large for shared memory
    dict(n_s=700, n_r=2500, nrp=50, npi=120), dict(n_s=1500, n_r=1500, which=0, weights=False),
], ids=str)
def test_sky_terms_match_fp64_engine(case):
    ctx, terms = _run(**case)
    batch = _lib.count_batch([(ctx, *t) for t in terms])
    for t, b in zip(terms, batch):
        ref = ctx.count(*t, engine="fp64")
        _same(b, ref, t[0])
        _same(ctx.count(*t), ref, t[0])
    ctx.close()


def test_sky_rows_shards_and_auto_match_fp64_engine():
    ctx, terms = _run(1200, 2600, keep=True)
    ref = ctx.count(*terms[0], engine="fp64")
    for parts in ([ctx.count(*terms[0], row_stride=5, row_offset=o) for o in range(5)],):
        assert np.array_equal(sum(q["num"] for q in parts), ref["num"])
        _close(sum(q["sums"] for q in parts), ref["sums"], ref["num"], "rows")
    parts = []
    for s in range(3):
        ctx.set_shard(s, 3)
        parts.append(ctx.count(*terms[0]))
    ctx.set_shard(0, 1)
    assert sum(q["n_window"] for q in parts) == ref["n_window"]
    assert np.array_equal(sum(q["num"] for q in parts), ref["num"])
    _same(ctx.count_auto("SS", 0), ctx.count_auto("SS", 0, engine="fp64"), "SS")
    ctx.close()


@pytest.mark.parametrize("which", [1, 2])
def test_sky_terms_in_several_launches_match_fp64_engine(which):
    """Enough region pairs for a launch per group of corels, beside one another."""
    ctx, terms = _run(5000, 20000, which=which, side=10, nrp=2, npi=2)
    l0 = ctx.launches()
    batch = _lib.count_batch([(ctx, *t) for t in terms])
    assert ctx.launches() - l0 > 1 + len(terms)  # the sums' launches, and more than one
    for t, b in zip(terms, batch):
        _same(b, ctx.count(*t, engine="fp64"), t[0])
    ctx.close()
