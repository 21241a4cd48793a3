"""Counts whose plan depends on what else a context holds or was told."""
import pytest

from corr_pc_gb300 import _lib, host
from test_gpu_box_tiles import _cat, _params, _same

pytestmark = pytest.mark.gpu

L = 250.0


def _box(which=0, n_s=900, n_d=12000):
    """A small pair of samples, and the density sample of 150,000 rows whose
    presence changes the automatic cell width (r_max to r_max / 2)."""
    s, d, big = _cat(n_s, 1, L, which=which), _cat(n_d, 2, L, which=which), _cat(150000, 3, L)
    out = []
    for c in (d, big):
        p = _params(which, n_s, L=L, rmax=20.0, npi=20, pmax=100.0)
        p.n_density = c.n
        out.append((p, host.prepare(p, [("S", s), ("D", c)])))
    (p, prep), (_, prep_big) = out
    return p, s, d, prep["S"], prep["D"], prep_big["D"]


@pytest.mark.parametrize("when", ["before", "after"])
@pytest.mark.parametrize("which", [0, 1])
def test_shards_on_contexts_of_other_contents_sum_to_the_whole_count(which, when):
    """Each shard on its own context, one of which also holds a larger catalogue
    in a slot that the count does not read."""
    p, s, d, ps, pd, pbig = _box(which)
    parts = []
    for sh in range(3):
        ctx = _lib.Context(p)
        if sh == 1 and when == "before":
            ctx.upload(5, pbig)
        ctx.upload(0, ps)
        ctx.upload(1, pd)
        if sh == 1 and when == "after":
            ctx.upload(5, pbig)
        if sh == 0:
            ref = ctx.count("SD", 1, 0, engine="fp64")
            ctx.count("SD", 1, 0)  # whole, with a plan of its own
        ctx.set_shard(sh, 3)
        parts.append(ctx.count("SD", 1, 0))
        ctx.close()
    total = {k: sum(q[k] for q in parts) for k in ("n_binned", "n_window", "num", "sums")}
    _same(total, ref, s, d)


@pytest.mark.parametrize("k", [1, 2, 3])
@pytest.mark.parametrize("order", ["set first", "set second"])
def test_set_and_automatic_cell_widths_count_together(order, k):
    """A catalogue uploaded with a set cell width against one uploaded with the
    automatic width."""
    p, s, d, ps, pd, _ = _box()
    ctx = _lib.Context(p)
    if order == "set first":
        ctx.set_tuning(k)
        ctx.upload(0, ps)
        ctx.set_tuning(0)
        ctx.upload(1, pd)
    else:
        ctx.upload(0, ps)
        ctx.set_tuning(k)
        ctx.upload(1, pd)
    got = ctx.count("SD", 1, 0)
    _same(got, ctx.count("SD", 1, 0, engine="fp64"), s, d)
    ctx.set_tuning(4)
    ctx.upload(1, pd)
    _same(ctx.count("SD", 1, 0), got, s, d)
    # from here on the three slots share one width: no count rebuilds a list
    ctx.upload(2, pd)
    for _ in range(2):
        n = ctx.launches()
        _same(ctx.count("SD", 1, 0), got, s, d)
        _same(ctx.count("SD", 2, 0), got, s, d)
    assert ctx.launches() - n == 4
    ctx.close()


def test_a_count_after_a_larger_upload_only_counts():
    """The cell lists follow the automatic width at the upload that changes it: a
    count enqueued later runs its own two kernels, no sort."""
    p, s, d, ps, pd, pbig = _box()
    ctx = _lib.Context(p)
    ctx.upload(0, ps)
    ctx.upload(1, pd)
    ref = ctx.count("SD", 1, 0)
    ctx.upload(2, pbig)
    n = ctx.launches()
    ctx.count_async("SD", 1, 0)
    _same(ctx.finish(), ref, s, d)
    assert ctx.launches() - n == 2
    ctx.close()


def test_a_batch_of_pairs_of_one_context():
    """More pair types of one context in a batch than it keeps unit lists of: each
    job has its own block, the first call's and the next one's."""
    p, s, d, ps, pd, _ = _box(1)
    ctx = _lib.Context(p)
    cats = [(0, s, ps), (1, d, pd)]
    for k in range(2, 7):
        c = _cat(400 + 211 * k, 10 + k, L, which=1)
        q = _params(1, 900, L=L, rmax=20.0, npi=20, pmax=100.0)
        q.n_density = c.n
        cats.append((k, c, host.prepare(q, [("S", s), ("D", c)])["D"]))
    for k, _, g in cats:
        ctx.upload(k, g)
    pairs = [(k, 0) for k in range(1, 7)] + [(k, 1) for k in range(2, 7)]
    refs = [ctx.count("SD", a, b, engine="fp64") for a, b in pairs]
    for _ in range(2):
        rs = _lib.count_batch([(ctx, "SD", a, b) for a, b in pairs])
        for (a, b), r, ref in zip(pairs, rs, refs):
            _same(r, ref, cats[a][1], cats[b][1], f"{a},{b}")
    ctx.close()


def test_autotuned_counts_keep_up_with_untuned_ones():
    """Sparse boxes, whose automatic cells of r_max no pair of the autotuners has: the
    pair kernel with what they keep takes at most a fifth longer than without them
    (cells of r_max / 2 take 1.4 times as long)."""
    n = 20000
    c = _cat(n, 4, L, which=0)
    p = _params(0, n, L=L, rmin=0.1, rmax=20.0, nrp=10, npi=20, pmax=100.0)
    prep = host.prepare(p, [("S", c), ("D", c)])
    ctxs = [_lib.Context(p) for _ in range(3)]
    for ctx in ctxs:
        ctx.upload(0, prep["D"])
        ctx.upload(1, prep["S"])

    def ms(ctx):
        return min(ctx.count("SD", 0, 1)["pair_kernel_ms"] for _ in range(20))

    ref, untuned = ctxs[0].count("SD", 0, 1), ms(ctxs[0])
    ctxs[0].autotune("SD", 0, 1, sample_stride=1)
    _lib.autotune_batch([(ctx, "SD", 0, 1) for ctx in ctxs[1:]], sample_stride=1)
    for ctx in ctxs:
        assert ms(ctx) <= 1.2 * untuned
        _same(ctx.count("SD", 0, 1), ref, c, c)
        ctx.close()
