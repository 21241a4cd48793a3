"""The fast sky kernel against the plain FP64 sky kernel on pairs that it leaves to
double precision: separations too small for single precision, galaxies at one
distance."""
import numpy as np
import pytest

from corr_pc_gb300 import _lib, host, synth
from test_gpu_sky_tiles import _same

pytestmark = pytest.mark.gpu


def _context(p, t, cats):
    ctx = _lib.Context(p, table=t)
    for k, c in enumerate(host.prepare(p, cats, table=t).values()):
        ctx.upload(k, c)
    return ctx


@pytest.mark.parametrize("which", [0, 1, 2])
def test_pairs_of_equal_distance_keep_the_fp64_values(which):
    """Every pair has Pi = 0, an edge of the Pi bins: the values added are those of
    the FP64 engine.  The sums differ by the order of n additions alone, each
    within 2^-53 of the largest partial sum."""
    p = synth._sky_params(which_corr=which, rmin=0.3, rmax=40.0, nrp=12, npi=16, pmax=40.0, njk=9)
    t = synth.flat_lcdm_table(p.z_max, p.dz)
    a = synth.sky_patch(700, 3, t, nside_jk=3, with_shapes=True, weights=True)
    b = synth.sky_patch(1900, 4, t, nside_jk=3, with_shapes=True, weights=True)
    for c in (a, b):
        c.z[:] = 0.25
    ctx = _context(p, t, [("S", a), ("D", b)])
    got, ref = ctx.count("SD", 1, 0), ctx.count("SD", 1, 0, engine="fp64")
    assert np.array_equal(got["num"], ref["num"]) and got["n_window"] == ref["n_window"]
    bound = np.array([2.25, 2.25, 5.1, 2.25, 5.1, 2.25, 2.25, 5.1, 2.25, 5.1, 5.1, 27.0, 400.0])
    n = ref["num"][..., None].astype(float)
    assert (np.abs(got["sums"] - ref["sums"]) <= 2 * n * n * bound * 2.0 ** -53).all()
    ctx.close()


def test_more_undecided_pairs_than_their_queue_holds():
    """1.44 million pairs closer than the separations that single precision can
    bin: past the 2^20 queued ones they are evaluated in the pair kernel."""
    p = synth._sky_params(which_corr=1, rmin=1e-3, rmax=1.0, nrp=9, npi=8, pmax=40.0, njk=4)
    t = synth.flat_lcdm_table(p.z_max, p.dz)
    cats = []
    for role, seed in (("S", 3), ("D", 4)):
        c = synth.sky_patch(1200, seed, t, nside_jk=2, with_shapes=True, weights=True)
        rng = np.random.default_rng(seed)
        c.x[:] = 5.0 + rng.uniform(-2e-3, 2e-3, c.n)
        c.y[:] = 5.0 + rng.uniform(-2e-3, 2e-3, c.n)
        c.z[:] = np.sort(rng.uniform(0.25, 0.252, c.n))
        cats.append((role, c))
    ctx = _context(p, t, cats)
    got, ref = ctx.count("SD", 1, 0), ctx.count("SD", 1, 0, engine="fp64")
    assert ref["n_window"] > 1 << 20
    _same(got, ref, "undecided")
    ctx.close()


def test_nearly_antipodal_pairs():
    """Galaxies so near that r_p bins reach half the sky, where the chord hardly
    changes with the angle: two caps on opposite sides, 64 fine bins below pi D_A."""
    t = synth.flat_lcdm_table(1.0, 0.0001)
    da = float(t.transverse[35])
    p = synth._sky_params(which_corr=1, rmin=(np.pi - 0.005) * da,
                          rmax=(np.pi + 0.0002) * da, nrp=64, npi=5, pmax=1.0, njk=4)
    p.lin_bin = 1
    cats = []
    for role, seed, ra, dec in (("S", 3, 10.0, 60.0), ("D", 4, 190.0, -60.0)):
        c = synth.sky_patch(400, seed, t, nside_jk=2, with_shapes=True, weights=True)
        rng = np.random.default_rng(seed)
        c.x[:] = ra + rng.uniform(-0.15, 0.15, c.n)
        c.y[:] = dec + rng.uniform(-0.08, 0.08, c.n)
        c.z[:] = 0.00355
        cats.append((role, c))
    ctx = _context(p, t, cats)
    got, ref = ctx.count("SD", 1, 0), ctx.count("SD", 1, 0, engine="fp64")
    assert ref["n_binned"] > 100000
    _same(got, ref, "antipodal")
    ctx.close()
