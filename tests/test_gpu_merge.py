"""GPU parity of the merge step (ht_merge_halos, ht_finalize_eulerian) with the oracle's
restatement of Merger.merge_catalog / finalize_eulerian: the surviving rows are identical
(same halos, same order, every field), reduced radii agree to one Float32 ulp (the cap
volumes are summed in a different order), velocities to two."""
import math

import numpy as np
import pytest
import torch

from oracle import catalog as oc
from gpu_helpers import to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def finder(ht, julia_table_path):
    tab, axes = ht.read_homeltab(julia_table_path)
    return ht.HaloFinder(6, tab, *axes)


def mk(x, y, z, R, vx=0.0, vy=0.0, vz=0.0, od=0.0):
    return [x, y, z, vx, vy, vz, R, 0.0, 0.0, 0.0, od]


def _ulps(a, b):
    a = np.asarray(a, np.float32).view(np.int32).astype(np.int64)
    b = np.asarray(b, np.float32).view(np.int32).astype(np.int64)
    return np.abs(a - b)


def _merge(ht, finder, rec, **kw):
    out = ht.catalog.merge_halos(finder, to_dev(rec), **kw)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def test_reference_cases(ht, finder):
    """test_merger.jl's small catalogs, through the device."""
    h = np.array([mk(0, 0, 0, 5, od=1), mk(1, 1, 1, 1, od=.5), mk(7, 0, 0, 3, od=.8),
                  mk(50, 50, 50, 2, od=.3)], np.float32)
    assert np.array_equal(_merge(ht, finder, h), oc.merge_catalog(h))
    assert _merge(ht, finder, h).shape[0] == 3
    eq = np.array([mk(0, 0, 0, 2), mk(.5, 0, 0, 2)], np.float32)
    assert np.array_equal(_merge(ht, finder, eq), eq[:1])
    chain = np.array([mk(0, 0, 0, 10)] + [mk(k, 0, 0, 10 - k) for k in range(1, 6)], np.float32)
    assert np.array_equal(_merge(ht, finder, chain), chain[:1])
    pair = np.array([mk(50, 50, 50, 3), mk(54, 50, 50, 2)], np.float32)
    got = _merge(ht, finder, pair, volume_reduction=True)
    assert _ulps(got[:, 6], oc.merge_catalog(pair, volume_reduction=True)[:, 6]).max() <= 1
    ties = np.array([mk(50, 50, 50, 2), mk(53, 50, 50, 2)], np.float32)
    for ft in (False, True):
        got = _merge(ht, finder, ties, volume_reduction=True, fortran_ties=ft)
        assert _ulps(got[:, 6], oc.merge_catalog(ties, True, ft)[:, 6]).max() <= 1
    assert _merge(ht, finder, np.zeros((0, 11), np.float32)).shape[0] == 0
    one = np.array([mk(1, 2, 3, 5, 1.0, 2.0, 3.0, .7)], np.float32)
    assert np.array_equal(_merge(ht, finder, one), one)


def _random_catalog(rng, n, box, width=11):
    # power-law radii: many small halos, a few large ones covering them
    r = np.minimum(0.8 * rng.pareto(2.5, n) + 0.8, 15.0)
    rec = rng.normal(0, 1, (n, width)).astype(np.float32)
    rec[:, :3] = rng.uniform(0, box, (n, 3))
    rec[:, 6] = r
    # a few exact radius ties and coincident x to exercise the tie-breaks
    rec[5:25, 6] = rec[4, 6]
    rec[30:40, 0] = rec[29, 0]
    return rec


@pytest.mark.parametrize("reduce", [False, True])
def test_random_catalog_matches_oracle(ht, finder, reduce):
    rng = np.random.default_rng(21)
    rec = _random_catalog(rng, 30000, 250.0)
    got = _merge(ht, finder, rec, volume_reduction=reduce)
    want = oc.merge_catalog(rec, volume_reduction=reduce)
    assert 5000 < want.shape[0] < 29000
    if not reduce:
        assert np.array_equal(got, want)
    else:
        # the survivors of the exclusion can differ only if a halo's remaining volume sits at
        # exactly zero; compare the rows, radii within one Float32 ulp
        assert got.shape == want.shape
        other = [c for c in range(11) if c != 6]
        assert np.array_equal(got[:, other], want[:, other])
        assert _ulps(got[:, 6], want[:, 6]).max() <= 1
        r0 = {tuple(row[:3]): row[6] for row in rec.tolist()}
        shrunk = sum(1 for row in got.tolist() if row[6] < r0[tuple(row[:3])])
        assert shrunk > 1000                    # the reduction is not a no-op here


def test_extended_records_and_input_order(ht, finder):
    rng = np.random.default_rng(4)
    rec = _random_catalog(rng, 8000, 120.0, width=33)
    got = _merge(ht, finder, rec)
    assert np.array_equal(got, oc.merge_catalog(rec))
    key = lambda m: sorted(map(tuple, m.tolist()))
    for s in range(2):
        perm = np.random.default_rng(s).permutation(len(rec))
        assert key(_merge(ht, finder, rec[perm])) == key(got)


@pytest.mark.parametrize("n,lo,hi,span", [
    (1, 2.0, 2.0, 10.0),          # one halo
    (257, 40.0, 60.0, 100.0),     # every halo wider than 3/4 of a cell (one CTA each)
    (3000, 1e-3, 1e-2, 100.0),    # every radius far below a cell (one thread each)
    (4000, 0.01, 30.0, 60.0),     # both kinds, long kill chains, one cell row and many
    (2500, 1.0, 3.0, 1e-3),       # all centres in one cell
])
@pytest.mark.parametrize("reduce", [False, True])
def test_search_sizes_match_oracle(ht, finder, n, lo, hi, span, reduce):
    rng = np.random.default_rng(n)
    rec = rng.normal(0, 1, (n, 11)).astype(np.float32)
    rec[:, :3] = rng.uniform(-span / 2, span, (n, 3))
    rec[:, 6] = np.exp(rng.uniform(np.log(lo), np.log(hi + 1e-9), n))
    got = _merge(ht, finder, rec, volume_reduction=reduce)
    want = oc.merge_catalog(rec, volume_reduction=reduce)
    if not reduce:
        assert np.array_equal(got, want)
        return
    # the reduced radius is the cube root of r^3 minus sums of cap volumes in another order:
    # FP64 sums of at most n caps, n 2^-53 of r^3, which a radius left with a share s of its
    # volume carries as n 2^-53 / (3 s); s > 1e-6 leaves every radius within one ulp
    assert got.shape == want.shape
    other = [c for c in range(11) if c != 6]
    assert np.array_equal(got[:, other], want[:, other])
    assert _ulps(got[:, 6], want[:, 6]).max(initial=0) <= 1


@pytest.mark.parametrize("n", [2, 3, 5, 9, 127, 128])
def test_chains_of_every_length(ht, finder, n):
    """Chains in which each halo covers the next one and nothing else: one is decided a round,
    n rounds, with the host looking at every round (below 128 halos) and at every fourth."""
    rec = np.zeros((n, 11), np.float32)
    r = 4.0 * 0.999 ** np.arange(n)
    rec[:, 0] = np.r_[0.0, np.cumsum(0.9 * r[:-1])]
    rec[:, 6] = r
    got = _merge(ht, finder, rec)
    assert np.array_equal(got, oc.merge_catalog(rec)) and got.shape[0] == (n + 1) // 2


@pytest.mark.parametrize("reduce", [False, True])
@pytest.mark.parametrize("low", [0.0, -1.0, -100.0])
def test_radii_that_cover_nothing(ht, finder, low, reduce):
    """Zero and negative radii (-1 marks a peak without collapse) among ordinary ones, in the
    corners of the cell grid too: such halos cover and overlap nothing, and a volume reduction
    leaves them no volume.  n 2^-53 / (3 s) bounds the radii as in the test above."""
    rng = np.random.default_rng(17)
    n = 2000
    rec = rng.normal(0, 1, (n, 11)).astype(np.float32)
    rec[:, :3] = rng.uniform(0, 10, (n, 3))
    rec[:8, :3] = [[10.0 * (c >> d & 1) for d in range(3)] for c in range(8)]
    rec[:, 6] = np.where(rng.random(n) < 0.4, low, rng.uniform(0.05, 0.4, n))
    rec[:8, 6] = low
    got = _merge(ht, finder, rec, volume_reduction=reduce)
    want = oc.merge_catalog(rec, volume_reduction=reduce)
    assert got.shape == want.shape and (reduce or (want[:, 6] == low).sum() > 500)
    other = [c for c in range(11) if c != 6]
    assert np.array_equal(got[:, other], want[:, other])
    assert _ulps(got[:, 6], want[:, 6]).max() <= (1 if reduce else 0)


@pytest.mark.parametrize("reduce", [False, True])
def test_nan_radius_leaves_the_others_alone(ht, finder, reduce):
    """A radius that is not a number is refused or, where the largest radius comes out finite,
    covers nothing and changes no other halo."""
    rng = np.random.default_rng(18)
    rec = rng.normal(0, 1, (3000, 11)).astype(np.float32)
    rec[:, :3] = rng.uniform(0, 10, (3000, 3))
    rec[:, 6] = rng.uniform(0.05, 0.4, 3000)
    rec[1234, 6] = np.nan
    try:
        got = _merge(ht, finder, rec, volume_reduction=reduce)
    except ht.HTError:
        return
    got = got[~np.isnan(got[:, 6])]
    want = oc.merge_catalog(np.delete(rec, 1234, 0), volume_reduction=reduce)
    assert got.shape == want.shape
    assert _ulps(got[:, 6], want[:, 6]).max() <= (1 if reduce else 0)


@pytest.mark.parametrize("ievol", [0, 1])
def test_finalize_eulerian_matches_oracle(ht, finder, ievol):
    cat = ht.catalog
    cp = cat.CosmologyParams()
    g = cat.dlinear_tables(cp)
    chi2z = cat.build_chi_to_z(cp, z_max=10.0, npts=400)
    cat.set_cosmology(finder, cp, chi2z, g)
    rng = np.random.default_rng(8 + ievol)
    rec = _random_catalog(rng, 5000, 300.0)
    rec[:, :3] += 1200.0                       # a lightcone shell at z ~ 0.4-0.5
    obs = (0.0, 0.0, 0.0)
    dev = to_dev(rec)
    cat.finalize_eulerian(finder, dev, obs, ievol=ievol, z_out=0.3)
    got = dev.cpu().numpy()
    want = oc.finalize_eulerian(rec, g, cp.Om, cp.OL, obs, chi2z.chis, chi2z.zs, chi2z.z_max,
                                ievol=ievol, z_out=0.3)
    assert np.array_equal(got[:, :3], want[:, :3])
    assert _ulps(got[:, 3:6], want[:, 3:6]).max() <= 2
    assert np.array_equal(got[:, 6:], want[:, 6:])
