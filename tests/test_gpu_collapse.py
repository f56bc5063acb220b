"""GPU parity of the collapse-table generator (ht_evolve_ellipses, ht_collapse_table) with
the oracle's C restatement of the reference's ellipsoid collapse, both integrators: the
fixed-step RK4 (EllipsoidalCollapse.jl:149-590, solver = :rk4) and the adaptive Tsit5
(:333-485, solver = :diffeq), and of the table sweep (CollapseTable.jl:22-76).

Both sides run the same FP64 operations in the same order (the device file is built
without fused multiply-adds, and the logarithm of the oblate shape branch and the Tsit5
controller's power are series that both carry), so the values agree to the bit."""
import numpy as np
import pytest
import torch

from oracle import collapse as oc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def planck(ht):
    cat = ht.catalog
    cp = cat.CosmologyParams(Om=0.315, OB=0.049, OL=0.685, h=0.674, ns=0.965, s8=0.808)
    return cp, cat.dlinear_tables(cp)


def _compare(got, want, max_flip=0, step_rel=5e-3, exact_frac=0.99):
    got, want = np.asarray(got, np.float64), np.asarray(want, np.float64)
    flip = (got <= 0) != (want <= 0)
    assert flip.sum() <= max_flip
    ok = (got > 0) & (want > 0)
    if not ok.any():                  # nothing collapses (e.g. iforce_strat 6): all -1
        assert np.array_equal(got, want)
        return
    assert np.mean(got[ok] == want[ok]) >= exact_frac
    rel = np.abs(got[ok] - want[ok]) / want[ok]
    assert rel.max() <= step_rel


def test_default_table_matches_oracle(ht, planck):
    cp, g = planck
    col = ht.collapse
    got = col.make_table(col.EllipsoidParams(cp, dlin_tables=g, solver="rk4"))  # (nz, ny, nx)
    want = np.transpose(oc.EllipsoidOracle(g, cp.Om, cp.OL).make_table(), (2, 1, 0))
    assert got.shape == want.shape == (20, 20, 50) and got.dtype == np.float32
    _compare(got, want)
    assert (got == -1.0).sum() > 2000 and (got > 0).sum() > 16000


def test_evolve_matches_oracle_every_event(ht, planck):
    cp, g = planck
    col = ht.collapse
    rng = np.random.default_rng(3)
    n = 600
    F = 10.0 ** rng.uniform(np.log10(1.2), np.log10(9.0), n)
    e = rng.uniform(0.0, 0.5, n)
    p = rng.uniform(-1.0, 1.0, n) * e
    F[:3], e[:3], p[:3] = (1.686, 5.0, 0.5), (0.0, 0.0, 0.0), (0.0, 0.0, 0.0)
    ep = col.EllipsoidParams(cp, dlin_tables=g, solver="rk4")
    eo = oc.EllipsoidOracle(g, cp.Om, cp.OL)
    for idynax in (1, 2, 3, 4, 5, 6):
        z, D, fc, st = (t.cpu().numpy() for t in
                        col.evolve_ellipses(F, e, p, ep, idynax=idynax, steps=True))
        want = np.array([eo.evolve(F[q], e[q], p[q], idynax) for q in range(n)])
        _compare(z, want[:, 0])
        _compare(D, want[:, 1])
        _compare(fc, want[:, 2])
        assert np.mean(st == want[:, 3]) >= 0.99
    assert col.evolve_ellipse_full(0.5, 0.0, 0.0, ep) == (-1.0, -1.0, -1.0)


@pytest.mark.parametrize("fs,vs", [(0, 2), (1, 2), (3, 2), (4, 1), (5, 2), (6, 2)])
def test_other_strategies_match_oracle(ht, planck, fs, vs):
    cp, g = planck
    col = ht.collapse
    rng = np.random.default_rng(10 + fs)
    n = 200
    F = 10.0 ** rng.uniform(np.log10(1.5), np.log10(8.0), n)
    e = rng.uniform(0.0, 0.5, n)
    p = rng.uniform(-1.0, 1.0, n) * e
    for solver in ("rk4", "diffeq"):
        ep = col.EllipsoidParams(cp, iforce_strat=fs, ivir_strat=vs, nstepmax=4000,
                                 dlin_tables=g, solver=solver)
        eo = oc.EllipsoidOracle(g, cp.Om, cp.OL, iforce_strat=fs, ivir_strat=vs,
                                nstepmax=4000, solver=solver)
        z = col.evolve_ellipses(F, e, p, ep)[0].cpu().numpy()
        want = np.array([eo.evolve(F[q], e[q], p[q])[0] for q in range(n)])
        _compare(z, want)


def test_invalid_parameters(ht, planck):
    cp, g = planck
    col = ht.collapse
    for kw in (dict(nstepmax=0), dict(ivir_strat=3), dict(iforce_strat=7), dict(tfac=0.0)):
        ep = col.EllipsoidParams(cp, dlin_tables=g, **kw)
        with pytest.raises(ht.HTError):
            col.evolve_ellipses([2.0], [0.1], [0.0], ep)
    ep = col.EllipsoidParams(cp, dlin_tables=g)
    with pytest.raises(ht.HTError):
        col.evolve_ellipses([2.0], [0.1], [0.0], ep, idynax=7)
    with pytest.raises(ht.HTError):   # the :diffeq path keeps no turnaround events
        col.evolve_ellipses([2.0], [0.1], [0.0], ep, idynax=4)
    z, D, fc = col.evolve_ellipses(np.zeros(0), np.zeros(0), np.zeros(0), ep)
    assert z.numel() == 0
    with pytest.raises(ht.HTError):
        col.make_table(ep, col.CollapseTableParams(Nx=1))


def test_generated_table_drives_the_finder(ht, planck, tmp_path):
    """A table made on the device, written as a HomelTab file and read back, gives the
    collapse criterion the same fcrit as the oracle's table (fsc_of_z at z = 0)."""
    cp, g = planck
    col = ht.collapse
    path = str(tmp_path / "HomelTab.dat")
    t = col.generate_table(path, Om=cp.Om, OB=cp.OB, OL=cp.OL, h=cp.h, solver="rk4")
    tab, axes = ht.read_homeltab(path)
    assert np.array_equal(tab, t)
    f = ht.HaloFinder(4, tab, *axes)
    want = np.transpose(oc.EllipsoidOracle(g, cp.Om, cp.OL).make_table(), (2, 1, 0))
    f2 = ht.HaloFinder(4, np.ascontiguousarray(want), *axes)
    assert f.fsc_of_z(0.0) == pytest.approx(f2.fsc_of_z(0.0), rel=1e-6)
    assert 1.6 < f.fsc_of_z(0.0) < 1.8


def test_tsit5_table_and_events_match_oracle(ht, planck):
    """The :diffeq path (adaptive Tsit5) on the device against the oracle's: the default
    table (the reference's default solver) and events 1-3 of random ellipsoids, with the
    iterations taken."""
    cp, g = planck
    col = ht.collapse
    got = col.make_table(col.EllipsoidParams(cp, dlin_tables=g))     # solver = "diffeq"
    want = np.transpose(oc.EllipsoidOracle(g, cp.Om, cp.OL, solver="diffeq").make_table(),
                        (2, 1, 0))
    print(f"\nTsit5 table: {np.mean(got == want):.4f} of the entries bit-identical")
    _compare(got, want, step_rel=0.2)
    assert (got > 0).sum() > 16900
    rng = np.random.default_rng(4)
    n = 400
    F = 10.0 ** rng.uniform(np.log10(1.2), np.log10(9.0), n)
    e = rng.uniform(0.0, 0.5, n)
    p = rng.uniform(-1.0, 1.0, n) * e
    F[:2], e[:2], p[:2] = (1.686, 0.5), (0.0, 0.0), (0.0, 0.0)
    ep = col.EllipsoidParams(cp, dlin_tables=g)
    eo = oc.EllipsoidOracle(g, cp.Om, cp.OL, solver="diffeq")
    for idynax in (1, 2, 3):
        z, D, fc, st = (t.cpu().numpy() for t in
                        col.evolve_ellipses(F, e, p, ep, idynax=idynax, steps=True))
        want = np.array([eo.evolve(F[q], e[q], p[q], idynax) for q in range(n)])
        _compare(z, want[:, 0], step_rel=0.2)
        _compare(D, want[:, 1], step_rel=0.2)
        assert np.mean(st == want[:, 3]) >= 0.99
    assert col.evolve_ellipse_full(0.5, 0.0, 0.0, ep) == (-1.0, -1.0, -1.0)


@pytest.mark.parametrize("solver", ["rk4", "diffeq"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (33, 2, 3), (5, 31, 2)])
def test_table_order_and_edges(ht, oracle, solver, shape):
    """Tables whose entries do not fill the last warp, at the extremes of the axes: shapes near
    the spherical limit (e_v = 0), oblate and prolate ones (p_v / e_v = -1, 1) and radii past
    the division-free form of the shape integrals' test.  Every entry equals the scalar call."""
    col = ht.collapse
    ep = col.EllipsoidParams(ht.catalog.CosmologyParams(Om=0.3, OL=0.7), solver=solver,
                             nstepmax=3000)
    tp = col.CollapseTableParams(Nx=shape[0], Ny=shape[1], Nz=shape[2])
    t = col.make_table(ep, tp)
    x1, x2, y1, y2, z1, z2 = tp.axes
    X = x1 + np.arange(tp.Nx) * ((x2 - x1) / (tp.Nx - 1))
    Y = y1 + np.arange(tp.Ny) * ((y2 - y1) / (tp.Ny - 1))
    Z = z1 + np.arange(tp.Nz) * ((z2 - z1) / (tp.Nz - 1))
    import math
    F = np.array([math.pow(10.0, x) for x in X])
    k, j, i = np.meshgrid(np.arange(tp.Nz), np.arange(tp.Ny), np.arange(tp.Nx), indexing="ij")
    z, _, _ = col.evolve_ellipses(F[i.ravel()], Y[j.ravel()], (Z[k] * Y[j]).ravel(), ep)
    assert np.array_equal(t.ravel(), z.cpu().numpy().astype(np.float32))
