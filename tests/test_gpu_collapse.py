"""GPU parity of the collapse-table generator (ht_evolve_ellipses, ht_collapse_table) with
the oracle's C restatement of the reference's ellipsoid collapse, both integrators: the
fixed-step RK4 (EllipsoidalCollapse.jl:149-590, solver = :rk4) and the adaptive Tsit5
(:333-485, solver = :diffeq), and of the table sweep (CollapseTable.jl:22-76).

Both sides run the same FP64 operations in the same order (the device file is built
without fused multiply-adds, and the logarithm of the oblate shape branch and the Tsit5
controller's power are series that both carry), so the values agree to the bit."""
import dataclasses
import os
import subprocess
import sys

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
def test_table_order_and_edges(ht, planck, solver, shape):
    """Tables whose entries do not fill the last warp, at the extremes of the axes: the
    spherical limit (e_v = 0), oblate and prolate shapes (p_v / e_v = -1, 1) and the largest
    e_v.  Every entry is the oracle's (the host's sqrt and division round as the operators
    that the device's forms stand for) and sits at its place in the table."""
    cp, g = planck
    col = ht.collapse
    ep = col.EllipsoidParams(cp, dlin_tables=g, solver=solver, nstepmax=3000)
    t = col.make_table(ep, col.CollapseTableParams(Nx=shape[0], Ny=shape[1], Nz=shape[2]))
    eo = oc.EllipsoidOracle(g, cp.Om, cp.OL, solver=solver, nstepmax=3000)
    assert np.array_equal(t, np.transpose(eo.make_table(*shape), (2, 1, 0)))


def _evolve_into(col, ep, args, out):
    """ht_evolve_ellipses on the current stream into out = (z, D, fc, steps)."""
    from huntian_b200 import _lib
    e, gr, keep = ep._structs()
    C = col.C
    _lib.check(_lib.load().ht_evolve_ellipses(
        0, C.byref(e), C.byref(gr), args[0].numel(), *(a.data_ptr() for a in args), 1,
        *(o.data_ptr() for o in out), torch.cuda.current_stream().cuda_stream))
    return keep


@pytest.mark.parametrize("solver", ["rk4", "diffeq"])
def test_captured_and_without_reciprocals(ht, planck, solver):
    """A call under stream capture, and one that does without the reciprocals of the growth
    table's spacings because one is too small for them (here beyond the range that is used):
    both give every bit of the ordinary call's results."""
    cp, g = planck
    col = ht.collapse
    rng = np.random.default_rng(5)
    n = 333
    F = 10.0 ** rng.uniform(np.log10(1.2), np.log10(9.0), n)
    e = rng.uniform(0.0, 0.5, n)
    args = [torch.as_tensor(v, device="cuda") for v in (F, e, rng.uniform(-1, 1, n) * e)]
    ep = col.EllipsoidParams(cp, dlin_tables=g, solver=solver, nstepmax=3000)
    want = col.evolve_ellipses(*args, ep, steps=True)
    assert (want[0] > 0).sum() > n // 2

    out = [torch.zeros_like(w) for w in want]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        keep = _evolve_into(col, ep, args, out)
    graph.replay()
    torch.cuda.synchronize()
    del keep, graph
    for a, b in zip(out, want):
        assert torch.equal(a, b)

    more = lambda t, last: np.r_[t, last]                       # noqa: E731
    g2 = dataclasses.replace(g, atab=more(g.atab, g.atab[-1] + 5e-13),
                             D_atab=more(g.D_atab, g.D_atab[-1]),
                             dlnD_dlnatab=more(g.dlnD_dlnatab, g.dlnD_dlnatab[-1]))
    assert 0 < g2.atab[-1] - g2.atab[-2] < 1e-12 and g.amaxtab <= g.atab[-1]
    got = col.evolve_ellipses(*args, col.EllipsoidParams(cp, dlin_tables=g2, solver=solver,
                                                         nstepmax=3000), steps=True)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


_NO_NEW = """
#include <cstdlib>
#include <new>
static std::size_t limit = 0;
extern "C" void refuse_from(std::size_t n) { limit = n; }
void* operator new(std::size_t n) {
    if (limit && n >= limit) throw std::bad_alloc();
    if (void* p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, std::size_t) noexcept { free(p); }
"""


def _child_without_memory(shim, path):
    import ctypes
    from conftest import load_package
    ht = load_package()
    col = ht.collapse
    refuse = ctypes.CDLL(shim).refuse_from
    refuse.argtypes = [ctypes.c_size_t]
    ep = col.EllipsoidParams(ht.catalog.CosmologyParams(Om=0.315, OL=0.685), solver="rk4")
    args = [torch.tensor(v, dtype=torch.float64, device="cuda")
            for v in ([2.0, 3.0], [0.1, 0.3], [0.0, 0.1])]
    out = [torch.zeros(2, dtype=t, device="cuda") for t in (torch.float64,) * 3 + (torch.int32,)]
    _evolve_into(col, ep, args, out)       # the driver's own first-use allocations
    out[0].zero_()
    refuse(16384)
    _evolve_into(col, ep, args, out)
    refuse(0)
    np.save(path, out[0].cpu().numpy())


def test_host_memory_refused(ht, tmp_path):
    """A host that has no memory left (operator new refuses 16 KB and more while the call runs,
    in a child process) is no reason for ht_evolve_ellipses to end the program."""
    here = os.path.dirname(os.path.abspath(__file__))
    src, so, out = (str(tmp_path / f) for f in ("no.cpp", "no.so", "z.npy"))
    with open(src, "w") as f:
        f.write(_NO_NEW)
    subprocess.run(["g++", "-O1", "-shared", "-fPIC", src, "-o", so], check=True)
    code = (f"import sys; sys.path.insert(0, {here!r}); import conftest; "
            f"import test_gpu_collapse as t; t._child_without_memory({so!r}, {out!r})")
    subprocess.run([sys.executable, "-c", code], check=True, cwd=here, timeout=600,
                   env=dict(os.environ, LD_PRELOAD=so))
    col = ht.collapse
    ep = col.EllipsoidParams(ht.catalog.CosmologyParams(Om=0.315, OL=0.685), solver="rk4")
    want = col.evolve_ellipses([2.0, 3.0], [0.1, 0.3], [0.0, 0.1], ep)[0].cpu().numpy()
    assert np.array_equal(np.load(out), want) and (want > 0).all()
