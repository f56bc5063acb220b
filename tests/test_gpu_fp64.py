"""The straight-line quotient, reciprocal, root and Carlson RD of ht_fp64.cuh against the
operators / and sqrt on the same device, bit for bit, over the ranges their callers admit.
RD is compared with the plain recurrence in torch, whose operations are separate kernels (no
product is fused into a sum)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT, load_package

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
RECIP, ROOT_OP, QUOT, RATIO, QUOT_ANY = range(5)
ONES = (1 << 52) - 1        # a significand of all ones


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    load_package()
    so = str(tmp_path_factory.mktemp("fp64") / "fp64_check.so")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-fmad=false", "-Xcompiler", "-fPIC", "-shared", "-cudart", "shared", "-I",
                    os.path.join(ROOT, "huntian.jl_b200", "csrc"),
                    os.path.join(HERE, "fp64_check.cu"), "-o", so], check=True)
    L = C.CDLL(so)
    L.fp64_op.argtypes = [C.c_int, C.c_longlong] + [C.c_void_p] * 3
    L.fp64_rd.argtypes = [C.c_longlong] + [C.c_void_p] * 4
    return L


def _op(lib, op, a, b):
    out = torch.empty_like(a)
    torch.cuda.synchronize()
    assert lib.fp64_op(op, a.numel(), a.data_ptr(), b.data_ptr(), out.data_ptr()) == 0
    torch.cuda.synchronize()
    return out


def _bits(t):
    return t.view(torch.int64)


def _same(got, want):
    return bool((_bits(got) == _bits(want)).all())


def _values(seed, n, lo, hi):
    """n positive doubles with exponents lo..hi - 1: random significands, significands within
    64 units of 1, 2 (all ones left out), 1.5 and sqrt 2, and few-bit ones."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    r = lambda a, b, m: torch.randint(a, b, (m,), generator=g, device="cuda")   # noqa: E731
    m = n // 8
    near = torch.tensor([0, ONES - 64, 1 << 51, int((2 ** 0.5 - 1) * 2 ** 52)], device="cuda")
    sig = torch.cat([r(0, ONES, n - 3 * m), near[r(0, 4, m)] + r(0, 64, m),
                     ONES - 1 - r(0, 64, m), (1 << r(0, 52, m)) | (1 << r(0, 52, m))])
    sig = sig[torch.randperm(n, generator=g, device="cuda")]
    return (sig | (r(lo, hi, n) + 1023 << 52)).view(torch.float64)


N = 1 << 23
E60 = 199                   # 2^199 < 1e60 < 2^200


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("lo,hi", [(-E60, E60), (-2, 2), (-60, 60)])
def test_quotients_and_roots_are_the_operators(lib, lo, hi, seed):
    a, b = _values(100 + seed, N, lo, hi), _values(200 + seed, N, lo, hi)
    assert _same(_op(lib, RECIP, a, b), 1.0 / b)
    assert _same(_op(lib, ROOT_OP, a, b), torch.sqrt(a))
    assert _same(_op(lib, QUOT, a, b), a / b)
    assert _same(_op(lib, QUOT, a * b, b), (a * b) / b)       # near whole quotients
    assert _same(_op(lib, RATIO, a, b), a / b)
    assert _same(_op(lib, QUOT_ANY, -a, b), -a / b)


def test_roots_next_to_ties(lib):
    """Squares, the doubles around them, and the doubles nearest to the squares of midpoints
    between two doubles: x = (m + 1/2)^2 for 53-bit m, in integer arithmetic."""
    rng = np.random.default_rng(5)
    m = [int(v) for v in rng.integers(1 << 52, 1 << 53, 100000)]
    m += [(1 << 52) + k for k in range(200)] + [(1 << 53) - 1 - k for k in range(200)]
    xs = []
    for v in m:
        for sq, sh in ((v * v, 0), ((2 * v + 1) ** 2, 2)):    # root v, v + 1/2
            for e in (0, 1):                                  # both parities of the exponent
                f = float(sq << e)                            # rounded to nearest
                xs += [f * 2.0 ** (-105 - sh)]
    x = torch.tensor(xs, dtype=torch.float64, device="cuda")
    x = torch.cat([x, torch.nextafter(x, 2 * x), torch.nextafter(x, 0 * x)])
    for scale in (1.0, 2.0 ** 180, 2.0 ** -180):
        assert _same(_op(lib, ROOT_OP, x * scale, x), torch.sqrt(x * scale))


def test_outside_the_range_and_all_ones(lib):
    """ratio and quot_any divide where the straight-line form does not hold; a significand of
    all ones is the one divisor that may come out a unit low."""
    v = [0.0, -0.0, 5e-324, 1e-310, 1e-300, 1e-250, 1e-61, 1e-60, 1e-30, 1.0, 1e30, 1e60, 1e61,
         1e250, 1.7e308, float("inf"), float("nan")]
    v += [-q for q in v]
    a, b = (t.reshape(-1).contiguous() for t in
            torch.meshgrid(*(torch.tensor(v, dtype=torch.float64, device="cuda"),) * 2,
                           indexing="ij"))
    for op in (RATIO, QUOT_ANY):
        got, want = _op(lib, op, a, b), a / b
        nan = torch.isnan(want)
        assert torch.equal(nan, torch.isnan(got)) and _same(got[~nan], want[~nan])
    e = torch.arange(-E60, E60, device="cuda")
    b = (ONES | (e + 1023 << 52)).view(torch.float64)
    for op, a, want in ((RECIP, b, 1.0 / b), (QUOT, torch.ones_like(b), 1.0 / b)):
        d = _bits(want) - _bits(_op(lib, op, a, b))
        assert int(d.min()) >= 0 and int(d.max()) <= 1
    a = _values(9, b.numel(), -60, 60)
    a = torch.where(_bits(a) << 12 == 0, 1.5 * a, a)         # no powers of two
    assert _same(_op(lib, QUOT, a, b), a / b)


def _rd(x, y, z):
    """EllipsoidalCollapse.jl:62-106 in plain float64 operations, 200 rounds at most."""
    c1, c2, c3, c4 = 3.0 / 14.0, 1.0 / 6.0, 9.0 / 22.0, 3.0 / 26.0
    c5, c6 = 0.25 * c3, 1.5 * c4
    s, fac = torch.zeros_like(x), torch.ones_like(x)
    ave = torch.zeros_like(x)
    done = torch.zeros_like(x, dtype=torch.bool)
    for _ in range(200):
        sx, sy, sz = torch.sqrt(x), torch.sqrt(y), torch.sqrt(z)
        lam = sx * (sy + sz) + sy * sz
        keep = lambda old, new: torch.where(done, old, new)      # noqa: B023, E731
        s = keep(s, s + fac / (sz * (z + lam)))
        fac = keep(fac, fac * 0.25)
        x, y, z = (keep(v, 0.25 * (v + lam)) for v in (x, y, z))
        ave = keep(ave, 0.2 * (x + y + 3.0 * z))
        d = [(ave - v) / ave for v in (x, y, z)]
        done |= torch.stack([q.abs() for q in d]).amax(0) <= 0.05
        if bool(done.all()):
            break
    dx, dy, dz = d
    ea, eb = dx * dy, dz * dz
    ec, ed = ea - eb, ea - 6.0 * eb
    ee = ed + ec + ec
    series = 1.0 + ed * (-c1 + c5 * ed - c6 * dz * ee) + dz * (c2 * ee + dz * (-c3 * ec + dz * c4 * ea))
    return 3.0 * s + fac * series / (ave * torch.sqrt(ave))


def test_rd_matches_the_plain_recurrence(lib):
    """Both forms (arguments inside and outside 1e-12 .. 1e12) and pairs of which one set ends
    rounds before the other; arguments chosen so that first averages lie on the stopping line."""
    rng = np.random.default_rng(6)
    n = 200000
    v = [10.0 ** rng.uniform(-3, 3, (3, n)), 10.0 ** rng.uniform(-11.9, 11.9, (3, n)),
         10.0 ** rng.uniform(-20, 20, (3, n)), 1.0 + rng.uniform(-0.3, 0.3, (3, n))]
    line = np.ones((3, n))                       # (ave - z) / ave near 0.05 after one round
    line[0] = line[1] = 1.0 + rng.uniform(0.4, 0.9, n)
    v = np.concatenate(v + [line], 1)[:, rng.permutation(5 * n)]
    x, y, z = (torch.as_tensor(np.ascontiguousarray(q), device="cuda") for q in v)
    out = torch.empty(2 * x.numel(), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert lib.fp64_rd(x.numel(), x.data_ptr(), y.data_ptr(), z.data_ptr(), out.data_ptr()) == 0
    torch.cuda.synchronize()
    want = _rd(x, y, z)
    assert bool(torch.isfinite(want).all())
    assert _same(out[:x.numel()], want) and _same(out[x.numel():], want)
