"""The work that programs have this framework do, as cases that can be timed and compared.

A halo-finding run takes every tile of its box through the same stage: the tile's density is
Fourier transformed once, smoothed with each filter of a bank and scanned for local maxima
(find, tile), the peaks are carried through the radial-shell collapse (walk), the collapsed
ones become halo records and are merged (halos).  Besides that it makes a collapse table once
per cosmology (table) and, offline, trains the network that orders the shell walk (train).
Fields are seeded Gaussian random fields with a BBKS spectrum and their 2LPT displacements,
as the benchmark's; sizes are those of the benchmark's and the tests' workloads.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DEV = torch.device("cuda", 0)
FCRIT = 1.686
FIELDS = ("delta", "etax", "etay", "etaz", "eta2x", "eta2y", "eta2z")


def _package():
    """The package directory huntian.jl_b200/, imported as huntian_b200."""
    name = "huntian_b200"
    if name not in sys.modules:
        pkg = os.path.join(ROOT, "huntian.jl_b200")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


ht = _package()
from huntian_b200 import synth  # noqa: E402

COSMO = synth.Cosmology()


def listed():
    return [
        # a small tile through the reference's peak-finding call, host arrays in and out, with
        # the Laplacian: the smallest call a program makes (sizes of the mirror tests)
        dict(name="tile_64", kind="tile", n=64, nbuff=8, nf=3, shear=1, host=True),
        # the 128^3 box with its 36-cell buffer through the same call, device arrays
        dict(name="tile_200", kind="tile", n=200, nbuff=36, nf=12, shear=0, host=False),
        # per-filter smoothing and scan of the 512^3 box's tile (a side with a factor of 31)
        dict(name="find_620", kind="find", n=620, nbuff=54, nf=6),
        # the same for the large tile, 1024^3 core and 64-cell buffer: the benchmark's loop
        # over its largest, smallest and two middle filters
        dict(name="find_1152", kind="find", n=1152, nbuff=64, nf=4),
        # shell collapse of a handful of peaks (one re-analysed region): latency
        dict(name="walk_few", kind="walk", box=60, nbuff=18, alatt=1.953125, nf=8, most=200,
             mode="batched", conv="gpu", lapd=False),
        # the 128^3 box, 30 filters, with the Laplacian field (extended output)
        dict(name="walk_200", kind="walk", box=128, nbuff=36, alatt=1.953125, nf=30, most=40000,
             mode="batched", conv="gpu", lapd=True),
        # the large tile's geometry (cell, 63-cell hunt radius, 80 filters) on a 192^3 core
        dict(name="walk_320", kind="walk", box=192, nbuff=64, alatt=1.46484375, nf=80,
             most=140000, mode="learned", conv="gpu", lapd=False),
        # the 512^3 box with 40 of its filters: the ordinary production tile
        dict(name="walk_620", kind="walk", box=512, nbuff=54, alatt=1.953125, nf=40,
             most=2200000, mode="learned", conv="gpu", lapd=False),
        # catalogue of a 512^3 tile: records of the collapsed peaks, then the exclusion
        dict(name="halos_2m", kind="halos", npk=2_800_000, box=512, shear=0, reduce=False),
        # the default collapse table by both integrators
        dict(name="table_rk4", kind="table", solver="rk4", nx=50, ny=20, nz=20),
        dict(name="table_diffeq", kind="table", solver="diffeq", nx=50, ny=20, nz=20),
        # one optimiser step of the walk-order network on a full training batch
        dict(name="train_65536", kind="train", batch=65536),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("tile", "find", "find", "walk", "walk", "walk", "halos", "table",
                       "train"))
    if kind == "tile":
        n = _log(rng, 48, 200)
        return dict(kind=kind, n=n, nbuff=rng.randint(4, n // 5), nf=rng.randint(2, 12),
                    shear=rng.randint(0, 1), host=rng.random() < 0.5)
    if kind == "find":
        n = rng.choice((576, 1152, 2 * _log(rng, 100, 400), 2 * _log(rng, 100, 400)))
        return dict(kind=kind, n=n, nbuff=rng.randint(8, min(64, n // 6)),
                    nf=rng.randint(2, 4 if n > 800 else 8))
    if kind == "walk":
        box = _log(rng, 40, 320)
        return dict(kind=kind, box=box, nbuff=min(rng.randint(14, 64), box // 2),
                    alatt=rng.uniform(1.4, 2.0), nf=rng.randint(4, 40),
                    most=_log(rng, 50, box ** 3 * 0.015),
                    mode=rng.choice(("batched", "learned", "learned", "plain")),
                    conv=rng.choice(("gpu", "gpu", "cpu")), lapd=rng.random() < 0.3)
    if kind == "halos":
        npk = _log(rng, 2000, 2_800_000)
        return dict(kind=kind, npk=npk, box=max(24, int((npk / 0.021) ** (1 / 3))),
                    shear=rng.randint(0, 1), reduce=False)
    if kind == "table":
        return dict(kind=kind, solver=rng.choice(("rk4", "diffeq")), nx=rng.randint(10, 50),
                    ny=rng.randint(5, 20), nz=rng.randint(5, 20))
    return dict(kind=kind, batch=_log(rng, 500, 65536))


# ------------------------------------------------------------------------- inputs ----

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _collapse_table():
    return ht.read_homeltab(os.path.join(ROOT, "tests", "golden", "HomelTab_julia.dat"))


def _alatt(case):
    """Cell size in Mpc/h: the box128 / box512 spacing, the large tile's from 1152 on."""
    return case.get("alatt", 1.46484375 if case["n"] > 1000 else 1.953125)


def _filters(nf, alatt, nbuff):
    """nf log-spaced radii, the largest within the buffer's hunt radius, as the drivers'."""
    rmin = 1.5 if alatt < 1.7 else 2.0
    return ht.log_filterbank(nf, rmin, max(1.2 * rmin, min(80.0, (nbuff - 1) * alatt / 1.75)))


def _window(q, n, alatt, Rf):
    """Top-hat window of integer |k|^2 = q on an n^3 grid, in the type of q."""
    x = torch.sqrt(q) * (2.0 * math.pi / (n * alatt) * Rf)
    w = 3.0 * (torch.sin(x) - x * torch.cos(x)) / x ** 3
    return torch.where(q == 0, torch.ones_like(w), w)


def _q(n, z0, z1):
    """|k|^2 of planes z0..z1 of the rfft grid as float64 integers."""
    f = torch.fft.fftfreq(n, d=1.0 / n, device=DEV, dtype=torch.float64)
    x = torch.arange(n // 2 + 1, device=DEV, dtype=torch.float64)
    return (f[z0:z1] ** 2).view(-1, 1, 1) + (f ** 2).view(1, -1, 1) + (x ** 2).view(1, 1, -1)


def _box_peaks(dk, n, alatt, filters):
    """1-based peak cells of the periodic box and their filter, by plain torch: local maxima
    of each smoothed field above the threshold that no larger filter took."""
    taken = torch.zeros((n,) * 3, dtype=torch.bool, device=DEV)
    cells, fidx = [], []
    for f, flt in enumerate(filters):
        w = _window(_q(n, 0, n).float(), n, alatt, flt[2])
        s = torch.fft.irfftn(dk * w, s=(n,) * 3)
        big = torch.nn.functional.pad(s[None, None], (1,) * 6, mode="circular")
        for d in range(3):
            k = [1, 1, 1]
            k[d] = 3
            big = torch.nn.functional.max_pool3d(big, tuple(k), stride=1)
        c = torch.nonzero(((s >= FCRIT) & (s == big[0, 0]) & ~taken).reshape(-1))[:, 0]
        taken.view(-1)[c] = True
        cells.append(c)
        fidx.append(torch.full_like(c, f))
        del w, s, big
    return torch.cat(cells), torch.cat(fidx)


def prepare(case, seed):
    return {"tile": _prep_tile, "find": _prep_find, "walk": _prep_walk, "halos": _prep_halos,
            "table": _prep_table, "train": _prep_train}[case["kind"]](case, seed)


def _prep_tile(case, seed):
    n, alatt = case["n"], _alatt(case)
    tab, axes = _collapse_table()
    dk = synth.gaussian_box(n, n * alatt, seed, COSMO, DEV)
    delta = torch.fft.irfftn(dk, s=(n,) * 3).contiguous()
    mask = torch.zeros((n,) * 3, dtype=torch.int8, device=DEV)
    filters = _filters(case["nf"], alatt, case["nbuff"])
    if case["host"]:
        delta, mask = delta.cpu().numpy(), mask.cpu().numpy()
    return {"kind": "tile", "case": case, "delta": delta, "mask": mask, "filters": filters,
            "alatt": alatt, "finder": ht.HaloFinder(4, tab, *axes)}


def _prep_find(case, seed):
    n, alatt = case["n"], _alatt(case)
    tab, axes = _collapse_table()
    s = {"kind": "find", "case": case, "alatt": alatt,
         "dk": synth.gaussian_box(n, n * alatt, seed, COSMO, DEV),
         "filters": _filters(case["nf"], alatt, case["nbuff"]),
         "finder": ht.HaloFinder(4, tab, *axes),
         "mask": torch.zeros((n,) * 3, dtype=torch.int8, device=DEV),
         "peaks": ht.HaloFinder.alloc_peaks(8_000_000 if n > 400 else 1_000_000, DEV, False),
         "ds": torch.zeros((n,) * 3, dtype=torch.float32, device=DEV), "pencil": None}
    if ht.HaloFinder.pencil_supported(n):
        s["pencil"] = torch.empty((n, n // 2 + 1, n), dtype=torch.complex64, device=DEV)
    return s


def _walk_inputs(case, seed):
    """(tile fields, cells i j k, filter index, filters) of a periodic box in its tile."""
    n, nbuff, alatt = case["box"], case["nbuff"], case["alatt"]
    dk = synth.gaussian_box(n, n * alatt, seed, COSMO, DEV)
    psi1, psi2 = synth.displacements(dk, n, n * alatt, ilpt=2)
    tile = dict(zip(FIELDS, (synth.wrap_pad(t, nbuff)
                             for t in [synth._irfft(dk, n)] + psi1 + psi2)))
    tile["lapd"] = (synth.wrap_pad(synth.laplacian(dk, n, n * alatt), nbuff)
                    if case["lapd"] else None)
    filters = _filters(case["nf"], alatt, nbuff)
    cells, fidx = _box_peaks(dk, n, alatt, filters)
    # as many for every seed: a random subset in scan order (over again if there are fewer)
    keep = torch.randperm(len(cells), generator=_gen(seed), device=DEV)[:case["most"]]
    keep = keep.sort().values[torch.arange(case["most"], device=DEV) % len(keep)]
    cells, fidx = cells[keep], fidx[keep]
    i, j, k = cells % n, cells // n % n, cells // (n * n)
    return tile, [(c + nbuff + 1).int() for c in (i, j, k)], fidx, filters


def _prep_walk(case, seed):
    tab, axes = _collapse_table()
    tile, ijk, fidx, filters = _walk_inputs(case, seed)
    alatt, nbuff = case["alatt"], case["nbuff"]
    finder = ht.HaloFinder(ht.nhunt_of(filters[0][2], alatt, nbuff), tab, *axes)
    Rf = torch.tensor([f[2] for f in filters], dtype=torch.float64, device=DEV)[fidx]
    ir2 = torch.tensor([ht.ir2min_of(f[2], alatt) for f in filters], dtype=torch.int32,
                       device=DEV)[fidx]
    npk = len(fidx)
    ones = torch.ones(npk, dtype=torch.float32, device=DEV)
    return {"kind": "walk", "case": case, "tile": tile, "finder": finder,
            "args": (*ijk, Rf, ir2, ones, ones * FCRIT, alatt),
            "mask": torch.zeros_like(tile["delta"], dtype=torch.int8),
            "model": ht.bracket.BracketModel.load(device=DEV) if case["mode"] == "learned"
            else None, "out": finder.alloc_results(npk, DEV), "npk": npk}


_TABLES = {}


def _cosmo_tables():
    """The run's chi -> z and growth tables, made once per program."""
    if not _TABLES:
        c = ht.catalog.CosmologyParams()
        _TABLES["all"] = (c, ht.catalog.build_chi_to_z(c, z_max=3.0, npts=200),
                          ht.catalog.dlinear_tables(c))
    return _TABLES["all"]


def _prep_halos(case, seed):
    """Collapse results as the walk leaves them: 72 % of the peaks collapsed, radii with the
    heavy tail of a real catalogue, cells in filter order (largest radii first, in part)."""
    tab, axes = _collapse_table()
    g, npk, box = _gen(seed), case["npk"], case["box"]
    rnd = lambda *s: torch.rand(s, generator=g, device=DEV)            # noqa: E731
    nrm = lambda *s: torch.randn(s, generator=g, device=DEV)           # noqa: E731
    cells = torch.randint(0, box ** 3, (npk,), generator=g, device=DEV)
    ijk = [(c + 1).int() for c in (cells % box, cells // box % box, cells // (box * box))]
    res = {nm: nrm(npk * ht.RESULT_WIDTH.get(nm, 1)) for nm in ht.RESULT_NAMES}
    r = torch.clamp(0.9 * rnd(npk) ** -0.42, max=25.0)
    res["RTHL"] = r
    r[torch.randperm(npk, generator=g, device=DEV)[int(0.72 * npk):]] = -1.0
    finder = ht.HaloFinder(4, tab, *axes)
    ht.catalog.set_cosmology(finder, *_cosmo_tables())
    peaks = {"i": ijk[0], "j": ijk[1], "k": ijk[2], "Rf": (1.5 + 10 * rnd(npk)).double(),
             "FcRf": FCRIT + rnd(npk), "d2Rf": nrm(npk) if case["shear"] else None, "z": None}
    return {"kind": "halos", "case": case, "finder": finder, "peaks": peaks, "results": res}


def _prep_table(case, seed):
    rng = np.random.default_rng(seed)
    Om = float(rng.uniform(0.27, 0.35))
    c = ht.catalog.CosmologyParams(Om=Om, OB=0.049, OL=1.0 - Om, h=0.674)
    col = ht.collapse
    return {"kind": "table", "ep": col.EllipsoidParams(c, solver=case["solver"]),
            "tp": col.CollapseTableParams(Nx=case["nx"], Ny=case["ny"], Nz=case["nz"])}


def _train_inputs(case, seed):
    """Standardised features and stop radii, correlated as the walk's are."""
    g, n = _gen(seed), case["batch"]
    F = torch.randn((n, 16), generator=g, device=DEV)
    F[:, 12:] = 0.0
    F = F * 0.7 + 0.3
    F[:, 12:] = 0.0
    t = 6.0 + 2.0 * F[:, 0] + F[:, 1].abs() + 0.5 * torch.randn(n, generator=g, device=DEV)
    return F.contiguous(), t.contiguous()


def _train_params(seed):
    p = ht.bracket.init_params(seed)
    return p, np.r_[np.full(12, 0.3), np.zeros(4)], np.r_[np.full(12, 1 / 0.7), np.zeros(4)]


def _prep_train(case, seed):
    tab, axes = _collapse_table()
    F, t = _train_inputs(case, seed)
    model = ht.bracket.BracketModel(*_train_params(seed), DEV)
    return {"kind": "train", "finder": ht.HaloFinder(4, tab, *axes), "F": F, "t": t,
            "model": model, "mom": torch.zeros_like(model.params),
            "vel": torch.zeros_like(model.params), "step": 0}


# -------------------------------------------------------------------------- a pass ----

def run(s):
    return {"tile": _run_tile, "find": _run_find, "walk": _run_walk, "halos": _run_halos,
            "table": _run_table, "train": _run_train}[s["kind"]](s)


def _run_tile(s):
    c, n = s["case"], s["case"]["n"]
    fc = [FCRIT] * len(s["filters"])
    r = ht.peak_find_tile_gpu(s["delta"], s["filters"], fc, s["mask"], 0.0, 0.0, 0.0,
                              s["alatt"], c["nbuff"], 1, c["shear"], max_peaks=n ** 3 // 8,
                              finder=s["finder"], return_device=not c["host"])
    cap = n ** 3 // 64    # the lists' lengths depend on the seed: zeros up to one length
    if c["host"]:
        p = r["peaks"]
        out = {"i": p.i, "j": p.j, "k": p.k, "ipp": p.ipp, "x": p.x, "y": p.y, "z": p.z,
               "delta": p.delta, "Rsmooth": p.Rsmooth, "d2Rf": r["d2Rf"]}
        return {**{k: np.pad(v, (0, cap - len(v))) for k, v in out.items()},
                "mask": r["mask"]}
    out = {k: r[k] for k in ("i", "j", "k", "delta", "lapd", "filter_idx")}
    return {**{k: _padded(v, cap) for k, v in out.items() if v is not None},
            "mask": r["mask"]}


def _padded(x, n):
    return torch.cat([x, x.new_zeros((n - x.shape[0], *x.shape[1:]))])


def _run_find(s):
    """One tile's loop over its filters, as a program with the tile's spectrum in hand runs
    it.  Returned: the mask, which holds every peak of every filter, and the rows of the
    last smoothed field that the scan reads (no others are defined)."""
    c, f = s["case"], s["finder"]
    n, nbuff, L = c["n"], c["nbuff"], c["n"] * s["alatt"]
    lo, hi = nbuff - 1, n - nbuff + 1
    s["mask"].zero_()
    s["peaks"]["count"].zero_()
    s["peaks"]["found"].zero_()
    if s["pencil"] is not None:
        f.spectrum_pencil(s["dk"], n, out=s["pencil"])
    for fi, flt in enumerate(s["filters"], start=1):
        if s["pencil"] is not None:
            f.smooth_pencil(s["pencil"], n, L, flt[2], 1, lo, hi, out=s["ds"])
        else:
            f.smooth_tile(s["dk"], n, L, flt[2], 1, out=s["ds"], planes=(lo, hi))
        f.peakfind_filter(s["ds"], s["mask"], nbuff, FCRIT, fi, s["peaks"]["i"].numel(),
                          s["peaks"])
    return {"mask": s["mask"], "ds": s["ds"][lo:hi, lo:hi]}


def _run_walk(s):
    """One tile's collapse: bind the fields, order the work, analyse every peak."""
    c, f, t = s["case"], s["finder"], s["tile"]
    s["mask"].zero_()
    f.bind_fields(*(t[k] for k in FIELDS), t["lapd"])
    cost = None
    if s["model"] is not None:
        F = ht.bracket.features(f, *s["args"])
        cost = ht.bracket.predict(f, s["model"], F)[:, 1].contiguous()
    f.analyse(*s["args"], nbuff=c["nbuff"], mask=s["mask"], conv=c["conv"], mode=c["mode"],
              out=s["out"], cost=cost)
    return {**s["out"], "mask": s["mask"]}


def _run_halos(s):
    c, cat = s["case"], ht.catalog
    rec = cat.pack_halos(s["finder"], s["peaks"], s["results"], c["box"], (0.0, 0.0, 0.0), 1.0,
                         ioutshear=c["shear"])
    merged = cat.merge_halos(s["finder"], rec, volume_reduction=c["reduce"])
    return {"records": rec, "merged": _padded(merged, rec.shape[0])}


def _run_table(s):
    return ht.collapse.make_table(s["ep"], s["tp"])


def _run_train(s):
    br, m = ht.bracket, s["model"]
    g, loss = br.grad(s["finder"], m, s["F"], s["t"])
    s["step"] += 1
    st = m.struct()
    _lib = ht.bracket._lib
    _lib.check(_lib.load().ht_bracket_adam(
        s["finder"].handle, m.params.data_ptr(), g.data_ptr(), s["mom"].data_ptr(),
        s["vel"].data_ptr(), s["step"], 2e-3, br.C.byref(st),
        torch.cuda.current_stream().cuda_stream))
    return {"grad": g, "loss": loss, "params": m.params}


# ---------------------------------------------------------------- work, tolerances ----

def work(case):
    """Bytes and operations of one pass that no implementation can do without."""
    kind = case["kind"]
    if kind in ("tile", "find"):
        # every filter: the spectrum in, the field of the scanned region out and back in
        n, nf = case["n"], case["nf"] * (2 if case.get("shear") else 1)
        reg = (n - 2 * case["nbuff"]) / n
        cells = float(n) ** 3
        return {"bytes": nf * cells * 4 * (1 + 2 * reg ** 2),
                "flops": nf * cells * 2.5 * 3 * math.log2(n)}
    if kind == "walk":
        # the tile's fields and mask once, and the results; 26 operations on the about 900
        # cells that a peak's collapse takes
        cells = (case["box"] + 2.0 * case["nbuff"]) ** 3
        npk = case["most"]
        return {"bytes": cells * (30 if case["lapd"] else 29) + npk * 200,
                "flops": npk * 26.0 * 900}
    if kind == "halos":
        w = 132 if case["shear"] else 44
        return {"bytes": case["npk"] * (72 + 0.72 * 1.4 * w) + case["npk"] * 0.72 * w,
                "flops": case["npk"] * 300.0}
    if kind == "table":
        per = 4 * 220 * (2500.0 if case["solver"] == "rk4" else 160.0)
        cells = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": cells * 4.0, "flops": cells * per}
    return {"bytes": case["batch"] * 68.0 + 9928 * 20, "flops": case["batch"] * 6.0 * 9664}


def tolerance(case):
    kind = case["kind"]
    if kind == "tile":      # 32-bit transforms; Laplacian and heights as the field
        return {"rel": 3e-6, "max": 2e-5, "differ": 1e-5}
    if kind == "find":      # a mask cell may flip where two cells tie to a rounding
        return {"rel": 2e-6, "max": 2e-5, "differ": 1e-6}
    if kind == "walk":      # 64-bit sums of 32-bit fields, results rounded to 32 bits
        return {"rel": 2e-7, "max": 1e-5, "differ": 1e-6}
    if kind in ("halos", "table"):
        return "exact"
    return {"rel": 1e-2, "max": 0.2}   # bf16 operands


# --------------------------------------------------------------- 64-bit restatement ----

def exact(case, seed):
    return {"tile": _exact_tile, "find": _exact_find, "walk": _exact_walk,
            "train": _exact_train}.get(case["kind"], lambda c, s: None)(case, seed)


def _smooth64(dk, n, alatt, Rf, laplace=False):
    w = torch.empty_like(dk)
    for z in range(0, n, 32):
        q = _q(n, z, min(n, z + 32))
        k2 = q * (2.0 * math.pi / (n * alatt)) ** 2
        w[z:z + 32] = dk[z:z + 32] * (k2 * torch.exp(-k2 * Rf * Rf / 8) if laplace
                                      else _window(q, n, alatt, Rf))
        if laplace and z == 0:
            w[0, 0, 0] = dk[0, 0, 0]
    return torch.fft.irfftn(w, s=(n,) * 3)


def _exact_find(case, seed):
    n, nbuff, alatt = case["n"], case["nbuff"], _alatt(case)
    dk = synth.gaussian_box(n, n * alatt, seed, COSMO, DEV).to(torch.complex128)
    ds = _smooth64(dk, n, alatt, _filters(case["nf"], alatt, nbuff)[-1][2])
    lo, hi = nbuff - 1, n - nbuff + 1
    return {"mask": None, "ds": ds[lo:hi, lo:hi]}


def _exact_tile(case, seed):
    """Heights and Laplacians at the peaks of a 64-bit scan of the 64-bit smoothed fields."""
    n, nb, alatt = case["n"], case["nbuff"], _alatt(case)
    dk = synth.gaussian_box(n, n * alatt, seed, COSMO, DEV)
    delta = torch.fft.irfftn(dk, s=(n,) * 3).contiguous()
    dk = torch.fft.rfftn(delta.double())
    mask = torch.zeros((n,) * 3, dtype=torch.bool, device=DEV)
    inner = torch.zeros_like(mask)
    inner[nb:n - nb, nb:n - nb, nb:n - nb] = True
    out = {"delta": [], "lapd": [], "Rf": [], "cell": []}
    for flt in _filters(case["nf"], alatt, nb):
        s = _smooth64(dk, n, alatt, flt[2])
        big = torch.nn.functional.max_pool3d(s[None, None], 3, stride=1, padding=1)[0, 0]
        c = torch.nonzero((inner & ~mask & (s >= FCRIT) & (s == big)).view(-1))[:, 0]
        mask.view(-1)[c] = True
        out["cell"].append(c)
        out["delta"].append(s.view(-1)[c])
        out["Rf"].append(torch.full((len(c),), flt[2], dtype=torch.float64, device=DEV))
        if case["shear"]:
            out["lapd"].append(_smooth64(dk, n, alatt, flt[2], True).reshape(-1)[c])
    d = {k: torch.cat(v) for k, v in out.items() if v}
    pad = lambda v: None if v is None else _padded(v, n ** 3 // 64)    # noqa: E731
    if not case["host"]:
        return {"delta": pad(d["delta"]), "lapd": pad(d.get("lapd"))}
    cell = d["cell"]
    pos = [alatt * (c + 1 - 0.5 * (n + 1)) for c in (cell % n, cell // n % n, cell // (n * n))]
    return {"x": pad(pos[0]), "y": pad(pos[1]), "z": pad(pos[2]), "delta": pad(d["delta"]),
            "Rsmooth": pad(d["Rf"]), "d2Rf": pad(d.get("lapd", torch.zeros_like(d["delta"])))}


def _exact_train(case, seed):
    """One step from zero moments in 64 bits, weights rounded to bf16 as they are kept."""
    F, t = _train_inputs(case, seed)
    p0, mean, istd = _train_params(seed)
    p = torch.as_tensor(p0, device=DEV).double().requires_grad_(True)
    X = (F.double() - torch.as_tensor(mean, device=DEV)) * torch.as_tensor(istd, device=DEV)
    o, W = 0, {}
    for name, shape in ht.bracket.LAYOUT:
        k = int(np.prod(shape))
        v = p[o:o + k].view(shape)
        if name[0] == "W":   # the value is the rounded weight, the gradient is the weight's
            v = v + (v.detach().float().bfloat16().double() - v.detach())
        W[name], o = v, o + k
    h = X
    for l in "123":
        h = torch.relu(h @ W["W" + l].T + W["b" + l])
    y = h @ W["W4"][:2].T + W["b4"][:2]
    d = t.double()[:, None] - y
    tau = torch.tensor(ht.bracket.QUANTILES, dtype=torch.float64, device=DEV)
    loss = torch.maximum(tau * d, (tau - 1) * d).sum() / len(t)
    loss.backward()
    return {"grad": p.grad, "loss": None, "params": None}


# The shell collapse in 64 bits, vectorised over peaks (all cells within the hunt radius of
# each peak are read; the SPH window sums are products with a matrix of weights).

def _kernel_integral(u0, u12):
    """int_{|u0|}^2 4 pi W(x) x (x^2 - u12) dx of the cubic-spline SPH kernel W."""
    a = np.abs(u0)
    outer = lambda x: (x**4 * (2 - x * (2.4 - x * (1 - x / 7))),                # noqa: E731
                       x**2 * (4 - x * (4 - x * (1.5 - 0.2 * x))))
    inner = lambda x: (x**4 * (1 - x * x * (1 - 3 * x / 7)),                    # noqa: E731
                       x**2 * (2 - x * x * (1.5 - 0.6 * x)))
    base = 1.6 * u12 - 6.4 / 7
    o, i = outer(a), inner(a)
    return np.where(a >= 1, base + o[0] - o[1] * u12,
                    base - 0.2 * (u12 - 1 / 7) + i[0] - i[1] * u12)


def _eig(E):
    """Ascending eigenvalues of (..., 6) symmetric matrices (11, 22, 33, 12, 13, 23)."""
    q = E[..., :3].mean(-1)
    b = E[..., :3] - q[..., None]
    c12, c13, c23 = E[..., 3], E[..., 4], E[..., 5]
    pp = torch.sqrt((b.square().sum(-1) + 2 * (c12**2 + c13**2 + c23**2)) / 6)
    det = (b[..., 0] * (b[..., 1] * b[..., 2] - c23**2) - c12 * (c12 * b[..., 2] - c23 * c13)
           + c13 * (c12 * c23 - b[..., 1] * c13))
    phi = torch.acos((det / (2 * pp**3)).clamp(-1, 1).nan_to_num(0.0)) / 3
    hi = q + 2 * pp * torch.cos(phi)
    lo = q + 2 * pp * torch.cos(phi + 2 * math.pi / 3)
    return torch.stack([lo, 3 * q - lo - hi, hi], -1)


def _shape(E):
    lam = _eig(E)
    tr = lam.sum(-1)
    e = torch.where(tr > 0, 0.5 * (lam[..., 2] - lam[..., 0]) / tr, torch.zeros_like(tr))
    p = torch.where(tr > 0, 0.5 * (lam[..., 2] + lam[..., 0] - 2 * lam[..., 1]) / tr,
                    torch.zeros_like(tr))
    return lam, tr, e, p


def _zvir(tab, axes, F, E):
    """Collapse redshift factor of overdensity F and strain E, -1 outside the table."""
    _, _, e, p = _shape(E)
    xs = (torch.log10(F.clamp(min=1e-300)), e,
          torch.where(e < 1e-5, torch.zeros_like(e), p / e))
    inside, at, fr = F > 0, [], []
    for d, x in enumerate(xs):
        a, b, n = axes[2 * d], axes[2 * d + 1], tab.shape[2 - d]
        inside = inside & (x >= a) & (x <= b)
        t = ((x - a) / ((b - a) / (n - 1))).nan_to_num(0.0).clamp(-1, n)
        i = torch.floor(t).clamp(0, n - 2)
        at.append(i.long())
        fr.append(t - i)
    v = 0.0
    for c in range(8):
        b = (c & 1, c >> 1 & 1, c >> 2)
        w = 1.0
        for d in range(3):
            w = w * (fr[d] if b[d] else 1 - fr[d])
        v = v + w * tab[at[2] + b[2], at[1] + b[1], at[0] + b[0]]
    return torch.where(inside, v, torch.full_like(v, -1.0))


def _exact_walk(case, seed):
    alatt, nbuff = case["alatt"], case["nbuff"]
    R = min(nbuff - 1, math.floor(_filters(case["nf"], alatt, nbuff)[0][2] * 1.75 / alatt))
    npk = case["most"]
    if npk * 4.2 * R ** 3 > 1.5e10:     # cells read, all peaks
        return None
    tile, ijk, fidx, filters = _walk_inputs(case, seed)
    tab, axes = _collapse_table()
    tab = torch.as_tensor(tab, device=DEV, dtype=torch.float64)
    r = np.arange(-R, R + 1)
    off = np.stack(np.meshgrid(r, r, r, indexing="ij")[::-1], -1).reshape(-1, 3)
    r2 = (off ** 2).sum(1)
    order = np.argsort(r2, kind="stable")
    order = order[r2[order] <= R * R]
    off, r2 = off[order], r2[order]
    ur2, start = np.unique(r2, return_index=True)
    m = len(ur2) - 1                       # the reference never closes the last shell
    off, last = off[:start[m]], np.r_[start[1:m + 1]] - 1
    rad = np.sqrt(ur2[:m].astype(np.float64))
    u0 = rad[:, None] - rad[None, :]
    with np.errstate(divide="ignore", invalid="ignore"):
        u12 = rad[:, None] ** 2 + rad[None, :] ** 2
        W = np.where(u0**2 < 4, _kernel_integral(u0, u12) / (u12 - u0**2) ** 2, 0.0)
        W *= 3.0 / (4 * math.pi) / alatt / rad[:, None]
        u = np.arange(1101) * 0.01
        ru = np.sqrt(u)
        akk = np.where(ru < 1, 1.5 / math.pi * (2 / 3 - u + 0.5 * u * ru),
                       np.where(ru <= 2, (2 - ru) ** 3 / (4 * math.pi), 0.0))
        akk[1100] = 0.0
        W[0] = np.where(rad < 2, 0.5 * np.interp(100 * rad**2, np.arange(1101), akk) / rad
                        * 3 / alatt, 0.0)
    W[:, 0] = 0.0
    T = lambda a: torch.as_tensor(a, device=DEV)                       # noqa: E731
    Wd, rd, r2d, lastd, offd = T(W), T(rad), T(ur2), T(last), T(off)
    nt = tile["delta"].shape[0]
    rows, n = [], len(fidx)
    P = max(1, int(1.2e7 // len(off)))
    for a in range(0, n, P):
        sl = slice(a, min(n, a + P))
        rows.append(_exact_chunk(case, tile, [c[sl].long() for c in ijk], fidx[sl], filters,
                                 nt, m, offd, lastd, r2d, rd, Wd, tab, axes))
    out = {k: torch.cat([x[k] for x in rows]).reshape(-1) for k in rows[0]}
    out["mask"] = None
    return out


def _exact_chunk(case, tile, ijk, fidx, filters, nt, m, off, last, r2, rad, W, tab, axes):
    alatt, gpu, n = case["alatt"], case["conv"] == "gpu", len(fidx)
    c = [v[:, None] - 1 + off[None, :, d] for d, v in enumerate(ijk)]
    at = c[0] + nt * c[1] + nt * nt * c[2]
    value = lambda k, ix=at: tile[k].reshape(-1)[ix].double()          # noqa: E731

    def shells(x):
        s = torch.cumsum(x, 1)[:, last]
        return torch.cat([s[:, :1], s[:, 1:] - s[:, :-1]], 1)

    d = [off[None, :, L].double() for L in range(3)]
    v = value("delta")
    cnt = torch.diff(torch.cat([last.new_full((1,), -1), last])).double()
    dF = shells(v) / cnt
    G = [shells(v * d[L]) / rad for L in range(3)]
    v = value("delta", c[2] + nt * c[0] + nt * nt * c[1])
    G += [shells(v * d[L]) / rad for L in range(3)]
    e = [value("eta" + L) for L in "xyz"]
    S1 = [shells(x) for x in e]
    G += [shells(2 * e[L] * d[L]) / rad for L in range(3)]
    G += [shells(e[L] * d[K] + e[K] * d[L]) / rad for L, K in ((0, 1), (0, 2), (1, 2))]
    del e
    S2 = [shells(value("eta2" + L)) for L in "xyz"]
    lap = shells(value("lapd")) if case["lapd"] else torch.zeros_like(dF)
    G = torch.stack(G, -1)
    G[:, 0] = 0.0                          # [peak, shell, 3 + 3 + 6]
    step = lambda x, p: 0.5 * (x[:, 1:] + x[:, :-1]) * torch.diff(rad ** p)    # noqa: E731
    zero = torch.zeros((n, 1), dtype=torch.float64, device=DEV)
    Fb = torch.cumsum(step(dF, 3), 1) / rad[1:] ** 3
    Fb = torch.cat([dF[:, :1], Fb], 1)
    srb = torch.cat([zero, torch.cumsum(step(Fb, 5), 1)], 1)
    Rf = torch.tensor([f[2] for f in filters], dtype=torch.float64, device=DEV)[fidx]
    ir2 = torch.tensor([min(math.floor((1.75 * f[2] / alatt) ** 2),
                            math.floor((40.0 / alatt - 1) ** 2)) for f in filters],
                       device=DEV)[fidx]
    sh = torch.arange(m, device=DEV)[None, :]          # 0-based shells
    first = lambda ok, other: torch.where(ok.any(1), ok.int().argmax(1), other)  # noqa: E731
    top = torch.full((n,), m - 1, device=DEV)
    pick = lambda x, s: x.gather(1, s.clamp(0, m - 1)[:, None])[:, 0]  # noqa: E731
    fc = float(np.float32(FCRIT))
    m0i = first((r2[None, :m] > ir2[:, None]) & (sh >= 1), top)
    high = pick(Fb, m0i) >= fc
    out_x = first((Fb < fc) & (sh >= m0i[:, None]), m0i)
    ge = (Fb >= fc) & (sh < m0i[:, None])
    in_x = torch.where(ge, sh + 1, torch.zeros_like(sh)).amax(1)       # shell above the last
    m0 = torch.where(high, out_x, in_x)
    ok = high | ge.any(1)
    top_s = int(m0.max()) + 1
    E = torch.einsum("st,ptc->psc", -0.5 * W[:top_s], G[..., 6:])
    z = _zvir(tab, axes, Fb[:, :top_s], E)
    hit = (z >= 1.0) & (sh[:, :top_s] < m0[:, None])
    ok &= hit.any(1)
    mp = torch.where(hit, sh[:, :top_s], torch.zeros_like(sh[:, :top_s])).amax(1)
    mu = mp + 1
    gs = torch.einsum("pst,ptc->psc", W[torch.stack([mp, mu], 1).clamp(max=m - 1)], G[..., :6])
    Es = lambda s: E[torch.arange(n, device=DEV), s.clamp(max=top_s - 1)]      # noqa: E731
    zp = z.gather(1, mp[:, None])[:, 0]
    zu = torch.where(mu == m0, -torch.ones_like(zp),
                     z.gather(1, mu.clamp(max=top_s - 1)[:, None])[:, 0])
    rp, rm = rad[mp], rad[mu.clamp(max=m - 1)]
    inter = (zu > 0) & (zp != zu)
    R3 = rp**3 + (rm**3 - rp**3) * (zp - 1.0) / torch.where(inter, zp - zu,
                                                           torch.ones_like(zp))
    RT = torch.where(inter, R3.clamp(min=0) ** (1 / 3), rp)
    ok &= RT > 0
    inter = zu > 0
    fr = torch.where(inter, (RT**3 - rp**3) / (rm**3 - rp**3), torch.zeros_like(RT))
    Fp, Fm = pick(Fb, mp), pick(Fb, mu)
    Fx = Fp + fr * (Fm - Fp)
    Em = Es(mp) + fr[:, None] * (Es(mu) - Es(mp))
    gp = torch.where(inter[:, None], gs[:, 0] + fr[:, None] * (gs[:, 1] - gs[:, 0]), gs[:, 1])
    tr = Em[:, :3].sum(1)
    lam, _, ev, pv = _shape(torch.where(tr != 0, Fx / tr, torch.ones_like(tr))[:, None] * Em)
    Frh = _eig(Es(mp)).sum(1)
    fin = Es(mp) * (Fx / Frh)[:, None]
    if gpu:
        fin = torch.where((Frh == 0)[:, None], Es(mp), fin)
    Sr = pick(srb, mp) + torch.where((zu > 0) & (zp != zu),
                                     0.5 * (Fp + Fx) * (RT**5 - rp**5), torch.zeros_like(RT))
    Sr = torch.where(Fx * RT**5 > 0, Sr / (Fx * RT**5), Sr)
    cum = lambda x, s: pick(torch.cumsum(x, 1), s)                     # noqa: E731
    ncum = torch.cumsum(cnt, 0)
    Sb = torch.stack([cum(x, mp) for x in S1 + S2], 1) / ncum[mp][:, None]
    s_in = (rad[None] <= RT[:, None]).sum(1) - 1
    d2 = cum(lap, s_in) / ncum[s_in] if gpu else \
        (cum(lap, s_in) - lap[:, 0]) / (ncum[s_in] - 1).clamp(min=1)
    # gradient at the filter scale, two shells (one on the device) inside the nearest
    smax = m if gpu else len(r2)
    dist = (r2[None, :smax].double() - (Rf / alatt)[:, None] ** 2).abs()
    dist[:, 0] = math.inf
    best, which = dist.min(1)
    which = (dist == best[:, None]).int().argmax(1)
    mrf = torch.where(best < 10, which - 1 if gpu else (which - 2).clamp(min=0), which * 0)
    grf = torch.einsum("pt,ptc->pc", W[mrf], G[..., :3])
    grf = torch.where((mrf == 0)[:, None], torch.full_like(grf, math.nan), grf)
    # largest collapse redshift of ten radii between RTHL / 2^(1/3) and RTHL
    zh = torch.full_like(RT, -math.inf)
    for jj in range(10):
        rc = RT * (0.5 + 0.5 * jj / 9) ** (1 / 3)
        above = lambda x, lo: first((rad[None, :m - 1] > x[:, None])           # noqa: E731
                                    & (sh[:, :m - 1] >= lo), top - 1)
        mid, lo, hi = above(rc, 0), above((rc - 2).clamp(min=0), 0), above(rc + 2, 1)
        w = W[mid] * ((sh >= lo[:, None]) & (sh <= hi[:, None]))
        Ez = -0.5 * torch.einsum("pt,ptc->pc", w, G[..., 6:])
        zh = torch.maximum(zh, _zvir(tab, axes, pick(Fb, mid), Ez) - 1.0)
    zh = torch.where(RT >= 3.0, zh, -torch.ones_like(zh))
    mat = fin[:, [0, 3, 4, 3, 1, 5, 4, 5, 2]]
    res = {"RTHL": RT, "Fbarx": Fx, "e_v": ev, "p_v": pv, "strain": mat, "eigs": lam,
           "Srb": Sr, "Sbar": Sb[:, :3], "Sbar2": Sb[:, 3:], "gradpk": gp[:, :3],
           "gradpkf": gp[:, 3:], "gradpkrf": grf, "d2F": d2, "zvir_half": zh}
    for k, x in res.items():
        none = -1.0 if k in ("RTHL", "zvir_half") else 0.0
        o = ok if x.dim() == 1 else ok[:, None]
        res[k] = torch.where(o, x, torch.full_like(x, none))
    return res
