"""What a user of this framework runs, at the sizes a user runs it.

The framework's main path is the Newton filter (six of the listed cases: both
precisions, grids from 36^3 to 192^3, square and rectangular planes, one
crystal and a batch); around it stand the Hamiltonian apply, the whole
pipeline, the subspace products, the local potential with its gradient, the
bulk band-structure fit with its gradient, and the spinor filter.

Inputs: zincblende dots cut to the box (a = 11.4895 bohr), a local potential
of one attractive well per atom (about 1.2 Ha deep, two species), normalised
random start states, Gaussian filters interpolated at Leja points.  The
spectrum is bounded by the kinetic cap plus the range of the potential.

The FP64 filter runs the 1024 Newton steps of the reference configurations.
The complex64 filters run 256: every step costs the same, and single
precision's rounding error grows in proportion to the steps (9e-6 of the
result at 256, 3e-5 at 1024).
"""
import functools
import math
import random

import numpy as np
import torch

import semi_empirical_pseudopotentials_gb300 as sep
from semi_empirical_pseudopotentials_gb300 import bulk, spinor

LENGTHS = (14, 16, 18, 20, 24, 32, 36, 40, 48, 56, 64, 72, 80, 96, 112, 128, 160, 192, 256)
A0 = 11.4895          # lattice constant, bohr
EKIN = 10.0           # kinetic cap of the filter program, hartree
EKIN_SPINOR = 20.0    # of the spinor filter program
EV = 27.2114
MAX_STEPS_C64 = 1.8e10   # pairs x points x Newton steps of the largest complex64 case
MAX_STEPS_F64 = 2.2e9    # and of the largest FP64 case (20 times slower a step)


def listed():
    return [
        # one H apply on host arrays, as the C program's hamiltonian() is called
        # through the fd.h-compatible layer on a toy system: latency
        dict(name="hpsi_f64_16x18x20", kind="hpsi", nx=16, ny=18, nz=20, ns=1),
        # the published small nanocrystal: 36^3, 16 start states x 10 targets
        dict(name="filter_c64_36", kind="filter", prec="mixed", nx=36, ny=36, nz=36, ns=16,
             ms=10, nc=256),
        # the plain FP64 filter of the smallest configuration: 64^3, 8 x 4
        dict(name="filter_f64_64", kind="filter", prec="f64", nx=64, ny=64, nz=64, ns=8, ms=4,
             nc=1024),
        # a nanorod-like box (the published 80 x 64 x 64 run, 48 of its states x 20 targets)
        dict(name="filter_c64_80x64x64", kind="filter", prec="mixed", nx=80, ny=64, nz=64, ns=48,
             ms=20, nc=256),
        # the headline workload: 2.5 nm dot on 128^3, 64 start states x 8 targets
        dict(name="filter_c64_128", kind="filter", prec="mixed", nx=128, ny=128, nz=128, ns=64,
             ms=8, nc=256),
        # the large dot's grid, a part of its states
        dict(name="filter_c64_192", kind="filter", prec="mixed", nx=192, ny=192, nz=192, ns=16,
             ms=8, nc=256),
        # many nanocrystals of uneven grids in one launch, 16 states x 4 targets each
        dict(name="batch_c64_48_112", kind="batch", sizes="48,112,56,96,64,80,72,64", ns=16, ms=4,
             nc=256),
        # the whole program on host arrays: energy range, filter, ortho, Ritz, sigma
        dict(name="pipeline_f64_48", kind="pipeline", nx=48, ny=48, nz=48, ns=8, ms=4, nc=512),
        # Gram matrix of the headline workload's 512 filtered states
        dict(name="gram_512", kind="gram", m=512, n=0, k=2097152),
        # V(r) of the 2.5 nm dot and the gradient in its radial tables (form-factor fit)
        dict(name="potential_128", kind="potential", nx=128, ny=128, nz=128),
        # two fit steps (bands and their gradient at new parameters) of wurtzite CdSe:
        # 42 k-points, about 380 plane waves, 16 bands
        dict(name="bulk_fit_42", kind="bulk", max_ke=5.0, nk=42, ne=16),
        # the spinor filter with the Gaussian spin-orbit operator of 64 atoms
        dict(name="spinor_filter_48", kind="spinor", n=48, natom=64, ns=4, ms=4, nc=64),
    ]


# ---- draws ------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _dims(rng, lo, hi):
    ok = [v for v in LENGTHS if lo <= v <= hi]
    n = ok[rng.randrange(len(ok))]
    if rng.random() < 0.5:
        return n, n, n
    near = [v for v in ok if 0.6 * n <= v <= 1.7 * n]
    return n, near[rng.randrange(len(near))], near[rng.randrange(len(near))]


def _draw_filter(rng):
    prec = "mixed" if rng.random() < 0.7 else "f64"
    nx, ny, nz = _dims(rng, 24, 192 if prec == "mixed" else 96)
    ns, ms = _log_int(rng, 1, 64), rng.randint(1, 20)
    nc = _log_int(rng, 32, 256 if prec == "mixed" else 1024)
    n = nx * ny * nz
    cap = MAX_STEPS_C64 if prec == "mixed" else MAX_STEPS_F64
    while ns > 1 and (((ns + 1) // 2) * n * nc > cap or ns * ms * n > 1.1e9):
        ns -= 1
    nc = max(32, min(nc, int(cap / (((ns + 1) // 2) * n))))
    return dict(kind="filter", prec=prec, nx=nx, ny=ny, nz=nz, ns=ns, ms=ms, nc=nc)


def draw(rng: random.Random):
    kind = rng.choices(("filter", "hpsi", "batch", "pipeline", "gram", "potential", "bulk",
                        "spinor"), (8, 1, 2, 1, 2, 1, 2, 2))[0]
    if kind == "filter":
        return _draw_filter(rng)
    if kind == "hpsi":
        nx, ny, nz = _dims(rng, 14, 64)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, ns=rng.randint(1, 8))
    if kind == "batch":
        sizes = [rng.choice([v for v in LENGTHS if 36 <= v <= 112])
                 for _ in range(rng.randint(2, 8))]
        return dict(kind=kind, sizes=",".join(map(str, sizes)), ns=rng.randint(2, 16),
                    ms=rng.randint(1, 8), nc=_log_int(rng, 32, 256))
    if kind == "pipeline":
        nx, ny, nz = _dims(rng, 36, 56)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, ns=rng.randint(2, 8), ms=rng.randint(2, 4),
                    nc=_log_int(rng, 200, 512))
    if kind == "gram":
        return dict(kind=kind, m=rng.randint(24, 512), n=rng.choice((0, rng.randint(8, 512))),
                    k=_log_int(rng, 40000, 2097152))
    if kind == "potential":
        nx, ny, nz = _dims(rng, 48, 128)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz)
    if kind == "bulk":
        return dict(kind=kind, max_ke=round(rng.uniform(1.6, 5.0), 2), nk=rng.randint(6, 42),
                    ne=2 * rng.randint(4, 8))
    return dict(kind=kind, n=rng.choice((32, 36, 40, 48)), natom=rng.randint(8, 64),
                ns=rng.randint(1, 4), ms=rng.randint(1, 4), nc=rng.randint(16, 64))


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spacing(n):
    return 0.75 if n >= 36 else 0.9


def _dot(half, rng):
    """Zincblende atoms inside the ellipsoid 5 bohr within the box, shifted a
    little: (xyz, types)."""
    r = np.maximum(np.asarray(half) - 5.0, 4.0)
    m = int(np.ceil(r.max() / A0)) + 1
    g = np.arange(-m, m + 1)
    cells = np.array(np.meshgrid(g, g, g, indexing="ij")).reshape(3, -1).T
    fcc = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    cat = (cells[:, None, :] + fcc[None]).reshape(-1, 3) * A0
    shift = rng.uniform(-1.0, 1.0, 3)
    xyz, types = [], []
    for t, sites in enumerate((cat, cat + A0 / 4)):
        keep = (((sites + shift) / r) ** 2).sum(1) <= 1.0
        xyz.append(sites[keep] + shift)
        types.append(np.full(int(keep.sum()), t, dtype=np.int32))
    return np.concatenate(xyz), np.concatenate(types)


def _potential(dims, h, seed):
    """Sum of Gaussian wells on the dot's atoms, [nz, ny, nx] on the GPU."""
    rng = np.random.default_rng(seed)
    half = [0.5 * n * h for n in dims]
    xyz, types = _dot(half, rng)
    depth = torch.tensor(np.where(types == 0, -0.7, -1.2) * (1 + 0.05 * rng.uniform(-1, 1)),
                         device="cuda")
    w = torch.tensor(np.where(types == 0, 1.45, 1.15), device="cuda")
    pos = torch.tensor(xyz, device="cuda")
    ax = [torch.exp(-0.5 * ((-half[d] + h * torch.arange(dims[d], device="cuda",
                                                         dtype=torch.float64))[None, :]
                            - pos[:, d:d + 1]) ** 2 / w[:, None] ** 2) for d in range(3)]
    plane = (ax[1][:, :, None] * ax[0][:, None, :]).reshape(len(types), -1)
    v = (ax[2] * depth[:, None]).T @ plane
    return v.reshape(dims[2], dims[1], dims[0])


@functools.lru_cache(maxsize=64)
def _leja(nc):
    """Leja points on [-2, 2] from 28 nc evenly spaced candidates and the origin."""
    z = np.append(np.linspace(-2.0, 2.0, 28 * nc), 0.0)
    out, s = np.empty(nc), np.zeros(len(z))
    k = 0
    for j in range(nc):
        out[j] = z[k]
        with np.errstate(divide="ignore"):
            s += np.log(np.abs(z - z[k]))
        k = int(np.argmax(s))
    return out


def _newton(el, nc, dE, vmin):
    """Divided differences of exp(-(E - el)^2 dt) at the Leja points -> (an, zn)."""
    zn = _leja(nc)
    dt = (nc / (2.5 * dE)) ** 2
    f = np.exp(-((zn[None, :] + 2.0) * dE / 4.0 + vmin - np.asarray(el)[:, None]) ** 2 * dt)
    c = np.zeros_like(f)
    c[:, 0] = f[:, 0]
    for j in range(1, nc):
        w = np.cumprod(zn[j] - zn[:j])
        c[:, j] = (f[:, j] - c[:, 0] - c[:, 1:j] @ w[:j - 1]) / w[j - 1]
    return np.ascontiguousarray(c), zn.copy()


def _targets(ms):
    """Energies where a dot of 8 electrons an atom pair has its band edges."""
    return np.linspace(0.0, 0.3, ms) if ms > 1 else np.array([0.1])


def _filter_inputs(dims, ns, ms, nc, seed):
    h = _spacing(min(dims))
    v = _potential(dims, h, seed)
    vmin, vmax = float(v.min()), float(v.max())
    dE = 1.1 * (EKIN + vmax - vmin)
    an, zn = _newton(_targets(ms), nc, dE, vmin)
    n = v.numel()
    start = torch.rand((ns, n), generator=_gen(seed + 1), device="cuda", dtype=torch.float64)
    start.mul_(2.0).sub_(1.0)
    for row in start:
        row /= torch.sqrt((row * row).sum() * h ** 3)
    return dict(dims=dims, h=h, v=v, vmin=vmin, dE=dE, an=an, zn=zn, start=start)


def _spinor_inputs(case, seed):
    n, h = case["n"], 0.6
    rng = np.random.default_rng(seed)
    v = _potential((n, n, n), h, seed)
    x = -0.5 * n * h + h * np.arange(n)
    # atoms between the grid points: Vso grows as 1 / r^2 at an atom
    cell = rng.integers(-int(0.32 * n), int(0.32 * n), (case["natom"], 3))
    xyz = h * (cell + rng.uniform(0.25, 0.75, cell.shape))
    vso = rng.uniform(0.02, 0.1, case["natom"])
    vmin, dE = float(v.min()) - 0.2, 1.1 * (EKIN_SPINOR + 2.0)
    an, zn = _newton(_targets(case["ms"]), case["nc"], dE, vmin)
    start = rng.uniform(-1, 1, (case["ns"], 2 * n ** 3)) + 1j * rng.uniform(
        -1, 1, (case["ns"], 2 * n ** 3))
    start /= np.linalg.norm(start, axis=1, keepdims=True) * h ** 1.5
    return dict(n=n, h=h, v=v, x=x, xyz=xyz, vso=vso, vmin=vmin, dE=dE, an=an + 0j, zn=zn,
                start=start, r2=0.49 * 6.0 * math.log(10.0))


def _bulk_inputs(case, seed):
    """Wurtzite CdSe with two parameter sets, as two steps of a fit have them."""
    rng = np.random.default_rng(seed)
    a, c = A0 / math.sqrt(2.0), A0 * 2.0 / math.sqrt(3.0)
    cell = np.array([[a, 0, 0], [-0.5 * a, math.sqrt(0.75) * a, 0], [0, 0, c]])
    frac = np.array([[1 / 3, 2 / 3, 0], [2 / 3, 1 / 3, 1 / 2], [1 / 3, 2 / 3, 3 / 8],
                     [2 / 3, 1 / 3, 7 / 8]])
    kpts = rng.uniform(-0.5, 0.5, (case["nk"], 3)) * (2 * math.pi / A0)
    params = np.array([[0.0424846, 0.671884, 0.136082, 0.514544],
                       [-0.22725, 3.69721, -2.24471, 0.676691]])
    params = params * (1 + 0.01 * rng.uniform(-1, 1, (2,) + params.shape))
    return dict(cell=cell, tau=frac @ cell, kpts=kpts, params=params,
                dl_de=rng.normal(size=(case["nk"], case["ne"])))


def _radial_tables():
    """1024-point radial tables of the two species, the last value zero."""
    r = 0.02513274122871834 * np.arange(1024)
    v = np.stack([-0.7 * np.exp(-r * r / 4.2) + 0.02 * np.exp(-r / 3) * np.cos(1.3 * r),
                  -1.2 * np.exp(-r * r / 2.7) + 0.03 * np.exp(-r / 3) * np.cos(1.7 * r)])
    return np.stack([r, r]), v - v[:, -1:]


def _potential_inputs(case, seed):
    dims = case["nx"], case["ny"], case["nz"]
    h = 0.81
    half = [0.5 * n * h for n in dims]
    rng = np.random.default_rng(seed)
    xyz, types = _dot(half, rng)
    rho = rng.normal(size=int(np.prod(dims))) ** 2
    tr, tv = _radial_tables()
    return dict(dims=dims, h=h, mins=[-x for x in half], xyz=xyz, types=types, tr=tr, tv=tv,
                rho=rho)


def _gram_inputs(case, seed):
    g = _gen(seed)
    a = torch.randn((case["m"], case["k"]), generator=g, device="cuda", dtype=torch.float64)
    for j in range(1, case["m"]):  # filtered states of neighbouring targets overlap
        a[j].add_(a[j - 1], alpha=0.3)
    a /= math.sqrt(case["k"])
    if not case["n"]:
        return a, None
    b = torch.randn((case["n"], case["k"]), generator=g, device="cuda", dtype=torch.float64)
    return a, b / math.sqrt(case["k"])


# ---- prepare and run --------------------------------------------------------
class _DeviceArray:
    """A device pointer of the library as torch sees it."""

    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(shape=tuple(shape), typestr="<f8", version=3,
                                             data=(ptr, False))


def _context(p, precision, ekinmax=EKIN):
    return sep.Context(p["dims"], (p["h"],) * 3, potl=p["v"].cpu().numpy().ravel(),
                       precision=precision, ekinmax=ekinmax)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("hpsi", "filter", "pipeline"):
        dims = case["nx"], case["ny"], case["nz"]
    if kind == "hpsi":
        h = _spacing(min(dims))
        v = _potential(dims, h, seed)
        rng = np.random.default_rng(seed)
        psi = rng.normal(size=(case["ns"], v.numel())) + 1j * rng.normal(
            size=(case["ns"], v.numel()))
        return dict(kind=kind, ctx=_context(dict(dims=dims, h=h, v=v), "f64"), psi=psi)
    if kind == "filter":
        p = _filter_inputs(dims, case["ns"], case["ms"], case["nc"], seed)
        ctx = _context(p, case["prec"])
        shape = (case["ns"], case["ms"], ctx.ngrid)
        out = torch.empty(shape, dtype=torch.float64, device="cuda")
        # a complex64 filter's states carry single precision and are kept as such
        kept = torch.empty(shape, dtype=torch.float32, device="cuda") \
            if case["prec"] == "mixed" else out
        return dict(kind=kind, ctx=ctx, start=p["start"], an=p["an"], zn=p["zn"], dE=p["dE"],
                    vmin=p["vmin"], out=out, kept=kept,
                    stream=torch.cuda.ExternalStream(ctx.stream()))
    if kind == "batch":
        sizes = [int(s) for s in case["sizes"].split(",")]
        ps = [_filter_inputs((n, n, n), case["ns"], case["ms"], case["nc"], seed + 7 * j)
              for j, n in enumerate(sizes)]
        ctxs = [_context(p, "mixed") for p in ps]
        b = sep.Batch(ctxs, [case["ns"]] * len(ps), case["ms"], case["nc"])
        outs, kept = [], []
        for j, p in enumerate(ps):
            b.set_coefficients(j, p["an"], p["zn"], 4.0 / p["dE"], p["vmin"])
            s, o = b.io(j)
            n = ctxs[j].ngrid
            torch.as_tensor(_DeviceArray(s, (case["ns"], n)), device="cuda").copy_(p["start"])
            outs.append(torch.as_tensor(_DeviceArray(o, (case["ns"], case["ms"], n)),
                                        device="cuda"))
            kept.append(torch.empty(outs[-1].shape, dtype=torch.float32, device="cuda"))
        return dict(kind=kind, batch=b, outs=outs, kept=kept)
    if kind == "pipeline":
        p = _filter_inputs(dims, case["ns"], case["ms"], case["nc"], seed)
        return dict(kind=kind, ctx=_context(p, "f64"), start=p["start"].cpu().numpy(),
                    el=_targets(case["ms"]), nc=case["nc"], vmin=p["vmin"])
    if kind == "gram":
        a, b = _gram_inputs(case, seed)
        ctx = sep.Context((16, 16, 16), (0.9,) * 3)
        out = torch.empty((case["m"], case["n"] or case["m"]), dtype=torch.float64, device="cuda")
        return dict(kind=kind, ctx=ctx, a=a, b=b, out=out)
    if kind == "potential":
        p = _potential_inputs(case, seed)
        ctx = sep.Context(p["dims"], (p["h"],) * 3)
        return dict(kind=kind, ctx=ctx, **p)
    if kind == "bulk":
        p = _bulk_inputs(case, seed)
        crystal = bulk.Crystal(cell=p["cell"], symbols=["Cd", "Cd", "Se", "Se"], tau=p["tau"], kpts=p["kpts"],
                               max_ke=case["max_ke"], ne=case["ne"], scale=A0)
        return dict(kind=kind, crystal=bulk.BulkCrystal(crystal), params=p["params"],
                    dl_de=p["dl_de"])
    if kind == "spinor":
        p = _spinor_inputs(case, seed)
        ctx = _context(dict(dims=(p["n"],) * 3, h=p["h"], v=p["v"]), "f64", EKIN_SPINOR)
        nlc, nl = spinor.neighbour_lists(p["x"], p["x"], p["x"], p["xyz"], p["vso"], p["r2"])
        path = spinor.SpinorPath(ctx, nlc, nl, sigma=p["h"])
        return dict(kind=kind, path=path, **{k: p[k] for k in ("start", "an", "zn", "dE", "vmin")})
    raise ValueError(kind)


def _split(x):
    """The first pair of states apart from the others."""
    return dict(first=x[:2], rest=x[2:]) if len(x) > 2 else dict(first=x)


def run(s):
    kind = s["kind"]
    if kind == "hpsi":
        return s["ctx"].hamiltonian(s["psi"])
    if kind == "filter":
        s["ctx"].filter_dev(s["start"].data_ptr(), s["start"].shape[0], s["an"], s["zn"],
                            4.0 / s["dE"], s["vmin"], s["out"].data_ptr())
        if s["kept"] is not s["out"]:
            with torch.cuda.stream(s["stream"]):
                s["kept"].copy_(s["out"])
        return _split(s["kept"])
    if kind == "batch":
        s["batch"].run()
        for k, o in zip(s["kept"], s["outs"]):
            k.copy_(o)
        return [_split(k) for k in s["kept"]]
    if kind == "pipeline":
        r = s["ctx"].pipeline(s["start"], s["el"], s["nc"], s["vmin"])
        return dict(eval=r["eval"], sigma=r["sigma"], kept=r["mkept"])
    if kind == "gram":
        m, k = s["a"].shape
        b = s["b"]
        s["ctx"].subspace_gemm_dev(s["a"].data_ptr(), None if b is None else b.data_ptr(), m,
                                   s["out"].shape[1], k, s["out"].data_ptr(), sym=b is None)
        return s["out"]
    if kind == "potential":
        n = [s["tr"].shape[1]] * 2
        v = s["ctx"].vbuild(s["xyz"], s["types"], s["tr"], s["tv"], n, s["mins"])
        dtab, _ = s["ctx"].vbuild_backward(s["xyz"], s["types"], s["tr"], s["tv"], n, s["mins"],
                                           s["rho"])
        return dict(v=v, dtab=dtab)
    if kind == "bulk":
        c, steps = s["crystal"], []
        for params in s["params"]:
            bands = c.bands(params, keep_vectors=True)
            _, grad = c.backward(params, s["dl_de"])
            steps.append(dict(bands=bands, grad=grad))
        return steps
    return s["path"].filter(s["start"], s["an"], s["zn"], 4.0 / s["dE"], s["vmin"])


# ---- what a pass cannot do without -----------------------------------------
def _fft_flops(n):
    return 10.0 * n * math.log2(n) + 12.0 * n   # transform pair, k^2, V psi and the shift


def work(case):
    kind = case["kind"]
    if kind in ("hpsi", "filter", "pipeline", "potential"):
        n = case["nx"] * case["ny"] * case["nz"]
    if kind == "hpsi":
        return dict(bytes=32.0 * n * case["ns"] + 8.0 * n, flops=case["ns"] * _fft_flops(n))
    if kind == "filter":
        ns, ms, nc = case["ns"], case["ms"], case["nc"]
        out = 4 if case["prec"] == "mixed" else 8
        return dict(bytes=n * ns * (8.0 + out * ms),
                    flops=((ns + 1) // 2) * (nc - 1) * _fft_flops(n) + 2.0 * ns * ms * nc * n)
    if kind == "batch":
        parts = [work(dict(kind="filter", prec="mixed", nx=int(s), ny=int(s), nz=int(s),
                           ns=case["ns"], ms=case["ms"], nc=case["nc"]))
                 for s in case["sizes"].split(",")]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "pipeline":
        m = case["ns"] * case["ms"]
        f = work(dict(case, kind="filter", prec="f64"))
        return dict(bytes=8.0 * n * case["ns"] + 16.0 * m,
                    flops=f["flops"] + (m + 1) // 2 * _fft_flops(n) + 6.0 * m * m * n)
    if kind == "gram":
        m, k = case["m"], case["k"]
        cols = case["n"] or m
        return dict(bytes=8.0 * k * (m + case["n"]) + 8.0 * m * cols,
                    flops=2.0 * m * cols * k * (1.0 if case["n"] else 0.5))
    if kind == "potential":
        half = [0.5 * 0.81 * x for x in (case["nx"], case["ny"], case["nz"])]
        r = [max(x - 5.0, 4.0) for x in half]
        atoms = 4.0 / 3.0 * math.pi * r[0] * r[1] * r[2] / (A0 ** 3 / 8)
        reach = min(4.0 / 3.0 * math.pi * 25.7 ** 3 / 0.81 ** 3, n)
        return dict(bytes=16.0 * n + 24.0 * atoms, flops=2 * 20.0 * atoms * reach)
    if kind == "bulk":
        nbv = A0 ** 3 / 2 * (2 * case["max_ke"]) ** 1.5 / (6 * math.pi ** 2)
        return dict(bytes=16.0 * case["nk"] * (3 + 2 * case["ne"]),
                    flops=2 * case["nk"] * (16.0 / 3.0 * nbv ** 3 + 8.0 * nbv ** 2 * case["ne"]))
    n, ns = case["n"] ** 3, case["ns"]
    points = 4.0 / 3.0 * math.pi * 2.6 ** 3 / 0.6 ** 3
    vso = case["natom"] * (24.0 * points ** 2 + 200.0 * points)
    return dict(bytes=32.0 * n * ns * (1 + case["ms"]),
                flops=case["nc"] * ns * (2 * _fft_flops(n) + vso + 16.0 * case["ms"] * n))


# ---- 64-bit references ------------------------------------------------------
def _kinetic(dims, h, cap=EKIN):
    ax = []
    for n in dims:
        j = torch.arange(n, device="cuda", dtype=torch.float64)
        j = torch.minimum(j, n - j)
        ax.append(0.5 * (2 * math.pi / (n * h) * j) ** 2)
    return (ax[2][:, None, None] + ax[1][None, :, None] + ax[0][None, None, :]).clamp(max=cap)


def _hamiltonian(psi, t, v):
    """(T + V) psi on complex grids [..., nz, ny, nx]."""
    return torch.fft.ifftn(torch.fft.fftn(psi, dim=(-3, -2, -1)) * t, dim=(-3, -2, -1)) + v * psi


def _exact_filter(p, states):
    """Newton filter of the first `states` start states -> [states, ms, N]."""
    an, zn, dE_1 = p["an"], p["zn"], 4.0 / p["dE"]
    st = p["start"][:states]
    if states % 2:
        st = torch.cat([st, torch.zeros_like(st[:1])])
    nx, ny, nz = p["dims"]
    psi = torch.complex(st[0::2].contiguous(), st[1::2].contiguous()).reshape(-1, nz, ny, nx)
    t = _kinetic(p["dims"], p["h"])
    acc = torch.zeros((len(psi), len(an)) + psi.shape[1:], dtype=torch.complex128, device="cuda")
    for j in range(len(zn)):
        if j:
            psi = dE_1 * _hamiltonian(psi, t, p["v"]) \
                - (2.0 + zn[j - 1] + p["vmin"] * dE_1) * psi
        for e in range(len(an)):
            acc[:, e].add_(psi, alpha=float(an[e, j]))
    acc = acc.reshape(len(psi), len(an), -1)
    return torch.stack([acc.real, acc.imag], 1).reshape(2 * len(psi), len(an), -1)[:states]


def _ran2(idum):
    """L'Ecuyer's two combined generators behind a 32-entry shuffle (Numerical Recipes' ran2)."""
    m1, m2, a1, a2, ndiv = 2147483563, 2147483399, 40014, 40692, 1 + 2147483562 // 32
    s1 = s2 = max(-idum, 1)
    iv = [0] * 32
    for j in range(39, -1, -1):
        s1 = a1 * s1 % m1
        if j < 32:
            iv[j] = s1
    iy = iv[0]
    while True:
        s1, s2 = a1 * s1 % m1, a2 * s2 % m2
        j = iy // ndiv
        iy, iv[j] = iv[j] - s2, s1
        if iy < 1:
            iy += m1 - 1
        yield min(iy / m1, 1.0 - 1.2e-7)


def _exact_pipeline(case, seed):
    p = _filter_inputs((case["nx"], case["ny"], case["nz"]), case["ns"], case["ms"], case["nc"],
                       seed)
    t, v, dv, shape = _kinetic(p["dims"], p["h"]), p["v"], p["h"] ** 3, p["v"].shape
    gen = _ran2(-874917403)
    psi = torch.tensor([2.0 * next(gen) - 1.0 for _ in range(v.numel())], device="cuda",
                       dtype=torch.float64)
    psi = (psi / torch.sqrt((psi * psi).sum() * dv)).reshape(shape) + 0j
    hp = _hamiltonian(psi, t, v)
    ene, old = 0.1, 0.0
    while abs((ene - old) / ene) > 1e-4:
        psi, old = hp / torch.sqrt((hp.abs() ** 2).sum() * dv), ene
        hp = _hamiltonian(psi, t, v)
        ene = float((psi.conj() * hp).sum().real) * dv
    p["dE"] = 1.1 * (ene - p["vmin"])
    p["an"], p["zn"] = _newton(_targets(case["ms"]), case["nc"], p["dE"], p["vmin"])
    x = _exact_filter(p, case["ns"]).reshape(case["ns"] * case["ms"], -1)
    x = x / torch.linalg.norm(x, dim=1, keepdim=True)
    q = torch.linalg.qr(x.T)[0].T.contiguous()
    hq = _hamiltonian(q.reshape(-1, *shape) + 0j, t, v).real.reshape(q.shape)
    w, u = torch.linalg.eigh(0.5 * (q @ hq.T + hq @ q.T))
    res = u.T @ hq - w[:, None] * (u.T @ q)
    return dict(eval=w, sigma=torch.linalg.norm(res, dim=1), kept=None)


def _exact_potential(case, seed):
    p = _potential_inputs(case, seed)
    r, tab = p["tr"][0], torch.tensor(p["tv"], device="cuda")
    dr, last = float(r[1]), len(r) - 2
    ax = [p["mins"][d] + p["h"] * torch.arange(p["dims"][d], device="cuda", dtype=torch.float64)
          for d in range(3)]
    nx, ny, nz = p["dims"]
    v = torch.zeros((nz, ny, nx), dtype=torch.float64, device="cuda")
    rho = torch.tensor(p["rho"], device="cuda").reshape(nz, ny, nx)
    dtab = torch.zeros_like(tab)
    reach = dr * (len(r) - 1)
    for pos, ty in zip(p["xyz"], p["types"]):
        box = []
        for d in range(3):
            lo = max(0, int((pos[d] - reach - p["mins"][d]) / p["h"]))
            hi = min(p["dims"][d], int((pos[d] + reach - p["mins"][d]) / p["h"]) + 2)
            box.append(slice(lo, hi))
        z, y, x = ((ax[d][box[d]] - pos[d]) ** 2 for d in (2, 1, 0))
        f = torch.sqrt(z[:, None, None] + y[None, :, None] + x[None, None, :]) / dr
        i = f.long()
        inside = (i <= last).double()
        i.clamp_(max=last)
        w = f - i
        at = (box[2], box[1], box[0])
        v[at] += inside * ((1 - w) * tab[ty][i] + w * tab[ty][i + 1])
        g = inside * rho[at]
        i = i.reshape(-1)
        dtab[ty] += torch.bincount(i, (g * (1 - w)).reshape(-1), len(r)) \
            + torch.bincount(i + 1, (g * w).reshape(-1), len(r))
    return dict(v=v.reshape(-1), dtab=dtab)


def _plane_waves(cell, max_ke):
    """Plane waves with |G|^2 / 2 < max_ke among the indices the fit program scans."""
    b = 2 * math.pi * np.linalg.inv(cell).T
    m = int(math.sqrt(max_ke) / np.linalg.norm(b, axis=1).min()) + 1
    n = np.arange(-m, m + 1)
    ijk = np.array(np.meshgrid(n, n, n, indexing="ij")).reshape(3, -1).T
    g = ijk @ b
    return g[(g * g).sum(1) / 2 < max_ke]


def _exact_bulk(case, seed):
    p = _bulk_inputs(case, seed)
    g = torch.tensor(_plane_waves(p["cell"], case["max_ke"]), device="cuda")
    d = g[:, None, :] - g[None, :, :]
    q2 = (d * d).sum(-1)
    tau = torch.tensor(p["tau"], device="cuda")
    weight = torch.tensor(p["dl_de"], device="cuda")
    steps = []
    for theta in p["params"]:
        params = torch.tensor(theta, device="cuda", requires_grad=True)
        pot = 0
        for t, (r0, r1) in zip(params, (tau[:2], tau[2:])):
            ff = t[0] * (q2 - t[1]) / (t[2] * torch.exp(t[3] * q2) + 1.0)
            pot = pot + ff * (torch.exp(-1j * (d @ r0)) + torch.exp(-1j * (d @ r1))) / len(tau)
        bands = []
        for k in torch.tensor(p["kpts"], device="cuda"):
            kin = 0.5 * ((g + k) ** 2).sum(-1)
            bands.append(EV * torch.linalg.eigvalsh(pot + torch.diag(kin))[:case["ne"]])
        bands = torch.stack(bands)
        (bands * weight).sum().backward()
        steps.append(dict(bands=bands, grad=params.grad))
    return steps


def _exact_spinor(case, seed):
    p = _spinor_inputs(case, seed)
    n, h = p["n"], p["h"]
    t = _kinetic((n, n, n), h, EKIN_SPINOR)
    x = torch.tensor(p["x"], device="cuda")
    lists = []
    c1 = 0.5 * math.sqrt(1.5 / math.pi)
    for pos, vs in zip(p["xyz"], p["vso"]):
        z, y, xx = torch.meshgrid(x - pos[2], x - pos[1], x - pos[0], indexing="ij")
        r2 = (z * z + y * y + xx * xx).reshape(-1)
        at = torch.nonzero(r2 < p["r2"])[:, 0]
        r2 = r2[at]
        r = torch.sqrt(r2)
        u = [c.reshape(-1)[at] / r for c in (xx, y, z)]
        ylm = torch.stack([-c1 * torch.complex(u[0], u[1]), math.sqrt(2) * c1 * u[2] + 0j,
                           c1 * torch.complex(u[0], -u[1])])  # m = 1, 0, -1
        vr = vs * torch.exp(-r2 / 0.49)
        k = (vr[:, None] + vr[None, :]) / (r2[:, None] + r2[None, :]) \
            * torch.exp(-0.5 * ((r[:, None] - r[None, :]) / h) ** 2)
        lists.append((at, ylm, k * (0.5 * h ** 3 / math.sqrt(2 * math.pi * h * h))))
    s2 = math.sqrt(2.0)

    def apply(psi):  # [ns, 2, N]
        grid = psi.reshape(-1, 2, n, n, n)
        out = _hamiltonian(grid, t, p["v"]).reshape(psi.shape)
        for at, (yp, y0, ym), k in lists:
            f = psi[:, :, at]
            sp, s0, sm = ((y.conj() * f) @ k.to(f.dtype) for y in (yp, y0, ym))
            up = yp * sp[:, 0] - ym * sm[:, 0] + s2 * (y0 * sp[:, 1] + ym * s0[:, 1])
            dn = -yp * sp[:, 1] - ym * sm[:, 1] + s2 * (y0 * sm[:, 0] + yp * s0[:, 0])
            out[:, 0, at] += up
            out[:, 1, at] += dn
        return out

    psi = torch.tensor(p["start"], device="cuda").reshape(case["ns"], 2, -1)
    dE_1 = 4.0 / p["dE"]
    acc = torch.zeros((case["ns"], case["ms"], 2, n ** 3), dtype=torch.complex128, device="cuda")
    for j in range(case["nc"]):
        if j:
            psi = dE_1 * apply(psi) - (2.0 + p["zn"][j - 1] + p["vmin"] * dE_1) * psi
        for e in range(case["ms"]):
            acc[:, e] += complex(p["an"][e, j]) * psi
    return acc.reshape(case["ns"], case["ms"], -1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "hpsi":
        dims = case["nx"], case["ny"], case["nz"]
        h = _spacing(min(dims))
        v = _potential(dims, h, seed)
        rng = np.random.default_rng(seed)
        shape = (case["ns"], v.numel())
        psi = rng.normal(size=shape) + 1j * rng.normal(size=shape)
        psi = torch.tensor(psi, device="cuda").reshape(-1, *v.shape)
        return _hamiltonian(psi, _kinetic(dims, h), v).reshape(shape).cpu().numpy()
    if kind in ("filter", "batch"):
        cells = [(case["nx"], case["ny"], case["nz"])] if kind == "filter" else \
            [(int(s),) * 3 for s in case["sizes"].split(",")]
        got = []
        for j, dims in enumerate(cells):
            p = _filter_inputs(dims, case["ns"], case["ms"], case["nc"], seed + 7 * j)
            r = dict(first=_exact_filter(p, min(2, case["ns"])))
            got.append(dict(r, rest=None) if case["ns"] > 2 else r)
        return got[0] if kind == "filter" else got
    if kind == "pipeline":
        return _exact_pipeline(case, seed)
    if kind == "gram":
        a, b = _gram_inputs(case, seed)
        return a @ (a if b is None else b).T
    if kind == "potential":
        return _exact_potential(case, seed)
    if kind == "bulk":
        return _exact_bulk(case, seed)
    return _exact_spinor(case, seed).cpu().numpy()
