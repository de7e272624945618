"""The spinor filter program on the GPU (sep_spinor_*, through the C ABI):
the spinor Hamiltonian, the Newton filter with complex coefficients, the
energy range and the whole program against the reference's own routines
(tests/golden/spinor_vso.npz, made by tests/golden/make_spinor_fixture.py
from spinors/filterSpinors/*.c) and against the oracle on a larger case.

Tolerances: H psi and the filter output as the CPU oracle's pins (samples
to 1e-12 of the largest, row sums and sums of squares to 1e-11); Vmin and
dE to 1e-9; the kept count exactly; Ritz values to 1e-9 (relative) and
sigma to 1e-7 (relative)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from oracle import spinor_oracle as so
from semi_empirical_pseudopotentials_gb300 import binding, spinor

pytestmark = pytest.mark.gpu

EKINMAX = 20.0  # filterSpinors/init.c:23


def load(golden):
    g = golden("spinor_vso.npz")
    raw = g["nlc"]
    return g, raw.reshape(-1).view(so.NLC_DTYPE).reshape(raw.shape[:2])


def check_sampled(g, name, got):
    got = np.asarray(got).reshape(-1, 2 * int(np.prod(g["dims"])))
    ref = g[name + "_sample"].reshape(got.shape[0], -1)
    scale = np.abs(ref).max()
    assert np.abs(got[:, g["sample_idx"]] - ref).max() <= 1e-12 * scale
    assert np.allclose(got.sum(axis=1), g[name + "_sum"], rtol=1e-11, atol=1e-12 * scale)
    assert np.allclose((np.abs(got) ** 2).sum(axis=1), g[name + "_sumsq"], rtol=1e-11, atol=0)


def path(g, nlc, form="gauss"):
    dims = tuple(int(v) for v in g["dims"])
    h = float(g["h"])
    ctx = binding.Context(dims, (h, h, h), potl=g["potl"], ekinmax=EKINMAX)
    assert np.array_equal(ctx_ksqr(ctx), g["ksqr"])
    if form == "gauss":
        return ctx, spinor.SpinorPath(ctx, nlc, g["nl"], sigma=h)
    return ctx, spinor.SpinorPath(ctx, nlc, g["nl"], elkb=g["elkb"])


def ctx_ksqr(ctx):
    import ctypes as C

    out = np.empty(ctx.ngrid)
    L = binding.lib()
    L.sep_ctx_ksqr.argtypes = [C.c_void_p, C.c_void_p]
    binding._check(L.sep_ctx_ksqr(ctx.h, out.ctypes.data))
    return out


@pytest.mark.parametrize("form", ["gauss", "kb"])
def test_spinor_hamiltonian_matches_reference(golden, form):
    g, nlc = load(golden)
    ctx, sp = path(g, nlc, form)
    check_sampled(g, "h_" + form, sp.hamiltonian(g["psi"]))


def test_spinor_newton_filter_matches_reference(golden):
    g, nlc = load(golden)
    ctx, sp = path(g, nlc)
    got = sp.filter(g["psi"][None, :], g["an"], g["zn"], float(g["dE_1"]), float(g["vmin"]))
    check_sampled(g, "filter_out", got[0])


def test_spinor_energy_range_matches_reference(golden):
    g, nlc = load(golden)
    ctx, sp = path(g, nlc)
    vmin, dE, _ = sp.energy_range()
    assert abs(vmin - float(g["run_vmin"])) <= 1e-9 * abs(float(g["run_vmin"]))
    assert abs(dE - float(g["run_dE"])) <= 1e-9 * float(g["run_dE"])


def test_spinor_pipeline_matches_reference_program(golden):
    """The reference's whole spinor program (energy range, coefficients,
    start spinors from its seed, filtering, portho, Hmat, sigma)."""
    g, nlc = load(golden)
    ctx, sp = path(g, nlc)
    n = ctx.ngrid
    ns = int(g["run_ns"])
    st = O.start_states(int(g["run_seed"]), 2 * ns, n, ctx.dv)
    spinors = np.stack([np.concatenate([st[2 * j], st[2 * j + 1]]) for j in range(ns)])
    res = sp.pipeline(spinors.astype(np.complex128), g["run_el"], int(g["run_nc"]))
    assert res["mkept"] == int(g["run_mkept"])
    assert abs(res["timing"]["dE"] - float(g["run_dE"])) <= 1e-9 * float(g["run_dE"])
    assert np.allclose(res["eval"], g["run_eval"], rtol=1e-9, atol=1e-12)
    assert np.allclose(res["sigma"], g["run_sigma"], rtol=1e-7, atol=1e-10)


def larger_case(seed=11, n=32, h=0.6, natom=12):
    rng = np.random.default_rng(seed)
    v = -0.5 * n * h + h * np.arange(n)
    rxyz = rng.uniform(-5.0, 5.0, size=(natom, 3))
    nlc, nl = so.neighbour_lists(v, v, v, rxyz, rng.uniform(-0.15, 0.15, natom),
                                 0.49 * 6.0 * np.log(10.0), 1200)
    zz, yy, xx = np.meshgrid(v, v, v, indexing="ij")
    pot = np.zeros(n ** 3)
    for a in range(natom):
        d2 = (xx - rxyz[a, 0]) ** 2 + (yy - rxyz[a, 1]) ** 2 + (zz - rxyz[a, 2]) ** 2
        pot -= 0.5 * np.exp(-0.4 * d2).ravel()
    return (n, n, n), h, nlc, nl, pot


def test_spinor_filter_against_oracle_on_a_larger_case():
    """32^3 grid, 12 atoms, 3 start spinors x 3 complex targets over 40
    Newton steps against the oracle's newton_filter."""
    dims, h, nlc, nl, pot = larger_case()
    ctx = binding.Context(dims, (h, h, h), potl=pot, ekinmax=EKINMAX)
    sp = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
    n = ctx.ngrid
    rng = np.random.default_rng(4)
    start = rng.normal(size=(3, 2 * n)) + 1j * rng.normal(size=(3, 2 * n))
    nc = 40
    an = rng.normal(size=(3, nc)) + 1j * rng.normal(size=(3, nc))
    an /= np.arange(1, nc + 1) ** 2
    zn = rng.uniform(-2.0, 2.0, nc)
    dE_1, vmin = 4.0 / 30.0, float(pot.min())
    got = sp.filter(start, an, zn, dE_1, vmin)
    ks = ctx_ksqr(ctx)
    for s in range(3):
        ref = so.newton_filter(start[s], an, zn, dE_1, vmin, pot, ks, dims, nlc, nl, h, h ** 3)
        assert np.abs(got[s] - ref).max() <= 1e-11 * np.abs(ref).max(), s


def test_spinor_pipeline_library_eigensolver_matches_cusolver():
    """The whole spinor program on the 32^3 case with the library's solver
    (on the real embedding of each Hermitian problem) and with cuSOLVER's
    Zheevd: the same kept count, Ritz values to 1e-10 and sigma to 1e-8."""
    dims, h, nlc, nl, pot = larger_case()
    out = {}
    for mode in (1, 0):
        ctx = binding.Context(dims, (h, h, h), potl=pot, ekinmax=EKINMAX)
        ctx.set_eigensolver(mode)
        sp = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
        n = ctx.ngrid
        st = O.start_states(-4242, 8, n, ctx.dv)
        spinors = np.stack([np.concatenate([st[2 * j], st[2 * j + 1]]) for j in range(4)])
        out[mode] = sp.pipeline(spinors.astype(np.complex128), [-0.8, -0.6, -0.4], 64)
        ctx.close()
    assert out[0]["mkept"] == out[1]["mkept"]
    assert np.abs(out[0]["eval"] - out[1]["eval"]).max() <= 1e-10
    assert np.abs(out[0]["sigma"] - out[1]["sigma"]).max() <= 1e-8


def test_spinor_pipeline_repeats():
    """The kept kernel's contributions are summed in list order, whatever order
    the blocks finish in, so H of the same spinors is the same to the bit, and
    the Ritz values of the same start spinors agree as the two solvers do
    above.  41 points of this case lie in the lists of three atoms, where the
    order of two additions shows."""
    dims, h, nlc, nl, pot = larger_case()
    points = np.concatenate([nlc["jxyz"][a, :nl[a]] for a in range(len(nl))])
    assert (np.bincount(points) >= 3).sum() == 41
    st = O.start_states(-4242, 8, int(np.prod(dims)), h ** 3)
    spinors = np.stack([np.concatenate([st[2 * j], st[2 * j + 1]]) for j in range(4)])
    ctx = binding.Context(dims, (h, h, h), potl=pot, ekinmax=EKINMAX)
    ctx.set_eigensolver(1)
    sp = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
    first = sp.hamiltonian(spinors.astype(np.complex128))
    assert all(np.array_equal(sp.hamiltonian(spinors.astype(np.complex128)), first)
               for _ in range(50))
    runs = [sp.pipeline(spinors.astype(np.complex128), [-0.8, -0.6, -0.4], 64) for _ in range(24)]
    ctx.close()
    for r in runs[1:]:
        assert r["mkept"] == runs[0]["mkept"]
        assert np.abs(r["eval"] - runs[0]["eval"]).max() <= 1e-10


def _list_entries(rng, n, ngrid):
    """n neighbour-list entries at random grid points, radii spread over (0.1, 2.6)."""
    e = np.zeros(n, dtype=spinor.NLC_DTYPE)
    e["jxyz"] = rng.choice(ngrid, n, replace=False)
    for f in ("y10", "y11", "y1_1"):
        e[f] = rng.normal(size=n) + 1j * rng.normal(size=n)
    e["r"] = rng.uniform(0.1, 2.6, n)
    e["r2"] = e["r"] ** 2
    e["Vr"] = 0.1 * np.exp(-e["r2"] / 0.49)
    return e


@pytest.mark.parametrize("counts", [(1, 31, 32, 33, 0), (63, 64, 65, 128), (200, 3, 129),
                                    (4096,) + (1,) * 299])
def test_kept_kernel_equals_the_operator_applied_alone(counts):
    """A context keeps the Gaussian form's K(j1, j2); sep_spinor_vso forms it in
    place.  H with the operator less H without it is Vso psi: both take the same
    products in the same order per atom, atoms add in any order, and H rounds
    the sum once more (tolerance 1e-13 of the largest value of H psi).  Lists
    around the 32- and 64-point tiles, an empty one, and one so long that the
    atoms' K (40 GB) would take more than an eighth of the device's memory and
    is not kept."""
    rng = np.random.default_rng(sum(counts))
    dims, h = (32, 32, 40), 0.5
    ngrid = int(np.prod(dims))
    nlc = np.zeros((len(counts), max(counts)), dtype=spinor.NLC_DTYPE)
    for a, n in enumerate(counts):
        nlc[a, :n] = _list_entries(rng, n, ngrid)
    nl = np.array(counts, dtype=np.int64)
    psi = rng.normal(size=(3, 2 * ngrid)) + 1j * rng.normal(size=(3, 2 * ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), precision="f64", ekinmax=20.0)
    full = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    bare = spinor.SpinorPath(ctx, nlc, np.zeros_like(nl), sigma=h).hamiltonian(psi)
    again = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    ctx.close()
    for s in range(3):
        ref = spinor.nonlocal_potential(psi[s], nlc, nl, h, h ** 3)
        assert np.abs(ref).max() > 0.0
        for got in (full, again):
            assert np.abs(got[s] - bare[s] - ref).max() <= 1e-13 * np.abs(full[s]).max()


@pytest.mark.parametrize("counts,nsp", [((64, 5, 0, 63), 1), ((129, 128), 45), ((681, 40), 2),
                                        ((700,), 1)])
def test_operator_on_the_tensor_cores(counts, nsp):
    """Lists of 64 points on take the digit-split contraction: against the
    operator applied alone (FP64 FMAs) to 1e-13 of the largest value of H psi
    (a term is good to 2^-53 of its row's largest K and its product's largest
    value, and 700 of them add up), as with the contraction switched off; over
    more spinors than one chunk takes (42), above 680 points, where products
    are formed twice, and around a tile of 128 rows."""
    rng = np.random.default_rng(sum(counts) + nsp)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    nlc = np.zeros((len(counts), max(counts)), dtype=spinor.NLC_DTYPE)
    for a, n in enumerate(counts):
        nlc[a, :n] = _list_entries(rng, n, ngrid)
    nl = np.array(counts, dtype=np.int64)
    psi = rng.normal(size=(nsp, 2 * ngrid)) + 1j * rng.normal(size=(nsp, 2 * ngrid))
    psi[:, :ngrid] *= np.logspace(-9, 0, ngrid)  # products of many magnitudes in a list
    out = {}
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), precision="f64", ekinmax=20.0)
    for tc in (1, 0):
        ctx.set_subspace("tc" if tc else "f64")
        out[tc] = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    bare = spinor.SpinorPath(ctx, nlc, np.zeros_like(nl), sigma=h).hamiltonian(psi)
    ctx.close()
    for s in range(nsp):
        ref = spinor.nonlocal_potential(psi[s], nlc, nl, h, h ** 3)
        for tc in (1, 0):
            assert np.abs(out[tc][s] - bare[s] - ref).max() <= 1e-13 * np.abs(out[0][s]).max()


def test_operator_with_values_that_are_not_finite():
    """A list point at its atom (r = 0) makes K infinite there: the sums stay
    with the FP64 kernel, and the same points are not finite as with the
    operator applied alone."""
    rng = np.random.default_rng(5)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    nlc = np.zeros((2, 100), dtype=spinor.NLC_DTYPE)
    for a in range(2):
        nlc[a] = _list_entries(rng, 100, ngrid)
    nlc["r"][1, 7] = nlc["r2"][1, 7] = 0.0
    nl = np.array([100, 100], dtype=np.int64)
    psi = rng.normal(size=(1, 2 * ngrid)) + 1j * rng.normal(size=(1, 2 * ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), precision="f64", ekinmax=20.0)
    got = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    ctx.close()
    ref = spinor.nonlocal_potential(psi[0], nlc, nl, h, h ** 3)
    assert not np.isfinite(ref).all()
    assert np.array_equal(np.isfinite(got[0]), np.isfinite(ref))


def _set_operator_of(ctx, nnlc, entries):
    """sep_spinor_set_operator for one atom with the given entries in a list that
    claims room for nnlc; returns the status."""
    nlc = np.ascontiguousarray(entries, dtype=spinor.NLC_DTYPE)
    nl = np.array([len(nlc)], dtype=np.int64)
    f = binding.lib().sep_spinor_set_operator
    f.argtypes = [C.c_void_p, C.c_long, C.c_long, C.c_void_p, C.c_void_p, C.c_double, C.c_int,
                  C.c_void_p]
    return f(ctx.h, 1, nnlc, nlc.ctypes.data, nl.ctypes.data, 0.5, 0, None)


def test_call_after_one_that_ran_out_of_memory():
    """A list with room for 2^34 entries (1.8 TB) cannot be allocated: the call
    says so, and the next call, which needs nothing of it, succeeds."""
    rng = np.random.default_rng(8)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    psi = rng.normal(size=(1, ngrid)) + 1j * rng.normal(size=(1, ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=rng.normal(size=ngrid), ekinmax=20.0)
    before = ctx.hamiltonian(psi)
    assert _set_operator_of(ctx, 2 ** 34, _list_entries(rng, 10, ngrid)) == -3  # SEP_ERR_NOMEM
    after = ctx.hamiltonian(psi)
    ctx.close()
    assert np.array_equal(after, before)


def test_operator_that_could_not_be_set():
    """A set call that fails after its arguments were checked has begun to take
    over the buffers of the operator before it: the context has no operator then
    (every spinor call says so), and takes a new one as a fresh context does.  One
    that is refused for its arguments leaves the operator as it was."""
    rng = np.random.default_rng(9)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    nlc = np.stack([_list_entries(rng, 90, ngrid) for _ in range(3)])
    nl = np.array([90, 70, 5], dtype=np.int64)
    psi = rng.normal(size=(2, 2 * ngrid)) + 1j * rng.normal(size=(2, 2 * ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=rng.normal(size=ngrid), ekinmax=20.0)
    path = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
    first = path.hamiltonian(psi)
    bad = nlc.copy()
    bad["jxyz"][0, 0] = ngrid
    with pytest.raises(binding.SepError, match="outside the grid"):
        spinor.SpinorPath(ctx, bad, nl, sigma=h)
    assert np.array_equal(path.hamiltonian(psi), first)
    assert _set_operator_of(ctx, 2 ** 34, _list_entries(rng, 10, ngrid)) == -3  # SEP_ERR_NOMEM
    for call in (lambda: path.hamiltonian(psi), path.energy_range,
                 lambda: path.filter(psi, np.ones((1, 2)), np.zeros(2), 0.1, -1.0),
                 lambda: path.pipeline(psi, [-0.5], 8)):
        with pytest.raises(binding.SepError, match="no spin-orbit operator set"):
            call()
    again = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    ctx.close()
    assert np.array_equal(again, first)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, complex(0.0, np.inf)])
def test_states_with_values_that_are_not_finite(bad):
    """One value of a spinor's up grid, a point of the first atom's list, is not
    finite: the other component is not finite on that list, through the operator
    alone, exactly where it is with the operator applied by itself, and has its
    values elsewhere; the other spinors of the call do not notice."""
    rng = np.random.default_rng(6)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    points = rng.permutation(ngrid)
    nlc = np.stack([_list_entries(rng, 150, ngrid) for _ in range(2)])
    nlc["jxyz"] = points[:300].reshape(2, 150)
    nl = np.array([150, 100], dtype=np.int64)
    psi = rng.normal(size=(3, 2 * ngrid)) + 1j * rng.normal(size=(3, 2 * ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), precision="f64", ekinmax=20.0)
    path = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
    clean = path.hamiltonian(psi)
    psi[1, nlc["jxyz"][0, 70]] = bad
    got = path.hamiltonian(psi)
    ctx.close()
    ref = spinor.nonlocal_potential(psi[1], nlc, nl, h, h ** 3)
    lost = ~np.isfinite(ref[ngrid:])
    assert lost.sum() == 150
    assert np.array_equal(~np.isfinite(got[1, ngrid:]), lost)
    assert np.array_equal(got[1, ngrid:][~lost], clean[1, ngrid:][~lost])
    assert np.array_equal(got[[0, 2]], clean[[0, 2]])


def _list_states(rng, kind, r, ngrid, points):
    """A spinor over the grid whose values on a list's points (radii r) are normal,
    constant, falling by nine or three decades towards or away from the atom,
    zero on the inner half, or of random magnitude."""
    psi = rng.normal(size=2 * ngrid) + 1j * rng.normal(size=2 * ngrid)
    out = r / r.max()
    f = {"normal": np.ones_like(r), "smooth": None, "towards9": 10.0 ** (9 * (out - 1)),
         "towards3": 10.0 ** (3 * (out - 1)), "away9": 10.0 ** (-9 * out),
         "node": np.where(out < 0.5, 0.0, 1.0), "any9": 10.0 ** rng.uniform(-9, 0, len(r))}[kind]
    for c in range(2):
        at = c * ngrid + points
        psi[at] = (1.0 + 0.3j) * (1 - 2 * c) if f is None else psi[at] * f
    return psi


def _row_errors(got, e, k, psi, ngrid, sigma, dv, held=None):
    """Per list point: the error of Vso psi against extended precision over the sum
    of the absolute values of what it adds up.  held: K's rows and the products
    rounded to that many bits below their largest, and summed exactly, instead."""
    LD = np.longdouble
    j, n = e["jxyz"], len(e)
    tmp = 0.5 / np.sqrt(2 * np.pi * sigma ** 2) * dv
    y = [e[f] for f in ("y11", "y10", "y1_1")]
    kl = k.astype(LD)
    if held:
        unit = np.ldexp(LD(1), np.frexp(k.max(1))[1] - held)
        kl = np.rint(kl / unit[:, None]) * unit[:, None]
    s, a = {}, {}
    for c in range(2):
        p = psi[c * ngrid + j]
        for m in range(3):
            yr, yi, pr, pi = (v.astype(LD) for v in (y[m].real, y[m].imag, p.real, p.imag))
            x = [yr * pr + yi * pi, yr * pi - yi * pr]
            a[m, c] = kl @ (np.abs(yr * pr) + np.abs(yi * pi) + np.abs(yr * pi) + np.abs(yi * pr))
            if held:
                for q in range(2):
                    u = np.ldexp(LD(1), int(np.frexp(np.abs(x[q]).max())[1]) - held)
                    x[q] = np.rint(x[q] / u) * u
            s[m, c] = [kl @ v for v in x]
    w = {(0, 0): [(0, (0, 0), 1), (2, (2, 0), -1), (1, (0, 1), 2 ** 0.5), (2, (1, 1), 2 ** 0.5)],
         (1, 0): [(0, (0, 1), -1), (2, (2, 1), -1), (1, (2, 0), 2 ** 0.5), (0, (1, 0), 2 ** 0.5)]}
    err, size = np.zeros(n, LD), np.zeros(n, LD)
    for (c, _), terms in w.items():
        re, im = np.zeros(n, LD), np.zeros(n, LD)
        for m, at, f in terms:
            yr, yi = y[m].real.astype(LD), y[m].imag.astype(LD)
            sr, si = s[at]
            g = LD(np.sqrt(LD(2))) if abs(f) > 1 else LD(f)
            re += g * tmp * (yr * sr - yi * si)
            im += g * tmp * (yr * si + yi * sr)
            size += abs(g) * tmp * (np.abs(yr) + np.abs(yi)) * a[at]
        if held:
            return re, im, size
        v = got[c * ngrid + j]
        err = np.maximum(err, np.maximum(np.abs(v.real - re), np.abs(v.imag - im)))
    return (err / size).astype(float)


@pytest.mark.parametrize("at,rc,take", [((0.13, -0.2, 0.07), 2.6, None), ((0.005, 0.0, 0.0), 2.6, None),
                                        ((0.0, 0.0, 0.0), 2.6, None), ((0.2, 0.2, 0.1), 3.0, 672),
                                        ((0.2, 0.2, 0.1), 3.0, 673), ((0.1, 0.2, 0.25), 1.4, None)])
def test_tensor_core_sums_are_as_accurate_as_the_fp64_ones(at, rc, take):
    """Vso psi of one atom (no potential, no kinetic energy to speak of) against
    extended precision, point by point, relative to the sum of the absolute
    values added up there: on the tensor cores it errs no more than by FP64 FMAs
    (root mean square over the points, a tenth for chance where nearly every row
    takes the FP64 sums; half as much again for the worst point).
    Atoms between grid points, near one and on one; lists of 92 to 673 points;
    states that are steep towards the atom, where K is largest and a split that
    is relative to the list's largest value alone loses their digits."""
    rng = np.random.default_rng(11)
    dims, h = (20, 20, 20), 0.5
    ngrid = int(np.prod(dims))
    ax = [(np.arange(d) - d // 2) * h for d in dims]
    nlc, nl = spinor.neighbour_lists(*ax, [at], [0.1], rc ** 2)
    nl = np.minimum(nl, take or nl)
    e = nlc[0, :nl[0]]
    assert len(e) == (take or len(e)) and len(e) >= 64
    r = np.where(e["r2"] > 1e10, 0.0, e["r"])
    k = (0.5 * (e["Vr"][:, None] + e["Vr"]) * np.exp(-((e["r"][:, None] - e["r"]) / h) ** 2 / 2)
         / (0.5 * (e["r2"][:, None] + e["r2"])))
    kinds = ["normal", "smooth", "towards9", "towards3", "away9", "node", "any9"]
    psi = np.stack([_list_states(rng, q, r, ngrid, e["jxyz"]) for q in kinds])
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), ekinmax=1e-200)
    out = {}
    for route in ("tc", "f64"):
        ctx.set_subspace(route)
        out[route] = spinor.SpinorPath(ctx, nlc, nl, sigma=h).hamiltonian(psi)
    ctx.close()
    for q in range(len(kinds)):
        err = {t: _row_errors(out[t][q], e, k, psi[q], ngrid, h, h ** 3) for t in out}
        rms = {t: np.sqrt((v ** 2).mean()) for t, v in err.items()}
        assert rms["tc"] <= 1.1 * rms["f64"]
        assert err["tc"].max() <= 1.5 * err["f64"].max()
        assert err["f64"].max() <= (len(e) + 20) * 2.0 ** -53
    # the comparison sees a digit less in each value
    re, im, size = _row_errors(None, e, k, psi[0], ngrid, h, h ** 3, held=47)
    full = _row_errors(None, e, k, psi[0], ngrid, h, h ** 3, held=63)
    lost = np.maximum(np.abs(re - full[0]), np.abs(im - full[1])) / size
    err = _row_errors(out["f64"][0], e, k, psi[0], ngrid, h, h ** 3)
    assert np.sqrt((lost ** 2).mean()) > np.sqrt((err ** 2).mean())


def test_one_long_list_among_many_short_ones():
    """The contraction takes every list as long as the longest, so an operator with
    one long list among a thousand short ones stays with the FP64 sums: the same
    bits with the tensor cores switched on and off, where lists that are all long
    differ in the last ones."""
    rng = np.random.default_rng(12)
    dims, h = (16, 16, 20), 0.5
    ngrid = int(np.prod(dims))
    psi = rng.normal(size=(2, 2 * ngrid)) + 1j * rng.normal(size=(2, 2 * ngrid))
    ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), ekinmax=20.0)
    for counts, same in (((300,) + (5,) * 999, True), ((300,) * 20, False)):
        nlc = np.zeros((len(counts), 300), dtype=spinor.NLC_DTYPE)
        for a, n in enumerate(counts):
            nlc[a, :n] = _list_entries(rng, n, ngrid)
        path = spinor.SpinorPath(ctx, nlc, np.array(counts, dtype=np.int64), sigma=h)
        out = []
        for route in ("tc", "f64"):
            ctx.set_subspace(route)
            out.append(path.hamiltonian(psi))
        assert np.array_equal(*out) == same
        assert np.abs(out[0] - out[1]).max() <= 1e-13 * np.abs(out[0]).max()
    ctx.close()


@pytest.mark.parametrize("call", ["filter", "hamiltonian"])
def test_operator_gives_its_kept_memory_back(call):
    """An operator of 8 lists of 2048 points keeps 1 GB (K, its digits, their
    workspace).  With 200 MB of the device left, a filter whose history needs 190
    MB of them per spinor (of which it takes 0.6) and an apply to 250 spinors (1.0
    GB) run all the same: the operator gives that memory back and forms K on each
    apply.  Same values as with room to spare, to the tolerance of the operator's
    other tests."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(13)
    dims, h = (32, 32, 40), 0.5
    ngrid = int(np.prod(dims))
    nlc = np.stack([_list_entries(rng, 2048, ngrid) for _ in range(8)])
    nl = np.full(8, 2048, dtype=np.int64)
    ns = 2 if call == "filter" else 250
    psi = rng.normal(size=(ns, 2 * ngrid)) + 1j * rng.normal(size=(ns, 2 * ngrid))

    def run(path):
        if call == "hamiltonian":
            return path.hamiltonian(psi)
        return path.filter(psi, np.eye(8, 130) + 0j, np.zeros(130), 1e-4, -1.0)

    out = []
    torch.cuda.empty_cache()
    for left in (None, 200 << 20):
        ctx = binding.Context(dims, (h, h, h), potl=np.zeros(ngrid), precision="f64", ekinmax=20.0)
        ctx.set_block_steps(128 if call == "filter" else 32)
        before = torch.cuda.mem_get_info()[0]
        path = spinor.SpinorPath(ctx, nlc, nl, sigma=h)
        assert before - torch.cuda.mem_get_info()[0] > 800 << 20
        hog = []
        try:
            while left and torch.cuda.mem_get_info()[0] > left + (64 << 20):
                room = torch.cuda.mem_get_info()[0] - left
                hog.append(torch.empty(min(room, 16 << 30), dtype=torch.uint8, device="cuda"))
            out.append(run(path))
        finally:
            hog.clear()
            torch.cuda.empty_cache()
            ctx.close()
    for s in range(ns):
        assert np.abs(out[1][s] - out[0][s]).max() <= 1e-13 * np.abs(out[0][s]).max()
