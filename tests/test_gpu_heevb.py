"""The library's batched Hermitian solver of the lowest eigenpairs
(csrc/sep_heevb.cu: one CTA per matrix, Householder tridiagonalisation,
bisection, inverse iteration, back-transformation), which replaces one zheev
per k-point of the bulk fit (pseudopotFitting/diag.c:12-48, lowest bands
fit.c:86-88), against numpy's eigh (LAPACK).

Tolerances relative to the largest |eigenvalue| s: eigenvalues 1e-12 s,
residuals |A x - lambda x| <= 1e-11 s, orthonormality 1e-11, and for exactly
degenerate eigenvalues the projector onto the cluster's vectors 1e-9 from
LAPACK's.
"""
import numpy as np
import pytest

import semi_empirical_pseudopotentials_gb300 as sep

pytestmark = pytest.mark.gpu


def _random_hermitian(rng, n):
    x = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return 0.5 * (x + x.conj().T)


def _with_spectrum(rng, lam):
    n = len(lam)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    return (q * lam) @ q.conj().T


def _check(a, nw, w, v):
    ref_w, ref_v = np.linalg.eigh(a)
    s = np.abs(ref_w).max()
    assert np.abs(w - ref_w[:nw]).max() <= 1e-12 * s
    r = a @ v - v * w
    assert np.abs(r).max() <= 1e-11 * s
    g = v.conj().T @ v
    assert np.abs(g - np.eye(nw)).max() <= 1e-11
    # degenerate clusters: compare projectors
    i = 0
    while i < nw:
        j = i + 1
        while j < nw and ref_w[j] - ref_w[j - 1] <= 1e-9 * s:
            j += 1
        if j < len(ref_w) and ref_w[j] - ref_w[j - 1] <= 1e-9 * s:
            i = j  # cluster cut by nw: skip
            continue
        p_got = v[:, i:j] @ v[:, i:j].conj().T
        p_ref = ref_v[:, i:j] @ ref_v[:, i:j].conj().T
        assert np.abs(p_got - p_ref).max() <= 1e-9, (i, j)
        i = j


@pytest.mark.parametrize("n,nmat,nw", [(2, 3, 2), (33, 4, 10), (100, 5, 32), (200, 3, 64),
                                       (387, 6, 32), (512, 2, 24)])
def test_random_hermitian_lowest_eigenpairs(n, nmat, nw):
    rng = np.random.default_rng(n)
    a = np.stack([_random_hermitian(rng, n) for _ in range(nmat)])
    w, v = sep.hermitian_lowest(a, nw)
    for m in range(nmat):
        _check(a[m], nw, w[m], v[m])


def test_degenerate_spectra():
    """Clusters of exactly equal eigenvalues (as at high-symmetry k-points),
    one crossing the last wanted band."""
    rng = np.random.default_rng(11)
    n = 150
    lam = np.sort(rng.uniform(-3, 3, n))
    lam[3:6] = lam[3]          # triple
    lam[10:12] = lam[10]       # pair
    lam[20:26] = lam[20]       # six
    lam[30:34] = lam[30]       # crosses nw = 32
    lam = np.sort(lam)
    a = np.stack([_with_spectrum(rng, lam) for _ in range(3)])
    w, v = sep.hermitian_lowest(a, 32)
    for m in range(3):
        _check(a[m], 32, w[m], v[m])


def test_eigenvalues_only_and_diagonal_input():
    rng = np.random.default_rng(5)
    a = np.stack([_random_hermitian(rng, 80), np.diag(np.arange(80.0)[::-1]).astype(complex)])
    w, v = sep.hermitian_lowest(a, 16, vectors=False)
    assert v is None
    for m in range(2):
        ref = np.linalg.eigvalsh(a[m])[:16]
        assert np.abs(w[m] - ref).max() <= 1e-12 * np.abs(np.linalg.eigvalsh(a[m])).max()


def test_bad_arguments():
    with pytest.raises(sep.SepError):
        sep.hermitian_lowest(np.eye(600, dtype=complex), 4)
    with pytest.raises(sep.SepError):
        sep.hermitian_lowest(np.eye(10, dtype=complex), 11)


@pytest.mark.parametrize("n,nmat", [(2, 1), (5, 3), (33, 1), (64, 2), (129, 1), (129, 40),
                                    (200, 80), (257, 5), (512, 1)])
def test_cluster_sizes(n, nmat):
    """The reduction takes 1 to 8 blocks per matrix by n and nmat: eigenvalues
    within 1e-12 of the largest and residuals within 1e-11, the bounds of the
    tests above, where most warps of a cluster have no column, at a single
    large matrix and with more matrices than clusters of two fit.  A third of
    each matrix's rows is diagonal, so steps without a reflector occur."""
    rng = np.random.default_rng(n + nmat)
    a = rng.normal(size=(nmat, n, n)) + 1j * rng.normal(size=(nmat, n, n))
    a = a + np.conj(np.transpose(a, (0, 2, 1)))
    k = n // 3
    diag = np.diagonal(a, axis1=1, axis2=2).copy()
    a[:, :k, :] = 0.0
    a[:, :, :k] = 0.0
    a[:, np.arange(n), np.arange(n)] = diag
    nw = min(n, 8)
    w, v = sep.hermitian_lowest(a, nw)
    for m in range(nmat):
        ref = np.linalg.eigvalsh(a[m])
        scale = np.abs(ref).max()
        assert np.abs(w[m] - ref[:nw]).max() <= 1e-12 * scale
        r = a[m] @ v[m] - v[m] * w[m]
        assert np.abs(r).max() <= 1e-11 * scale


@pytest.mark.parametrize("n,nw", [(2, 2), (3, 2), (31, 31), (32, 32), (33, 33), (65, 64),
                                  (300, 64), (512, 64)])
def test_inverse_iteration_groups(n, nw):
    """One matrix with all wanted eigenvalues in one group (1e-6 apart: their
    vectors are orthogonalised against each other), one with none in a group
    (apart by more than 1e-3 of the norm, as far as nw allows) and one of both,
    at sizes around a warp and the largest; bounds of the tests above."""
    rng = np.random.default_rng(1000 + n)
    far = np.linspace(-1.0, 1.0, n)
    close = np.where(np.arange(n) < nw, -1.0 + 1e-6 * np.arange(n), np.linspace(0.5, 1.0, n))
    mixed = np.sort(np.where(np.arange(n) % 3 == 0, far, np.roll(far, 1) + 1e-5))
    a = np.stack([_with_spectrum(rng, lam) for lam in (close, far, mixed)])
    w, v = sep.hermitian_lowest(a, nw)
    for m in range(3):
        _check(a[m], nw, w[m], v[m])


@pytest.mark.parametrize("nmat,nw", [(1, 1), (38, 64), (39, 64), (607, 4), (609, 4)])
def test_multisection_point_counts(nmat, nw):
    """16 or 4 points per round, by the number of eigenvalues wanted in all
    (2,432 is the last that takes 16), against LAPACK to the bound above; a
    matrix with a zero off-diagonal and equal eigenvalues among them."""
    n = 66
    rng = np.random.default_rng(nmat)
    a = np.stack([_random_hermitian(rng, n) for _ in range(nmat)])
    a[0] = np.diag(np.repeat([-2.0, 0.0, 1e-300, 3.0, 5.0, 5.5], n // 6)).astype(complex)
    w, _ = sep.hermitian_lowest(a, nw, vectors=False)
    ref = np.linalg.eigvalsh(a)
    assert np.abs(w - ref[:, :nw]).max() <= 1e-12 * np.abs(ref).max()
