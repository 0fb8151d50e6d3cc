"""The eigensolver's Rayleigh–Ritz kernel by itself (``omb_rayleigh_ritz``) on matrices that an
ordinary solve seldom forms, and the solves whose projected matrices are not finite.

Tolerances: with κ the condition number of the scaled G, the inverse Cholesky factor carries
≈ n·ε₆₄·κ; κ ≤ 100 and n ≤ 36 give 4e-13, so CᴴGC − 1 and the residual of the wanted pairs
(relative to ‖S‖) are held to 1e-12."""

from __future__ import annotations

import numpy as np
import pytest

from conftest import P_WG, gaussian_epsinv

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (2, 1), (6, 2), (9, 3), (15, 5), (16, 6), (17, 6), (32, 11), (33, 11), (36, 12)]


@pytest.fixture(scope="module")
def omb():
    import omb200
    return omb200


def hermitian(rng, lam):
    n = len(lam)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    a = (q * lam) @ q.conj().T
    return 0.5 * (a + a.conj().T)


def check(G, S, m, got, tol=1e-12):
    lam, C, rank = got
    assert rank == len(G)
    assert np.all(np.diff(lam) >= 0)
    assert np.max(np.abs(C.conj().T @ G @ C - np.eye(m))) < tol
    assert np.linalg.norm(S @ C - (G @ C) * lam) < tol * np.linalg.norm(S)


@pytest.mark.parametrize("n,m", SIZES)
def test_non_finite_projections_have_an_order(omb, n, m):
    """A NaN or an infinity in S, on the Cholesky path and on the one for near-dependent directions:
    the call returns (its Ritz values not finite, or the entries that the bad one does not reach),
    and the next call on good matrices is right."""
    from omb200.ops import rayleigh_ritz
    rng = np.random.default_rng(n)
    G = hermitian(rng, np.linspace(1, 10, n))
    S = hermitian(rng, np.linspace(0.3, 30, n))
    Gd = G.copy()  # two almost equal directions: SVQB drops one
    if n > 2 * m:
        Gd[:, -1], Gd[-1, :] = Gd[:, 0], Gd[0, :]
        Gd[-1, -1] = Gd[0, 0]
        Gd[0, -1] = Gd[-1, 0] = Gd[0, 0]
    for bad in (np.nan, np.inf, -np.inf, complex(1.0, np.nan)):
        for at in ((0, 0), (0, n - 1), (n - 1, n - 1)):
            T = S.copy()
            T[at] = T[at[::-1]] = bad
            if at[0] == at[1]:
                T[at] = np.real(bad) if not np.isnan(bad) else np.nan
            for g in (G, Gd):
                lam, C, rank = rayleigh_ritz(g, T, m)
                assert m <= rank <= n and lam.shape == (m,) and C.shape == (n, m)
    lam, _, _ = rayleigh_ritz(G, np.full((n, n), np.nan), m)
    assert np.all(np.isnan(lam))
    check(G, S, m, rayleigh_ritz(G, S, m))


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("n,m", SIZES)
def test_pairs_of_graded_matrices(omb, n, m, prec):
    """Well-separated pairs, the refinement's ordinary case: eigenvalues from 0.3 to 300, G of condition
    number 100.  (The FP32 tolerances stop the refinement earlier: at |E| ≤ 1e-6, so errors of ≈1e-12·n.)"""
    from omb200.ops import rayleigh_ritz
    rng = np.random.default_rng(100 + n)
    G = hermitian(rng, np.geomspace(0.1, 10, n))
    L = np.linalg.cholesky(G)
    T = hermitian(rng, np.geomspace(0.3, 300, n))
    S = L @ T @ L.conj().T
    S = 0.5 * (S + S.conj().T)
    lam, C, rank = got = rayleigh_ritz(G, S, m, precision=prec)
    check(G, S, m, got, tol=1e-12 if prec == "fp64" else 1e-10)
    assert np.allclose(lam, np.geomspace(0.3, 300, n)[:m], rtol=0, atol=1e-12 * 300 if prec == "fp64" else 1e-10 * 300)


@pytest.mark.parametrize("gap", [0.0, 1e-14, 1e-11, 1e-8, 1e-5])
@pytest.mark.parametrize("n,m", [s for s in SIZES if s[1] >= 2])
def test_close_wanted_pairs(omb, n, m, gap):
    """Two (then all) wanted eigenvalues `gap` apart: too close for the first-order refinement of the FP32
    sweeps, so the FP64 Jacobi takes over; the pairs are as accurate as separated ones."""
    from omb200.ops import rayleigh_ritz
    rng = np.random.default_rng(200 + n)
    for close in (2, m):
        lam = np.linspace(1.0, 30.0, n)
        lam[:close] = 0.4 + gap * np.arange(close)
        G = hermitian(rng, np.linspace(1, 10, n))
        L = np.linalg.cholesky(G)
        S = L @ hermitian(rng, lam) @ L.conj().T
        S = 0.5 * (S + S.conj().T)
        got = rayleigh_ritz(G, S, m)
        check(G, S, m, got)
        assert np.allclose(got[0], lam[:m], rtol=0, atol=1e-12 * 30)


def test_overflowing_operator_is_an_error(omb):
    """An FP32 operator application that overflows (ε⁻¹ near the largest float): OMB_ERR_NAN from an FP32
    solve, OMB_ERR_NOT_CONVERGED from a mixed one (whose FP64 phase runs on and does not get
    there), and the context still solves."""
    g = omb.Grid(6.0, 4.0, 24, 16)
    ei = gaussian_epsinv(P_WG)
    for prec, code in (("fp32", 7), ("mixed", 3)):
        with pytest.raises(omb.OmbError) as ex:
            omb.solve_omega2(1.2, ei * (3e38 / ei.max()), g, omb.B200Solver(precision=prec), nev=2)
        assert ex.value.code == code
    ev, _ = omb.solve_omega2(1.2, ei, g, nev=2)
    assert np.all(ev > 0)
