"""Parity of the device eigensolves (solve_ω², solve_k) with the FP64 oracle, through the
C ABI, on the reference's own test fixture (``ME/test/runtests.jl:29-45``) and analytic
known answers.

Tolerances: eigenvalue / k relative error ≤ 1e-9 (the target after the FP64 polish),
residual ‖M̂h − ω²h‖ ≤ 1e-8 of the converged unit eigenvector (plus the |Δk| < k_tol
offset of the final Newton update), FP32-only runs at the reference's FP32 tolerance 1e-5
(``ME/test/runtests.jl:205-218``)."""

from __future__ import annotations

import numpy as np
import pytest

import oracle as O
from conftest import OMEGA0, P_WG, gaussian_epsinv

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def omb():
    import omb200
    return omb200


@pytest.fixture(scope="module")
def case():
    grid = O.Grid(6.0, 4.0, 24, 16)
    ei = gaussian_epsinv(P_WG)
    km, kv = O.solve_k(OMEGA0, ei, grid, nev=2, k_tol=1e-12, eig_tol=1e-11)
    return grid, ei, km, kv


def _resid(k, ei, grid, h, w2):
    return np.linalg.norm(O.Operator(k, ei, grid).M(h) - w2 * h)


def _overlap(a, b):
    return abs(np.vdot(a, b)) / (np.linalg.norm(a) * np.linalg.norm(b))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_solve_omega2_parity(omb, case, prec):
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    k0 = O.k_guess(OMEGA0, ei)
    ref, refv, _ = O.solve_omega2(k0, ei, grid, nev=3, tol=1e-11)
    ev, evecs, info = omb.solve_omega2(k0, ei, g, omb.B200Solver(precision=prec), nev=3, return_info=True)
    assert np.all(info["status"] == 0)
    assert np.allclose(ev, ref, rtol=1e-9, atol=0)
    for a, v in zip(ev, evecs):
        assert np.isclose(np.linalg.norm(v), 1.0, rtol=1e-10)
        assert _resid(k0, ei, grid, v, a) < 1.5e-8


@pytest.mark.parametrize("prec,precond,newton", [
    ("mixed", "mpb", "inner"), ("fp64", "mpb", "inner"), ("mixed", "diag", "inner"),
    ("fp64", "mpb", "outer"), ("fp64", "diag", "outer"),
])
def test_solve_k_parity(omb, case, prec, precond, newton):
    grid, ei, km_ref, kv_ref = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    solver = omb.B200Solver(precision=prec, preconditioner=precond, newton=newton)
    km, kv, info = omb.solve_k(OMEGA0, ei, g, solver, nev=2, return_info=True)
    assert np.all(info["status"] == 0), info
    assert np.allclose(km, km_ref, rtol=1e-9, atol=0), (km, km_ref)
    for k, h, href in zip(km, kv, kv_ref):
        assert np.isclose(np.linalg.norm(h), 1.0, rtol=1e-10)
        assert _resid(k, ei, grid, h, OMEGA0 ** 2) < 5e-8
        assert _overlap(h, href) > 1 - 1e-8
        E = O.E_field(k, h, ei, grid)
        e = E[np.argmax(np.abs(E))]
        assert abs(e.imag) <= 1e-9 * abs(e) and e.real > 0
    # n_g from the adjoint slope: ∂ω²/∂k = 2⟨h|∂M̂/∂k|h⟩
    for k, h, d in zip(km, kv, info["dw2dk"]):
        assert np.isclose(d, 2 * O.Operator(k, ei, grid).HMkH(h), rtol=1e-6)


def test_solve_k_fp32(omb, case):
    grid, ei, km_ref, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    km, kv = omb.solve_k(OMEGA0, ei, g, omb.B200Solver(precision="fp32"), nev=2)
    assert np.allclose(km, km_ref, rtol=1e-5)


def test_uniform_medium_known_answer(omb):
    g = omb.Grid(6.0, 4.0, 24, 16)
    eps = 2.5
    ei = np.zeros((3, 3, 24, 16))
    for a in range(3):
        ei[a, a] = 1 / eps
    km, _ = omb.solve_k(OMEGA0, ei, g, nev=2)
    assert np.allclose(km, OMEGA0 * np.sqrt(eps), rtol=1e-10)


def test_round_trip_and_bounds(omb, case):
    # ME/test/runtests.jl:76-82
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    km, _ = omb.solve_k(OMEGA0, ei, g, nev=1)
    assert np.sqrt(P_WG[1]) < km[0] / OMEGA0 < np.sqrt(P_WG[0])
    ev, _ = omb.solve_omega2(km[0], ei, g, nev=1)
    assert np.isclose(ev[0], OMEGA0 ** 2, rtol=1e-9)


def test_batch_matches_single(omb, case):
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    omegas = [1 / 1.45, 1 / 1.55, 1 / 1.65]
    batch = omb.solve_k_batch([{"omega": w, "eps_inv": ei, "grid": g, "nev": 2} for w in omegas])
    for w, (km, kv) in zip(omegas, batch):
        ref, _ = O.solve_k(w, ei, grid, nev=2, k_tol=1e-12, eig_tol=1e-11)
        assert np.allclose(km, ref, rtol=1e-9)


def test_warm_start_guess(omb, case):
    grid, ei, km_ref, kv_ref = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    ret, info = omb.solve_k_batch([{"omega": OMEGA0, "eps_inv": ei, "grid": g, "nev": 2,
                                    "kguess": km_ref[0], "Hguess": kv_ref}], return_info=True)
    km = ret[0][0]
    assert np.allclose(km, km_ref, rtol=1e-9)
    _, info0 = omb.solve_k_batch([{"omega": OMEGA0, "eps_inv": ei, "grid": g, "nev": 2}],
                                 return_info=True)
    assert info[0]["iterations"].sum() < info0[0]["iterations"].sum()


@pytest.mark.parametrize("newton", ["inner", "outer"])
def test_sweep_warm_start(omb, case, newton):
    """A frequency sweep in one batch (OMB_WARM_SWEEP): the same k as independent solves
    (and the oracle), and the members started from the solved neighbour need fewer
    iterations than their cold solves."""
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    omegas = [1 / 1.50, 1 / 1.53, 1 / 1.56, 1 / 1.59]
    probs = [{"omega": w, "eps_inv": ei, "grid": g, "nev": 2} for w in omegas]
    prec = "fp64" if newton == "outer" else "mixed"
    cold, info_c = omb.solve_k_batch(probs, omb.B200Solver(precision=prec, newton=newton), return_info=True)
    warm, info_w = omb.solve_k_batch(probs, omb.B200Solver(precision=prec, newton=newton, warm_start="sweep"),
                                     return_info=True)
    for w, (kc, _), (kw, vw), iw in zip(omegas, cold, warm, info_w):
        assert np.all(iw["status"] == 0)
        assert np.allclose(kw, kc, rtol=1e-9)
        ref, _ = O.solve_k(w, ei, grid, nev=2, k_tol=1e-12, eig_tol=1e-11)
        assert np.allclose(kw, ref, rtol=1e-9)
        for b in range(2):
            assert _resid(kw[b], ei, grid, vw[b], w * w) < 2e-8
    # the anchor is the ω nearest the mean (index 1 or 2); the other three start warm
    it_c = np.array([i["iterations"].sum() for i in info_c])
    it_w = np.array([i["iterations"].sum() for i in info_w])
    assert it_w.sum() < it_c.sum()


def test_cells_warm_start(omb):
    """A taper of cross-sections at one ω in one batch (OMB_WARM_CELLS, the batched form of
    eme(...; warmstart=true)): every cell matches its own oracle solve, and the cells started
    from the middle one need fewer iterations than their cold solves."""
    from conftest import gaussian_epsinv
    grid = O.Grid(6.0, 4.0, 24, 16)
    g = omb.Grid(6.0, 4.0, 24, 16)
    cells = [gaussian_epsinv((4.2, 2.1, 1.0 + 0.04 * c, 0.6)) for c in range(5)]
    probs = [{"omega": OMEGA0, "eps_inv": e, "grid": g, "nev": 2} for e in cells]
    cold, info_c = omb.solve_k_batch(probs, omb.B200Solver(), return_info=True)
    warm, info_w = omb.solve_k_batch(probs, omb.B200Solver(warm_start="cells"), return_info=True)
    for e, (kc, _), (kw, vw), iw in zip(cells, cold, warm, info_w):
        assert np.all(iw["status"] == 0)
        assert np.allclose(kw, kc, rtol=1e-9)
        ref, _ = O.solve_k(OMEGA0, e, grid, nev=2, k_tol=1e-12, eig_tol=1e-11)
        assert np.allclose(kw, ref, rtol=1e-9)
        for b in range(2):
            assert _resid(kw[b], e, grid, vw[b], OMEGA0 ** 2) < 2e-8
    it_c = np.array([i["iterations"].sum() for i in info_c])
    it_w = np.array([i["iterations"].sum() for i in info_w])
    assert it_w.sum() < it_c.sum()


def test_kguess_bands(omb, case):
    """Per-band Newton starts reach the same k."""
    grid, ei, km_ref, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    ret = omb.solve_k_batch([{"omega": OMEGA0, "eps_inv": ei, "grid": g, "nev": 2,
                              "kguess_bands": km_ref * 1.01}])
    assert np.allclose(ret[0][0], km_ref, rtol=1e-9)


def test_uneven_batch(omb):
    """One batch mixing grids, cells, frequencies and band counts (the shape of the
    uneven-grid sweep): every instance matches its own oracle solve."""
    specs = [  # (Nx, Ny, Dx, Dy, ω, nev, bump)
        (24, 16, 6.0, 4.0, 1 / 1.55, 2, P_WG),
        (32, 24, 6.0, 4.5, 1 / 1.45, 3, (4.6, 2.1, 1.1, 0.7)),
        (20, 20, 5.0, 5.0, 1 / 1.60, 1, (3.98, 2.09, 0.9, 0.9)),
        (24, 16, 6.0, 4.0, 1 / 1.50, 3, P_WG),
        (48, 32, 6.0, 4.0, 1 / 1.55, 2, P_WG),
    ]
    probs, refs = [], []
    for Nx, Ny, Dx, Dy, w, nev, p in specs:
        ei = gaussian_epsinv(p, Dx, Dy, Nx, Ny)
        probs.append({"omega": w, "eps_inv": ei, "grid": omb.Grid(Dx, Dy, Nx, Ny), "nev": nev})
        refs.append(O.solve_k(w, ei, O.Grid(Dx, Dy, Nx, Ny), nev=nev, k_tol=1e-12, eig_tol=1e-11)[0])
    for warm in ("none", "sweep"):
        out, info = omb.solve_k_batch(probs, omb.B200Solver(warm_start=warm), return_info=True)
        for (km, kv), i, ref, pr in zip(out, info, refs, probs):
            assert np.all(i["status"] == 0)
            assert np.allclose(km, ref, rtol=1e-9)
            assert len(kv) == pr["nev"] and all(v.shape == (2 * pr["grid"].N,) for v in kv)


@pytest.mark.parametrize("nev", [1, 2, 4, 5, 7, 10, 11])
def test_rayleigh_ritz_block_sizes(omb, case, nev):
    """Blocks of nev + 1 columns, so Rayleigh–Ritz bases of up to 6, 9, 15, 18, 24, 33 and 36: one,
    two and three 16-wide tiles per dimension of k_rr, even and odd sizes, and the largest.
    FP64 at 1e-10, so eigenvalue errors are ≈ residual²/gap: rtol 1e-9 as for the other solves."""
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    k0 = O.k_guess(OMEGA0, ei)
    ref, _, _ = O.solve_omega2(k0, ei, grid, nev=nev + 2, tol=1e-9, maxiter=600)
    ev, evecs, info = omb.solve_omega2(k0, ei, g, omb.B200Solver(precision="fp64"), nev=nev, tol=1e-10, return_info=True)
    assert np.all(info["status"] == 0)
    assert np.allclose(ev, ref[:nev], rtol=1e-9, atol=0)
    V = np.stack(evecs, axis=1)
    assert np.allclose(V.conj().T @ V, np.eye(nev), atol=1e-10)


def test_more_tracks_than_a_scan(omb, case):
    """270 problems of two bands: 540 tracks, 270 per lane, so the live-tile prefixes take two rounds of
    the 256-thread scan and are too many for the streaming kernels' shared-memory copy.  Every band
    converges, and a sample agrees with the same problems solved alone (k rtol 1e-9)."""
    grid, ei, _, _ = case
    g = omb.Grid(6.0, 4.0, 24, 16)
    om = OMEGA0 * (1 + 0.0005 * np.arange(270))
    res, info = omb.solve_k_batch([{"omega": w, "eps_inv": ei, "grid": g, "nev": 2} for w in om], return_info=True)
    assert all(np.all(i["status"] == 0) for i in info)
    for j in (0, 1, 134, 135, 255, 256, 269):
        km, _ = omb.solve_k(om[j], ei, g, nev=2)
        assert np.allclose(res[j][0], km, rtol=1e-9, atol=0)


# 128² cell of 3 × 2 μm: bands 2 and 3 have k = 0.830169 and 0.830165
NEAR_PAIR = ((3.554630006558236, 2.003322750103637, 0.4164621074304316, 0.48672393048774054), 0.6064630733279459)


def test_near_degenerate_pair_converges_from_any_start(omb):
    """Two bands 4.5e-6 apart in k, to residuals of 3e-12 from 40 random blocks: the recurrences of
    AX and AP lose accuracy while the pair separates, and without starting again from X about one start in
    six ended with residuals of 1e-8 to 1e-5 that no longer fell."""
    P, w = NEAR_PAIR
    g = omb.Grid(3.0, 2.0, 128, 128)
    ei = gaussian_epsinv(P, 3.0, 2.0, 128, 128)
    ks = []
    for seed in range(1, 41):
        km, _, info = omb.solve_k(w, ei, g, omb.B200Solver(precision="mixed", seed=seed), nev=4, k_tol=1e-12, eig_tol=3e-12,
                                  return_info=True)
        assert np.all(info["status"] == 0), (seed, info)
        ks.append(km)
    # residual 3e-12: λ to 1e-12 or better, so k to 1e-11 whatever the start
    assert np.allclose(ks, ks[0], rtol=0, atol=1e-11)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("off", [1.2, 2.0])
def test_indefinite_epsinv(omb, prec, off):
    """ε⁻¹ with positive diagonals and off-diagonal entries large enough to make it indefinite in the middle of
    the cell: the lowest eigenvalues are negative, and found (a negative Ritz value is no sign of a broken
    block).  Residual 1e-7: eigenvalues to 1e-7 at worst."""
    g = omb.Grid(6.0, 4.0, 24, 16)
    ei = gaussian_epsinv(P_WG)
    ei[0, 1] = ei[1, 0] = off * ei[0, 0] * np.exp(-np.linspace(-2, 2, 24)[:, None] ** 2)
    op = O.Operator(1.2, ei, O.Grid(6.0, 4.0, 24, 16))
    A = op.M_block(np.eye(2 * g.N, dtype=np.complex128))
    ref = np.linalg.eigvalsh(0.5 * (A + A.conj().T))[:3]
    assert ref[2] < 0
    ev, _ = omb.solve_omega2(1.2, ei, g, omb.B200Solver(precision=prec), nev=3, tol=1e-7)
    assert np.allclose(ev, ref, rtol=0, atol=1e-7)


@pytest.mark.parametrize("seed", [20315, 21121, 23116])
def test_fp32_phase_hands_over_at_its_floor(omb, seed):
    """Frequency sweeps of a narrow LiNbO₃ ridge on 256², started by the learned network, whose FP32 residuals
    settle just above the level that ends the FP32 phase: the phase ends once k has settled, instead of
    taking Newton steps by the noise of k (40 to 60 of the 60 that a band has in most of these solves), so
    that 10 steps in all are enough (5 are usual)."""
    import importlib.util
    import os
    from conftest import ROOT
    spec = importlib.util.spec_from_file_location("speed_cases", os.path.join(ROOT, "perf", "cases.py"))
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    s = cases.prepare({"do": "sweep", "family": "ridge", "nx": 256, "ny": 256, "nev": 2, "widths": 1, "omegas": 4,
                       "warm": "sweep_learned"}, seed)
    for _ in range(8):
        _, info = omb.solve_k_batch(s["problems"], s["solver"], k_tol=1e-12, eig_tol=3e-12, max_eigsolves=10, return_info=True)
        for i in info:
            assert np.all(i["status"] == 0) and np.max(i["newton_steps"]) <= 10
