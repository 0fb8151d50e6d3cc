"""The workloads this library's speed is judged on, called as a user's program calls them.

Each case is one pass through the public Python API (or, for callers that own their device
buffers, one C entry point): mode solves of single cross-sections from the smallest grids to
512×512, batches of them, the reverse-mode rule, a z-periodic cell, one operator application
and the material pass of a smoothing plan.  The cross-sections are the families the
configurations and tests use (a Si₃N₄ rectangle in SiO₂, an x-cut LiNbO₃ ridge, a row of
rectangles with slots between them), with dimensions, position and frequency drawn from the
seed.  The cores sit a fraction of a pixel off the centre of the cell, so that no two pixels
tie for the largest |E| that fixes a mode's phase.

Solves run at ``k_tol = 1e-12, eig_tol = 3e-12``: tolerances of the kind that gradients, group
indices and phase-accurate fields are computed at (modes are then defined to ≈1e-10).
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "optimode.jl_b200"))

import omb200 as omb  # noqa: E402
from omb200 import _lib  # noqa: E402

K_TOL, EIG_TOL = 1e-12, 3e-12
OMEGA0 = 1.0 / 1.55


def listed():
    return [
        # a quick mode check while a design is being drawn: latency is all that counts
        {"name": "solve_48x40", "do": "solve", "family": "rect", "nx": 48, "ny": 40, "nev": 1, "mode": "mixed"},
        # the plain single solve of the reference's examples: TE and TM of a Si3N4 wire
        {"name": "solve_128", "do": "solve", "family": "rect", "nx": 128, "ny": 128, "nev": 2, "mode": "mixed"},
        # the reference's own settings: FP64, its preconditioner, its band-by-band Newton loop
        {"name": "solve_192x128_fp64", "do": "solve", "family": "ridge", "nx": 192, "ny": 128, "nev": 2, "mode": "reference"},
        # one design point of the LiNbO3 ridge at production resolution
        {"name": "solve_256", "do": "solve", "family": "ridge", "nx": 256, "ny": 256, "nev": 4, "mode": "mixed"},
        # a large multi-core cross-section
        {"name": "solve_512", "do": "solve", "family": "slots", "nx": 512, "ny": 512, "nev": 4, "mode": "mixed"},
        # a frequency sweep of three ridge widths, four frequencies each, from learned anchors
        {"name": "sweep_256", "do": "sweep", "family": "ridge", "nx": 256, "ny": 256, "nev": 4, "widths": 3, "omegas": 4,
         "warm": "sweep_learned"},
        # unrelated problems of mixed grids and band counts in one batch
        {"name": "batch_uneven", "do": "uneven", "count": 10, "nx": 256, "ny": 192, "warm": "none"},
        # the gradient of one mode on a small, odd grid
        {"name": "pullback_96x80", "do": "pullback", "family": "rect", "nx": 96, "ny": 80, "nev": 1},
        # the gradient of an inverse-design step through both modes of the wire
        {"name": "pullback_256", "do": "pullback", "family": "rect", "nx": 256, "ny": 256, "nev": 2},
        # Bloch modes of a Bragg-corrugated wire
        {"name": "periodic_32x24x16", "do": "periodic", "nx": 32, "ny": 24, "nz": 16, "nev": 2},
        # the operator inside somebody else's iteration, on that program's device buffers
        {"name": "apply_256", "do": "apply", "family": "ridge", "nx": 256, "ny": 256, "ncol": 4},
        # the permittivity of one geometry at many frequencies, left on the device
        {"name": "smooth_256", "do": "smooth", "nx": 256, "ny": 256, "nsets": 48},
    ]


# every grid side the FFT passes support from 40 points up, by what a solve of it costs
_SIDES = (40, 48, 64, 80, 96, 128, 160, 192, 256)


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "sweep", "uneven", "pullback", "periodic", "apply", "smooth"])
    nx, ny = rng.choice(_SIDES), rng.choice(_SIDES)
    family = rng.choice(["rect", "ridge"])
    if kind == "solve":
        if rng.random() < 0.25:
            return {"do": "solve", "family": "slots", "nx": rng.choice((320, 384, 512)), "ny": rng.choice((192, 256, 320, 384)),
                    "nev": rng.randint(1, 4), "mode": "mixed"}
        return {"do": "solve", "family": family, "nx": nx, "ny": ny, "nev": rng.randint(1, 2 if family == "rect" else 4),
                "mode": rng.choice(["mixed", "mixed", "fp64", "reference"])}
    if kind == "sweep":
        return {"do": "sweep", "family": "ridge", "nx": nx, "ny": ny, "nev": rng.randint(1, 4), "widths": rng.randint(1, 3),
                "omegas": rng.randint(2, 4), "warm": "sweep"}
    if kind == "uneven":
        return {"do": "uneven", "count": rng.randint(2, 10), "nx": rng.choice((96, 128, 160, 192)), "ny": rng.choice((80, 96, 128)),
                "warm": "none"}
    if kind == "pullback":
        return {"do": "pullback", "family": "rect", "nx": nx, "ny": ny, "nev": rng.randint(1, 2)}
    if kind == "periodic":
        return {"do": "periodic", "nx": rng.choice((24, 32, 40, 48)), "ny": rng.choice((16, 20, 24, 32)), "nz": rng.choice((8, 12, 16)),
                "nev": rng.randint(1, 2)}
    if kind == "apply":
        return {"do": "apply", "family": family, "nx": nx, "ny": ny, "ncol": rng.randint(1, 262144 // (nx * ny) if nx * ny > 32768 else 8)}
    return {"do": "smooth", "nx": nx, "ny": ny, "nsets": int(round(math.exp(rng.uniform(0, math.log(48)))))}


# ---- cross-sections ------------------------------------------------------------------------

_CELL = {"rect": (6.0, 4.0), "ridge": (8.0, 5.0), "slots": (8.0, 5.0)}


def _box(x0, x1, y0, y1):
    return [(x0, y0), (x1, y0), (x1, y1), (x0, y1)]


def _shapes(family, r, dx, dy, width=None):
    """(convex outlines with diagonal ε, highest priority first; ε around them)."""
    jit = lambda v, s=0.02: v * (1 + s * r.uniform(-1, 1))  # noqa: E731
    cx, cy = r.uniform(0.15, 0.35) * dx, r.uniform(0.15, 0.35) * dy
    if family == "rect":
        w, h = jit(1.7) if width is None else width, jit(0.7)
        return [(_box(cx - w / 2, cx + w / 2, cy - h / 2, cy + h / 2), (3.98, 3.98, 3.98))], (2.09, 2.09, 2.09)
    sub = (2.09, 2.09, 2.09)
    if family == "ridge":
        w, slab, etch = jit(1.5) if width is None else width, jit(0.3), jit(0.3)
        side = etch / math.tan(math.radians(70.0))
        y0 = cy - 0.3
        ln = (4.97, 4.61, 4.97)
        top = [(cx - w / 2 - side, y0 + slab), (cx + w / 2 + side, y0 + slab), (cx + w / 2, y0 + slab + etch), (cx - w / 2, y0 + slab + etch)]
        return [(top, ln), (_box(-40, 40, y0, y0 + slab), ln), (_box(-40, 40, -40, y0), sub)], (1.0, 1.0, 1.0)
    out, x, y0 = [], cx - 1.9, cy - 0.5
    for w, gap, e in ((1.4, 0.3, 4.2), (0.5, 0.25, 3.98), (1.0, 0.0, 4.2)):
        w, gap = jit(w), jit(gap)
        out.append((_box(x, x + w, y0, y0 + 0.65), (e, e, e)))
        x += w + gap
    return out + [(_box(-40, 40, -40, y0), sub)], (1.0, 1.0, 1.0)


def _epsinv(shapes, around, Dx, Dy, nx, ny):
    """Sub-pixel averaged ε⁻¹ (3, 3, nx, ny): harmonic along the interface normal, arithmetic across it."""
    dx, dy = Dx / nx, Dy / ny
    X, Y = np.meshgrid(-Dx / 2 + np.arange(nx) * dx, -Dy / 2 + np.arange(ny) * dy, indexing="ij")
    e = np.array(around)[:, None, None] * np.ones((3, nx, ny))
    h = 1.0 / e
    n, best = np.zeros((2, nx, ny)), np.zeros((nx, ny))
    for verts, eps in reversed(shapes):
        v = np.array(verts)
        t = np.roll(v, -1, axis=0) - v
        t /= np.linalg.norm(t, axis=1)[:, None]
        d = np.stack([(X - p[0]) * q[1] - (Y - p[1]) * q[0] for p, q in zip(v, t)])
        at = d.argmax(0)
        nn = np.stack([t[at, 1], -t[at, 0]])
        f = np.clip(0.5 - d.max(0) / (np.abs(nn[0]) * dx + np.abs(nn[1]) * dy), 0, 1)
        ev = np.array(eps)[:, None, None]
        e, h = f * ev + (1 - f) * e, f / ev + (1 - f) * h
        edge = f * (1 - f)
        n = np.where(edge >= best, nn, n)
        best = np.where(f >= 1, 0, np.maximum(best, edge))
    n = np.where(best > 0, n, 0)
    P = np.zeros((3, 3, nx, ny))
    P[0, 0], P[1, 1], P[0, 1], P[1, 0] = n[0] ** 2, n[1] ** 2, n[0] * n[1], n[0] * n[1]
    Q = np.eye(3)[:, :, None, None] - P
    out = np.einsum("abxy,bxy,bcxy->acxy", P, h, P) + np.einsum("abxy,bxy,bcxy->acxy", Q, 1 / e, Q)
    return np.asfortranarray(0.5 * (out + out.swapaxes(0, 1)))


def _cell(family, nx, ny, r, width=None):
    Dx, Dy = _CELL[family]
    shapes, around = _shapes(family, r, Dx / nx, Dy / ny, width)
    return omb.Grid(Dx, Dy, nx, ny), _epsinv(shapes, around, Dx, Dy, nx, ny)


def _omega(r):
    return OMEGA0 * (1 + 0.01 * r.uniform(-1, 1))


def _solver(mode, warm="none"):
    if mode == "reference":
        return omb.B200Solver(precision="fp64", preconditioner="mpb", newton="outer", warm_start=warm)
    return omb.B200Solver(precision=mode, warm_start=warm)


def _problems(case, r):
    if case["do"] == "sweep":
        probs = []
        for w in np.linspace(1.0, 2.0, 3)[:case["widths"]]:
            g, e = _cell(case["family"], case["nx"], case["ny"], r, w * (1 + 0.02 * r.uniform(-1, 1)))
            for j in range(case["omegas"]):
                probs.append({"omega": _omega(r) * 1.55 / (1.5 + 0.025 * j), "eps_inv": e, "grid": g, "nev": case["nev"]})
        return probs
    # uneven: sides from half the given ones up, one to three bands
    sx = [s for s in _SIDES if case["nx"] // 2 <= s <= case["nx"]]
    sy = [s for s in _SIDES if case["ny"] // 2 <= s <= case["ny"]]
    q = np.random.RandomState(case["count"])  # the shape of the batch belongs to the case, its contents to the seed
    probs = []
    for _ in range(case["count"]):
        family = ("rect", "ridge")[q.randint(2)]
        g, e = _cell(family, int(q.choice(sx)), int(q.choice(sy)), r)
        probs.append({"omega": _omega(r), "eps_inv": e, "grid": g, "nev": int(q.randint(1, 3 if family == "rect" else 4))})
    return probs


def _bragg(case, r):
    g = omb.Grid3(6.0, 4.0, 0.25, case["nx"], case["ny"], case["nz"])
    shapes, around = _shapes("rect", r, 6.0 / case["nx"], 4.0 / case["ny"])
    (x0, y0), _, (x1, y1), _ = shapes[0][0]
    wide = _epsinv(shapes, around, 6.0, 4.0, case["nx"], case["ny"])
    slim = _epsinv([(_box(x0 + 0.15, x1 - 0.15, y0, y1), shapes[0][1])], around, 6.0, 4.0, case["nx"], case["ny"])
    half = case["nz"] // 2
    return g, np.asfortranarray(np.stack([wide] * half + [slim] * (case["nz"] - half), axis=-1))


def _cotangents(case, n2, r):
    """A smooth seeded field cotangent per band (the gradient of an overlap) and one for k."""
    nx, ny = case["nx"], case["ny"]
    gx, gy = np.fft.fftfreq(nx) * nx / 6.0, np.fft.fftfreq(ny) * ny / 4.0
    env = np.exp(-(gx[None, :] ** 2 + gy[:, None] ** 2) / 4.0)[..., None]
    out = []
    for _ in range(case["nev"]):
        v = ((r.standard_normal((ny, nx, 2)) + 1j * r.standard_normal((ny, nx, 2))) * env).reshape(-1)
        out.append(v / np.linalg.norm(v))
    return r.standard_normal(case["nev"]), out


# ---- the calls -----------------------------------------------------------------------------

def prepare(case, seed):
    r = np.random.RandomState(seed)
    s = {"do": case["do"]}
    if case["do"] == "solve":
        s["grid"], s["eps"] = _cell(case["family"], case["nx"], case["ny"], r)
        s["omega"], s["nev"], s["solver"] = _omega(r), case["nev"], _solver(case["mode"])
    elif case["do"] in ("sweep", "uneven"):
        s["problems"], s["solver"] = _problems(case, r), _solver("mixed", case["warm"])
    elif case["do"] == "pullback":
        s["grid"], s["eps"] = _cell(case["family"], case["nx"], case["ny"], r)
        s["omega"] = _omega(r)
        s["kbar"], s["evbar"] = _cotangents(case, 2 * s["grid"].N, r)
        s["kmags"], s["evecs"] = omb.solve_k(s["omega"], s["eps"], s["grid"], _solver("fp64"), nev=case["nev"], k_tol=1e-12,
                                             eig_tol=1e-12)
        s["solver"] = _solver("mixed")
    elif case["do"] == "periodic":
        s["grid"], s["eps"] = _bragg(case, r)
        s["omega"], s["nev"], s["solver"] = _omega(r), case["nev"], _solver("mixed")
    elif case["do"] == "apply":
        g, e = _cell(case["family"], case["nx"], case["ny"], r)
        h = _block(case, r)
        s["grid"], s["k"], s["ncol"] = g, 2.0 * _omega(r), case["ncol"]
        s["eps"] = torch.tensor(e.reshape(-1, order="F"), dtype=torch.float32, device="cuda")
        s["h"] = torch.tensor(h, dtype=torch.complex64, device="cuda")
        s["out"] = torch.empty_like(s["h"])
        s["lib"] = _lib.load()
    else:
        g = omb.Grid(8.0, 5.0, case["nx"], case["ny"])
        shapes, _ = _shapes("ridge", r, 8.0 / case["nx"], 5.0 / case["ny"])
        s["plan"] = omb.SmoothingPlan([np.array(v) for v, _ in shapes], [0, 0, 1, 2], g)
        s["mats"] = _materials(case, r)
        n = g.N * case["nsets"]
        s["eps"] = torch.empty(27 * n, dtype=torch.float64, device="cuda")
        s["epsinv"] = torch.empty(9 * n, dtype=torch.float64, device="cuda")
        s["stream"] = torch.cuda.current_stream()
    return s


def _block(case, r):
    n2 = 2 * case["nx"] * case["ny"]
    h = r.standard_normal((case["ncol"], n2)) + 1j * r.standard_normal((case["ncol"], n2))
    return (h / np.linalg.norm(h, axis=1)[:, None]).astype(np.complex64)


def _materials(case, r):
    """ε, ∂ε/∂ω and ∂²ε/∂ω² columns of LiNbO₃, SiO₂ and air over a band of frequencies (one-pole dispersion)."""
    w = np.linspace(0.55, 0.75, case["nsets"]) * (1 + 0.005 * r.uniform(-1, 1))
    out = np.zeros((27, 3, case["nsets"]))
    for m, diag in enumerate(((4.6, 4.2, 4.6), (2.05, 2.05, 2.05))):
        for a, e in enumerate(diag):
            q = 1 - 0.04 * w ** 2
            for d, f in enumerate((1 / q, 0.08 * w / q ** 2, 0.08 / q ** 2 + 2 * (0.08 * w) ** 2 / q ** 3)):
                out[9 * d + 4 * a, m] = 1.0 * (d == 0) + (e - 1) * f
    out[[0, 4, 8], 2] = 1.0
    return out


def run(s):
    do = s["do"]
    if do == "solve":
        return omb.solve_k(s["omega"], s["eps"], s["grid"], s["solver"], nev=s["nev"], k_tol=K_TOL, eig_tol=EIG_TOL)
    if do in ("sweep", "uneven"):
        return omb.solve_k_batch(s["problems"], s["solver"], k_tol=K_TOL, eig_tol=EIG_TOL)
    if do == "pullback":
        return omb.pullback(s["omega"], s["eps"], s["grid"], s["kmags"], s["evecs"], s["kbar"], s["evbar"], s["solver"])
    if do == "periodic":
        return omb.solve_k_periodic(s["omega"], s["eps"], s["grid"].Dz, s["grid"], s["solver"], nev=s["nev"], k_tol=K_TOL, eig_tol=EIG_TOL)
    if do == "apply":
        g = s["grid"]
        _lib.check(s["lib"].omb_apply_M_noalloc(g.Nx, g.Ny, g.Dx, g.Dy, s["k"], s["eps"].data_ptr(), s["ncol"], s["h"].data_ptr(),
                                                s["out"].data_ptr(), torch.cuda.current_stream().cuda_stream))
        return s["out"]
    s["plan"].smooth_eps_device(s["mats"], s["eps"], s["epsinv"], s["stream"])
    return s["eps"], s["epsinv"]


def work(case):
    """Inputs read and outputs written once; solves: 60 block iterations per mode, pull-backs 150
    MINRES iterations per mode, each with one operator application per column and its vector algebra."""
    sizes = [(case["nx"] * case["ny"] * case.get("nz", 1), case.get("nev", 1))]
    if case["do"] in ("sweep", "uneven"):
        sizes = [(p["grid"].N, p["nev"]) for p in _problems(case, np.random.RandomState(0))]
    b = f = 0.0
    for n, nev in sizes:
        apply1 = 30 * n * math.log2(n) + 110 * n
        if case["do"] == "apply":
            return {"bytes": n * (36 + 32 * case["ncol"]), "flops": apply1 * case["ncol"]}
        if case["do"] == "smooth":
            return {"bytes": 8 * 36 * n * case["nsets"] + 8 * n, "flops": 30 * n * case["nsets"]}
        if case["do"] == "pullback":
            b += n * (144 + 64 * nev)
            f += nev * 150 * (apply1 + 120 * n)
            continue
        b += n * (72 + 32 * nev)
        for band in range(nev):
            m = band + 2
            f += 60 * (m * apply1 + 2 * n * 8 * (9 * m * m + 12 * m * m))
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------

class _Op:
    """M̂(k) on a flat (ny·nx or nz·ny·nx)-ordered field of two transverse coefficients."""

    def __init__(self, grid, epsinv):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        nz, Dz = getattr(grid, "Nz", 1), getattr(grid, "Dz", 1.0)
        self.shape = (nz, grid.Ny, grid.Nx)
        fr = lambda n, d: torch.tensor(np.fft.fftfreq(n) * n / d, device=dev)  # noqa: E731
        self.gx, self.gy, self.gz = fr(grid.Nx, grid.Dx)[None, None, :], fr(grid.Ny, grid.Dy)[None, :, None], fr(nz, Dz)[:, None, None]
        e = torch.tensor(np.ascontiguousarray(epsinv), device=dev)
        self.e = e.reshape(3, 3, grid.Nx, grid.Ny, nz).permute(0, 1, 4, 3, 2).contiguous()
        self.dev, self.n2 = dev, 2 * nz * grid.Ny * grid.Nx

    def basis(self, k):
        one = torch.ones(self.shape, dtype=torch.float64, device=self.dev)
        kz, gx, gy = (k - self.gz) * one, self.gx * one, self.gy * one
        p2 = gx * gx + gy * gy
        at0 = p2 == 0
        p = torch.sqrt(torch.where(at0, one, p2))
        mag = torch.sqrt(p2 + kz * kz)
        n = (torch.where(at0, 0 * one, gy / p), torch.where(at0, one, -gx / p), 0 * one)
        m = (torch.where(at0, torch.sign(kz), -gx * kz / (p * mag)), torch.where(at0, 0 * one, -gy * kz / (p * mag)),
             torch.where(at0, 0 * one, -p2 / (p * mag)))
        return mag, torch.stack(m), torch.stack(n)

    def curl(self, k, H):  # columns (c, n2) → fft of −mag(h1 n̂ − h2 m̂), (c, 3, nz, ny, nx)
        mag, m, n = self.basis(k)
        h = H.reshape(-1, *self.shape, 2)
        return torch.fft.fftn(-mag * (h[..., 0][:, None] * n - h[..., 1][:, None] * m), dim=(-3, -2, -1))

    def contract(self, D):
        return torch.einsum("abzyx,qbzyx->qazyx", self.e.to(torch.complex128), D)

    def __call__(self, k, H):
        mag, m, n = self.basis(k)
        E = torch.fft.ifftn(self.contract(self.curl(k, H)), dim=(-3, -2, -1))
        return torch.stack([-mag * (E * n).sum(1), mag * (E * m).sum(1)], dim=-1).reshape(-1, self.n2)

    def precond(self, k):
        one = torch.ones(self.shape, dtype=torch.float64, device=self.dev)
        return (1 / (self.gx ** 2 + self.gy ** 2 + (k - self.gz) ** 2) * one).reshape(-1, 1).expand(-1, 2).reshape(-1)


def _orth(S):
    for _ in range(2):
        S = S / torch.linalg.norm(S, dim=1, keepdim=True)
        G = S.conj() @ S.T
        L = torch.linalg.cholesky(G + 1e-15 * torch.eye(len(G), device=S.device))
        S = torch.linalg.solve_triangular(L.conj(), S, upper=False)
    return S


def _lowest(op, k, X, need, tol, most=1200):
    """Lowest Ritz pairs of M̂(k) from the rows of X: block LOBPCG, every product formed afresh."""
    M, P, pre = len(X), None, op.precond(k)
    X = _orth(X)
    for _ in range(most):
        AX = op(k, X)
        w, c = torch.linalg.eigh(X.conj() @ AX.T)
        X, AX = c.T @ X, c.T @ AX
        R = AX - w[:, None] * X
        if float(torch.linalg.norm(R[:need], dim=1).max()) < tol:
            break
        W = R * pre
        for _ in range(2):
            W = W - (W @ X.conj().T) @ X
        S = _orth(torch.cat([X, W] + ([P] if P is not None else [])))
        w, c = torch.linalg.eigh(S.conj() @ op(k, S).T)
        X = c[:, :M].T @ S
        P = c[M:, :M].T @ S[M:]
        P = P - (P @ X.conj().T) @ X
    return w, X


def _modes(op, omega, nev, k=None, tol=2e-13):
    """k and phase-fixed modes (rows) of the lowest bands at omega: Newton on k, band after band."""
    g = torch.Generator(device="cpu").manual_seed(1)
    X = torch.complex(*torch.randn(2, nev + 3, op.n2, dtype=torch.float64, generator=g)).to(op.dev)
    k = omega / math.sqrt(float(torch.stack([op.e[a, a] for a in range(3)]).min())) ** -1 if k is None else k
    ks, vs = [], []
    for b in range(nev):
        for step in range(40):
            w, X = _lowest(op, k, X, b + 1, 1e-4 if step == 0 and b == 0 else (1e-9 if step < 3 else max(tol, 3e-15 * op.n2 ** 0.5)))
            dk = (float(w[b]) - omega ** 2) / _slope(op, k, X[b])
            k -= dk
            if abs(dk) < 1e-13 and step > 3:
                break
        E = op.contract(op.curl(k, X[b:b + 1]))[0].permute(1, 2, 3, 0).reshape(-1)
        at = E[E.abs().argmax()]
        ks.append(k)
        vs.append(X[b] * at.conj() / at.abs())
    return ks, vs


def _slope(op, k, h):
    t = torch.tensor(k, dtype=torch.float64, device=op.dev, requires_grad=True)
    D = op.curl(t, h[None])
    v = (D.conj() * op.contract(D)).real.sum() / (op.n2 / 2)
    return float(torch.autograd.grad(v, t)[0])


def _adjoint(op, k, h, w2, b):
    """λ ⟂ h with (M̂ − ω²)λ = b − h⟨h, b⟩: preconditioned MINRES (Paige and Saunders 1975)."""
    away = lambda v: v - h * torch.vdot(h, v)  # noqa: E731
    pre = op.precond(k)
    A = lambda v: away(op(k, v[None])[0] - w2 * v)  # noqa: E731
    r1 = r2 = away(b)
    y = away(pre * r1)
    beta1 = beta = math.sqrt(float(torch.vdot(r1, y).real))
    x, w, wo = torch.zeros_like(b), torch.zeros_like(b), torch.zeros_like(b)
    old = dbar = eps = 0.0
    phibar, cs, sn, low = beta1, -1.0, 0.0, 0
    for it in range(6000):
        v = y / beta
        y = A(v)
        if it:
            y = y - (beta / old) * r1
        alfa = float(torch.vdot(v, y).real)
        y = y - (alfa / beta) * r2
        r1, r2 = r2, away(y)
        y = away(pre * r2)
        old, beta = beta, math.sqrt(max(0.0, float(torch.vdot(r2, y).real)))
        olde, delta, gbar = eps, cs * dbar + sn * alfa, sn * dbar - cs * alfa
        eps, dbar = sn * beta, -cs * beta
        gamma = math.hypot(gbar, beta)
        cs, sn = gbar / gamma, beta / gamma
        phi, phibar = cs * phibar, sn * phibar
        wo, w = w, (v - olde * wo - delta * w) / gamma
        x = x + phi * w
        low = low + 1 if phibar < 1e-13 * beta1 else 0
        if low > 3 or beta == 0.0:
            break
    return away(x)


def _exact_pullback(case, r):
    grid, e = _cell(case["family"], case["nx"], case["ny"], r)
    omega = _omega(r)
    kbar, evbar = _cotangents(case, 2 * grid.N, r)
    op = _Op(grid, e)
    N = op.n2 // 2
    ks, hs = _modes(op, omega, case["nev"])
    wbar, ebar = 0.0, torch.zeros(3, 3, *op.shape, dtype=torch.float64, device=op.dev)
    for k, h, kb, eb in zip(ks, hs, kbar, evbar):
        lam = _adjoint(op, k, h, omega ** 2, torch.tensor(eb, device=op.dev))
        t = torch.tensor(k, dtype=torch.float64, device=op.dev, requires_grad=True)
        D, L = op.curl(t, h[None]), op.curl(t, lam[None])
        kh = -float(torch.autograd.grad((L.conj() * op.contract(D)).real.sum() / N, t)[0])
        s = (kb + kh) / _slope(op, k, h)
        D, L = D.detach()[0], (L.detach() + s * D.detach())[0]
        G = torch.einsum("azyx,bzyx->abzyx", L.conj(), D).real / N
        off = G + G.transpose(0, 1)
        ebar -= torch.where(torch.eye(3, device=op.dev)[:, :, None, None, None] > 0, G, off)
        wbar += 2 * omega * s
    return float(wbar), np.ascontiguousarray(ebar[:, :, 0].permute(0, 1, 3, 2).cpu().numpy())


def exact(case, seed):
    r = np.random.RandomState(seed)
    do = case["do"]
    if do == "solve":
        grid, e = _cell(case["family"], case["nx"], case["ny"], r)
        ks, hs = _modes(_Op(grid, e), _omega(r), case["nev"])
        return np.array(ks), [h.cpu().numpy() for h in hs]
    if do == "periodic":
        grid, e = _bragg(case, r)
        ks, hs = _modes(_Op(grid, e), _omega(r), case["nev"])
        return np.array(ks), [h.cpu().numpy() for h in hs]
    if do == "pullback":
        return _exact_pullback(case, r)
    if do == "apply":
        grid, e = _cell(case["family"], case["nx"], case["ny"], r)
        h = torch.tensor(_block(case, r).astype(np.complex128))
        op = _Op(grid, e.astype(np.float32).astype(np.float64))
        return op(2.0 * _omega(r), h.to(op.dev))
    return None  # batches: dozens of eigensolves of this kind; smoothing: minutes of per-pixel rational algebra
