// Adjoint pull-back of solve_k on the device (omb_pullback).
//
// Per band b with mode (k_b, h_b) and cotangents (k̄_b, ē_b) (reference:
// rrule(solve_k), lib/MaxwellEigenmodes/src/solve.jl:213-289; GPU variant
// src/solvers/gpu.jl:292-365):
//   ∂ω²/∂k = 2⟨h|∂M̂/∂k|h⟩                                   (HMₖH pass)
//   (M̂ − ω²) λ = ē − h⟨h,ē⟩,  λ ⟂ h                         (deflated, preconditioned MINRES)
//   D0 = fft(kx_tc h),  Λd = fft(kx_tc λ)                   (H2D passes)
//   ẽ = bfft(ε⁻¹ D0)/N,  λ̃e = bfft(ε⁻¹ Λd)/N                (D2E passes)
//   k̄ₕ = −∇ₖ(mag, m̂, n̂) · (m̄, n̄, māg) from ẽ, λ̃e, h, λ     (one reduction kernel)
//   s = (k̄ + k̄ₕ)/(∂ω²/∂k),  ω̄ += 2ωs
//   ε̄⁻¹ += ε⁻¹_bar(D0/N, Λd + s·D0)                          (one pointwise kernel: the
//          eigenvalue-path term ε⁻¹_bar(d, fft(kx_tc(s h))) is bilinear in D0, so it folds
//          into the same pass)
//
// MINRES (C. C. Paige & M. A. Saunders, SIAM J. Numer. Anal. 12 (1975)) with a symmetric
// positive-definite preconditioner: for a Hermitian operator the Lanczos coefficients and
// Givens rotations are real, only the vectors are complex.  Every vector stays orthogonal to
// h (the right-hand side is, and the preconditioned vector is projected), which deflates the
// eigenvalue ω² of the operator.  All recurrence scalars live in device memory; one
// iteration is a fixed launch sequence replayed from a CUDA graph: the three operator passes and three
// vector kernels, whose last CTA sums the dot products and takes the scalar step.  Every band of the
// pull-back is a row of each launch: a solve is bound by the latency of its launches (a vector of a
// 256² cell is 2 MB, resident in L2), not by bytes, so the bands share it.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "context.h"
#include "vec.cuh"

namespace omb {

constexpr int ADJ_NT = 256;
constexpr int ADJ_BLOCKS = 296;  // 2 × 148 SMs for the streaming vector kernels

struct MinresState {
  double shift;          // ω²
  double beta1, beta, oldb, alfa, dbar, epsln, oldeps, phibar, cs, sn, gamma, delta, phi;
  double dot_ey_r, dot_ey_i, dot_ez_r, dot_ez_i;
  double rtol;
  double phibar_mark;  // phibar at itn_mark (stagnation test)
  int active;          // operator columns of the solve (0 once it is over)
  int itn, maxit, done, status;  // status: 0 running, 1 converged, 2 maxiter, 3 breakdown,
                                 // 4 maxiter with the residual below LOOSE_TOL
  int itn_mark;
  int flat_windows;  // consecutive windows in which phibar did not halve
};

// Below rtol the recurrence residual phibar can flatten at the rounding floor of the FP64
// operator (≈1e-12 of β₁ for right-hand sides dominated by modes near the deflated
// eigenvalue), while the iterate has long converged.  The solve also ends, converged, when
// phibar ≤ STALL_TOL·β₁ and did not halve over the last STALL_WINDOW iterations.
constexpr double STALL_TOL = 1e-10;
constexpr int STALL_WINDOW = 50;
// A solve that reaches its iteration cap is still accepted when its relative residual is
// below √ε₆₄ ≈ 1.5e-8, the default relative tolerance of the reference's GMRES
// (IterativeSolvers `gmres`, lib/MaxwellEigenmodes/src/grads/solve.jl:56-66, which returns
// whatever it reached after maxiter = 1000).
constexpr double LOOSE_TOL = 1.4901161193847656e-08;
// Near-degenerate bands make (M̂ − ω²) ill-conditioned on the complement of the deflated
// eigenvector, and the FP64 recurrence then flattens at ≈ε₆₄·cond above LOOSE_TOL.  A solve
// whose phibar has not halved over FLAT_WINDOWS consecutive windows while below FLAT_TOL·β₁
// ends there, accepted (status 4): more iterations would not lower it.
constexpr double FLAT_TOL = 1e-6;
constexpr int FLAT_WINDOWS = 4;

// Sums of four doubles over the CTA, valid in thread 0 (every thread calls it).
__device__ __forceinline__ void block_sum4(double (&v)[4]) {
  __shared__ double sm[4][ADJ_NT / 32];
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
#pragma unroll
    for (int q = 0; q < 4; ++q) sm[q][w] = v[q];
  __syncthreads();
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      double s = 0;
      for (int i = 0; i < ADJ_NT / 32; ++i) s += sm[q][i];
      v[q] = s;
    }
  __syncthreads();
}

// block-reduce two complex partial sums (4 doubles) into part[blockIdx.x*4 + 0..3]
__device__ __forceinline__ void block_reduce4(double a, double b, double c, double d, double* part) {
  double v[4] = {a, b, c, d};
  block_sum4(v);
  if (threadIdx.x == 0)
#pragma unroll
    for (int q = 0; q < 4; ++q) part[4 * blockIdx.x + q] = v[q];
}

// Arrival of a CTA of row blockIdx.y of the grid: true in every thread of the last one, which resets
// the counter.  What the others wrote before is then visible.
__device__ __forceinline__ bool last_block(unsigned* ticket) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    if (last) *ticket = 0;
  }
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// Grid-wide sums: block partials, then the last CTA adds them with all its threads in a fixed order.
// True in thread 0 of that CTA, with the sums in v.  (One thread adding 296 partials in a kernel of its
// own took ≈10 µs.)
__device__ __forceinline__ bool grid_sum4(double (&v)[4], double* part, unsigned* ticket) {
  block_reduce4(v[0], v[1], v[2], v[3], part);
  if (!last_block(ticket)) return false;
#pragma unroll
  for (int q = 0; q < 4; ++q) v[q] = 0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += ADJ_NT)
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] += __ldcg(part + 4 * i + q);
  block_sum4(v);
  return threadIdx.x == 0;
}

// One band's solve: all bands of a pull-back run together, a row of CTAs (blockIdx.y) each.
struct AdjBand {
  double2 *x, *v, *w, *w2, *r1, *r2, *y, *Av;
  double2* b;        // right-hand side
  const double2* e;  // unit eigenvector (deflation direction)
  double* part;      // partial sums, 4 per CTA
  unsigned* ticket;
  MinresState* S;
  double k;
};
struct AdjGeom {
  int N, Nx, Ny, Nz;  // pixels (two coefficients each); Nz = 1 for a 2D cell
  double inv_dx, inv_dy, inv_dz, eps_mean;
};

// Diagonal preconditioner ⟨ε⟩/|w|² at pixel p (w = k ẑ − G; g_z of the pixel's slab)
__device__ __forceinline__ double prec_scale(unsigned p, const AdjGeom& G, double k) {
  const unsigned rest = p / (unsigned)G.Nx, ix = p - rest * (unsigned)G.Nx;
  const unsigned iz = rest / (unsigned)G.Ny, iy = rest - iz * (unsigned)G.Ny;
  const double gx = freq_index((int)ix, G.Nx) * G.inv_dx, gy = freq_index((int)iy, G.Ny) * G.inv_dy;
  const double wz = k - freq_index((int)iz, G.Nz) * G.inv_dz;
  return G.eps_mean / (gx * gx + gy * gy + wz * wz);
}

__device__ __forceinline__ void dot_acc(double& re, double& im, double2 a, double2 b) {  // += conj(a)·b
  re += a.x * b.x + a.y * b.y;
  im += a.x * b.y - a.y * b.x;
}
// a − c·b for a complex c
__device__ __forceinline__ double2 sub_mul(double2 a, double cr, double ci, double2 b) {
  return make_double2(a.x - (cr * b.x - ci * b.y), a.y - (cr * b.y + ci * b.x));
}

// init: r1 = r2 = b, z = P b, partials ⟨e,z⟩, ⟨b,z⟩ (y holds z); then the scalars
__global__ void __launch_bounds__(ADJ_NT) k_minres_init(const AdjBand* __restrict__ bands, AdjGeom G) {
  const AdjBand V = bands[blockIdx.y];
  double d[4] = {0, 0, 0, 0};
  for (int p = blockIdx.x * ADJ_NT + threadIdx.x; p < G.N; p += gridDim.x * ADJ_NT) {
    const double s = prec_scale(p, G, V.k);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const size_t i = 2 * (size_t)p + c;
      const double2 bb = V.b[i], zero = make_double2(0, 0);
      const double2 z = make_double2(bb.x * s, bb.y * s);
      V.r1[i] = bb; V.r2[i] = bb; V.y[i] = z;
      V.x[i] = zero; V.w[i] = zero; V.w2[i] = zero;
      dot_acc(d[0], d[1], V.e[i], z);
      dot_acc(d[2], d[3], bb, z);
    }
  }
  if (!grid_sum4(d, V.part, V.ticket)) return;
  MinresState* S = V.S;
  S->dot_ez_r = d[0]; S->dot_ez_i = d[1];
  const double b2 = d[2];
  S->itn = 0; S->done = 0; S->status = 0; S->active = 1;
  S->oldb = 0; S->dbar = 0; S->epsln = 0; S->oldeps = 0; S->cs = -1; S->sn = 0;
  if (!(b2 > 0) || !isfinite(b2)) {  // zero right-hand side: λ = 0
    S->beta1 = S->beta = 0; S->phibar = 0; S->done = 1; S->status = 1; S->active = 0;
    return;
  }
  S->beta1 = S->beta = sqrt(b2);
  S->phibar = S->beta1;
  S->phibar_mark = S->beta1;
  S->itn_mark = 0;
  S->flat_windows = 0;
}

// v = (z − ⟨e,z⟩e)/beta  (start of the first iteration)
__global__ void __launch_bounds__(ADJ_NT) k_minres_first_v(const AdjBand* __restrict__ bands, AdjGeom G) {
  const AdjBand V = bands[blockIdx.y];
  const MinresState* S = V.S;
  if (S->done) return;
  const double inv = 1.0 / S->beta, er = S->dot_ez_r, ei = S->dot_ez_i;
  for (int i = blockIdx.x * ADJ_NT + threadIdx.x; i < 2 * G.N; i += gridDim.x * ADJ_NT) {
    const double2 z = sub_mul(V.y[i], er, ei, V.e[i]);
    V.v[i] = make_double2(z.x * inv, z.y * inv);
  }
}

// y = Av − shift·v − (beta/oldb)·r1 ; sums ⟨e,y⟩, ⟨v,y⟩ = alfa (real for a Hermitian operator, v ⟂ e)
__global__ void __launch_bounds__(ADJ_NT) k_minres_a(const AdjBand* __restrict__ bands, AdjGeom G) {
  const AdjBand V = bands[blockIdx.y];
  MinresState* S = V.S;
  if (S->done) return;
  const double sh = S->shift;
  const double c1 = S->itn >= 1 ? S->beta / S->oldb : 0.0;
  double d[4] = {0, 0, 0, 0};
  for (int i = blockIdx.x * ADJ_NT + threadIdx.x; i < 2 * G.N; i += gridDim.x * ADJ_NT) {
    const double2 av = V.Av[i], v = V.v[i], r1 = V.r1[i], e = V.e[i];
    const double2 y = make_double2(av.x - sh * v.x - c1 * r1.x, av.y - sh * v.y - c1 * r1.y);
    V.y[i] = y;
    dot_acc(d[0], d[1], e, y);
    dot_acc(d[2], d[3], v, y);
  }
  if (!grid_sum4(d, V.part, V.ticket)) return;
  S->dot_ey_r = d[0]; S->dot_ey_i = d[1];
  S->alfa = d[2];
}

// Lanczos coefficient β_{k+1} and the Givens rotation of MINRES (all real)
__device__ __forceinline__ void minres_rotate(MinresState* S, double b2) {
  S->oldb = S->beta;
  S->beta = b2 > 0 ? sqrt(b2) : 0.0;
  S->oldeps = S->epsln;
  const double alfa = S->alfa;
  S->delta = S->cs * S->dbar + S->sn * alfa;
  const double gbar = S->sn * S->dbar - S->cs * alfa;
  S->epsln = S->sn * S->beta;
  S->dbar = -S->cs * S->beta;
  double gamma = sqrt(gbar * gbar + S->beta * S->beta);
  if (gamma < 1e-300) gamma = 1e-300;
  S->gamma = gamma;
  S->cs = gbar / gamma;
  S->sn = S->beta / gamma;
  S->phi = S->cs * S->phibar;
  S->phibar = S->sn * S->phibar;
  S->itn++;
  if (!isfinite(S->phibar) || !isfinite(S->phi)) { S->done = 1; S->status = 3; S->active = 0; return; }
  if (S->phibar <= S->rtol * S->beta1) { S->done = 2; S->status = 1; return; }  // finish this update
  if (S->itn - S->itn_mark >= STALL_WINDOW) {
    const bool flat = S->phibar > 0.5 * S->phibar_mark;
    if (S->phibar <= STALL_TOL * S->beta1 && flat) {
      S->done = 2; S->status = 1; return;
    }
    S->flat_windows = flat ? S->flat_windows + 1 : 0;
    if (S->flat_windows >= FLAT_WINDOWS && S->phibar <= FLAT_TOL * S->beta1) {
      S->done = 2; S->status = 4; return;
    }
    S->phibar_mark = S->phibar;
    S->itn_mark = S->itn;
  }
  if (S->beta == 0.0) { S->done = 2; S->status = 1; return; }                   // invariant subspace
  if (S->itn >= S->maxit) { S->done = 2; S->status = S->phibar <= LOOSE_TOL * S->beta1 ? 4 : 2; }
}

// y ← y − ⟨e,y⟩e − (alfa/beta) r2 ; r1 ← r2 ; r2 ← y ; z = P r2 (into y) ; sums ⟨e,z⟩, ⟨r2,z⟩ (the
// square of β_{k+1}: ⟨r2, z − e⟨e,z⟩⟩ = ⟨r2, z⟩ since r2 ⟂ e)
__global__ void __launch_bounds__(ADJ_NT) k_minres_b(const AdjBand* __restrict__ bands, AdjGeom G) {
  const AdjBand V = bands[blockIdx.y];
  MinresState* S = V.S;
  if (S->done) return;
  const double c2 = S->alfa / S->beta, er0 = S->dot_ey_r, ei0 = S->dot_ey_i;
  double d[4] = {0, 0, 0, 0};
  for (int p = blockIdx.x * ADJ_NT + threadIdx.x; p < G.N; p += gridDim.x * ADJ_NT) {
    const double s = prec_scale(p, G, V.k);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const size_t i = 2 * (size_t)p + c;
      const double2 e = V.e[i], r2 = V.r2[i], y = sub_mul(V.y[i], er0, ei0, e);
      const double2 yn = make_double2(y.x - c2 * r2.x, y.y - c2 * r2.y);
      V.r1[i] = r2;
      V.r2[i] = yn;
      const double2 z = make_double2(yn.x * s, yn.y * s);
      V.y[i] = z;
      dot_acc(d[0], d[1], e, z);
      dot_acc(d[2], d[3], yn, z);
    }
  }
  if (!grid_sum4(d, V.part, V.ticket)) return;
  S->dot_ez_r = d[0]; S->dot_ez_i = d[1];
  minres_rotate(S, d[2]);
}

// w_k = (v − oldeps·w_{k−2} − delta·w_{k−1})/gamma ; x += phi·w_k ; v ← (z − ⟨e,z⟩e)/β_{k+1}; a solve
// whose last update this was is then over
__global__ void __launch_bounds__(ADJ_NT) k_minres_c(const AdjBand* __restrict__ bands, AdjGeom G) {
  const AdjBand V = bands[blockIdx.y];
  MinresState* S = V.S;
  if (S->done == 1) return;
  const double ig = 1.0 / S->gamma, oe = S->oldeps, de = S->delta, ph = S->phi;
  const bool next = S->done == 0 && S->beta > 0;
  const double ib = next ? 1.0 / S->beta : 0.0, er = S->dot_ez_r, ei = S->dot_ez_i;
  const bool ends = S->done == 2;
  for (int i = blockIdx.x * ADJ_NT + threadIdx.x; i < 2 * G.N; i += gridDim.x * ADJ_NT) {
    const double2 v = V.v[i], wa = V.w2[i], wb = V.w[i];
    const double2 wn = make_double2((v.x - oe * wa.x - de * wb.x) * ig, (v.y - oe * wa.y - de * wb.y) * ig);
    V.w2[i] = wb;
    V.w[i] = wn;
    double2 x = V.x[i];
    x.x += ph * wn.x; x.y += ph * wn.y;
    V.x[i] = x;
    if (next) {
      const double2 z = sub_mul(V.y[i], er, ei, V.e[i]);
      V.v[i] = make_double2(z.x * ib, z.y * ib);
    }
  }
  if (ends && last_block(V.ticket) && threadIdx.x == 0) { S->done = 1; S->active = 0; }
}

// t ← t − ⟨e,t⟩e for the right-hand sides (t = b) or the solutions (t = x): the sum, then the update
// with it
__global__ void __launch_bounds__(ADJ_NT) k_dot_e(const AdjBand* __restrict__ bands, AdjGeom G, int of_x) {
  const AdjBand V = bands[blockIdx.y];
  const double2* t = of_x ? V.x : V.b;
  double d[4] = {0, 0, 0, 0};
  for (int i = blockIdx.x * ADJ_NT + threadIdx.x; i < 2 * G.N; i += gridDim.x * ADJ_NT) dot_acc(d[0], d[1], V.e[i], t[i]);
  if (!grid_sum4(d, V.part, V.ticket)) return;
  V.S->dot_ey_r = d[0]; V.S->dot_ey_i = d[1];
}
__global__ void __launch_bounds__(ADJ_NT) k_sub_proj(const AdjBand* __restrict__ bands, AdjGeom G, int of_x) {
  const AdjBand V = bands[blockIdx.y];
  double2* t = of_x ? V.x : V.b;
  const double cr = V.S->dot_ey_r, ci = V.S->dot_ey_i;
  for (int i = blockIdx.x * ADJ_NT + threadIdx.x; i < 2 * G.N; i += gridDim.x * ADJ_NT) t[i] = sub_mul(t[i], cr, ci, V.e[i]);
}

// k̄ₕ partials from ẽ = EC/N, λ̃e = ED/N (planar), h and λ (interleaved), basis at k
// (z-periodic cells: the basis at k − g_z, and beside k̄ₕ's sum the same per-plane-wave terms
// weighted by g_z/Λ, whose negative is the eigenvector channel's period cotangent Λ̄_H,
// lib/MaxwellEigenmodes/src/grads/period.jl:113-117, 171-175)
__global__ void __launch_bounds__(ADJ_NT) k_adj_kbar(const double2* __restrict__ EC, const double2* __restrict__ ED,
                                                     const double2* __restrict__ h, const double2* __restrict__ lam,
                                                     int Nx, int Ny, int Nz, double inv_dx, double inv_dy,
                                                     double inv_dz, double k, double* part) {
  const long long N = (long long)Nx * Ny * Nz;
  const double sN = 1.0 / (double)N;
  double acc = 0, accL = 0;
  for (long long p = blockIdx.x * (long long)ADJ_NT + threadIdx.x; p < N; p += (long long)gridDim.x * ADJ_NT) {
    const int ix = (int)(p % Nx);
    const long long rest = p / Nx;
    const int iy = (int)(rest % Ny), iz = (int)(rest / Ny);
    const double gz = freq_index(iz, Nz) * inv_dz;
    const Basis<double> B = basis_at<double>(k - gz, freq_index(ix, Nx) * inv_dx, freq_index(iy, Ny) * inv_dy);
    const double m[3] = {B.mx, B.my, B.mz}, n[3] = {B.nx, B.ny, 0.0};
    const double2 h1 = h[2 * p], h2 = h[2 * p + 1], l1 = lam[2 * p], l2 = lam[2 * p + 1];
    double km[3], kn[3];
    for (int c = 0; c < 3; ++c) {
      const double2 le = ED[c * N + p], ee = EC[c * N + p];
      // Re(λ̃e·conj(h₂) + ẽ·conj(λ₂)) and −Re(λ̃e·conj(h₁) + ẽ·conj(λ₁)), with the 1/N scale
      km[c] = (le.x * h2.x + le.y * h2.y + ee.x * l2.x + ee.y * l2.y) * sN;
      kn[c] = -(le.x * h1.x + le.y * h1.y + ee.x * l1.x + ee.y * l1.y) * sN;
    }
    const double magbar = n[0] * kn[0] + n[1] * kn[1] + n[2] * kn[2] + m[0] * km[0] + m[1] * km[1] + m[2] * km[2];
    // ∇ₖmag_m_n (ME/src/maxwell.jl:560-566) with dk̂ = ẑ: u = (m × n)/mag, q = u × ẑ
    const double u[3] = {(m[1] * n[2] - m[2] * n[1]) / B.mag, (m[2] * n[0] - m[0] * n[2]) / B.mag,
                         (m[0] * n[1] - m[1] * n[0]) / B.mag};
    const double q[3] = {u[1], -u[0], 0.0};
    const double mq[3] = {m[1] * q[2] - m[2] * q[1], m[2] * q[0] - m[0] * q[2], m[0] * q[1] - m[1] * q[0]};
    const double nq[3] = {n[1] * q[2] - n[2] * q[1], n[2] * q[0] - n[0] * q[2], n[0] * q[1] - n[1] * q[0]};
    const double kmag = magbar * u[2] * B.mag;
    const double kmm = -(km[0] * mq[0] + km[1] * mq[1] + km[2] * mq[2]) * B.mag;  // m̄ = kx̄_m·mag
    const double knn = -(kn[0] * nq[0] + kn[1] * nq[1] + kn[2] * nq[2]) * B.mag;
    acc += kmag + kmm + knn;
    accL += (kmag + kmm + knn) * gz * inv_dz;
  }
  block_reduce4(acc, accL, 0, 0, part);
}

// ε̄⁻¹ (6 unique entries) += ε⁻¹_bar(d, lt), d = D0/N, lt = Λd + s·D0
__global__ void __launch_bounds__(ADJ_NT) k_adj_eibar(const double2* __restrict__ D0, const double2* __restrict__ LD,
                                                      long long N, double s, double* __restrict__ eib) {
  const double sN = 1.0 / (double)N;
  for (long long p = blockIdx.x * (long long)ADJ_NT + threadIdx.x; p < N; p += (long long)gridDim.x * ADJ_NT) {
    double2 d[3], l[3];
    for (int c = 0; c < 3; ++c) {
      const double2 a = D0[c * N + p], b = LD[c * N + p];
      d[c] = make_double2(a.x * sN, a.y * sN);
      l[c] = make_double2(b.x + s * a.x, b.y + s * a.y);
    }
    auto re = [](double2 a, double2 b) { return a.x * b.x + a.y * b.y; };  // Re(a·conj(b))
    double* o = eib + 6 * p;
    o[0] -= re(l[0], d[0]);                 // xx
    o[1] -= re(l[1], d[1]);                 // yy
    o[2] -= re(l[2], d[2]);                 // zz
    o[3] -= re(l[1], d[0]) + re(l[0], d[1]);  // xy (summed (x,y)+(y,x), mirrored)
    o[4] -= re(l[2], d[0]) + re(l[0], d[2]);  // xz
    o[5] -= re(l[2], d[1]) + re(l[1], d[2]);  // yz
  }
}

// expand to (3,3,Nx,Ny) and, if requested, ε̄ = −Y ε̄⁻¹ Y with Y = ε⁻¹ (sliceinv_3x3 pull-back,
// ME/src/grads/linalg.jl:40-47; Y is symmetric so Yᵀ = Y)
__global__ void __launch_bounds__(ADJ_NT) k_adj_expand(const double* __restrict__ eib, const double2* __restrict__ e64,
                                                       long long N, double* __restrict__ out_ei, double* __restrict__ out_e) {
  for (long long p = blockIdx.x * (long long)ADJ_NT + threadIdx.x; p < N; p += (long long)gridDim.x * ADJ_NT) {
    const double* o = eib + 6 * p;
    const double Gb[3][3] = {{o[0], o[3], o[4]}, {o[3], o[1], o[5]}, {o[4], o[5], o[2]}};
    for (int a = 0; a < 3; ++a)
      for (int b = 0; b < 3; ++b) out_ei[9 * p + a + 3 * b] = Gb[a][b];
    if (out_e) {
      const double2 y0 = e64[3 * p], y1 = e64[3 * p + 1], y2 = e64[3 * p + 2];
      const double Y[3][3] = {{y0.x, y1.y, y2.x}, {y1.y, y0.y, y2.y}, {y2.x, y2.y, y1.x}};
      double T[3][3];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) T[a][b] = Y[a][0] * Gb[0][b] + Y[a][1] * Gb[1][b] + Y[a][2] * Gb[2][b];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b)
          out_e[9 * p + a + 3 * b] = -(T[a][0] * Y[0][b] + T[a][1] * Y[1][b] + T[a][2] * Y[2][b]);
    }
  }
}

}  // namespace omb

using namespace omb;

// The pull-back on an uploaded problem; Nz > 1 is a z-periodic cell, for which L_bar (when
// non-NULL) receives the period cotangent Λ̄ (lib/MaxwellEigenmodes/src/grads/period.jl:136-200).
static int pullback_impl(omb_ctx* ctx, Problem& P, double omega, int nev, const double* kmags, const double* evecs,
                         const double* kbar, const double* evbar, const omb_options& O, double* omega_bar,
                         double* epsinv_bar, double* eps_bar, double* L_bar, int32_t* iterations) {
  cudaStream_t st = ctx->stream;
  const long long N = (long long)P.N(), n2 = 2 * N;
  const bool periodic = P.Nz > 1;
  for (int b = 0; b < nev; ++b)
    if (!(kmags[b] > 0) || !std::isfinite(kmags[b])) return fail(OMB_ERR_INVALID_ARG, "kmags must be finite and positive");
  const AdjGeom G{(int)N, P.Nx, P.Ny, P.Nz, 1.0 / P.Dx, 1.0 / P.Dy, periodic ? 1.0 / P.Dz : 0.0, P.eps_mean};
  const int rb = row_blocks(P.Nx, P.Ny) * P.Nz;  // HMₖH partials: row blocks of every slab
  DevBuf<double> eib;
  OMB_CU(eib.alloc(6 * N, st));
  OMB_CU(eib.zero());
  double wbar = 0.0, Lbar = 0.0;
  // The bands of a chunk run together: at a few hundred KB to a few MB per vector one band's launches
  // leave most SMs idle.  A band holds up to 10 vectors and 6 planar fields (38·N complex numbers); a
  // chunk is limited to 4 GiB of them, and to what a nearly full device still has (halved until its
  // vectors and fields fit; one band needs no more than this).
  int chunk = (int)std::max<long long>(1, std::min<long long>(nev, ((long long)4 << 30) / (38 * N * (long long)sizeof(double2))));
  for (int b0 = 0, nb = 0; b0 < nev; b0 += nb) {
    nb = std::min(chunk, nev - b0);
    // bands with a field cotangent (the others need no adjoint solve)
    std::vector<int> mb;  // MINRES index → band of the chunk
    for (int j = 0; j < nb && evbar; ++j) {
      const double* h = evbar + 4 * N * (size_t)(b0 + j);
      bool any = false;
      for (long long i = 0; i < 2 * n2 && !any; ++i) any = h[i] != 0.0;
      if (any) mb.push_back(j);
    }
    const int nm = (int)mb.size();
    DevBuf<double2> ev, vecs, scr;
    DevBuf<double> kd, part, hpart, hred;
    DevBuf<MinresState> S;
    DevBuf<unsigned> tick;
    DevBuf<AdjBand> dband;
    cudaError_t ae = ev.alloc(n2 * nb, st);
    if (ae == cudaSuccess) ae = vecs.alloc(9 * n2 * nm, st);  // x v w w2 r1 r2 y Av b
    if (ae == cudaSuccess) ae = scr.alloc(6 * 3 * N * nb, st);
    if (ae == cudaErrorMemoryAllocation && nb > 1) {
      cudaGetLastError();  // (a failed allocation leaves no other trace)
      chunk = (nb + 1) / 2;
      nb = 0;
      continue;
    }
    OMB_CU(ae);
    OMB_CU(kd.alloc(nb, st));
    OMB_CU(hpart.alloc(2 * (size_t)rb * nb, st));
    OMB_CU(hred.alloc(4 * (size_t)nb, st));
    double2* SA = scr.p;                // D0 = fft(kx_tc h), per band of the chunk
    double2* SB = SA + 3 * N * nb;      // Λd = fft(kx_tc λ)
    double2* SC = SB + 3 * N * nb;      // copies consumed by the D2E passes, operator scratch
    double2* SD = SC + 3 * N * nb;
    double2* EC = SD + 3 * N * nb;      // N·ẽ
    double2* ED = EC + 3 * N * nb;      // N·λ̃e
    OMB_CU(cudaMemcpyAsync(kd.p, kmags + b0, nb * sizeof(double), cudaMemcpyHostToDevice, st));
    OMB_CU(cudaMemcpyAsync(ev.p, evecs + 4 * N * (size_t)b0, n2 * nb * sizeof(double2), cudaMemcpyHostToDevice, st));
    // operator units, kind by kind: HMₖH on h; HMₖH with the ẑ× action weighted by g_z/Λ (∂ω²/∂Λ); H2D on
    // h; M̂ on v → Av; H2D on λ; D2E on the two copies
    enum { U_HK = 0, U_HL = 1, U_D0 = 2, U_M = 3, U_LD = 4, U_EC = 5, U_ED = 6, U_KINDS = 7 };
    std::vector<OpUnit<double>> hu(U_KINDS * (size_t)nb);
    std::vector<AdjBand> hband(nm);
    auto unit = [&](int j, const double2* in, double2* out, double2* s) {
      OpUnit<double> u = make_unit<double>(P);
      u.in = in; u.out = out; u.scr = s; u.k_dev = kd.p + j; u.partial = hpart.p + 2 * (size_t)rb * j;
      u.in_cs = n2; u.out_cs = n2; u.scr_cs = 3 * N; u.ncol = 1;
      return u;
    };
    if (nm > 0) {
      OMB_CU(S.alloc(nm, st));
      OMB_CU(tick.alloc(nm, st));
      OMB_CU(tick.zero());
      OMB_CU(dband.alloc(nm, st));
      OMB_CU(part.alloc(4 * (size_t)ADJ_BLOCKS * nm, st));
    }
    for (int j = 0; j < nb; ++j) {
      const double2* e = ev.p + n2 * j;
      hu[U_HK * nb + j] = unit(j, e, nullptr, SC + 3 * N * j);
      hu[U_HL * nb + j] = unit(j, e, nullptr, SC + 3 * N * j);
      hu[U_HL * nb + j].zx_weight_gz = 1;
      hu[U_D0 * nb + j] = unit(j, e, nullptr, SA + 3 * N * j);
    }
    for (int m = 0; m < nm; ++m) {
      const int j = mb[m];
      double2* v0 = vecs.p + 9 * n2 * m;
      hband[m] = AdjBand{v0, v0 + n2, v0 + 2 * n2, v0 + 3 * n2, v0 + 4 * n2, v0 + 5 * n2, v0 + 6 * n2, v0 + 7 * n2,
                         v0 + 8 * n2, ev.p + n2 * j, part.p + 4 * (size_t)ADJ_BLOCKS * m, tick.p + m, S.p + m,
                         kmags[b0 + j]};
      hu[U_M * nb + m] = unit(j, hband[m].v, hband[m].Av, SC + 3 * N * j);
      hu[U_M * nb + m].ncol_dev = &S.p[m].active;
      hu[U_LD * nb + m] = unit(j, hband[m].x, nullptr, SB + 3 * N * j);
      hu[U_EC * nb + m] = unit(j, nullptr, EC + 3 * N * j, SC + 3 * N * j);
      hu[U_ED * nb + m] = unit(j, nullptr, ED + 3 * N * j, SD + 3 * N * j);
      hu[U_EC * nb + m].out_cs = hu[U_ED * nb + m].out_cs = 3 * N;
    }
    DevBuf<OpUnit<double>> du, dexp;
    OMB_CU(du.alloc(hu.size(), st));
    OMB_CU(cudaMemcpyAsync(du.p, hu.data(), hu.size() * sizeof(OpUnit<double>), cudaMemcpyHostToDevice, st));
    if (periodic) OMB_CU(dexp.alloc((size_t)(P.Nz + 1) * nb, st));
    const TwTables& tw = ctx->tw;
    auto run = [&](OpKind kind, int u, int n) -> cudaError_t {
      return periodic ? launch_op3d<double>(kind, du.p + u * nb, n, P.Nx, P.Ny, P.Nz, 1, tw, dexp.p, st)
                      : launch_op<double>(kind, du.p + u * nb, n, P.Nx, P.Ny, 1, tw, st);
    };
    // ∂ω²/∂k = 2⟨h|∂M̂/∂k|h⟩ and, on a periodic cell, ∂ω²/∂Λ = 2⟨h|∂M̂/∂Λ|h⟩ (period.jl:150-151); the device
    // partials hold Re⟨h|kx_ct(…)⟩ = −HMₖH
    const bool want_L = periodic && L_bar;
    std::vector<double> hk(4 * (size_t)nb, 0.0);
    OMB_CU(run(OP_HMKH, U_HK, nb));
    k_reduce_partials<<<nb, 256, 0, st>>>(hpart.p, rb, nb, hred.p);
    OMB_CU(cudaGetLastError());
    if (want_L) {
      OMB_CU(run(OP_HMKH, U_HL, nb));
      k_reduce_partials<<<nb, 256, 0, st>>>(hpart.p, rb, nb, hred.p + 2 * nb);
      OMB_CU(cudaGetLastError());
    }
    OMB_CU(cudaMemcpyAsync(hk.data(), hred.p, (want_L ? 4 : 2) * (size_t)nb * sizeof(double), cudaMemcpyDeviceToHost, st));
    // D0 = fft(kx_tc h) into SA
    OMB_CU(run(OP_H2D, U_D0, nb));
    OMB_CU(cudaStreamSynchronize(st));
    for (int j = 0; j < nb; ++j) {
      const double dw2dk = -2.0 * hk[2 * j];
      if (!(dw2dk > 0) || !std::isfinite(dw2dk)) return fail(OMB_ERR_NAN, "non-positive ∂ω²/∂k in the pull-back");
    }
    std::vector<double> kbar_h(nb, 0.0), Lbar_h(nb, 0.0);
    if (iterations)
      for (int j = 0; j < nb; ++j) iterations[b0 + j] = 0;
    if (nm < nb) OMB_CU(cudaMemsetAsync(SB, 0, 3 * N * nb * sizeof(double2), st));
    if (nm > 0) {
      MinresState s0{};
      s0.shift = omega * omega;
      s0.rtol = 1e-12;
      s0.maxit = std::max(4 * O.maxiter, 3000);
      std::vector<MinresState> hs(nm, s0);
      OMB_CU(cudaMemcpyAsync(S.p, hs.data(), nm * sizeof(MinresState), cudaMemcpyHostToDevice, st));
      OMB_CU(cudaMemcpyAsync(dband.p, hband.data(), nm * sizeof(AdjBand), cudaMemcpyHostToDevice, st));
      for (int m = 0; m < nm; ++m)
        OMB_CU(cudaMemcpyAsync(hband[m].b, evbar + 4 * N * (size_t)(b0 + mb[m]), n2 * sizeof(double2),
                               cudaMemcpyHostToDevice, st));
      const AdjBand* D = dband.p;
      const int nbx = (int)std::min<long long>(ADJ_BLOCKS, (N + ADJ_NT - 1) / ADJ_NT);
      const dim3 gv(nbx, nm);
      // b = ē − h⟨h,ē⟩
      k_dot_e<<<gv, ADJ_NT, 0, st>>>(D, G, 0);
      k_sub_proj<<<gv, ADJ_NT, 0, st>>>(D, G, 0);
      k_minres_init<<<gv, ADJ_NT, 0, st>>>(D, G);
      k_minres_first_v<<<gv, ADJ_NT, 0, st>>>(D, G);
      OMB_CU(cudaGetLastError());
      // one MINRES iteration of every band; 8 per graph replay, host checks the flags between replays
      auto iter = [&]() -> cudaError_t {
        cudaError_t e = run(OP_M, U_M, nm);
        if (e != cudaSuccess) return e;
        k_minres_a<<<gv, ADJ_NT, 0, st>>>(D, G);
        k_minres_b<<<gv, ADJ_NT, 0, st>>>(D, G);
        k_minres_c<<<gv, ADJ_NT, 0, st>>>(D, G);
        return cudaGetLastError();
      };
      OMB_CU(iter());  // eager once (sets kernel attributes outside the capture)
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t exec = nullptr;
      OMB_CU(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
      cudaError_t ce = cudaSuccess;
      for (int i = 0; i < 8 && ce == cudaSuccess; ++i) ce = iter();
      cudaError_t ee = cudaStreamEndCapture(st, &graph);
      if (ce != cudaSuccess) { if (graph) cudaGraphDestroy(graph); return cuda_fail(ce, "MINRES capture"); }
      OMB_CU(ee);
      OMB_CU(cudaGraphInstantiate(&exec, graph, 0));
      const int cap = s0.maxit / 8 + 2;
      for (int it = 0; it < cap; ++it) {
        cudaError_t e = cudaGraphLaunch(exec, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(hs.data(), S.p, nm * sizeof(MinresState), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) { cudaGraphExecDestroy(exec); cudaGraphDestroy(graph); return cuda_fail(e, "MINRES"); }
        bool all = true;
        for (const MinresState& q : hs) all = all && q.done;
        if (all) break;
      }
      cudaGraphExecDestroy(exec);
      cudaGraphDestroy(graph);
      for (int m = 0; m < nm; ++m) {
        const MinresState& sh = hs[m];
        const int b = b0 + mb[m];
        if (iterations) iterations[b] = sh.itn;
        if (sh.status == 3) return fail(OMB_ERR_NAN, "MINRES breakdown in the adjoint solve");
        if (sh.status != 1 && sh.status != 4) {
          char msg[160];
          snprintf(msg, sizeof msg, "adjoint MINRES did not converge (band %d: relative residual %.3g after %d iterations)",
                   b, sh.beta1 > 0 ? sh.phibar / sh.beta1 : 0.0, sh.itn);
          return fail(OMB_ERR_NOT_CONVERGED, msg);
        }
      }
      // λ ⟂ h (re-projection against round-off), then Λd = fft(kx_tc λ) into SB
      k_dot_e<<<gv, ADJ_NT, 0, st>>>(D, G, 1);
      k_sub_proj<<<gv, ADJ_NT, 0, st>>>(D, G, 1);
      OMB_CU(cudaGetLastError());
      OMB_CU(run(OP_H2D, U_LD, nm));
      // ẽ·N and λ̃e·N through the D2E passes on copies (the passes work in place)
      OMB_CU(cudaMemcpyAsync(SC, SA, 3 * N * nb * sizeof(double2), cudaMemcpyDeviceToDevice, st));
      OMB_CU(cudaMemcpyAsync(SD, SB, 3 * N * nb * sizeof(double2), cudaMemcpyDeviceToDevice, st));
      OMB_CU(run(OP_D2E, U_EC, nm));
      OMB_CU(run(OP_D2E, U_ED, nm));
      for (int m = 0; m < nm; ++m) {
        const int j = mb[m];
        k_adj_kbar<<<nbx, ADJ_NT, 0, st>>>(EC + 3 * N * j, ED + 3 * N * j, hband[m].e, hband[m].x, P.Nx, P.Ny, P.Nz,
                                           G.inv_dx, G.inv_dy, G.inv_dz, kmags[b0 + j], hband[m].part);
        OMB_CU(cudaGetLastError());
      }
      std::vector<double> hp(4 * (size_t)ADJ_BLOCKS * nm);
      OMB_CU(cudaMemcpyAsync(hp.data(), part.p, hp.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
      OMB_CU(cudaStreamSynchronize(st));
      for (int m = 0; m < nm; ++m) {
        const double* q = hp.data() + 4 * (size_t)ADJ_BLOCKS * m;
        double acc = 0, accL = 0;
        for (int i = 0; i < nbx; ++i) {
          acc += q[4 * i];
          accL += q[4 * i + 1];
        }
        kbar_h[mb[m]] = -acc;
        Lbar_h[mb[m]] = -accL;
      }
    }
    for (int j = 0; j < nb; ++j) {
      const double dw2dk = -2.0 * hk[2 * j], dw2dL = want_L ? -2.0 * hk[2 * (nb + j)] : 0.0;
      const double kt = (kbar ? kbar[b0 + j] : 0.0) + kbar_h[j], s = kt / dw2dk;
      k_adj_eibar<<<ADJ_BLOCKS, ADJ_NT, 0, st>>>(SA + 3 * N * j, SB + 3 * N * j, N, s, eib.p);
      OMB_CU(cudaGetLastError());
      wbar += 2.0 * omega * s;
      Lbar += Lbar_h[j] + kt * (-dw2dL / dw2dk);
    }
  }
  DevBuf<double> oei, oe;
  OMB_CU(oei.alloc(9 * N, st));
  if (eps_bar) OMB_CU(oe.alloc(9 * N, st));
  k_adj_expand<<<ADJ_BLOCKS, ADJ_NT, 0, st>>>(eib.p, P.e64.p, N, oei.p, eps_bar ? oe.p : nullptr);
  OMB_CU(cudaGetLastError());
  OMB_CU(cudaMemcpyAsync(epsinv_bar, oei.p, 9 * N * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (eps_bar) OMB_CU(cudaMemcpyAsync(eps_bar, oe.p, 9 * N * sizeof(double), cudaMemcpyDeviceToHost, st));
  OMB_CU(cudaStreamSynchronize(st));
  *omega_bar = wbar;
  if (L_bar) *L_bar = Lbar;
  return OMB_OK;
}

static int pullback_args(omb_ctx* ctx, double omega, int nev, const double* kmags, const double* evecs,
                         double* omega_bar, double* epsinv_bar) {
  if (!ctx) return fail(OMB_ERR_INVALID_ARG, "ctx is NULL");
  if (nev <= 0 || !kmags || !evecs || !omega_bar || !epsinv_bar)
    return fail(OMB_ERR_INVALID_ARG, "need nev > 0 and non-NULL kmags, evecs, omega_bar, epsinv_bar");
  if (!(omega > 0) || !std::isfinite(omega)) return fail(OMB_ERR_INVALID_ARG, "omega must be finite and positive");
  return OMB_OK;
}

extern "C" int omb_pullback(omb_ctx* ctx, const omb_grid* grid, double omega, const double* epsinv, int nev,
                            const double* kmags, const double* evecs, const double* kbar, const double* evbar,
                            const omb_options* opt, double* omega_bar, double* epsinv_bar, double* eps_bar,
                            int32_t* iterations) {
  int rc = pullback_args(ctx, omega, nev, kmags, evecs, omega_bar, epsinv_bar);
  if (rc) return rc;
  omb_options dflt;
  omb_options_default(&dflt);
  OMB_CU(cudaSetDevice(ctx->device));
  Problem P;
  rc = upload_problem(ctx, grid, epsinv, P);
  if (rc) return rc;
  return pullback_impl(ctx, P, omega, nev, kmags, evecs, kbar, evbar, opt ? *opt : dflt, omega_bar, epsinv_bar,
                       eps_bar, nullptr, iterations);
}

extern "C" int omb_pullback_periodic(omb_ctx* ctx, const omb_grid3* grid, double omega, const double* epsinv,
                                     int nev, const double* kmags, const double* evecs, const double* kbar,
                                     const double* evbar, const omb_options* opt, double* omega_bar,
                                     double* epsinv_bar, double* L_bar, int32_t* iterations) {
  int rc = pullback_args(ctx, omega, nev, kmags, evecs, omega_bar, epsinv_bar);
  if (rc) return rc;
  if (!grid) return fail(OMB_ERR_INVALID_ARG, "grid is NULL");
  if (grid->Nz < 8) return fail(OMB_ERR_UNSUPPORTED, "a z-periodic cell needs Nz >= 8 slabs (a supported length)");
  omb_options dflt;
  omb_options_default(&dflt);
  OMB_CU(cudaSetDevice(ctx->device));
  Problem P;
  const omb_grid g2{grid->Nx, grid->Ny, grid->Dx, grid->Dy};
  rc = upload_problem(ctx, &g2, epsinv, P, grid->Nz, grid->Dz);
  if (rc) return rc;
  return pullback_impl(ctx, P, omega, nev, kmags, evecs, kbar, evbar, opt ? *opt : dflt, omega_bar, epsinv_bar,
                       nullptr, L_bar, iterations);
}
