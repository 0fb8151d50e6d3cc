// Small dense Hermitian algebra for the Rayleigh–Ritz step, one CTA per problem (FP64).
//
// Matrices live in shared memory, row-major with leading dimension `ld`, complex double.
// The eigensolver is the cyclic Jacobi method for complex Hermitian matrices with the
// round-robin (tournament) ordering of Brent & Luk, so the n/2 rotations of a round act on
// disjoint index pairs.  Each 2×2 rotation first removes the phase of A_pq
// (D = diag(1, e^{-iφ})) and then applies the real symmetric Jacobi rotation with
// t = sign(ζ)/(|ζ| + √(1+ζ²)), ζ = (A_qq − A_pp)/(2|A_pq|) (Golub & Van Loan, Matrix
// Computations, §8.5).  A round is two barriers: one thread per pair computes its rotation
// (reciprocal square roots only, no divisions by |A_pq|), then every element of the new
// matrix is formed from the four old elements it depends on, A' = JᴴAJ, into a second
// buffer, while V ← VJ is updated in place by column pairs.  Sweeps stop when the
// off-diagonal Frobenius norm falls below 1e-13·‖A‖_F (eigenvalue perturbation
// ≲ 1e-26‖A‖²/gap; rounding keeps the off-diagonal near n·1e-16‖A‖, so a tighter test
// would never pass) or after `max_sweeps`.
#pragma once

#include "omb_common.cuh"

namespace omb {

// Per index a of a round: partner pa and the coefficients of the two-sided update,
// (JᴴA)_a· = α_a A_a· + β_a A_pa·  and  (AJ)_·a = γ_a A_·a + δ_a A_·pa.
struct RotIdx { double2 al, be, ga, de; int pa; };

// Round-robin pairing: players 0..ne-1 (ne even); player 0 fixed, the rest rotate.
__device__ __forceinline__ void rr_pair(int round, int i, int ne, int& p, int& q) {
  auto pos = [&](int k) { return k == 0 ? 0 : 1 + ((k - 1 + round) % (ne - 1)); };
  int a = pos(i), b = pos(ne - 1 - i);
  p = a < b ? a : b;
  q = a < b ? b : a;
}

__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// Jacobi eigen-decomposition of the n×n Hermitian matrix A (overwritten with its
// eigenvalues on the diagonal); V (n×n) receives the eigenvectors as columns.
// `A2` is n×n scratch (leading dimension ld), `ri` ≥ n entries, `red` ≥ 2·(warps) doubles.
// Sweeps stop once ‖offdiag‖²_F ≤ tol2·‖A‖²_F.
__device__ inline void jacobi_eigh(double2* A, double2* V, int n, int ld, double2* A2, RotIdx* ri, double* red,
                                   double tol2 = 1e-26, int max_sweeps = 20) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int e = tid; e < n * n; e += nt) {
    const int r = e / n, c = e % n;
    V[r * ld + c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    if (r == c) A[r * ld + c].y = 0.0;
  }
  __syncthreads();
  if (n <= 1) return;
  double2* cur = A;
  double2* nxt = A2;
  const int ne = n + (n & 1);
  const int npair = ne / 2;
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    // convergence check: off-diagonal vs total Frobenius norm
    double off = 0, tot = 0;
    for (int e = tid; e < n * n; e += nt) {
      const int r = e / n, c = e % n;
      const double2 v = cur[r * ld + c];
      const double a2 = v.x * v.x + v.y * v.y;
      tot += a2;
      if (r != c) off += a2;
    }
    for (int o = 16; o > 0; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if ((tid & 31) == 0) { red[2 * (tid >> 5)] = off; red[2 * (tid >> 5) + 1] = tot; }
    __syncthreads();
    double so = 0, st = 0;
    for (int w = 0; w < (nt + 31) / 32; ++w) { so += red[2 * w]; st += red[2 * w + 1]; }
    __syncthreads();
    if (so <= tol2 * st || so == 0.0) break;
    for (int round = 0; round < ne - 1; ++round) {
      // 1. rotations of this round (identity for the odd player out and settled pairs)
      for (int i = tid; i < npair; i += nt) {
        int p, q;
        rr_pair(round, i, ne, p, q);
        const double2 one = make_double2(1.0, 0.0), zero = make_double2(0.0, 0.0);
        RotIdx rp{one, zero, one, zero, q}, rq{one, zero, one, zero, p};
        if (q < n) {
          const double2 apq = cur[p * ld + q];
          const double g2 = apq.x * apq.x + apq.y * apq.y;
          const double app = cur[p * ld + p].x, aqq = cur[q * ld + q].x;
          if (g2 > 1e-300 && g2 > 1e-36 * fabs(app * aqq)) {
            const double rg = rsqrt(g2);                    // 1/|A_pq|
            const double er = apq.x * rg, ei = apq.y * rg;  // e^{iφ}
            const double zeta = 0.5 * (aqq - app) * rg;
            const double h = 1.0 + zeta * zeta;
            const double t = (zeta >= 0 ? 1.0 : -1.0) * __drcp_rn(fabs(zeta) + h * rsqrt(h));
            const double c = rsqrt(1.0 + t * t), sn = t * c;
            // rows:    A_p· ← c A_p· − s e A_q·,    A_q· ← s A_p· + c e A_q·
            // columns: A_·p ← c A_·p − s ē A_·q,    A_·q ← s A_·p + c ē A_·q
            rp.al = make_double2(c, 0.0);         rp.be = make_double2(-sn * er, -sn * ei);
            rq.al = make_double2(c * er, c * ei); rq.be = make_double2(sn, 0.0);
            rp.ga = make_double2(c, 0.0);         rp.de = make_double2(-sn * er, sn * ei);
            rq.ga = make_double2(c * er, -c * ei); rq.de = make_double2(sn, 0.0);
          }
          ri[q] = rq;
        }
        ri[p] = rp;
      }
      __syncthreads();
      // 2. A' = JᴴAJ element by element into the other buffer; V ← VJ by column pairs
      for (int e = tid; e < n * n; e += nt) {
        const int i = e / n, j = e % n;
        const RotIdx a = ri[i], b = ri[j];
        double2 v = zmul(zmul(a.al, cur[i * ld + j]), b.ga);
        if (b.pa < n) v = v + zmul(zmul(a.al, cur[i * ld + b.pa]), b.de);
        if (a.pa < n) {
          v = v + zmul(zmul(a.be, cur[a.pa * ld + j]), b.ga);
          if (b.pa < n) v = v + zmul(zmul(a.be, cur[a.pa * ld + b.pa]), b.de);
        }
        nxt[i * ld + j] = v;
      }
      for (int e = tid; e < n * npair; e += nt) {
        const int i = e / npair, k = e % npair;
        int p, q;
        rr_pair(round, k, ne, p, q);
        if (q >= n) continue;
        const RotIdx rp = ri[p], rq = ri[q];
        const double2 vp = V[i * ld + p], vq = V[i * ld + q];
        V[i * ld + p] = zmul(rp.ga, vp) + zmul(rp.de, vq);
        V[i * ld + q] = zmul(rq.ga, vq) + zmul(rq.de, vp);
      }
      __syncthreads();
      double2* tmp = cur; cur = nxt; nxt = tmp;
    }
  }
  if (cur != A) {
    for (int e = tid; e < n * n; e += nt) A[(e / n) * ld + e % n] = cur[(e / n) * ld + e % n];
    __syncthreads();
  }
  for (int e = tid; e < n; e += nt) A[e * ld + e].y = 0.0;
  __syncthreads();
}

// ---- FP32 Jacobi refined to FP64 ------------------------------------------------------------
//
// A round of the FP64 Jacobi above is a chain of dependent FP64 operations (three reciprocal
// square roots, a reciprocal, two barriers; ≈2.5 K cycles at n = 15), and a matrix needs 6–8
// sweeps of n − 1 rounds.  The sweeps below run on an FP32 copy (one barrier and ≈300 cycles a
// round), and their eigenvectors are then brought to FP64 by the quadratically convergent
// refinement of T. Ogita and K. Aishima ("Iterative refinement for symmetric eigenvalue
// decomposition", Japan J. Indust. Appl. Math. 35, 2018), whose steps are three small matrix
// products in FP64: with R = I − XᴴX, S = XᴴAX and λ_j = S_jj/(1 − R_jj),
//   E_ij = (S_ij + λ_j R_ij)/(λ_j − λ_i)  (i ≠ j),  E_jj = R_jj/2,  X ← X(I + E).
// The error after a step is of the order of ‖E‖², so the step whose largest |E_ij| is below
// `tol_e` is the last one.  Where a wanted pair is too close for the first-order formula
// (|E_ij| > E_MAX) the caller falls back to the FP64 Jacobi.
constexpr int EIG_NT = 256;          // threads: a 16×16 map over matrix elements
// sweeps end once every rotation had tan² ≤ JAC32_ANGLE2 or |A_pq|² ≤ JAC32_NOISE2·‖A‖²
constexpr float JAC32_ANGLE2 = 1e-6f, JAC32_NOISE2 = 2e-13f;
constexpr double E_MAX = 0.1;

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
struct Rot32 { float c, s, er, ei; };  // rows: p ← c p − s e q, q ← s p + c e q; columns with ē

// The rotation that annihilates A_pq (identity when it is below the FP32 noise of a unit-norm
// matrix); `big` reports a rotation that another sweep has to follow.
__device__ __forceinline__ Rot32 rot32(float2 apq, float app, float aqq, bool& big) {
  const float g2 = apq.x * apq.x + apq.y * apq.y;
  Rot32 r{1.f, 0.f, 1.f, 0.f};
  if (g2 > 1e-17f) {
    const float rg = rsqrtf(g2);
    r.er = apq.x * rg;
    r.ei = apq.y * rg;
    const float zeta = 0.5f * (aqq - app) * rg;
    const float h = 1.f + zeta * zeta;
    const float t = copysignf(__fdividef(1.f, fabsf(zeta) + h * rsqrtf(h)), zeta);
    r.c = rsqrtf(1.f + t * t);
    r.s = t * r.c;
    if (t * t > JAC32_ANGLE2 && g2 > JAC32_NOISE2) big = true;
  }
  return r;
}
// column k of the pair list of a round: index 0 stays, the others rotate (round < ne − 1)
__device__ __forceinline__ int pair_pos(int k, int round, int ne) {
  if (k == 0) return 0;
  const int x = k - 1 + round;
  return 1 + (x >= ne - 1 ? x - (ne - 1) : x);
}

// Eigenvectors of the ne×ne (even; zero-padded) unit-norm Hermitian matrix `A` into V, the
// eigenvalues on the diagonal of the buffer returned; A2 is scratch.  Thread items: the 2×2
// blocks (pair, pair) of A, formed into the other buffer from their four old elements, and the
// (pair, row) entries of V, updated in place; each thread computes the rotations it needs from
// the old matrix, so a round is one barrier.
__device__ inline float2* jacobi32(float2* A, float2* A2, float2* V, int ne, int ldf) {
  const int tid = threadIdx.x;
  const int np = ne / 2, na = np * np, items = na + np * ne;
  constexpr int SLOTS = 4;  // ne ≤ 36: na + np·ne ≤ 972
  int ij[SLOTS];
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int e = tid + q * EIG_NT;
    const int w = e < na ? np : ne, b = e < na ? e : e - na;
    ij[q] = e < items ? (b / w) | ((b % w) << 8) | (e < na ? 0 : 1 << 16) : -1;
  }
  float2* cur = A;
  float2* nxt = A2;
  for (int sweep = 0; sweep < 9; ++sweep) {
    bool big = false;
    for (int round = 0; round < ne - 1; ++round) {
#pragma unroll
      for (int q = 0; q < SLOTS; ++q) {
        if (ij[q] < 0) break;
        const int I = ij[q] & 255, J = (ij[q] >> 8) & 255;
        const int p = pair_pos(I, round, ne), s = pair_pos(ne - 1 - I, round, ne);
        const Rot32 a = rot32(cur[p * ldf + s], cur[p * ldf + p].x, cur[s * ldf + s].x, big);
        const float2 ea = make_float2(a.er, a.ei), eac = make_float2(a.er, -a.ei);
        if (ij[q] >> 16) {
          const float2 vp = V[J * ldf + p], vs = cmulf(V[J * ldf + s], eac);
          V[J * ldf + p] = make_float2(a.c * vp.x - a.s * vs.x, a.c * vp.y - a.s * vs.y);
          V[J * ldf + s] = make_float2(a.s * vp.x + a.c * vs.x, a.s * vp.y + a.c * vs.y);
        } else {
          const int u = pair_pos(J, round, ne), v = pair_pos(ne - 1 - J, round, ne);
          const Rot32 b = rot32(cur[u * ldf + v], cur[u * ldf + u].x, cur[v * ldf + v].x, big);
          const float2 ebc = make_float2(b.er, -b.ei);
          const float2 pu = cur[p * ldf + u], pv = cmulf(cur[p * ldf + v], ebc);
          const float2 su = cmulf(cur[s * ldf + u], ea), sv = cmulf(cmulf(cur[s * ldf + v], ebc), ea);
          // columns, then rows
          const float2 p1 = make_float2(b.c * pu.x - b.s * pv.x, b.c * pu.y - b.s * pv.y);
          const float2 p2 = make_float2(b.s * pu.x + b.c * pv.x, b.s * pu.y + b.c * pv.y);
          const float2 s1 = make_float2(b.c * su.x - b.s * sv.x, b.c * su.y - b.s * sv.y);
          const float2 s2 = make_float2(b.s * su.x + b.c * sv.x, b.s * su.y + b.c * sv.y);
          const bool diag = I == J;
          const float2 z = make_float2(0.f, 0.f);
          nxt[p * ldf + u] = make_float2(a.c * p1.x - a.s * s1.x, diag ? 0.f : a.c * p1.y - a.s * s1.y);
          nxt[p * ldf + v] = diag ? z : make_float2(a.c * p2.x - a.s * s2.x, a.c * p2.y - a.s * s2.y);
          nxt[s * ldf + u] = diag ? z : make_float2(a.s * p1.x + a.c * s1.x, a.s * p1.y + a.c * s1.y);
          nxt[s * ldf + v] = make_float2(a.s * p2.x + a.c * s2.x, diag ? 0.f : a.s * p2.y + a.c * s2.y);
        }
      }
      __syncthreads();
      float2* t = cur; cur = nxt; nxt = t;
    }
    if (!__syncthreads_or(big)) break;
  }
  return cur;
}

// Eigen-decomposition of the n×n Hermitian T (leading dimension ld, kept): the columns of the
// matrix returned (X or Y) are the eigenvectors in ascending order up to rounding, lam their
// eigenvalues.  W holds ld·(n + 1) double2 and is scratch, as is Y (the same size).  Returns nullptr where
// the refinement does not apply (non-finite or zero T; a pair with one of the lowest M columns too
// close to be separated).  TL: 16×16 tiles per dimension covering n.
template <int TL>
__device__ inline double2* eigh_refined(const double2* T, double2* X, double2* Y, double2* W, int n, int M,
                                        int ld, double* lam, double* red, int* order, double tol_e) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int ne = n + (n & 1), ldf = ne | 1;
  // unit-norm FP32 copy, padded to an even size
  double tot = 0;
#pragma unroll
  for (int a = 0; a < TL; ++a)
#pragma unroll
    for (int b = 0; b < TL; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      if (i < n && j < n) { const double2 v = T[i * ld + j]; tot += v.x * v.x + v.y * v.y; }
    }
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if ((tid & 31) == 0) red[tid >> 5] = tot;
  __syncthreads();
  tot = 0;
#pragma unroll
  for (int w = 0; w < EIG_NT / 32; ++w) tot += red[w];
  if (!(tot > 0) || !isfinite(tot)) return nullptr;
  const double scale = rsqrt(tot);
  float2* A = reinterpret_cast<float2*>(W);
  float2* A2 = A + ne * ldf;
  float2* V = reinterpret_cast<float2*>(Y);
  for (int i = ty; i < ne; i += 16)
    for (int j = tx; j < ne; j += 16) {
      const bool in = i < n && j < n;
      const double2 v = in ? T[i * ld + j] : make_double2(0, 0);
      A[i * ldf + j] = make_float2((float)(v.x * scale), (float)(v.y * scale));
      V[i * ldf + j] = make_float2(i == j ? 1.f : 0.f, 0.f);
    }
  __syncthreads();
  const float2* D = jacobi32(A, A2, V, ne, ldf);
  // ascending order of the FP32 eigenvalues (the padding column is never moved, index n)
  if (tid < n) {
    const float d = D[tid * ldf + tid].x;
    int rank = 0;
    for (int j = 0; j < n; ++j) {
      const float dj = D[j * ldf + j].x;
      rank += dj < d || (dj == d && j < tid);
    }
    order[rank] = tid;
  }
  __syncthreads();
  for (int i = ty; i < n; i += 16)
    for (int j = tx; j < n; j += 16) {
      const float2 v = V[i * ldf + order[j]];
      X[i * ld + j] = make_double2((double)v.x, (double)v.y);
    }
  __syncthreads();
  double2* E = W;
  for (int step = 0; step < 6; ++step) {
    // Y = T X and R = I − XᴴX (into E)
    double2 t1[TL][TL], t2[TL][TL];
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) t1[a][b] = t2[a][b] = make_double2(0, 0);
#pragma unroll 2
    for (int k = 0; k < n; ++k) {
      double2 xj[TL];
#pragma unroll
      for (int b = 0; b < TL; ++b) xj[b] = tx + 16 * b < n ? X[k * ld + tx + 16 * b] : make_double2(0, 0);
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = ty + 16 * a;
        if (i >= n) continue;
        const double2 tik = T[i * ld + k], xi = X[k * ld + i];
#pragma unroll
        for (int b = 0; b < TL; ++b) {
          t1[a][b] = cmac(t1[a][b], tik, xj[b]);
          t2[a][b].x += xi.x * xj[b].x + xi.y * xj[b].y;  // conj(X_ki)·X_kj
          t2[a][b].y += xi.x * xj[b].y - xi.y * xj[b].x;
        }
      }
    }
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i < n && j < n) {
          Y[i * ld + j] = t1[a][b];
          t2[a][b] = make_double2((i == j ? 1.0 : 0.0) - t2[a][b].x, -t2[a][b].y);
        }
      }
    __syncthreads();
    // S = XᴴY (kept in t1); λ from its diagonal
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) t1[a][b] = make_double2(0, 0);
#pragma unroll 2
    for (int k = 0; k < n; ++k) {
      double2 yj[TL];
#pragma unroll
      for (int b = 0; b < TL; ++b) yj[b] = tx + 16 * b < n ? Y[k * ld + tx + 16 * b] : make_double2(0, 0);
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = ty + 16 * a;
        if (i >= n) continue;
        const double2 xi = X[k * ld + i];
#pragma unroll
        for (int b = 0; b < TL; ++b) {
          t1[a][b].x += xi.x * yj[b].x + xi.y * yj[b].y;
          t1[a][b].y += xi.x * yj[b].y - xi.y * yj[b].x;
        }
      }
    }
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i == j && i < n) lam[i] = t1[a][b].x / (1.0 - t2[a][b].x);
      }
    __syncthreads();
    bool more = false, bad = false;
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i >= n || j >= n) continue;
        const double2 s = t1[a][b], r = t2[a][b];
        double2 e = make_double2(0.5 * r.x, 0.5 * r.y);
        if (i != j) {
          const double lj = lam[j], inv = 1.0 / (lj - lam[i]);
          const double2 f = make_double2((s.x + lj * r.x) * inv, (s.y + lj * r.y) * inv);
          const double f1 = fabs(f.x) + fabs(f.y);
          if (f1 <= E_MAX) e = f;             // (false for a NaN or infinite quotient)
          else if (i < M || j < M) bad = true;  // unwanted close pairs may stay mixed
        } else {
          e.y = 0;
        }
        const double e1 = fabs(e.x) + fabs(e.y);
        if (!(e1 <= E_MAX)) bad = true;
        if (e1 > tol_e) more = true;
        E[i * ld + j] = e;
      }
    if (__syncthreads_or(bad)) return nullptr;
    // X ← X + X E, into Y
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        t1[a][b] = i < n && j < n ? X[i * ld + j] : make_double2(0, 0);
      }
#pragma unroll 2
    for (int k = 0; k < n; ++k) {
      double2 ej[TL];
#pragma unroll
      for (int b = 0; b < TL; ++b) ej[b] = tx + 16 * b < n ? E[k * ld + tx + 16 * b] : make_double2(0, 0);
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = ty + 16 * a;
        if (i >= n) continue;
        const double2 xi = X[i * ld + k];
#pragma unroll
        for (int b = 0; b < TL; ++b) t1[a][b] = cmac(t1[a][b], xi, ej[b]);
      }
    }
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i < n && j < n) Y[i * ld + j] = t1[a][b];
      }
    more = __syncthreads_or(more);
    double2* t = X; X = Y; Y = t;
    if (!more) return X;
  }
  return nullptr;
}

// Indices of the eigenvalues (diagonal of A) in ascending order → order[0..n).
__device__ inline void sort_diag(const double2* A, int n, int ld, int* order) {
  if (threadIdx.x == 0) {
    for (int i = 0; i < n; ++i) order[i] = i;
    for (int i = 1; i < n; ++i) {
      int v = order[i], j = i - 1;
      while (j >= 0 && A[order[j] * ld + order[j]].x > A[v * ld + v].x) { order[j + 1] = order[j]; --j; }
      order[j + 1] = v;
    }
  }
  __syncthreads();
}

}  // namespace omb
