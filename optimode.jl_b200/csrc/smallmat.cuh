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

#include <cmath>

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

// Position of entry i of the n values at(0), …, at(n − 1) in ascending order, ties by index and NaNs
// counted as +∞: the positions are a permutation of 0..n−1 whatever the values are, so an index read
// back from a table filled by them is always one of the n.
template <typename F> __host__ __device__ __forceinline__ int rank_of(const F& at, int n, int i) {
  using V = decltype(at(0));
  auto key = [&](int j) { const V v = at(j); return v == v ? v : (V)INFINITY; };
  const V d = key(i);
  int r = 0;
  for (int j = 0; j < n; ++j) {
    const V e = key(j);
    r += e < d || (e == d && j < i);
  }
  return r;
}

// ---- FP32 Jacobi refined to FP64 ------------------------------------------------------------
//
// A round of the FP64 Jacobi above is a chain of dependent FP64 operations (three reciprocal
// square roots, a reciprocal, two barriers; ≈2.5 K cycles at n = 15), and a matrix needs 6–8
// sweeps of n − 1 rounds.  The sweeps below run on an FP32 copy (≈470 cycles a
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

// acc + conj(a)·b as a chain of two FMAs per half (like cmac)
__device__ __forceinline__ double2 cmacc(double2 c, double2 a, double2 b) {
  return make_double2(fma(a.y, b.y, fma(a.x, b.x, c.x)), fma(-a.y, b.x, fma(a.x, b.y, c.y)));
}
// c·a + w·b (c real)
__device__ __forceinline__ float2 rotf(float c, float2 a, float2 w, float2 b) {
  return make_float2(fmaf(-w.y, b.y, fmaf(w.x, b.x, c * a.x)), fmaf(w.y, b.x, fmaf(w.x, b.y, c * a.y)));
}
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Shared-memory accesses by 32-bit address.
__device__ __forceinline__ float lds1(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ float4 lds4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts2(uint32_t a, float2 v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sts4(uint32_t a, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// rows: p ← c p − w q, q ← w̄ p + c q;  columns: p ← c p − w̄ q, q ← w p + c q
struct Rot32 { float c; float2 w; };

// The rotation that annihilates A_pq of a unit-norm matrix: with d = A_qq − A_pp and
// h = √(d² + 4|A_pq|²), c² = (1 + |d|/h)/2 and w = sign(d)·A_pq/(h c) — two reciprocal square roots in
// sequence and no branch, so that the two rotations a thread needs overlap (1e-9 added to |d| makes
// equal entries with A_pq = 0 the identity).  `big` reports one that another sweep has to follow.
__device__ __forceinline__ Rot32 rot32(float2 apq, float app, float aqq, bool& big) {
  const float g2 = fmaf(apq.x, apq.x, apq.y * apq.y), d = aqq - app, ad = fabsf(d) + 1e-9f;
  const float rh = rsqrt_ftz(fmaf(ad, ad, 4.f * g2));
  const float c2 = fmaf(0.5f * ad, rh, 0.5f);
  const float rc = rsqrt_ftz(c2);
  const float f = copysignf(rh * rc, d);
  big |= (g2 > JAC32_NOISE2) & (g2 * f * f > JAC32_ANGLE2 * c2);
  return Rot32{c2 * rc, make_float2(f * apq.x, f * apq.y)};
}

// The dynamic shared memory of k_rr; its matrices are addressed as offsets into it (an offset can be
// swapped between buffers and the accesses stay shared-space ones).
extern __shared__ __align__(16) unsigned char rr_smem_raw[];

// Eigenvectors of the ne×ne (even; zero-padded) unit-norm Hermitian matrix at float2 offset oA into
// oV, the eigenvalues on the diagonal of the matrix at the offset returned; the ne·ldf elements
// after each are scratch (the other buffer).  Rows and columns are kept in the order of the
// tournament, whose players all move to the next position after a round: position k always meets
// ne − 1 − k, an element is read from one buffer and written at its next position in the other, so
// every address is fixed, and a sweep of ne − 1 rounds ends in the order it began with.  A round is
// two barriers: one thread per pair computes its rotation, then each thread takes the 2×2 blocks
// (pair, pair) of A and the (pair, row) entries of V that are its items.  What counts is the number of
// instructions in a warp's chain (≈4 cycles each): 10 K / 35 K / 284 K cycles
// per matrix at n = 6 / 15 / 36, against 12 K / 53 K / 339 K with each thread working out its rotations and
// addresses by itself in one-barrier rounds.
template <int TL>
__device__ inline int jacobi32(int oA, int oV, int ne, int ldf, float4* rots) {
  const int tid = threadIdx.x;
  const int np = ne / 2, na = np * np, v0 = (na + 31) & ~31;  // (whole warps take one kind of item)
  constexpr int SLOTS = TL == 1 ? 1 : TL == 2 ? 3 : 4;        // ne ≤ 36: v0 + np·ne ≤ 1000
  auto nx = [&](int k) { return k == 0 ? 0 : (k == ne - 1 ? 1 : k + 1); };
  const uint32_t smem = (uint32_t)__cvta_generic_to_shared(rr_smem_raw), srot = (uint32_t)__cvta_generic_to_shared(rots);
  const uint32_t sA = smem + 8 * oA, sV = smem + 8 * oV;
  const bool pair = tid < np;
  const int kp = pair ? tid : 0, ks = ne - 1 - kp;
  const uint32_t r_ps = sA + 8 * (kp * ldf + ks), r_pp = sA + 8 * (kp * ldf + kp), r_ss = sA + 8 * (ks * ldf + ks);
  // items: rotation addresses, the elements read (A: the block's corners; V: two) and written
  uint32_t qa[SLOTS], qb[SLOTS], r_e[SLOTS][4], w_e[SLOTS][4];
  int kind[SLOTS];
#pragma unroll
  for (int q = 0; q < SLOTS; ++q) {
    const int e = tid + q * EIG_NT, ev = e - v0;
    kind[q] = e < na ? 1 : (ev >= 0 && ev < np * ne ? 2 : 0);
    const int I = e < na ? e / np : ev / ne, J = e < na ? e % np : ev % ne;
    const int p = I, s = ne - 1 - I, u = J, v = ne - 1 - J;
    qa[q] = srot + 16 * I;
    qb[q] = srot + 16 * J;
    if (e < na) {
      r_e[q][0] = sA + 8 * (p * ldf + u); r_e[q][1] = sA + 8 * (p * ldf + v);
      r_e[q][2] = sA + 8 * (s * ldf + u); r_e[q][3] = sA + 8 * (s * ldf + v);
      w_e[q][0] = sA + 8 * (nx(p) * ldf + nx(u)); w_e[q][1] = sA + 8 * (nx(p) * ldf + nx(v));
      w_e[q][2] = sA + 8 * (nx(s) * ldf + nx(u)); w_e[q][3] = sA + 8 * (nx(s) * ldf + nx(v));
    } else {
      r_e[q][0] = sV + 8 * (J * ldf + p); r_e[q][1] = sV + 8 * (J * ldf + s);
      w_e[q][0] = sV + 8 * (J * ldf + nx(p)); w_e[q][1] = sV + 8 * (J * ldf + nx(s));
      r_e[q][2] = r_e[q][3] = w_e[q][2] = w_e[q][3] = 0;
    }
  }
  uint32_t from = 0, to = 8 * ne * ldf;  // offsets of the buffer read and the one written
  for (int sweep = 0; sweep < 9; ++sweep) {
    bool big = false;
#pragma unroll 1
    for (int round = 0; round < ne - 1; ++round) {
      if (pair) {
        const float2 aps = lds2(r_ps + from);
        const float app = lds1(r_pp + from), ass = lds1(r_ss + from);
        const Rot32 r = rot32(aps, app, ass, big);
        sts4(srot + 16 * kp, make_float4(r.c, r.w.x, r.w.y, 0.f));
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < SLOTS; ++q) {
        if (kind[q] == 0) continue;
        const float4 a = lds4(qa[q]);
        const float2 e0 = lds2(r_e[q][0] + from), e1 = lds2(r_e[q][1] + from);
        const float2 aw = make_float2(a.y, a.z), ac = make_float2(a.y, -a.z);  // w, w̄
        const float2 awn = make_float2(-a.y, -a.z), acn = make_float2(-a.y, a.z);
        if (kind[q] == 2) {
          sts2(w_e[q][0] + to, rotf(a.x, e0, acn, e1));
          sts2(w_e[q][1] + to, rotf(a.x, e1, aw, e0));
        } else {
          const float4 b = lds4(qb[q]);
          const float2 e2 = lds2(r_e[q][2] + from), e3 = lds2(r_e[q][3] + from);
          const float2 bw = make_float2(b.y, b.z), bcn = make_float2(-b.y, b.z);
          // columns, then rows (the annihilated pair is left at its rounding, below the noise that
          // ends the sweeps)
          const float2 p1 = rotf(b.x, e0, bcn, e1), p2 = rotf(b.x, e1, bw, e0);
          const float2 s1 = rotf(b.x, e2, bcn, e3), s2 = rotf(b.x, e3, bw, e2);
          sts2(w_e[q][0] + to, rotf(a.x, p1, awn, s1));
          sts2(w_e[q][1] + to, rotf(a.x, p2, awn, s2));
          sts2(w_e[q][2] + to, rotf(a.x, s1, ac, p1));
          sts2(w_e[q][3] + to, rotf(a.x, s2, ac, p2));
        }
      }
      __syncthreads();
      const uint32_t t = from; from = to; to = t;
    }
    if (!__syncthreads_or(big)) break;
  }
  return (int)(from / 8);
}

// Eigen-decomposition of the n×n Hermitian T (leading dimension ld, kept): the columns of the
// matrix whose offset is returned (oX or oY) are the eigenvectors in ascending order up to rounding,
// lam their eigenvalues.  Offsets count double2 in rr_smem_raw; W and Y hold ld·(n + 1) of them and
// are scratch.  Returns −1 where
// the refinement does not apply (non-finite or zero T; a pair with one of the lowest M columns too
// close to be separated).  TL: 16×16 tiles per dimension covering n.
template <int TL>
__device__ inline int eigh_refined(int oT, int oX, int oY, int oW, int n, int M, int ld, double* lam,
                                   float* red, float4* rots, int* order, double tol_e) {
  double2* const sm = reinterpret_cast<double2*>(rr_smem_raw);
  const double2* const T = sm + oT;
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
  float totf = (float)tot;
  for (int o = 16; o > 0; o >>= 1) totf += __shfl_xor_sync(0xffffffffu, totf, o);
  if ((tid & 31) == 0) red[tid >> 5] = totf;
  __syncthreads();
  totf = 0;
#pragma unroll
  for (int w = 0; w < EIG_NT / 32; ++w) totf += red[w];
  if (!(totf > 1e-30f && totf < 1e30f)) return -1;
  const double scale = rsqrtf(totf);
  float2* const smf = reinterpret_cast<float2*>(rr_smem_raw);
  float2* A = smf + 2 * oW;
  float2* V = smf + 2 * oY;
  for (int i = ty; i < ne; i += 16)
    for (int j = tx; j < ne; j += 16) {
      const bool in = i < n && j < n;
      const double2 v = in ? T[i * ld + j] : make_double2(0, 0);
      A[i * ldf + j] = make_float2((float)(v.x * scale), (float)(v.y * scale));
      V[i * ldf + j] = make_float2(i == j ? 1.f : 0.f, 0.f);
    }
  __syncthreads();
  const int at = jacobi32<TL>(2 * oW, 2 * oY, ne, ldf, rots);
  const float2* D = A + at;
  V += at;
  // ascending order of the FP32 eigenvalues (the padding stays at index n)
  if (tid < n) order[rank_of([&](int j) { return D[j * ldf + j].x; }, n, tid)] = tid;
  __syncthreads();
  for (int i = ty; i < n; i += 16)
    for (int j = tx; j < n; j += 16) {
      const float2 v = V[i * ldf + order[j]];
      sm[oX + i * ld + j] = make_double2((double)v.x, (double)v.y);
    }
  __syncthreads();
  double2* const E = sm + oW;
  for (int step = 0; step < 6; ++step) {
    const double2* X = sm + oX;
    double2* Y = sm + oY;
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
      for (int b = 0; b < TL; ++b) xj[b] = X[k * ld + min(tx + 16 * b, n - 1)];
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = min(ty + 16 * a, n - 1);  // (threads outside the matrix repeat an edge)
        const double2 tik = T[i * ld + k], xi = X[k * ld + i];
#pragma unroll
        for (int b = 0; b < TL; ++b) {
          t1[a][b] = cmac(t1[a][b], tik, xj[b]);
          t2[a][b] = cmacc(t2[a][b], xi, xj[b]);
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
      for (int b = 0; b < TL; ++b) yj[b] = Y[k * ld + min(tx + 16 * b, n - 1)];
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = min(ty + 16 * a, n - 1);  // (threads outside the matrix repeat an edge)
        const double2 xi = X[k * ld + i];
#pragma unroll
        for (int b = 0; b < TL; ++b) {
          t1[a][b] = cmacc(t1[a][b], xi, yj[b]);
        }
      }
    }
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i == j && i < n) lam[i] = t1[a][b].x * (1.0 + t2[a][b].x);  // 1/(1 − R_jj) to second order
      }
    __syncthreads();
    bool more = false, bad = false;
    // one thread per pair i < j: E_ji = conj(R_ij − E_ij), the same formula with S and R taken as exactly
    // Hermitian.  (From the two roundings of S_ij and S_ji the columns of a pair would be orthogonal only to
    // ε‖T‖/|λ_j − λ_i|: 1e-10 for a pair 1e-5 apart.)
#pragma unroll
    for (int a = 0; a < TL; ++a)
#pragma unroll
      for (int b = 0; b < TL; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        if (i > j || i >= n || j >= n) continue;
        const double2 s = t1[a][b], r = t2[a][b];
        double2 e = make_double2(0.5 * r.x, i == j ? 0.0 : 0.5 * r.y);
        if (i != j) {
          const double lj = lam[j];
          const double inv = (double)__frcp_rn((float)(lj - lam[i]));  // (a relative error of 1e-7: 1e-15 in a last step)
          const double2 f = make_double2((s.x + lj * r.x) * inv, (s.y + lj * r.y) * inv);
          const double f1 = fabs(f.x) + fabs(f.y);
          if (f1 <= E_MAX) e = f;             // (false for a NaN or infinite quotient)
          else if (i < M || j < M) bad = true;  // unwanted close pairs may stay mixed
        }
        const double2 h = i == j ? e : make_double2(r.x - e.x, e.y - r.y);
        const double e1 = fmax(fabs(e.x) + fabs(e.y), fabs(h.x) + fabs(h.y));
        if (!(e1 <= E_MAX)) bad = true;
        if (e1 > tol_e) more = true;
        E[i * ld + j] = e;
        E[j * ld + i] = h;
      }
    if (__syncthreads_or(bad)) return -1;
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
      for (int b = 0; b < TL; ++b) ej[b] = E[k * ld + min(tx + 16 * b, n - 1)];
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = min(ty + 16 * a, n - 1);  // (threads outside the matrix repeat an edge)
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
    const int o = oX; oX = oY; oY = o;
    if (!more) return oX;
  }
  return -1;
}

}  // namespace omb
