// Rayleigh–Ritz, control and Newton kernels of the device LOBPCG (FP64, precision-agnostic).
#include "lobpcg.cuh"

namespace omb {

// The track's summed Gram matrices G = ZᴴZ and S = ZᴴAZ (upper triangles), scaled to unit
// diagonal of G, and their reduction to the standard problem T = L⁻¹SL⁻ᴴ with G = LLᴴ.  Thread
// (ty, tx) holds the elements (ty + 16a, tx + 16b) of G, S and Z in registers; step j eliminates
// column j from all three at once (G ← its Schur complement, S ← E_j S E_jᴴ, Z ← Z E_jᴴ, so that Z
// ends as L⁻ᴴ up to the pivots' roots): the only data exchanged are the three columns j, published
// by their owners in a double-buffered shared copy, so a step is one barrier and the factorisation
// and both triangular solves are n steps instead of 3n.  T (Hermitian) and Z go to shared memory.
// Returns false when a pivot falls to the floor (near-dependent directions).
struct RRCols { double2 g[2][NMAX], s[2][NMAX], z[2][NMAX]; double d[2][NMAX]; };
template <int TL>
__device__ __forceinline__ bool rr_reduce(const double2* __restrict__ acc, int n, int ld, double drop, RRCols& col,
                                          double* dsc, double2* T, double2* Z) {
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  double2 g[TL][TL], s[TL][TL], z[TL][TL];
#pragma unroll
  for (int a = 0; a < TL; ++a)
#pragma unroll
    for (int b = 0; b < TL; ++b) {
      const int i = ty + 16 * a, k = tx + 16 * b;
      g[a][b] = s[a][b] = z[a][b] = make_double2(0, 0);
      if (i >= n || k >= n) continue;
      const int lo = min(i, k), hi = max(i, k);
      const double gi = acc[i * NMAX + i].x, gk = acc[k * NMAX + k].x;
      const double di = gi > 0 && isfinite(gi) ? rsqrt(gi) : 0.0, dk = gk > 0 && isfinite(gk) ? rsqrt(gk) : 0.0;
      const double2 vg = acc[lo * NMAX + hi], vs = acc[NMAX * NMAX + lo * NMAX + hi];
      const double f = di * dk, sg = i < k ? f : (i > k ? -f : 0.0);
      g[a][b] = make_double2(vg.x * f, vg.y * sg);
      s[a][b] = make_double2(vs.x * f, vs.y * sg);
      z[a][b].x = i == k ? 1.0 : 0.0;
      if (i == k) { dsc[i] = di; col.d[0][i] = g[a][b].x; }
      if (k == 0) { col.g[0][i] = g[a][b]; col.s[0][i] = s[a][b]; col.z[0][i] = z[a][b]; }
    }
  __syncthreads();
  // the pivot of step j + 1 and its reciprocal are formed during step j, in every thread, from column
  // j and the published diagonal, so the reciprocal is off the chain of the updates
  double d = col.d[0][0], inv = 1.0 / d;
  for (int j = 0; j < n; ++j) {
    const int cb = j & 1;
    if (!(d > drop)) return false;  // the same value in every thread
    const int jn = min(j + 1, n - 1);
    const double2 gn = col.g[cb][jn];
    const double dn = fma(-(gn.x * gn.x + gn.y * gn.y), inv, col.d[cb][jn]);
    const double invn = 1.0 / dn;
    const double2 sjj = col.s[cb][j];
#pragma unroll
    for (int b = 0; b < TL; ++b) {
      const int k = tx + 16 * b, kc = min(k, n - 1);  // (threads outside the matrix repeat an edge)
      const double2 gk = col.g[cb][kc], sk = col.s[cb][kc];
      const double invk = k > j ? inv : 0.0;  // l is zero at and before the pivot
      const double2 nl = make_double2(-gk.x * invk, gk.y * invk);  // −conj(l_kj)
#pragma unroll
      for (int a = 0; a < TL; ++a) {
        const int i = ty + 16 * a, ic = min(i, n - 1);
        const double2 gi = col.g[cb][ic], si = col.s[cb][ic], zi = col.z[cb][ic];
        const double invi = i > j ? inv : 0.0;
        const double2 ni = make_double2(-gi.x * invi, -gi.y * invi);  // −l_ij
        const double2 gm = i > j ? gi : make_double2(0, 0);
        g[a][b] = cmac(g[a][b], gm, nl);
        // S_ik − l_i S_jk − conj(l_k)(S_ij − l_i S_jj)
        s[a][b] = cmac(cmac(s[a][b], ni, make_double2(sk.x, -sk.y)), nl, cmac(si, ni, sjj));
        z[a][b] = cmac(z[a][b], nl, zi);
        if (k == j + 1 && i < n) { col.g[cb ^ 1][i] = g[a][b]; col.s[cb ^ 1][i] = s[a][b]; col.z[cb ^ 1][i] = z[a][b]; }
        if (i == k && i < n) col.d[cb ^ 1][i] = g[a][b].x;
      }
    }
    d = dn;
    inv = invn;
    __syncthreads();
  }
  // unit pivots: the diagonal of the final Schur complements is still in its owners' registers
  double* piv = reinterpret_cast<double*>(col.g);
#pragma unroll
  for (int a = 0; a < TL; ++a) {
    const int i = ty + 16 * a;
    if (tx == (i & 15) && i < n) piv[i] = rsqrt(g[a][a].x);
  }
  __syncthreads();
#pragma unroll
  for (int a = 0; a < TL; ++a)
#pragma unroll
    for (int b = 0; b < TL; ++b) {
      const int i = ty + 16 * a, k = tx + 16 * b;
      if (i >= n || k >= n) continue;
      const double pk = piv[k], f = piv[i] * pk;
      Z[i * ld + k] = make_double2(z[a][b].x * pk, z[a][b].y * pk);
      if (i < k) continue;
      const double2 t = make_double2(s[a][b].x * f, i == k ? 0.0 : s[a][b].y * f);
      T[i * ld + k] = t;
      T[k * ld + i] = make_double2(t.x, -t.y);
    }
  __syncthreads();
  return true;
}

// One CTA per track: a latency-bound chain, so the time is what its barriers and dependent FP64
// operations take.  The reduction is n one-barrier steps (rr_reduce), the eigenproblem FP32 Jacobi
// sweeps refined to FP64 (eigh_refined), and L⁻ᴴ is applied as a matrix product.
__global__ void __launch_bounds__(RR_NT) k_rr(TrackState* const* __restrict__ states,
                                               double2* const* __restrict__ gram_accs,
                                               double2* const* __restrict__ coefs,
                                               float2* const* __restrict__ coefs32, int ntracks, int nmax,
                                               IterParams prm) {
  const int t = blockIdx.x;
  if (t >= ntracks) return;
  TrackState& s = *states[t];
  if (s.done) return;
  const int M = s.M;
  const int n = M + s.nWa + s.nP;
  const double jtol2 = prm.jacobi_tol2;
  const int ld = rr_ld(nmax);
  const int mat = (int)rr_mat(nmax);
  double2* T = reinterpret_cast<double2*>(rr_smem_raw);
  double2* X = T + mat;
  double2* W = X + mat;
  double2* Y = W + mat;
  double2* Z = Y + mat;
  __shared__ RRCols cols;
  __shared__ RotIdx ri[NMAX];
  __shared__ double red[64];
  __shared__ float redf[EIG_NT / 32];
  __shared__ float4 rots[NMAX];
  __shared__ int order[NMAX];
  __shared__ double dsc[NMAX];
  __shared__ double theta[NMAX];
  __shared__ double lam[NMAX];
  __shared__ int keep[NMAX];
  __shared__ int rank;
  const int tid = threadIdx.x, nt = blockDim.x;
  double2* acc = gram_accs[t];
  const bool chol_ok = n <= 16   ? rr_reduce<1>(acc, n, ld, prm.gram_drop, cols, dsc, T, Z)
                       : n <= 32 ? rr_reduce<2>(acc, n, ld, prm.gram_drop, cols, dsc, T, Z)
                                 : rr_reduce<3>(acc, n, ld, prm.gram_drop, cols, dsc, T, Z);
  int r = n;
  const double2* Ev;  // eigenvectors of the projected problem (columns)
  double2* G = T;     // SVQB path: scaled Gram matrix, then the projected one
  double2* B = W;     // SVQB path: the kept basis
  if (chol_ok) {
    // the accumulators are read: clear them for the next iteration
    for (int a = tid / 16; a < n; a += nt / 16)
      for (int b = a + tid % 16; b < n; b += 16)
        acc[a * NMAX + b] = acc[NMAX * NMAX + a * NMAX + b] = make_double2(0, 0);
    const double tol_e = 0.03 * sqrt(sqrt(jtol2));  // the last step leaves ‖E‖² ≲ 1e-3·√jtol2
    const int at = n <= 16   ? eigh_refined<1>(0, mat, 3 * mat, 2 * mat, n, M, ld, lam, redf, rots, order, tol_e)
                   : n <= 32 ? eigh_refined<2>(0, mat, 3 * mat, 2 * mat, n, M, ld, lam, redf, rots, order, tol_e)
                             : eigh_refined<3>(0, mat, 3 * mat, 2 * mat, n, M, ld, lam, redf, rots, order, tol_e);
    Ev = T + at;
    if (at < 0) {
      __syncthreads();
      jacobi_eigh(T, X, n, ld, W, ri, red, jtol2);
      for (int i = tid; i < n; i += nt) lam[i] = T[i * ld + i].x;
      Ev = X;
    }
  } else {
    // SVQB on the scaled Gram matrix
    double2* S = X;
    double2* V = Y;
    __syncthreads();
    for (int e = tid; e < 2 * n * n; e += nt) {
      const int which = e / (n * n), ab = e % (n * n), a = ab / n, b = ab % n;
      if (a > b) continue;
      const double f = dsc[a] * dsc[b];
      double2 g = acc[which * NMAX * NMAX + a * NMAX + b];
      g.x *= f;
      g.y *= a == b ? 0.0 : f;
      double2* Mx = which ? S : G;
      Mx[a * ld + b] = g;
      Mx[b * ld + a] = make_double2(g.x, -g.y);
    }
    __syncthreads();
    for (int e = tid; e < 2 * n * n; e += nt) {
      const int which = e / (n * n), ab = e % (n * n), a = ab / n, b = ab % n;
      if (a <= b) acc[which * NMAX * NMAX + a * NMAX + b] = make_double2(0, 0);
    }
    jacobi_eigh(G, V, n, ld, B, ri, red, jtol2);
    if (tid == 0) {
      double tmax = 0;
      for (int i = 0; i < n; ++i) { theta[i] = G[i * ld + i].x; tmax = fmax(tmax, theta[i]); }
      int rr = 0;
      for (int i = 0; i < n; ++i)
        if (theta[i] > prm.gram_drop * tmax) keep[rr++] = i;
      rank = rr;
    }
    __syncthreads();
    r = rank;
    if (r < M) {
      if (tid == 0) {
        s.status = TS_ORTHO; s.done = 1; s.op_ncol = 0; s.pw_ncol = 0; s.hmkh_ncol = 0;
        s.rr_n = n; s.rr_rank = r;
      }
      return;
    }
    // B = V_keep Θ^{-1/2}   (n × r)
    for (int e = tid; e < n * r; e += nt) {
      const int l = e / r, j = e % r;
      const double f = 1.0 / sqrt(theta[keep[j]]);
      const double2 v = V[l * ld + keep[j]];
      B[l * ld + j] = make_double2(v.x * f, v.y * f);
    }
    __syncthreads();
    // V ← S B (n × r), then G ← Bᴴ V (r × r)
    for (int e = tid; e < n * r; e += nt) {
      const int l = e / r, j = e % r;
      double2 acc = make_double2(0, 0);
      for (int m = 0; m < n; ++m) {
        const double2 a = S[l * ld + m], b = B[m * ld + j];
        acc.x += a.x * b.x - a.y * b.y;
        acc.y += a.x * b.y + a.y * b.x;
      }
      V[l * ld + j] = acc;
    }
    __syncthreads();
    for (int e = tid; e < r * r; e += nt) {
      const int i = e / r, j = e % r;
      double2 acc = make_double2(0, 0);
      for (int l = 0; l < n; ++l) {
        const double2 a = B[l * ld + i], b = V[l * ld + j];
        acc.x += a.x * b.x + a.y * b.y;  // conj(a)·b
        acc.y += a.x * b.y - a.y * b.x;
      }
      G[i * ld + j] = acc;
    }
    __syncthreads();
    jacobi_eigh(G, V, r, ld, S, ri, red, jtol2);  // S is folded into G = Bᴴ S B
    for (int i = tid; i < r; i += nt) lam[i] = G[i * ld + i].x;
    Ev = V;
  }
  __syncthreads();
  // ascending Ritz values (non-finite ones, which end the track after the update, have a place too)
  if (tid < r) order[rank_of([&](int j) { return lam[j]; }, r, tid)] = tid;
  __syncthreads();
  // coefficients of the new X in the Z columns (D L⁻ᴴ U, or D B U), and of the new P for the active
  // columns: the W and P parts of the Ritz vectors
  double2* coef = coefs[t];
  float2* coef32 = coefs32[t];
  const double2* Bz = chol_ok ? Z : B;
  const int nPn = (s.nWa + s.nP > 0) ? (M - s.nlocked) : 0;
  for (int e = tid; e < n * MMAX; e += nt) {
    const int l = e / MMAX, m = e % MMAX;
    if (m >= M) continue;
    const int um = order[m];
    double2 c = make_double2(0, 0);
    for (int j = chol_ok ? l : 0; j < r; ++j) c = cmac(c, Bz[l * ld + j], Ev[j * ld + um]);
    c.x *= dsc[l];
    c.y *= dsc[l];
    coef[l * MMAX + m] = c;
    coef32[l * MMAX + m] = make_float2((float)c.x, (float)c.y);
    const int mp = m - s.nlocked;
    if (mp >= 0 && mp < nPn) {
      if (l < M) c = make_double2(0, 0);
      coef[NMAX * MMAX + l * MMAX + mp] = c;
      coef32[NMAX * MMAX + l * MMAX + mp] = make_float2((float)c.x, (float)c.y);
    }
  }
  for (int m = tid; m < M; m += nt) s.lam[m] = lam[order[m]];
  if (tid == 0) { s.nP_next = nPn; s.rr_n = n; s.rr_rank = r; }
}

// Newton step of one track (one thread) from the partial sums of its HMkH pass.
__device__ __forceinline__ void newton_track(TrackState& s, const double* hp, int nb, const IterParams& prm) {
  double re = 0;
  for (int b = 0; b < nb; ++b) re += hp[2 * b];
  const double h = -re;
  const double dw2dk = 2.0 * h;
  const int j = s.band;
  const double dk = (s.lam[j] - s.omega2) / dw2dk;
  s.hmkh_ncol = 0;
  if (!(dw2dk > 0) || !isfinite(dk)) { finish(s, TS_NAN); return; }
  s.k_eig = s.k;
  s.hmkh = h;
  s.k -= dk;
  s.dk_last = dk;
  s.newton_steps++;
  s.newton_phase++;
  s.since_newton = 0;
  if (s.mode == MODE_NEWTON_OUTER) s.iter_phase = 0;  // the reference budgets each eigensolve
  double maxres = 0;
  for (int i = 0; i < s.need; ++i) maxres = fmax(maxres, s.resid[i]);
  if (s.mode == MODE_NEWTON_INNER) maxres = s.resid[j];  // the returned band (see control_track)
  if (!(s.k > 0)) { finish(s, TS_NAN); return; }
  if (prm.last_phase && maxres < prm.tol && fabs(dk) < prm.k_tol) { finish(s, TS_CONVERGED); return; }
  if (s.newton_steps >= prm.max_newton) { finish(s, prm.last_phase ? TS_MAXITER : TS_PHASE_DONE); return; }
  // k moved: recompute AX, AW and AP at the new k (keeping the P direction keeps LOBPCG's
  // momentum across Newton steps) and restart locking
  const int M = s.M;
  s.nlocked = 0;
  s.nWa = M;
  s.op_col0 = 0;
  s.op_ncol = 2 * M + s.nP;
  s.pw_ncol = 0;
  s.resid_best = 1e300;
  s.stall = 0;
}

// Inclusive scan over the first threads of a CTA of NEWTON_NT threads (warp shuffles, then the warps'
// totals), plus `carry`; every thread calls it.
__device__ __forceinline__ long long cta_scan(long long v, long long carry, long long* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) sh[w] = v;
  __syncthreads();
  for (int i = 0; i < w; ++i) v += sh[i];
  return v + carry;
}

// One CTA: a thread per track takes its Newton step and counts its live tiles; prefix sums of the
// counts and costs follow.  (As two kernels, the second a 1024-thread scan with 20 barriers, they took
// 3.5 + 7.2 µs of every iteration.)
__global__ void __launch_bounds__(NEWTON_NT)
    k_newton(TrackState* const* __restrict__ states, double* const* __restrict__ hmkh_parts,
             const int* __restrict__ hmkh_nb, const long long* __restrict__ n2, int ntracks, int rg, int ru,
             int* __restrict__ pre_g, int* __restrict__ pre_u, long long* __restrict__ wpre_g,
             long long* __restrict__ wpre_u, IterParams prm) {
  __shared__ long long sh[4][NEWTON_NT / 32];
  __shared__ long long last[4];
  const int tid = threadIdx.x;
  if (tid == 0) { pre_g[0] = pre_u[0] = 0; wpre_g[0] = wpre_u[0] = 0; }
  long long carry[4] = {0, 0, 0, 0};
  for (int base = 0; base < ntracks; base += NEWTON_NT) {
    const int t = base + tid;
    long long v[4] = {0, 0, 0, 0};
    if (t < ntracks) {
      TrackState& s = *states[t];
      if (!s.done && s.hmkh_ncol != 0) newton_track(s, hmkh_parts[t], hmkh_nb[t], prm);
      if (!s.done) {
        const int n = s.M + s.nWa + s.nP;
        v[0] = (n2[t] + rg - 1) / rg;
        v[1] = (n2[t] + ru - 1) / ru;
        v[2] = v[0] * gram_tile_cost(n) + GRAM_TRACK_COST;
        v[3] = v[1] * update_tile_cost(n, s.M);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = cta_scan(v[q], carry[q], sh[q]);
    if (t < ntracks) {
      pre_g[t + 1] = (int)v[0]; pre_u[t + 1] = (int)v[1];
      wpre_g[t + 1] = v[2]; wpre_u[t + 1] = v[3];
    }
    if (base + NEWTON_NT < ntracks) {
      if (tid == NEWTON_NT - 1)
        for (int q = 0; q < 4; ++q) last[q] = v[q];
      __syncthreads();
      for (int q = 0; q < 4; ++q) carry[q] = last[q];
      __syncthreads();
    }
  }
}

}  // namespace omb
