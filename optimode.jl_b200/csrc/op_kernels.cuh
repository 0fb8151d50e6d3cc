// Fused plane-wave Helmholtz operator passes (sm_100a): the units they work on and their modes (the
// kernels are in op_kernels_2l.cuh, op_kernels_split.cuh and op_cluster.cuh).
//
// One operator application M̂(k)H = kx_ct · (1/N)·bfft · ε⁻¹ · fft · kx_tc H
// (reference: _M!, lib/MaxwellEigenmodes/src/maxwell.jl:471-481) runs as three passes:
//
//   row_in  : per grid row, regenerate (mag, m̂, n̂) from (k, gx, gy) in registers, form
//             the 3-component field (kx_tc, kxinv_tc or zx_tc), FFT along x,
//             store planar to the scratch field (stays in L2 between passes);
//   col     : per tile of TX adjacent columns, FFT along y, per-pixel 3×3 ε⁻¹ contraction
//             (6 unique entries: float4 + float2 loads) or ε_ave scaling, FFT back along y,
//             in place;
//   row_out : per grid row, FFT back along x, then the curl epilogue (kx_ct or kxinv_ct)
//             that writes the 2-component output, optionally reducing ⟨H_in, out⟩.
//
// The same passes with other prologue/epilogue choices give the MPB-style preconditioner
// (_P!, maxwell.jl:459-469), ⟨H|∂M̂/∂k|H⟩ (HMₖH, maxwell.jl:267-269), E = ε⁻¹·fft(kx_tc H)
// (E⃗, fields.jl:194-210) and the adjoint's _H2d!/_d2ẽ! (fields.jl:81-93).
//
// Layouts: H is the reference's column-major (2, Nx, Ny) complex vector (component
// fastest); scratch fields are planar [c][iy][ix]; ε⁻¹ is stored as 6 unique entries
// (xx, yy, zz, xy) + (xz, yz) per pixel.
#pragma once

#include "dft_small.cuh"

namespace omb {

template <typename T> struct OpUnit {
  const cplx<T>* in;      // 2-component input block (or planar 3-component for RI_LOAD3)
  cplx<T>* out;           // 2-component output block (or planar 3-component for RO_STORE3)
  cplx<T>* scr;           // planar 3·N scratch per column
  const float4* e32a;     // (xx, yy, zz, xy) FP32
  const float2* e32b;     // (xz, yz)         FP32
  const double2* e64;     // 3 double2 per pixel: (xx,yy), (zz,xy), (xz,yz)
  const T* eave;          // 3/tr(ε⁻¹) per pixel
  const T* e9;            // ε⁻¹ in the reference's (3, 3, Nx, Ny) layout (PW_EPS9 only)
  const double* k_dev;    // wavevector magnitude (device, so the solver can update it)
  double* partial;        // per-(column, row-block) partial sums for RO_KXCT_DOT
  const int* ncol_dev;    // optional device-side column count
  const int* col0_dev;    // optional device-side first column of in/out (scratch is not offset)
  long long in_cs, out_cs, scr_cs;  // column strides in complex elements
  int Nx, Ny, ncol;
  int part_stride;        // partial sums per column (≥ gridDim.x of row_out)
  T inv_dx, inv_dy;
  // z-periodic cells: one unit per z-slab (or per z-line set) of a 3D field
  long long comp_stride;  // component stride of planar 3-component fields (0: Nx·Ny of the pass)
  double kz_shift;        // g_z of the slab: the passes see k − g_z (w = k ẑ − G)
  double inv_dz;          // 1/Λ of a z-periodic cell (0 for a 2D cell)
  int zx_weight_gz;       // RI_ZXTC only: weight ẑ×H by g_z/Λ (⟨H|∂M̂/∂Λ|H⟩, the period derivative)
};

enum RowIn : int { RI_KXTC = 0, RI_KXINV = 1, RI_ZXTC = 2, RI_LOAD3 = 3, RI_HCART = 4 };
enum RowOut : int { RO_KXCT = 0, RO_KXINVCT = 1, RO_STORE3 = 2, RO_KXCT_DOT = 3 };
enum ColStep : int { CS_NONE = 0, CS_FWD = 1, CS_INV = 2 };
enum ColPw : int { PW_NONE = 0, PW_EPS = 1, PW_EAVE = 2, PW_EPS9 = 3 };

template <typename T> __device__ __forceinline__ void load_eps(const OpUnit<T>& U, size_t p, T e[6]);
template <> __device__ __forceinline__ void load_eps<float>(const OpUnit<float>& U, size_t p, float e[6]) {
  float4 a = __ldg(U.e32a + p);
  float2 b = __ldg(U.e32b + p);
  e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w; e[4] = b.x; e[5] = b.y;
}
template <> __device__ __forceinline__ void load_eps<double>(const OpUnit<double>& U, size_t p, double e[6]) {
  double2 a = __ldg(U.e64 + 3 * p), b = __ldg(U.e64 + 3 * p + 1), c = __ldg(U.e64 + 3 * p + 2);
  e[0] = a.x; e[1] = a.y; e[2] = b.x; e[3] = b.y; e[4] = c.x; e[5] = c.y;
}

template <typename T> __device__ __forceinline__ int unit_ncol(const OpUnit<T>& U) {
  return U.ncol_dev ? *U.ncol_dev : U.ncol;
}
template <typename T> __device__ __forceinline__ int unit_col0(const OpUnit<T>& U) {
  return U.col0_dev ? *U.col0_dev : 0;
}

}  // namespace omb
