// Allocation-free FP32 operator apply (omb_apply_M_noalloc).
//
// Some callers cannot allocate device memory at the moment they need the operator:
// host frameworks that own the whole device pool (a Julia or PyTorch caching allocator
// that forbids foreign cudaMalloc/cudaFree), callers with a fixed device-memory budget
// decided up front, and hot loops that must not pay the latency and the implicit device
// synchronisation of cudaMalloc/cudaFree.  This entry point takes every input and output as
// caller-owned device memory and allocates nothing itself: the intermediate 3-component
// field of the three FFT passes lives in a file-scope static device array of fixed size,
// and so do the twiddle tables.
//
// Limits and rules:
//  * Nx·Ny·ncol ≤ OMB_NOALLOC_MAX_PIXEL_COLUMNS (262144: e.g. 256×256 with 4 columns or
//    512×512 with 1); larger requests are rejected with OMB_ERR_INVALID_ARG.
//  * The array (6 MiB) is held by every GPU that loads the library until exit.
//  * All calls share it, so calls that overlap on the GPU (different streams, or
//    different host threads) race; serialise them on one stream.
//  * The first call in a CUDA context does a one-time set-up with that context current
//    (it resolves the arrays' device addresses with cudaGetSymbolAddress and uploads the
//    twiddle tables with a blocking copy); make that first call before any stream capture
//    (a first call on a capturing stream is refused with OMB_ERR_INVALID_ARG).  The set-up
//    is keyed on the context, so a new primary context after cudaDeviceReset repeats it.
//  * The pass descriptor travels as a kernel argument; the field needs no clearing (the first pass
//    writes every element the later passes read).
//  * The passes are the two-level register-FFT passes of omb_apply.  ε⁻¹ is read in the
//    reference's (3, 3, Nx, Ny) layout.
#include <cuda.h>

#include <cmath>
#include <mutex>

#include "context.h"
#include "ops_impl.cuh"

namespace omb {

constexpr long long NOALLOC_MAX_PIXEL_COLUMNS = 262144;
constexpr size_t NOALLOC_FIELD_BYTES = 3 * (size_t)NOALLOC_MAX_PIXEL_COLUMNS * sizeof(float2);

// scratch: the 3·N·ncol field
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_FIELD_BYTES];

#define OMB_NOALLOC_LENS(X) X(8) X(12) X(16) X(20) X(24) X(32) X(40) X(48) X(64) X(80) X(96) \
  X(128) X(160) X(192) X(256) X(320) X(384) X(512)
#define OMB_LEN_SUM(n) +3 * n
// per length L: [exp(-2πi m/L), m < L | TW1 | TW3] (the layout of the context's tables)
constexpr int NOALLOC_TW_TOTAL = 0 OMB_NOALLOC_LENS(OMB_LEN_SUM);
#undef OMB_LEN_SUM
static __device__ __align__(16) float2 g_noalloc_tw[NOALLOC_TW_TOTAL];

struct NoallocDevice {
  unsigned long long ctx_id = 0;     // context the set-up was done in (0: none yet)
  unsigned char* scratch = nullptr;  // device address of g_noalloc_scratch
  float2* tw = nullptr;              // device address of g_noalloc_tw
  int tw_off[513] = {};
};
static NoallocDevice g_noalloc_dev[64];
static std::mutex g_noalloc_mu;

using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

// Unique id of the calling thread's current context (the runtime has made it current).
static int current_ctx_id(unsigned long long* id) {
  static CtxGetCurrentFn get_cur = nullptr;
  static CtxGetIdFn get_id = nullptr;
  if (!get_cur || !get_id) {
    void* a = nullptr;
    void* b = nullptr;
    cudaDriverEntryPointQueryResult qa{}, qb{};
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) != cudaSuccess || !a ||
        cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) != cudaSuccess || !b)
      return fail(OMB_ERR_CUDA, "omb_apply_M_noalloc: cuCtxGetCurrent/cuCtxGetId not available from the driver");
    get_cur = reinterpret_cast<CtxGetCurrentFn>(a);
    get_id = reinterpret_cast<CtxGetIdFn>(b);
  }
  CUcontext c = nullptr;
  if (get_cur(&c) != CUDA_SUCCESS || !c || get_id(c, id) != CUDA_SUCCESS)
    return fail(OMB_ERR_CUDA, "omb_apply_M_noalloc: no current CUDA context");
  return OMB_OK;
}

static int noalloc_setup(int dev, cudaStream_t st) {
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoallocDevice& D = g_noalloc_dev[dev];
  unsigned long long id = 0;
  int rc = current_ctx_id(&id);
  if (rc) return rc;
  if (D.ctx_id == id) return OMB_OK;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(st, &cs);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamIsCapturing");
  if (cs != cudaStreamCaptureStatusNone)
    return fail(OMB_ERR_INVALID_ARG,
                "omb_apply_M_noalloc: the first call in a CUDA context does a blocking set-up; make one call "
                "outside any stream capture first");
  void* p = nullptr;
  e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(noalloc scratch)");
  D.scratch = static_cast<unsigned char*>(p);
  e = cudaGetSymbolAddress(&p, g_noalloc_tw);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(noalloc twiddles)");
  D.tw = static_cast<float2*>(p);
  static float2 host_tw[NOALLOC_TW_TOTAL];  // fixed host table, no heap use
  const double two_pi = 6.283185307179586476925286766559;
  auto w_of = [&](int m, int L) {
    m %= L;
    double c = std::cos(-two_pi * (double)m / (double)L), s = std::sin(-two_pi * (double)m / (double)L);
    if (m == 0) { c = 1; s = 0; }
    if (4 * m == L) { c = 0; s = -1; }
    if (2 * m == L) { c = -1; s = 0; }
    if (4 * m == 3 * L) { c = 0; s = 1; }
    return make_float2((float)c, (float)s);
  };
  int off = 0;
  auto fill = [&](int L) {
    D.tw_off[L] = off;
    for (int m = 0; m < L; ++m) host_tw[off + m] = w_of(m, L);
    const int A = plan2_a(L), B = A ? L / A : 0;
    for (int k1 = 0; k1 < A; ++k1)
      for (int n2 = 0; n2 < B; ++n2) {
        host_tw[off + L + k1 * B + n2] = w_of(n2 * k1, L);
        host_tw[off + 2 * L + n2 * A + k1] = w_of(n2 * k1, L);
      }
    off += 3 * L;
  };
#define OMB_FILL(n) fill(n);
  OMB_NOALLOC_LENS(OMB_FILL)
#undef OMB_FILL
  e = cudaMemcpyToSymbol(g_noalloc_tw, host_tw, sizeof(host_tw));
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyToSymbol(noalloc twiddles)");
  D.ctx_id = id;
  return OMB_OK;
}

// The three passes in the component-parallel form (op_kernels_split.cuh) with the pass descriptor and k
// passed by value: at this entry point's sizes a launch is at most one CTA per SM or so and its time is
// one CTA's chain of latencies, which three times the threads shorten; and nothing has to be written
// to the device ahead of it.  256×256 with 4 columns: 31.6 → 23.5 µs a call
// (against a descriptor kernel and the one-thread-per-slot passes).
struct NoallocUnit {
  OpUnit<float> u;
  double k;
};
__host__ __device__ constexpr int noalloc_tx(int NY) { return NY > 256 ? 4 : 8; }
template <int NX>
__global__ void __launch_bounds__(sp_row_threads(NX, sp_rows(NX)), sp_row_min_blocks<float>(sp_row_threads(NX, sp_rows(NX)), NX))
    k_noalloc_row_in(const __grid_constant__ NoallocUnit P, const float2* __restrict__ tw) {
  row_in_sp<float, NX, RI_KXTC, false, sp_rows(NX)>(P.u, P.k, tw);
}
template <int NY>
__global__ void __launch_bounds__(sp_col_threads(NY, noalloc_tx(NY)))
    k_noalloc_col(const __grid_constant__ NoallocUnit P, const float2* __restrict__ tw) {
  col_sp<NY, CS_FWD, PW_EPS9, CS_INV, noalloc_tx(NY)>(P.u, blockIdx.y, tw);
}
template <int NX>
__global__ void __launch_bounds__(sp_row_threads(NX, sp_rows(NX)), sp_row_min_blocks<float>(sp_row_threads(NX, sp_rows(NX)), NX))
    k_noalloc_row_out(const __grid_constant__ NoallocUnit P, const float2* __restrict__ tw) {
  row_out_sp<float, NX, RO_KXCT, true, sp_rows(NX)>(P.u, P.k, tw);
}

template <typename K> static cudaError_t noalloc_launch(K kern, dim3 g, int nt, size_t smem, cudaStream_t st,
                                                         const NoallocUnit& P, const float2* tw) {
  if (smem > 32 * 1024) {
    // (every call: the attribute belongs to the CUDA context, which may be a new one)
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  kern<<<g, nt, smem, st>>>(P, tw);
  return cudaGetLastError();
}

template <int NX> static cudaError_t noalloc_rows(bool in, int Ny, int ncol, const NoallocUnit& P,
                                                  const float2* tw, cudaStream_t st) {
  constexpr int G = sp_rows(NX), NT = sp_row_threads(NX, G);
  const size_t sm = (size_t)3 * G * l2_row_lstr<float2, NX>() * sizeof(float2);
  const dim3 g((Ny + G - 1) / G, ncol, 1);
  return in ? noalloc_launch(k_noalloc_row_in<NX>, g, NT, sm, st, P, tw)
            : noalloc_launch(k_noalloc_row_out<NX>, g, NT, sm, st, P, tw);
}
template <int NY> static cudaError_t noalloc_col(int Nx, int ncol, const NoallocUnit& P, const float2* tw,
                                                 cudaStream_t st) {
  constexpr int TX = noalloc_tx(NY), NT = sp_col_threads(NY, TX);
  const size_t sm = (size_t)3 * TX * l2_col_lstr<float2, NY, TX>() * sizeof(float2);
  const dim3 g((Nx + TX - 1) / TX, ncol, 1);
  return noalloc_launch(k_noalloc_col<NY>, g, NT, sm, st, P, tw);
}

}  // namespace omb

using namespace omb;

extern "C" int omb_apply_M_noalloc(int32_t Nx, int32_t Ny, double Dx, double Dy, double k, const float* d_epsinv,
                                   int32_t ncol, const void* d_H_in, void* d_H_out, void* stream) {
  omb_grid g{Nx, Ny, Dx, Dy};
  int rc = check_grid(&g);
  if (rc) return rc;
  if (!(k > 0) || !std::isfinite(k)) return fail(OMB_ERR_INVALID_ARG, "k must be finite and positive");
  if (ncol <= 0 || !d_epsinv || !d_H_in || !d_H_out)
    return fail(OMB_ERR_INVALID_ARG, "need ncol > 0 and non-NULL device pointers");
  if ((long long)Nx * Ny * ncol > NOALLOC_MAX_PIXEL_COLUMNS)
    return fail(OMB_ERR_INVALID_ARG, "omb_apply_M_noalloc: Nx*Ny*ncol = " + std::to_string((long long)Nx * Ny * ncol) +
                                         " exceeds its fixed scratch of " + std::to_string(NOALLOC_MAX_PIXEL_COLUMNS) +
                                         " pixel-columns (use omb_apply for larger blocks)");
  int dev = 0;
  OMB_CU(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(OMB_ERR_UNSUPPORTED, "device index above 63");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = noalloc_setup(dev, st);
  if (rc) return rc;
  const NoallocDevice& D = g_noalloc_dev[dev];
  const size_t N = (size_t)Nx * Ny;
  NoallocUnit P{};
  P.k = k;
  OpUnit<float>& u = P.u;
  u.in = static_cast<const float2*>(d_H_in);
  u.out = static_cast<float2*>(d_H_out);
  u.scr = reinterpret_cast<float2*>(D.scratch);
  u.e9 = d_epsinv;
  u.in_cs = u.out_cs = (long long)(2 * N);
  u.scr_cs = (long long)(3 * N);
  u.Nx = Nx; u.Ny = Ny; u.ncol = ncol;
  u.part_stride = row_blocks(Nx, Ny);
  u.inv_dx = (float)(1.0 / Dx); u.inv_dy = (float)(1.0 / Dy);
  cudaError_t e = cudaSuccess;
  switch (Nx) {
#define OMB_CASE(n) case n: e = noalloc_rows<n>(true, Ny, ncol, P, D.tw + D.tw_off[n], st); break;
    OMB_NOALLOC_LENS(OMB_CASE)
#undef OMB_CASE
  }
  if (e != cudaSuccess) return cuda_fail(e, "omb_apply_M_noalloc row pass");
  switch (Ny) {
#define OMB_CASE(n) case n: e = noalloc_col<n>(Nx, ncol, P, D.tw + D.tw_off[n], st); break;
    OMB_NOALLOC_LENS(OMB_CASE)
#undef OMB_CASE
  }
  if (e != cudaSuccess) return cuda_fail(e, "omb_apply_M_noalloc column pass");
  switch (Nx) {
#define OMB_CASE(n) case n: e = noalloc_rows<n>(false, Ny, ncol, P, D.tw + D.tw_off[n], st); break;
    OMB_NOALLOC_LENS(OMB_CASE)
#undef OMB_CASE
  }
  if (e != cudaSuccess) return cuda_fail(e, "omb_apply_M_noalloc row pass");
  return OMB_OK;
}
