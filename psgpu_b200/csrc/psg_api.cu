// psg_api.cu -- error reporting and library information of the C API.
#include <stdarg.h>
#include <stdio.h>
#include <math.h>
#include <string.h>

#include "psg_common.cuh"
#include "psgpu_internal.h"

static thread_local char g_err[1024];

extern "C" void psg_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof g_err, fmt, ap);
  va_end(ap);
}

extern "C" const char* psg_last_error(void) { return g_err; }

extern "C" void psg_clear_error(void) { g_err[0] = 0; }

extern "C" int psg_version(void) { return PSG_VERSION; }

// ---------------------------------------------------------------------------
// building-block check: the line FFT of psg_fft.cuh applied to `nlines`
// contiguous lines of n complex doubles (one warp-level thread group per
// line).  Used by the unit tests; unnormalised, sign -1 forward / +1 inverse.
// ---------------------------------------------------------------------------
#include "psg_fft.cuh"
#include "psg_tma.cuh"

namespace {
template <int N, int SIGN, bool SWAP>
__global__ void linefft_kernel(const psg::cpx<double>* in, psg::cpx<double>* out,
                               const psg::cpx<double>* tw, int nlines) {
  using F = psg::LineFFT<N, SIGN, double, SWAP>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  psg::cpx<double>* s_tw = reinterpret_cast<psg::cpx<double>*>(smem_raw);
  psg::cpx<double>* s_ex = s_tw + N;
  for (int i = threadIdx.x; i < N; i += blockDim.x) s_tw[i] = tw[i];
  __syncthreads();
  const int gpb = blockDim.x / F::G;
  const int grp = threadIdx.x / F::G, g = threadIdx.x % F::G;
  const int line = blockIdx.x * gpb + grp;
  const bool live = line < nlines;
  psg::cpx<double> v[F::E];
#pragma unroll
  for (int e = 0; e < F::E; ++e)
    v[e] = live ? in[(long)line * N + F::in_index(g, e)] : psg::czero<double>();
  F::run(v, g, s_tw, s_ex + grp * F::SMEM, psg::WarpSync());
  if (live) {
#pragma unroll
    for (int e = 0; e < F::E; ++e) out[(long)line * N + F::out_index(g, e)] = v[e];
  }
}

template <int N, int SIGN, bool SWAP>
int launch_linefft(const double* in, double* out, int nlines) {
  using F = psg::LineFFT<N, SIGN, double, SWAP>;
  const long len = (long)nlines * N;
  psg::cpx<double>*d_in = nullptr, *d_out = nullptr, *d_tw = nullptr;
  psg::cpx<double> h_tw[N];
  F::host_table(h_tw);
  int rc = PSG_OK;
  const int threads = 128;
  const int gpb = threads / F::G;
  const size_t smem = sizeof(psg::cpx<double>) * (N + gpb * F::SMEM);
  if (cudaMalloc(&d_in, sizeof(psg::cpx<double>) * len) != cudaSuccess ||
      cudaMalloc(&d_out, sizeof(psg::cpx<double>) * len) != cudaSuccess ||
      cudaMalloc(&d_tw, sizeof(psg::cpx<double>) * N) != cudaSuccess) {
    psg_set_error("cudaMalloc failed");
    rc = PSG_ERR_CUDA;
  }
  if (rc == PSG_OK) {
    cudaMemcpy(d_in, in, sizeof(psg::cpx<double>) * len, cudaMemcpyHostToDevice);
    cudaMemcpy(d_tw, h_tw, sizeof(psg::cpx<double>) * N, cudaMemcpyHostToDevice);
    cudaFuncSetAttribute(linefft_kernel<N, SIGN, SWAP>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    linefft_kernel<N, SIGN, SWAP><<<(nlines + gpb - 1) / gpb, threads, smem>>>(d_in, d_out, d_tw, nlines);
    cudaError_t e = cudaMemcpy(out, d_out, sizeof(psg::cpx<double>) * len, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) { psg_set_error("%s", cudaGetErrorString(e)); rc = PSG_ERR_CUDA; }
  }
  cudaFree(d_in); cudaFree(d_out); cudaFree(d_tw);
  return rc;
}
}  // namespace

extern "C" int psg_debug_linefft(int n, int sign, int swap, const double* in, double* out,
                                 int nlines) {
  if (!in || !out || nlines <= 0 || (sign != 1 && sign != -1)) {
    psg_set_error("bad arguments");
    return PSG_ERR_ARG;
  }
#define PSG_LF(NN)                                                                   \
  case NN:                                                                           \
    if (swap)                                                                        \
      return sign < 0 ? launch_linefft<NN, -1, true>(in, out, nlines)                \
                      : launch_linefft<NN, 1, true>(in, out, nlines);                \
    return sign < 0 ? launch_linefft<NN, -1, false>(in, out, nlines)                 \
                    : launch_linefft<NN, 1, false>(in, out, nlines);
  switch (n) {
    PSG_LF(16) PSG_LF(32) PSG_LF(64) PSG_LF(128) PSG_LF(256) PSG_LF(512)
    default:
      psg_set_error("line length %d unsupported", n);
      return PSG_ERR_UNSUPPORTED;
  }
#undef PSG_LF
}

// ---------------------------------------------------------------------------
// The same check of the forms that the engines run: FP64 and FP32 lines, plain and
// with merged twiddles, and two FP32 lines in one packed transform, with either
// exchange (lines 2 p and 2 p + 1; an odd last line is paired with itself).
// ---------------------------------------------------------------------------
#include "psg_fft2.cuh"

namespace {
// psg_debug_line_form's forms (include/psgpu.h)
enum LineForm { kPlain = 0, kMerged = 1, kPacked = 2, kPackedMerged = 3, kPackedMergedWide = 4 };

template <typename T, int N, int SIGN, bool SWAP, int FORM>
__global__ void __launch_bounds__(128)
line_form_kernel(const double2* __restrict__ in, double2* __restrict__ out, const psg::cpx<T>* __restrict__ tw,
                 int nlines) {
  using P = psg::LineFFT<N, SIGN, T, SWAP>;
  constexpr bool PACKED = FORM >= kPacked;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  psg::cpx<T>* s_tw = reinterpret_cast<psg::cpx<T>*>(smem_raw);
  for (int i = threadIdx.x; i < N; i += blockDim.x) s_tw[i] = tw[i];
  __syncthreads();
  const int gpb = blockDim.x / P::G, grp = threadIdx.x / P::G, g = threadIdx.x % P::G;
  // 16 bytes of exchange per entry, whatever the form takes
  float4* ex = reinterpret_cast<float4*>(s_tw + N) + grp * P::SMEM;
  const int item = blockIdx.x * gpb + grp, per = PACKED ? 2 : 1;
  const bool live = item * per < nlines;
  const long l0 = live ? (long)item * per : 0, l1 = PACKED && l0 + 1 < nlines ? l0 + 1 : l0;
  if constexpr (PACKED) {
    psg::Pk v[P::E];
#pragma unroll
    for (int e = 0; e < P::E; ++e) {
      const double2 a = in[l0 * N + P::in_index(g, e)], b = in[l1 * N + P::in_index(g, e)];
      v[e] = psg::Pk{make_float2((float)a.x, (float)b.x), make_float2((float)a.y, (float)b.y)};
    }
    if constexpr (FORM == kPacked)
      psg::LineFFT2<N, SIGN, SWAP>::run(v, g, s_tw, reinterpret_cast<float2*>(ex), psg::WarpSync());
    else if constexpr (FORM == kPackedMerged)
      psg::LineFFT2M<N, SIGN, SWAP>::run(v, g, s_tw, reinterpret_cast<float2*>(ex), psg::WarpSync());
    else
      psg::LineFFT2M<N, SIGN, SWAP>::run(v, g, s_tw, ex, psg::WarpSync());
    if (!live) return;
#pragma unroll
    for (int e = 0; e < P::E; ++e) {
      const int k = P::out_index(g, e);
      out[l0 * N + k] = make_double2(v[e].re.x, v[e].im.x);
      if (l1 != l0) out[l1 * N + k] = make_double2(v[e].re.y, v[e].im.y);
    }
  } else {
    psg::cpx<T> v[P::E];
#pragma unroll
    for (int e = 0; e < P::E; ++e) {
      const double2 a = in[l0 * N + P::in_index(g, e)];
      v[e] = psg::cpx<T>{(T)a.x, (T)a.y};
    }
    psg::cpx<T>* ext = reinterpret_cast<psg::cpx<T>*>(ex);
    if constexpr (FORM == kMerged) psg::LineFFTM<N, SIGN, T, SWAP>::run(v, g, s_tw, ext, psg::WarpSync());
    else P::run(v, g, s_tw, ext, psg::WarpSync());
    if (!live) return;
#pragma unroll
    for (int e = 0; e < P::E; ++e) out[l0 * N + P::out_index(g, e)] = make_double2(v[e].x, v[e].y);
  }
}

template <typename T, int N, int SIGN, bool SWAP, int FORM>
int launch_line_form(const double* in, double* out, int nlines) {
  using P = psg::LineFFT<N, SIGN, T, SWAP>;
  psg::cpx<T> h_tw[N];
  if (FORM == kPlain || FORM == kPacked) P::host_table(h_tw);
  else psg::LineFFTM<N, SIGN, T, SWAP>::host_table(h_tw);
  const size_t bytes = sizeof(double2) * (size_t)nlines * N;
  unsigned char* d = nullptr;  // in, out, table
  PSG_CUDA_TRY(cudaMalloc(&d, 2 * bytes + sizeof h_tw));
  cudaError_t e = cudaMemcpy(d, in, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + 2 * bytes, h_tw, sizeof h_tw, cudaMemcpyHostToDevice);
  const int threads = 128, gpb = threads / P::G, items = FORM >= kPacked ? (nlines + 1) / 2 : nlines;
  const size_t smem = sizeof h_tw + sizeof(float4) * gpb * P::SMEM;
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(line_form_kernel<T, N, SIGN, SWAP, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
  if (e == cudaSuccess) {
    line_form_kernel<T, N, SIGN, SWAP, FORM><<<(items + gpb - 1) / gpb, threads, smem>>>(
        reinterpret_cast<double2*>(d), reinterpret_cast<double2*>(d + bytes),
        reinterpret_cast<psg::cpx<T>*>(d + 2 * bytes), nlines);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + bytes, bytes, cudaMemcpyDeviceToHost);
  cudaFree(d);
  PSG_CUDA_TRY(e);
  return PSG_OK;
}

template <int N, int SIGN, bool SWAP>
int line_form(int form, int precision, const double* in, double* out, int nlines) {
  if (precision == 64) {
    if (form == kPlain) return launch_line_form<double, N, SIGN, SWAP, kPlain>(in, out, nlines);
    if (form == kMerged) return launch_line_form<double, N, SIGN, SWAP, kMerged>(in, out, nlines);
  } else {
    switch (form) {
      case kPlain: return launch_line_form<float, N, SIGN, SWAP, kPlain>(in, out, nlines);
      case kMerged: return launch_line_form<float, N, SIGN, SWAP, kMerged>(in, out, nlines);
      case kPacked: return launch_line_form<float, N, SIGN, SWAP, kPacked>(in, out, nlines);
      case kPackedMerged: return launch_line_form<float, N, SIGN, SWAP, kPackedMerged>(in, out, nlines);
      case kPackedMergedWide: return launch_line_form<float, N, SIGN, SWAP, kPackedMergedWide>(in, out, nlines);
    }
  }
  psg_set_error("line form %d in precision %d unsupported", form, precision);
  return PSG_ERR_UNSUPPORTED;
}
}  // namespace

extern "C" int psg_debug_line_form(int n, int sign, int swap, int form, int precision, const double* in,
                                   double* out, int nlines) {
  if (!in || !out || nlines <= 0 || (sign != 1 && sign != -1) || (precision != 32 && precision != 64)) {
    psg_set_error("bad arguments");
    return PSG_ERR_ARG;
  }
  // the engines' transforms: inverse, forward, and forward on the inverse's output registers
  if (swap && sign > 0) {
    psg_set_error("no inverse transform takes the swapped plan");
    return PSG_ERR_UNSUPPORTED;
  }
#define PSG_LF(NN)                                                                          \
  case NN:                                                                                  \
    if (swap) return line_form<NN, -1, true>(form, precision, in, out, nlines);             \
    return sign < 0 ? line_form<NN, -1, false>(form, precision, in, out, nlines)            \
                    : line_form<NN, 1, false>(form, precision, in, out, nlines);
  switch (n) {
    PSG_LF(16) PSG_LF(32) PSG_LF(64) PSG_LF(128) PSG_LF(256)
    default:
      psg_set_error("line length %d unsupported", n);
      return PSG_ERR_UNSUPPORTED;
  }
#undef PSG_LF
}

// ---------------------------------------------------------------------------
// The bounded-wait path, exercised: a block arms an mbarrier for a transfer
// that is never issued and waits `polls` times; the wait runs out, the kernel
// records PSG_DEV_TIMEOUT in the status word and returns (no copy is in flight,
// so nothing outlives the block).  The host reads the status as the engines do.
// ---------------------------------------------------------------------------
namespace {
__global__ void wait_nothing(int polls, int* status) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    psg::mbar_init(&bar, 1);
    psg::mbar_expect_tx(&bar, 16);  // 16 bytes that never arrive
    psg::mbar_wait_polls(&bar, 0, polls, status);
  }
}
}  // namespace

extern "C" int psg_debug_wait_timeout(int polls, int* status_out) {
  if (polls < 1 || polls > (1 << 20) || !status_out) {
    psg_set_error("bad arguments");
    return PSG_ERR_ARG;
  }
  int* d = nullptr;
  PSG_CUDA_TRY(cudaMalloc(&d, sizeof(int)));
  cudaError_t e = cudaMemset(d, 0, sizeof(int));
  if (e == cudaSuccess) {
    wait_nothing<<<1, 32>>>(polls, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(status_out, d, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  PSG_CUDA_TRY(e);
  return PSG_OK;
}
