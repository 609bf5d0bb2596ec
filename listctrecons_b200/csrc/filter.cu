// Stage 3: ramp-filter taps (host) and row convolution kernels.
//
// The reference convolves each detector row with 2*ns taps, out[is] = sum_{k<ns}
// h[is-k+ns] * row[k] (CUDA/Filter.cu:42-46), i.e. out = row * T with the Toeplitz matrix
// T[k][is] = h[is-k+ns].  LCT_FILTER_FP32 keeps that sum's order (FP32 FMA, k increasing) so
// results are bit-exact with the reference kernel.  LCT_FILTER_BF16X3 runs the same product as a GEMM on the
// tensor cores (filter_tc.cu).
#include <cmath>
#include <mutex>

#include "lct_internal.h"
#include "tc_ptx.cuh"

namespace lct {

// ---------------------------------------------------------------------------------------
// Taps.  With W(f) a frequency window, every kernel here is
//   h(n) = (1/ds) * 2 * integral_0^{1/2} f W(f) cos(2 pi n f) df,
// which for W = 1 is exactly the reference's Ram-Lak expression (Src/Filter.cpp:13-19) and
// for W = sinc(f) the Shepp-Logan kernel -2 / (pi^2 ds (4n^2 - 1)) (Shepp & Logan 1974;
// Kak & Slaney, "Principles of Computerized Tomographic Imaging", ch. 3), both with the
// reference's scaling (the discrete sum's ds factor folded into the taps).
// ---------------------------------------------------------------------------------------

// continuous-argument kernels (x in samples), FP64
static double ramlak_x(double x, double ds) {
  if (x == 0.0) return 0.25 / ds;
  const double px = kRefPi * x;
  return (std::sin(px) / px + (std::cos(px) - 1.0) / (px * px)) / (2.0 * ds);
}

static double shepp_logan_x(double x, double ds) {
  // (1/pi) [ (1 - cos(pi u1 / 2)) / (pi u1) + (1 - cos(pi u2 / 2)) / (pi u2) ], u = 1 +- 2x
  auto term = [](double u) {
    if (std::fabs(u) < 1e-12) return 0.0;
    return (1.0 - std::cos(kRefPi * u / 2.0)) / (kRefPi * u);
  };
  return (term(1.0 + 2.0 * x) + term(1.0 - 2.0 * x)) / kRefPi / ds;
}

static double base_kernel(int kind, double x, double ds) {
  return kind == LCT_FILTER_SHEPP_LOGAN ? shepp_logan_x(x, ds) : ramlak_x(x, ds);
}

static double windowed(int kind, int window, int n, double ds) {
  switch (window) {
    case LCT_WINDOW_HANN:  // 0.5 + 0.5 cos(2 pi f): a [1/4, 1/2, 1/4] smoothing of the taps
      return 0.5 * base_kernel(kind, n, ds) +
             0.25 * (base_kernel(kind, n - 1, ds) + base_kernel(kind, n + 1, ds));
    case LCT_WINDOW_HAMMING:  // 0.54 + 0.46 cos(2 pi f)
      return 0.54 * base_kernel(kind, n, ds) +
             0.23 * (base_kernel(kind, n - 1, ds) + base_kernel(kind, n + 1, ds));
    case LCT_WINDOW_COSINE:  // cos(pi f): mean of the kernel half a sample either side
      return 0.5 * (base_kernel(kind, n - 0.5, ds) + base_kernel(kind, n + 0.5, ds));
    default:
      return base_kernel(kind, n, ds);
  }
}

}  // namespace lct

using namespace lct;

LCT_API int lct_filter_taps(int kind, int window, int ns, float ds, float* h) {
  if (!h || ns <= 0 || !(ds > 0.f)) return LCT_ERR_ARG;
  if (kind != LCT_FILTER_RAMLAK && kind != LCT_FILTER_SHEPP_LOGAN) return LCT_ERR_ARG;
  if (window < LCT_WINDOW_NONE || window > LCT_WINDOW_COSINE) return LCT_ERR_ARG;
  for (int i = 0; i < 2 * ns; ++i) {
    int n = i - ns;
    if (kind == LCT_FILTER_RAMLAK && window == LCT_WINDOW_NONE) {
      // Src/Filter.cpp:13-19, the same expression (double, stored as float)
      if (n == 0)
        h[i] = 0.25 / ds;
      else
        h[i] = (std::sin(n * kRefPi) / (n * kRefPi) +
                (std::cos(n * kRefPi) - 1) / (n * n * kRefPi * kRefPi)) /
               (2 * ds);
    } else {
      h[i] = (float)windowed(kind, window, n, (double)ds);
    }
  }
  return LCT_OK;
}

namespace lct {

// ---------------------------------------------------------------------------------------
// FP32 convolution in the reference's order.  Bound: the FP32 FMA pipe, so the operands have to
// come cheaply: shared memory returns 128 bytes per clock and SM, a quarter of what 128 FMA lanes
// would ask for if every FMA loaded one operand.  A thread therefore makes a tile of 8 rows x 8
// consecutive outputs: per k it loads the 8 rows' samples (two 16-byte broadcasts of the rows
// interleaved [k][row]) and ONE tap -- output j at k + 1 uses output j - 1's tap at k, so the
// other seven stay in registers (a ring of eight, its positions fixed by unrolling k by 8) -- for
// 64 FMAs, issued as 32 packed FP32 pairs of two rows (each lane rounded as a scalar fmaf, k
// increasing: bit-exact with the reference's sum).
// Taps are padded by one word in nine so that lanes 8 outputs apart fall on different banks.
// 56,128 rows of 672 (with their rebin): 1.03 ms, 2.18 ms with 16 rows x 1 output per thread, which
// asked shared memory for 17 words per 16 FMAs (23 of the chip's 74 TFLOP/s).
// ---------------------------------------------------------------------------------------
constexpr int kFiltR = 8;         // rows per thread, and per row group in shared memory
constexpr int kFiltC = 8;         // outputs per thread
constexpr int kFiltBlk = 8 * kFiltR + 4;  // words of 8 k: padded, so that staging stores spread over the banks
constexpr int kFiltThreads = 256; // most threads of a CTA

// front padding that puts tap index ns on a multiple of 8, and the padded taps' words
__host__ __device__ __forceinline__ int filt_front(int ns) { return 8 + (8 - (ns & 7)) % 8; }
__host__ __device__ __forceinline__ int filt_tap_words(int ns) {
  return ((filt_front(ns) + 2 * ns + 8) * 9 / 8 + 8) / 4 * 4;
}

// grid ceil(row groups / rg); CTA: rg groups of 8 rows x all ns outputs, thread items
// (row group, 8 outputs) flattened so that a warp may hold two row groups' ends
__global__ void __launch_bounds__(kFiltThreads, 2)
    filter_fp32_kernel(const float* __restrict__ h, float* __restrict__ rows, long long nrows, int ns,
                       int rg) {
  extern __shared__ __align__(16) float sm[];
  const int front = filt_front(ns);
  float* s_h = sm;                        // tap i at (i + front) * 9 / 8
  float* s_r = sm + filt_tap_words(ns);   // [rg][ns / 8][8 k][8 rows] + 4 words per 8 k
  const long long r0 = (long long)blockIdx.x * rg * kFiltR;
#pragma unroll 4
  for (int i = threadIdx.x; i < front + 2 * ns + 8; i += blockDim.x) {
    const int k = i - front;
    s_h[i + (i >> 3)] = (k >= 0 && k < 2 * ns) ? h[k] : 0.0f;
  }
  // asynchronous 4-byte copies (transposing, all in flight at once: a small CTA would otherwise
  // wait for its loads in turn); rows past the end are zero-filled
  const int nsb = (ns + 7) / 8;
  for (int r = 0; r < rg * kFiltR; ++r) {
    const unsigned bytes = r0 + r < nrows ? 4u : 0u;
    const float* src = rows + (bytes ? r0 + r : r0) * ns;
    const uint32_t dst = smem_u32(s_r + (r / kFiltR) * nsb * kFiltBlk + r % kFiltR);
#pragma unroll 4
    for (int k = threadIdx.x; k < ns; k += blockDim.x)
      cp_async4(dst + 4u * ((k >> 3) * kFiltBlk + (k & 7) * kFiltR), src + k, bytes);
  }
  cp_async_wait_all();
  __syncthreads();
  const int groups = (ns + kFiltC - 1) / kFiltC;
  const bool vec = (ns & 3) == 0 && (reinterpret_cast<uintptr_t>(rows) & 15) == 0;
  for (int item = threadIdx.x; item < groups * rg; item += blockDim.x) {
    const int gr = item / groups, cg = item - gr * groups;
    const float* x = s_r + gr * nsb * kFiltBlk;
    const float* t = s_h + cg * 9 + (ns + front) / 8 * 9;  // tap of output 0 at k = 0
    float2 acc[kFiltC][kFiltR / 2];
#pragma unroll
    for (int j = 0; j < kFiltC; ++j)
#pragma unroll
      for (int q = 0; q < kFiltR / 2; ++q) acc[j][q] = make_float2(0.0f, 0.0f);
    float2 ring[8];  // (tap, tap): output j at k = k0 + u in ring[(j - u) & 7]
#pragma unroll
    for (int j = 1; j < 8; ++j) ring[j] = make_float2(t[j], t[j]);
    auto step = [&](int u) {  // u = k mod 8, a constant after unrolling
      const float tap = u == 0 ? t[0] : t[-u - 1];
      ring[(8 - u) & 7] = make_float2(tap, tap);
      const float4 a = *reinterpret_cast<const float4*>(x + u * kFiltR);
      const float4 b = *reinterpret_cast<const float4*>(x + u * kFiltR + 4);
      const float2 v[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y),
                           make_float2(b.z, b.w)};
#pragma unroll
      for (int j = 0; j < kFiltC; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[j][q] = __ffma2_rn(ring[(j - u) & 7], v[q], acc[j][q]);
    };
    int k = 0;
    for (; k + 8 <= ns; k += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) step(u);
      t -= 9;
      x += kFiltBlk;
    }
#pragma unroll
    for (int u = 0; u < 7; ++u)
      if (k + u < ns) step(u);
    const int is0 = cg * kFiltC;
#pragma unroll
    for (int r = 0; r < kFiltR; ++r) {
      const long long row = r0 + gr * kFiltR + r;
      if (row >= nrows) break;
      float* o = rows + row * ns + is0;
      float y[kFiltC];
#pragma unroll
      for (int j = 0; j < kFiltC; ++j) y[j] = (r & 1) ? acc[j][r / 2].y : acc[j][r / 2].x;
      if (vec && is0 + kFiltC <= ns) {
        *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
        *reinterpret_cast<float4*>(o + 4) = make_float4(y[4], y[5], y[6], y[7]);
      } else {
#pragma unroll
        for (int j = 0; j < kFiltC; ++j)
          if (is0 + j < ns) o[j] = y[j];
      }
    }
  }
}

// Row groups per CTA: the fewest warps on the busiest SM, counting the lanes that the last warp of
// a CTA leaves idle; ties to the smaller CTA.
static int filt_row_groups(long long row_groups, int ns, int sms, size_t* smem) {
  const int groups = (ns + kFiltC - 1) / kFiltC;
  int best = 1;
  long long best_cost = 0;
  for (int rg = 1; rg == 1 || (groups * rg <= kFiltThreads && rg <= 32); ++rg) {
    const size_t b = sizeof(float) * (filt_tap_words(ns) + (size_t)rg * ((ns + 7) / 8) * kFiltBlk);
    if (rg > 1 && b > 96 * 1024) break;
    const long long ctas = (row_groups + rg - 1) / rg;
    const long long cost = (ctas + sms - 1) / sms * ((groups * rg + 31) / 32);
    if (rg == 1 || cost < best_cost) {
      best = rg;
      best_cost = cost;
      *smem = b;
    }
  }
  return best;
}

int launch_filter_rows(int ns, const float* d_h, float* d_rows, long long nrows, int mode,
                       cudaStream_t s) {
  if (nrows <= 0) return LCT_OK;
  if (mode == LCT_FILTER_BF16X3 || mode == LCT_FILTER_BF16X6)
    return launch_filter_tc(ns, d_h, d_rows, nrows, mode, s);
  static std::mutex mu;
  static int sms_of[64] = {0};                 // 0: attribute not set yet on that device
  static unsigned long long ctx_of[64] = {0};  // and in that context
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  const unsigned long long ctx = context_id();
  {
    std::lock_guard<std::mutex> lock(mu);  // host threads may share a device
    if (dev >= 64 || !sms_of[dev] || ctx_of[dev] != ctx) {
      int st = cuda_status(cudaFuncSetAttribute(filter_fp32_kernel,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                200 * 1024));
      if (!st) st = cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      if (st) return st;
      if (dev < 64) {
        sms_of[dev] = sms;
        ctx_of[dev] = ctx;
      }
    } else {
      sms = sms_of[dev];
    }
  }
  const long long row_groups = (nrows + kFiltR - 1) / kFiltR;
  size_t smem = 0;
  const int rg = filt_row_groups(row_groups, ns, sms, &smem);
  const long long nblk = (row_groups + rg - 1) / rg;
  if (nblk > 0x7fffffffLL) return LCT_ERR_ARG;
  const int items = (ns + kFiltC - 1) / kFiltC * rg;
  const int threads = std::min(kFiltThreads, (items + 31) / 32 * 32);
  filter_fp32_kernel<<<(unsigned)nblk, threads, smem, s>>>(d_h, d_rows, nrows, ns, rg);
  return launch_status();
}

}  // namespace lct

LCT_API int lct_filter_rows(int ns, const float* d_h, float* d_rows, int64_t nrows, int mode,
                            lct_stream stream) {
  if (ns <= 0 || ns > 3072 || !d_h || !d_rows || nrows < 0) return LCT_ERR_ARG;
  if (mode != LCT_FILTER_FP32 && mode != LCT_FILTER_BF16X3 && mode != LCT_FILTER_BF16X6)
    return LCT_ERR_ARG;
  return launch_filter_rows(ns, d_h, d_rows, nrows, mode, (cudaStream_t)stream);
}
