// Stage 3 on the tensor cores: the row convolution as a Toeplitz GEMM, BF16x3 on tcgen05.
//
// out[r][n] = sum_k rows[r][k] * h[n - k + ns]  (CUDA/Filter.cu:42-46) is out = R * T with
// T[k][n] = h[n - k + ns].  Both operands are split into bf16 high and low parts
// (x = hi + lo + O(2^-18 x)), and the product is accumulated in FP32 as
//   R*T ~= Rhi*Thi + Rhi*Tlo + Rlo*Thi
// (the dropped Rlo*Tlo term and the split residue are ~2^-16 relative per product).
//
// GEMM D[M x N] = A[M x K] B[K x N] with A = rows (K-major, as stored) and B given K-major as
// B^T[n][k] = h[n - k + ns] (itself Toeplitz, materialised once per taps), both zero padded to whole K
// slices.  Persistent CTAs take tiles of D, 128 rows x up to 256 columns (tc_width), columns fastest (a
// row block's planes then come from L2 for its second and third tile):
//   * warp 0 issues TMA loads (tiled, 64-byte swizzle, no multicast) of 32-deep K slices -- P planes of
//     A (128 x 32) and of B (width x 32) -- into a ring of 3 to 6 stages;
//   * warp 1 issues tcgen05.mma.kind::f16 (M128, N up to 256, K16, BF16 in, FP32 accumulate in TMEM; 3 or
//     6 products per K16 step) into one of two accumulators and frees each stage with tcgen05.commit;
//   * warps 2-5 drain the other accumulator (tcgen05.ld 32x32b) and store the columns n < ns.
// Bound: tensor pipe and TMA.  Loading an M128 operand costs about 64 clocks and a column of N 0.4, so
// N is as wide as TMEM takes twice.  117,312 rows of 736, P = 3: 0.53 ms; 128 x 128 tiles, one per CTA with
// load, math and store in turn, 0.69 ms.
// Every mbarrier wait is bounded; a wait that runs out raises the device status word, the CTA
// stops issuing work, waits (bounded) for the copies it started, frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <mutex>

#include "lct_internal.h"
#include "tc_ptx.cuh"

namespace lct {

constexpr int kTcM = 128, kTcN = 256, kTcK = 32, kTcThreads = 192, kTcMaxStages = 6;
constexpr uint32_t kTcSmem = 225 * 1024;  // dynamic shared memory: stages and alignment

// P = bf16 planes per operand: P = 2 -> 3 products (BF16x3), P = 3 -> 6 products (BF16x6).
// a stage: P planes of A (128 x 32) and of B (width x 32)
constexpr uint32_t kTcTileA = kTcM * kTcK * 2;
__host__ __device__ constexpr uint32_t tc_tile_b(int width) { return (uint32_t)width * kTcK * 2; }

// planes are padded to whole 64-byte K slices, so that every row of a TMA box is aligned (404 columns
// padded to 408, 816-byte rows: 3,500 clocks a stage instead of 2,200)
__host__ __device__ inline int tc_pad(int ns) { return (ns + kTcK - 1) / kTcK * kTcK; }

// ---------------------------------------------------------------------------------------
// operand preparation
// ---------------------------------------------------------------------------------------
// x = p[0] + p[1] (+ p[2]) + residue: each plane the bf16 rounding of what the previous left
template <int P>
__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16 (&p)[P]) {
#pragma unroll
  for (int i = 0; i < P; ++i) {
    p[i] = __float2bfloat16_rn(x);
    x -= __bfloat162float(p[i]);
  }
}

// rows fp32 [M][ns] -> P planes [M][kpad] (zero columns k >= ns); plane stride m * kpad.  A thread
// block takes one row
template <int P>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ rows, long long m,
                                                         int ns, int kpad,
                                                         __nv_bfloat16* __restrict__ planes) {
  const long long r = blockIdx.x;
  if (r >= m) return;
  const long long pstride = m * kpad;
  for (int k = threadIdx.x; k < kpad; k += blockDim.x) {
    __nv_bfloat16 v[P];
    split_bf16<P>(k < ns ? rows[r * ns + k] : 0.0f, v);
#pragma unroll
    for (int i = 0; i < P; ++i) planes[i * pstride + r * kpad + k] = v[i];
  }
}

// The same split, 4 columns per thread and kSplitRows rows per block: 16-byte loads and 8-byte
// stores (4 bf16) per plane instead of scalar ones.  Needs ns and kpad multiples of 4 and a
// 16-byte aligned row base; every element is split exactly as above.
constexpr int kSplitRows = 4;

template <int P>
__global__ void __launch_bounds__(256) split_rows4_kernel(const float4* __restrict__ rows,
                                                          long long m, int ns4, int kpad4,
                                                          uint2* __restrict__ planes) {
  const long long r0 = (long long)blockIdx.x * kSplitRows;
  const long long pstride4 = m * kpad4;  // plane stride in groups of 4
  for (int j = 0; j < kSplitRows; ++j) {
    const long long r = r0 + j;
    if (r >= m) return;
    for (int k4 = threadIdx.x; k4 < kpad4; k4 += blockDim.x) {
      const float4 x = k4 < ns4 ? __ldg(rows + r * ns4 + k4) : make_float4(0.f, 0.f, 0.f, 0.f);
      __nv_bfloat16 v0[P], v1[P], v2[P], v3[P];
      split_bf16<P>(x.x, v0);
      split_bf16<P>(x.y, v1);
      split_bf16<P>(x.z, v2);
      split_bf16<P>(x.w, v3);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        uint2 q;
        q.x = (unsigned)__bfloat16_as_ushort(v0[i]) | ((unsigned)__bfloat16_as_ushort(v1[i]) << 16);
        q.y = (unsigned)__bfloat16_as_ushort(v2[i]) | ((unsigned)__bfloat16_as_ushort(v3[i]) << 16);
        planes[i * pstride4 + r * kpad4 + k4] = q;
      }
    }
  }
}

// B^T[n][k] = h[n - k + ns] for n, k < ns, else 0; P planes [kpad][kpad]
template <int P>
__global__ void __launch_bounds__(256) toeplitz_kernel(const float* __restrict__ h, int ns, int kpad,
                                                       __nv_bfloat16* __restrict__ planes) {
  const int n = blockIdx.x;
  const long long pstride = (long long)kpad * kpad;
  for (int k = threadIdx.x; k < kpad; k += blockDim.x) {
    __nv_bfloat16 v[P];
    split_bf16<P>((n < ns && k < ns) ? h[n - k + ns] : 0.0f, v);
#pragma unroll
    for (int i = 0; i < P; ++i) planes[i * pstride + (long long)n * kpad + k] = v[i];
  }
}

// ---------------------------------------------------------------------------------------
// the GEMM: grid min(tiles, SMs), 192 threads; tiles of 128 rows x `width` columns, S stages.
// Products per K16 step: P = 2: (0,0) (0,1) (1,0);  P = 3: those and (0,2) (1,1) (2,0).
// ---------------------------------------------------------------------------------------
template <int P>
struct TcMaps {
  CUtensorMap a[P];
  CUtensorMap b[P];
};

template <int P>
__global__ void __launch_bounds__(kTcThreads, 1)
    filter_tc_kernel(const __grid_constant__ TcMaps<P> maps, float* __restrict__ out, long long m,
                     int ns, int width, int S, int n_tiles_n, long long n_tiles, int* status) {
  const uint32_t tile_b = tc_tile_b(width), stage = P * (kTcTileA + tile_b);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ __align__(8) uint64_t bars[2 * kTcMaxStages + 5];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;

  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t stage0 = smem_u32(smem);
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kTcMaxStages]);
  const uint32_t accf0 = smem_u32(&bars[2 * kTcMaxStages]), acce0 = accf0 + 16, mdone = accf0 + 32;
  const int ktiles = (ns + kTcK - 1) / kTcK;

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accf0 + 8 * i, 1);
      mbar_init(acce0 + 8 * i, 4);  // one arrival per epilogue warp
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(2 * kTcN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_slot, 0);
  auto aborted = [&] { return *reinterpret_cast<volatile int*>(&s_abort) != 0; };

  if (warp == 0) {
    if (lane == 0) {
      long long kg = 0;  // slices issued
      bool stop = false;
      for (long long t = blockIdx.x; t < n_tiles && !stop; t += gridDim.x) {
        const int n0 = (int)(t % n_tiles_n) * width, m0 = (int)(t / n_tiles_n) * kTcM;
        for (int kt = 0; kt < ktiles; ++kt, ++kg) {
          const int s = (int)(kg % S);
          if (kg >= S && !mbar_wait(empty0 + 8 * s, (uint32_t)(((kg / S) - 1) & 1))) {
            atomicExch(&s_abort, 1);
            stop = true;
            break;
          }
          if (aborted()) {
            stop = true;
            break;
          }
          const uint32_t st = stage0 + s * stage, fb = full0 + 8 * s;
          mbar_expect_tx(fb, stage);
#pragma unroll
          for (int i = 0; i < P; ++i) tma_load_2d(st + i * kTcTileA, &maps.a[i], kt * kTcK, m0, fb);
#pragma unroll
          for (int i = 0; i < P; ++i)
            tma_load_2d(st + P * kTcTileA + i * tile_b, &maps.b[i], kt * kTcK, n0, fb);
        }
      }
      if (aborted())  // copies still in flight land on their full barriers before the CTA may exit
        for (long long q = (kg > S ? kg - S : 0); q < kg; ++q)
          mbar_wait(full0 + 8 * (int)(q % S), (uint32_t)((q / S) & 1));
    }
  } else if (warp == 1) {
    // the whole warp runs the loop, so that descriptors stay warp-uniform; one elected lane issues
    long long kg = 0, it = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, ++it) {
      const int buf = (int)(it & 1), n0 = (int)(t % n_tiles_n) * width;
      const int n = min(width, (ns - n0 + 15) / 16 * 16);
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
                             ((uint32_t)(kTcM >> 4) << 24);
      const uint32_t d = tmem + (uint32_t)(buf * kTcN);
      ok = __all_sync(0xFFFFFFFFu, it < 2 || mbar_wait(acce0 + 8 * buf, (uint32_t)(((it >> 1) - 1) & 1)));
      for (int kt = 0; kt < ktiles && ok; ++kt, ++kg) {
        const int s = (int)(kg % S);
        ok = __all_sync(0xFFFFFFFFu, mbar_wait(full0 + 8 * s, (uint32_t)((kg / S) & 1)) && !aborted());
        if (!ok) break;
        tc_fence_after();
        const uint32_t st = stage0 + s * stage;
        if (elect_one()) {
          uint64_t a[P], b[P];
#pragma unroll
          for (int i = 0; i < P; ++i) {
            a[i] = desc_sw64(st + i * kTcTileA);
            b[i] = desc_sw64(st + P * kTcTileA + i * tile_b);
          }
#pragma unroll
          for (int j = 0; j < kTcK / 16; ++j) {
            const uint64_t dk = (uint64_t)((j * 32) >> 4);  // 16 bf16 = 32 bytes along K
            umma_bf16(d, a[0] + dk, b[0] + dk, idesc, (kt | j) ? 1u : 0u);
            umma_bf16(d, a[0] + dk, b[1] + dk, idesc, 1u);
            umma_bf16(d, a[1] + dk, b[0] + dk, idesc, 1u);
            if (P == 3) {
              umma_bf16(d, a[0] + dk, b[P - 1] + dk, idesc, 1u);
              umma_bf16(d, a[1] + dk, b[1] + dk, idesc, 1u);
              umma_bf16(d, a[P - 1] + dk, b[0] + dk, idesc, 1u);
            }
          }
          umma_commit(empty0 + 8 * s);
          if (kt == ktiles - 1) umma_commit(accf0 + 8 * buf);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) atomicExch(&s_abort, 1);
    }
    if (elect_one()) umma_commit(mdone);  // every MMA issued above has finished once this arrives
    __syncwarp();
    if (!mbar_wait(mdone, 0)) atomicExch(&s_abort, 1);
  } else {
    // epilogue: the warp of quadrant q holds rows 32 q .. + 31 of the tile
    const int q = warp & 3;
    // 32-byte stores (whole sectors) where every row starts on 32 bytes, 16-byte ones on 16 bytes
    const bool vec8 = ((ns & 7) == 0) && ((reinterpret_cast<uintptr_t>(out) & 31) == 0);
    const bool vec = ((ns & 3) == 0) && ((reinterpret_cast<uintptr_t>(out) & 15) == 0);
    long long it = 0;
    for (long long t = blockIdx.x; t < n_tiles; t += gridDim.x, ++it) {
      const int buf = (int)(it & 1), n0 = (int)(t % n_tiles_n) * width;
      const long long row = (t / n_tiles_n) * kTcM + q * 32 + lane;
      // warp-uniform decision: the TMEM loads below are .sync.aligned
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(accf0 + 8 * buf, (uint32_t)((it >> 1) & 1)))) {
        if (lane == 0) atomicExch(&s_abort, 1);
        break;
      }
      if (__any_sync(0xFFFFFFFFu, aborted())) break;
      tc_fence_after();
      float* orow = out + row * ns;
      const int cols = min(width, ns - n0);
#pragma unroll 1
      for (int c = 0; c < cols; c += 32) {
        uint32_t r[32];
        tmem_ld32(tmem + (uint32_t)(buf * kTcN + c) + ((uint32_t)(q * 32) << 16), r);
        const int col0 = n0 + c;
        if (row < m) {
          if (vec8 && c + 32 <= cols) {
#pragma unroll
            for (int i = 0; i < 32; i += 8)
              stg256(orow + col0 + i, r[i], r[i + 1], r[i + 2], r[i + 3], r[i + 4], r[i + 5], r[i + 6], r[i + 7]);
          } else if (vec && c + 32 <= cols) {
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              *reinterpret_cast<float4*>(orow + col0 + i) =
                  make_float4(__uint_as_float(r[i]), __uint_as_float(r[i + 1]),
                              __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c + i < cols) orow[col0 + i] = __uint_as_float(r[i]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acce0 + 8 * buf);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && aborted() && status) atomicExch(status, kDevWaitTimeout);
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(2 * kTcN)
                 : "memory");
}

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

// 2-D bf16 tensor [rows][cols] (cols contiguous), box {kTcK, box_rows}, 64-byte swizzle
static int make_map(CUtensorMap* map, const void* base, long long rows, int cols, int box_rows) {
  auto fn = tensor_map_encoder();
  if (!fn) return LCT_ERR_UNSUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  cuuint32_t box[2] = {(cuuint32_t)kTcK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LCT_OK : LCT_ERR_ARG;
}

static int planes_of(int mode) { return mode == LCT_FILTER_BF16X6 ? 3 : 2; }

// scratch: P Toeplitz planes [kpad][kpad], then P row planes [rows_cap][kpad]
size_t tc_scratch_bytes(int ns, long long rows_cap, int mode) {
  const long long kp = tc_pad(ns);
  const int P = planes_of(mode);
  return sizeof(__nv_bfloat16) * (size_t)P * ((size_t)rows_cap * kp + (size_t)kp * kp);
}

int tc_build_toeplitz(int ns, const float* d_h, void* scratch, int mode, cudaStream_t s) {
  const int kp = tc_pad(ns);
  __nv_bfloat16* b = static_cast<__nv_bfloat16*>(scratch);
  if (planes_of(mode) == 3)
    toeplitz_kernel<3><<<kp, 256, 0, s>>>(d_h, ns, kp, b);
  else
    toeplitz_kernel<2><<<kp, 256, 0, s>>>(d_h, ns, kp, b);
  return launch_status();
}

// Tile width: few wide tiles cost fewer operand loads, many narrow ones fill the last round of SMs and
// leave less epilogue exposed at the end.  Per MMA about 64 + 0.37 width clocks, or what TMA takes to
// deliver the stage (29 bytes per clock and SM in rows of 64 bytes, few SMs loading or all).  736 columns,
// clocks per MMA: 256 wide 211, 192 wide 185, 128 wide 144.
static int tc_width(int ns, long long mt, int P, int sms) {
  const int prods = P == 3 ? 6 : 3;
  const double steps = (double)((ns + kTcK - 1) / kTcK) * 2 * prods;
  int best = kTcN;
  double best_cost = 1e300;
  for (int nt = (ns + kTcN - 1) / kTcN; nt <= (ns + 63) / 64; ++nt) {
    const int w = ((ns + nt - 1) / nt + 15) / 16 * 16;
    const long long tiles = mt * ((ns + w - 1) / w);
    const double mma = std::max(64.0 + 0.37 * w, P * (kTcTileA + (double)tc_tile_b(w)) / (2 * prods) / 29.0);
    const double cost = (double)((tiles + sms - 1) / sms) * steps * mma + 20.0 * w;
    if (cost < best_cost) {
      best_cost = cost;
      best = w;
    }
  }
  return best;
}

template <int P>
static int tc_filter_p(int ns, float* d_rows, long long nrows, void* scratch, cudaStream_t s) {
  const int kp = tc_pad(ns);
  const long long mt = (nrows + kTcM - 1) / kTcM;
  if (mt > 65535) return LCT_ERR_ARG;
  __nv_bfloat16* b = static_cast<__nv_bfloat16*>(scratch);
  __nv_bfloat16* a = b + (size_t)P * kp * kp;  // 64-byte aligned: kp is a multiple of 32
  if (ns % 4 == 0 && reinterpret_cast<uintptr_t>(d_rows) % 16 == 0 &&
      reinterpret_cast<uintptr_t>(a) % 8 == 0)
    split_rows4_kernel<P><<<(unsigned)((nrows + kSplitRows - 1) / kSplitRows), 256, 0, s>>>(
        reinterpret_cast<const float4*>(d_rows), nrows, ns / 4, kp / 4, reinterpret_cast<uint2*>(a));
  else
    split_rows_kernel<P><<<(unsigned)nrows, 256, 0, s>>>(d_rows, nrows, ns, kp, a);
  int st = launch_status();
  if (st) return st;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  {
    static std::mutex mu;  // host threads may share a device
    static int sms_of[64] = {0};                 // 0: attribute not set yet on that device
    static unsigned long long ctx_of[64] = {0};  // and in that context
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !sms_of[dev] || ctx_of[dev] != ctx) {
      if ((st = cuda_status(cudaFuncSetAttribute(filter_tc_kernel<P>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kTcSmem))))
        return st;
      if ((st = cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)))) return st;
      if (dev < 64) {
        sms_of[dev] = sms;
        ctx_of[dev] = ctx;
      }
    } else {
      sms = sms_of[dev];
    }
  }
  const int w = tc_width(ns, mt, P, sms);
  TcMaps<P> maps;
  for (int i = 0; i < P; ++i) {
    if ((st = make_map(&maps.a[i], a + (size_t)i * nrows * kp, nrows, kp, kTcM))) return st;
    if ((st = make_map(&maps.b[i], b + (size_t)i * kp * kp, kp, kp, w))) return st;
  }
  const uint32_t stage = P * (kTcTileA + tc_tile_b(w));
  const int S = (int)std::min<uint32_t>(kTcMaxStages, (kTcSmem - 1024) / stage);
  const int nt = (ns + w - 1) / w;
  filter_tc_kernel<P><<<(unsigned)std::min<long long>(mt * nt, sms), kTcThreads, S * stage + 1024, s>>>(
      maps, d_rows, nrows, ns, w, S, nt, mt * nt, device_status_ptr());
  return launch_status();
}

// split + GEMM over nrows rows (nrows <= rows_cap the scratch was sized for), in place
int tc_filter(int ns, float* d_rows, long long nrows, void* scratch, long long rows_cap, int mode,
              cudaStream_t s) {
  if (nrows <= 0) return LCT_OK;
  if (nrows > rows_cap || nrows > 0x7fffffffLL) return LCT_ERR_ARG;
  return planes_of(mode) == 3 ? tc_filter_p<3>(ns, d_rows, nrows, scratch, s)
                              : tc_filter_p<2>(ns, d_rows, nrows, scratch, s);
}

// stage-level entry: stream-ordered scratch for this call
int launch_filter_tc(int ns, const float* d_h, float* d_rows, long long nrows, int mode,
                     cudaStream_t s) {
  if (nrows <= 0) return LCT_OK;
  void* scratch = nullptr;
  if (scratch_alloc(&scratch, tc_scratch_bytes(ns, nrows, mode), s))
    return LCT_ERR_ALLOC;
  int st = tc_build_toeplitz(ns, d_h, scratch, mode, s);
  if (!st) st = tc_filter(ns, d_rows, nrows, scratch, nrows, mode, s);
  int st2 = scratch_free(scratch, s);
  return st ? st : st2;
}

}  // namespace lct
