// Learned 2.5D residual correction after backprojection (no reference counterpart; the
// reference stops at the FDK volume, Src/Reconstructor.cpp).
//
// Network: 5 neighbouring slices of the (calibrated) FDK volume as channels -> 8 zero-padded
// 3x3 convolutions (5->32, 6 x 32->32, 32->1), ReLU between them -> a residual r added to the
// centre slice.  BF16 weights and activations, FP32 accumulation.
//
// HBM layout: every activation / delta is bf16 [B][H + 2][4][wp][8]: per padded row four planes of
// eight channels, 16 bytes per pixel and plane; pixel x of row y at column x + 1 of row y + 1, wp = W + 2
// rounded up to 8.  Rows 0 and H + 1 and the columns outside the image stay zero.  The network input has one plane (5 channels, 3 zero).  A
// staged tile is one TMA box, and in shared memory eight pixels of a plane are one unswizzled core
// matrix: an operand may start at any pixel, so ONE box serves all nine taps.  (TMA sees 8-byte
// elements, two per pixel, in blocks of 8 pixels where a box is wider than 128.)
// Weights are packed per layer as bf16 [32][9 taps x 32 channels].
//
// Convolution on tcgen05, persistent and warp-specialised: a tile is 8 output rows x up to 128 pixels.
// Pixels are the M operand, and the three vertical taps of one column offset the N operand: input row r
// (of ten), column offset dx and 16 channels are ONE M128 x N96 x K16 MMA that adds tap (dy, dx) to the
// accumulators of output rows r - 2, r - 1 and r, 32 columns apart in tensor memory, so a pixel's
// channels are read from shared memory 3 x 10 / 8 times instead of 9 (N64 and N32 at the tile's edges).
// Two buffers of 8 x 32 columns fill tensor memory; the packed weights sit in shared memory for the
// CTA's lifetime.  Per output the taps add in the order (dx, dy, channel half).  Launches of few tiles take
// lower ones (conv_height).  The first tiles' boxes load while the CTA stages its weights and zeroes its
// accumulators (64^2 x 16 slices: 83 us a forward pass, 93 with the loads after that).
// Bound: shared-memory operand reads (7 KB per MMA), then HBM.  512 x 512, 32 slices: 190 us per
// hidden layer; one tap per MMA (M128 x N32, three boxes per tile) 308 us.
// Fused epilogues: bias + ReLU -> bf16 (forward), ReLU mask of the previous activation -> bf16 delta
// (backward data), FP32 residual (training), and the acceptance gate writing the corrected volume
// (inference).
// Weight gradients: tcgen05 with K = pixels (both operands MN-major from the same layout).
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <new>
#include <type_traits>
#include <vector>

#include "lct_internal.h"
#include "tc_ptx.cuh"

namespace lct {

constexpr int kCnnLayers = 8, kCnnC = 32, kCnnTaps = 9, kCnnK = kCnnTaps * kCnnC;  // K = 288
constexpr int kCnnParams = 57249;     // sum over layers of cin*cout*9 + cout
constexpr int kWSlot = kCnnC * kCnnK;  // packed weights of one layer, elements
constexpr int kConvHeights = 3;   // output rows of a tile: 8, 4 or 2 (conv_height)
LCT_HD constexpr int conv_rows(int height) { return 8 >> height; }
constexpr int kConvMaxN = 128;    // pixels of a tile, a multiple of 8 (its box starts on a block)
constexpr int kConvThreads = 320; // warp 0 copies, warp 1 MMA + TMEM, warps 2-9 epilogue
constexpr int kConvMaxStages = 8;
constexpr uint32_t kConvZero = 128 * 16 + 32;  // a plane of zeros for the network input's absent channels
constexpr uint32_t kSmemMax = 226 * 1024;      // dynamic shared memory of the CNN kernels

LCT_HD constexpr int cnn_cin(int l) { return l == 0 ? 5 : 32; }
LCT_HD constexpr int cnn_cout(int l) { return l == kCnnLayers - 1 ? 1 : 32; }
LCT_HD constexpr int cnn_off(int l) { return l == 0 ? 0 : 1472 + (l - 1) * 9248; }

enum ConvEpi : int { kEpiRelu = 0, kEpiMask = 1, kEpiResid = 2, kEpiGate = 3 };

struct ConvArgs {
  int H, W, wp, n_px, tiles_x, tiles_y, stages;
  int rows;                        // output rows of a tile
  uint32_t stage_bytes;
  long long n_tiles;
  const __nv_bfloat16* w;          // packed weights
  const float* bias;               // [32] (forward epilogues; [1] for the last layer)
  float* out_f;                    // Resid: r [B][H][W]; Gate: corrected slices [B][H][W]
  const float* xc;                 // Gate: plain slices [B][H][W]
  __nv_bfloat16* out_act;          // Relu / Mask: [B][H + 2][4][wp][8]
  const __nv_bfloat16* mask_act;   // Mask: activation whose sign gates the delta
  float calib, inv_scale, bound;   // Gate
  unsigned long long* n_reject;    // Gate
  int* status;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// tile t: slice b, first output row y0, first pixel x0
__device__ __forceinline__ void conv_tile(const ConvArgs& a, long long t, int& x0, int& y0, int& b) {
  const long long per = (long long)a.tiles_x * a.tiles_y;
  b = (int)(t / per);
  const int r = (int)(t % per);
  y0 = (r / a.tiles_x) * a.rows;
  x0 = (r % a.tiles_x) * a.n_px;
}

__device__ __forceinline__ bool conv_aborted(int* flag) {
  return *reinterpret_cast<volatile int*>(flag) != 0;
}

// bytes of a plane of a staged row: a convolution's (the pixels and a block of 8), a gradient's
// activation (the pixels and one on each side)
LCT_HD constexpr uint32_t conv_plane(int n_px) { return (uint32_t)(n_px + 8) * 16; }
LCT_HD constexpr uint32_t dw_plane(int n_px) { return (uint32_t)(n_px + 2) * 16; }

// PLANES: planes of the input (1: the network input, whose channels 8..15 read a zeroed plane of
// shared memory and whose second half of 16 channels does not exist; 4: an activation).
// ROWS: output rows of a tile.
// Every wait is bounded; on a timeout the CTA drains its copies and MMAs, raises the device status
// word and leaves its remaining tiles unwritten.
template <int EPI, int PLANES, int ROWS>
__global__ void __launch_bounds__(kConvThreads, 1)
    conv_tc_kernel(const __grid_constant__ CUtensorMap mbox, const ConvArgs a) {
  constexpr bool kLast = EPI == kEpiResid || EPI == kEpiGate;
  constexpr int kHalves = PLANES == 1 ? 1 : 2;  // K16 steps per tap
  constexpr int kCo = kLast ? 16 : 32;          // accumulator columns of an output row
  constexpr int kIn = ROWS + 2;                 // input rows of a tile
  constexpr uint32_t kBuf = ROWS * kCo;         // columns of a buffer
  constexpr uint32_t kTmem = 2 * kBuf;
  constexpr uint32_t kWPlane = 3 * kCo * 16, kWBlock = 2 * kWPlane;  // weights of (dx, half), [2][3 kCo][8]
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[2 * kConvMaxStages + 5];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;

  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int N = a.n_px, S = a.stages;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kConvMaxStages]);
  const uint32_t accf0 = smem_u32(&bars[2 * kConvMaxStages]), acce0 = accf0 + 16, mdone = accf0 + 32;
  // stages, (PLANES 1) the zero plane, weights; an operand's rows past the tile's pixels read on into
  // what follows, which only reaches accumulator rows that are not stored
  const uint32_t cs = conv_plane(N), rs = PLANES * cs;
  const uint32_t stage0 = smem_u32(smem), zero0 = stage0 + (uint32_t)S * a.stage_bytes;
  const uint32_t w0 = zero0 + (PLANES == 1 ? kConvZero : 0u);

  // tile t as the k-th of this CTA: one box (rows and columns outside the padded image read as zero)
  auto load = [&](long long t, long long k) {
    int x0, y0, b;
    conv_tile(a, t, x0, y0, b);
    const int s = (int)(k % S);
    mbar_expect_tx(full0 + 8 * s, kIn * rs);
    tma_load_5d(stage0 + s * a.stage_bytes, &mbox, 0, x0 / 8, 0, y0, b, full0 + 8 * s);
  };
  long long issued = 0;  // thread 0: tiles loaded
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(accf0 + 8 * i, 1);
      mbar_init(acce0 + 8 * i, 8);  // one arrival per epilogue warp
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    // the first tiles' loads under the set-up that follows
    for (; issued < S && blockIdx.x + issued * gridDim.x < a.n_tiles; ++issued)
      load(blockIdx.x + issued * gridDim.x, issued);
  }
  if (PLANES == 1)
    for (uint32_t i = threadIdx.x * 16; i < kConvZero; i += kConvThreads * 16)
      *reinterpret_cast<uint4*>(smem + (zero0 - stage0) + i) = make_uint4(0u, 0u, 0u, 0u);
  // weights: block (dx, half), plane of 8 channels, row (2 - dy) kCo + co
  for (int i = threadIdx.x; i < 3 * kHalves * 2 * 3 * kCo; i += kConvThreads) {
    const int row = i % (3 * kCo), c = i / (3 * kCo) % 2, blk = i / (6 * kCo);
    const int dy = 2 - row / kCo, co = row % kCo, dx = blk / kHalves, h = blk % kHalves;
    *reinterpret_cast<uint4*>(smem + (w0 - stage0) + blk * kWBlock + c * kWPlane + row * 16) =
        __ldg(reinterpret_cast<const uint4*>(a.w + co * kCnnK + (dy * 3 + dx) * kCnnC + 16 * h + 8 * c));
  }
  fence_async_smem();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(kTmem)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_slot, 0);  // uniform to the compiler
  if (warp >= 2) {  // accumulators start at zero, and the epilogue leaves them so
    for (uint32_t c = warp < 6 ? 0 : kBuf; c < (warp < 6 ? kBuf : kTmem); c += 16)
      tmem_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c);
    tmem_wait_st();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();

  if (warp == 0) {
    // producer: the tiles past the first S
    if (lane == 0) {
      long long k = issued;
      for (long long t = blockIdx.x + k * gridDim.x; t < a.n_tiles; t += gridDim.x, ++k) {
        if (!mbar_wait(empty0 + 8 * (int)(k % S), (uint32_t)(((k / S) - 1) & 1))) {
          atomicExch(&s_abort, 1);
          break;
        }
        if (conv_aborted(&s_abort)) break;
        load(t, k);
      }
      if (conv_aborted(&s_abort))  // let copies in flight land before the CTA exits
        for (long long q = (k > S ? k - S : 0); q < k; ++q)
          mbar_wait(full0 + 8 * (int)(q % S), (uint32_t)((q / S) & 1));
    }
  } else if (warp == 1) {
    // the whole warp runs the loop, so that descriptors and addresses stay warp-uniform values; one
    // elected lane issues
    long long k = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < a.n_tiles && ok; t += gridDim.x, ++k) {
      const int buf = (int)(k & 1), s = (int)(k % S);
      ok = __all_sync(0xFFFFFFFFu, (k < 2 || mbar_wait(acce0 + 8 * buf, (uint32_t)(((k >> 1) - 1) & 1))) &&
                                       mbar_wait(full0 + 8 * s, (uint32_t)((k / S) & 1)));
      if (!ok && lane == 0) atomicExch(&s_abort, 1);
      if (!ok || __any_sync(0xFFFFFFFFu, conv_aborted(&s_abort))) break;
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)buf * kBuf, st = stage0 + s * a.stage_bytes;
      if (elect_one()) {
#pragma unroll
        for (int dx = 0; dx < 3; ++dx)
#pragma unroll
          for (int r = 0; r < kIn; ++r) {
            // output rows j0 .. j1 take tap r - j of input row r
            const int j0 = r < 2 ? 0 : r - 2, j1 = r < ROWS ? r : ROWS - 1, n = (j1 - j0 + 1) * kCo;
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
#pragma unroll
            for (int h = 0; h < kHalves; ++h) {
              const uint32_t at = st + r * rs + 2 * h * cs + 16 * dx;
              const uint32_t wt = w0 + (dx * kHalves + h) * kWBlock + (2 - (r - j0)) * kCo * 16;
              umma_bf16(d + j0 * kCo, desc_plain(at, PLANES == 1 ? zero0 - at : cs, 128),
                        desc_plain(wt, kWPlane, 128), idesc, 1u);
            }
          }
        umma_commit(empty0 + 8 * s);
        umma_commit(accf0 + 8 * buf);
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(mdone);  // every MMA issued above has finished once this arrives
    __syncwarp();
    if (!mbar_wait(mdone, 0)) atomicExch(&s_abort, 1);
  } else {
    // epilogue: the two warps of quadrant q hold pixels 32 q .. + 31, a lane one pixel, half of the
    // output rows each
    constexpr int kRows = ROWS / 2;
    const int px = (warp & 3) * 32 + lane, j0 = warp < 6 ? 0 : kRows;
    const uint32_t tl = (uint32_t)((warp & 3) * 32) << 16;
    float bias[EPI == kEpiRelu ? 32 : 1];
    if constexpr (EPI == kEpiRelu) {
#pragma unroll
      for (int i = 0; i < 32; ++i) bias[i] = __ldg(a.bias + i);
    } else {
      bias[0] = kLast ? __ldg(a.bias) : 0.f;
    }
    const long long rowq = (long long)a.wp * 4;  // 16-byte units of a padded row
    long long k = 0;
    for (long long t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++k) {
      const int buf = (int)(k & 1);
      int x0, y0, b;
      conv_tile(a, t, x0, y0, b);
      y0 += j0;
      const int x = x0 + px, rows = min(kRows, a.H - y0);
      const bool in = px < N && x < a.W;
      // plane 0 of the pixel in this warp's first row, and the pixel in an unpadded volume
      const long long at = ((long long)b * (a.H + 2) + y0 + 1) * rowq + x + 1;
      const long long o0 = ((long long)b * a.H + y0) * a.W + x;
      // what the epilogue reads of other arrays is loaded before the wait
      uint4 m[EPI == kEpiMask ? 4 * kRows : 1];
      float xc[EPI == kEpiGate ? kRows : 1];
      if constexpr (EPI == kEpiMask) {
#pragma unroll
        for (int j = 0; j < kRows; ++j)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            m[4 * j + c] = in && j < rows ? __ldg(reinterpret_cast<const uint4*>(a.mask_act) + at + j * rowq +
                                                  (long long)c * a.wp)
                                          : make_uint4(0u, 0u, 0u, 0u);
      }
      if constexpr (EPI == kEpiGate) {
#pragma unroll
        for (int j = 0; j < kRows; ++j) xc[j] = in && j < rows ? __ldg(a.xc + o0 + (long long)j * a.W) : 0.f;
      }
      // warp-uniform decision: the TMEM accesses below are .sync.aligned
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(accf0 + 8 * buf, (uint32_t)((k >> 1) & 1)))) {
        if (lane == 0) atomicExch(&s_abort, 1);
        break;
      }
      if (__any_sync(0xFFFFFFFFu, conv_aborted(&s_abort))) break;
      tc_fence_after();
      const uint32_t ta = tmem + (uint32_t)buf * kBuf + (uint32_t)(j0 * kCo) + tl;
#pragma unroll
      for (int j = 0; j < kRows; ++j) {
        const bool mine = in && j < rows;
        if constexpr (!kLast) {
          uint32_t r[32];
          tmem_ld32(ta + j * 32, r);
          tmem_zero16(ta + j * 32);  // the next tile accumulates from zero
          tmem_zero16(ta + j * 32 + 16);
          uint4* dst = reinterpret_cast<uint4*>(a.out_act) + at + j * rowq;
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float u = __uint_as_float(r[8 * c + e]);
              if constexpr (EPI == kEpiRelu) {
                v[e] = fmaxf(u + bias[8 * c + e], 0.f);
              } else {
                const uint4 q = m[4 * j + c];
                const uint32_t w = e < 2 ? q.x : (e < 4 ? q.y : (e < 6 ? q.z : q.w));
                v[e] = (int16_t)(e & 1 ? w >> 16 : w & 0xFFFFu) > 0 ? u : 0.f;
              }
            }
            if (mine)
              dst[(long long)c * a.wp] = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                                                    pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
          }
        } else {
          uint32_t r[16];
          tmem_ld16(ta + j * 16, r);
          tmem_zero16(ta + j * 16);
          const long long o = o0 + (long long)j * a.W;
          const float rr = __uint_as_float(r[0]) + bias[0];
          if constexpr (EPI == kEpiResid) {
            if (mine) a.out_f[o] = rr;
          } else {
            bool rej = false;
            if (mine) {
              const float plain = a.calib * xc[j];
              const float dlt = rr * a.inv_scale;
              const bool keep = fabsf(dlt) <= a.bound;  // NaN fails the test: plain is kept
              a.out_f[o] = keep ? plain + dlt : plain;
              rej = !keep;
            }
            const unsigned msk = __ballot_sync(0xFFFFFFFFu, rej);
            if (lane == 0 && msk && a.n_reject)
              atomicAdd(a.n_reject, (unsigned long long)__popc(msk));
          }
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acce0 + 8 * buf);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && conv_aborted(&s_abort) && a.status) atomicExch(a.status, kDevWaitTimeout);
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmem) : "memory");
}

// Network input: channel k of slice b = k_in * plane(b, k), k < 5 (channels 5..7 zero; the pads stay
// zero).  plane(b, k) = b*5 + k for stacked training inputs [B][5][H][W], or the volume slice
// clamp(z0 + b + k - 2, 0, nz - 1) for inference over a volume [nz][H][W].
__global__ void __launch_bounds__(256) cnn_prep_kernel(const float* __restrict__ src, int vol_mode, int z0,
                                                       int nz, int B, int H, int W, int wp, float k_in,
                                                       __nv_bfloat16* __restrict__ a0) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long long)B * H * W) return;
  const int x = (int)(i % W);
  const long long q = i / W;
  const int y = (int)(q % H), b = (int)(q / H);
  float v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    long long plane;
    if (vol_mode) {
      int z = z0 + b + k - 2;
      z = z < 0 ? 0 : (z > nz - 1 ? nz - 1 : z);
      plane = z;
    } else {
      plane = (long long)b * 5 + k;
    }
    v[k] = __fmul_rn(k_in, __ldg(src + (plane * H + y) * W + x));
  }
  uint4* dst = reinterpret_cast<uint4*>(a0 + (((long long)b * (H + 2) + y + 1) * wp + x + 1) * 8);
  *dst = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], 0.f), 0u);
}

// MSE loss of (k_in x_c + r) against s t and its gradient 2 d / n -> channel 0 of the last
// layer's delta (bf16, padded layout); sum of d^2 accumulated in FP64.
__global__ void __launch_bounds__(256) cnn_loss_kernel(const float* __restrict__ in5,
                                                       const float* __restrict__ r,
                                                       const float* __restrict__ tgt, int B,
                                                       int H, int W, int wp, float k_in, float s,
                                                       float two_over_n, __nv_bfloat16* dz,
                                                       double* loss) {
  __shared__ float red[8];
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long hw = (long long)H * W;
  float d2 = 0.f;
  if (p < B * hw) {
    const long long b = p / hw, pix = p % hw;
    const int y = (int)(pix / W), x = (int)(pix % W);
    const float xc = in5[(b * 5 + 2) * hw + pix];
    const float yv = __fadd_rn(__fmul_rn(k_in, xc), r[p]);
    const float d = __fsub_rn(yv, __fmul_rn(s, tgt[p]));
    d2 = d * d;
    // plane 0, channel 0; the other channels of this delta stay zero
    *reinterpret_cast<uint4*>(dz + ((b * (H + 2) + y + 1) * 4 * wp + x + 1) * 8) =
        make_uint4(pack_bf16x2(__fmul_rn(d, two_over_n), 0.f), 0u, 0u, 0u);
  }
  for (int o = 16; o; o >>= 1) d2 += __shfl_xor_sync(0xFFFFFFFFu, d2, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = d2;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) sum += red[w];
    atomicAdd(loss, sum);
  }
}

// Weight and bias gradients of one layer, no transposes: with K = pixels, both operands are MN-major
// core matrices of the layout (8 pixels x 8 channels, 128 contiguous bytes).  For a group of three delta
// rows j and the five activation rows o around them,
//   D_dx[32 j + co][32 o + ci] += sum_p dz[row j, p][co] * act[row o, p + dx - 1][ci]
// is one M128 x N160 x K16 MMA per dx and 16 pixels: M the planes of consecutive delta rows (the fourth
// row is discarded), N those of the activation rows, shifted by the start of the operand.  The blocks
// with o - j = dy in 0..2 are the gradient's; nine of fifteen useful, but loading an M128 operand costs
// about 64 clocks and a column 0.4, so few wide MMAs beat nine exact ones.  The network input has one
// plane: 32 o becomes 8 o and N 48.
// A tile is 6 rows x up to 64 pixels: one box of eight activation rows and one of six delta rows
// (whatever lies outside the image reads as zero).  A CTA accumulates over all its tiles in three TMEM
// accumulators, sums the blocks over j in shared memory and adds them to the gradient once.  Four
// further warps sum the staged deltas per channel: the bias gradient.
// Bound: the MMAs' operand loads (about 137 clocks each, 1.7 us per tile and SM, 32 of 40 us).  16 x 256^2:
// 39-41 us per layer; with one tap's activations as M128 and N32, and a separate pass for the biases,
// 57-87 + 24 us.
constexpr int kDwThreads = 192, kDwSums = kDwThreads / 32 - 2, kDwGroups = 2, kDwRows = 3 * kDwGroups, kDwMaxP = 64, kDwMaxStages = 4;
constexpr int kDwPitch = 33, kDwPart = 9 * kCnnC * kDwPitch;  // a warp's gradient blocks: [ci][tap][co], padded rows

template <int PLANES>  // planes of the activation: 1 (network input) or 4
__global__ void __launch_bounds__(kDwThreads, 1)
    cnn_dw_tc_kernel(const __grid_constant__ CUtensorMap mact, const __grid_constant__ CUtensorMap mdz,
                     const ConvArgs a, int cin, int cout, float* __restrict__ gw, float* __restrict__ gb) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(8) uint64_t bars[2 * kDwMaxStages + 1];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;
  __shared__ float s_bias[kDwSums][32];
  const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int P = a.n_px, S = a.stages;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[kDwMaxStages]);
  const uint32_t mdone = smem_u32(&bars[2 * kDwMaxStages]);
  const uint32_t stage0 = smem_u32(smem);
  const uint32_t cs = dw_plane(P), rs = PLANES * cs;  // activation plane, row
  const uint32_t zs = (uint32_t)P * 16, zoff = ((kDwRows + 2) * rs + 127) / 128 * 128;  // delta plane, offset
  constexpr int kCi = PLANES * 8, kN = PLANES == 1 ? 48 : 160;  // columns of an activation row, of D_dx
  constexpr uint32_t kCols = PLANES == 1 ? 256 : 512;
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                              ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int s = 0; s < S; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1 + kDwSums);  // the MMAs and the summing warps
    }
    mbar_init(mdone, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(&tmem_slot)),
                 "r"(kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __shfl_sync(0xFFFFFFFFu, tmem_slot, 0);

  if (warp == 0) {
    if (lane == 0) {
      long long k = 0;
      for (long long t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++k) {
        const int s = (int)(k % S);
        if (k >= S && !mbar_wait(empty0 + 8 * s, (uint32_t)(((k / S) - 1) & 1))) {
          atomicExch(&s_abort, 1);
          break;
        }
        if (conv_aborted(&s_abort)) break;
        int x0, y0, b;
        conv_tile(a, t, x0, y0, b);
        const uint32_t fb = full0 + 8 * s, st = stage0 + s * a.stage_bytes;
        mbar_expect_tx(fb, (kDwRows + 2) * rs + kDwRows * 4 * zs);
        tma_load_4d(st, &mact, 2 * x0, 0, y0, b, fb);
        tma_load_4d(st + zoff, &mdz, 2 * x0, 0, y0, b, fb);
      }
      if (conv_aborted(&s_abort))  // let copies in flight land before the CTA exits
        for (long long q = (k > S ? k - S : 0); q < k; ++q)
          mbar_wait(full0 + 8 * (int)(q % S), (uint32_t)((q / S) & 1));
    }
  } else if (warp == 1) {
    long long k = 0;
    uint32_t more = 0;  // 0 for the first MMA of each accumulator
    for (long long t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++k) {
      const int s = (int)(k % S);
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(full0 + 8 * s, (uint32_t)((k / S) & 1)))) {
        if (lane == 0) atomicExch(&s_abort, 1);
        break;
      }
      tc_fence_after();
      int x0, y0, b;
      conv_tile(a, t, x0, y0, b);
      const int groups = (min(P, a.W - x0) + 15) / 16;
      const uint32_t st = stage0 + s * a.stage_bytes;
      if (elect_one()) {
#pragma unroll
        for (int q = 0; q < kDwGroups; ++q) {
          uint64_t za = desc_plain(st + zoff + 12 * q * zs, 128, zs), ab = desc_plain(st + 3 * q * rs, 128, cs);
          for (int g = 0; g < groups; ++g, za += 16, ab += 16) {
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) umma_bf16(tmem + dx * kN, za, ab + (uint64_t)dx, kIdesc, more);
            more = 1;
          }
        }
        umma_commit(empty0 + 8 * s);
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(mdone);
  } else if (warp >= 2) {
    // bias gradient: lane = (plane, pixel mod 8), every fourth delta row; the eight lanes of a plane read
    // 128 consecutive bytes (lane = (pixel mod 8, plane): planes a multiple of 128 bytes apart, 4-way
    // bank conflicts in the memory that feeds the MMAs; 2-3 us of a 16 x 256^2 layer)
    float sum[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    long long k = 0;
    for (long long t = blockIdx.x; t < a.n_tiles; t += gridDim.x, ++k) {
      const int s = (int)(k % S);
      if (!__all_sync(0xFFFFFFFFu, mbar_wait(full0 + 8 * s, (uint32_t)((k / S) & 1)))) {
        if (lane == 0) atomicExch(&s_abort, 1);
        break;
      }
      int x0, y0, b;
      conv_tile(a, t, x0, y0, b);
      const int px = min(P, a.W - x0), zrows = min(kDwRows, a.H - y0);
      for (int r = warp - 2; r < zrows; r += kDwSums) {
        const uint8_t* p = smem + (size_t)s * a.stage_bytes + zoff + (uint32_t)(4 * r + (lane >> 3)) * zs;
#pragma unroll 4
        for (int i = lane & 7; i < px; i += 8) {
          const uint4 q = *reinterpret_cast<const uint4*>(p + i * 16);
          const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            sum[2 * e] += __uint_as_float(w[e] << 16);
            sum[2 * e + 1] += __uint_as_float(w[e] & 0xFFFF0000u);
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * s);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      sum[e] += __shfl_xor_sync(0xFFFFFFFFu, sum[e], 1);
      sum[e] += __shfl_xor_sync(0xFFFFFFFFu, sum[e], 2);
      sum[e] += __shfl_xor_sync(0xFFFFFFFFu, sum[e], 4);
      if ((lane & 7) == 0) s_bias[warp - 2][lane + e] = sum[e];  // channel 8 (lane / 8) + e
    }
  }
  __syncwarp();
  const bool done = __all_sync(0xFFFFFFFFu, mbar_wait(mdone, 0));
  __syncthreads();
  tc_fence_after();
  if (!done || conv_aborted(&s_abort)) {
    if (threadIdx.x == 0 && a.status) atomicExch(a.status, kDevWaitTimeout);
  } else {
    // warp j < 3 holds delta row j, lane = co: block (o, dx) is tap dy = o - j.  The stages are free now:
    // each of the three warps lays its blocks out there, and every thread sums them over j on its way to
    // the gradient.  [ci][tap] in the gradient's own order and rows of 33, so neither side meets a bank
    // conflict ([tap][ci][co], summed over j by the three warps in turn: 32-way conflicts, 48 -> 44.5 us)
    float* part = reinterpret_cast<float*>(smem);  // [j][ci][tap][co]
    if (warp < 3) {
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        uint32_t r[PLANES == 1 ? 16 : 32];
        const uint32_t at =
            tmem + (uint32_t)((tap % 3) * kN + (warp + tap / 3) * kCi) + ((uint32_t)(warp * 32) << 16);
        if constexpr (PLANES == 1)
          tmem_ld16(at, r);
        else
          tmem_ld32(at, r);
        float* p = part + warp * kDwPart + tap * kDwPitch + lane;
#pragma unroll
        for (int ci = 0; ci < kCi; ++ci) p[ci * 9 * kDwPitch] = __uint_as_float(r[ci]);
      }
    }
    __syncthreads();
    // one warp adds the biases: all CTAs meet on one 128-byte line, and an atomic of each summing warp and
    // channel took its L2 slice about 5 us
    if (threadIdx.x < cout) {
      float b = 0.f;
#pragma unroll
      for (int w = 0; w < kDwSums; ++w) b += s_bias[w][threadIdx.x];
      atomicAdd(&gb[threadIdx.x], b);
    }
    const int per = 9 * cin;
    for (int co = warp; co < cout; co += kDwThreads / 32)
      for (int i = lane; i < per; i += 32) {
        const float* p = part + i * kDwPitch + co;
        atomicAdd(&gw[co * per + i], (p[0] + p[kDwPart]) + p[2 * kDwPart]);
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kCols)
                 : "memory");
}

__global__ void cnn_adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                                float* __restrict__ m, float* __restrict__ v, int n, float lr,
                                float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

// FP32 master weights -> bf16 GEMM operands.  Forward slot l: [co][tap*32 + ci].  Backward
// (data) slot l: [ci][tap*32 + co] holding W[co][ci][8 - tap] (the flipped, transposed kernel).
__global__ void cnn_pack_kernel(const float* __restrict__ p, __nv_bfloat16* __restrict__ wf,
                                __nv_bfloat16* __restrict__ wb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kCnnLayers * kWSlot) return;
  const int l = i / kWSlot, rem = i % kWSlot, row = rem / kCnnK, k = rem % kCnnK;
  const int tap = k / kCnnC, c = k % kCnnC;
  const int cin = cnn_cin(l), cout = cnn_cout(l);
  const float* w = p + cnn_off(l);
  float f = 0.f, bwd = 0.f;
  if (row < cout && c < cin) f = w[(row * cin + c) * 9 + tap];
  if (l > 0 && row < cin && c < cout) bwd = w[(c * cin + row) * 9 + (8 - tap)];
  wf[i] = __float2bfloat16_rn(f);
  wb[i] = __float2bfloat16_rn(bwd);
}

}  // namespace lct

using namespace lct;

struct lct_cnn {
  int device = 0, cap = 0, H = 0, W = 0, wp = 0, sms = 148;
  int n_px = 16, dw_px = 16;       // tile widths of the convolutions and of the weight gradients
  bool train = false;
  int n_act = 0;                   // activations: outputs of layers 0..6 (training), or 2
  long long act_elems = 0;         // of one activation / delta; the network input has a quarter
  float* d_p = nullptr;  // params, grads, Adam m, Adam v: 4 x kCnnParams
  float* d_g = nullptr;
  float* d_m = nullptr;
  float* d_v = nullptr;
  __nv_bfloat16* d_wf = nullptr;  // 8 forward slots
  __nv_bfloat16* d_wb = nullptr;  // 8 backward slots (slot 0 unused)
  // boxes of the convolutions' inputs and of the weight gradients; activations: [0] the network input,
  // [1 + i] buffer i
  CUtensorMap m_in[kConvHeights][kCnnLayers], m_dwa[kCnnLayers];
  CUtensorMap m_zin[kConvHeights][3], m_dwz[3];  // the same for the deltas
  __nv_bfloat16* d_in = nullptr;  // network input
  __nv_bfloat16* d_act = nullptr; // n_act activation buffers
  __nv_bfloat16* d_dz = nullptr;  // training: 3 delta buffers
  float* d_r = nullptr;           // training: residual [cap][H][W]
  double* d_loss = nullptr;
  unsigned long long* d_rej = nullptr;
  float calib = 1.f, in_scale = 1.f;
  int adam_t = 0;
  long long last_n = 0;
};

namespace lct {

static __nv_bfloat16* act_buf(lct_cnn* c, int i) { return c->d_act + (size_t)i * c->act_elems; }
static __nv_bfloat16* dz_buf(lct_cnn* c, int i) { return c->d_dz + (size_t)i * c->act_elems; }
// buffer of layer l's output (training keeps every activation; inference ping-pongs two), and map index
// of layer l's input
static int out_buf(const lct_cnn* c, int l) { return c->train ? l : (l & 1); }
static int in_map(const lct_cnn* c, int l) { return l == 0 ? 0 : 1 + out_buf(c, l - 1); }

// Boxes of the convolutions: bf16 [cap][H + 2][planes][wp / 8][8 pixels] as 8-byte elements, box
// {8 pixels, px / 8 + 1 blocks, planes, rows, 1}.
static int conv_map(CUtensorMap* m, __nv_bfloat16* base, const lct_cnn* c, int planes, int rows) {
  auto fn = tensor_map_encoder();
  if (!fn) return LCT_ERR_UNSUPPORTED;
  const size_t plane = (size_t)16 * c->wp, row = plane * planes, slice = row * (c->H + 2);
  cuuint64_t dims[5] = {16, (cuuint64_t)c->wp / 8, (cuuint64_t)planes, (cuuint64_t)(c->H + 2), (cuuint64_t)c->cap};
  cuuint64_t strides[4] = {128, plane, row, slice};
  cuuint32_t box[5] = {16, (cuuint32_t)(c->n_px / 8 + 1), (cuuint32_t)planes, (cuuint32_t)(rows + 2), 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 5, base, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LCT_OK : LCT_ERR_UNSUPPORTED;
}

// Boxes of the gradients: bf16 [cap][H + 2][planes][wp][8] as 8-byte elements, box {px, planes, rows, 1}.  inner: only the
// image's pixels, from row 0 and column 0 of the image (stores outside are dropped); else with the pads.
static int act_map(CUtensorMap* m, __nv_bfloat16* base, const lct_cnn* c, int planes, int px, int rows,
                   bool inner) {
  auto fn = tensor_map_encoder();
  if (!fn) return LCT_ERR_UNSUPPORTED;
  const size_t col = 16, plane = col * c->wp, row = plane * planes, slice = row * (c->H + 2);
  cuuint64_t dims[4] = {(cuuint64_t)(inner ? c->W : c->wp) * 2, (cuuint64_t)planes,
                        (cuuint64_t)(inner ? c->H : c->H + 2), (cuuint64_t)c->cap};
  cuuint64_t strides[3] = {plane, row, slice};
  cuuint32_t box[4] = {(cuuint32_t)(px * 2), (cuuint32_t)planes, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  uint8_t* p = reinterpret_cast<uint8_t*>(base) + (inner ? row + col : 0);
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, p, dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? LCT_OK : LCT_ERR_UNSUPPORTED;
}

// Tile width for an image of W pixels: as few tiles of at most `most` pixels as it takes, alike in width,
// a multiple of `step`
static int tile_px(int W, int most, int step) {
  const int tiles = (W + most - 1) / most;
  return ((W + tiles - 1) / tiles + step - 1) / step * step;
}

template <int EPI, int PLANES, int ROWS>
static int launch_conv_rows(const CUtensorMap& in, ConvArgs a, int B, int sms, cudaStream_t s) {
  a.rows = ROWS;
  a.tiles_y = (a.H + ROWS - 1) / ROWS;
  a.n_tiles = (long long)B * a.tiles_x * a.tiles_y;
  if (a.n_tiles <= 0) return LCT_OK;
  a.stage_bytes = ((ROWS + 2) * PLANES * conv_plane(a.n_px) + 127) / 128 * 128;
  const bool last = EPI == kEpiResid || EPI == kEpiGate;
  const uint32_t fixed = (PLANES == 1 ? kConvZero : 0u) + 3u * (PLANES == 1 ? 1u : 2u) * 2u * 3u * (last ? 16u : 32u) * 16u;
  const uint32_t tail = 128 * 16;  // an operand of the last plane may read this far past it
  a.stages = std::min<int>(kConvMaxStages, (int)((kSmemMax - fixed - tail) / a.stage_bytes));
  const size_t smem = (size_t)a.stages * a.stage_bytes + fixed + tail;
  const unsigned grid = (unsigned)std::min<long long>(a.n_tiles, sms);  // tensor memory: one CTA per SM
  conv_tc_kernel<EPI, PLANES, ROWS><<<grid, kConvThreads, smem, s>>>(in, a);
  return launch_status();
}

// Height of the tiles: the fewest rows whose tiles are still one for each SM.  Such a launch is bound by one
// tile's MMAs (60 in series for eight rows, 3.3 us; 36 for four; 24 of fewer columns for two, 1 us), not by
// operand reads or the rows that neighbouring tiles both load; a second tile for some SMs costs more than it
// saves (96^2 x 4 slices, 192 tiles of two rows: 84 us a forward pass, 80 with eight rows; two CTAs per SM no
// better).  Forward pass of 8 layers as a program calls it, us, eight rows / the fewest: 64^2 x 4 slices
// 79 / 65, 128^2 80 / 66 (in a graph 58 / 39, the loads' overlap included), 96^2 x 4 80 / 72.  The same values: a pixel's taps add in the same order.
static int conv_height(const ConvArgs& a, int B, int sms) {
  int h = kConvHeights - 1;
  while (h > 0 && (long long)B * a.tiles_x * ((a.H + conv_rows(h) - 1) / conv_rows(h)) > sms) --h;
  return h;
}

// in(height): the input's boxes for tiles of that height
template <int EPI, int PLANES, class Boxes>
static int launch_conv(Boxes in, const ConvArgs& a, int B, int sms, cudaStream_t s) {
  switch (conv_height(a, B, sms)) {
    case 2: return launch_conv_rows<EPI, PLANES, conv_rows(2)>(in(2), a, B, sms, s);
    case 1: return launch_conv_rows<EPI, PLANES, conv_rows(1)>(in(1), a, B, sms, s);
    default: return launch_conv_rows<EPI, PLANES, conv_rows(0)>(in(0), a, B, sms, s);
  }
}

static ConvArgs conv_args(const lct_cnn* c) {
  ConvArgs a = {};
  a.H = c->H;
  a.W = c->W;
  a.wp = c->wp;
  a.n_px = c->n_px;
  a.tiles_x = (c->W + a.n_px - 1) / a.n_px;
  a.status = device_status_ptr();
  return a;
}

template <int ROWS>
static int conv_attributes() {
  auto attr = [](auto kernel) {
    return cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
  };
  int st;
  if ((st = attr(conv_tc_kernel<kEpiRelu, 1, ROWS>))) return st;
  if ((st = attr(conv_tc_kernel<kEpiRelu, 4, ROWS>))) return st;
  if ((st = attr(conv_tc_kernel<kEpiMask, 4, ROWS>))) return st;
  if ((st = attr(conv_tc_kernel<kEpiResid, 4, ROWS>))) return st;
  if ((st = attr(conv_tc_kernel<kEpiGate, 4, ROWS>))) return st;
  if ((st = attr(cnn_dw_tc_kernel<1>))) return st;
  return attr(cnn_dw_tc_kernel<4>);
}

// attributes (which load a kernel) of the tile heights that passes of 1 .. cap slices take
static int conv_prepare(const lct_cnn* c) {
  static std::mutex mu;  // host threads may create workspaces on one device together
  static unsigned long long done[64][kConvHeights] = {};  // the context they are set in, plus one
  if (c->device < 0 || c->device >= 64) return LCT_ERR_UNSUPPORTED;
  const unsigned long long ctx = context_id() + 1;
  const ConvArgs a = conv_args(c);
  std::lock_guard<std::mutex> lock(mu);
  for (int h = conv_height(a, c->cap, c->sms); h <= conv_height(a, 1, c->sms); ++h) {
    if (done[c->device][h] == ctx) continue;
    const int st = h == 0   ? conv_attributes<conv_rows(0)>()
                   : h == 1 ? conv_attributes<conv_rows(1)>()
                            : conv_attributes<conv_rows(2)>();
    if (st) return st;
    done[c->device][h] = ctx;
  }
  return LCT_OK;
}

static int run_pack(lct_cnn* c, cudaStream_t s) {
  cnn_pack_kernel<<<(kCnnLayers * kWSlot + 255) / 256, 256, 0, s>>>(c->d_p, c->d_wf, c->d_wb);
  return launch_status();
}

static int run_prep(lct_cnn* c, const float* src, int vol_mode, int z0, int nz, int B,
                    cudaStream_t s) {
  const long long n = (long long)B * c->H * c->W;
  const float k_in = c->calib * c->in_scale;
  cnn_prep_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(src, vol_mode, z0, nz, B, c->H,
                                                             c->W, c->wp, k_in, c->d_in);
  return launch_status();
}

// hidden layers 0..6 of the forward pass on B slices already in d_in
static int run_hidden(lct_cnn* c, int B, cudaStream_t s) {
  ConvArgs a = conv_args(c);
  int st;
  for (int l = 0; l < kCnnLayers - 1; ++l) {
    a.bias = c->d_p + cnn_off(l) + cnn_cin(l) * cnn_cout(l) * 9;
    a.w = c->d_wf + (size_t)l * kWSlot;
    a.out_act = act_buf(c, out_buf(c, l));
    auto in = [&, m = in_map(c, l)](int h) -> const CUtensorMap& { return c->m_in[h][m]; };
    st = l == 0 ? launch_conv<kEpiRelu, 1>(in, a, B, c->sms, s) : launch_conv<kEpiRelu, 4>(in, a, B, c->sms, s);
    if (st) return st;
  }
  return LCT_OK;
}

static int last_bias_and_args(lct_cnn* c, ConvArgs& a) {
  a = conv_args(c);
  const int l = kCnnLayers - 1;
  a.bias = c->d_p + cnn_off(l) + cnn_cin(l) * cnn_cout(l) * 9;
  a.w = c->d_wf + (size_t)l * kWSlot;
  return LCT_OK;
}

static int cnn_forward_impl(lct_cnn* c, const float* d_in5, int B, cudaStream_t s) {
  int st;
  if ((st = run_prep(c, d_in5, 0, 0, 0, B, s))) return st;
  if ((st = run_hidden(c, B, s))) return st;
  ConvArgs a;
  last_bias_and_args(c, a);
  a.out_f = c->d_r;
  auto in = [&, m = in_map(c, kCnnLayers - 1)](int h) -> const CUtensorMap& { return c->m_in[h][m]; };
  return launch_conv<kEpiResid, 4>(in, a, B, c->sms, s);
}

static int cnn_backward_impl(lct_cnn* c, const float* d_in5, const float* d_target, int B,
                             cudaStream_t s) {
  int st;
  const long long n = (long long)B * c->H * c->W;
  if ((st = cuda_status(cudaMemsetAsync(c->d_g, 0, sizeof(float) * kCnnParams, s)))) return st;
  if ((st = cuda_status(cudaMemsetAsync(c->d_loss, 0, sizeof(double), s)))) return st;
  cnn_loss_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(
      d_in5, c->d_r, d_target, B, c->H, c->W, c->wp, c->calib * c->in_scale, c->in_scale,
      (float)(2.0 / (double)n), dz_buf(c, 2), c->d_loss);
  if ((st = launch_status())) return st;
  c->last_n = n;
  ConvArgs a = conv_args(c);
  ConvArgs da = conv_args(c);
  da.n_px = c->dw_px;
  da.rows = kDwRows;
  da.tiles_x = (c->W + da.n_px - 1) / da.n_px;
  da.tiles_y = (c->H + kDwRows - 1) / kDwRows;
  da.n_tiles = (long long)B * da.tiles_x * da.tiles_y;
  const unsigned dw_grid = (unsigned)std::min<long long>(da.n_tiles, c->sms);
  int cur = 2;
  for (int l = kCnnLayers - 1; l >= 0; --l) {
    float* gw = c->d_g + cnn_off(l);
    float* gb = gw + cnn_cin(l) * cnn_cout(l) * 9;
    const int planes = l == 0 ? 1 : 4;
    da.stage_bytes = ((kDwRows + 2) * planes * dw_plane(da.n_px) + 127) / 128 * 128 +
                     kDwRows * 4 * (uint32_t)da.n_px * 16;
    // the last group's discarded delta row, and the network input's sixth activation row, read past it
    const uint32_t tail = 4 * (uint32_t)da.n_px * 16 + 2 * dw_plane(da.n_px);
    da.stages = std::min<int>(kDwMaxStages, (int)((kSmemMax - tail) / da.stage_bytes));
    const size_t dw_smem = std::max((size_t)da.stages * da.stage_bytes + tail, sizeof(float) * 3 * kDwPart);
    auto dw = l == 0 ? cnn_dw_tc_kernel<1> : cnn_dw_tc_kernel<4>;
    dw<<<dw_grid, kDwThreads, dw_smem, s>>>(c->m_dwa[in_map(c, l)], c->m_dwz[cur], da, cnn_cin(l), cnn_cout(l),
                                            gw, gb);
    if ((st = launch_status())) return st;
    if (l == 0) break;
    const int nxt = cur == 2 ? 0 : (cur ^ 1);
    a.w = c->d_wb + (size_t)l * kWSlot;
    a.out_act = dz_buf(c, nxt);
    a.mask_act = act_buf(c, out_buf(c, l - 1));
    auto in = [&](int h) -> const CUtensorMap& { return c->m_zin[h][cur]; };
    if ((st = launch_conv<kEpiMask, 4>(in, a, B, c->sms, s))) return st;
    cur = nxt;
  }
  return LCT_OK;
}

static int cnn_adam_impl(lct_cnn* c, float lr, float b1, float b2, float eps, cudaStream_t s) {
  ++c->adam_t;
  const float c1 = (float)(1.0 / (1.0 - std::pow((double)b1, c->adam_t)));
  const float c2 = (float)(1.0 / (1.0 - std::pow((double)b2, c->adam_t)));
  cnn_adam_kernel<<<(kCnnParams + 255) / 256, 256, 0, s>>>(c->d_p, c->d_g, c->d_m, c->d_v,
                                                          kCnnParams, lr, b1, b2, eps, c1, c2);
  int st = launch_status();
  return st ? st : run_pack(c, s);
}

// He-normal weights (std sqrt(2 / (9 cin)), the last layer x0.1 so training starts near the
// identity), zero biases; splitmix64 + Box-Muller, so a seed gives the same network everywhere.
static void init_params(std::vector<float>& p, uint64_t seed) {
  uint64_t st = seed ^ 0x6c6374636e6eULL;
  auto next = [&st]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
  };
  auto unif = [&]() { return ((double)(next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); };
  p.assign(kCnnParams, 0.f);
  for (int l = 0; l < kCnnLayers; ++l) {
    const int nw = cnn_cin(l) * cnn_cout(l) * 9;
    const double sd = std::sqrt(2.0 / (9.0 * cnn_cin(l))) * (l == kCnnLayers - 1 ? 0.1 : 1.0);
    for (int i = 0; i < nw; ++i) {
      const double u1 = unif(), u2 = unif();
      p[cnn_off(l) + i] = (float)(sd * std::sqrt(-2.0 * std::log(u1)) *
                                  std::cos(2.0 * 3.141592653589793 * u2));
    }
  }
}

static void free_cnn(lct_cnn* c) {
  if (!c) return;
  cudaFree(c->d_p);
  cudaFree(c->d_wf);
  cudaFree(c->d_in);
  cudaFree(c->d_act);
  cudaFree(c->d_dz);
  cudaFree(c->d_r);
  cudaFree(c->d_loss);
  cudaFree(c->d_rej);
  delete c;
}

}  // namespace lct

LCT_API int lct_cnn_param_count(int64_t* n) {
  if (!n) return LCT_ERR_ARG;
  *n = kCnnParams;
  return LCT_OK;
}

LCT_API int lct_cnn_create(int max_slices, int ny, int nx, int flags, uint64_t seed,
                           lct_cnn** out) {
  if (!out || max_slices <= 0 || ny <= 0 || nx <= 0) return LCT_ERR_ARG;
  *out = nullptr;
  if ((flags & ~LCT_CNN_TRAIN) != 0) return LCT_ERR_ARG;
  const long long wp = ((long long)nx + 2 + 7) / 8 * 8;
  if (wp > (1LL << 30) || ny > (1 << 30)) return LCT_ERR_ARG;
  lct_cnn* c = new (std::nothrow) lct_cnn;
  if (!c) return LCT_ERR_ALLOC;
  c->cap = max_slices;
  c->H = ny;
  c->W = nx;
  c->wp = (int)wp;
  c->train = (flags & LCT_CNN_TRAIN) != 0;
  c->n_px = tile_px(nx, kConvMaxN, 8);
  c->dw_px = tile_px(nx, kDwMaxP, 16);
  c->n_act = c->train ? kCnnLayers - 1 : 2;
  c->act_elems = (long long)max_slices * (ny + 2) * wp * kCnnC;
  int st = cuda_status(cudaGetDevice(&c->device));
  if (!st) st = cuda_status(cudaDeviceGetAttribute(&c->sms, cudaDevAttrMultiProcessorCount, c->device));
  if (!st) st = conv_prepare(c);
  if (!st) st = cuda_status(cudaMalloc(&c->d_p, sizeof(float) * 4 * kCnnParams));
  if (!st) {
    c->d_g = c->d_p + kCnnParams;
    c->d_m = c->d_g + kCnnParams;
    c->d_v = c->d_m + kCnnParams;
    st = cuda_status(cudaMemset(c->d_p, 0, sizeof(float) * 4 * kCnnParams));
  }
  if (!st) st = cuda_status(cudaMalloc(&c->d_wf, sizeof(__nv_bfloat16) * 2 * kCnnLayers * kWSlot));
  if (!st) c->d_wb = c->d_wf + kCnnLayers * kWSlot;
  const size_t act_bytes = sizeof(__nv_bfloat16) * (size_t)c->act_elems;
  if (!st) st = cuda_status(cudaMalloc(&c->d_in, act_bytes / 4));
  if (!st) st = cuda_status(cudaMemset(c->d_in, 0, act_bytes / 4));
  if (!st) st = cuda_status(cudaMalloc(&c->d_act, act_bytes * c->n_act));
  if (!st) st = cuda_status(cudaMemset(c->d_act, 0, act_bytes * c->n_act));
  if (!st && c->train) {
    st = cuda_status(cudaMalloc(&c->d_dz, act_bytes * 3));
    if (!st) st = cuda_status(cudaMemset(c->d_dz, 0, act_bytes * 3));
    if (!st) st = cuda_status(cudaMalloc(&c->d_r, sizeof(float) * (size_t)max_slices * ny * nx));
  }
  if (!st) st = cuda_status(cudaMalloc(&c->d_loss, sizeof(double)));
  if (!st) st = cuda_status(cudaMalloc(&c->d_rej, sizeof(unsigned long long)));
  for (int i = 0; i <= c->n_act && !st; ++i) {  // i = 0: the network input
    __nv_bfloat16* p = i == 0 ? c->d_in : act_buf(c, i - 1);
    const int planes = i == 0 ? 1 : 4;
    for (int h = 0; h < kConvHeights && !st; ++h) st = conv_map(&c->m_in[h][i], p, c, planes, conv_rows(h));
    if (!st && c->train) st = act_map(&c->m_dwa[i], p, c, planes, c->dw_px + 2, kDwRows + 2, false);
  }
  for (int i = 0; i < 3 && !st && c->train; ++i) {
    for (int h = 0; h < kConvHeights && !st; ++h) st = conv_map(&c->m_zin[h][i], dz_buf(c, i), c, 4, conv_rows(h));
    if (!st) st = act_map(&c->m_dwz[i], dz_buf(c, i), c, 4, c->dw_px, kDwRows, true);
  }
  if (!st) {
    std::vector<float> p;
    init_params(p, seed);
    st = cuda_status(cudaMemcpy(c->d_p, p.data(), sizeof(float) * kCnnParams, cudaMemcpyHostToDevice));
  }
  if (!st) st = run_pack(c, nullptr);
  if (!st) st = cuda_status(cudaDeviceSynchronize());
  if (st) {
    free_cnn(c);
    return st;
  }
  *out = c;
  return LCT_OK;
}

// Parameter, gradient, loss and counter copies wait for every stream first: the caller's training
// or inference may be queued on a non-blocking stream that the default stream does not order.
LCT_API int lct_cnn_set_params(lct_cnn* c, const float* params, int on_device) {
  if (!c || !params) return LCT_ERR_ARG;
  int st = cuda_status(cudaDeviceSynchronize());
  if (st) return st;
  st = cuda_status(cudaMemcpy(c->d_p, params, sizeof(float) * kCnnParams,
                                  on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
  if (!st) st = cuda_status(cudaMemset(c->d_m, 0, sizeof(float) * 2 * kCnnParams));
  c->adam_t = 0;
  if (!st) st = run_pack(c, nullptr);
  if (!st) st = cuda_status(cudaDeviceSynchronize());
  return st;
}

LCT_API int lct_cnn_get_params(const lct_cnn* c, float* params, int on_device) {
  if (!c || !params) return LCT_ERR_ARG;
  const int st = cuda_status(cudaDeviceSynchronize());
  if (st) return st;
  return cuda_status(cudaMemcpy(params, c->d_p, sizeof(float) * kCnnParams,
                                on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost));
}

LCT_API int lct_cnn_get_grads(const lct_cnn* c, float* grads, int on_device) {
  if (!c || !grads || !c->train) return LCT_ERR_ARG;
  const int st = cuda_status(cudaDeviceSynchronize());
  if (st) return st;
  return cuda_status(cudaMemcpy(grads, c->d_g, sizeof(float) * kCnnParams,
                                on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost));
}

LCT_API int lct_cnn_set_scales(lct_cnn* c, float calib, float in_scale) {
  if (!c || !(calib > 0.f) || !(in_scale > 0.f) || !std::isfinite(calib) || !std::isfinite(in_scale))
    return LCT_ERR_ARG;
  c->calib = calib;
  c->in_scale = in_scale;
  return LCT_OK;
}

LCT_API int lct_cnn_get_scales(const lct_cnn* c, float* calib, float* in_scale) {
  if (!c || !calib || !in_scale) return LCT_ERR_ARG;
  *calib = c->calib;
  *in_scale = c->in_scale;
  return LCT_OK;
}

LCT_API int lct_cnn_forward(lct_cnn* c, const float* d_in5, int n_slices, float* d_resid,
                            lct_stream stream) {
  if (!c || !d_in5 || n_slices <= 0 || n_slices > c->cap) return LCT_ERR_ARG;
  if (!c->train) return LCT_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  int st = cnn_forward_impl(c, d_in5, n_slices, s);
  if (!st && d_resid)
    st = cuda_status(cudaMemcpyAsync(d_resid, c->d_r, sizeof(float) * (size_t)n_slices * c->H * c->W,
                                     cudaMemcpyDeviceToDevice, s));
  return st;
}

LCT_API int lct_cnn_backward(lct_cnn* c, const float* d_in5, const float* d_target, int n_slices,
                             lct_stream stream) {
  if (!c || !d_in5 || !d_target || n_slices <= 0 || n_slices > c->cap) return LCT_ERR_ARG;
  if (!c->train) return LCT_ERR_UNSUPPORTED;
  return cnn_backward_impl(c, d_in5, d_target, n_slices, (cudaStream_t)stream);
}

LCT_API int lct_cnn_adam_step(lct_cnn* c, float lr, float beta1, float beta2, float eps,
                              lct_stream stream) {
  if (!c || !c->train || !(lr >= 0.f) || !(beta1 >= 0.f && beta1 < 1.f) ||
      !(beta2 >= 0.f && beta2 < 1.f) || !(eps > 0.f))
    return LCT_ERR_ARG;
  return cnn_adam_impl(c, lr, beta1, beta2, eps, (cudaStream_t)stream);
}

LCT_API int lct_cnn_train_step(lct_cnn* c, const float* d_in5, const float* d_target,
                               int n_slices, float lr, lct_stream stream) {
  if (!c || !d_in5 || !d_target || n_slices <= 0 || n_slices > c->cap || !(lr >= 0.f))
    return LCT_ERR_ARG;
  if (!c->train) return LCT_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  int st = cnn_forward_impl(c, d_in5, n_slices, s);
  if (!st) st = cnn_backward_impl(c, d_in5, d_target, n_slices, s);
  if (!st) st = cnn_adam_impl(c, lr, 0.9f, 0.999f, 1e-8f, s);
  return st;
}

LCT_API int lct_cnn_last_loss(const lct_cnn* c, double* loss) {
  if (!c || !loss || !c->train) return LCT_ERR_ARG;
  if (c->last_n <= 0) return LCT_ERR_ARG;  // no backward pass yet
  double sum = 0.0;
  int st = cuda_status(cudaDeviceSynchronize());
  if (!st) st = cuda_status(cudaMemcpy(&sum, c->d_loss, sizeof(double), cudaMemcpyDeviceToHost));
  if (!st) *loss = sum / (double)c->last_n;
  return st;
}

namespace lct {

// Gated inference of the slices [z0, z1) of a volume of nz slices (passes of at most max_slices;
// the 5-slice inputs read the neighbours, edge slices replicated).  Rejections add to the
// counter that cnn_reset_rejects clears.
int cnn_infer_range(lct_cnn* c, const float* d_vol, float* d_out, int nz, int z0, int z1,
                    float bound, cudaStream_t s) {
  if (!c || !d_vol || !d_out || nz <= 0 || d_vol == d_out || !(bound >= 0.f)) return LCT_ERR_ARG;
  if (z0 < 0 || z1 > nz || z0 > z1) return LCT_ERR_ARG;
  const long long plane = (long long)c->H * c->W;
  int st = LCT_OK;
  for (int zb = z0; zb < z1 && !st; zb += c->cap) {
    const int B = z1 - zb < c->cap ? z1 - zb : c->cap;
    if ((st = run_prep(c, d_vol, 1, zb, nz, B, s))) break;
    if ((st = run_hidden(c, B, s))) break;
    ConvArgs a;
    last_bias_and_args(c, a);
    a.out_f = d_out + (size_t)zb * plane;
    a.xc = d_vol + (size_t)zb * plane;
    a.calib = c->calib;
    a.inv_scale = 1.f / c->in_scale;
    a.bound = bound;
    a.n_reject = c->d_rej;
    auto in = [&, m = in_map(c, kCnnLayers - 1)](int h) -> const CUtensorMap& { return c->m_in[h][m]; };
    st = launch_conv<kEpiGate, 4>(in, a, B, c->sms, s);
  }
  return st;
}

int cnn_reset_rejects(lct_cnn* c, cudaStream_t s) {
  return cuda_status(cudaMemsetAsync(c->d_rej, 0, sizeof(unsigned long long), s));
}

int cnn_passes(const lct_cnn* c, int nslices) { return (nslices + c->cap - 1) / c->cap; }

}  // namespace lct

LCT_API int lct_cnn_infer_volume(lct_cnn* c, const float* d_vol, float* d_out, int nz,
                                 float bound, int64_t* n_rejected, lct_stream stream) {
  if (!c || !d_vol || !d_out || nz <= 0 || d_vol == d_out || !(bound >= 0.f)) return LCT_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  int st = cnn_reset_rejects(c, s);
  if (!st) st = cnn_infer_range(c, d_vol, d_out, nz, 0, nz, bound, s);
  if (!st && n_rejected) {
    unsigned long long v = 0;
    st = cuda_status(cudaMemcpyAsync(&v, c->d_rej, sizeof(v), cudaMemcpyDeviceToHost, s));
    if (!st) st = cuda_status(cudaStreamSynchronize(s));
    if (!st) *n_rejected = (int64_t)v;
  }
  return st;
}

LCT_API int lct_cnn_get_shape(const lct_cnn* c, int* max_slices, int* ny, int* nx) {
  if (!c || !max_slices || !ny || !nx) return LCT_ERR_ARG;
  *max_slices = c->cap;
  *ny = c->H;
  *nx = c->W;
  return LCT_OK;
}

LCT_API int lct_cnn_last_rejected(const lct_cnn* c, int64_t* n) {
  if (!c || !n) return LCT_ERR_ARG;
  unsigned long long v = 0;
  int st = cuda_status(cudaDeviceSynchronize());
  if (!st) st = cuda_status(cudaMemcpy(&v, c->d_rej, sizeof(v), cudaMemcpyDeviceToHost));
  if (!st) *n = (int64_t)v;
  return st;
}

LCT_API void lct_cnn_destroy(lct_cnn* c) { free_cnn(c); }
