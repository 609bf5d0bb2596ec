// Status codes, CUDA error bookkeeping, the device status word and geometry checks.
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>

#include "lct_internal.h"

namespace lct {

static thread_local int t_last_cuda_error = 0;

void set_cuda_error(cudaError_t e) { t_last_cuda_error = (int)e; }

int cuda_status(cudaError_t e) {
  if (e == cudaSuccess) return LCT_OK;
  set_cuda_error(e);
  return LCT_ERR_CUDA;
}

int launch_status() { return cuda_status(cudaGetLastError()); }

int device_sms() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) == cudaSuccess &&
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
    return sms;
  cudaGetLastError();
  return 148;
}

// cudaDeviceReset destroys a device's context with all that lives in it -- pools, module addresses,
// kernel attributes -- and the next call starts another, so what the library keeps per device is kept
// for the context's id.
unsigned long long context_id() {
  static std::once_flag once;
  static PFN_cuCtxGetId_v12000 get = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get = reinterpret_cast<PFN_cuCtxGetId_v12000>(p);
  });
  unsigned long long id = 0;
  if (!get || get(nullptr, &id) == CUDA_SUCCESS) return id;
  cudaFree(nullptr);  // no context yet: starts the device's
  return get(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}

// One word per device, kept in the module's own global memory (no allocation).
static __device__ int g_device_status = 0;

int* device_status_ptr() {
  static std::mutex mu;
  static int* ptrs[64] = {nullptr};
  static unsigned long long ctx[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  const unsigned long long id = context_id();
  std::lock_guard<std::mutex> lock(mu);
  if (!ptrs[dev] || ctx[dev] != id) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_device_status) != cudaSuccess) return nullptr;
    ptrs[dev] = static_cast<int*>(p);
    ctx[dev] = id;
  }
  return ptrs[dev];
}

// Scratch of the stage entry points.  The default pool unmaps what is freed at every
// synchronisation, so a call that takes a gigabyte of scratch after each one paid for mapping it
// again (a 3,600-view block of 735 x 31: 15-160 ms a call for a 5 ms kernel).  One pool per device and
// context keeps up to kScratchKeep bytes (1/32 of the device's memory if that is less) mapped between calls.
// The pool is stream-ordered and thread-safe like the default one; what exceeds the bound goes back
// at the next synchronisation, the rest when the driver needs it for another allocation of the
// process or lct_scratch_release asks.
constexpr size_t kScratchKeep = 4ull << 30;
static std::mutex g_scratch_mu;
// by device and context; never destroyed, as calls may outlive static objects
static auto& g_scratch_pool = *new std::map<std::pair<int, unsigned long long>, cudaMemPool_t>;

static cudaMemPool_t scratch_pool() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  const std::pair<int, unsigned long long> ctx{dev, context_id()};
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const auto it = g_scratch_pool.find(ctx);
  if (it != g_scratch_pool.end()) return it->second;
  cudaMemPoolProps p = {};
  p.allocType = cudaMemAllocationTypePinned;
  p.handleTypes = cudaMemHandleTypeNone;
  p.location.type = cudaMemLocationTypeDevice;
  p.location.id = dev;
  cudaMemPool_t pool = nullptr;
  size_t free_b = 0, total = 0;
  uint64_t keep = kScratchKeep;
  if (cudaMemGetInfo(&free_b, &total) == cudaSuccess) keep = std::min<uint64_t>(keep, total / 32);
  if (cudaMemPoolCreate(&pool, &p) != cudaSuccess) {
    cudaGetLastError();  // no pools on this device: the default one
    return nullptr;
  }
  if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess)
    cudaGetLastError();
  return g_scratch_pool[ctx] = pool;
}

int scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  *p = nullptr;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaMemPool_t pool = nullptr;
  // a captured call's scratch belongs to its graph
  if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
    pool = scratch_pool();
  return cuda_status(pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s));
}

int scratch_free(void* p, cudaStream_t s) { return cuda_status(cudaFreeAsync(p, s)); }

int check_geom(const lct_geom* g) {
  if (!g) return LCT_ERR_ARG;
  if (g->ns <= 0 || g->nt <= 0 || g->n_angle <= 0 || g->n_angle_add < g->n_angle) return LCT_ERR_ARG;
  if (!(g->ds > 0.f) || !(g->dt > 0.f) || !(g->dso > 0.f) || g->n_proj_turn < 2) return LCT_ERR_ARG;
  if (!std::isfinite(g->orbit) || g->orbit == 0.f || !std::isfinite(g->pitch)) return LCT_ERR_ARG;
  if (g->z_dir != 1 && g->z_dir != -1) return LCT_ERR_ARG;
  if ((long long)g->ns * g->nt * (long long)g->n_angle_add > (1LL << 40)) return LCT_ERR_ARG;
  return LCT_OK;
}

int check_img(const lct_img* ig) {
  if (!ig) return LCT_ERR_ARG;
  if (ig->nx <= 0 || ig->ny <= 0 || ig->nz <= 0) return LCT_ERR_ARG;
  if (!(ig->dx > 0.f) || !(ig->dy > 0.f) || !std::isfinite(ig->dz)) return LCT_ERR_ARG;
  return LCT_OK;
}

// CUDA/Backprojector.cu:33-42 with ia_step = 1 (:151).  FP32, same operation order.
BpWindow bp_window(const lct_geom& g, const lct_img& ig, int iz, float dz_per_view,
                   int na1_half) {
  float zc = ((float)iz - ig.wz) * ig.dz;
  int a_middle = (int)roundf((zc - g.source_z0) / dz_per_view);
  a_middle = a_middle < 0 ? 0 : a_middle;
  a_middle = a_middle > g.n_angle - 1 ? g.n_angle - 1 : a_middle;
  BpWindow w;
  w.a_min = (a_middle - na1_half >= 0) ? (a_middle - na1_half) : 0;
  w.a_max = (a_middle + na1_half < g.n_angle) ? (a_middle + na1_half) : g.n_angle - 1;
  w.a_mid = a_middle;
  return w;
}

}  // namespace lct

using namespace lct;

LCT_API const char* lct_status_string(int status) {
  switch (status) {
    case LCT_OK: return "ok";
    case LCT_ERR_ARG: return "invalid argument";
    case LCT_ERR_CUDA: return "CUDA error";
    case LCT_ERR_ALLOC: return "allocation failed";
    case LCT_ERR_RANGE: return "requested reconstruction is outside of allowed data range";
    case LCT_ERR_DEVICE: return "device status word raised";
    case LCT_ERR_UNSUPPORTED: return "unsupported option";
    case LCT_ERR_IO: return "file missing or short";
    case LCT_ERR_SCRATCH: return "problem larger than the fixed scratch of the allocation-free entry point";
    default: return "unknown status";
  }
}

LCT_API int lct_last_cuda_error(void) { return t_last_cuda_error; }

LCT_API int lct_scratch_release(void) {
  int dev = 0;
  int st = cuda_status(cudaGetDevice(&dev));
  if (st) return st;
  const std::pair<int, unsigned long long> ctx{dev, context_id()};
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  const auto it = g_scratch_pool.find(ctx);
  return it == g_scratch_pool.end() ? LCT_OK : cuda_status(cudaMemPoolTrimTo(it->second, 0));
}

LCT_API int lct_version(void) { return 100; }

LCT_API int lct_device_status(int* code_out) {
  int* p = device_status_ptr();
  if (!p) return LCT_ERR_CUDA;
  int v = 0;
  int st = cuda_status(cudaMemcpy(&v, p, sizeof(int), cudaMemcpyDeviceToHost));
  if (st) return st;
  int zero = 0;
  st = cuda_status(cudaMemcpy(p, &zero, sizeof(int), cudaMemcpyHostToDevice));
  if (code_out) *code_out = v;
  if (st) return st;
  return v ? LCT_ERR_DEVICE : LCT_OK;
}
