// scratch.cu -- the stream-ordered scratch of the entry points.
//
// Short calls (a dot product, a COO multiply, a conversion) need a few
// kilobytes to a few megabytes of device memory while they run.  The device's
// default memory pool gives its free memory back to the system at every
// synchronisation, so a call after a synchronisation maps it anew: 110 us for
// one allocation, 220 us more for a COO multiply (452 against 230 us).  Scratch
// therefore comes from a pool of the library's own, one per device, that
// keeps up to SCRATCH_KEEP bytes between calls; what exceeds it goes back at
// the next synchronisation as before, and mgb_scratch_release() gives back
// the rest.  Allocations stay ordered on their stream, so threads and streams
// share the pool as they shared the default one; under stream capture they
// become nodes of the graph.
#include <cuda.h>  // CUcontext / CUresult types only: the driver calls are resolved at run time

#include <mutex>

#include "mgb_internal.cuh"

namespace mgb {
namespace {

constexpr uint64_t SCRATCH_KEEP = 32ull << 20;

// cuCtxGetCurrent / cuCtxGetId through the runtime's driver entry points (no
// link against the driver library).  Context IDs are unique for the life of
// the process, unlike context handles, which a new context may reuse.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

}  // namespace

unsigned long long current_ctx_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_current = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  });
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (get_current == nullptr || get_id == nullptr || get_current(&c) != CUDA_SUCCESS || c == nullptr ||
      get_id(c, &id) != CUDA_SUCCESS)
    return 0;
  return id;
}

namespace {

struct PoolSlot {
  unsigned long long ctx_id;  // unique ID of the context the pool belongs to (0: none)
  cudaMemPool_t pool;
};
std::mutex g_pool_mutex;
PoolSlot g_pool[64] = {};

// The current device's pool, made on first use (and again in a new context);
// null where there is none to be had: the default pool serves then.
cudaMemPool_t scratch_pool(cudaStream_t s, bool make) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return nullptr;
  }
  const unsigned long long id = current_ctx_id();
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  PoolSlot& slot = g_pool[dev];
  if (slot.pool != nullptr && id != 0 && slot.ctx_id == id) return slot.pool;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (!make || id == 0 || cudaStreamIsCapturing(s, &capturing) != cudaSuccess ||
      capturing != cudaStreamCaptureStatusNone) {
    (void)cudaGetLastError();
    return nullptr;
  }
  cudaMemPoolProps props = {};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  uint64_t keep = SCRATCH_KEEP;
  // another thread's capture is not disturbed by the pool's creation
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  (void)cudaThreadExchangeStreamCaptureMode(&mode);
  cudaError_t e = cudaMemPoolCreate(&pool, &props);
  if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
  (void)cudaThreadExchangeStreamCaptureMode(&mode);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    if (pool != nullptr) (void)cudaMemPoolDestroy(pool);
    return nullptr;
  }
  slot.pool = pool;
  slot.ctx_id = id;
  return pool;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  const cudaMemPool_t pool = scratch_pool(s, true);
  return pool != nullptr ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

}  // namespace mgb

extern "C" int mgb_scratch_release(void) {
  const cudaMemPool_t pool = mgb::scratch_pool(nullptr, false);
  if (pool == nullptr) return MGB_SUCCESS;
  MGB_CUDA_CHECK(cudaDeviceSynchronize());
  MGB_CUDA_CHECK(cudaMemPoolTrimTo(pool, 0));
  return MGB_SUCCESS;
}
