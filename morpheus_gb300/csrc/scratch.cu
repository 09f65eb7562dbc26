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
  static thread_local PoolSlot last = {};  // a context's ID is never used again
  const unsigned long long id = current_ctx_id();
  if (id != 0 && last.ctx_id == id) return last.pool;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    (void)cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  PoolSlot& slot = g_pool[dev];
  if (slot.pool != nullptr && id != 0 && slot.ctx_id == id) {
    last = slot;
    return slot.pool;
  }
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
  last = slot;
  return pool;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  const cudaMemPool_t pool = scratch_pool(s, true);
  return pool != nullptr ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

// Host words: one page per device, 64 words of 64 bytes.  A context that went
// away took its page with it; words still out of an older page are forgotten.
namespace {
struct HostPage {
  unsigned long long ctx_id;
  char *host, *device;
  uint64_t used;  // a bit per word
};
HostPage g_page[64] = {};
}  // namespace

HostWord::HostWord(cudaStream_t s) : s_(s) {
  if (cudaGetDevice(&dev_) != cudaSuccess || dev_ < 0 || dev_ >= 64) {
    (void)cudaGetLastError();
    return;
  }
  const unsigned long long id = current_ctx_id();
  if (id == 0) return;
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  HostPage& page = g_page[dev_];
  if (page.host == nullptr || page.ctx_id != id) {
    void *h = nullptr, *d = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // another thread's capture is not disturbed
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    cudaError_t e = cudaHostAlloc(&h, 64 * 64, cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer(&d, h, 0);
    (void)cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      if (h != nullptr) (void)cudaFreeHost(h);
      return;
    }
    page = HostPage{id, static_cast<char*>(h), static_cast<char*>(d), 0};
  }
  if (page.used == ~0ull) return;
  index_ = __builtin_ctzll(~page.used);
  page.used |= 1ull << index_;
  host_ = page.host + 64 * index_;
  device_ = page.device + 64 * index_;
}

cudaError_t HostWord::wait() {
  const cudaError_t e = cudaStreamSynchronize(s_);
  waited_ = e == cudaSuccess;
  return e;
}

HostWord::~HostWord() {
  if (host_ == nullptr) return;
  if (!waited_ && wait() != cudaSuccess) {  // a kernel may still write the word: nobody gets it again
    (void)cudaGetLastError();
    return;
  }
  std::lock_guard<std::mutex> lock(g_pool_mutex);
  HostPage& page = g_page[dev_];
  if (static_cast<char*>(host_) == page.host + 64 * index_) page.used &= ~(1ull << index_);
}

}  // namespace mgb

extern "C" int mgb_scratch_release(void) {
  const cudaMemPool_t pool = mgb::scratch_pool(nullptr, false);
  if (pool == nullptr) return MGB_SUCCESS;
  MGB_CUDA_CHECK(cudaDeviceSynchronize());
  MGB_CUDA_CHECK(cudaMemPoolTrimTo(pool, 0));
  return MGB_SUCCESS;
}
