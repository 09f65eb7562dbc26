// scratch.cu -- the stream-ordered scratch of the entry points.
//
// Short calls (a dot product, a COO multiply, a conversion) need a few
// kilobytes to a few megabytes of device memory while they run.  The device's
// default memory pool gives its free memory back to the system at every
// synchronisation, so a call after a synchronisation maps it anew: 110 us for
// one allocation, 220 us more for a COO multiply (452 against 230 us).  Scratch
// therefore comes from a pool of the library's own, one per context, that
// keeps up to SCRATCH_KEEP bytes between calls; what exceeds it goes back at
// the next synchronisation as before, and mgb_scratch_release() gives back
// the rest.  Allocations stay ordered on their stream, so threads and streams
// share the pool as they shared the default one; under stream capture they
// become nodes of the graph.
#include <cuda.h>  // CUcontext / CUresult types only: the driver calls are resolved at run time

#include <mutex>
#include <new>

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

// What the library keeps per CUDA context: the scratch pool and a page of 64
// mapped host words.  One entry for every context that called, found again when
// a program changes between contexts; entries stay until the process ends (a
// context that went away took its pool and page with it, and IDs are not used
// again).
struct ContextState {
  unsigned long long ctx_id;
  cudaMemPool_t pool;
  char *page, *page_device;
  uint64_t used;  // host words handed out, a bit each
  ContextState* next;
};
std::mutex g_mutex;
ContextState* g_contexts = nullptr;

// The current context's entry, made on first use; null without a context ID.
// g_mutex held.
ContextState* context_state(unsigned long long id) {
  if (id == 0) return nullptr;
  for (ContextState* c = g_contexts; c != nullptr; c = c->next)
    if (c->ctx_id == id) return c;
  ContextState* c = new (std::nothrow) ContextState{};
  if (c == nullptr) return nullptr;
  c->ctx_id = id;
  c->next = g_contexts;
  g_contexts = c;
  return c;
}

// The current context's pool, made on first use; null where there is none to be
// had: the default pool serves then.
cudaMemPool_t scratch_pool(cudaStream_t s, bool make) {
  static thread_local struct {
    unsigned long long ctx_id;
    cudaMemPool_t pool;
  } last = {};
  const unsigned long long id = current_ctx_id();
  if (id != 0 && last.ctx_id == id) return last.pool;
  std::lock_guard<std::mutex> lock(g_mutex);
  ContextState* c = context_state(id);
  if (c == nullptr) return nullptr;
  if (c->pool != nullptr) {
    last = {id, c->pool};
    return c->pool;
  }
  int dev = 0;
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (!make || cudaGetDevice(&dev) != cudaSuccess || cudaStreamIsCapturing(s, &capturing) != cudaSuccess ||
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
  c->pool = pool;
  last = {id, pool};
  return pool;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  const cudaMemPool_t pool = scratch_pool(s, true);
  return pool != nullptr ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

HostWord::HostWord(cudaStream_t s) : s_(s) {
  const unsigned long long id = current_ctx_id();
  std::lock_guard<std::mutex> lock(g_mutex);
  ContextState* c = context_state(id);
  if (c == nullptr) return;
  if (c->page == nullptr) {
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
    c->page = static_cast<char*>(h);
    c->page_device = static_cast<char*>(d);
  }
  if (c->used == ~0ull) return;
  index_ = __builtin_ctzll(~c->used);
  c->used |= 1ull << index_;
  used_ = &c->used;
  host_ = c->page + 64 * index_;
  device_ = c->page_device + 64 * index_;
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
  std::lock_guard<std::mutex> lock(g_mutex);
  *used_ &= ~(1ull << index_);
}

}  // namespace mgb

extern "C" int mgb_scratch_release(void) {
  const cudaMemPool_t pool = mgb::scratch_pool(nullptr, false);
  if (pool == nullptr) return MGB_SUCCESS;
  MGB_CUDA_CHECK(cudaDeviceSynchronize());
  MGB_CUDA_CHECK(cudaMemPoolTrimTo(pool, 0));
  return MGB_SUCCESS;
}
