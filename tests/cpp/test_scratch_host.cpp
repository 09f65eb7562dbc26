// Host logic of csrc/scratch.cu against a fake CUDA runtime: no GPU, no driver.
// Linked with that file's object instead of the CUDA runtime.
#include <math.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>

#include <cuda.h>
#include <cuda_runtime.h>

#include "mgb_internal.cuh"

namespace {
unsigned long long g_ctx = 1;  // the "current context"
int g_syncs = 0, g_failed = 0;
cudaError_t g_sync_result = cudaSuccess;
std::set<void*> g_pools;
std::set<void*> g_host;

CUresult fake_ctx_get_current(CUcontext* c) {
  *c = reinterpret_cast<CUcontext>(g_ctx);
  return CUDA_SUCCESS;
}
CUresult fake_ctx_get_id(CUcontext c, unsigned long long* id) {
  *id = reinterpret_cast<unsigned long long>(c);
  return CUDA_SUCCESS;
}

void expect(bool ok, const char* what) {
  if (ok) return;
  g_failed++;
  std::printf("FAILED: %s\n", what);
}
}  // namespace

namespace mgb {
int record_cuda_error(cudaError_t) { return MGB_ERR_CUDA; }
}  // namespace mgb

extern "C" {
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
  *f = !std::strcmp(name, "cuCtxGetId") ? reinterpret_cast<void*>(&fake_ctx_get_id)
                                        : reinterpret_cast<void*>(&fake_ctx_get_current);
  *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  void* m = std::malloc(1);
  g_pools.insert(m);
  *p = static_cast<cudaMemPool_t>(m);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t, cudaMemPool_t pool, cudaStream_t) {
  *p = pool;  // which pool it came from is all that the checks look at
  return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t, cudaStream_t) {
  *p = nullptr;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = std::calloc(1, n);
  g_host.insert(*p);
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
  *d = h;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void*) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  g_syncs++;
  return g_sync_result;
}
}

int main() {
  using mgb::HostWord;
  // a call that waits for its stream gives the word back without another wait
  void* first;
  {
    HostWord w(nullptr);
    expect(w.ok(), "a word");
    first = w.host();
    expect(w.wait() == cudaSuccess, "wait");
  }
  expect(g_syncs == 1, "one synchronisation when the call waited");
  // a call that returns early: the stream is waited for before anybody else gets the word
  {
    HostWord w(nullptr);
    expect(w.host() == first, "the word is used again");
  }
  expect(g_syncs == 2, "a synchronisation on the way out of a call that did not wait");
  // the wait fails: the word is not handed out again
  g_sync_result = cudaErrorLaunchFailure;
  { HostWord w(nullptr); }
  g_sync_result = cudaSuccess;
  {
    HostWord w(nullptr);
    expect(w.ok() && w.host() != first, "a word that may still be written is not handed out");
  }
  // two contexts used in turn keep one pool and one page each
  void* from[2] = {nullptr, nullptr};
  for (int k = 0; k < 20; k++) {
    g_ctx = 1 + k % 2;
    void* p = nullptr;
    expect(mgb::scratch_alloc(&p, 256, nullptr) == cudaSuccess, "scratch");
    expect(p != nullptr && (from[k % 2] == nullptr || from[k % 2] == p), "a context keeps its pool");
    from[k % 2] = p;
    HostWord w(nullptr);
    expect(w.ok() && w.wait() == cudaSuccess, "a word in either context");
  }
  expect(from[0] != from[1] && g_pools.size() == 2 && g_host.size() == 2, "one pool and one page per context");
  g_ctx = 0;  // no context: the default pool serves
  void* p = &g_ctx;
  expect(mgb::scratch_alloc(&p, 256, nullptr) == cudaSuccess && p == nullptr, "no context, no pool");
  expect(!HostWord(nullptr).ok(), "no context, no word");
  std::printf("%d failed\n", g_failed);
  return g_failed != 0;
}
