// spmv_coo.cu -- COO SpMV for sm_103a (row-sorted keys).
//
// Replaces the reference's CUDA COO path (impl/Coo/Cuda/Morpheus_Multiply_Impl.hpp:50-176:
// flat kernel impl/Coo/Kernels/Morpheus_Multiply_Impl.hpp:121-208, carry pass
// impl/DenseVector/Kernels/Morpheus_Segmented_Reduction_Impl.hpp:40-162 and a
// serial <<<1,1>>> tail).  Like that path the matrix must be sorted by row;
// columns may be in any order and duplicates are allowed.  Semantics are the
// Serial multiply (impl/Coo/Serial/Morpheus_Multiply_Impl.hpp:38-59):
// y = 0 if init, then y[I[n]] += V[n] * x[J[n]].
//
// Design: fixed chunks of 256 or 512 consecutive entries, one warp each, cut
// into 32 contiguous lane ranges (the lane-segment scheme of spmv_csr.cu, so
// every FP64 FMA is issued by all 32 lanes).  Row indices, columns and values
// are copied into padded shared memory a step ahead (cp.async, two buffers); a lane
// detects row ends by comparing consecutive row indices.  Rows that cross
// lanes are combined by one segmented shuffle scan per chunk.  The first and
// last row of a chunk may continue in a neighbouring chunk, so their sums are
// written as carries and a small second kernel adds each row's carries in
// chunk order; interior rows are stored directly: deterministic, no atomics,
// no searches.  With init, rows without entries are zero-filled by the lane
// that sees the gap, so y is written once per row.
#include "csr_chunk.cuh"

namespace mgb {
namespace {

constexpr int COO_WARPS = 4;
constexpr int COO_CTAS = 5;                 // register budget per SM (shared memory allows 2 to 4)
constexpr int64_t COO_CHUNK = 2048;         // entries per warp chunk at most (allocation-free calls)

// Entries per chunk: 512, and 256 where FP64 takes steps of four entries (below
// COO_SHORT).  Larger chunks leave the last wave nearly empty at some sizes;
// smaller ones pay carries.  us:
//   FP64, power-law COO of 5.3 M entries, 10.6 M, 15 M, 24 M:
//     256: 43.1, 77.8, 101.5, 153.5   512: 45.1, 80.2, 107.1, 160.2   1024: 50.9, 88.7   2048: 51.8, 90.0
//   from COO_SHORT on (steps of eight), power-law of 30 M, 27-point stencils of 26 M and 109 M:
//     256: 231, 189, 758   512: 209, 145, 554   1024: 220, 160   2048: 214, 166, 607
//   FP32, power-law of 3 M, 10.6 M, 21 M, 30 M, 27-point stencils of 26 M and 109 M:
//     256: 29.5, 72.5, 131.2, 181.7, 126.8, 489.8   512: 26.6, 70.8, 127.9, 176.2, 106.5, 389.2
//     1024 or 2048: 29.6, 77.4, 139.6, 186.6, 134.7, 472.0   (single staging 28.9, 81.0, 136.0, 199.1, 131.5, 552.5)
constexpr int64_t COO_SHORT = 24 << 20;
template <typename T>
inline int64_t coo_chunk_size(int64_t nnz) {
  return sizeof(T) == 8 && nnz < COO_SHORT ? 256 : 512;
}

template <typename T>
__device__ __forceinline__ T gather_x(const T* __restrict__ x, int32_t c, int64_t ncols) {
  return ((uint64_t)(int64_t)c < (uint64_t)ncols) ? __ldg(x + c) : T(0);
}

// IDX: entry and row index type inside the kernel (int32_t when nnz < 2^31 -
// 4096: measured on GB300, power-law COO 252 -> 221 us, same arithmetic).
// SEG: entries per lane per staging step.
template <typename T, typename IDX, int SEG>
__global__ void __launch_bounds__(COO_WARPS * 32, COO_CTAS)
spmv_coo_segments(int64_t nrows, int64_t ncols, int64_t nnz, int64_t chunk, const int32_t* __restrict__ ri,
                  const int32_t* __restrict__ ci, const T* __restrict__ va, const T* __restrict__ x,
                  T* __restrict__ y, int init, int32_t* __restrict__ carry_row, T* __restrict__ carry_val) {
  constexpr int PAD = SEG + 1;  // padded lane stride in shared memory
  __shared__ T s_val[COO_WARPS][2][32 * PAD];
  __shared__ int32_t s_col[COO_WARPS][2][32 * PAD];
  __shared__ int32_t s_row[COO_WARPS][2][32 * PAD];
  const int lane = threadIdx.x & 31;
  const int w = threadIdx.x >> 5;
  const IDX nchunks = (nnz + chunk - 1) / chunk;
  const IDX KW = chunk / 32;  // entries per lane, a multiple of SEG
  for (IDX k = (IDX)blockIdx.x * COO_WARPS + w; k < nchunks; k += (IDX)gridDim.x * COO_WARPS) {
    const IDX base = k * chunk;
    const IDX cend = min(base + chunk, nnz);
    const IDX la = base + (IDX)lane * KW;
    const IDX lb = min(la + KW, cend);
    const bool active = la < lb;
    const IDX first_row = __ldg(ri + base);
    const IDX last_row = __ldg(ri + cend - 1);
    // row of the entry before this lane's range, and of the entry after it
    const IDX prev = (active && la > 0) ? (IDX)__ldg(ri + la - 1) : -1;
    const IDX next = (active && lb < cend) ? (IDX)__ldg(ri + lb) : -2;

    auto finalize = [&](IDX row, T total) {
      if (row == first_row) {
        carry_row[2 * k] = (int32_t)row;
        carry_val[2 * k] = total;
        if (first_row == last_row) {
          carry_row[2 * k + 1] = (int32_t)row;
          carry_val[2 * k + 1] = T(0);
        }
      } else if (row == last_row) {
        carry_row[2 * k + 1] = (int32_t)row;
        carry_val[2 * k + 1] = total;
      } else if (row >= 0 && row < nrows) {
        y[row] = total;
      }
    };
    auto zero_gap = [&](IDX from, IDX to) {  // rows (from, to), init only
      for (IDX g = max(from + 1, (IDX)0); g < min(to, (IDX)nrows); g++) y[g] = T(0);
    };

    IDX cur = -1;          // row being accumulated
    bool cur_here = false;     // it started inside this lane's range
    IDX hrow = -1;
    T hval = T(0), acc = T(0);

    // step s + 1 is copied (cp.async) while step s's x reads are in flight
    auto stage = [&](IDX st, int b) {
      if (st < KW) {
#pragma unroll
        for (int q = 0; q < SEG; q++) {
          const int f = q * 32 + lane;
          const int L = f / SEG, j = f % SEG;
          const IDX e = base + (IDX)L * KW + st + j;
          const bool in = e < cend;
          csr::copy_or_zero(s_row[w][b] + L * PAD + j, ri + (in ? e : base), in);
          csr::copy_or_zero(s_col[w][b] + L * PAD + j, ci + (in ? e : base), in);
          csr::copy_or_zero(s_val[w][b] + L * PAD + j, va + (in ? e : base), in);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    __syncwarp();  // the chunk before is done with the buffers
    stage(0, 0);
    int buf = 0;
    for (IDX st = 0; st < KW; st += SEG, buf ^= 1) {
      __syncwarp();  // the reads of the buffer filled next are done
      stage(st + SEG, buf ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      __syncwarp();
      const T* sv = s_val[w][buf];
      const int32_t* sc = s_col[w][buf];
      const int32_t* sr = s_row[w][buf];
      T v[SEG], xv[SEG];
      int32_t rw[SEG];
#pragma unroll
      for (int kk = 0; kk < SEG; kk++) {
        const bool valid = la + st + kk < lb;
        rw[kk] = sr[lane * PAD + kk];
        v[kk] = valid ? sv[lane * PAD + kk] : T(0);
        xv[kk] = valid ? gather_x(x, sc[lane * PAD + kk], ncols) : T(0);
      }
#pragma unroll
      for (int kk = 0; kk < SEG; kk++) {
        const IDX e = la + st + kk;
        if (e < lb && rw[kk] != cur) {  // a new row starts at e (or the lane's first row)
          if (cur >= 0) {
            if (cur_here) finalize(cur, acc); else { hrow = cur; hval = acc; }
          }
          const IDX before = (cur >= 0) ? cur : prev;
          if (init && rw[kk] - before > 1) zero_gap(before, rw[kk]);
          cur = rw[kk];
          cur_here = (e > la) || (prev != cur);
          const bool carried = (cur == first_row) || (cur == last_row);
          acc = (init || carried || !cur_here || cur < 0 || cur >= nrows) ? T(0) : y[cur];
        }
        acc = fmadd(v[kk], xv[kk], acc);
      }
    }
    // the lane's last row: continues into the next lane, or ends here
    bool has_tail = false;
    if (active) {
      if (next == cur) {
        has_tail = true;
      } else {
        if (cur_here) finalize(cur, acc); else { hrow = cur; hval = acc; }
      }
    }
    const IDX key = has_tail ? cur : -1 - (IDX)lane;
    T cv = has_tail ? acc : T(0);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T u = __shfl_up_sync(0xffffffffu, cv, d);
      const IDX k2 = __shfl_up_sync(0xffffffffu, key, d);
      if (lane >= d && k2 == key) cv += u;
    }
    const T vprev = __shfl_up_sync(0xffffffffu, cv, 1);
    const IDX kprev = __shfl_up_sync(0xffffffffu, key, 1);
    if (hrow >= 0) finalize(hrow, (lane > 0 && kprev == hrow) ? hval + vprev : hval);
    // rows after the last entry of the matrix (init): whole warp fills
    if (init && k == nchunks - 1)
      for (int64_t g = max((int64_t)last_row + 1, (int64_t)0) + lane; g < nrows; g += 32) y[g] = T(0);
  }
}

// Shared-memory carve-out of the kernel above (power-law matrix, 2e6 rows, FP64 /
// FP32; single staging with 24 warps per SM: 223 / 200 us): 35 %: 280 / 208,
// 45: 226 / 194, 60 and 70: 213 / 186 (12 / 16 warps per SM).
// FP64 of fewer than COO_SHORT entries: four entries per step, so that a
// carve-out of 45 % holds 16 warps and leaves L1 more lines.  Steps of eight at
// 60 % / four at 45 % (single staging before), us, each with its chunks: power-law
// COO of 7.6 M entries 65.6 / 61.1 (76.8), 12 M 94.1 / 85.3 (91.2), 13.7 M 103.1 / 93.8
// (100.7), 15 M 112.8 / 101.5 (122.4), 24 M 171.4 / 153.5 (176.3), 30 M 209.4 / 231.4
// (220.8); 5-point rows, 20 M 132.4 / 120.9 (158.7), 27-point, 26 M 145.1 / 189.4 (164.7);
// HYB with a COO part of 8 M entries 288 / 278 (277 to 279).
template <typename T, typename IDX, int SEG, int PERCENT>
int launch_segments(const mgb_coo* A, int64_t chunk, int64_t nchunks, const T* x, T* y, int init, int32_t* cr, T* cv,
                    cudaStream_t s) {
  static std::atomic<bool> done[64];
  if (int st = csr::set_carveout_once(spmv_coo_segments<T, IDX, SEG>, done, PERCENT)) return st;
  const int64_t blocks = (nchunks + COO_WARPS - 1) / COO_WARPS;
  spmv_coo_segments<T, IDX, SEG><<<(unsigned)blocks, COO_WARPS * 32, 0, s>>>(
      A->nrows, A->ncols, A->nnz, chunk, A->row_indices, A->column_indices, static_cast<const T*>(A->values), x, y,
      init, cr, cv);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}
template <typename T>
int coo_segments(const mgb_coo* A, int64_t chunk, int64_t nchunks, const T* x, T* y, int init, int32_t* cr, T* cv,
                 cudaStream_t s) {
  if constexpr (sizeof(T) == 8) {
    if (A->nnz < COO_SHORT) return launch_segments<T, int32_t, 4, 45>(A, chunk, nchunks, x, y, init, cr, cv, s);
  }
  if (A->nnz < ((int64_t)1 << 31) - 4096)
    return launch_segments<T, int32_t, 8, 60>(A, chunk, nchunks, x, y, init, cr, cv, s);
  return launch_segments<T, int64_t, 8, 60>(A, chunk, nchunks, x, y, init, cr, cv, s);
}

// Adds the carries of each row.  carry_row is non-decreasing.  A thread adds the
// few carries of most rows in chunk order; a row of many (5e6 entries: 39,000) is
// added by the CTA that its first one falls to, in an order that the matrix alone
// fixes.  One thread for all of them: the multiply of 2e7 entries with such a row
// 3,390 us, with a CTA 264.
constexpr int FIXUP_FEW = 32;
template <typename T>
__global__ void __launch_bounds__(256) coo_carry_fixup(int64_t ncarry, int64_t nrows,
                                                       const int32_t* __restrict__ cr, const T* __restrict__ cv,
                                                       T* __restrict__ y, int init) {
  __shared__ int64_t s_head[256 / FIXUP_FEW + 1];  // heads of many are more than FIXUP_FEW apart
  __shared__ T s_part[8];
  __shared__ int s_heads;
  if (threadIdx.x == 0) s_heads = 0;
  __syncthreads();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  const int32_t r = i < ncarry ? cr[i] : -1;
  if (i < ncarry && (i == 0 || cr[i - 1] != r)) {
    if (i + FIXUP_FEW < ncarry && cr[i + FIXUP_FEW] == r) {
      s_head[atomicAdd(&s_heads, 1)] = i;
    } else {
      T s = T(0);
      for (int64_t j = i; j < ncarry && cr[j] == r; j++) s += cv[j];
      if (r >= 0 && r < nrows) y[r] = init ? s : y[r] + s;
    }
  }
  __syncthreads();
  for (int k = 0; k < s_heads; k++) {
    const int64_t head = s_head[k];
    const int32_t row = cr[head];
    int64_t end = ncarry;  // the first carry of another row
    for (int64_t lo = head + FIXUP_FEW + 1; lo < end;) {
      const int64_t mid = (lo + end) >> 1;
      if (cr[mid] == row) lo = mid + 1; else end = mid;
    }
    T s = T(0);
#pragma unroll 8
    for (int64_t j = head + threadIdx.x; j < end; j += 256) s += cv[j];
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0 && row >= 0 && row < nrows) {
      for (int w = 1; w < 8; w++) s += s_part[w];
      y[row] = init ? s : y[row] + s;
    }
    __syncthreads();  // the next row's parts
  }
}

}  // namespace

template <typename T>
int launch_coo(const mgb_coo* A, const T* x, T* y, int init, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(!bad_sizes(A->nrows, A->ncols, A->nnz), MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(A->nrows < ((int64_t)1 << 31), MGB_ERR_INVALID_INPUT);
  if (A->nrows == 0) return MGB_SUCCESS;
  MGB_REQUIRE(y != nullptr, MGB_ERR_BAD_ARGUMENT);
  if (A->nnz == 0) {
    if (init) MGB_CUDA_CHECK(cudaMemsetAsync(y, 0, sizeof(T) * A->nrows, s));
    return MGB_SUCCESS;
  }
  MGB_REQUIRE(A->row_indices && A->column_indices && A->values && x, MGB_ERR_BAD_ARGUMENT);
  const int64_t chunk = coo_chunk_size<T>(A->nnz);
  const int64_t nchunks = (A->nnz + chunk - 1) / chunk;
  const int64_t ncarry = 2 * nchunks;
  void* scratch = nullptr;
  const size_t rows_bytes = ((sizeof(int32_t) * ncarry + 255) / 256) * 256;
  MGB_CUDA_CHECK(scratch_alloc(&scratch, rows_bytes + sizeof(T) * ncarry, s));
  int32_t* cr = static_cast<int32_t*>(scratch);
  T* cv = reinterpret_cast<T*>(static_cast<char*>(scratch) + rows_bytes);
  int st = coo_segments<T>(A, chunk, nchunks, x, y, init, cr, cv, s);
  cudaError_t e = cudaSuccess;
  if (st == MGB_SUCCESS) {
    coo_carry_fixup<T><<<(unsigned)((ncarry + 255) / 256), 256, 0, s>>>(ncarry, A->nrows, cr, cv, y, init);
    e = cudaGetLastError();
  }
  cudaError_t ef = cudaFreeAsync(scratch, s);
  if (st != MGB_SUCCESS) return st;
  if (e != cudaSuccess) return record_cuda_error(e);
  if (ef != cudaSuccess) return record_cuda_error(ef);
  return MGB_SUCCESS;
}

template int launch_coo<double>(const mgb_coo*, const double*, double*, int, cudaStream_t);
template int launch_coo<float>(const mgb_coo*, const float*, float*, int, cudaStream_t);

}  // namespace mgb

extern "C" {

int mgb_spmv_coo_f64(const mgb_coo* A, const double* x, double* y, int init, void* stream) {
  return mgb::launch_coo<double>(A, x, y, init, mgb::as_stream(stream));
}

int mgb_spmv_coo_f32(const mgb_coo* A, const float* x, float* y, int init, void* stream) {
  return mgb::launch_coo<float>(A, x, y, init, mgb::as_stream(stream));
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free COO SpMV.
//
// For callers that cannot allocate device memory while they run: real-time
// loops of a host application that forbids allocation once it is running,
// embedded hosts that reserve all device memory up front, and plugins whose
// host process owns the allocator.  mgb_spmv_coo_f64 takes
// its carry buffer from the library's scratch pool; this variant takes it from a fixed
// file-scope device array instead, so it never calls cudaMalloc, cudaFree or
// any allocating routine.
//
// Limits and rules:
//  * The array is COO_NOALLOC_BYTES (4 MiB) of device memory that every GPU
//    which loads this library holds until the process exits.  It holds two
//    carries (int32 row + double value) per chunk of up to 2048 entries (chunks
//    grow with the matrix until their carries fit), so A->nnz may be at most
//    357,892,096; larger matrices get MGB_ERR_INVALID_INPUT before any
//    work is queued.
//  * The first call on a device looks up the array's device address with
//    cudaGetSymbolAddress (once per device, with that device current) and
//    caches it with the unique ID of the current CUDA context; make that
//    first call before any stream capture.  A later call that finds another
//    context current (after cudaDeviceReset, or a context the caller made
//    current through the driver API) looks the address up again, so the
//    first call in each new context is a set-up call too.  Where the driver
//    gives no context ID, every call looks the address up.
//  * Every call uses the same array and leaves the previous call's carries
//    in it.  Nothing in it needs to start at zero: each call writes every
//    carry slot it reads.  Calls that overlap on the GPU (other streams, other
//    host threads) race on the array; serialise them.
// ---------------------------------------------------------------------------
#include <mutex>

namespace mgb {
namespace {
constexpr size_t COO_NOALLOC_BYTES = size_t(4) << 20;
}  // namespace
}  // namespace mgb

static __device__ __align__(256) unsigned char g_coo_noalloc_scratch[mgb::COO_NOALLOC_BYTES];

namespace mgb {
namespace {

struct NoallocSlot {
  unsigned long long ctx_id;  // unique ID of the context the address belongs to (0: none)
  void* ptr;
};
std::mutex g_noalloc_mutex;
NoallocSlot g_noalloc[128] = {};

// Device address of the scratch array in the current context: looked up on
// the first call per device and again whenever the current context changed.
int noalloc_scratch(void** out) {
  int dev = 0;
  MGB_CUDA_CHECK(cudaGetDevice(&dev));
  MGB_REQUIRE(dev >= 0 && dev < 128, MGB_ERR_RUNTIME);
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  NoallocSlot& slot = g_noalloc[dev];
  const unsigned long long id = current_ctx_id();
  if (slot.ptr == nullptr || id == 0 || slot.ctx_id != id) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_coo_noalloc_scratch);
    if (e != cudaSuccess) return record_cuda_error(e);
    slot.ptr = p;
    slot.ctx_id = id != 0 ? id : current_ctx_id();  // the look-up may have created the context
  }
  *out = slot.ptr;
  return MGB_SUCCESS;
}

int launch_coo_noalloc_f64(const mgb_coo* A, const double* x, double* y, int init, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(!bad_sizes(A->nrows, A->ncols, A->nnz), MGB_ERR_BAD_ARGUMENT);
  int64_t chunk = coo_chunk_size<double>(A->nnz), nchunks, ncarry;
  size_t rows_bytes;
  for (;; chunk <<= 1) {  // chunks as large as the array needs them, up to COO_CHUNK
    nchunks = (A->nnz + chunk - 1) / chunk;
    ncarry = 2 * nchunks;
    rows_bytes = ((sizeof(int32_t) * (size_t)ncarry + 255) / 256) * 256;
    if (rows_bytes + sizeof(double) * (size_t)ncarry <= COO_NOALLOC_BYTES) break;
    MGB_REQUIRE(chunk < COO_CHUNK, MGB_ERR_INVALID_INPUT);
  }
  MGB_REQUIRE(A->nrows < ((int64_t)1 << 31), MGB_ERR_INVALID_INPUT);
  if (A->nrows == 0) return MGB_SUCCESS;
  MGB_REQUIRE(y != nullptr, MGB_ERR_BAD_ARGUMENT);
  if (A->nnz == 0) {
    if (init) MGB_CUDA_CHECK(cudaMemsetAsync(y, 0, sizeof(double) * A->nrows, s));
    return MGB_SUCCESS;
  }
  MGB_REQUIRE(A->row_indices && A->column_indices && A->values && x, MGB_ERR_BAD_ARGUMENT);
  void* scratch = nullptr;
  int st = noalloc_scratch(&scratch);
  if (st != MGB_SUCCESS) return st;
  int32_t* cr = static_cast<int32_t*>(scratch);
  double* cv = reinterpret_cast<double*>(static_cast<char*>(scratch) + rows_bytes);
  st = coo_segments<double>(A, chunk, nchunks, x, y, init, cr, cv, s);  // nnz is far below 2^31 here
  if (st != MGB_SUCCESS) return st;
  coo_carry_fixup<double><<<(unsigned)((ncarry + 255) / 256), 256, 0, s>>>(ncarry, A->nrows, cr, cv, y, init);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

}  // namespace
}  // namespace mgb

extern "C" int mgb_spmv_coo_f64_noalloc(const mgb_coo* A, const double* x, double* y, int init, void* stream) {
  return mgb::launch_coo_noalloc_f64(A, x, y, init, mgb::as_stream(stream));
}
