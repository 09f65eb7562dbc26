// convert.cu -- format conversions on the GPU, bit-exact with the reference's
// Serial convert (the reference's CUDA convert throws NotImplementedException
// for every pair: impl/<Fmt>/Cuda/Morpheus_Convert_Impl.hpp).
//
// Every X -> COO builds the reference's pre-sort array in the reference's
// order (including the (0,0,0) tail entries left when exact zeros are dropped)
// and, only if that array is not sorted, applies a stable (row, col) sort
// (equal to the reference's two stable counting sorts,
// impl/Coo/Serial/Morpheus_Sort_Impl.hpp:109-164).  Every COO -> Y follows the
// reference's placement loop: slot numbers restart whenever the row changes,
// later entries overwrite earlier ones at the same slot, remainders keep COO
// order.  Output sizes come from *_plan calls, which also apply the
// reference's fill-tolerance test (impl/Morpheus_Utils.hpp:91-105, in FP32).
#include <algorithm>
#include <climits>
#include <cstdint>
#include <vector>

#include "primitives.cuh"

namespace mgb {
namespace {

using prim::blocks_for;
using prim::Scratch;

inline unsigned grid_for(int64_t n) { return blocks_for(n, 256, (int64_t)num_sms() * 16); }

// core/src/impl/Morpheus_Utils.hpp:91-105 (single-precision arithmetic)
bool exceeds_tolerance(int64_t num_rows, int64_t num_entries, int64_t num_columns) {
  const float max_fill = 10.0f;
  const float threshold = 100e6f;
  const float size = float(num_columns) * float(num_rows);
  const float fill_ratio = size / std::max(1.0f, float(num_entries));
  return fill_ratio > max_fill && size > threshold;
}

template <typename T>
__global__ void fill_kernel(T* p, T v, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

template <typename T>
int fill(T* p, T v, int64_t n, cudaStream_t s) {
  if (n <= 0) return MGB_SUCCESS;
  fill_kernel<T><<<grid_for(n), 256, 0, s>>>(p, v, n);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

using prim::Words;
using prim::words_alloc;
using prim::words_read;

// MGB_ERR_INVALID_INPUT if any row is outside [0, nrows) or column outside
// [0, ncols): the reference has no check and indexes out of bounds there.
inline bool words_valid(const Words& h) { return (h.seen & prim::COO_BAD_INDEX) == 0; }
inline bool words_rows_sorted(const Words& h) { return (h.seen & prim::COO_ROWS_UNSORTED) == 0; }
// sorted by (row, column) without equal pairs: no two entries share a place
inline bool words_distinct(const Words& h) { return (h.seen & (prim::COO_UNSORTED | prim::COO_DUPLICATE)) == 0; }

int sorted_and_dup(const int32_t* r, const int32_t* c, int64_t n, bool* sorted, bool* dup, cudaStream_t s) {
  Scratch sc(s);
  int32_t* d;
  MGB_SCRATCH(sc, d, 2);
  int st = prim::coo_sorted_flags(r, c, n, d, d + 1, s);
  if (st) return st;
  int32_t h[2];
  MGB_CUDA_CHECK(cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, s));
  MGB_CUDA_CHECK(cudaStreamSynchronize(s));
  *sorted = h[0] != 0;
  if (dup) *dup = h[1] != 0;
  return MGB_SUCCESS;
}

// In-place stable (row, col) sort of a COO array with rows in [0, nbins).
template <typename T>
int sort_coo_inplace(int32_t* rows, int32_t* cols, T* vals, int64_t n, int64_t nbins, Scratch& sc, cudaStream_t s) {
  if (n <= 1) return MGB_SUCCESS;
  return prim::row_sort<T, true>(rows, cols, vals, n, nbins, nullptr, rows, cols, vals, sc, s);
}

// The reference's "if (!is_sorted(dst)) sort_by_row_and_column(dst)" on a
// freshly built COO; rows of the pre-sort array are in [0, nrows).
template <typename T>
int sort_if_unsorted(mgb_coo* dst, cudaStream_t s) {
  if (dst->nnz <= 1) return MGB_SUCCESS;
  bool sorted = false;
  int st = sorted_and_dup(dst->row_indices, dst->column_indices, dst->nnz, &sorted, nullptr, s);
  if (st || sorted) return st;
  Scratch sc(s);
  return sort_coo_inplace<T>(dst->row_indices, dst->column_indices, static_cast<T*>(dst->values), dst->nnz,
                             dst->nrows, sc, s);
}

int check_coo_dst(const mgb_coo* d, int64_t nrows, int64_t ncols, int64_t nnz) {
  MGB_REQUIRE(d != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(d->nrows == nrows && d->ncols == ncols && d->nnz == nnz, MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(nnz == 0 || (d->row_indices && d->column_indices && d->values), MGB_ERR_BAD_ARGUMENT);
  return MGB_SUCCESS;
}

template <typename T>
int zero_coo(mgb_coo* d, cudaStream_t s) {
  if (d->nnz <= 0) return MGB_SUCCESS;
  MGB_CUDA_CHECK(cudaMemsetAsync(d->row_indices, 0, sizeof(int32_t) * d->nnz, s));
  MGB_CUDA_CHECK(cudaMemsetAsync(d->column_indices, 0, sizeof(int32_t) * d->nnz, s));
  MGB_CUDA_CHECK(cudaMemsetAsync(d->values, 0, sizeof(T) * d->nnz, s));
  return MGB_SUCCESS;
}

// ---------------------------------------------------------------- CSR <-> COO
// impl/Csr/Serial/Morpheus_Convert_Impl.hpp:70-97
// rows[j + shift] = the row of CSR entry j, one warp per 32 rows, 32 entries
// per store (a thread per row wrote 4 bytes at a time: 608 us for the 437 MB of
// the 27-point stencil at 160^3).  Entries before the first offset or past
// the last one (offsets that do not span the entries) get row 0.
__global__ void __launch_bounds__(256) expand_rows(const int32_t* __restrict__ ro, int64_t nrows, int64_t nnz,
                                                   int32_t* __restrict__ rows, int64_t shift) {
  __shared__ prim::WarpRows s_rows[8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t* out = rows + shift;
  for (int64_t r0 = ((int64_t)blockIdx.x * 8 + w) * 32; r0 < nrows; r0 += (int64_t)gridDim.x * 256)
    prim::warp_row_walk(ro, r0, nrows, s_rows[w], lane, 0, 1, [](int64_t, int) { return 0; },
                        [&](bool in, bool, int q, int64_t c0, int i, int) {
                          if (in && c0 + i >= 0 && c0 + i < nnz) __stcs(out + c0 + i, (int32_t)(r0 + q));
                        });
  const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x, nt = (int64_t)gridDim.x * 256;
  const int64_t first = min((int64_t)ro[0], nnz), last = max((int64_t)ro[nrows], (int64_t)0);
  for (int64_t j = t; j < first; j += nt) out[j] = 0;
  for (int64_t j = last + t; j < nnz; j += nt) out[j] = 0;
}

template <typename T>
int csr_to_coo(const mgb_csr* src, mgb_coo* dst, cudaStream_t s) {
  MGB_REQUIRE(src != nullptr, MGB_ERR_BAD_ARGUMENT);
  int st = check_coo_dst(dst, src->nrows, src->ncols, src->nnz);
  if (st) return st;
  if (src->nnz == 0) return MGB_SUCCESS;
  expand_rows<<<grid_for(src->nrows), 256, 0, s>>>(src->row_offsets, src->nrows, src->nnz, dst->row_indices, 0);
  MGB_LAUNCH_CHECK();
  if (dst->column_indices != src->column_indices)
    MGB_CUDA_CHECK(cudaMemcpyAsync(dst->column_indices, src->column_indices, sizeof(int32_t) * src->nnz,
                                   cudaMemcpyDeviceToDevice, s));
  if (dst->values != src->values)
    MGB_CUDA_CHECK(cudaMemcpyAsync(dst->values, src->values, sizeof(T) * src->nnz, cudaMemcpyDeviceToDevice, s));
  return MGB_SUCCESS;
}

// impl/Csr/Serial/Morpheus_Convert_Impl.hpp:99-151: counting scatter, COO order within a row
struct CsrPlan {
  int32_t* start = nullptr;  // of sorted rows: the row offsets
  Words h{};
};
int csr_plan(const mgb_coo* src, CsrPlan* p, Scratch& sc, cudaStream_t s) {
  Words* dw;
  int st = words_alloc(sc, &dw, s);
  if (st) return st;
  int32_t* gaps;
  MGB_SCRATCH(sc, p->start, src->nrows + 1);
  MGB_SCRATCH(sc, gaps, prim::gap_words(src->nrows));
  st = prim::coo_pass(src->row_indices, src->column_indices, src->nnz, src->nrows, src->ncols, dw, nullptr, p->start,
                      gaps, false, s);
  if (st) return st;
  st = words_read(dw, &p->h, s);
  if (st) return st;
  if (prim::gaps_left(p->h)) return prim::coo_pass_gaps(src->row_indices, src->nrows, dw, gaps, p->start, s);
  return words_valid(p->h) ? MGB_SUCCESS : MGB_ERR_INVALID_INPUT;
}

template <typename T>
int csr_fill(const mgb_coo* src, const CsrPlan& p, mgb_csr* dst, Scratch& sc, cudaStream_t s) {
  const int64_t n = src->nnz, N = src->nrows;
  MGB_REQUIRE(dst->nrows == N && dst->ncols == src->ncols && dst->nnz == n, MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(dst->row_offsets != nullptr, MGB_ERR_BAD_ARGUMENT);
  if (!words_rows_sorted(p.h))
    return prim::row_sort<T, false>(src->row_indices, src->column_indices, static_cast<const T*>(src->values), n, N,
                                    dst->row_offsets, nullptr, dst->column_indices, static_cast<T*>(dst->values), sc,
                                    s);
  MGB_CUDA_CHECK(cudaMemcpyAsync(dst->row_offsets, p.start, sizeof(int32_t) * (N + 1), cudaMemcpyDeviceToDevice, s));
  if (n == 0) return MGB_SUCCESS;
  MGB_CUDA_CHECK(cudaMemcpyAsync(dst->column_indices, src->column_indices, sizeof(int32_t) * n,
                                 cudaMemcpyDeviceToDevice, s));
  MGB_CUDA_CHECK(cudaMemcpyAsync(dst->values, src->values, sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
  return MGB_SUCCESS;
}

template <typename T>
int coo_to_csr(const mgb_coo* src, mgb_csr* dst, cudaStream_t s) {
  MGB_REQUIRE(src != nullptr && dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(dst->nrows == src->nrows && dst->ncols == src->ncols && dst->nnz == src->nnz, MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(dst->row_offsets != nullptr, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  CsrPlan p;
  const int st = csr_plan(src, &p, sc, s);
  return st ? st : csr_fill<T>(src, p, dst, sc, s);
}

// ---------------------------------------------------------------- DIA -> COO
// impl/Dia/Serial/Morpheus_Convert_Impl.hpp:72-118 (slab order = diagonal-major)
template <typename T>
__global__ void dia_flags(const int32_t* __restrict__ offs, const T* __restrict__ vals, int64_t nrows,
                          int64_t ncols, int64_t pitch, int64_t total, uint8_t* flags) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / pitch, row = t - i * pitch;
    const int64_t col = row + offs[i];
    flags[t] = (row < nrows && col >= 0 && col < ncols && vals[t] != T(0)) ? 1 : 0;
  }
}

template <typename T>
__global__ void dia_scatter(const int32_t* __restrict__ offs, const T* __restrict__ vals, int64_t pitch,
                            int64_t total, const uint8_t* __restrict__ flags, const int64_t* __restrict__ pos,
                            int64_t limit, int32_t* rows, int32_t* cols, T* out) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    if (!flags[t]) continue;
    const int64_t p = pos[t];
    if (p >= limit) continue;
    const int64_t i = t / pitch, row = t - i * pitch;
    rows[p] = (int32_t)row;
    cols[p] = (int32_t)(row + offs[i]);
    out[p] = vals[t];
  }
}

// writes the DIA entries (nonzero, in range) into dst at [0, found); returns found
template <typename T>
int dia_part_to_coo(const mgb_dia* src, mgb_coo* dst, int64_t limit, int64_t* found, cudaStream_t s) {
  *found = 0;
  const int64_t total = src->pitch * src->ndiags;
  if (total == 0) return MGB_SUCCESS;
  Scratch sc(s);
  uint8_t* flags;
  int64_t *pos, *d_total;
  MGB_SCRATCH(sc, flags, total);
  MGB_SCRATCH(sc, pos, total);
  MGB_SCRATCH(sc, d_total, 1);
  dia_flags<T><<<grid_for(total), 256, 0, s>>>(src->diagonal_offsets, static_cast<const T*>(src->values),
                                               src->nrows, src->ncols, src->pitch, total, flags);
  MGB_LAUNCH_CHECK();
  int st = prim::exclusive_scan<uint8_t, int64_t>(flags, pos, total, s, d_total);
  if (st) return st;
  dia_scatter<T><<<grid_for(total), 256, 0, s>>>(src->diagonal_offsets, static_cast<const T*>(src->values),
                                                 src->pitch, total, flags, pos, limit, dst->row_indices,
                                                 dst->column_indices, static_cast<T*>(dst->values));
  MGB_LAUNCH_CHECK();
  return prim::to_host(d_total, found, s);
}

int check_dia(const mgb_dia* d) {
  MGB_REQUIRE(d != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(d->nrows >= 0 && d->ncols >= 0 && d->nnz >= 0 && d->ndiags >= 0, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(d->ndiags == 0 || (d->pitch >= d->nrows && d->diagonal_offsets && d->values), MGB_ERR_BAD_ARGUMENT);
  return MGB_SUCCESS;
}

template <typename T>
int dia_to_coo(const mgb_dia* src, mgb_coo* dst, cudaStream_t s) {
  int st = check_dia(src);
  if (st) return st;
  st = check_coo_dst(dst, src->nrows, src->ncols, src->nnz);
  if (st || src->nnz == 0) return st;
  st = zero_coo<T>(dst, s);
  if (st) return st;
  int64_t found = 0;
  st = dia_part_to_coo<T>(src, dst, dst->nnz, &found, s);
  if (st) return st;
  MGB_REQUIRE(found <= src->nnz, MGB_ERR_RUNTIME);  // the reference would write past dst
  return sort_if_unsorted<T>(dst, s);
}

// ---------------------------------------------------------------- COO -> DIA
// impl/Dia/Serial/Morpheus_Convert_Impl.hpp:120-169

// place values(row, slot) = v; owner != nullptr resolves collisions to the
// highest COO position (the reference's loop order: last write wins)
template <typename T>
__global__ void dia_place(const int32_t* __restrict__ r, const int32_t* __restrict__ c, const T* __restrict__ v,
                          int64_t n, int64_t nrows, const int32_t* __restrict__ slot, int64_t pitch, T* vals,
                          int32_t* owner, int pass) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t at = r[i] + pitch * (int64_t)slot[(int64_t)c[i] - r[i] + nrows - 1];
    if (owner == nullptr) vals[at] = v[i];
    else if (pass == 0) atomicMax(owner + at, (int32_t)i);
    else if (owner[at] == (int32_t)i) vals[at] = v[i];
  }
}

// ---- slabs from row-sorted entries, tile by tile
//
// A CTA owns R consecutive rows of D diagonals at a time: the rows' entries
// (one contiguous range, found and told apart by the row starts: the row
// indices are not read) go through shared memory to their (diagonal, row) place, and the tile is written column by column, padding included, in
// consecutive rows.  So every value of the slab is written once, in full
// sectors, and nothing is cleared before.  Placing each entry with its own
// 8-byte store into a cleared slab took 2,012 us on the 27-point stencil at
// 160^3 (HBM 35 %; the entries, the slab and the row starts once are 400 us
// at the copy rate).  The tile's rows are padded to an odd stride: the
// entries of a row go to different banks.  Diagonals are looked up in a table
// in shared memory while they are few (DIA_HASH_DIAGS), else in the bin ->
// slot array.
constexpr int DIA_TILE_THREADS = 128;
constexpr int DIA_TILE_BYTES = 16 * 1024;
constexpr int DIA_TILE_ROWS = 512;  // at most
constexpr int DIA_HASH_DIAGS = 256;  // at most a quarter of the table's slots
constexpr int DIA_HASH_LOG2 = 10;
constexpr int DIA_HASH_SLOTS = 1 << DIA_HASH_LOG2;
constexpr int32_t DIA_HASH_FREE = INT32_MIN;  // no offset: |offset| < 2^31 - 1

struct DiaTable {
  int2* e;  // x: diagonal offset (DIA_HASH_FREE: none), y: its slot
};
__device__ __forceinline__ unsigned dia_hash(int32_t d) {
  return ((uint32_t)d * 0x9E3779B1u) >> (32 - DIA_HASH_LOG2);
}

// every thread; the caller synchronises.  Equal offsets keep the lowest slot.
__device__ __forceinline__ void dia_table_clear(DiaTable t) {
  for (int i = threadIdx.x; i < DIA_HASH_SLOTS; i += blockDim.x) t.e[i] = make_int2(DIA_HASH_FREE, INT32_MAX);
}
__device__ __forceinline__ void dia_table_fill(DiaTable t, const int32_t* __restrict__ offs, int nd) {
  for (int k = threadIdx.x; k < nd; k += blockDim.x) {
    const int32_t d = offs[k];
    unsigned h = dia_hash(d);
    for (int p = 0; p < DIA_HASH_SLOTS; p++) {
      const int32_t was = atomicCAS(&t.e[h].x, DIA_HASH_FREE, d);
      if (was == DIA_HASH_FREE || was == d) break;
      h = (h + 1) & (DIA_HASH_SLOTS - 1);
    }
    atomicMin(&t.e[h].y, k);
  }
}
__device__ __forceinline__ int dia_table_find(DiaTable t, int32_t d) {
  unsigned h = dia_hash(d);
  int2 e = t.e[h];
  while (e.x != d) {
    if (e.x == DIA_HASH_FREE) return -1;
    h = (h + 1) & (DIA_HASH_SLOTS - 1);
    e = t.e[h];
  }
  return e.y;
}

// First position in [b, e) with c[position] >= col, columns in order.
__device__ __forceinline__ int64_t lower_column(const int32_t* __restrict__ c, int64_t b, int64_t e, int64_t col) {
  while (b < e) {
    const int64_t mid = (b + e) >> 1;
    if (__ldg(c + mid) < col) b = mid + 1; else e = mid;
  }
  return b;
}

// REM (HDC): also rem[row] = the row's entries on no stored diagonal.  LONGS:
// rows of more than `longest` entries, most of them on none, are not walked, the
// stored diagonals' entries are searched in them (a tridiagonal matrix of 1e6
// rows with a full last one: the conversion 19,600 us with a warp per row here
// and in the remainder, 250).
template <typename T, bool REM, bool LONGS>
__global__ void __launch_bounds__(DIA_TILE_THREADS, 10)
dia_fill_tiles(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
               int64_t nrows, int64_t pitch, int nd, const int32_t* __restrict__ offs,
               const int32_t* __restrict__ bin_slot, T* __restrict__ out, int32_t* __restrict__ rem, int R, int D,
               int longest) {
  constexpr int WARPS = DIA_TILE_THREADS / 32;
  extern __shared__ __align__(16) unsigned char dia_smem[];
  T* tile = reinterpret_cast<T*>(dia_smem);
  __shared__ int2 h_table[DIA_HASH_SLOTS];
  __shared__ int32_t s_rem[REM ? DIA_TILE_ROWS : 1];
  __shared__ prim::WarpRows s_rows[WARPS];
  const DiaTable table{h_table};
  const bool hashed = nd <= DIA_HASH_DIAGS;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, S = R + 1;
  const int groups = R / 32;                              // of 32 rows
  const int share = groups < WARPS ? WARPS / groups : 1;  // warps that share a group's entries
  if constexpr (REM)
    for (int i = threadIdx.x; i < R; i += DIA_TILE_THREADS) s_rem[i] = 0;
  if (hashed) dia_table_clear(table);
  for (int i = threadIdx.x; i < D * S; i += DIA_TILE_THREADS) tile[i] = T(0);
  __syncthreads();
  if (hashed) dia_table_fill(table, offs, nd);
  __syncthreads();
  const int64_t ntiles = (pitch + R - 1) / R;
  struct Entry {
    int32_t col;
    T val;
  };
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t r0 = t * R;
    for (int d0 = 0; d0 < nd; d0 += D) {
      const int dn = min(D, nd - d0);
      for (int g = w / share; g < groups; g += WARPS / share) {
        const int64_t g0 = r0 + 32 * g;
        if (g0 >= nrows) break;
        unsigned longs = 0;
        if constexpr (LONGS)
          longs = __ballot_sync(0xffffffffu,
                                start[min(g0 + lane + 1, nrows)] - start[min(g0 + lane, nrows)] > longest);
        for (int64_t p = g0;;) {  // the rows up to the next long one, and that one
          const int64_t end = longs ? g0 + __ffs(longs) - 1 : min(g0 + 32, nrows);
          const int q0 = (int)(p - g0);
          if (!LONGS || p < end)
            prim::warp_row_walk(
                start, p, LONGS ? end : nrows, s_rows[w], lane, w % share, share,
                [&](int64_t c0, int i) { return Entry{__ldcs(c + c0 + i), __ldcs(v + c0 + i)}; },
                [&](bool in, bool, int q, int64_t, int, Entry x) {
                  if (!in) return;
                  if (LONGS) q += q0;
                  const int32_t d = x.col - (int32_t)g0 - q;
                  const int found = hashed ? dia_table_find(table, d) : bin_slot[(int64_t)d + nrows - 1];
                  const int s = found - d0;
                  if (s >= 0 && s < dn) tile[s * S + 32 * g + q] = x.val;
                  if (REM && found < 0 && d0 == 0) atomicAdd(s_rem + 32 * g + q, 1);
                });
          if (!LONGS || !longs) break;
          const int64_t b = start[end], e = start[end + 1];
          const int q = 32 * g + (int)(end - g0);
          int hits = 0;
          for (int d = (d0 == 0 ? 0 : d0) + 32 * (w % share) + lane; d < (d0 == 0 ? nd : d0 + dn); d += 32 * share) {
            const int64_t col = end + offs[d], at = lower_column(c, b, e, col);
            if (at == e || c[at] != col) continue;
            hits++;
            if (d < d0 + dn) tile[(d - d0) * S + q] = v[at];
          }
          if (d0 == 0) {
            hits = __reduce_add_sync(0xffffffffu, hits);
            if (lane == 0) atomicAdd(s_rem + q, (w % share == 0 ? (int)(e - b) : 0) - hits);
          }
          longs &= longs - 1;
          p = end + 1;
        }
      }
      __syncthreads();
      if (REM && d0 == 0)
        for (int q = threadIdx.x; q < R; q += DIA_TILE_THREADS) {
          if (r0 + q < nrows) rem[r0 + q] = s_rem[q];
          s_rem[q] = 0;
        }
      for (int d = w; d < dn; d += WARPS)
        for (int q = lane; q < R; q += 32) {
          if (r0 + q < pitch) __stcs(out + r0 + q + pitch * (int64_t)(d0 + d), tile[d * S + q]);
          tile[d * S + q] = T(0);
        }
      __syncthreads();
    }
  }
}

// Tile shape for nd diagonals: the most rows (32..512) whose tile of all
// diagonals fits DIA_TILE_BYTES, else 32 rows of as many diagonals as fit
// (the rows' entries are then read once per group of diagonals).
template <typename T>
void dia_tile_shape(int64_t nd, int* R, int* D) {
  *R = DIA_TILE_ROWS;
  while (*R > 32 && nd * (*R + 1) * (int64_t)sizeof(T) > DIA_TILE_BYTES) *R >>= 1;
  *D = (int)std::min<int64_t>(nd, DIA_TILE_BYTES / ((*R + 1) * (int64_t)sizeof(T)));
}
// More diagonals and the entries are placed one by one instead (a COO source) or
// made a COO first (CSR): every group of D diagonals reads the rows' entries
// again, and beyond DIA_HASH_DIAGS each looks its slot up in global memory.  Whole
// conversions, us, tiles / placed (150,000 rows, half of the slots filled; HDC 100,000):
//   diagonals     63         125        187        249        373          497
//   FP64 COO      165 / 132  210 / 205  285 / 270  378 / 340   793 /  488  1336 /  647
//        CSR      183 / 301  322 / 462  441 / 603  624 / 777  1593 / 1162  2620 / 1545
//   FP64 HDC COO  202 / 266  263 / 551  342 / 735  472 / 909  1149 / 1282  1836 / 1645
//        HDC CSR  222 / 411  298 / 743  420 / 980  563 /1190  1279 / 1648  1997 / 2110
//   FP32 CSR         -       283 / 395     -       495 / 646   978 /  942  1514 / 1248
//   FP32 HDC COO  177 / 261  231 / 516  269 / 693  367 / 845   688 / 1180  1068 / 1507
// and, 1,200,000 rows, one group: FP64 62 diagonals 561 / 973, FP32 124 995 / 1728
// (slabs beyond L2 are where placing costs most).  HDC's other way also reads the
// entries several times, so its line is later.
constexpr int64_t HDC_TILE_GROUPS = 6;

template <typename T>
int launch_dia_fill(const mgb_coo* src, const int32_t* start, int64_t pitch, int64_t nd, const int32_t* offs,
                    const int32_t* bin_slot, T* out, int32_t* rem, bool longs, cudaStream_t s) {
  int R, D;
  dia_tile_shape<T>(nd, &R, &D);
  const size_t smem = sizeof(T) * (size_t)D * (R + 1);
  // one resident wave: every CTA sets its table up once
  const int64_t per_sm = std::min<int64_t>(10, (200 * 1024) / (int64_t)(smem + 12 * 1024));
  const unsigned grid = blocks_for((pitch + R - 1) / R, 1, (int64_t)num_sms() * std::max<int64_t>(1, per_sm));
  const T* v = static_cast<const T*>(src->values);
  // a search of 32 diagonals costs about what 1,500 entries of the walk do
  const int longest = 2048 * (int)((nd + 31) / 32);
  const auto run = [&](auto kernel) {
    kernel<<<grid, DIA_TILE_THREADS, smem, s>>>(src->column_indices, v, start, src->nrows, pitch, (int)nd, offs,
                                                bin_slot, out, rem, R, D, longest);
  };
  if (rem == nullptr) run(dia_fill_tiles<T, false, false>);
  else if (!longs) run(dia_fill_tiles<T, true, false>);
  else run(dia_fill_tiles<T, true, true>);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}
inline bool dia_tiled(int64_t nd) { return nd > 0 && nd <= DIA_HASH_DIAGS; }
template <typename T>
bool hdc_tiled(int64_t nd) {
  if (nd == 0) return false;
  int R, D;
  dia_tile_shape<T>(nd, &R, &D);
  return (nd + D - 1) / D <= HDC_TILE_GROUPS;
}

// Argument checks of a COO source (the index pass checks the index ranges, read
// back with the caller's other words).
int check_coo_args(const mgb_coo* src, bool diagonals = true) {
  MGB_REQUIRE(src != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(src->nrows >= 0 && src->ncols >= 0 && src->nnz >= 0, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(src->nnz == 0 || (src->row_indices && src->column_indices && src->values), MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(!diagonals || src->nrows + src->ncols < INT32_MAX, MGB_ERR_INVALID_INPUT);
  return MGB_SUCCESS;
}

// One pass over the entries' indices into *dw (and the diagonal counts unless
// null); start: a CSR matrix's offsets, else, if asked for, row starts in
// scratch.
struct IndexPass {
  const int32_t* start = nullptr;
  int32_t *own = nullptr, *gaps = nullptr;
};
int index_pass(const mgb_coo* src, const int32_t* ro, bool starts, bool huge, Words* dw, int32_t* diag, IndexPass* p,
               Scratch& sc, cudaStream_t s) {
  if (ro != nullptr) {
    p->start = ro;
    int2* pieces;
    MGB_SCRATCH(sc, pieces, prim::max_row_pieces(src->nnz));
    return prim::csr_pass(ro, src->column_indices, src->nnz, src->nrows, src->ncols, dw, diag, pieces, s);
  }
  if (starts) {
    MGB_SCRATCH(sc, p->own, src->nrows + 1);
    MGB_SCRATCH(sc, p->gaps, prim::gap_words(src->nrows));
  }
  p->start = p->own;
  return prim::coo_pass(src->row_indices, src->column_indices, src->nnz, src->nrows, src->ncols, dw, diag, p->own,
                        p->gaps, huge, s);
}

// The pass, then the sizes (queued by `sizes`) and one host read; sizes and read
// again where the pass left long gaps.
template <typename SIZES>
int pass_and_sizes(const mgb_coo* src, const int32_t* ro, bool starts, bool huge, Words* dw, int32_t* diag,
                   IndexPass* p, Words* h, Scratch& sc, cudaStream_t s, SIZES sizes) {
  int st = index_pass(src, ro, starts, huge, dw, diag, p, sc, s);
  for (;;) {
    if (!st) st = sizes();
    if (!st) st = words_read(dw, h, s);
    if (st || !prim::gaps_left(*h)) return st;
    st = prim::coo_pass_gaps(src->row_indices, src->nrows, dw, p->gaps, p->own, s);
  }
}

// COO -> DIA sizes: one pass over the indices counts the diagonals, checks
// the ranges and the order and (starts) finds the row starts; the occupied
// bins are counted; one host read.
// ro: the offsets of a CSR matrix, whose entries src then holds without row
// indices (here and in the plans below).
struct DiaPlan {
  int32_t* counts = nullptr;
  const int32_t* start = nullptr;
  int64_t* sums = nullptr;
  Words h{};
};
int dia_plan(const mgb_coo* src, const int32_t* ro, bool starts, DiaPlan* p, Scratch& sc, cudaStream_t s) {
  int st = ro ? MGB_SUCCESS : check_coo_args(src);
  if (st) return st;
  Words* dw;
  st = words_alloc(sc, &dw, s);
  if (st) return st;
  const int64_t nb = src->nrows + src->ncols - 1;
  MGB_SCRATCH(sc, p->counts, nb > 0 ? nb : 1);
  if (src->nnz > 0 && nb > 0) MGB_SCRATCH(sc, p->sums, prim::bin_tiles(nb));
  IndexPass pass;
  st = pass_and_sizes(src, ro, starts, false, dw, p->counts, &pass, &p->h, sc, s, [&] {
    return p->sums ? prim::select_bins(p->counts, nb, 1, p->sums, &dw->total, nullptr, s) : MGB_SUCCESS;
  });
  if (st) return st;
  p->start = pass.start;
  if (!words_valid(p->h)) return MGB_ERR_INVALID_INPUT;
  if (exceeds_tolerance(src->nrows, src->nnz, p->h.total)) return MGB_ERR_FORMAT_CONVERSION;
  return MGB_SUCCESS;
}

int coo_to_dia_plan(const mgb_coo* src, int64_t* ndiags, cudaStream_t s) {
  MGB_REQUIRE(ndiags != nullptr, MGB_ERR_BAD_ARGUMENT);
  *ndiags = 0;
  Scratch sc(s);
  DiaPlan p;
  const int st = dia_plan(src, nullptr, false, &p, sc, s);
  if (st == MGB_SUCCESS || st == MGB_ERR_FORMAT_CONVERSION) *ndiags = p.h.total;
  return st;
}

template <typename T>
int dia_fill(const mgb_coo* src, const DiaPlan& p, mgb_dia* dst, cudaStream_t s) {
  Scratch sc(s);
  int st;
  const int64_t nd = p.h.total;
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(dst->nrows == src->nrows && dst->ncols == src->ncols && dst->nnz == src->nnz && dst->ndiags == nd &&
                  dst->pitch >= src->nrows,
              MGB_ERR_INVALID_INPUT);
  if (nd == 0) return MGB_SUCCESS;
  MGB_REQUIRE(dst->diagonal_offsets && dst->values, MGB_ERR_BAD_ARGUMENT);
  const int64_t n = src->nnz, nb = src->nrows + src->ncols - 1;
  st = prim::select_bins_apply(p.counts, nb, 1, p.sums, src->nrows, -1, dst->diagonal_offsets, s);
  if (st) return st;
  const int32_t* slot = p.counts;  // bin -> slot now
  const T* v = static_cast<const T*>(src->values);
  T* out = static_cast<T*>(dst->values);
  const bool distinct = words_distinct(p.h);
  if (distinct && dia_tiled(nd))
    return launch_dia_fill<T>(src, p.start, dst->pitch, nd, dst->diagonal_offsets, slot, out, nullptr, false, s);
  MGB_CUDA_CHECK(cudaMemsetAsync(dst->values, 0, sizeof(T) * dst->pitch * nd, s));
  if (distinct) {
    dia_place<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices, v, n, src->nrows, slot,
                                             dst->pitch, out, nullptr, 0);
    MGB_LAUNCH_CHECK();
  } else {
    int32_t* owner;
    MGB_SCRATCH(sc, owner, dst->pitch * nd);
    st = fill<int32_t>(owner, -1, dst->pitch * nd, s);
    if (st) return st;
    for (int pass = 0; pass < 2; pass++) {
      dia_place<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices, v, n, src->nrows, slot,
                                               dst->pitch, out, owner, pass);
      MGB_LAUNCH_CHECK();
    }
  }
  return MGB_SUCCESS;
}

template <typename T>
int coo_to_dia(const mgb_coo* src, mgb_dia* dst, cudaStream_t s) {
  Scratch sc(s);
  DiaPlan p;
  const int st = dia_plan(src, nullptr, true, &p, sc, s);
  return st ? st : dia_fill<T>(src, p, dst, s);
}

// ---------------------------------------------------------------- ELL -> COO
// impl/Ell/Serial/Morpheus_Convert_Impl.hpp:68-109
__global__ void ell_row_counts(const int32_t* __restrict__ ci, int64_t nrows, int64_t width, int64_t pitch,
                               int32_t* counts) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = 0;
    for (int64_t k = 0; k < width; k++) c += ci[r + pitch * k] != MGB_INVALID_INDEX;
    counts[r] = c;
  }
}

// per row: ELL slots in order, then (HYB) the row's COO-prefix entries
template <typename T>
__global__ void ell_rows_to_coo(const int32_t* __restrict__ ci, const T* __restrict__ ev, int64_t nrows,
                                int64_t width, int64_t pitch, const int32_t* __restrict__ pos, int64_t limit,
                                const int32_t* __restrict__ coo_start, const int32_t* __restrict__ coo_count,
                                const int32_t* __restrict__ cc, const T* __restrict__ cv, int32_t* rows,
                                int32_t* cols, T* out) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x) {
    int64_t p = pos[r];
    for (int64_t k = 0; k < width; k++) {
      const int32_t c = ci[r + pitch * k];
      if (c != MGB_INVALID_INDEX) {
        if (p < limit) { rows[p] = (int32_t)r; cols[p] = c; out[p] = ev[r + pitch * k]; }
        p++;
      }
    }
    if (coo_count) {
      const int64_t a = coo_start[r], cnt = coo_count[r];
      for (int64_t j = a; j < a + cnt; j++) {
        if (p < limit) { rows[p] = (int32_t)r; cols[p] = cc[j]; out[p] = cv[j]; }
        p++;
      }
    }
  }
}

int check_ell(const mgb_ell* e) {
  MGB_REQUIRE(e != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(e->nrows >= 0 && e->ncols >= 0 && e->nnz >= 0 && e->width >= 0, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(e->width == 0 || (e->pitch >= e->nrows && e->column_indices && e->values), MGB_ERR_BAD_ARGUMENT);
  return MGB_SUCCESS;
}

__global__ void add_i32(int32_t* a, const int32_t* __restrict__ b, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    a[i] += b[i];
}

// ELL (+ optional HYB COO-prefix) -> pre-sort COO in row-major order;
// *found = entries produced (entries beyond dst->nnz are counted, not written)
template <typename T>
int ell_like_to_coo(const mgb_ell* e, const mgb_coo* cpart, int64_t coo_prefix, mgb_coo* dst, int64_t* found,
                    cudaStream_t s) {
  const int64_t N = e->nrows;
  *found = 0;
  if (N == 0) return MGB_SUCCESS;
  Scratch sc(s);
  int32_t *counts, *pos, *coo_counts = nullptr, *coo_start = nullptr;
  int64_t* d_total;
  MGB_SCRATCH(sc, counts, N + 1);
  MGB_SCRATCH(sc, pos, N + 1);
  MGB_SCRATCH(sc, d_total, 1);
  if (e->width > 0) {
    ell_row_counts<<<grid_for(N), 256, 0, s>>>(e->column_indices, N, e->width, e->pitch, counts);
    MGB_LAUNCH_CHECK();
  } else {
    MGB_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int32_t) * N, s));
  }
  MGB_CUDA_CHECK(cudaMemsetAsync(counts + N, 0, sizeof(int32_t), s));
  int st;
  if (cpart && coo_prefix > 0) {
    MGB_SCRATCH(sc, coo_counts, N + 1);
    MGB_SCRATCH(sc, coo_start, N + 1);
    st = prim::histogram(cpart->row_indices, coo_prefix, coo_counts, N, s);
    if (st) return st;
    MGB_CUDA_CHECK(cudaMemsetAsync(coo_counts + N, 0, sizeof(int32_t), s));
    st = prim::exclusive_scan<int32_t, int32_t>(coo_counts, coo_start, N + 1, s);
    if (st) return st;
    add_i32<<<grid_for(N), 256, 0, s>>>(counts, coo_counts, N);
    MGB_LAUNCH_CHECK();
  }
  st = prim::exclusive_scan<int32_t, int32_t>(counts, pos, N + 1, s, d_total);
  if (st) return st;
  ell_rows_to_coo<T><<<grid_for(N), 256, 0, s>>>(
      e->column_indices, static_cast<const T*>(e->values), N, e->width, e->pitch, pos, dst->nnz, coo_start,
      coo_counts, cpart ? cpart->column_indices : nullptr, cpart ? static_cast<const T*>(cpart->values) : nullptr,
      dst->row_indices, dst->column_indices, static_cast<T*>(dst->values));
  MGB_LAUNCH_CHECK();
  return prim::to_host(d_total, found, s);
}

template <typename T>
int ell_to_coo(const mgb_ell* src, mgb_coo* dst, cudaStream_t s) {
  int st = check_ell(src);
  if (st) return st;
  st = check_coo_dst(dst, src->nrows, src->ncols, src->nnz);
  if (st || src->nnz == 0) return st;
  st = zero_coo<T>(dst, s);
  if (st) return st;
  int64_t found = 0;
  st = ell_like_to_coo<T>(src, nullptr, 0, dst, &found, s);
  if (st) return st;
  MGB_REQUIRE(found <= src->nnz, MGB_ERR_RUNTIME);
  return sort_if_unsorted<T>(dst, s);
}

// ---------------------------------------------------------------- HYB -> COO
// impl/Hyb/Serial/Morpheus_Convert_Impl.hpp:62-108.  The COO part is consumed
// row by row while its row index equals the current row: exactly its longest
// prefix with non-decreasing in-range rows.
__global__ void first_consume_break(const int32_t* __restrict__ r, int64_t n, int64_t nrows,
                                    unsigned long long* out) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = r[i];
    if (v < 0 || v >= nrows || (i > 0 && v < r[i - 1])) atomicMin(out, (unsigned long long)i);
  }
}

template <typename T>
int hyb_to_coo(const mgb_hyb* src, mgb_coo* dst, cudaStream_t s) {
  MGB_REQUIRE(src != nullptr, MGB_ERR_BAD_ARGUMENT);
  int st = check_ell(&src->ell);
  if (st) return st;
  const mgb_coo* c = &src->coo;
  MGB_REQUIRE(c->nnz >= 0 && (c->nnz == 0 || (c->row_indices && c->column_indices && c->values)),
              MGB_ERR_BAD_ARGUMENT);
  const int64_t nnz = src->ell.nnz + c->nnz;
  st = check_coo_dst(dst, src->ell.nrows, src->ell.ncols, nnz);
  if (st || nnz == 0) return st;
  st = zero_coo<T>(dst, s);
  if (st) return st;
  int64_t prefix = c->nnz;
  if (c->nnz > 0) {
    Scratch sc(s);
    unsigned long long* d;
    MGB_SCRATCH(sc, d, 1);
    const unsigned long long big = ~0ull;
    MGB_CUDA_CHECK(cudaMemcpyAsync(d, &big, sizeof(big), cudaMemcpyHostToDevice, s));
    first_consume_break<<<grid_for(c->nnz), 256, 0, s>>>(c->row_indices, c->nnz, src->ell.nrows, d);
    MGB_LAUNCH_CHECK();
    unsigned long long h;
    st = prim::to_host(d, &h, s);
    if (st) return st;
    if (h != big) prefix = (int64_t)h;
  }
  int64_t found = 0;
  st = ell_like_to_coo<T>(&src->ell, c, prefix, dst, &found, s);
  if (st) return st;
  MGB_REQUIRE(found <= nnz, MGB_ERR_RUNTIME);
  return sort_if_unsorted<T>(dst, s);
}

// ------------------------------------------------------- COO -> ELL / HYB
// slot of entry i = i - (start of its run of equal row indices): the
// reference's loop restarts n whenever the row index changes
// (impl/Ell/Serial/Morpheus_Convert_Impl.hpp:160-172, Hyb :174-195).
__global__ void run_flags(const int32_t* __restrict__ r, int64_t n, uint8_t* f) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    f[i] = (i == 0 || r[i] != r[i - 1]) ? 1 : 0;
}
__global__ void run_starts(const uint8_t* __restrict__ f, const int32_t* __restrict__ excl, int64_t n,
                           int32_t* starts) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (f[i]) starts[excl[i]] = (int32_t)i;
}
__global__ void run_slots(const uint8_t* __restrict__ f, const int32_t* __restrict__ excl,
                          const int32_t* __restrict__ starts, int64_t n, int32_t* slot) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    slot[i] = (int32_t)(i - starts[excl[i] + f[i] - 1]);
}
// Slot of every entry in its run (the reference's placement counter, which
// restarts whenever the row changes), for rows in any order.
int compute_slots(const mgb_coo* src, int32_t* slot, Scratch& sc, cudaStream_t s) {
  const int64_t n = src->nnz;
  if (n == 0) return MGB_SUCCESS;
  uint8_t* f;
  int32_t *excl, *starts;
  MGB_SCRATCH(sc, f, n);
  MGB_SCRATCH(sc, excl, n);
  MGB_SCRATCH(sc, starts, n);
  run_flags<<<grid_for(n), 256, 0, s>>>(src->row_indices, n, f);
  MGB_LAUNCH_CHECK();
  if (int st = prim::exclusive_scan<uint8_t, int32_t>(f, excl, n, s)) return st;
  run_starts<<<grid_for(n), 256, 0, s>>>(f, excl, n, starts);
  MGB_LAUNCH_CHECK();
  run_slots<<<grid_for(n), 256, 0, s>>>(f, excl, starts, n, slot);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

// ELL placement of entries with slot < W; owner resolves collisions to the
// highest position.  Entries with slot >= W are marked for the COO part.
template <typename T>
__global__ void ell_place(const int32_t* __restrict__ r, const int32_t* __restrict__ c, const T* __restrict__ v,
                          const int32_t* __restrict__ slot, int64_t n, int64_t W, int64_t pitch, int32_t* eci,
                          T* ev, int32_t* owner, int pass, uint8_t* to_coo) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = slot[i];
    if (k >= W) {
      if (to_coo && pass == 0) to_coo[i] = 1;
      continue;
    }
    if (to_coo && pass == 0) to_coo[i] = 0;
    const int64_t at = r[i] + pitch * k;
    if (pass == 0) {
      atomicMax(owner + at, (int32_t)i);
    } else if (owner[at] == (int32_t)i) {
      eci[at] = c[i];
      ev[at] = v[i];
    }
  }
}

template <typename T>
__global__ void coo_part_scatter(const int32_t* __restrict__ r, const int32_t* __restrict__ c,
                                 const T* __restrict__ v, const uint8_t* __restrict__ f,
                                 const int64_t* __restrict__ pos, int64_t n, int64_t limit, int32_t* orow,
                                 int32_t* ocol, T* oval) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    if (f[i] && pos[i] < limit) {
      orow[pos[i]] = r[i];
      ocol[pos[i]] = c[i];
      oval[pos[i]] = v[i];
    }
}

// ELL slab of a COO whose rows are in any order.
template <typename T>
int place_ell(const mgb_coo* src, mgb_ell* e, int64_t W, const int32_t* slot, uint8_t* to_coo, Scratch& sc,
              cudaStream_t s) {
  const int64_t n = src->nnz;
  const int64_t slab = e->pitch * e->width;
  int st = fill<int32_t>(e->column_indices, MGB_INVALID_INDEX, slab, s);
  if (st) return st;
  if (slab) MGB_CUDA_CHECK(cudaMemsetAsync(e->values, 0, sizeof(T) * slab, s));
  if (n == 0) return MGB_SUCCESS;
  int32_t* owner;
  MGB_SCRATCH(sc, owner, slab > 0 ? slab : 1);
  st = fill<int32_t>(owner, -1, slab, s);
  if (st) return st;
  for (int pass = 0; pass < 2; pass++) {
    ell_place<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices,
                                             static_cast<const T*>(src->values), slot, n, W, e->pitch,
                                             e->column_indices, static_cast<T*>(e->values), owner, pass, to_coo);
    MGB_LAUNCH_CHECK();
  }
  return MGB_SUCCESS;
}

// ELL slab of row-sorted entries: a CTA takes R rows and a segment of the slot
// columns, brings the rows' entries through shared memory and writes every slot
// of the segment, padding included, in consecutive rows: the slab is written
// once in full sectors and not cleared before.  Where the rows' entries (one
// contiguous range) do not fit ELL_TILE, ELL_TILE / R slots of every row at a
// time are staged.  A pad after every 32 staged entries spreads rows of even
// length over the banks.  Segments (grid y) divide the width where the rows
// alone are too few CTAs (COO -> ELL of 33 rows of 1e6 entries: 68,000 us with
// whole rows per CTA, 520 with segments).  Placing
// each entry alone into a cleared slab: 27-point stencil on 120 x 120 x 121, COO
// -> ELL in all 2,667 us, this way 525.
constexpr int ELL_TILE = 2048;
constexpr int ELL_TILE_ROWS = 256;
constexpr int ELL_SEGMENT = 64;  // slot columns of a segment at least
__device__ __forceinline__ int ell_pad(int i) { return i + (i >> 5); }

// The tile's rows whose entries do not fit: blocks of their slots (out of line,
// for the registers of the kernel).
template <typename T>
__device__ __noinline__ void ell_fill_long(const int32_t* __restrict__ c, const T* __restrict__ v,
                                           const int32_t* s_start, int32_t* s_c, T* s_v, int64_t r0, int64_t pitch,
                                           int64_t k_begin, int64_t k_end, int64_t W, int32_t* __restrict__ eci,
                                           T* __restrict__ ev, int R) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int block = ELL_TILE / R;  // a power of two, as R
  for (int64_t k0 = k_begin; k0 < k_end; k0 += block) {
    for (int i = threadIdx.x; i < ELL_TILE; i += 256) {
      const int q = i / block;
      const int64_t k = k0 + i % block;
      if (k < s_start[q + 1] - s_start[q]) {
        s_c[ell_pad(i)] = __ldcs(c + s_start[q] + k);
        s_v[ell_pad(i)] = __ldcs(v + s_start[q] + k);
      }
    }
    __syncthreads();
    const int64_t k1 = min(k0 + block, k_end);
    for (int q = lane; q < R && r0 + q < pitch; q += 32) {
      const int64_t len = min((int64_t)(s_start[q + 1] - s_start[q]), W);
      for (int64_t k = k0 + w; k < k1; k += 8) {
        const int i = ell_pad(q * block + (int)(k - k0));
        __stcs(eci + r0 + q + pitch * k, k < len ? s_c[i] : MGB_INVALID_INDEX);
        __stcs(ev + r0 + q + pitch * k, k < len ? s_v[i] : T(0));
      }
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(256, 8)
ell_fill_tiles(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
               int64_t nrows, int64_t pitch, int64_t width, int64_t W, int32_t* __restrict__ eci, T* __restrict__ ev,
               int R, int64_t segment) {
  __shared__ T s_v[ELL_TILE + ELL_TILE / 32];
  __shared__ int32_t s_c[ELL_TILE + ELL_TILE / 32];
  __shared__ int32_t s_start[ELL_TILE_ROWS + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t ntiles = (pitch + R - 1) / R;
  const int64_t k_begin = blockIdx.y * segment, k_end = min(k_begin + segment, width);
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t r0 = t * R;
    for (int q = threadIdx.x; q <= R; q += 256) s_start[q] = start[min(r0 + q, nrows)];
    __syncthreads();
    const int32_t e0 = s_start[0], n = s_start[R] - e0;
    if (n > ELL_TILE) {
      ell_fill_long<T>(c, v, s_start, s_c, s_v, r0, pitch, k_begin, k_end, W, eci, ev, R);
      continue;
    }
    for (int i = threadIdx.x; i < n; i += 256) {
      s_c[ell_pad(i)] = __ldcs(c + e0 + i);
      s_v[ell_pad(i)] = __ldcs(v + e0 + i);
    }
    __syncthreads();
    for (int q = lane; q < R; q += 32) {
      const int64_t row = r0 + q;
      if (row >= pitch) break;
      const int32_t b = s_start[q];
      const int64_t len = min((int64_t)(s_start[q + 1] - b), W);
      for (int64_t k = k_begin + w; k < k_end; k += 8) {
        int32_t col = MGB_INVALID_INDEX;
        T val = T(0);
        if (k < len) {
          const int i = ell_pad(b - e0 + (int)k);
          col = s_c[i];
          val = s_v[i];
        }
        __stcs(eci + row + pitch * k, col);
        __stcs(ev + row + pitch * k, val);
      }
    }
    __syncthreads();
  }
}

template <typename T>
int launch_ell_fill(const mgb_coo* src, const int32_t* start, mgb_ell* e, int64_t W, cudaStream_t s) {
  if (e->pitch * e->width == 0) return MGB_SUCCESS;
  // as many rows as keep the mean tile at 5/8 of the staging (rows of unequal length: most tiles fit)
  const int64_t mean = src->nnz / std::max<int64_t>(1, src->nrows) + 1;
  int R = ELL_TILE_ROWS;
  while (R > 32 && R * mean > ELL_TILE * 5 / 8) R >>= 1;
  const int64_t resident = (int64_t)num_sms() * 8;
  const unsigned tiles = blocks_for((e->pitch + R - 1) / R, 1, resident);
  // segments of whole staging blocks (multiples of ELL_SEGMENT, as ELL_TILE / R divides it), about one wave of CTAs
  const int64_t parts = std::max<int64_t>(1, std::min(resident / tiles, e->width / ELL_SEGMENT));
  const int64_t segment = ((e->width + parts - 1) / parts + ELL_SEGMENT - 1) / ELL_SEGMENT * ELL_SEGMENT;
  const dim3 grid(tiles, (unsigned)((e->width + segment - 1) / segment));
  ell_fill_tiles<T><<<grid, 256, 0, s>>>(src->column_indices, static_cast<const T*>(src->values), start, src->nrows,
                                         e->pitch, e->width, W, e->column_indices, static_cast<T*>(e->values), R,
                                         segment);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

// HYB's COO part of row-sorted entries: excess[r] = the row's entries past
// the ELL width; with their exclusive scan, one warp per 32 rows copies the
// rows that have some.  Rows with HUGE_ROW of them or more, where the index pass
// saw such a row, are listed in pieces, and a CTA copies each piece (1e6 short
// rows and one of 500,000: the conversion 8,180 us with a warp per row, 330).
constexpr int EXCESS_PIECE = 2048;
__global__ void row_excess(const int32_t* __restrict__ start, int64_t nrows, int64_t W, int32_t* excess) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * blockDim.x)
    excess[r] = (int32_t)max((int64_t)(start[r + 1] - start[r]) - W, (int64_t)0);
}
template <typename T>
__global__ void __launch_bounds__(256)
copy_excess(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
            const int32_t* __restrict__ base, int64_t nrows, int64_t W, int32_t* __restrict__ orow,
            int32_t* __restrict__ ocol, T* __restrict__ oval, int2* __restrict__ pieces, int32_t* npieces) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * 8;
  for (int64_t r0 = ((int64_t)blockIdx.x * 8 + (threadIdx.x >> 5)) * 32; r0 < nrows; r0 += warps * 32) {
    const int64_t r = r0 + lane;
    int32_t from = 0, n = 0, to = 0;
    if (r < nrows) {
      from = (int32_t)min((int64_t)start[r] + W, (int64_t)INT32_MAX);
      n = max(start[r + 1] - from, 0);
      to = base[r];
    }
    for (unsigned m = __ballot_sync(0xffffffffu, n > 0); m; m &= m - 1) {
      const int j = __ffs(m) - 1;
      const int32_t f = __shfl_sync(0xffffffffu, from, j), k = __shfl_sync(0xffffffffu, n, j);
      const int32_t o = __shfl_sync(0xffffffffu, to, j);
      if (k >= prim::HUGE_ROW && pieces != nullptr) {
        const int32_t np = (int32_t)(((int64_t)k + EXCESS_PIECE - 1) / EXCESS_PIECE);
        int32_t at = 0;
        if (lane == 0) at = atomicAdd(npieces, np);
        at = __shfl_sync(0xffffffffu, at, 0);
        for (int32_t i = lane; i < np; i += 32) pieces[at + i] = make_int2((int32_t)(r0 + j), i);
        continue;
      }
#pragma unroll 4
      for (int32_t i = lane; i < k; i += 32) {
        orow[o + i] = (int32_t)(r0 + j);
        ocol[o + i] = c[f + i];
        oval[o + i] = v[f + i];
      }
    }
  }
}
template <typename T>
__global__ void __launch_bounds__(256)
copy_excess_pieces(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
                   const int32_t* __restrict__ base, int64_t W, int32_t* __restrict__ orow, int32_t* __restrict__ ocol,
                   T* __restrict__ oval, const int2* __restrict__ pieces, const int32_t* __restrict__ npieces) {
  for (int32_t p = blockIdx.x; p < *npieces; p += gridDim.x) {
    const int2 piece = pieces[p];
    const int64_t skip = (int64_t)piece.y * EXCESS_PIECE;
    const int64_t f = start[piece.x] + W + skip, o = base[piece.x] + skip;
    const int n = (int)min((int64_t)EXCESS_PIECE, start[piece.x + 1] - f);
    for (int i = threadIdx.x; i < n; i += 256) {
      orow[o + i] = piece.x;
      ocol[o + i] = c[f + i];
      oval[o + i] = v[f + i];
    }
  }
}

// The longest row and, for width > 0, the entries that a width-W ELL part
// holds (sum of min(length, width)), over row starts or a row histogram.
struct RowsFromStart {
  const int32_t* p;
  __device__ int operator()(int64_t r) const { return p[r + 1] - p[r]; }
};
struct RowsFromCounts {
  const int32_t* p;
  __device__ int operator()(int64_t r) const { return p[r]; }
};
template <typename LEN>
__global__ void __launch_bounds__(256) row_sizes(LEN len, int64_t nrows, int64_t width, Words* d) {
  __shared__ int64_t s_sum[8];
  __shared__ int32_t s_max[8];
  int64_t sum = 0;
  int32_t mx = 0;
  for (int64_t r = (int64_t)blockIdx.x * 256 + threadIdx.x; r < nrows; r += (int64_t)gridDim.x * 256) {
    const int32_t n = len(r);
    mx = max(mx, n);
    sum += min((int64_t)n, width);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = sum;
    s_max[threadIdx.x >> 5] = mx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; i++) {
      sum += s_sum[i];
      mx = max(mx, s_max[i]);
    }
    atomicAdd(reinterpret_cast<unsigned long long*>(&d->total), (unsigned long long)sum);
    atomicMax(&d->maxv, mx);
  }
}

// COO -> ELL / HYB sizes: one pass over the indices (ranges, order, row
// starts) and one over the rows; one host read.  A COO whose rows are not
// sorted has no row starts: its row histogram and a second read follow.
struct RowPlan {
  const int32_t* start = nullptr;
  Words h{};
};
int row_plan(const mgb_coo* src, const int32_t* ro, int64_t width, RowPlan* p, Scratch& sc, cudaStream_t s) {
  const int64_t N = src->nrows;
  Words* dw;
  int st = words_alloc(sc, &dw, s);
  if (st) return st;
  const unsigned grid = blocks_for(N, 256, (int64_t)num_sms() * 8);
  IndexPass pass;
  st = pass_and_sizes(src, ro, true, true, dw, nullptr, &pass, &p->h, sc, s, [&] {
    row_sizes<<<grid, 256, 0, s>>>(RowsFromStart{pass.start}, N, width, dw);
    MGB_LAUNCH_CHECK();
    return (int)MGB_SUCCESS;
  });
  if (st) return st;
  p->start = pass.start;
  if (!words_valid(p->h)) return MGB_ERR_INVALID_INPUT;
  if (words_rows_sorted(p->h)) return MGB_SUCCESS;
  const int32_t seen = p->h.seen;
  MGB_CUDA_CHECK(cudaMemsetAsync(dw, 0, sizeof(Words), s));
  int32_t* counts;
  MGB_SCRATCH(sc, counts, N);
  st = prim::histogram(src->row_indices, src->nnz, counts, N, s);
  if (st) return st;
  row_sizes<<<grid, 256, 0, s>>>(RowsFromCounts{counts}, N, width, dw);
  MGB_LAUNCH_CHECK();
  st = words_read(dw, &p->h, s);
  p->h.seen = seen;
  return st;
}

// Sizes of a COO's ELL form; h.maxv is the ELL width.
int ell_plan(const mgb_coo* src, const int32_t* ro, RowPlan* p, Scratch& sc, cudaStream_t s) {
  int st = ro ? MGB_SUCCESS : check_coo_args(src);
  if (st) return st;
  if (src->nrows == 0) return src->nnz > 0 ? MGB_ERR_INVALID_INPUT : MGB_SUCCESS;  // every row out of range
  st = row_plan(src, ro, 0, p, sc, s);
  if (st) return st;
  p->h.maxv = std::max(p->h.maxv, 0);
  if (exceeds_tolerance(src->nrows, src->nnz, p->h.maxv)) return MGB_ERR_FORMAT_CONVERSION;
  return MGB_SUCCESS;
}

int coo_to_ell_plan(const mgb_coo* src, int64_t* epr, cudaStream_t s) {
  MGB_REQUIRE(epr != nullptr, MGB_ERR_BAD_ARGUMENT);
  *epr = 0;
  Scratch sc(s);
  RowPlan p;
  const int st = ell_plan(src, nullptr, &p, sc, s);
  if (st == MGB_SUCCESS || st == MGB_ERR_FORMAT_CONVERSION) *epr = p.h.maxv;
  return st;
}

template <typename T>
int ell_fill(const mgb_coo* src, const RowPlan& p, mgb_ell* dst, cudaStream_t s) {
  const int64_t W = p.h.maxv;
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(dst->nrows == src->nrows && dst->ncols == src->ncols && dst->nnz == src->nnz &&
                  dst->entries_per_row == W && dst->width >= W && dst->pitch >= src->nrows,
              MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(dst->width * dst->pitch == 0 || (dst->column_indices && dst->values), MGB_ERR_BAD_ARGUMENT);
  if (src->nrows == 0) return MGB_SUCCESS;
  if (words_rows_sorted(p.h)) return launch_ell_fill<T>(src, p.start, dst, W, s);
  Scratch sc(s);
  int32_t* slot;
  MGB_SCRATCH(sc, slot, src->nnz);
  if (int st = compute_slots(src, slot, sc, s)) return st;
  return place_ell<T>(src, dst, W, slot, nullptr, sc, s);
}

template <typename T>
int coo_to_ell(const mgb_coo* src, mgb_ell* dst, cudaStream_t s) {
  Scratch sc(s);
  RowPlan p;
  const int st = ell_plan(src, nullptr, &p, sc, s);
  return st ? st : ell_fill<T>(src, p, dst, s);
}

// impl/Hyb/Serial/Morpheus_Convert_Impl.hpp:110-151 (width = max(1, nnz/nrows)
// unless the caller passes one)
int hyb_plan(const mgb_coo* src, const int32_t* ro, int64_t width, int64_t* W, RowPlan* p, Scratch& sc,
             cudaStream_t s) {
  MGB_REQUIRE(width >= 0, MGB_ERR_BAD_ARGUMENT);
  int st = ro ? MGB_SUCCESS : check_coo_args(src);
  if (st) return st;
  MGB_REQUIRE(src->nrows > 0, MGB_ERR_INVALID_INPUT);  // the reference divides by nrows
  *W = width > 0 ? width : std::max<int64_t>(1, src->nnz / src->nrows);
  st = row_plan(src, ro, *W, p, sc, s);
  if (st) return st;
  if (exceeds_tolerance(src->nrows, p->h.total, *W)) return MGB_ERR_FORMAT_CONVERSION;
  return MGB_SUCCESS;
}

int coo_to_hyb_plan(const mgb_coo* src, int64_t width, int64_t* epr, int64_t* ell_nnz, int64_t* coo_nnz,
                    cudaStream_t s) {
  MGB_REQUIRE(epr && ell_nnz && coo_nnz && width >= 0, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  RowPlan p;
  int64_t W = 0;
  const int st = hyb_plan(src, nullptr, width, &W, &p, sc, s);
  if (st == MGB_SUCCESS || st == MGB_ERR_FORMAT_CONVERSION) {
    *epr = W;
    *ell_nnz = p.h.total;
    *coo_nnz = src->nnz - p.h.total;
  }
  return st;
}

template <typename T>
int hyb_fill(const mgb_coo* src, const RowPlan& p, int64_t W, mgb_hyb* dst, cudaStream_t s) {
  Scratch sc(s);
  int st;
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  const int64_t en = p.h.total, cn = src->nnz - p.h.total;
  mgb_ell* e = &dst->ell;
  mgb_coo* c = &dst->coo;
  MGB_REQUIRE(e->nrows == src->nrows && e->ncols == src->ncols && e->nnz == en && e->entries_per_row == W &&
                  e->width >= W && e->pitch >= src->nrows,
              MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(c->nrows == src->nrows && c->ncols == src->ncols && c->nnz == cn, MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(e->width * e->pitch == 0 || (e->column_indices && e->values), MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(cn == 0 || (c->row_indices && c->column_indices && c->values), MGB_ERR_BAD_ARGUMENT);
  const int64_t n = src->nnz;
  if (words_rows_sorted(p.h)) {
    st = launch_ell_fill<T>(src, p.start, e, W, s);
    if (st || cn == 0) return st;
    int32_t *excess, *base;
    MGB_SCRATCH(sc, excess, src->nrows);
    MGB_SCRATCH(sc, base, src->nrows);
    row_excess<<<grid_for(src->nrows), 256, 0, s>>>(p.start, src->nrows, W, excess);
    MGB_LAUNCH_CHECK();
    st = prim::exclusive_scan<int32_t, int32_t>(excess, base, src->nrows, s);
    if (st) return st;
    const bool longs = (p.h.seen & prim::COO_HUGE_ROW) && cn >= prim::HUGE_ROW;
    int2* pieces = nullptr;
    int32_t* npieces = nullptr;
    if (longs) {
      MGB_SCRATCH(sc, npieces, 1);
      MGB_SCRATCH(sc, pieces, 2 * (cn / EXCESS_PIECE) + 1);  // listed rows' pieces are more than half full
      MGB_CUDA_CHECK(cudaMemsetAsync(npieces, 0, sizeof(int32_t), s));
    }
    const T* v = static_cast<const T*>(src->values);
    T* ov = static_cast<T*>(c->values);
    copy_excess<T><<<grid_for(src->nrows), 256, 0, s>>>(src->column_indices, v, p.start, base, src->nrows, W,
                                                        c->row_indices, c->column_indices, ov, pieces, npieces);
    MGB_LAUNCH_CHECK();
    if (!longs) return MGB_SUCCESS;
    copy_excess_pieces<T><<<blocks_for(cn, EXCESS_PIECE, (int64_t)num_sms() * 8), 256, 0, s>>>(
        src->column_indices, v, p.start, base, W, c->row_indices, c->column_indices, ov, pieces, npieces);
    MGB_LAUNCH_CHECK();
    return MGB_SUCCESS;
  }
  st = zero_coo<T>(c, s);
  if (st) return st;
  int32_t* slot;
  uint8_t* to_coo;
  MGB_SCRATCH(sc, slot, n);
  MGB_SCRATCH(sc, to_coo, n);
  st = compute_slots(src, slot, sc, s);
  if (st) return st;
  st = place_ell<T>(src, e, W, slot, to_coo, sc, s);
  if (st || n == 0) return st;
  int64_t* pos;
  MGB_SCRATCH(sc, pos, n);
  st = prim::exclusive_scan<uint8_t, int64_t>(to_coo, pos, n, s);
  if (st) return st;
  coo_part_scatter<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices,
                                                  static_cast<const T*>(src->values), to_coo, pos, n, cn,
                                                  c->row_indices, c->column_indices, static_cast<T*>(c->values));
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

template <typename T>
int coo_to_hyb(const mgb_coo* src, mgb_hyb* dst, cudaStream_t s) {
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  RowPlan p;
  int64_t W = 0;
  const int st = hyb_plan(src, nullptr, dst->ell.entries_per_row, &W, &p, sc, s);
  return st ? st : hyb_fill<T>(src, p, W, dst, s);
}

// ---------------------------------------------------------------- HDC -> COO
// impl/Hdc/Serial/Morpheus_Convert_Impl.hpp:64-130
template <typename T>
int hdc_to_coo(const mgb_hdc* src, mgb_coo* dst, cudaStream_t s) {
  MGB_REQUIRE(src != nullptr, MGB_ERR_BAD_ARGUMENT);
  int st = check_dia(&src->dia);
  if (st) return st;
  const mgb_csr* c = &src->csr;
  MGB_REQUIRE(c->nnz >= 0 && c->row_offsets != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(c->nnz == 0 || (c->column_indices && c->values), MGB_ERR_BAD_ARGUMENT);
  const int64_t nnz = src->dia.nnz + c->nnz;
  st = check_coo_dst(dst, src->dia.nrows, src->dia.ncols, nnz);
  if (st || nnz == 0) return st;
  st = zero_coo<T>(dst, s);
  if (st) return st;
  int64_t found = 0;
  st = dia_part_to_coo<T>(&src->dia, dst, nnz, &found, s);
  if (st) return st;
  MGB_REQUIRE(found + c->nnz <= nnz, MGB_ERR_RUNTIME);
  if (c->nnz > 0) {
    expand_rows<<<grid_for(c->nrows), 256, 0, s>>>(c->row_offsets, c->nrows, c->nnz, dst->row_indices, found);
    MGB_LAUNCH_CHECK();
    MGB_CUDA_CHECK(cudaMemcpyAsync(dst->column_indices + found, c->column_indices, sizeof(int32_t) * c->nnz,
                                   cudaMemcpyDeviceToDevice, s));
    MGB_CUDA_CHECK(cudaMemcpyAsync(static_cast<T*>(dst->values) + found, c->values, sizeof(T) * c->nnz,
                                   cudaMemcpyDeviceToDevice, s));
  }
  return sort_if_unsorted<T>(dst, s);
}

// ---------------------------------------------------------------- COO -> HDC
// impl/Hdc/Serial/Morpheus_Convert_Impl.hpp:132-226
// first matching stored offset (the reference's break on the first match)
__global__ void hdc_classify(const int32_t* __restrict__ r, const int32_t* __restrict__ c, int64_t n,
                             const int32_t* __restrict__ offs, int64_t nd, int32_t* dslot, uint8_t* is_csr) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t d = c[i] - r[i];
    int64_t lo = 0, hi = nd;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (offs[mid] < d) lo = mid + 1; else hi = mid;
    }
    const bool hit = lo < nd && offs[lo] == d;
    dslot[i] = hit ? (int32_t)lo : -1;
    is_csr[i] = hit ? 0 : 1;
  }
}

template <typename T>
__global__ void hdc_dia_place(const int32_t* __restrict__ r, const T* __restrict__ v, const int32_t* __restrict__ dslot,
                              int64_t n, int64_t pitch, T* vals, int32_t* owner, int pass) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    if (dslot[i] < 0) continue;
    const int64_t at = r[i] + pitch * (int64_t)dslot[i];
    if (owner == nullptr) vals[at] = v[i];
    else if (pass == 0) atomicMax(owner + at, (int32_t)i);
    else if (owner[at] == (int32_t)i) vals[at] = v[i];
  }
}

// CSR remainder of row-sorted entries: base = the exclusive scan of the rows'
// remainders.  Entries are row-sorted, so those of 32 rows that lie on no
// stored diagonal go, in order, to the consecutive places from base[first
// row] on: one warp per 32 rows, ranks by ballot.  Long rows are left in pieces
// to hdc_remainder_pieces.
template <typename T, bool LONGS>
__global__ void __launch_bounds__(256)
hdc_remainder(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
              const int32_t* __restrict__ base, int64_t nrows, int nd, const int32_t* __restrict__ offs,
              const int32_t* __restrict__ bin_slot, int64_t limit, int32_t* __restrict__ ocol,
              T* __restrict__ oval, prim::RowPieces pieces) {
  __shared__ int2 h_table[DIA_HASH_SLOTS];
  __shared__ prim::WarpRows s_rows[8];
  const DiaTable table{h_table};
  const bool hashed = nd <= DIA_HASH_DIAGS;
  if (hashed) dia_table_clear(table);
  __syncthreads();
  if (hashed) dia_table_fill(table, offs, nd);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int64_t r0 = ((int64_t)blockIdx.x * 8 + w) * 32; r0 < nrows; r0 += (int64_t)gridDim.x * 256) {
    int64_t to = base[r0];
    if (to == base[min(r0 + 32, nrows)]) continue;  // every entry on a stored diagonal
    auto place = [&](bool in, int q, int64_t e, int32_t col) {
      const int32_t d = col - (int32_t)(r0 + q);
      const bool miss = in && (hashed ? dia_table_find(table, d) : bin_slot[(int64_t)d + nrows - 1]) < 0;
      const unsigned m = __ballot_sync(0xffffffffu, miss);
      const int64_t p = to + __popc(m & ((1u << lane) - 1));
      if (miss && p < limit) {
        ocol[p] = col;
        oval[p] = v[e];
      }
      to += __popc(m);
    };
    if (LONGS && prim::long_group(start, r0, nrows) &&
        prim::warp_rows_apart(start, r0, nrows, pieces, lane, [&](bool in, int q, int32_t e, int32_t first) {
          if (e - lane == first) to = base[r0 + q];
          place(in, q, e, in ? __ldcs(c + e) : (int32_t)(r0 + q));
        }))
      continue;
    prim::warp_row_walk(
        start, r0, nrows, s_rows[w], lane, 0, 1, [&](int64_t c0, int i) { return __ldcs(c + c0 + i); },
        [&](bool in, bool, int q, int64_t c0, int i, int32_t col) { place(in, q, c0 + i, col); });
  }
}

// A CTA per piece of a long row.  The row's entries before the piece that lie on
// a stored diagonal are counted by searching for every diagonal's column below
// the piece's first one; within the piece, a warp per 256 entries.
template <typename T>
__global__ void __launch_bounds__(256)
hdc_remainder_pieces(const int32_t* __restrict__ c, const T* __restrict__ v, const int32_t* __restrict__ start,
                     const int32_t* __restrict__ base, int64_t nrows, int nd, const int32_t* __restrict__ offs,
                     const int32_t* __restrict__ bin_slot, int64_t limit, int32_t* __restrict__ ocol,
                     T* __restrict__ oval, prim::RowPieces pieces) {
  constexpr int PER_WARP = prim::ROW_PIECE / 8, STEPS = PER_WARP / 32;
  __shared__ int2 h_table[DIA_HASH_SLOTS];
  __shared__ int s_hits[8], s_misses[8];
  const DiaTable table{h_table};
  const bool hashed = nd <= DIA_HASH_DIAGS;
  if (hashed) dia_table_clear(table);
  __syncthreads();
  if (hashed) dia_table_fill(table, offs, nd);
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t n = min((int64_t)*pieces.count, pieces.limit);
  for (int64_t piece = blockIdx.x; piece < n; piece += gridDim.x) {
    const int32_t row = pieces.list[piece].x;
    if (row < 0) continue;
    const int64_t b = start[row], e = start[row + 1], e0 = b + (int64_t)pieces.list[piece].y * prim::ROW_PIECE;
    const int64_t first = __ldg(c + e0);
    int hits = 0;
    for (int d = threadIdx.x; d < nd; d += 256) {
      const int64_t col = (int64_t)row + offs[d];
      if (col >= first) continue;
      const int64_t at = lower_column(c, b, e0, col);
      hits += at < e0 && c[at] == col;
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    const int64_t w0 = e0 + (int64_t)w * PER_WARP;
    int32_t col[STEPS];
    unsigned miss[STEPS];
    int misses = 0;
#pragma unroll
    for (int k = 0; k < STEPS; k++) {
      const int64_t at = w0 + 32 * k + lane;
      col[k] = at < e ? __ldg(c + at) : row;
      const int32_t d = col[k] - row;
      const bool out = at < e && (hashed ? dia_table_find(table, d) : bin_slot[(int64_t)d + nrows - 1]) < 0;
      miss[k] = __ballot_sync(0xffffffffu, out);
      misses += __popc(miss[k]);
    }
    if (lane == 0) {
      s_hits[w] = hits;
      s_misses[w] = misses;
    }
    __syncthreads();
    int64_t to = base[row] + (e0 - b);
    for (int i = 0; i < 8; i++) to += (i < w ? s_misses[i] : 0) - s_hits[i];
#pragma unroll
    for (int k = 0; k < STEPS; k++) {
      const int64_t p = to + __popc(miss[k] & ((1u << lane) - 1));
      if (((miss[k] >> lane) & 1) && p < limit) {
        ocol[p] = col[k];
        oval[p] = v[w0 + 32 * k + lane];
      }
      to += __popc(miss[k]);
    }
    __syncthreads();  // the next piece's counts
  }
}

// COO -> HDC sizes: one pass over the indices as for DIA, then the true
// diagonals (>= floor(0.2 N) entries) and their entry count; one host read.
struct HdcPlan {
  int32_t* counts = nullptr;
  const int32_t* start = nullptr;
  int64_t* sums = nullptr;
  int32_t min_elem = 0;
  Words h{};
};
int32_t hdc_min_elem(const mgb_coo* src) {
  return (int32_t)((double)src->nrows * 0.2);  // HdcMatrix::true_diagonal_ratio
}
int hdc_plan(const mgb_coo* src, const int32_t* ro, bool starts, HdcPlan* p, Scratch& sc, cudaStream_t s) {
  int st = ro ? MGB_SUCCESS : check_coo_args(src);
  if (st) return st;
  MGB_REQUIRE(src->nrows > 0 && src->ncols > 0, MGB_ERR_INVALID_INPUT);
  const int64_t nb = src->nrows + src->ncols - 1;
  p->min_elem = hdc_min_elem(src);
  Words* dw;
  st = words_alloc(sc, &dw, s);
  if (st) return st;
  MGB_SCRATCH(sc, p->counts, nb);
  MGB_SCRATCH(sc, p->sums, prim::bin_tiles(nb));
  IndexPass pass;
  st = pass_and_sizes(src, ro, starts, true, dw, p->counts, &pass, &p->h, sc, s, [&] {
    return prim::select_bins(p->counts, nb, p->min_elem, p->sums, &dw->total, &dw->total2, s);
  });
  if (st) return st;
  p->start = pass.start;
  if (!words_valid(p->h)) return MGB_ERR_INVALID_INPUT;
  if (exceeds_tolerance(src->nrows, p->h.total2, p->h.total)) return MGB_ERR_FORMAT_CONVERSION;
  return MGB_SUCCESS;
}

int coo_to_hdc_plan(const mgb_coo* src, int64_t* ndiags, int64_t* dia_nnz, int64_t* csr_nnz, cudaStream_t s) {
  MGB_REQUIRE(ndiags && dia_nnz && csr_nnz, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  HdcPlan p;
  const int st = hdc_plan(src, nullptr, false, &p, sc, s);
  if (st == MGB_SUCCESS || st == MGB_ERR_FORMAT_CONVERSION) {
    *ndiags = p.h.total;
    *dia_nnz = p.h.total2;
    *csr_nnz = src->nnz - p.h.total2;
  }
  return st;
}

template <typename T>
int hdc_fill(const mgb_coo* src, const HdcPlan& p, mgb_hdc* dst, cudaStream_t s) {
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  int st;
  const int64_t nd = p.h.total, dn = p.h.total2, cn = src->nnz - p.h.total2;
  mgb_dia* D = &dst->dia;
  mgb_csr* C = &dst->csr;
  MGB_REQUIRE(D->nrows == src->nrows && D->ncols == src->ncols && D->nnz == dn && D->ndiags == nd &&
                  D->pitch >= src->nrows,
              MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(C->nrows == src->nrows && C->ncols == src->ncols && C->nnz == cn, MGB_ERR_INVALID_INPUT);
  MGB_REQUIRE(C->row_offsets && (nd == 0 || (D->diagonal_offsets && D->values)), MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(cn == 0 || (C->column_indices && C->values), MGB_ERR_BAD_ARGUMENT);
  const int64_t n = src->nnz, N = src->nrows, nb = src->nrows + src->ncols - 1;
  if (nd > 0) {
    // the midpoint bin is recorded as offset 0 (exact only for square matrices)
    st = prim::select_bins_apply(p.counts, nb, p.min_elem, p.sums, N, nb / 2, D->diagonal_offsets, s);
    if (st) return st;
    // std::sort of the stored offsets (impl/Hdc/Serial/Morpheus_Convert_Impl.hpp:193-195):
    // they are in order already unless the midpoint bin is not offset 0
    if (src->nrows != src->ncols) {
      std::vector<int32_t> h((size_t)nd);
      MGB_CUDA_CHECK(cudaMemcpyAsync(h.data(), D->diagonal_offsets, sizeof(int32_t) * nd, cudaMemcpyDeviceToHost, s));
      MGB_CUDA_CHECK(cudaStreamSynchronize(s));
      std::sort(h.begin(), h.end());
      MGB_CUDA_CHECK(cudaMemcpyAsync(D->diagonal_offsets, h.data(), sizeof(int32_t) * nd, cudaMemcpyHostToDevice, s));
      MGB_CUDA_CHECK(cudaStreamSynchronize(s));  // h lives on this stack frame
    }
  }
  if (n == 0) {
    if (nd > 0) MGB_CUDA_CHECK(cudaMemsetAsync(D->values, 0, sizeof(T) * D->pitch * nd, s));
    MGB_CUDA_CHECK(cudaMemsetAsync(C->row_offsets, 0, sizeof(int32_t) * (N + 1), s));
    return MGB_SUCCESS;
  }
  const T* v = static_cast<const T*>(src->values);
  // A square matrix's bins are its offsets, so the entries off the true
  // diagonals are exactly the cn counted ones; the midpoint bin of another
  // shape is not (below).
  if (src->nrows == src->ncols && words_distinct(p.h)) {
    if (nd == 0) {
      MGB_CUDA_CHECK(cudaMemcpyAsync(C->row_offsets, p.start, sizeof(int32_t) * (N + 1), cudaMemcpyDeviceToDevice, s));
      MGB_CUDA_CHECK(cudaMemcpyAsync(C->column_indices, src->column_indices, sizeof(int32_t) * n,
                                     cudaMemcpyDeviceToDevice, s));
      MGB_CUDA_CHECK(cudaMemcpyAsync(C->values, v, sizeof(T) * n, cudaMemcpyDeviceToDevice, s));
      return MGB_SUCCESS;
    }
    if (hdc_tiled<T>(nd)) {
      // rows that one warp has too much with: 32 of less than HUGE_ROW do as little as the mean allows
      const bool longs = (p.h.seen & prim::COO_HUGE_ROW) || n / N > prim::LONG_GROUP / 32;
      int32_t* rem;
      MGB_SCRATCH(sc, rem, N + 1);
      MGB_CUDA_CHECK(cudaMemsetAsync(rem + N, 0, sizeof(int32_t), s));
      st = launch_dia_fill<T>(src, p.start, D->pitch, nd, D->diagonal_offsets, p.counts, static_cast<T*>(D->values),
                              rem, longs, s);
      if (st) return st;
      st = prim::exclusive_scan<int32_t, int32_t>(rem, C->row_offsets, N + 1, s);
      if (st || cn == 0) return st;
      prim::RowPieces pieces{nullptr, nullptr, prim::max_row_pieces(n)};
      if (longs)
        if (int e = prim::row_pieces_alloc(&pieces, sc, s)) return e;
      const auto run = [&](auto kernel) {
        kernel<<<blocks_for(N, 256, (int64_t)num_sms() * 8), 256, 0, s>>>(
            src->column_indices, v, p.start, C->row_offsets, N, (int)nd, D->diagonal_offsets, p.counts, cn,
            C->column_indices, static_cast<T*>(C->values), pieces);
      };
      if (longs) run(hdc_remainder<T, true>);
      else run(hdc_remainder<T, false>);
      MGB_LAUNCH_CHECK();
      if (!longs) return MGB_SUCCESS;
      hdc_remainder_pieces<T><<<blocks_for(pieces.limit, 1, (int64_t)num_sms() * 8), 256, 0, s>>>(
          src->column_indices, v, p.start, C->row_offsets, N, (int)nd, D->diagonal_offsets, p.counts, cn,
          C->column_indices, static_cast<T*>(C->values), pieces);
      MGB_LAUNCH_CHECK();
      return MGB_SUCCESS;
    }
  }
  if (nd > 0) MGB_CUDA_CHECK(cudaMemsetAsync(D->values, 0, sizeof(T) * D->pitch * nd, s));
  int32_t* dslot;
  uint8_t* is_csr;
  int64_t *cpos, *d_csr;
  MGB_SCRATCH(sc, dslot, n);
  MGB_SCRATCH(sc, is_csr, n);
  MGB_SCRATCH(sc, cpos, n);
  MGB_SCRATCH(sc, d_csr, 1);
  hdc_classify<<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices, n, D->diagonal_offsets, nd, dslot,
                                           is_csr);
  MGB_LAUNCH_CHECK();
  st = prim::exclusive_scan<uint8_t, int64_t>(is_csr, cpos, n, s, d_csr);
  if (st) return st;
  // a non-square matrix with a true diagonal in the midpoint bin sends more
  // entries to CSR than were counted (the reference writes out of bounds):
  // the scatter below stops at cn, and the count is checked at the end
  if (nd > 0) {
    if (words_distinct(p.h)) {
      hdc_dia_place<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, v, dslot, n, D->pitch, static_cast<T*>(D->values),
                                                    nullptr, 0);
      MGB_LAUNCH_CHECK();
    } else {
      int32_t* owner;
      MGB_SCRATCH(sc, owner, D->pitch * nd);
      st = fill<int32_t>(owner, -1, D->pitch * nd, s);
      if (st) return st;
      for (int pass = 0; pass < 2; pass++) {
        hdc_dia_place<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, v, dslot, n, D->pitch,
                                                      static_cast<T*>(D->values), owner, pass);
        MGB_LAUNCH_CHECK();
      }
    }
  }
  // CSR part: entries in COO order (csr_entries counter of the reference),
  // row_offsets = exclusive scan of per-row counts, last = csr_nnz
  int32_t *rows_c, *counts_c;
  MGB_SCRATCH(sc, rows_c, cn > 0 ? cn : 1);
  MGB_SCRATCH(sc, counts_c, N + 1);
  if (cn > 0) {
    MGB_CUDA_CHECK(cudaMemsetAsync(C->column_indices, 0, sizeof(int32_t) * cn, s));
    MGB_CUDA_CHECK(cudaMemsetAsync(C->values, 0, sizeof(T) * cn, s));
    // slots the scatter leaves empty hold row N, which the histogram ignores
    st = fill<int32_t>(rows_c, (int32_t)N, cn, s);
    if (st) return st;
    coo_part_scatter<T><<<grid_for(n), 256, 0, s>>>(src->row_indices, src->column_indices, v, is_csr, cpos, n, cn,
                                                    rows_c, C->column_indices, static_cast<T*>(C->values));
    MGB_LAUNCH_CHECK();
  }
  st = prim::histogram(rows_c, cn, counts_c, N, s);
  if (st) return st;
  MGB_CUDA_CHECK(cudaMemsetAsync(counts_c + N, 0, sizeof(int32_t), s));
  st = prim::exclusive_scan<int32_t, int32_t>(counts_c, C->row_offsets, N + 1, s);
  if (st) return st;
  const int32_t last = (int32_t)cn;
  int64_t ncsr = 0;
  MGB_CUDA_CHECK(cudaMemcpyAsync(C->row_offsets + N, &last, sizeof(int32_t), cudaMemcpyHostToDevice, s));
  MGB_CUDA_CHECK(cudaMemcpyAsync(&ncsr, d_csr, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  MGB_CUDA_CHECK(cudaStreamSynchronize(s));  // 'last' and 'ncsr' live on this stack frame
  MGB_REQUIRE(ncsr <= cn, MGB_ERR_RUNTIME);
  return MGB_SUCCESS;
}

template <typename T>
int coo_to_hdc(const mgb_coo* src, mgb_hdc* dst, cudaStream_t s) {
  MGB_REQUIRE(dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s);
  HdcPlan p;
  const int st = hdc_plan(src, nullptr, true, &p, sc, s);
  return st ? st : hdc_fill<T>(src, p, dst, s);
}

// ------------------------------------------------- plan and fill, one pass
// mgb_convert_coo_plan leaves what the index pass found in the caller's
// workspace, and mgb_convert_coo_planned_* fills from there: the indices are
// read for the sizes once, where a *_plan call and its conversion each read
// them (260 us of 2,342 for the selector's switch of the 160^3 stencil), and
// nothing that size is allocated.  mgb_convert_csr_plan does the same for the
// entries of a CSR matrix, whose offsets take the place of the row starts: its
// row indices are neither made nor read.
enum { PLAN_CSR = 1, PLAN_DIA = 2, PLAN_ELL = 3, PLAN_HYB = 4, PLAN_HDC = 5 };  // formats_e

size_t plan_bytes(int64_t nrows, int64_t ncols, int64_t nnz, int format) {
  size_t b = Scratch::padded(sizeof(Words)) + Scratch::padded(sizeof(int32_t) * (size_t)(nrows + 1)) +
             Scratch::padded(sizeof(int32_t) * (size_t)prim::gap_words(nrows)) +
             Scratch::padded(sizeof(int2) * (size_t)prim::max_row_pieces(nnz));
  const int64_t nb = std::max<int64_t>(1, nrows + ncols - 1);
  if (format == PLAN_DIA || format == PLAN_HDC)
    b += Scratch::padded(sizeof(int32_t) * (size_t)nb) + Scratch::padded(sizeof(int64_t) * (size_t)prim::bin_tiles(nb));
  return b;
}

int coo_plan_bytes(const mgb_coo* src, int format, int64_t* bytes) {
  MGB_REQUIRE(bytes != nullptr && format >= PLAN_CSR && format <= PLAN_HDC, MGB_ERR_BAD_ARGUMENT);
  int st = check_coo_args(src, format != PLAN_CSR);
  if (st) return st;
  *bytes = (int64_t)plan_bytes(src->nrows, src->ncols, src->nnz, format);
  return MGB_SUCCESS;
}

enum { SOURCE_COO = 1, SOURCE_CSR = 2 };

// The plan was made of a source of this kind and of src's sizes.
bool plan_of(const mgb_coo_plan* plan, int64_t kind, const mgb_coo* src) {
  return plan->source[0] == kind && plan->source[1] == src->nrows && plan->source[2] == src->ncols &&
         plan->source[3] == src->nnz;
}

inline bool bad_workspace(const void* ws) { return reinterpret_cast<uintptr_t>(ws) % 256 != 0; }

// The common part: src's entries with, for a CSR matrix, its offsets.
int plan_any(const mgb_coo* src, const int32_t* ro, int format, int64_t hyb_width, void* ws, int64_t bytes,
             mgb_coo_plan* plan, cudaStream_t s) {
  MGB_REQUIRE(ws != nullptr && !bad_workspace(ws) && bytes >= (int64_t)plan_bytes(src->nrows, src->ncols, src->nnz, format),
              MGB_ERR_BAD_ARGUMENT);
  *plan = mgb_coo_plan{};
  plan->format = format;
  const int64_t made_of[4] = {ro ? SOURCE_CSR : SOURCE_COO, src->nrows, src->ncols, src->nnz};
  std::copy(made_of, made_of + 4, plan->source);
  Scratch sc(s, ws, (size_t)bytes);
  int st;
  if (format == PLAN_CSR) {
    CsrPlan p;
    st = csr_plan(src, &p, sc, s);
    plan->seen = p.h.seen;
    plan->parts[1] = p.start;
    if (!words_rows_sorted(p.h)) plan->fill_bytes = prim::row_sort_bytes(src->nnz, src->nrows);
  } else if (format == PLAN_DIA) {
    DiaPlan p;
    st = dia_plan(src, ro, true, &p, sc, s);
    plan->sizes[0] = p.h.total;
    plan->seen = p.h.seen;
    plan->parts[0] = p.counts, plan->parts[1] = const_cast<int32_t*>(p.start), plan->parts[2] = p.sums;
  } else if (format == PLAN_HDC) {
    HdcPlan p;
    st = hdc_plan(src, ro, true, &p, sc, s);
    plan->sizes[0] = p.h.total;
    plan->sizes[1] = p.h.total2;
    plan->sizes[2] = src->nnz - p.h.total2;
    plan->seen = p.h.seen;
    plan->parts[0] = p.counts, plan->parts[1] = const_cast<int32_t*>(p.start), plan->parts[2] = p.sums;
  } else {
    RowPlan p;
    int64_t W = 0;
    if (format == PLAN_ELL) {
      st = ell_plan(src, ro, &p, sc, s);
      plan->sizes[0] = p.h.maxv;
    } else {
      st = hyb_plan(src, ro, hyb_width, &W, &p, sc, s);
      plan->sizes[0] = W;
      plan->sizes[1] = p.h.total;
      plan->sizes[2] = src->nnz - p.h.total;
    }
    plan->seen = p.h.seen;
    plan->parts[1] = const_cast<int32_t*>(p.start);
  }
  return st;
}

int coo_plan(const mgb_coo* src, int format, int64_t hyb_width, void* ws, int64_t bytes, mgb_coo_plan* plan,
             cudaStream_t s) {
  MGB_REQUIRE(plan != nullptr && format >= PLAN_CSR && format <= PLAN_HDC, MGB_ERR_BAD_ARGUMENT);
  int st = check_coo_args(src, format != PLAN_CSR);
  if (st) return st;
  return plan_any(src, nullptr, format, hyb_width, ws, bytes, plan, s);
}

// src: the plan's source, or the entries of its CSR matrix.
template <typename T>
int fill_planned(const mgb_coo* src, const mgb_coo_plan* plan, void* dst, void* ws, int64_t bytes, cudaStream_t s) {
  auto* counts = static_cast<int32_t*>(plan->parts[0]);
  auto* start = static_cast<int32_t*>(plan->parts[1]);
  auto* sums = static_cast<int64_t*>(plan->parts[2]);
  Words h{};
  h.seen = plan->seen;
  h.total = plan->sizes[0];
  if (plan->format == PLAN_CSR) {
    MGB_REQUIRE(!bad_workspace(ws), MGB_ERR_BAD_ARGUMENT);
    Scratch sc(s, ws, (size_t)std::max<int64_t>(bytes, 0));
    CsrPlan p;
    p.start = start, p.h = h;
    return csr_fill<T>(src, p, static_cast<mgb_csr*>(dst), sc, s);
  }
  if (plan->format == PLAN_DIA) {
    DiaPlan p;
    p.counts = counts, p.start = start, p.sums = sums, p.h = h;
    return dia_fill<T>(src, p, static_cast<mgb_dia*>(dst), s);
  }
  if (plan->format == PLAN_HDC) {
    HdcPlan p;
    p.counts = counts, p.start = start, p.sums = sums, p.h = h;
    p.h.total2 = plan->sizes[1];
    p.min_elem = hdc_min_elem(src);
    return hdc_fill<T>(src, p, static_cast<mgb_hdc*>(dst), s);
  }
  RowPlan p;
  p.start = start, p.h = h;
  if (plan->format == PLAN_ELL) {
    p.h.maxv = (int32_t)plan->sizes[0];
    return ell_fill<T>(src, p, static_cast<mgb_ell*>(dst), s);
  }
  MGB_REQUIRE(plan->format == PLAN_HYB, MGB_ERR_BAD_ARGUMENT);
  p.h.total = plan->sizes[1];
  return hyb_fill<T>(src, p, plan->sizes[0], static_cast<mgb_hyb*>(dst), s);
}

template <typename T>
int coo_planned(const mgb_coo* src, const mgb_coo_plan* plan, void* dst, void* ws, int64_t bytes, cudaStream_t s) {
  MGB_REQUIRE(plan != nullptr && dst != nullptr, MGB_ERR_BAD_ARGUMENT);
  if (int st = check_coo_args(src, plan->format != PLAN_CSR)) return st;
  MGB_REQUIRE(plan_of(plan, SOURCE_COO, src), MGB_ERR_BAD_ARGUMENT);
  return fill_planned<T>(src, plan, dst, ws, bytes, s);
}

// The entries of a CSR matrix without row indices: every routine that fills
// from row starts takes them.
mgb_coo csr_entries(const mgb_csr* A) {
  return mgb_coo{A->nrows, A->ncols, A->nnz, nullptr, A->column_indices, A->values};
}

int csr_source_bytes(const mgb_csr* src, int format, int64_t* bytes) {
  MGB_REQUIRE(src != nullptr && bytes != nullptr && format >= PLAN_DIA && format <= PLAN_HDC, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(!bad_sizes(src->nrows, src->ncols, src->nnz), MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(src->nrows + src->ncols < INT32_MAX, MGB_ERR_INVALID_INPUT);
  *bytes = (int64_t)plan_bytes(src->nrows, src->ncols, src->nnz, format);
  return MGB_SUCCESS;
}

// format 0 in the plan: not a case for the fills from row starts (offsets that
// do not span the entries, columns out of order or repeated in a row, more
// diagonals than the tiles take, a HDC that is not square): the matrix goes
// through its COO form.
template <typename T>
bool csr_fillable(const mgb_csr* src, int format, const mgb_coo_plan& p) {
  if (p.seen & prim::COO_BAD_OFFSETS) return false;
  if (format == PLAN_ELL || format == PLAN_HYB) return true;
  Words h{};
  h.seen = p.seen;
  if (!words_distinct(h) || (format == PLAN_HDC && src->nrows != src->ncols)) return false;
  return p.sizes[0] == 0 || (format == PLAN_DIA ? dia_tiled(p.sizes[0]) : hdc_tiled<T>(p.sizes[0]));
}

template <typename T>
int csr_source_plan(const mgb_csr* src, int format, int64_t hyb_width, void* ws, int64_t bytes, mgb_coo_plan* plan,
                    cudaStream_t s) {
  int64_t need = 0;
  MGB_REQUIRE(plan != nullptr, MGB_ERR_BAD_ARGUMENT);
  int st = csr_source_bytes(src, format, &need);
  if (st) return st;
  *plan = mgb_coo_plan{};
  MGB_REQUIRE(src->row_offsets != nullptr && (src->nnz == 0 || (src->column_indices && src->values)),
              MGB_ERR_BAD_ARGUMENT);
  if (src->nrows == 0) return MGB_SUCCESS;  // format 0
  const mgb_coo e = csr_entries(src);
  st = plan_any(&e, src->row_offsets, format, hyb_width, ws, bytes, plan, s);
  if (plan->seen & prim::COO_BAD_OFFSETS) st = MGB_SUCCESS;
  if (st == MGB_SUCCESS && !csr_fillable<T>(src, format, *plan)) *plan = mgb_coo_plan{};
  return st;
}

template <typename T>
int csr_source_planned(const mgb_csr* src, const mgb_coo_plan* plan, void* dst, cudaStream_t s) {
  MGB_REQUIRE(src != nullptr && plan != nullptr && dst != nullptr && plan->format >= PLAN_DIA, MGB_ERR_BAD_ARGUMENT);
  const mgb_coo e = csr_entries(src);
  MGB_REQUIRE(src->row_offsets != nullptr && (src->nnz == 0 || (src->column_indices && src->values)),
              MGB_ERR_BAD_ARGUMENT);
  // the fills below read no row indices: only what csr_source_plan<T> lets through may come here
  MGB_REQUIRE(plan_of(plan, SOURCE_CSR, &e) && plan->parts[1] == src->row_offsets &&
                  csr_fillable<T>(src, plan->format, *plan),
              MGB_ERR_BAD_ARGUMENT);
  return fill_planned<T>(&e, plan, dst, nullptr, 0, s);
}

// ---------------------------------------------------------------- sort API
template <typename T>
int coo_sort(mgb_coo* A, void* ws, int64_t bytes, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr && A->nnz >= 0, MGB_ERR_BAD_ARGUMENT);
  if (A->nnz <= 1) return MGB_SUCCESS;
  MGB_REQUIRE(A->row_indices && A->column_indices && A->values, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(ws == nullptr || reinterpret_cast<uintptr_t>(ws) % 256 == 0, MGB_ERR_BAD_ARGUMENT);
  Scratch sc(s, ws, (size_t)std::max<int64_t>(bytes, 0));
  Words* dw;
  int st = words_alloc(sc, &dw, s);
  if (st) return st;
  st = prim::reduce_max_i32(A->row_indices, A->nnz, &dw->maxv, s);
  if (st) return st;
  // rows and columns must be >= 0 (the counting sort indexes by them)
  st = prim::coo_pass(A->row_indices, A->column_indices, A->nnz, INT32_MAX, INT32_MAX, dw, nullptr, nullptr, nullptr, false, s);
  if (st) return st;
  Words hw;
  st = words_read(dw, &hw, s);
  if (st) return st;
  if (!words_valid(hw)) return MGB_ERR_INVALID_INPUT;
  return sort_coo_inplace<T>(A->row_indices, A->column_indices, static_cast<T*>(A->values), A->nnz,
                             (int64_t)hw.maxv + 1, sc, s);
}

int coo_is_sorted(const mgb_coo* A, int* out, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr && out != nullptr && A->nnz >= 0, MGB_ERR_BAD_ARGUMENT);
  *out = 1;
  if (A->nnz <= 1) return MGB_SUCCESS;
  bool sorted = false;
  int st = sorted_and_dup(A->row_indices, A->column_indices, A->nnz, &sorted, nullptr, s);
  if (st) return st;
  *out = sorted ? 1 : 0;
  return MGB_SUCCESS;
}

}  // namespace
}  // namespace mgb

#define MGB_CONV_PAIR(NAME, SRC, DST)                                                            \
  int mgb_convert_##NAME##_f64(const SRC* src, DST* dst, void* stream) {                         \
    return mgb::NAME<double>(src, dst, mgb::as_stream(stream));                                  \
  }                                                                                              \
  int mgb_convert_##NAME##_f32(const SRC* src, DST* dst, void* stream) {                         \
    return mgb::NAME<float>(src, dst, mgb::as_stream(stream));                                   \
  }

extern "C" {

MGB_CONV_PAIR(csr_to_coo, mgb_csr, mgb_coo)
MGB_CONV_PAIR(coo_to_csr, mgb_coo, mgb_csr)
MGB_CONV_PAIR(dia_to_coo, mgb_dia, mgb_coo)
MGB_CONV_PAIR(coo_to_dia, mgb_coo, mgb_dia)
MGB_CONV_PAIR(ell_to_coo, mgb_ell, mgb_coo)
MGB_CONV_PAIR(coo_to_ell, mgb_coo, mgb_ell)
MGB_CONV_PAIR(hyb_to_coo, mgb_hyb, mgb_coo)
MGB_CONV_PAIR(coo_to_hyb, mgb_coo, mgb_hyb)
MGB_CONV_PAIR(hdc_to_coo, mgb_hdc, mgb_coo)
MGB_CONV_PAIR(coo_to_hdc, mgb_coo, mgb_hdc)

int mgb_convert_coo_to_dia_plan(const mgb_coo* src, int64_t* ndiags, void* stream) {
  return mgb::coo_to_dia_plan(src, ndiags, mgb::as_stream(stream));
}
int mgb_convert_coo_to_ell_plan(const mgb_coo* src, int64_t* entries_per_row, void* stream) {
  return mgb::coo_to_ell_plan(src, entries_per_row, mgb::as_stream(stream));
}
int mgb_convert_coo_to_hyb_plan(const mgb_coo* src, int64_t width, int64_t* entries_per_row, int64_t* ell_nnz,
                                int64_t* coo_nnz, void* stream) {
  return mgb::coo_to_hyb_plan(src, width, entries_per_row, ell_nnz, coo_nnz, mgb::as_stream(stream));
}
int mgb_convert_coo_to_hdc_plan(const mgb_coo* src, int64_t* ndiags, int64_t* dia_nnz, int64_t* csr_nnz,
                                void* stream) {
  return mgb::coo_to_hdc_plan(src, ndiags, dia_nnz, csr_nnz, mgb::as_stream(stream));
}
int mgb_convert_coo_workspace_bytes(const mgb_coo* src, int format, int64_t* bytes) {
  return mgb::coo_plan_bytes(src, format, bytes);
}
int mgb_convert_coo_plan(const mgb_coo* src, int format, int64_t hyb_width, void* workspace, int64_t bytes,
                         mgb_coo_plan* plan, void* stream) {
  return mgb::coo_plan(src, format, hyb_width, workspace, bytes, plan, mgb::as_stream(stream));
}
int mgb_convert_coo_planned_f64(const mgb_coo* src, const mgb_coo_plan* plan, void* dst, void* workspace,
                                int64_t bytes, void* stream) {
  return mgb::coo_planned<double>(src, plan, dst, workspace, bytes, mgb::as_stream(stream));
}
int mgb_convert_coo_planned_f32(const mgb_coo* src, const mgb_coo_plan* plan, void* dst, void* workspace,
                                int64_t bytes, void* stream) {
  return mgb::coo_planned<float>(src, plan, dst, workspace, bytes, mgb::as_stream(stream));
}
int mgb_convert_csr_workspace_bytes(const mgb_csr* src, int format, int64_t* bytes) {
  return mgb::csr_source_bytes(src, format, bytes);
}
int mgb_convert_csr_plan_f64(const mgb_csr* src, int format, int64_t hyb_width, void* workspace, int64_t bytes,
                             mgb_coo_plan* plan, void* stream) {
  return mgb::csr_source_plan<double>(src, format, hyb_width, workspace, bytes, plan, mgb::as_stream(stream));
}
int mgb_convert_csr_plan_f32(const mgb_csr* src, int format, int64_t hyb_width, void* workspace, int64_t bytes,
                             mgb_coo_plan* plan, void* stream) {
  return mgb::csr_source_plan<float>(src, format, hyb_width, workspace, bytes, plan, mgb::as_stream(stream));
}
int mgb_convert_csr_planned_f64(const mgb_csr* src, const mgb_coo_plan* plan, void* dst, void* stream) {
  return mgb::csr_source_planned<double>(src, plan, dst, mgb::as_stream(stream));
}
int mgb_convert_csr_planned_f32(const mgb_csr* src, const mgb_coo_plan* plan, void* dst, void* stream) {
  return mgb::csr_source_planned<float>(src, plan, dst, mgb::as_stream(stream));
}
int mgb_coo_sort_by_row_and_column_f64(mgb_coo* A, void* stream) {
  return mgb::coo_sort<double>(A, nullptr, 0, mgb::as_stream(stream));
}
int mgb_coo_sort_by_row_and_column_f32(mgb_coo* A, void* stream) {
  return mgb::coo_sort<float>(A, nullptr, 0, mgb::as_stream(stream));
}
int mgb_coo_sort_workspace_bytes(const mgb_coo* A, int64_t* bytes) {
  MGB_REQUIRE(A != nullptr && bytes != nullptr && A->nnz >= 0 && A->nrows >= 0, MGB_ERR_BAD_ARGUMENT);
  *bytes = (int64_t)mgb::Scratch::padded(sizeof(mgb::Words)) + mgb::prim::row_sort_bytes(A->nnz, A->nrows);
  return MGB_SUCCESS;
}
int mgb_coo_sort_by_row_and_column_ws_f64(mgb_coo* A, void* workspace, int64_t bytes, void* stream) {
  return mgb::coo_sort<double>(A, workspace, bytes, mgb::as_stream(stream));
}
int mgb_coo_sort_by_row_and_column_ws_f32(mgb_coo* A, void* workspace, int64_t bytes, void* stream) {
  return mgb::coo_sort<float>(A, workspace, bytes, mgb::as_stream(stream));
}
int mgb_coo_is_sorted(const mgb_coo* A, int* sorted, void* stream) {
  return mgb::coo_is_sorted(A, sorted, mgb::as_stream(stream));
}

}  // extern "C"
