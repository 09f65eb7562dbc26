// primitives.cuh -- device-wide building blocks for the GPU conversions:
// exclusive scan, reductions, the pass over COO indices and the stable (row,
// col) sort of COO entries.  All scratch is stream-ordered or
// the caller's.
#pragma once

#include "mgb_internal.cuh"

namespace mgb {
namespace prim {

// RAII stream-ordered scratch; freed with cudaFreeAsync on the same stream.
// A caller's workspace, where there is one, is used up first (256-byte
// pieces, in the order asked for; never freed here).
class Scratch {
 public:
  explicit Scratch(cudaStream_t s, void* workspace = nullptr, size_t bytes = 0)
      : s_(s), ws_(static_cast<char*>(workspace)), left_(workspace ? bytes : 0) {}
  ~Scratch() {
    for (int i = 0; i < n_; i++) cudaFreeAsync(p_[i], s_);
  }
  Scratch(const Scratch&) = delete;
  Scratch& operator=(const Scratch&) = delete;
  static size_t padded(size_t bytes) { return (bytes + 255) / 256 * 256; }
  template <typename T>
  cudaError_t get(T** out, size_t count) {
    *out = nullptr;
    const size_t need = padded(count ? count * sizeof(T) : 16);
    if (need <= left_) {
      *out = reinterpret_cast<T*>(ws_);
      ws_ += need;
      left_ -= need;
      return cudaSuccess;
    }
    if (n_ >= 32) return cudaErrorMemoryAllocation;
    void* p = nullptr;
    cudaError_t e = scratch_alloc(&p, count ? count * sizeof(T) : 16, s_);
    if (e == cudaSuccess) {
      p_[n_++] = p;
      *out = static_cast<T*>(p);
    }
    return e;
  }

 private:
  cudaStream_t s_;
  char* ws_;
  size_t left_;
  void* p_[32];
  int n_ = 0;
};

#define MGB_SCRATCH(sc, ptr, count) MGB_CUDA_CHECK((sc).get(&(ptr), (size_t)(count)))

// Exclusive scan of n values (any integer type in, any integer type out,
// 64-bit accumulation).  Optionally writes the total to *d_total (device).
template <typename Tin, typename Tout>
int exclusive_scan(const Tin* in, Tout* out, int64_t n, cudaStream_t s, int64_t* d_total = nullptr);

// Max over n int32 values into *d_out (device); n == 0 writes INT32_MIN.
int reduce_max_i32(const int32_t* in, int64_t n, int32_t* d_out, cudaStream_t s);

// Counts of keys in [0, nbins) (out of range keys are ignored).
int histogram(const int32_t* keys, int64_t n, int32_t* counts, int64_t nbins, cudaStream_t s);

// 1 if (row, col) pairs are sorted lexicographically (duplicates allowed),
// else 0, written to *d_flag (device).  Also *d_dup = 1 if an adjacent
// duplicate (row, col) exists (only meaningful when sorted).
int coo_sorted_flags(const int32_t* rows, const int32_t* cols, int64_t n, int32_t* d_flag,
                     int32_t* d_dup, cudaStream_t s);

// Sort the keys of each segment [seg[i], seg[i+1]) ascending (keys unique
// within a segment, so any sort is stable).  nseg segments, seg has nseg+1
// entries (int32 offsets into keys).
int segmented_sort_u64(uint64_t* keys, const int32_t* seg, int64_t nseg, int64_t nkeys, cudaStream_t s);

// COO entries brought into row order: start (nrows + 1 entries; null: kept in
// scratch) = the first entry of every row, ocol / oval (and orow unless null)
// = the entries by row and, within a row, in source order (COLS false) or by
// column and then source order (COLS true: the reference's two stable counting
// sorts, by column and then by row).  Rows must lie in [0, nrows).  The outputs
// may be the inputs.  Synchronises the stream for n > 512.  Scratch: up to
// row_sort_bytes (rows beyond 4,096 entries: 16 n more).
template <typename T, bool COLS>
int row_sort(const int32_t* rows, const int32_t* cols, const T* vals, int64_t n, int64_t nrows, int32_t* start,
             int32_t* orow, int32_t* ocol, T* oval, Scratch& sc, cudaStream_t s);
int64_t row_sort_bytes(int64_t n, int64_t nrows);

// ---- one pass over COO indices ------------------------------------------------
// Device words an entry point reads back with one copy and one stream
// synchronisation: what the index pass saw, and the plan's sizes, computed by
// kernels queued one after another.
constexpr int32_t COO_BAD_INDEX = 1;      // a row outside [0, nrows) or a column outside [0, ncols)
constexpr int32_t COO_ROWS_UNSORTED = 2;  // a row smaller than the one before it
constexpr int32_t COO_UNSORTED = 4;       // a (row, column) smaller than the one before it
constexpr int32_t COO_DUPLICATE = 8;      // a (row, column) equal to the one before it
constexpr int32_t COO_BAD_OFFSETS = 16;   // CSR row offsets that do not rise from 0 to the number of entries
constexpr int32_t COO_HUGE_ROW = 32;      // where it is looked for: maybe a row of HUGE_ROW entries or more (never missed)
constexpr int HUGE_ROW = 4096;
struct Words {
  int64_t total, total2;  // plan sizes
  int32_t seen;           // COO_* bits
  int32_t maxv;
  int32_t gaps, huge;     // of the row starts, still to be filled
  int32_t pieces, pad;    // of long rows
};
int words_alloc(Scratch& sc, Words** d, cudaStream_t s);          // zeroed
int words_read(const Words* d, Words* h, cudaStream_t s);         // synchronises

// Reads every (row, column) once, queued without a synchronisation:
// d->seen |= the COO_* bits; diag != nullptr (nrows + ncols - 1 counters,
// zeroed here): the entries on each diagonal, bin column - row + nrows - 1;
// start != nullptr (nrows + 1 entries): the first entry of every row, valid
// when the rows are in range and non-decreasing, with gaps = gap_words(nrows)
// words of scratch, and once coo_pass_gaps has filled the long gaps where the
// words read back say that there are some (gaps_left); huge: also COO_HUGE_ROW.
// Entries out of range are reported and not counted.
int64_t gap_words(int64_t nrows);
int coo_pass(const int32_t* rows, const int32_t* cols, int64_t n, int64_t nrows, int64_t ncols, Words* d,
             int32_t* diag, int32_t* start, int32_t* gaps, bool huge, cudaStream_t s);

inline bool gaps_left(const Words& h) {
  return !(h.seen & (COO_BAD_INDEX | COO_ROWS_UNSORTED)) && (h.gaps | h.huge) != 0;
}
// also clears the gaps and the sizes (total, total2, maxv) in *d
int coo_pass_gaps(const int32_t* rows, int64_t nrows, Words* d, const int32_t* gaps, int32_t* start, cudaStream_t s);

// The same for the entries of a CSR matrix (its rows are in order), one read
// of the columns; d->seen also COO_BAD_OFFSETS.  pieces: max_row_pieces(n) of
// scratch.
int csr_pass(const int32_t* ro, const int32_t* cols, int64_t n, int64_t nrows, int64_t ncols, Words* d,
             int32_t* diag, int2* pieces, cudaStream_t s);

// The bins with counts[b] >= threshold, in order: how many to *d_total, their
// counts' sum to *d_sum (if not null), and tile prefixes in sums
// (bin_tiles(nb) entries) for select_bins_apply, which replaces counts[b] by
// the bin's slot (-1: not selected) and writes offsets[slot] = b - nrows + 1
// (zero_bin: the bin recorded as offset 0, -1 for none).
int64_t bin_tiles(int64_t nb);
int select_bins(const int32_t* counts, int64_t nb, int32_t threshold, int64_t* sums, int64_t* d_total, int64_t* d_sum,
                cudaStream_t s);
int select_bins_apply(int32_t* counts, int64_t nb, int32_t threshold, const int64_t* sums, int64_t nrows,
                      int64_t zero_bin, int32_t* offsets, cudaStream_t s);

// Copy a device scalar to the host (synchronises the stream).
template <typename T>
int to_host(const T* d, T* h, cudaStream_t s) {
  MGB_CUDA_CHECK(cudaMemcpyAsync(h, d, sizeof(T), cudaMemcpyDeviceToHost, s));
  MGB_CUDA_CHECK(cudaStreamSynchronize(s));
  return MGB_SUCCESS;
}

// ---- counting into few hot bins --------------------------------------------
// A histogram whose entries fall into few distinct bins per CTA (the
// diagonals of a banded or stencil matrix: 27 bins for a 27-point stencil,
// however many entries) serialises on global atomics.  CtaHist counts in
// shared memory first, in an open-addressing table of HIST_SLOTS (key, count)
// pairs, and the CTA flushes the table with one global atomic per occupied
// slot.  A key that is in the table already costs one shared-memory read (two
// or three after a collision) and one shared-memory increment, which the
// hardware merges over the lanes that hit the same slot; the lookup is a plain
// read, and the compare-and-swap is left to the first occurrence of a key.
// A key that finds no free slot within HIST_PROBES probes marks the table
// full; from then on a key that two probes do not find goes straight to the
// global counter, so scattered keys pay little for the try while the hot
// ones, which came first, still hit the table.  The counts are exact in every
// case.  Measured on the 27-point stencil's 109 M entries (160^3): merging
// the lanes with __match_any_sync and probing by compare-and-swap took
// 1,270 us (bound by the SM's issue slots, HBM at 4 %).
constexpr int HIST_SLOTS_LOG2 = 11;
constexpr int HIST_SLOTS = 1 << HIST_SLOTS_LOG2;
constexpr int HIST_PROBES = 8;
constexpr uint32_t HIST_EMPTY = ~0u;  // no key of the table (keys from here on are counted globally)

// Resident CTAs of 256 threads per SM of the kernels that walk CSR rows into a
// table: their grid is one wave (a CTA's table is set up and flushed once).
constexpr int DIAG_CTAS = 6;

struct CtaHist {
  uint32_t* keys;   // HIST_SLOTS keys, HIST_EMPTY where free
  int32_t* counts;  // HIST_SLOTS counts
  int* full;        // set once a key found no slot
};

// every thread of the CTA, followed by __syncthreads()
__device__ __forceinline__ void hist_init(CtaHist h) {
  for (int i = threadIdx.x; i < HIST_SLOTS; i += blockDim.x) {
    h.keys[i] = HIST_EMPTY;
    h.counts[i] = 0;
  }
  if (threadIdx.x == 0) *h.full = 0;
}

__device__ __forceinline__ unsigned hist_home(uint32_t key) { return (key * 0x9E3779B1u) >> (32 - HIST_SLOTS_LOG2); }

// counts n occurrences of key < HIST_EMPTY (global[key] += n, in the end).  MERGE: lanes
// that go to the global counter with the same key add once (runs of equal
// keys: the rows of row-sorted entries; n = 1).
template <bool MERGE = false>
__device__ __forceinline__ void hist_add32(CtaHist h, int32_t* global, uint32_t key, int32_t n = 1) {
  unsigned slot = hist_home(key);
  volatile uint32_t* keys = h.keys;
  uint32_t k = keys[slot];
  if (k == key) {
    atomicAdd(h.counts + slot, n);
    return;
  }
  const int probes = *reinterpret_cast<volatile int*>(h.full) ? 2 : HIST_PROBES;
  for (int p = 0; p < probes; p++) {
    if (k == HIST_EMPTY) k = atomicCAS(h.keys + slot, HIST_EMPTY, key);
    if (k == HIST_EMPTY || k == key) {
      atomicAdd(h.counts + slot, n);
      return;
    }
    slot = (slot + 1) & (HIST_SLOTS - 1);
    k = keys[slot];
  }
  if (probes == HIST_PROBES) *reinterpret_cast<volatile int*>(h.full) = 1;
  if constexpr (MERGE) {
    const unsigned same = __match_any_sync(__activemask(), key);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(global + key, __popc(same));
  } else {
    atomicAdd(global + key, n);
  }
}

// A lane's keys, one after the other: equal ones in a row are counted in a
// register.  run_end once, after the last key.
struct KeyRun {
  uint32_t key = HIST_EMPTY;
  int32_t n = 0;
};
__device__ __forceinline__ void run_end(CtaHist h, int32_t* global, const KeyRun& k) {
  if (k.n) hist_add32(h, global, k.key, k.n);
}
__device__ __forceinline__ void run_add(CtaHist h, int32_t* global, KeyRun& k, uint32_t key) {
  if (key != k.key) {
    run_end(h, global, k);
    k.key = key;
    k.n = 0;
  }
  k.n++;
}

// the same for keys that may not fit the table's 32 bits
__device__ __forceinline__ void hist_add(CtaHist h, int32_t* global, uint64_t key) {
  if (key < HIST_EMPTY) hist_add32(h, global, (uint32_t)key);
  else atomicAdd(global + key, 1);
}

// every thread of the CTA, after a __syncthreads() that follows the last hist_add
__device__ __forceinline__ void hist_flush(CtaHist h, int32_t* global) {
  for (int i = threadIdx.x; i < HIST_SLOTS; i += blockDim.x) {
    const uint32_t k = h.keys[i];
    if (k != HIST_EMPTY && h.counts[i]) atomicAdd(global + k, h.counts[i]);
  }
}

// ---- entries of CSR rows, one warp per 32 rows ------------------------------
// Visits the entries of the rows [r0, min(r0 + 32, nrows)) in groups of 32
// consecutive ones, a lane per entry, however long the rows are.  The rows'
// first entries are marked in a bitmap of 1,024 entries at a time; an entry's
// row is the number of marks up to it (one population count), through a list
// of the rows that are not empty.  Entry e = c0 + i: v = load(c0, i) for four
// groups ahead of their f(in, head, q, c0, i, v), which every lane of the warp
// calls (in: the lane holds an entry, of row r0 + q; head: the row's first; full
// groups are compiled with in = true).  The warps that share the rows take every
// `step`th group from `first` on.  Searching every fourth entry's row among
// the offsets and moving on from there took 160 instructions per 128 entries.
struct WarpRows {
  uint32_t bits[32];
  int32_t row[32];
};
template <typename LOAD, typename F>
__device__ __forceinline__ void warp_row_walk(const int32_t* __restrict__ ro, int64_t r0, int64_t nrows, WarpRows& w,
                                              int lane, int first, int step, LOAD load, F f) {
  constexpr unsigned ALL = 0xffffffffu;
  const int32_t a = ro[min(r0 + lane, nrows)], z = ro[min(r0 + lane + 1, nrows)];
  const int64_t b = __shfl_sync(ALL, a, 0), t = __shfl_sync(ALL, z, 31);
  const bool some = z > a;
  const unsigned m = __ballot_sync(ALL, some);
  const unsigned upto = ALL >> (31 - lane);
  __syncwarp();
  if (some) w.row[__popc(m & (upto >> 1))] = lane;
  for (int64_t c0 = b; c0 < t; c0 += 1024) {
    w.bits[lane] = 0;
    __syncwarp();
    const int64_t at = a - c0;
    if (some && at >= 0 && at < 1024) atomicOr(w.bits + (at >> 5), 1u << (at & 31));
    __syncwarp();
    const uint32_t word = w.bits[lane];
    int pre = __popc(word);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int u = __shfl_up_sync(ALL, pre, d);
      if (lane >= d) pre += u;
    }
    pre += __popc(__ballot_sync(ALL, some && a < c0)) - __popc(word) - 1;
    const int n = (int)min(t - c0, (int64_t)1024);
    auto emit = [&](bool in, int g, auto v) {
      const uint32_t marks = __shfl_sync(ALL, word, g);
      const int k = (__shfl_sync(ALL, pre, g) + __popc(marks & upto)) & 31;
      f(in, (marks >> lane) & 1, m == ALL ? k : w.row[k], c0, 32 * g + lane, v);
    };
    int j = first;
    for (; j + 3 * step < (n >> 5); j += 4 * step) {
      decltype(load(c0, 0)) v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] = load(c0, 32 * (j + u * step) + lane);
#pragma unroll
      for (int u = 0; u < 4; u++) emit(true, j + u * step, v[u]);
    }
    for (; 32 * j < n; j += step) {
      decltype(load(c0, 0)) v{};
      const bool in = 32 * j + lane < n;
      if (in) v = load(c0, 32 * j + lane);
      emit(in, j, v);
    }
    __syncwarp();
  }
}

// Groups of 32 rows with more than LONG_GROUP entries have too many for one warp.
// Their rows of more than LONG_ROW: listed in pieces of ROW_PIECE entries (x: row, or
// -1 for none, y: piece), which a second kernel takes by CTAs.  The list is
// bounded (512 KB): rows beyond it stay with their warps, of which so many long
// rows keep enough busy.
constexpr int LONG_GROUP = 8192;
constexpr int LONG_ROW = 512;
constexpr int ROW_PIECE = 2048;
struct RowPieces {
  int2* list;
  int32_t* count;  // zeroed
  int64_t limit;
};
inline int64_t max_row_pieces(int64_t nnz) {
  const int64_t n = nnz / LONG_ROW + 1;
  return n < 65536 ? n : 65536;
}

// The list (limit set) and its count, from sc.
inline int row_pieces_alloc(RowPieces* p, Scratch& sc, cudaStream_t s) {
  MGB_SCRATCH(sc, p->list, p->limit + 1);
  p->count = reinterpret_cast<int32_t*>(p->list + p->limit);
  MGB_CUDA_CHECK(cudaMemsetAsync(p->count, 0, sizeof(int32_t), s));
  return MGB_SUCCESS;
}

// Asked before warp_rows_apart, which kernels call out of line: few groups need
// it, and inlined it costs the others registers.
__device__ __forceinline__ bool long_group(const int32_t* __restrict__ ro, int64_t r0, int64_t nrows) {
  return (int64_t)ro[min(r0 + 32, nrows)] - ro[r0] > LONG_GROUP;
}
// The rows [r0, min(r0 + 32, nrows)) of a long group, where one of them is long:
// lists the long ones and calls f(in, q, e, first) for 32 entries e of another
// row r0 + q at a time (first: the row's first entry), every lane of the warp.
// Otherwise false, and nothing is done.
template <typename F>
__device__ __forceinline__ bool warp_rows_apart(const int32_t* __restrict__ ro, int64_t r0, int64_t nrows,
                                                RowPieces pieces, int lane, F f) {
  constexpr unsigned ALL = 0xffffffffu;
  const int32_t a = ro[min(r0 + lane, nrows)], z = ro[min(r0 + lane + 1, nrows)];
  const int64_t len = (int64_t)z - a;
  unsigned longs = __ballot_sync(ALL, len > LONG_ROW);
  if (!longs) return false;
  const int32_t np = len > LONG_ROW ? (int32_t)((len + ROW_PIECE - 1) / ROW_PIECE) : 0;
  int32_t upto = np;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int32_t u = __shfl_up_sync(ALL, upto, d);
    if (lane >= d) upto += u;
  }
  const int32_t total = __shfl_sync(ALL, upto, 31);
  int32_t base = 0;
  if (lane == 0) base = *reinterpret_cast<volatile int32_t*>(pieces.count) >= pieces.limit
                            ? (int32_t)pieces.limit : atomicAdd(pieces.count, total);
  base = __shfl_sync(ALL, base, 0);
  if ((int64_t)base + total > pieces.limit) {  // full: the places left hold nothing
    for (int64_t i = base + lane; i < pieces.limit; i += 32) pieces.list[i] = make_int2(-1, 0);
    longs = 0;
  }
  for (int q = 0; q < 32; q++) {
    const int64_t n = __shfl_sync(ALL, len, q);
    const int32_t first = __shfl_sync(ALL, a, q);
    if ((longs >> q) & 1) {
      const int32_t k = __shfl_sync(ALL, np, q), at = base + __shfl_sync(ALL, upto, q) - k;
      for (int32_t i = lane; i < k; i += 32) pieces.list[at + i] = make_int2((int32_t)(r0 + q), i);
    } else {
      for (int64_t j = 0; j < n; j += 32) f(j + lane < n, q, (int32_t)(first + j + lane), first);
    }
  }
  return true;
}

// Calls f(row, e, first) for every entry e of the listed pieces, a thread each;
// CTAs of 256 threads.
template <typename F>
__device__ __forceinline__ void for_row_pieces(const int32_t* __restrict__ ro, RowPieces pieces, F f) {
  const int64_t n = min((int64_t)*pieces.count, pieces.limit);
  for (int64_t p = blockIdx.x; p < n; p += gridDim.x) {
    const int2 piece = pieces.list[p];
    if (piece.x < 0) continue;
    const int32_t first = ro[piece.x], end = ro[piece.x + 1];
    const int64_t e0 = first + (int64_t)piece.y * ROW_PIECE, e1 = min(e0 + ROW_PIECE, (int64_t)end);
    for (int64_t e = e0 + threadIdx.x; e < e1; e += 256) f(piece.x, (int32_t)e, first);
  }
}

// Counts the diagonals (bin column - row + nrows - 1) of the entries of the same
// 32 rows so that a lane keeps its position in the row while the rows go by:
// 32 / L rows of L entries at a time, which are consecutive entries too.  On a
// stencil's or band's rows a lane's diagonal then stays the same from row to
// row, and its KeyRun takes eight steps with one comparison of them all (six
// instructions per step; a look into the table and a shared-memory atomic per
// entry made it 70).  Where the diagonals change, each lane starts a run at the
// first of the eight; if the others are not on it either, or a column is
// outside the matrix, they go through the table one by one, and after four
// eights in a row like that (columns that follow no diagonal) the warp is told
// to walk its other rows.
// ORDER: *down / *equal as for entries of one row that follow each other;
// *bad: a column beyond the matrix.
// False, and nothing counted, unless the lengths change so seldom that the
// steps outweigh the changes (one costs about what 96 entries of the walk do),
// no row is longer than the warp, and the offsets do not decrease.
// 27-point stencil, 160^3, walk -> here: csr_pass 236 -> 148 us, csr_diag 193 ->
// 136 (the columns at the copy rate: 66); entries one by one after each change
// of length: 170 / 156; the next eight loaded ahead with four CTAs per SM: 151 /
// 140, and rows that have to be walked 5-10 % slower than with six.
template <bool ORDER>
__device__ __forceinline__ bool warp_equal_rows(const int32_t* __restrict__ ro, int64_t r0, int64_t nrows,
                                                const int32_t* __restrict__ c, uint32_t nc, int lane, CtaHist h,
                                                int32_t* counts, KeyRun& run, int& misses, bool* bad, bool* down,
                                                bool* equal) {
  constexpr unsigned ALL = 0xffffffffu;
  constexpr int STEPS = 8;
  if (misses >= 4) return false;
  const int32_t a = ro[min(r0 + lane, nrows)], len = ro[min(r0 + lane + 1, nrows)] - a;
  const int32_t left = __shfl_up_sync(ALL, len, 1);
  unsigned heads = __ballot_sync(ALL, lane == 0 || len != left);
  const int32_t total = __shfl_sync(ALL, a + len, 31) - __shfl_sync(ALL, a, 0);
  if (96 * __popc(heads) > total || __any_sync(ALL, (unsigned)len > 32u)) return false;
  const uint32_t diag0 = (uint32_t)(nrows - 1 - r0);
  while (heads) {
    const int q0 = __ffs(heads) - 1;
    heads &= heads - 1;
    const int q1 = heads ? __ffs(heads) - 1 : 32;
    const int L = __shfl_sync(ALL, len, q0);
    const int32_t e0 = __shfl_sync(ALL, a, q0);
    if (L == 0) continue;
    const int P = 32 / L, sub = lane / L;
    const bool inner = lane > sub * L;  // not the row's first
    const int end = sub < P ? q1 : 0;
    const int32_t* p = c + e0 + lane;
    for (int q = q0; q < q1; q += STEPS * P, p += STEPS * P * L) {
      uint32_t v[STEPS];
#pragma unroll
      for (int u = 0; u < STEPS; u++) v[u] = q + u * P + sub < end ? (uint32_t)__ldcs(p + u * P * L) : 0;
      int32_t n = 0;
      auto same = [&] {  // every entry on its lane's run
        const uint32_t want = run.key - diag0 + (q + sub);
        uint32_t other = 0, last = 0;
        n = 0;
#pragma unroll
        for (int u = 0; u < STEPS; u++)
          if (q + u * P + sub < end) {
            other |= v[u] ^ (want + u * P);
            last = v[u];
            n++;
          }
        return !__any_sync(ALL, other != 0 || last >= nc || v[0] >= nc);
      };
      bool all = same();
      if (!all) {  // runs start at the first of the steps
        const uint32_t key = v[0] - (q + sub) + diag0;
        if (n > 0 && v[0] < nc && key != run.key) {
          run_end(h, counts, run);
          run.key = key;
          run.n = 0;
        }
        all = same();
        misses += !all;
      } else {
        misses = 0;
      }
      if (all) {
        run.n += n;
        if constexpr (ORDER) {  // alike in all steps
          const uint32_t before = __shfl_up_sync(ALL, v[0], 1);
          *down |= n > 0 && inner && v[0] < before;
          *equal |= n > 0 && inner && v[0] == before;
        }
        continue;
      }
#pragma unroll 1
      for (int u = 0; u < STEPS && q + u * P < q1; u++) {
        const int row = q + u * P + sub;
        const bool in = row < end;
        const uint32_t col = in ? (uint32_t)__ldg(p + u * P * L) : 0;
        if constexpr (ORDER) {
          const uint32_t before = __shfl_up_sync(ALL, col, 1);
          *down |= in && inner && col < before;
          *equal |= in && inner && col == before;
        }
        if (!in) continue;
        if (col >= nc) *bad = true;
        else run_add(h, counts, run, col - row + diag0);
      }
    }
  }
  return true;
}

// global[key] += 1 with the lanes of a warp holding the same key merged
// (row counts of row-sorted entries: consecutive lanes share a row)
__device__ __forceinline__ void warp_merged_add(int32_t* global, int64_t key) {
  const unsigned same = __match_any_sync(__activemask(), (unsigned long long)key);
  if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(global + key, __popc(same));
}

#define MGB_CTA_HIST(name)                                  \
  __shared__ uint32_t name##_keys[::mgb::prim::HIST_SLOTS]; \
  __shared__ int32_t name##_counts[::mgb::prim::HIST_SLOTS]; \
  __shared__ int name##_full;                               \
  const ::mgb::prim::CtaHist name{name##_keys, name##_counts, &name##_full}

inline unsigned blocks_for(int64_t n, int threads, int64_t cap = 1 << 20) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > cap) b = cap;
  return (unsigned)b;
}

}  // namespace prim
}  // namespace mgb
