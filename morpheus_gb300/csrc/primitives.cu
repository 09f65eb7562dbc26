// primitives.cu -- scan, reductions, histograms and sorts used by convert.cu.
#include <climits>
#include <type_traits>
#include <utility>

#include "primitives.cuh"

namespace mgb {
namespace prim {
namespace {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// exclusive scan of one int64 per thread across the block; returns the
// exclusive prefix, *total = block sum
__device__ int64_t block_exclusive_scan(int64_t v, int64_t* total) {
  __shared__ int64_t s_warp[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int64_t inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int64_t u = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += u;
  }
  if (lane == 31) s_warp[w] = inc;
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    int64_t x = lane < nw ? s_warp[lane] : 0;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int64_t u = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += u;
    }
    if (lane < nw) s_warp[lane] = x;  // inclusive warp prefix
  }
  __syncthreads();
  const int64_t warp_excl = w ? s_warp[w - 1] : 0;
  *total = s_warp[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_excl + inc - v;
}

template <typename Tin>
__global__ void __launch_bounds__(SCAN_THREADS) scan_tile_sums(const Tin* __restrict__ in, int64_t n,
                                                               int64_t* __restrict__ sums) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  int64_t v = 0;
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const int64_t i = base + (int64_t)k * SCAN_THREADS + threadIdx.x;
    if (i < n) v += (int64_t)in[i];
  }
  int64_t total;
  block_exclusive_scan(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// exclusive scan of sums[0..nb) in place by one block; total -> *d_total
__global__ void __launch_bounds__(1024) scan_sums(int64_t* sums, int64_t nb, int64_t* d_total) {
  const int64_t per = (nb + blockDim.x - 1) / blockDim.x;
  const int64_t b0 = (int64_t)threadIdx.x * per;
  int64_t local = 0;
  for (int64_t i = b0; i < b0 + per && i < nb; i++) local += sums[i];
  int64_t total;
  int64_t run = block_exclusive_scan(local, &total);
  for (int64_t i = b0; i < b0 + per && i < nb; i++) {
    const int64_t v = sums[i];
    sums[i] = run;
    run += v;
  }
  if (threadIdx.x == 0 && d_total) *d_total = total;
}

template <typename Tin, typename Tout>
__global__ void __launch_bounds__(SCAN_THREADS) scan_apply(const Tin* __restrict__ in, Tout* __restrict__ out,
                                                           int64_t n, const int64_t* __restrict__ sums) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
  int64_t v[SCAN_ITEMS];
  int64_t local = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const int64_t i = base + k;
    v[k] = i < n ? (int64_t)in[i] : 0;
    local += v[k];
  }
  int64_t total;
  int64_t run = block_exclusive_scan(local, &total) + sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const int64_t i = base + k;
    if (i < n) out[i] = (Tout)run;
    run += v[k];
  }
}

__global__ void fill_i32(int32_t* p, int32_t v, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    p[i] = v;
}

__global__ void max_i32_kernel(const int32_t* __restrict__ in, int64_t n, int32_t* out) {
  int32_t m = INT_MIN;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, in[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// counts[k] += 1 for every key in [0, nbins); few hot keys per CTA are
// counted in shared memory first (CtaHist)
__global__ void histogram_kernel(const int32_t* __restrict__ keys, int64_t n, int32_t* counts, int64_t nbins) {
  MGB_CTA_HIST(h);
  hist_init(h);
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t k = keys[i];
    if (k >= 0 && k < nbins) hist_add32<true>(h, counts, (uint32_t)k);
  }
  __syncthreads();
  hist_flush(h, counts);
}

__global__ void sorted_flags_kernel(const int32_t* __restrict__ r, const int32_t* __restrict__ c, int64_t n,
                                    int32_t* flag, int32_t* dup) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i + 1 < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t r0 = r[i], r1 = r[i + 1];
    if (c == nullptr) {
      if (r0 > r1) *flag = 0;
    } else {
      const int32_t c0 = c[i], c1 = c[i + 1];
      if (r0 > r1 || (r0 == r1 && c0 > c1)) *flag = 0;
      if (dup && r0 == r1 && c0 == c1) *dup = 1;
    }
  }
}

// One pass over the indices (coo_pass).  Each thread takes four consecutive
// entries (16-byte loads where the arrays are aligned) and its predecessor
// from the neighbouring lane, so rows and columns are read once for the range
// check, the order flags, the diagonal counts and the row starts together
// (five kernels before: 480 us of index reads and an intermediate bin array
// on the 27-point stencil at 160^3; the HBM floor of the pass is 131 us).
// Row starts: the entry where the row changes from p to q is the start of
// the rows p + 1..q; gaps longer than PASS_GAP are listed by their entry and
// filled by fill_gaps, a warp each, those beyond PASS_HUGE by its whole grid (COO
// -> CSR of 10,000 entries in 5e7 rows: 3,260 us with the CTA that met the gap
// filling it, 195); the rows before the first and after the last entry are left to
// this kernel's grid.
// Rows that go down make the starts useless, and entries in random order have
// gaps of a third of the matrix each: the first such row that a CTA sees stops
// the writing of starts in that CTA at once and in the others at their next
// tile.
constexpr uint32_t PASS_GAP = 256;
constexpr uint32_t PASS_HUGE = 1 << 16;
// of non-decreasing rows at most so many gaps
__host__ __device__ inline int64_t max_gaps(int64_t nrows) { return nrows / PASS_GAP + 1; }
__host__ __device__ inline int64_t max_huge(int64_t nrows) { return nrows / PASS_HUGE + 1; }

// out of line: the pass has no registers to spare for it
__device__ __noinline__ void list_gap(Words* d, int32_t* gaps, int64_t nrows, int32_t at, bool huge) {
  const int64_t g = atomicAdd(huge ? &d->huge : &d->gaps, 1);
  if (g < (huge ? max_huge(nrows) : max_gaps(nrows))) gaps[(huge ? max_gaps(nrows) : 0) + g] = at;
}

// HUGE: looks for rows of HUGE_ROW entries (COO_HUGE_ROW).
template <bool DIAG, bool STARTS, bool HUGE>
__global__ void __launch_bounds__(256, STARTS ? (DIAG && HUGE ? 6 : 8) : 1) coo_pass_kernel(const int32_t* __restrict__ r, const int32_t* __restrict__ c,
                                                       int64_t n, int64_t nrows, int64_t ncols, bool vec,
                                                       Words* d, int32_t* __restrict__ diag,
                                                       int32_t* __restrict__ start, int32_t* __restrict__ gaps) {
  int32_t* seen = &d->seen;
  __shared__ uint32_t h_keys[DIAG ? HIST_SLOTS : 1];
  __shared__ int32_t h_counts[DIAG ? HIST_SLOTS : 1];
  __shared__ int h_full;
  __shared__ int s_bits, s_stop;
  volatile int* stop = &s_stop;
  const CtaHist h{h_keys, h_counts, &h_full};
  if constexpr (DIAG) hist_init(h);
  if (threadIdx.x == 0) {
    s_bits = 0;
    s_stop = 0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  // valid indices are below 2^31: unsigned comparisons (order flags that
  // negative indices upset do not matter, such a matrix is refused)
  const uint32_t nr = (uint32_t)min(nrows, (int64_t)1 << 31), nc = (uint32_t)min(ncols, (int64_t)1 << 31);
  const uint32_t mid = (uint32_t)(nrows - 1);
  int bits = 0;
  for (int64_t base = (int64_t)blockIdx.x * 1024; base < n; base += (int64_t)gridDim.x * 1024) {
    const int64_t i0 = base + (int64_t)threadIdx.x * 4;
    const int m = (int)min((int64_t)4, n - i0);  // this thread's entries (<= 0: none)
    if (STARTS && (*reinterpret_cast<volatile int32_t*>(seen) & COO_ROWS_UNSORTED)) *stop = 1;
    uint32_t rr[4] = {0, 0, 0, 0}, cc[4] = {0, 0, 0, 0};
    if (vec && m == 4) {
      const int4 a = __ldg(reinterpret_cast<const int4*>(r + i0)), b = __ldg(reinterpret_cast<const int4*>(c + i0));
      rr[0] = a.x; rr[1] = a.y; rr[2] = a.z; rr[3] = a.w;
      cc[0] = b.x; cc[1] = b.y; cc[2] = b.z; cc[3] = b.w;
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (k < m) { rr[k] = r[i0 + k]; cc[k] = c[i0 + k]; }
    }
    uint32_t pr = __shfl_up_sync(0xffffffffu, rr[3], 1), pc = __shfl_up_sync(0xffffffffu, cc[3], 1);
    if (lane == 0 && m > 0 && i0 > 0) { pr = r[i0 - 1]; pc = c[i0 - 1]; }
    if (i0 == 0) { pr = rr[0]; pc = 0; }  // the first entry: nothing before it
    // a row of HUGE_ROW entries has two that are HUGE_ROW - 1024 apart, the first at a multiple of 1024
    if (HUGE && threadIdx.x == 0 && base + HUGE_ROW - 1024 < n && r[base + HUGE_ROW - 1024] == (int32_t)rr[0])
      bits |= COO_HUGE_ROW;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      if (k >= m) break;
      const bool ok = rr[k] < nr && cc[k] < nc;
      if (!ok) bits |= COO_BAD_INDEX;
      if (rr[k] == pr) {
        if (cc[k] < pc) bits |= COO_UNSORTED;
        if (cc[k] == pc && (k > 0 || i0 > 0)) bits |= COO_DUPLICATE;
      } else {
        if (rr[k] < pr) {
          bits |= COO_ROWS_UNSORTED | COO_UNSORTED;
          if (STARTS && !*stop) {
            *stop = 1;
            atomicOr(seen, COO_ROWS_UNSORTED);
          }
        }
        if constexpr (STARTS) {
          if (rr[k] == pr + 1) {
            if (rr[k] < nr) start[rr[k]] = (int32_t)(i0 + k);
          } else if (rr[k] > pr && rr[k] < nr && !*stop) {
            const int32_t at = (int32_t)(i0 + k);
            if (rr[k] - pr > PASS_GAP) {
              list_gap(d, gaps, nrows, at, rr[k] - pr > PASS_HUGE);
            } else {
              for (uint32_t q = pr + 1; q <= rr[k]; q++) start[q] = at;
            }
          }
        }
      }
      if (DIAG && ok) hist_add32(h, diag, cc[k] - rr[k] + mid);
      pr = rr[k];
      pc = cc[k];
    }
  }
  if (bits) atomicOr(&s_bits, bits);
  __syncthreads();
  if (threadIdx.x == 0 && s_bits) atomicOr(seen, s_bits);
  if constexpr (DIAG) hist_flush(h, diag);
  if constexpr (STARTS) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x, nt = (int64_t)gridDim.x * 256;
    const int64_t first = n > 0 ? min((int64_t)r[0], nrows) : nrows;
    const int64_t last = n > 0 ? max((int64_t)r[n - 1], (int64_t)-1) : nrows;
    for (int64_t q = t; q <= first; q += nt) start[q] = 0;
    for (int64_t q = last + 1 + t; q <= nrows; q += nt) start[q] = (int32_t)n;
  }
}

// The rows of the listed gaps start at the entry behind the gap (valid and
// non-decreasing rows).
__global__ void __launch_bounds__(256) fill_gaps(const int32_t* __restrict__ r, int64_t nrows, const Words* d,
                                                 const int32_t* __restrict__ gaps, int32_t* __restrict__ start) {
  const int64_t warps = (int64_t)gridDim.x * 8, n = min((int64_t)d->gaps, max_gaps(nrows));
  for (int64_t g = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); g < n; g += warps) {
    const int32_t at = gaps[g];
    for (int64_t q = (int64_t)r[at - 1] + 1 + (threadIdx.x & 31); q <= r[at]; q += 32) start[q] = at;
  }
  const int64_t huge = min((int64_t)d->huge, max_huge(nrows));
  for (int64_t g = 0; g < huge; g++) {
    const int32_t at = gaps[max_gaps(nrows) + g];
    const int64_t first = (int64_t)r[at - 1] + 1, last = r[at];
    for (int64_t q = first + (int64_t)blockIdx.x * 256 + threadIdx.x; q <= last; q += (int64_t)gridDim.x * 256)
      start[q] = at;
  }
}

// Rows of a long group: their COO_* bits, -1 where they are walked as any.
template <bool DIAG>
__device__ __noinline__ int csr_pass_apart(const int32_t* __restrict__ ro, const int32_t* __restrict__ c, int64_t r0,
                                           int64_t nrows, uint32_t nc, int lane, CtaHist h, int32_t* diag,
                                           RowPieces pieces) {
  int bits = COO_HUGE_ROW;
  const bool apart = warp_rows_apart(ro, r0, nrows, pieces, lane, [&](bool in, int q, int32_t e, int32_t first) {
    if (!in) return;
    const uint32_t col = c[e], before = e > first ? c[e - 1] : 0;
    if (col >= nc) bits |= COO_BAD_INDEX;
    if (col < before) bits |= COO_UNSORTED;
    if (e > first && col == before) bits |= COO_DUPLICATE;
    if (DIAG && col < nc) hist_add32(h, diag, col - (uint32_t)(r0 + q) + (uint32_t)(nrows - 1));
  });
  return apart ? bits : -1;
}

template <bool DIAG>
__global__ void __launch_bounds__(256, DIAG_CTAS) csr_pass_kernel(const int32_t* __restrict__ ro, const int32_t* __restrict__ c,
                                                       int64_t n, int64_t nrows, int64_t ncols, int32_t* seen,
                                                       int32_t* __restrict__ diag, RowPieces pieces) {
  __shared__ uint32_t h_keys[DIAG ? HIST_SLOTS : 1];
  __shared__ int32_t h_counts[DIAG ? HIST_SLOTS : 1];
  __shared__ int h_full, s_bits;
  __shared__ WarpRows s_rows[8];
  const CtaHist h{h_keys, h_counts, &h_full};
  if constexpr (DIAG) hist_init(h);
  if (threadIdx.x == 0) s_bits = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t nc = (uint32_t)min(ncols, (int64_t)1 << 31);
  bool bad = false, offsets = false, down = false, equal = false;
  int longs = 0;
  KeyRun run;
  int misses = 0;
  for (int64_t r0 = ((int64_t)blockIdx.x * 8 + w) * 32; r0 < nrows; r0 += (int64_t)gridDim.x * 256) {
    const int64_t r = r0 + lane;
    if (r < nrows) {
      const int32_t a = ro[r], z = ro[r + 1];
      offsets |= a > z || a < 0 || z > n || (r == 0 && a != 0) || (r == nrows - 1 && z != n);
    }
    if (__any_sync(0xffffffffu, offsets)) break;  // nothing of such rows is read
    uint32_t last = 0;  // column of the entry before the group
    const uint32_t diag0 = (uint32_t)(nrows - 1 - r0);
    if (DIAG && warp_equal_rows<true>(ro, r0, nrows, c, nc, lane, h, diag, run, misses, &bad, &down, &equal)) continue;
    if (long_group(ro, r0, nrows)) {
      const int b = csr_pass_apart<DIAG>(ro, c, r0, nrows, nc, lane, h, diag, pieces);
      if (b >= 0) {
        longs |= b;
        continue;
      }
    }
    warp_row_walk(
        ro, r0, nrows, s_rows[w], lane, 0, 1, [&](int64_t c0, int i) { return (uint32_t)__ldcs(c + c0 + i); },
        [&](bool in, bool head, int q, int64_t, int, uint32_t col) {
          uint32_t before = __shfl_up_sync(0xffffffffu, col, 1);
          if (lane == 0) before = last;
          last = __shfl_sync(0xffffffffu, col, 31);
          if (!in) return;
          bad |= col >= nc;
          down |= !head && col < before;
          equal |= !head && col == before;
          if (DIAG && col < nc) hist_add32(h, diag, col - q + diag0);
        });
  }
  if constexpr (DIAG) run_end(h, diag, run);
  const int bits = (bad ? COO_BAD_INDEX : 0) | (offsets ? COO_BAD_OFFSETS : 0) | (down ? COO_UNSORTED : 0) |
                   (equal ? COO_DUPLICATE : 0) | longs;
  if (bits) atomicOr(&s_bits, bits);
  __syncthreads();
  if (threadIdx.x == 0 && s_bits) atomicOr(seen, s_bits);
  if constexpr (DIAG) hist_flush(h, diag);
}

// The entries of the long rows: most of them alone on their diagonals, so they
// are counted globally.  CSR -> ELL of 64 rows of 500,000 entries: 27,100 us
// through COO, 95,400 with a warp per 32 rows, 350 with pieces.
template <bool DIAG>
__global__ void __launch_bounds__(256) csr_pass_pieces(const int32_t* __restrict__ ro, const int32_t* __restrict__ c,
                                                       int64_t nrows, int64_t ncols, int32_t* seen,
                                                       int32_t* __restrict__ diag, RowPieces pieces) {
  if (*pieces.count == 0 || (*reinterpret_cast<volatile int32_t*>(seen) & COO_BAD_OFFSETS)) return;
  const uint32_t nc = (uint32_t)min(ncols, (int64_t)1 << 31);
  bool bad = false, down = false, equal = false;
  for_row_pieces(ro, pieces, [&](int32_t row, int32_t e, int32_t first) {
    const uint32_t col = __ldg(c + e), before = e > first ? __ldg(c + e - 1) : 0;
    bad |= col >= nc;
    down |= col < before;
    equal |= e > first && col == before;
    if (DIAG && col < nc) atomicAdd(diag + (col - (uint32_t)row + (uint32_t)(nrows - 1)), 1);
  });
  const int bits = (bad ? COO_BAD_INDEX : 0) | (down ? COO_UNSORTED : 0) | (equal ? COO_DUPLICATE : 0);
  if (bits) atomicOr(seen, bits);
}

// ---- selection of bins -----------------------------------------------------
__global__ void __launch_bounds__(SCAN_THREADS) bin_tile_sums(const int32_t* __restrict__ counts, int64_t nb,
                                                              int32_t thr, int64_t* __restrict__ sums,
                                                              unsigned long long* d_sum) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE;
  int64_t v = 0, e = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const int64_t i = base + (int64_t)k * SCAN_THREADS + threadIdx.x;
    const int32_t x = i < nb ? counts[i] : 0;
    if (i < nb && x >= thr) {
      v++;
      e += x;
    }
  }
  int64_t total;
  block_exclusive_scan(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
  if (d_sum != nullptr && total > 0) {
    block_exclusive_scan(e, &total);
    if (threadIdx.x == 0) atomicAdd(d_sum, (unsigned long long)total);
  }
}

__global__ void __launch_bounds__(SCAN_THREADS) bin_apply(int32_t* __restrict__ counts, int64_t nb, int32_t thr,
                                                          const int64_t* __restrict__ sums, int64_t nrows,
                                                          int64_t zero_bin, int32_t* __restrict__ offsets) {
  const int64_t base = (int64_t)blockIdx.x * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
  bool f[SCAN_ITEMS];
  int64_t local = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    f[k] = base + k < nb && counts[base + k] >= thr;
    local += f[k];
  }
  int64_t total;
  int64_t slot = block_exclusive_scan(local, &total) + sums[blockIdx.x];
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; k++) {
    const int64_t b = base + k;
    if (b >= nb) break;
    counts[b] = f[k] ? (int32_t)slot : -1;
    if (f[k]) offsets[slot++] = b == zero_bin ? 0 : (int32_t)(b - nrows + 1);
  }
}

// ---- segmented sort ------------------------------------------------------

constexpr int SEG_SMALL = 32;
constexpr int SEG_MED = 4096;
constexpr int SEG_MED_THREADS = 512;

__global__ void classify_segments(const int32_t* __restrict__ seg, int64_t nseg, int32_t* lists, int64_t cap,
                                  int32_t* counters) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nseg; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t len = seg[i + 1] - seg[i];
    if (len <= 1) continue;
    const int cls = len <= SEG_SMALL ? 0 : (len <= SEG_MED ? 1 : 2);
    const int32_t slot = atomicAdd(counters + cls, 1);
    lists[cls * cap + slot] = (int32_t)i;
  }
}

__global__ void sort_small_segments(uint64_t* keys, const int32_t* __restrict__ seg, const int32_t* __restrict__ list,
                                    const int32_t* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t w = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); w < *count; w += nw) {
    const int32_t s = list[w];
    const int32_t b = seg[s], len = seg[s + 1] - b;
    uint64_t v = lane < len ? keys[b + lane] : ~0ull;
    // bitonic sort across the 32 lanes
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const uint64_t o = __shfl_xor_sync(0xffffffffu, v, j);
        const bool up = ((lane & k) == 0);
        const bool lower = ((lane & j) == 0);
        const uint64_t mn = v < o ? v : o, mx = v < o ? o : v;
        v = (lower == up) ? mn : mx;
      }
    }
    if (lane < len) keys[b + lane] = v;
  }
}

// bitonic sort of m (power of two, <= SEG_MED) keys in shared memory
__device__ void bitonic_smem(uint64_t* sk, int m) {
  for (int k = 2; k <= m; k <<= 1) {
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int p = i ^ j;
        if (p > i) {
          const uint64_t a = sk[i], b = sk[p];
          const bool up = ((i & k) == 0);
          if ((a > b) == up) { sk[i] = b; sk[p] = a; }
        }
      }
      __syncthreads();
    }
  }
}

__global__ void __launch_bounds__(SEG_MED_THREADS) sort_medium_segments(uint64_t* keys, const int32_t* __restrict__ seg,
                                                                        const int32_t* __restrict__ list,
                                                                        const int32_t* __restrict__ count) {
  __shared__ uint64_t sk[SEG_MED];
  for (int64_t w = blockIdx.x; w < *count; w += gridDim.x) {
    const int32_t s = list[w];
    const int32_t b = seg[s], len = seg[s + 1] - b;
    int m = 64;
    while (m < len) m <<= 1;
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) sk[i] = i < len ? keys[b + i] : ~0ull;
    __syncthreads();
    bitonic_smem(sk, m);
    for (int i = threadIdx.x; i < len; i += blockDim.x) keys[b + i] = sk[i];
  }
}

// large segments: sort 4096-chunks in shared memory, then merge runs pairwise
// (merge path: each thread emits a contiguous slice of the output)
__device__ int64_t merge_corank(const uint64_t* a, int64_t na, const uint64_t* b, int64_t nb, int64_t k) {
  // number of elements taken from a among the first k outputs (stable: a first on ties)
  int64_t lo = k > nb ? k - nb : 0, hi = k < na ? k : na;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (a[mid] <= b[k - mid - 1]) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__global__ void __launch_bounds__(SEG_MED_THREADS) sort_large_segments(uint64_t* keys, uint64_t* tmp,
                                                                       const int32_t* __restrict__ seg,
                                                                       const int32_t* __restrict__ list,
                                                                       const int32_t* __restrict__ count) {
  __shared__ uint64_t sk[SEG_MED];
  for (int64_t w = blockIdx.x; w < *count; w += gridDim.x) {
    const int32_t s = list[w];
    const int64_t b = seg[s], len = seg[s + 1] - b;
    uint64_t* src = keys + b;
    uint64_t* dst = tmp + b;
    for (int64_t c0 = 0; c0 < len; c0 += SEG_MED) {
      const int cl = (int)min((int64_t)SEG_MED, len - c0);
      __syncthreads();
      for (int i = threadIdx.x; i < SEG_MED; i += blockDim.x) sk[i] = i < cl ? src[c0 + i] : ~0ull;
      __syncthreads();
      bitonic_smem(sk, SEG_MED);
      for (int i = threadIdx.x; i < cl; i += blockDim.x) src[c0 + i] = sk[i];
    }
    __syncthreads();
    bool in_src = true;
    for (int64_t width = SEG_MED; width < len; width <<= 1) {
      const uint64_t* from = in_src ? src : dst;
      uint64_t* to = in_src ? dst : src;
      for (int64_t a0 = 0; a0 < len; a0 += 2 * width) {
        const int64_t na = min(width, len - a0);
        const int64_t nb = max((int64_t)0, min(width, len - a0 - width));
        const int64_t tot = na + nb;
        const int64_t per = (tot + blockDim.x - 1) / blockDim.x;
        const int64_t k0 = min(tot, (int64_t)threadIdx.x * per), k1 = min(tot, k0 + per);
        const uint64_t* A = from + a0;
        const uint64_t* B = from + a0 + na;
        int64_t ia = merge_corank(A, na, B, nb, k0);
        int64_t ib = k0 - ia;
        for (int64_t k = k0; k < k1; k++) {
          if (ib >= nb || (ia < na && A[ia] <= B[ib])) to[a0 + k] = A[ia++];
          else to[a0 + k] = B[ib++];
        }
      }
      __syncthreads();
      in_src = !in_src;
    }
    if (!in_src)
      for (int64_t i = threadIdx.x; i < len; i += blockDim.x) src[i] = dst[i];
    __syncthreads();
  }
}

// ---- sort by row ---------------------------------------------------------
// An entry on its way to its row: position in the source, column, value bits
// (16 bytes, so that one aligned store brings it there).
struct __align__(16) RowRecord {
  uint32_t i;
  int32_t col;
  uint64_t val;
};
__device__ __forceinline__ RowRecord load_record(const RowRecord* p) {
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  return RowRecord{u.x, (int32_t)u.y, (uint64_t)u.z | ((uint64_t)u.w << 32)};
}
__device__ __forceinline__ uint64_t bits_of(double v) { return (uint64_t)__double_as_longlong(v); }
__device__ __forceinline__ uint64_t bits_of(float v) { return (uint64_t)__float_as_uint(v); }
template <typename T> __device__ __forceinline__ T value_of(uint64_t b);
template <> __device__ __forceinline__ double value_of<double>(uint64_t b) { return __longlong_as_double((long long)b); }
template <> __device__ __forceinline__ float value_of<float>(uint64_t b) { return __uint_as_float((unsigned)b); }

// The order within a row: by source position (COLS false: a stable partition
// by row), or by column and then position.
template <bool COLS>
__device__ __forceinline__ uint64_t record_key(const RowRecord& r) {
  return COLS ? ((uint64_t)(uint32_t)r.col << 32) | r.i : r.i;
}

// rank[i] = how many entries of the row came to its counter before (any
// order).  Lanes of a warp with the same row add once; the search for them is
// left out where no neighbouring lanes share a row.  *scattered = warps whose
// rows fall by more than a quarter of the matrix from one lane to the next.
__global__ void __launch_bounds__(256) row_ranks(const int32_t* __restrict__ rows, int64_t n, int64_t nrows,
                                                 int32_t* counts, int32_t* __restrict__ rank, int32_t* scattered) {
  __shared__ int32_t cta_falls;
  if (threadIdx.x == 0) cta_falls = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int32_t far = (int32_t)(nrows >> 2);
  int32_t falls = 0;
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;; i += (int64_t)gridDim.x * 256) {
    const bool in = i < n;
    const unsigned active = __ballot_sync(0xffffffffu, in);
    if (!active) break;
    const int32_t r = in ? __ldcs(rows + i) : -1;
    const int32_t up = __shfl_up_sync(0xffffffffu, r, 1);
    falls += __any_sync(0xffffffffu, in && lane > 0 && up - r > far);
    if (!__any_sync(0xffffffffu, in && lane > 0 && up == r)) {
      if (in) rank[i] = atomicAdd(counts + r, 1);
      continue;
    }
    const unsigned same = __match_any_sync(0xffffffffu, r);
    const int leader = __ffs(same) - 1;
    int32_t base = 0;
    if (in && lane == leader) base = atomicAdd(counts + r, __popc(same));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (in) rank[i] = base + __popc(same & ((1u << lane) - 1));
  }
  if (lane == 0 && falls) atomicAdd(&cta_falls, falls);
  __syncthreads();
  if (threadIdx.x == 0 && cta_falls) atomicAdd(scattered, cta_falls);
}

// Records to their rows.  Each is one 16-byte store, half a sector, to a
// place that only its row tells: while the records stay within L2 (129 MB) the
// other half of the sector arrives before the sector is written back.  Beyond
// that, entries in arbitrary order are written for the lower and then the
// upper half of the rows (PASS 1 and 2, each reads all of `rows`); entries
// whose rows are near each other in most warps (*scattered tells) need no
// second pass and pay an empty launch.  PASS 0: everything at once.
// CSR from shuffled triplets, one pass -> two: 15.2M entries (power law) 960
// -> 909 us, 19.3M (27 diagonals, FP32) 1,040 -> 943, 45M 3,200 -> 2,940;
// 7.6M (121 MB) 501 -> 500, 4.6M 341 -> 354, which is why the line is at L2's
// size; three passes were worth 0.5-2 % beyond 30M only.  Row-sorted triplets,
// 16M: 508 in one pass, 517 with an empty second, 542 in two.
constexpr int64_t SCATTER_L2 = (int64_t)128 << 20;
template <typename T, int PASS>
__global__ void __launch_bounds__(256) row_scatter(const int32_t* __restrict__ rows, const int32_t* __restrict__ cols,
                                                   const T* __restrict__ vals, const int32_t* __restrict__ start,
                                                   const int32_t* __restrict__ rank, int64_t n, int64_t nrows,
                                                   const int32_t* __restrict__ scattered, RowRecord* rec) {
  const bool halves = PASS != 0 && __ldg(scattered) > n / 64;
  if (PASS == 2 && !halves) return;
  const int32_t mid = (int32_t)(nrows >> 1);
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
    const int32_t r = __ldcs(rows + i);
    if (PASS == 1 && halves && r >= mid) continue;
    if (PASS == 2 && r < mid) continue;
    const int64_t at = (int64_t)__ldg(start + r) + __ldcs(rank + i);
    const uint64_t v = bits_of(__ldcs(vals + i));
    reinterpret_cast<uint4*>(rec)[at] =
        make_uint4((unsigned)i, (unsigned)__ldcs(cols + i), (unsigned)v, (unsigned)(v >> 32));
  }
}

// Rows of at most SORT_SHORT entries are sorted in tiles: CTA t takes the rows
// that start in [t, t + 1) * SORT_WINDOW.  Longer ones are listed (lists: medium
// ones first, then those beyond SORT_MED).
constexpr int SORT_WINDOW = 1024;
constexpr int SORT_SHORT = 512;
constexpr int SORT_MED = 4096;
constexpr int SORT_CAP = SORT_WINDOW + SORT_SHORT;  // entries of a tile, a long last row left out
constexpr int SORT_PER = SORT_CAP / 256;

__global__ void sort_plan(const int32_t* __restrict__ start, int64_t nrows, int64_t ntiles, int32_t* tile_row,
                          int32_t* medium, int32_t* large, int32_t* counters) {
  const int lane = threadIdx.x & 31;
  for (int64_t r0 = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); r0 <= nrows;
       r0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = r0 + lane;
    int len = 0;
    if (r <= nrows) {
      const int64_t s = start[r];
      const int64_t k_lo = r == 0 ? 0 : (int64_t)start[r - 1] / SORT_WINDOW + 1;
      const int64_t k_hi = r == nrows ? ntiles : s / SORT_WINDOW;
      for (int64_t k = k_lo; k <= k_hi; k++) tile_row[k] = (int32_t)r;
      if (r < nrows) len = start[r + 1] - (int32_t)s;
    }
#pragma unroll
    for (int cls = 0; cls < 2; cls++) {
      const bool mine = cls == 0 ? len > SORT_SHORT && len <= SORT_MED : len > SORT_MED;
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (!m) continue;
      int32_t base = 0;
      if (lane == __ffs(m) - 1) base = atomicAdd(counters + cls, __popc(m));
      base = __shfl_sync(0xffffffffu, base, __ffs(m) - 1);
      if (mine) (cls == 0 ? medium : large)[base + __popc(m & ((1u << lane) - 1))] = (int32_t)r;
    }
  }
}

// One thread per entry: its place is its row's start plus the number of
// smaller keys in the row, counted over the row's keys in shared memory (the
// lanes of a row read the same word).  Sorting each row with a warp's or a
// CTA's bitonic network spent 1,100 us on the 1e6 lognormal rows (15 M entries)
// that this kernel sorts with the gather of columns and values in: rows of
// 15 entries leave most of a network's lanes idle, and its barriers bound it.
template <typename T, bool COLS>
__global__ void __launch_bounds__(256)
sort_tiles(const RowRecord* __restrict__ rec, const int32_t* __restrict__ start, const int32_t* __restrict__ tile_row,
           int32_t* __restrict__ orow, int32_t* __restrict__ ocol, T* __restrict__ oval) {
  using Key = typename std::conditional<COLS, uint64_t, uint32_t>::type;
  __shared__ Key s_key[SORT_CAP];
  __shared__ uint16_t s_head[SORT_CAP], s_end[SORT_CAP];  // an entry's row start; at a row start, the row's end
  __shared__ int32_t s_row[SORT_CAP];                     // at a row start, the row
  __shared__ int s_warp[8];
  const int64_t r0 = tile_row[blockIdx.x], r1 = tile_row[blockIdx.x + 1];
  if (r0 >= r1) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int32_t base = start[r0];
  int32_t end = start[r1];
  if (end - start[r1 - 1] > SORT_SHORT) end = start[r1 - 1];  // a long last row
  const int m = end - base;
  for (int e = threadIdx.x; e < SORT_CAP; e += 256) s_head[e] = 0;
  RowRecord mine[SORT_PER];
#pragma unroll
  for (int k = 0; k < SORT_PER; k++) {
    const int e = k * 256 + threadIdx.x;
    if (e < m) {
      mine[k] = load_record(rec + base + e);
      s_key[e] = (Key)record_key<COLS>(mine[k]);
    }
  }
  __syncthreads();
  for (int64_t r = r0 + threadIdx.x; r < r1; r += 256) {
    const int b = start[r] - base, t = start[r + 1] - base;
    if (b < t && b < m) {
      s_head[b] = (uint16_t)b;
      s_end[b] = (uint16_t)(t - b > SORT_SHORT ? b : t);  // a long row inside the tile: nothing to do here
      s_row[b] = (int32_t)r;
    }
  }
  __syncthreads();
  // every entry's row start: the largest marked position up to it
  int run[SORT_PER];
  int top = 0;
#pragma unroll
  for (int k = 0; k < SORT_PER; k++) run[k] = top = max(top, (int)s_head[threadIdx.x * SORT_PER + k]);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, top, d);
    if (lane >= d) top = max(top, o);
  }
  if (lane == 31) s_warp[w] = top;
  int before = __shfl_up_sync(0xffffffffu, top, 1);
  if (lane == 0) before = 0;
  __syncthreads();
  for (int i = 0; i < w; i++) before = max(before, s_warp[i]);
#pragma unroll
  for (int k = 0; k < SORT_PER; k++) s_head[threadIdx.x * SORT_PER + k] = (uint16_t)max(run[k], before);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < SORT_PER; k++) {
    const int e = k * 256 + threadIdx.x;
    if (e >= m) break;
    const int h = s_head[e], t = s_end[h];
    if (t == h) continue;
    const Key key = s_key[e];
    int at = h;
#pragma unroll 4
    for (int j = h; j < t; j++) at += s_key[j] < key ? 1 : 0;
    if (orow != nullptr) orow[base + at] = s_row[h];
    ocol[base + at] = mine[k].col;
    oval[base + at] = value_of<T>(mine[k].val);
  }
}

constexpr int SORT_LONG_THREADS = 512;
constexpr int SORT_RUN = 128;

// The order of up to SORT_MED records by one CTA: mine[k] (record
// k * SORT_LONG_THREADS + threadIdx.x of rec) belongs at pos[k].  Every thread
// keeps its records in registers and only moves keys: the place in a run of
// SORT_RUN by counting, then doubled runs by one binary search of the
// neighbouring run per level.  (A bitonic network over 16-byte records: 129 us
// where a few rows of thousands of entries are all there is.)
constexpr int SORT_LONG_PER = SORT_MED / SORT_LONG_THREADS;
template <bool COLS>
using SortKey = typename std::conditional<COLS, uint64_t, uint32_t>::type;

template <bool COLS>
__device__ __forceinline__ void order_records(const RowRecord* __restrict__ rec, int len, RowRecord* mine, int* pos,
                                              SortKey<COLS>* from, SortKey<COLS>* to) {
  using Key = SortKey<COLS>;
#pragma unroll
  for (int k = 0; k < SORT_LONG_PER; k++) {
    const int e = k * SORT_LONG_THREADS + threadIdx.x;
    if (e < len) {
      mine[k] = load_record(rec + e);
      from[e] = (Key)record_key<COLS>(mine[k]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < SORT_LONG_PER; k++) {
    const int e = k * SORT_LONG_THREADS + threadIdx.x;
    if (e < len) {
      const int c0 = e & ~(SORT_RUN - 1), c1 = min(c0 + SORT_RUN, len);
      const Key key = (Key)record_key<COLS>(mine[k]);
      int at = c0;
#pragma unroll 8
      for (int j = c0; j < c1; j++) at += from[j] < key ? 1 : 0;
      pos[k] = at;
      to[at] = key;
    }
  }
  __syncthreads();
  for (int width = SORT_RUN; width < len; width <<= 1) {
    Key* t = from;
    from = to;
    to = t;
#pragma unroll
    for (int k = 0; k < SORT_LONG_PER; k++) {
      const int e = k * SORT_LONG_THREADS + threadIdx.x;
      if (e < len) {
        const Key key = (Key)record_key<COLS>(mine[k]);
        const int own = pos[k] & ~(width - 1), other = own ^ width;
        int lo = min(other, len), hi = min(other + width, len);
        const int first = lo;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (from[mid] < key) lo = mid + 1; else hi = mid;
        }
        pos[k] = min(own, other) + (pos[k] - own) + (lo - first);
        to[pos[k]] = key;
      }
    }
    __syncthreads();
  }
}

// One CTA per row of SORT_SHORT < length <= SORT_MED.
template <typename T, bool COLS>
__global__ void __launch_bounds__(SORT_LONG_THREADS, 2)
sort_medium_rows(const RowRecord* __restrict__ rec, const int32_t* __restrict__ start,
                 const int32_t* __restrict__ list, const int32_t* __restrict__ count, int32_t* __restrict__ orow,
                 int32_t* __restrict__ ocol, T* __restrict__ oval) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  SortKey<COLS>* keys = reinterpret_cast<SortKey<COLS>*>(sort_smem);
  for (int64_t w = blockIdx.x; w < *count; w += gridDim.x) {
    const int32_t r = list[w];
    const int32_t b = start[r], len = start[r + 1] - b;
    RowRecord mine[SORT_LONG_PER];
    int pos[SORT_LONG_PER];
    order_records<COLS>(rec + b, len, mine, pos, keys, keys + SORT_MED);
#pragma unroll
    for (int k = 0; k < SORT_LONG_PER; k++) {
      if (k * SORT_LONG_THREADS + (int)threadIdx.x < len) {
        if (orow != nullptr) orow[b + pos[k]] = r;
        ocol[b + pos[k]] = mine[k].col;
        oval[b + pos[k]] = value_of<T>(mine[k].val);
      }
    }
    __syncthreads();  // the next row's keys
  }
}

// Rows beyond SORT_MED, in pieces of SORT_MED records (x: row, y: piece) that
// CTAs take: each piece is ordered by itself, then runs of doubled length are
// merged, one launch per level, a CTA per piece of the output.  (One CTA per row
// for all of it: sorting a row of 2e6 entries 118 ms, with pieces 0.8.)
// The runs alternate between rec and tmp; a row is done, where it is then, when
// it is one run.
__device__ __forceinline__ int merge_levels(int64_t len) {
  int n = 0;
  for (int64_t width = SORT_MED; width < len; width <<= 1) n++;
  return n;
}

__global__ void list_sort_pieces(const int32_t* __restrict__ start, const int32_t* __restrict__ list,
                                 const int32_t* __restrict__ count, int2* pieces, int32_t* npieces) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < *count; w += warps) {
    const int32_t r = list[w];
    const int32_t n = (int32_t)(((int64_t)start[r + 1] - start[r] + SORT_MED - 1) / SORT_MED);
    int32_t at = 0;
    if (lane == 0) at = atomicAdd(npieces, n);
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int32_t i = lane; i < n; i += 32) pieces[at + i] = make_int2(r, i);
  }
}

template <bool COLS>
__global__ void __launch_bounds__(SORT_LONG_THREADS, 2)
sort_pieces(RowRecord* rec, const int32_t* __restrict__ start, const int2* __restrict__ pieces,
            const int32_t* __restrict__ npieces) {
  extern __shared__ __align__(16) unsigned char sort_smem[];
  SortKey<COLS>* keys = reinterpret_cast<SortKey<COLS>*>(sort_smem);
  for (int32_t p = blockIdx.x; p < *npieces; p += gridDim.x) {
    const int2 piece = pieces[p];
    const int64_t b = start[piece.x] + (int64_t)piece.y * SORT_MED;
    const int len = (int)min((int64_t)SORT_MED, start[piece.x + 1] - b);
    RowRecord mine[SORT_LONG_PER];
    int pos[SORT_LONG_PER];
    order_records<COLS>(rec + b, len, mine, pos, keys, keys + SORT_MED);
#pragma unroll
    for (int k = 0; k < SORT_LONG_PER; k++)
      if (k * SORT_LONG_THREADS + (int)threadIdx.x < len) rec[b + pos[k]] = mine[k];
    __syncthreads();  // the next piece's keys
  }
}

// number of records taken from a among the first k of a and b merged
template <bool COLS>
__device__ int64_t merge_corank(const RowRecord* a, int64_t na, const RowRecord* b, int64_t nb, int64_t k) {
  int64_t lo = k > nb ? k - nb : 0, hi = k < na ? k : na;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (record_key<COLS>(a[mid]) <= record_key<COLS>(b[k - mid - 1])) lo = mid + 1; else hi = mid;
  }
  return lo;
}

template <bool COLS>
__global__ void __launch_bounds__(SORT_LONG_THREADS)
merge_pieces(const RowRecord* __restrict__ src, RowRecord* __restrict__ dst, const int32_t* __restrict__ start,
             const int2* __restrict__ pieces, const int32_t* __restrict__ npieces, int64_t width) {
  __shared__ SortKey<COLS> s_key[SORT_MED];
  __shared__ int64_t s_from[2];
  for (int32_t p = blockIdx.x; p < *npieces; p += gridDim.x) {
    const int2 piece = pieces[p];
    const int64_t b = start[piece.x], len = start[piece.x + 1] - b;
    if (len <= width) continue;
    const int64_t k0 = (int64_t)piece.y * SORT_MED, k1 = min(k0 + SORT_MED, len);
    const int64_t a0 = k0 / (2 * width) * (2 * width);  // the pair of runs that the piece lies in
    const int64_t na = min(width, len - a0), nb = max((int64_t)0, min(width, len - a0 - width));
    const RowRecord *A = src + b + a0, *B = A + na;
    if (threadIdx.x < 2) s_from[threadIdx.x] = merge_corank<COLS>(A, na, B, nb, (threadIdx.x ? k1 : k0) - a0);
    __syncthreads();
    const int64_t ia = s_from[0], ib = k0 - a0 - ia;
    const int m = (int)(k1 - k0), ma = (int)(s_from[1] - ia);  // records of the piece, those from A
    RowRecord mine[SORT_LONG_PER];
#pragma unroll
    for (int k = 0; k < SORT_LONG_PER; k++) {
      const int e = k * SORT_LONG_THREADS + threadIdx.x;
      if (e < m) {
        mine[k] = load_record(e < ma ? A + ia + e : B + ib + (e - ma));
        s_key[e] = (SortKey<COLS>)record_key<COLS>(mine[k]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < SORT_LONG_PER; k++) {
      const int e = k * SORT_LONG_THREADS + threadIdx.x;
      if (e < m) {
        const SortKey<COLS> key = (SortKey<COLS>)record_key<COLS>(mine[k]);
        int lo = e < ma ? ma : 0, hi = e < ma ? m : ma;
        const int first = lo;
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (s_key[mid] < key) lo = mid + 1; else hi = mid;
        }
        dst[b + k0 + (e < ma ? e : e - ma) + (lo - first)] = mine[k];
      }
    }
    __syncthreads();  // the next piece's keys
  }
}

template <typename T>
__global__ void __launch_bounds__(SORT_LONG_THREADS)
write_pieces(const RowRecord* __restrict__ rec, const RowRecord* __restrict__ tmp, const int32_t* __restrict__ start,
             const int2* __restrict__ pieces, const int32_t* __restrict__ npieces, int32_t* __restrict__ orow,
             int32_t* __restrict__ ocol, T* __restrict__ oval) {
  for (int32_t p = blockIdx.x; p < *npieces; p += gridDim.x) {
    const int2 piece = pieces[p];
    const int64_t b = start[piece.x], end = start[piece.x + 1];
    const RowRecord* from = merge_levels(end - b) & 1 ? tmp : rec;
    const int64_t k0 = b + (int64_t)piece.y * SORT_MED, k1 = min(k0 + SORT_MED, end);
    for (int64_t k = k0 + threadIdx.x; k < k1; k += SORT_LONG_THREADS) {
      const RowRecord x = load_record(from + k);
      if (orow != nullptr) orow[k] = piece.x;
      ocol[k] = x.col;
      oval[k] = value_of<T>(x.val);
    }
  }
}

}  // namespace

template <typename Tin, typename Tout>
int exclusive_scan(const Tin* in, Tout* out, int64_t n, cudaStream_t s, int64_t* d_total) {
  if (n <= 0) {
    if (d_total) MGB_CUDA_CHECK(cudaMemsetAsync(d_total, 0, sizeof(int64_t), s));
    return MGB_SUCCESS;
  }
  Scratch sc(s);
  const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
  int64_t* sums;
  MGB_SCRATCH(sc, sums, nb);
  scan_tile_sums<Tin><<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, n, sums);
  MGB_LAUNCH_CHECK();
  scan_sums<<<1, 1024, 0, s>>>(sums, nb, d_total);
  MGB_LAUNCH_CHECK();
  scan_apply<Tin, Tout><<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, out, n, sums);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

template int exclusive_scan<int32_t, int32_t>(const int32_t*, int32_t*, int64_t, cudaStream_t, int64_t*);
template int exclusive_scan<uint8_t, int64_t>(const uint8_t*, int64_t*, int64_t, cudaStream_t, int64_t*);
template int exclusive_scan<uint8_t, int32_t>(const uint8_t*, int32_t*, int64_t, cudaStream_t, int64_t*);

int reduce_max_i32(const int32_t* in, int64_t n, int32_t* d_out, cudaStream_t s) {
  fill_i32<<<1, 32, 0, s>>>(d_out, INT_MIN, 1);
  MGB_LAUNCH_CHECK();
  if (n <= 0) return MGB_SUCCESS;
  max_i32_kernel<<<blocks_for(n, 256, (int64_t)num_sms() * 8), 256, 0, s>>>(in, n, d_out);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int histogram(const int32_t* keys, int64_t n, int32_t* counts, int64_t nbins, cudaStream_t s) {
  MGB_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int32_t) * (nbins > 0 ? nbins : 0), s));
  if (n <= 0 || nbins <= 0) return MGB_SUCCESS;
  histogram_kernel<<<blocks_for(n, 256, (int64_t)num_sms() * 16), 256, 0, s>>>(keys, n, counts, nbins);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int coo_sorted_flags(const int32_t* rows, const int32_t* cols, int64_t n, int32_t* d_flag, int32_t* d_dup,
                     cudaStream_t s) {
  fill_i32<<<1, 32, 0, s>>>(d_flag, 1, 1);
  MGB_LAUNCH_CHECK();
  if (d_dup) MGB_CUDA_CHECK(cudaMemsetAsync(d_dup, 0, sizeof(int32_t), s));
  if (n <= 1) return MGB_SUCCESS;
  sorted_flags_kernel<<<blocks_for(n, 256, (int64_t)num_sms() * 16), 256, 0, s>>>(rows, cols, n, d_flag, d_dup);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int words_alloc(Scratch& sc, Words** d, cudaStream_t s) {
  MGB_SCRATCH(sc, *d, 1);
  MGB_CUDA_CHECK(cudaMemsetAsync(*d, 0, sizeof(Words), s));
  return MGB_SUCCESS;
}

int words_read(const Words* d, Words* h, cudaStream_t s) { return to_host(d, h, s); }

int64_t gap_words(int64_t nrows) { return max_gaps(nrows) + max_huge(nrows); }

int coo_pass(const int32_t* rows, const int32_t* cols, int64_t n, int64_t nrows, int64_t ncols, Words* d,
             int32_t* diag, int32_t* start, int32_t* gaps, bool huge, cudaStream_t s) {
  const int64_t nb = nrows + ncols - 1;
  if (diag != nullptr && nb > 0) MGB_CUDA_CHECK(cudaMemsetAsync(diag, 0, sizeof(int32_t) * nb, s));
  if (n <= 0 && start == nullptr) return MGB_SUCCESS;
  const bool vec = (reinterpret_cast<uintptr_t>(rows) | reinterpret_cast<uintptr_t>(cols)) % 16 == 0;
  const unsigned grid = blocks_for(n / 4 + 1, 256, (int64_t)num_sms() * 8);
  const auto run = [&](auto kernel) {
    kernel<<<grid, 256, 0, s>>>(rows, cols, n, nrows, ncols, vec, d, diag, start, gaps);
  };
  if (diag != nullptr && start != nullptr && huge) run(coo_pass_kernel<true, true, true>);
  else if (diag != nullptr && start != nullptr) run(coo_pass_kernel<true, true, false>);
  else if (diag != nullptr) run(coo_pass_kernel<true, false, false>);
  else if (start != nullptr) run(coo_pass_kernel<false, true, true>);
  else run(coo_pass_kernel<false, false, false>);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int csr_pass(const int32_t* ro, const int32_t* cols, int64_t n, int64_t nrows, int64_t ncols, Words* d,
             int32_t* diag, int2* pieces, cudaStream_t s) {
  const int64_t nb = nrows + ncols - 1;
  if (diag != nullptr && nb > 0) MGB_CUDA_CHECK(cudaMemsetAsync(diag, 0, sizeof(int32_t) * nb, s));
  if (nrows <= 0) return MGB_SUCCESS;
  const RowPieces longs{pieces, &d->pieces, max_row_pieces(n)};
  const unsigned grid = blocks_for(nrows, 256, (int64_t)num_sms() * DIAG_CTAS);
  if (diag != nullptr) csr_pass_kernel<true><<<grid, 256, 0, s>>>(ro, cols, n, nrows, ncols, &d->seen, diag, longs);
  else csr_pass_kernel<false><<<grid, 256, 0, s>>>(ro, cols, n, nrows, ncols, &d->seen, diag, longs);
  MGB_LAUNCH_CHECK();
  if (n <= LONG_GROUP) return MGB_SUCCESS;
  const unsigned pgrid = blocks_for(longs.limit, 1, (int64_t)num_sms() * 4);
  if (diag != nullptr) csr_pass_pieces<true><<<pgrid, 256, 0, s>>>(ro, cols, nrows, ncols, &d->seen, diag, longs);
  else csr_pass_pieces<false><<<pgrid, 256, 0, s>>>(ro, cols, nrows, ncols, &d->seen, diag, longs);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int coo_pass_gaps(const int32_t* rows, int64_t nrows, Words* d, const int32_t* gaps, int32_t* start, cudaStream_t s) {
  fill_gaps<<<blocks_for(nrows, 1024, (int64_t)num_sms() * 8), 256, 0, s>>>(rows, nrows, d, gaps, start);
  MGB_LAUNCH_CHECK();
  MGB_CUDA_CHECK(cudaMemsetAsync(&d->total, 0, 2 * sizeof(int64_t), s));
  MGB_CUDA_CHECK(cudaMemsetAsync(&d->maxv, 0, 3 * sizeof(int32_t), s));  // and gaps, huge
  return MGB_SUCCESS;
}

int64_t bin_tiles(int64_t nb) { return (nb + SCAN_TILE - 1) / SCAN_TILE; }

int select_bins(const int32_t* counts, int64_t nb, int32_t threshold, int64_t* sums, int64_t* d_total, int64_t* d_sum,
                cudaStream_t s) {
  bin_tile_sums<<<(unsigned)bin_tiles(nb), SCAN_THREADS, 0, s>>>(counts, nb, threshold, sums,
                                                                 reinterpret_cast<unsigned long long*>(d_sum));
  MGB_LAUNCH_CHECK();
  scan_sums<<<1, 1024, 0, s>>>(sums, bin_tiles(nb), d_total);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int select_bins_apply(int32_t* counts, int64_t nb, int32_t threshold, const int64_t* sums, int64_t nrows,
                      int64_t zero_bin, int32_t* offsets, cudaStream_t s) {
  bin_apply<<<(unsigned)bin_tiles(nb), SCAN_THREADS, 0, s>>>(counts, nb, threshold, sums, nrows, zero_bin, offsets);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

int segmented_sort_u64(uint64_t* keys, const int32_t* seg, int64_t nseg, int64_t nkeys, cudaStream_t s) {
  if (nseg <= 0 || nkeys <= 1) return MGB_SUCCESS;
  Scratch sc(s);
  int32_t* lists;
  int32_t* counters;
  MGB_SCRATCH(sc, lists, 3 * nseg);
  MGB_SCRATCH(sc, counters, 4);
  MGB_CUDA_CHECK(cudaMemsetAsync(counters, 0, 4 * sizeof(int32_t), s));
  classify_segments<<<blocks_for(nseg, 256, (int64_t)num_sms() * 16), 256, 0, s>>>(seg, nseg, lists, nseg, counters);
  MGB_LAUNCH_CHECK();
  int32_t h[4];
  MGB_CUDA_CHECK(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, s));
  MGB_CUDA_CHECK(cudaStreamSynchronize(s));
  if (h[0] > 0) {
    sort_small_segments<<<blocks_for((int64_t)h[0] * 32, 256, (int64_t)num_sms() * 32), 256, 0, s>>>(
        keys, seg, lists, counters);
    MGB_LAUNCH_CHECK();
  }
  if (h[1] > 0) {
    sort_medium_segments<<<(unsigned)min((int64_t)h[1], (int64_t)num_sms() * 8), SEG_MED_THREADS, 0, s>>>(
        keys, seg, lists + nseg, counters + 1);
    MGB_LAUNCH_CHECK();
  }
  if (h[2] > 0) {
    uint64_t* tmp;
    MGB_SCRATCH(sc, tmp, nkeys);
    sort_large_segments<<<(unsigned)min((int64_t)h[2], (int64_t)num_sms() * 4), SEG_MED_THREADS, 0, s>>>(
        keys, tmp, seg, lists + 2 * nseg, counters + 2);
    MGB_LAUNCH_CHECK();
  }
  return MGB_SUCCESS;
}

int64_t row_sort_bytes(int64_t n, int64_t nrows) {
  return (int64_t)(Scratch::padded(sizeof(RowRecord) * (size_t)n) + Scratch::padded(sizeof(int32_t) * (size_t)n) +
                   2 * Scratch::padded(sizeof(int32_t) * (size_t)(nrows + 1)) +
                   Scratch::padded(sizeof(int32_t) * (size_t)(n / SORT_WINDOW + 2)) +
                   Scratch::padded(sizeof(int32_t) * (size_t)(n / SORT_SHORT + 1)) +
                   Scratch::padded(sizeof(int32_t) * (size_t)(n / SORT_MED + 1)) + 256);
}

template <typename T, bool COLS>
int row_sort(const int32_t* rows, const int32_t* cols, const T* vals, int64_t n, int64_t nrows, int32_t* start,
             int32_t* orow, int32_t* ocol, T* oval, Scratch& sc, cudaStream_t s) {
  RowRecord* rec;
  int32_t *counts, *rank, *tile_row, *medium, *large, *counters;
  MGB_SCRATCH(sc, rec, n);
  MGB_SCRATCH(sc, rank, n);
  MGB_SCRATCH(sc, counts, nrows + 1);
  if (start == nullptr) MGB_SCRATCH(sc, start, nrows + 1);
  const int64_t ntiles = n / SORT_WINDOW + 1;
  MGB_SCRATCH(sc, tile_row, ntiles + 1);
  MGB_SCRATCH(sc, medium, n / SORT_SHORT + 1);
  MGB_SCRATCH(sc, large, n / SORT_MED + 1);
  MGB_SCRATCH(sc, counters, 3);  // medium rows, large rows, scattered warps
  MGB_CUDA_CHECK(cudaMemsetAsync(counts, 0, sizeof(int32_t) * (nrows + 1), s));
  MGB_CUDA_CHECK(cudaMemsetAsync(counters, 0, 3 * sizeof(int32_t), s));
  const unsigned grid = blocks_for(n, 256, (int64_t)num_sms() * 8);
  row_ranks<<<grid, 256, 0, s>>>(rows, n, nrows, counts, rank, counters + 2);
  MGB_LAUNCH_CHECK();
  int st = exclusive_scan<int32_t, int32_t>(counts, start, nrows + 1, s);
  if (st) return st;
  if (n * (int64_t)sizeof(RowRecord) > SCATTER_L2) {
    row_scatter<T, 1><<<grid, 256, 0, s>>>(rows, cols, vals, start, rank, n, nrows, counters + 2, rec);
    MGB_LAUNCH_CHECK();
    row_scatter<T, 2><<<grid, 256, 0, s>>>(rows, cols, vals, start, rank, n, nrows, counters + 2, rec);
  } else {
    row_scatter<T, 0><<<grid, 256, 0, s>>>(rows, cols, vals, start, rank, n, nrows, counters + 2, rec);
  }
  MGB_LAUNCH_CHECK();
  sort_plan<<<blocks_for(nrows + 1, 256, (int64_t)num_sms() * 8), 256, 0, s>>>(start, nrows, ntiles, tile_row, medium,
                                                                                large, counters);
  MGB_LAUNCH_CHECK();
  int32_t h[2] = {0, 0};
  if (n > SORT_SHORT) {
    MGB_CUDA_CHECK(cudaMemcpyAsync(h, counters, sizeof(h), cudaMemcpyDeviceToHost, s));
    MGB_CUDA_CHECK(cudaStreamSynchronize(s));
  }
  sort_tiles<T, COLS><<<(unsigned)ntiles, 256, 0, s>>>(rec, start, tile_row, orow, ocol, oval);
  MGB_LAUNCH_CHECK();
  constexpr int keys = 2 * SORT_MED * (int)sizeof(SortKey<COLS>);
  if (h[0] > 0) {
    MGB_CUDA_CHECK(cudaFuncSetAttribute(sort_medium_rows<T, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, keys));
    sort_medium_rows<T, COLS><<<(unsigned)min((int64_t)h[0], (int64_t)num_sms() * 3), SORT_LONG_THREADS, keys, s>>>(
        rec, start, medium, counters, orow, ocol, oval);
    MGB_LAUNCH_CHECK();
  }
  if (h[1] > 0) {
    RowRecord* tmp;
    int2* pieces;
    int32_t* npieces;
    const int64_t most = 2 * (n / SORT_MED);  // a row's pieces are at least half full on average
    MGB_SCRATCH(sc, tmp, n);
    MGB_SCRATCH(sc, pieces, most);
    MGB_SCRATCH(sc, npieces, 1);
    MGB_CUDA_CHECK(cudaMemsetAsync(npieces, 0, sizeof(int32_t), s));
    list_sort_pieces<<<blocks_for(h[1], 8, (int64_t)num_sms() * 8), 256, 0, s>>>(start, large, counters + 1, pieces,
                                                                                npieces);
    MGB_LAUNCH_CHECK();
    const unsigned pgrid = blocks_for(most, 1, (int64_t)num_sms() * 4);
    MGB_CUDA_CHECK(cudaFuncSetAttribute(sort_pieces<COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize, keys));
    sort_pieces<COLS><<<pgrid, SORT_LONG_THREADS, keys, s>>>(rec, start, pieces, npieces);
    MGB_LAUNCH_CHECK();
    RowRecord *from = rec, *to = tmp;
    for (int64_t width = SORT_MED; width < n; width <<= 1) {
      merge_pieces<COLS><<<pgrid, SORT_LONG_THREADS, 0, s>>>(from, to, start, pieces, npieces, width);
      MGB_LAUNCH_CHECK();
      std::swap(from, to);
    }
    write_pieces<T><<<pgrid, SORT_LONG_THREADS, 0, s>>>(rec, tmp, start, pieces, npieces, orow, ocol, oval);
    MGB_LAUNCH_CHECK();
  }
  return MGB_SUCCESS;
}
#define MGB_ROW_SORT(T, COLS)                                                                                        \
  template int row_sort<T, COLS>(const int32_t*, const int32_t*, const T*, int64_t, int64_t, int32_t*, int32_t*,     \
                                 int32_t*, T*, Scratch&, cudaStream_t);
MGB_ROW_SORT(double, false)
MGB_ROW_SORT(double, true)
MGB_ROW_SORT(float, false)
MGB_ROW_SORT(float, true)

}  // namespace prim
}  // namespace mgb
