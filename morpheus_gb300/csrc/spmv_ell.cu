// spmv_ell.cu -- ELL and HYB SpMV for sm_103a.
//
// ELL replaces impl/Ell/Cuda/Morpheus_Multiply_Impl.hpp:41-80 (kernel
// impl/Ell/Kernels/Morpheus_Multiply_Impl.hpp:37-65).  Semantics are the
// Serial multiply (impl/Ell/Serial/Morpheus_Multiply_Impl.hpp:38-67): y = 0 if
// init, then for each row and each of the `width` padded slots whose column
// is not the invalid index (-1), y[i] += values(i, n) * x[col].
//
// HYB replaces impl/Hyb/Cuda/Morpheus_Multiply_Impl.hpp:42-53: the ELL part
// with init, then the COO part accumulating into y.
//
// Layout: slot (i, n) at [i + pitch * n], pitch = nrows (column-major, the
// reference's CUDA LayoutLeft).  Padding values are never read.  Three
// kernels; the rule and the figures are at launch_ell.
#include "mgb_internal.cuh"

namespace mgb {
namespace {

constexpr int ELL_THREADS = 256;

template <typename T, int RPT> struct EllVec;
template <> struct EllVec<double, 4> {
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2 a = __ldcs(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcs(reinterpret_cast<const double2*>(p) + 1);
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
  }
};
template <> struct EllVec<double, 2> {
  static __device__ __forceinline__ void load(const double* p, double* o) {
    const double2 v = __ldcs(reinterpret_cast<const double2*>(p)); o[0] = v.x; o[1] = v.y;
  }
};
template <typename T> struct EllVec<T, 1> {
  static __device__ __forceinline__ void load(const T* p, T* o) { o[0] = __ldcs(p); }
};

template <int RPT> struct IdxVec;
template <> struct IdxVec<4> {
  static __device__ __forceinline__ void load(const int32_t* p, int32_t* o) {
    const int4 v = __ldcs(reinterpret_cast<const int4*>(p)); o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
  }
};
template <> struct IdxVec<2> {
  static __device__ __forceinline__ void load(const int32_t* p, int32_t* o) {
    const int2 v = __ldcs(reinterpret_cast<const int2*>(p)); o[0] = v.x; o[1] = v.y;
  }
};
template <> struct IdxVec<1> {
  static __device__ __forceinline__ void load(const int32_t* p, int32_t* o) { o[0] = __ldcs(p); }
};

// RPT consecutive rows per thread, a slot at a time.  RPT = 4: one 16-byte load
// of the indices and, only where one of the 4 slots holds an entry, two of the
// values (RPT = 2: half of each); pitch and pointers have to allow it.
// MINB: resident CTAs of 256 threads per SM the kernel is compiled for (0:
// no register cap); the launcher picks it.
template <typename T, int RPT, int MINB>
__global__ void __launch_bounds__(ELL_THREADS, MINB)
spmv_ell_rows(int64_t nrows, int64_t ncols, int64_t width, int64_t pitch,
              const int32_t* __restrict__ ci, const T* __restrict__ va,
              const T* __restrict__ x, T* __restrict__ y, int init) {
  const int64_t ngroups = (nrows + RPT - 1) / RPT;
  for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row0 = g * RPT;
    const bool full = row0 + RPT <= nrows;
    T acc[RPT];
#pragma unroll
    for (int i = 0; i < RPT; i++) acc[i] = (row0 + i < nrows && !init) ? y[row0 + i] : T(0);
    for (int64_t n = 0; n < width; n++) {
      const int64_t base = row0 + pitch * n;
      int32_t c[RPT];
      if (full) {
        IdxVec<RPT>::load(ci + base, c);
      } else {
#pragma unroll
        for (int i = 0; i < RPT; i++) c[i] = (row0 + i < nrows) ? __ldcs(ci + base + i) : -1;
      }
      bool any = false;
#pragma unroll
      for (int i = 0; i < RPT; i++) any |= ((uint64_t)(int64_t)c[i] < (uint64_t)ncols);
      if (any) {
        T v[RPT];
        if (full) {
          EllVec<T, RPT>::load(va + base, v);
        } else {
#pragma unroll
          for (int i = 0; i < RPT; i++) v[i] = (row0 + i < nrows) ? __ldcs(va + base + i) : T(0);
        }
#pragma unroll
        for (int i = 0; i < RPT; i++)
          if ((uint64_t)(int64_t)c[i] < (uint64_t)ncols) acc[i] = fmadd(v[i], __ldg(x + c[i]), acc[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < RPT; i++)
      if (row0 + i < nrows) y[row0 + i] = acc[i];
  }
}

// A thread per row, B slots at a time: their indices are loaded a step ahead,
// their values and x elements are in flight together, and a slot that no row
// of the warp fills takes no FMA (the FP64 pipe is busy for the slot even
// where no lane has work).  The sums run in slot order.
constexpr int ELL_PAIR_THREADS = 128;

template <typename T, int B>
__global__ void __launch_bounds__(ELL_PAIR_THREADS, 16)
spmv_ell_pairs(int64_t nrows, int64_t ncols, int64_t width, int64_t pitch, const int32_t* __restrict__ ci,
               const T* __restrict__ va, const T* __restrict__ x, T* __restrict__ y, int init) {
  const int64_t row = (int64_t)blockIdx.x * ELL_PAIR_THREADS + threadIdx.x;
  if (row >= nrows) return;
  T acc = init ? T(0) : y[row];
  const int32_t* cp = ci + row;
  const T* vp = va + row;
  int32_t c[B];
#pragma unroll
  for (int u = 0; u < B; u++) c[u] = u < width ? __ldcs(cp + u * pitch) : -1;
  for (int64_t k0 = 0; k0 < width; k0 += B, vp += B * pitch) {
    cp += B * pitch;
    int32_t next[B];
#pragma unroll
    for (int u = 0; u < B; u++) next[u] = k0 + B + u < width ? __ldcs(cp + u * pitch) : -1;
    T v[B], xv[B];
#pragma unroll
    for (int u = 0; u < B; u++)
      if ((uint64_t)(int64_t)c[u] < (uint64_t)ncols) {
        v[u] = __ldcs(vp + u * pitch);
        xv[u] = __ldg(x + c[u]);
      }
#pragma unroll
    for (int u = 0; u < B; u++) {
      const bool in = (uint64_t)(int64_t)c[u] < (uint64_t)ncols;
      if (__any_sync(__activemask(), in)) {
        if (in) acc = fmadd(v[u], xv[u], acc);
      }
    }
#pragma unroll
    for (int u = 0; u < B; u++) c[u] = next[u];
  }
  y[row] = acc;
}

}  // namespace

template <typename T, int RPT, int MINB>
int launch_ell_rows(const mgb_ell* A, const T* x, T* y, int init, cudaStream_t s) {
  const int64_t groups = (A->nrows + RPT - 1) / RPT;
  int64_t blocks = (groups + ELL_THREADS - 1) / ELL_THREADS;
  const int64_t cap = (int64_t)num_sms() * 64;
  if (blocks > cap) blocks = cap;
  spmv_ell_rows<T, RPT, MINB><<<(unsigned)blocks, ELL_THREADS, 0, s>>>(
      A->nrows, A->ncols, A->width, A->pitch, A->column_indices, static_cast<const T*>(A->values), x, y, init);
  MGB_LAUNCH_CHECK();
  return MGB_SUCCESS;
}

// Which kernel (us on one GB300; p: pairs, 1 / 4: rows per thread of spmv_ell_rows):
//                                     FP64   p     1     4        FP32   p     1     4
//   27-point stencil, 195,112 rows        16.4  18.4  39.7          16.4  15.2  29.9
//                     1,000,000           63.8  65.6  87.8          58.7  41.2  48.7
//                     4,096,000          236   246   241           212   154   173
//   power-law HYB part, width 34 -> 64 (with its COO part)
//                        50,000 rows      34.9  39.0  48.2          30.7  24.6  44.6
//                       400,000           86.5 101    92.2          86.9  62.4  90.3
//                     1,234,567          206   228    -            192   145    -
//                     2,000,000          297   330   279           278   204   240
//   5-point stencil,    202,500 rows      16.8  20.5  20.5          16.0  14.9  16.3
//                     1,000,000           61.7  69.8  47.0          49.8  30.7  30.8
//                     4,194,304          232   256   145           182   107   109
//   9-point stencil,  2,254,502           128    -    96 (2 rows)   -     64    90 (2 rows)
// FP32: one row per thread everywhere (8 CTAs per SM).  FP64: pairs, except
// mostly-padding slabs of more rows than threads fit the GPU, where four rows
// per thread (two where the pitch is not a multiple of 4) read the padding's
// indices in the fewest instructions.  At that line (311,296 rows on 152 SMs) and
// above, four / pairs: 5-point 324,900 rows 24.6 / 25.5, 518,400 25.9 / 36.4, 722,500
// 28.7 / 47.1; 9-point 518,400 28.6 / 36.9; HYB part 320,000 82 / 76, 500,000 94 / 91,
// 600,000 98 / 110, 850,000 165 / 142, 1,200,000 184 / 191.  Between 0.3 and 0.5 M rows the
// two are within what the arrays' place in memory makes of it (21 to 25 us for the
// same slab of 324,900 rows).
template <typename T>
int launch_ell(const mgb_ell* A, const T* x, T* y, int init, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(!bad_sizes(A->nrows, A->ncols, A->nnz) && A->width >= 0, MGB_ERR_BAD_ARGUMENT);
  if (A->nrows == 0) return MGB_SUCCESS;
  MGB_REQUIRE(y != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(A->width == 0 || (A->pitch >= A->nrows && A->column_indices && A->values && x),
              MGB_ERR_BAD_ARGUMENT);
  if constexpr (sizeof(T) == 4) {
    return launch_ell_rows<T, 1, 8>(A, x, y, init, s);
  } else {
    const uintptr_t ap = reinterpret_cast<uintptr_t>(A->values), ai = reinterpret_cast<uintptr_t>(A->column_indices);
    const bool vec4 = (A->pitch % 4 == 0) && (ap % 16 == 0) && (ai % 16 == 0);
    const bool padded = 2 * A->nnz < A->nrows * A->width;
    const int64_t ctas = (A->nrows + ELL_PAIR_THREADS - 1) / ELL_PAIR_THREADS;
    const bool vec2 = (A->pitch % 2 == 0) && (ap % 16 == 0) && (ai % 8 == 0);
    if (padded && A->nrows > (int64_t)num_sms() * 2048) {
      if (vec4) return launch_ell_rows<T, 4, 0>(A, x, y, init, s);
      if (vec2) return launch_ell_rows<T, 2, 0>(A, x, y, init, s);
    }
    spmv_ell_pairs<T, 2><<<(unsigned)ctas, ELL_PAIR_THREADS, 0, s>>>(A->nrows, A->ncols, A->width, A->pitch,
                                                                     A->column_indices,
                                                                     static_cast<const T*>(A->values), x, y, init);
    MGB_LAUNCH_CHECK();
    return MGB_SUCCESS;
  }
}

template int launch_ell<double>(const mgb_ell*, const double*, double*, int, cudaStream_t);
template int launch_ell<float>(const mgb_ell*, const float*, float*, int, cudaStream_t);

template <typename T>
int launch_hyb(const mgb_hyb* A, const T* x, T* y, int init, cudaStream_t s) {
  MGB_REQUIRE(A != nullptr, MGB_ERR_BAD_ARGUMENT);
  MGB_REQUIRE(A->ell.nrows == A->coo.nrows, MGB_ERR_INVALID_INPUT);
  int st = launch_ell<T>(&A->ell, x, y, init, s);
  if (st != MGB_SUCCESS) return st;
  if (A->coo.nnz == 0) return MGB_SUCCESS;
  return launch_coo<T>(&A->coo, x, y, 0, s);
}

}  // namespace mgb

extern "C" {

int mgb_spmv_ell_f64(const mgb_ell* A, const double* x, double* y, int init, void* stream) {
  return mgb::launch_ell<double>(A, x, y, init, mgb::as_stream(stream));
}
int mgb_spmv_ell_f32(const mgb_ell* A, const float* x, float* y, int init, void* stream) {
  return mgb::launch_ell<float>(A, x, y, init, mgb::as_stream(stream));
}
int mgb_spmv_hyb_f64(const mgb_hyb* A, const double* x, double* y, int init, void* stream) {
  return mgb::launch_hyb<double>(A, x, y, init, mgb::as_stream(stream));
}
int mgb_spmv_hyb_f32(const mgb_hyb* A, const float* x, float* y, int init, void* stream) {
  return mgb::launch_hyb<float>(A, x, y, init, mgb::as_stream(stream));
}

}  // extern "C"
