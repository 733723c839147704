// spmv_sym.cu -- the products of SparseMatrixBase that scatter with atomic
// additions, for every segment format:
//  * vectorProduct of a symmetric matrix (SparseMatrixBase.hpp:296-330):
//    one triangle is stored; a stored a_rc with c < r also adds
//    alpha a_rc x[r] to y[c];
//  * transposedVectorProduct (SparseMatrixBase.hpp:542-588):
//    y[c] += alpha x[r] a_rc over the stored elements.
// As in the reference, y is first multiplied by beta unless beta == 1 (read
// even when beta == 0), and the scattered additions are atomic, so their
// order -- and the last bits of y -- is not fixed.  G lanes take one row,
// G from the mean row length (as Light CSR picks it); elements are reached
// through the formats' getGlobalIndex (segview.cuh), so one kernel serves
// CSR, Ellpack, SlicedEllpack, ChunkedEllpack, BiEllpack and AdaptiveCSR.
#include "internal.cuh"
#include "segview.cuh"

namespace tnlb {
namespace {

template <typename Real>
__global__ void k_scale_in_place(int64_t n, Real b, Real* __restrict__ y)
{
   for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
      y[i] = y[i] * b;
}

template <typename Real, int G>
__global__ void k_spmv_symmetric(SegView v, const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                                 const Real* __restrict__ x, Real* __restrict__ y, Real alpha, int32_t begin,
                                 int32_t end)
{
   const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   const int64_t row = begin + gid / G;
   const int lane = (int)(gid % G);
   Real sum = Real(0);
   if (row < end) {
      const Real xr = x[row];
      for (int32_t local = lane;; local += G) {
         const int64_t gi = global_index_of(v, (int32_t)row, local);
         if (gi < 0) break;
         const int32_t c = cols[gi];
         if (c < 0) continue;  // padding
         const Real a = vals[gi];
         if (c < row) atomicAdd(y + c, alpha * a * xr);
         sum += a * x[c];
      }
   }
   sum = group_sum<G>(sum);
   if (row < end && lane == 0) atomicAdd(y + row, alpha * sum);
}

template <typename Real, int G>
__global__ void k_spmv_transposed(SegView v, const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                                  const Real* __restrict__ x, Real* __restrict__ y, Real alpha, int32_t n,
                                  int32_t begin, int32_t end)
{
   const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   const int64_t row = gid / G;
   const int lane = (int)(gid % G);
   if (row >= n) return;
   const Real axr = alpha * x[row];
   for (int32_t local = lane;; local += G) {
      const int64_t gi = global_index_of(v, (int32_t)row, local);
      if (gi < 0) break;
      const int32_t c = cols[gi];
      if (c >= begin && c < end && c != -1) atomicAdd(y + c, axr * vals[gi]);
   }
}

// The same two products with a window of y in shared memory: one block per SM
// takes a contiguous run of rows, adds what falls on the columns around them
// there and the window to y at the end, so that of a banded matrix's elements
// only the window's entries reach memory as atomic additions, and those
// coalesced.  CSR rows are taken by G lanes, kScatterRows rows in flight; Col:
// column-major Ellpack and SlicedEllpack, a lane a row, whose slots the lanes
// read together.  A^T x of 13.5M entries at 500,009 rows in a band of 12,600
// (FP64): 147 us with every addition in memory, 79 so, 88 with all of the shared
// memory as window: 163 KB leave the L1 cache enough for x and for the additions
// outside.
// A block first looks at some of its columns and adds all in memory where the
// window does not pay (scatter_pays).
constexpr int kScatterThreads = 1024, kScatterRows = 4;
constexpr int kScatterBytes = 163 * 1024;
extern __shared__ __align__(16) unsigned char scatter_smem[];

// The column of one slot of a row among [r0, r1), or -1: of 32 neighbouring rows in
// 8 places, one for each of the block's first 256 threads.
template <bool Col>
__device__ __forceinline__ int32_t scatter_sample(const SegView& v, const int32_t* __restrict__ cols, int32_t r0,
                                                  int32_t r1)
{
   const int32_t r = r0 + (int32_t)((threadIdx.x >> 5) * (int64_t)(r1 - r0) / 8) + (int32_t)(threadIdx.x & 31);
   if (threadIdx.x >= 256 || r >= r1) return -1;
   const uint32_t any = threadIdx.x * 2654435761u >> 8;
   if constexpr (Col) {
      const bool sliced = v.format == TNLB_SLICED_ELLPACK;
      const int32_t w = sliced ? v.slice_w[r / kSellSlice] : v.segment_size;
      const int64_t base = sliced ? v.slice_off[r / kSellSlice] + (int64_t)(r % kSellSlice) : r;
      return w > 0 ? cols[base + (int64_t)(any % (uint32_t)w) * (sliced ? kSellSlice : v.aligned_size)] : -1;
   }
   else {
      const int32_t at = v.offsets[r], len = v.offsets[r + 1] - at;
      return len > 0 ? cols[at + (int32_t)(any % (uint32_t)len)] : -1;
   }
}

// Clears the window of `width` entries from `lo` and tells whether it pays for the
// rows whose sampled columns the threads hold: an eighth of them lies in it, and
// no column is kScatterHot of the 256.  Additions to one place in shared memory
// follow one another, about 50 cycles each, which those to the L2 cache need not.
// FP64, transposed, 27 entries a row at 500,009 rows, us by the kernels above, by
// additions in memory here, and by the window: band of 40,000 150, 110, 93; of
// 120,000 (17% inside) 149, 110, 95; random 148, 105, 103; a tenth of each 3000
// rows' entries in one column 324, 128, 312; 63,000 entries in the first and the
// last column 259, 144, 1123 (95 where only the blocks that hold them add in
// memory).
constexpr int kScatterHot = 5, kScatterBins = 8192;
template <typename Real>
__device__ __forceinline__ bool scatter_pays(int32_t c, int32_t lo, uint32_t width)
{
   int* words = reinterpret_cast<int*>(scatter_smem);
   const uint32_t clear = max(width * (uint32_t)(sizeof(Real) / sizeof(int)), (uint32_t)kScatterBins);
   for (uint32_t j = threadIdx.x; j < clear; j += kScatterThreads) words[j] = 0;
   const int valid = __syncthreads_count(c >= 0);
   const int inside = __syncthreads_count(c >= 0 && (uint32_t)(c - lo) < width);
   int* bin = words + ((uint32_t)c * 2654435761u >> 19);
   const bool hot = __syncthreads_or(c >= 0 && atomicAdd(bin, 1) >= kScatterHot - 1);
   if (c >= 0) *bin = 0;
   __syncthreads();
   return 8 * inside >= valid && !hot;
}

template <typename Real, bool Symmetric, bool Col, int G>
__global__ void __launch_bounds__(kScatterThreads, 1)
   k_scatter_window(SegView v, const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                    const Real* __restrict__ x, Real* __restrict__ y, Real alpha, int32_t row0, int32_t row1,
                    int32_t per_block, int32_t columns, int32_t room, int32_t begin, int32_t end)
{
   Real* win = reinterpret_cast<Real*>(scatter_smem);
   const int32_t r0 = (int32_t)imin64(row0 + (int64_t)blockIdx.x * per_block, row1);
   const int32_t r1 = (int32_t)imin64((int64_t)r0 + per_block, row1);
   const int64_t mid = ((int64_t)r0 + r1) / 2;
   const int32_t lo = (int32_t)imin64(imax64(mid - room / 2, 0), imax64((int64_t)columns - room, 0));
   uint32_t width = (uint32_t)imin64(room, columns - lo);
   if (!scatter_pays<Real>(scatter_sample<Col>(v, cols, r0, r1), lo, width)) width = 0;
   auto add = [&](int32_t c, Real t) {
      const uint32_t at = (uint32_t)(c - lo);
      if (at < width)
         atomicAdd(win + at, t);
      else
         atomicAdd(y + c, t);
   };
   // one element of row r; what it adds to the row's own sum
   auto element = [&](int32_t r, Real xr, int32_t c, Real a) -> Real {
      if (Symmetric) {
         if (c < 0) return Real(0);
         if (c < r) add(c, alpha * a * xr);
         return a * x[c];
      }
      if (c >= begin && c < end && c != -1) add(c, alpha * xr * a);
      return Real(0);
   };
   if constexpr (Col) {
      const bool sliced = v.format == TNLB_SLICED_ELLPACK;
      const int64_t step = sliced ? kSellSlice : v.aligned_size;
      for (int32_t r = r0 + (int32_t)threadIdx.x; r < r1; r += kScatterThreads) {
         const int32_t w = sliced ? v.slice_w[r / kSellSlice] : v.segment_size;
         const int64_t base = sliced ? v.slice_off[r / kSellSlice] + (int64_t)(r % kSellSlice) : r;
         const Real xr = x[r];
         Real sum = Real(0);
         for (int32_t k = 0; k < w; k += kScatterRows) {
            int32_t c[kScatterRows];
            Real a[kScatterRows];
#pragma unroll
            for (int u = 0; u < kScatterRows; u++) {
               c[u] = -1;
               a[u] = Real(0);
               if (k + u < w) {
                  c[u] = ld_stream(cols + base + (k + u) * step);
                  a[u] = ld_stream(vals + base + (k + u) * step);
               }
            }
#pragma unroll
            for (int u = 0; u < kScatterRows; u++)
               if (c[u] != -1) sum += element(r, xr, c[u], a[u]);
         }
         if (Symmetric) add(r, alpha * sum);
      }
   }
   else {
      const int lane = threadIdx.x % G;
      constexpr int32_t kStep = kScatterThreads / G;
      for (int32_t q = r0 + (int32_t)threadIdx.x / G; q - (int32_t)threadIdx.x / G < r1; q += kStep * kScatterRows) {
         int32_t at[kScatterRows], e[kScatterRows], c[kScatterRows];
         Real a[kScatterRows], xr[kScatterRows];
#pragma unroll
         for (int u = 0; u < kScatterRows; u++) {
            const int32_t r = q + u * kStep;
            at[u] = r < r1 ? v.offsets[r] + lane : 0;
            e[u] = r < r1 ? v.offsets[r + 1] : 0;
            xr[u] = r < r1 ? x[r] : Real(0);
         }
#pragma unroll
         for (int u = 0; u < kScatterRows; u++) {
            c[u] = -1;
            a[u] = Real(0);
            if (at[u] < e[u]) {
               c[u] = ld_stream(cols + at[u]);
               a[u] = ld_stream(vals + at[u]);
            }
         }
#pragma unroll
         for (int u = 0; u < kScatterRows; u++) {
            const int32_t r = q + u * kStep;
            Real sum = Real(0);
            if (c[u] != -1) sum = element(r, xr[u], c[u], a[u]);
            for (int32_t k = at[u] + G; k < e[u]; k += G) {
               const int32_t ck = ld_stream(cols + k);
               if (ck != -1) sum += element(r, xr[u], ck, ld_stream(vals + k));
            }
            if (Symmetric) {
               sum = group_sum<G>(sum);
               if (lane == 0 && r < r1) add(r, alpha * sum);
            }
         }
      }
   }
   __syncthreads();
   for (uint32_t j = threadIdx.x; j < width; j += kScatterThreads)
      if (win[j] != Real(0)) atomicAdd(y + lo + j, win[j]);
}

int lanes_for(const tnlb_segments* seg)
{
   if (seg->n <= 0) return 2;
   const int64_t e = (seg->storage + seg->n - 1) / seg->n;
   if (e <= 2) return 2;
   if (e <= 4) return 4;
   if (e <= 8) return 8;
   if (e <= 16) return 16;
   return 32;
}

// Launches k_scatter_window over the rows [row0, row1) where it is expected to be
// the faster one (false: not launched).  Measured against the kernels above on
// grids, band matrices (9 to 45 entries a row) and power-law rows:
//  * column-major formats, whose slots those kernels read lane by lane: 1.3 to 3
//    times as fast from 8000 entries an SM, 0.7 to 1.2 at 2600 to 4000 (random
//    columns, 4 to 42 a row, 0.95 to 2.1 from 8000);
//  * transposed CSR: 1.1 to 2.1 times from 14,000 entries an SM (random columns
//    1.1 to 1.8), 0.9 at 10,000,
//    where the clearing and the flush of the window count; 0.3 to 0.7 on
//    power-law rows, which one block's lanes cannot share, so rows are short;
//  * symmetric CSR: 0.8 to 1.1, so never.
constexpr int64_t kScatterColEntries = 8000, kScatterCsrEntries = 14000;
constexpr int32_t kScatterCsrRow = 64;
template <typename Real, bool Symmetric>
bool launch_scatter(const tnlb_segments* seg, const int32_t* cols, const Real* vals, const Real* x, Real* y,
                    Real alpha, int32_t row0, int32_t row1, int32_t columns, int32_t begin, int32_t end,
                    cudaStream_t st, cudaError_t* err)
{
   const bool csr = !Symmetric && (seg->format == TNLB_CSR || seg->format == TNLB_ADAPTIVE_CSR) && seg->max_row >= 0 &&
                    seg->max_row <= kScatterCsrRow;
   const bool col = (seg->format == TNLB_ELLPACK || seg->format == TNLB_SLICED_ELLPACK) &&
                    seg->organization == TNLB_COLUMN_MAJOR;
   int dev = 0, sms = 0;
   if (!(csr || col) || cudaGetDevice(&dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      return false;
   }
   const int64_t rows = (int64_t)row1 - row0;
   const int32_t per_block = (int32_t)((rows + sms - 1) / sms);
   if (seg->elements < (int64_t)sms * (col ? kScatterColEntries : kScatterCsrEntries) || per_block < 1) return false;
   const int32_t room = (int32_t)(kScatterBytes / sizeof(Real));
   const int G = lanes_for(seg);
   auto* k = k_scatter_window<Real, Symmetric, true, 32>;
   if constexpr (!Symmetric)
      if (!col)
         k = G <= 4    ? k_scatter_window<Real, false, false, 4>
             : G == 8  ? k_scatter_window<Real, false, false, 8>
             : G == 16 ? k_scatter_window<Real, false, false, 16>
                       : k_scatter_window<Real, false, false, 32>;
   if (cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, kScatterBytes) != cudaSuccess) {
      cudaGetLastError();
      return false;
   }
   k<<<(unsigned)((rows + per_block - 1) / per_block), kScatterThreads, kScatterBytes, st>>>(
      view_of(seg), cols, vals, x, y, alpha, row0, row1, per_block, columns, room, begin, end);
   *err = cudaGetLastError();
   return true;
}

template <typename Real>
tnlb_status symmetric_t(const tnlb_segments* seg, const int32_t* cols, const Real* vals, const Real* x, Real* y,
                        Real alpha, Real beta, int32_t begin, int32_t end, cudaStream_t st)
{
   const int64_t n = seg->n;
   if (beta != Real(1)) {
      k_scale_in_place<Real><<<grid_for(n, 256 * 4), 256, 0, st>>>(n, beta, y);
      TNLB_CHECK_LAUNCH();
   }
   const int64_t rows = (int64_t)end - begin;
   if (rows <= 0) return TNLB_OK;
   cudaError_t e = cudaSuccess;
   if (launch_scatter<Real, true>(seg, cols, vals, x, y, alpha, begin, end, seg->n, 0, 0, st, &e)) {
      TNLB_CUDA_TRY(e);
      return TNLB_OK;
   }
   const SegView v = view_of(seg);
   const int G = lanes_for(seg);
#define TNLB_SYM(GG)                                                                                           \
   case GG:                                                                                                    \
      k_spmv_symmetric<Real, GG><<<grid_for(rows * GG, 256), 256, 0, st>>>(v, cols, vals, x, y, alpha, begin, \
                                                                            end);                              \
      break;
   switch (G) {
      TNLB_SYM(2)
      TNLB_SYM(4)
      TNLB_SYM(8)
      TNLB_SYM(16)
      TNLB_SYM(32)
   }
#undef TNLB_SYM
   TNLB_CHECK_LAUNCH();
   return TNLB_OK;
}

template <typename Real>
tnlb_status transposed_t(const tnlb_segments* seg, const int32_t* cols, const Real* vals, int32_t columns,
                         const Real* x, Real* y, Real alpha, Real beta, int32_t begin, int32_t end, cudaStream_t st)
{
   if (beta != Real(1) && columns > 0) {
      k_scale_in_place<Real><<<grid_for(columns, 256 * 4), 256, 0, st>>>(columns, beta, y);
      TNLB_CHECK_LAUNCH();
   }
   const int64_t n = seg->n;
   if (n <= 0 || end <= begin) return TNLB_OK;
   cudaError_t e = cudaSuccess;
   if (launch_scatter<Real, false>(seg, cols, vals, x, y, alpha, 0, (int32_t)n, columns, begin, end, st, &e)) {
      TNLB_CUDA_TRY(e);
      return TNLB_OK;
   }
   const SegView v = view_of(seg);
   const int G = lanes_for(seg);
#define TNLB_TR(GG)                                                                                              \
   case GG:                                                                                                      \
      k_spmv_transposed<Real, GG><<<grid_for(n * GG, 256), 256, 0, st>>>(v, cols, vals, x, y, alpha, (int32_t)n, \
                                                                          begin, end);                           \
      break;
   switch (G) {
      TNLB_TR(2)
      TNLB_TR(4)
      TNLB_TR(8)
      TNLB_TR(16)
      TNLB_TR(32)
   }
#undef TNLB_TR
   TNLB_CHECK_LAUNCH();
   return TNLB_OK;
}

}  // namespace
}  // namespace tnlb

using namespace tnlb;

extern "C" tnlb_status tnlb_spmv_symmetric(const tnlb_segments* seg, tnlb_real real, const int32_t* d_cols,
                                          const void* d_values, const void* d_x, void* d_y, double alpha,
                                          double beta, int32_t begin, int32_t end, tnlb_stream stream)
{
   clear_error();
   TNLB_REQUIRE(seg != nullptr, TNLB_ERR_INVALID_ARGUMENT, "null segments");
   TNLB_REQUIRE(real == TNLB_F32 || real == TNLB_F64, TNLB_ERR_INVALID_ARGUMENT, "unknown real type");
   if (end == 0) end = seg->n;
   TNLB_REQUIRE(begin >= 0 && begin <= end && end <= seg->n, TNLB_ERR_INVALID_ARGUMENT,
                "vectorProduct: row range [begin, end) outside the matrix");
   if (seg->n == 0) return TNLB_OK;
   TNLB_REQUIRE(d_y != nullptr && (seg->storage == 0 || (d_cols && d_values && d_x)), TNLB_ERR_INVALID_ARGUMENT,
                "null array");
   const cudaStream_t st = (cudaStream_t)stream;
   if (real == TNLB_F64)
      return symmetric_t<double>(seg, d_cols, (const double*)d_values, (const double*)d_x, (double*)d_y, alpha, beta,
                                 begin, end, st);
   return symmetric_t<float>(seg, d_cols, (const float*)d_values, (const float*)d_x, (float*)d_y, (float)alpha,
                             (float)beta, begin, end, st);
}

extern "C" tnlb_status tnlb_spmv_transposed(const tnlb_segments* seg, tnlb_real real, const int32_t* d_cols,
                                           const void* d_values, int32_t columns, const void* d_x, void* d_y,
                                           double alpha, double beta, int32_t begin, int32_t end, tnlb_stream stream)
{
   clear_error();
   TNLB_REQUIRE(seg != nullptr, TNLB_ERR_INVALID_ARGUMENT, "null segments");
   TNLB_REQUIRE(real == TNLB_F32 || real == TNLB_F64, TNLB_ERR_INVALID_ARGUMENT, "unknown real type");
   TNLB_REQUIRE(columns >= 0, TNLB_ERR_INVALID_ARGUMENT,
                "transposedVectorProduct: size of the output vector does not match the number of matrix columns");
   if (end == 0) end = columns;
   TNLB_REQUIRE(begin >= 0 && begin <= end && end <= columns, TNLB_ERR_INVALID_ARGUMENT,
                "transposedVectorProduct: column range [begin, end) outside the matrix");
   if (columns == 0) return TNLB_OK;
   TNLB_REQUIRE(d_y != nullptr && (seg->storage == 0 || (d_cols && d_values && d_x)), TNLB_ERR_INVALID_ARGUMENT,
                "null array");
   const cudaStream_t st = (cudaStream_t)stream;
   if (real == TNLB_F64)
      return transposed_t<double>(seg, d_cols, (const double*)d_values, columns, (const double*)d_x, (double*)d_y,
                                  alpha, beta, begin, end, st);
   return transposed_t<float>(seg, d_cols, (const float*)d_values, columns, (const float*)d_x, (float*)d_y,
                              (float)alpha, (float)beta, begin, end, st);
}
