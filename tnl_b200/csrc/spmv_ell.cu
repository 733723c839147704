// spmv_ell.cu -- y = alpha*A*x + beta*y for Ellpack, SlicedEllpack,
// ChunkedEllpack and BiEllpack segments (both element organizations).
//
//  * Ellpack, column-major (the reference's GPU default): one thread per row
//    walking slots row + alignedSize*k -- consecutive rows give coalesced
//    loads (ReducingOperations_Ellpack.h:186-199).  Row-major: G lanes per
//    row (EllpackCudaReductionKernel, ReducingKernels_Ellpack.h:12-74).
//  * SlicedEllpack (slice 32), column-major: one warp per slice, lane = row,
//    slot k of the slice is 32 consecutive elements (256 B in FP64), loop
//    unrolled by 4 to keep loads in flight; G > 1 splits the slot range of a
//    slice over G warps of a block and combines them in shared memory
//    (reduceSegmentsSlicedEllpackKernel, ReducingKernels_SlicedEllpack.h:100-323).
//    Row-major: G lanes per row.
//  * ChunkedEllpack: one block per slice, one thread per chunk, per-chunk
//    partials in shared memory, then each row sums its chunks
//    (ChunkedEllpackReduceSegmentsKernel, ReducingKernels_ChunkedEllpack.h:13-98).
//  * BiEllpack: one warp per strip of 32 rows; lane = sorted position, groups
//    of halving height 32,16,8,4,2,1; the result is moved to the original
//    row through the permutation with one shuffle
//    (BiEllpackReduceSegmentsKernel, ReducingKernels_BiEllpack.h:70-217).
#include <cooperative_groups.h>

#include "internal.cuh"
#include "reduce.cuh"

namespace tnlb {
namespace {

template <typename Real>
__device__ __forceinline__ void keep_range(Real* y, int64_t row, Real v, Real alpha, Real beta, int32_t begin,
                                           int32_t end)
{
   if (row >= begin && row < end) keep(y, (int32_t)row, v, alpha, beta);
}

template <typename Real>
__device__ __forceinline__ Real fma_slot(const int32_t* cols, const Real* vals, const Real* x, int64_t g, Real acc)
{
   const int32_t c = ld_stream(cols + g);
   const Real v = ld_stream(vals + g);
   return c >= 0 ? acc + v * ld_gather(x + c) : acc;
}

// ------------------------------------------------------------- Ellpack

template <typename Real>
__global__ void k_ell_col(const int32_t* __restrict__ cols, const Real* __restrict__ vals, const Real* __restrict__ x,
                          Real* __restrict__ y, int32_t n, int32_t width, int32_t aligned, int32_t begin, int32_t end,
                          Real alpha, Real beta)
{
   const int64_t row = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (row >= end) return;
   Real sum = 0;
   int32_t k = 0;
   if (width <= 8) {
      // narrow rows (stencils): every slot's load issued at once
      int32_t c[8];
      Real v[8];
#pragma unroll
      for (int u = 0; u < 8; u++) {
         c[u] = -1;
         v[u] = Real(0);
         if (u < width) {
            c[u] = ld_stream(cols + row + (int64_t)aligned * u);
            v[u] = ld_stream(vals + row + (int64_t)aligned * u);
         }
      }
#pragma unroll
      for (int u = 0; u < 8; u++)
         if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
      k = width;
   }
   for (; k + 4 <= width; k += 4) {
      int32_t c[4];
      Real v[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
         c[u] = ld_stream(cols + row + (int64_t)aligned * (k + u));
         v[u] = ld_stream(vals + row + (int64_t)aligned * (k + u));
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
         if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
   }
   for (; k < width; k++) sum = fma_slot(cols, vals, x, row + (int64_t)aligned * k, sum);
   keep(y, (int32_t)row, sum, alpha, beta);
}

template <typename Real, int G>
__global__ void k_ell_row(const int32_t* __restrict__ cols, const Real* __restrict__ vals, const Real* __restrict__ x,
                          Real* __restrict__ y, int32_t width, int32_t begin, int32_t end, Real alpha, Real beta)
{
   const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   const int64_t row = begin + gid / G;
   const int lane = (int)(gid % G);
   Real sum = 0;
   if (row < end)
      for (int32_t k = lane; k < width; k += G) sum = fma_slot(cols, vals, x, row * width + k, sum);
   sum = group_sum<G>(sum);
   if (row < end && lane == 0) keep(y, (int32_t)row, sum, alpha, beta);
}

// ------------------------------------------------------- SlicedEllpack

// The runs of slices that k_sell_window may take, and the window of each: `room`
// entries of x around the run's rows.
constexpr int kWindowPercent = 60;
struct SellWindow {
   int32_t per_block, columns, room;  // slices of a run, a multiple of 8; 0: no windows
   __device__ __forceinline__ int32_t lo(int64_t s0, int64_t s1) const
   {
      const int64_t mid = (s0 + s1) / 2 * kSellSlice;
      return (int32_t)imin64(imax64(mid - room / 2, 0), imax64((int64_t)columns - room, 0));
   }
   __device__ __forceinline__ uint32_t width(int32_t lo) const { return (uint32_t)imin64(room, columns - lo); }
   // Whether kWindowPercent of the columns of run `b` lie in its window, from 32
   // slots of 8 of its slices.  Called by whole blocks of at least 256 threads; the answer is the
   // same in each.
   __device__ __forceinline__ bool taken(int32_t b, const int32_t* cols, const int32_t* slice_off,
                                         const int32_t* slice_w, int32_t slices) const
   {
      const int64_t s0 = (int64_t)b * per_block, s1 = imin64(s0 + per_block, slices);
      const int32_t l = lo(s0, s1);
      int32_t c = -1;
      if (threadIdx.x < 256) {
         const int64_t s = s0 + (threadIdx.x >> 5) * (s1 - s0) / 8;
         const int32_t w = slice_w[s];
         if (w > 0) c = cols[(int64_t)slice_off[s] + (int64_t)(w - 1) / 2 * kSellSlice + (threadIdx.x & 31)];
      }
      const int valid = __syncthreads_count(c >= 0);
      return 100 * __syncthreads_count(c >= 0 && (uint32_t)(c - l) < width(l)) >= kWindowPercent * valid;
   }
};

// G warps per slice (G = 1, 2, 4, 8); the block holds 8/G slices.  Runs that
// k_sell_window takes are left out.
template <typename Real, int G>
__global__ void __launch_bounds__(256) k_sell_col(const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                                                  const Real* __restrict__ x, Real* __restrict__ y,
                                                  const int32_t* __restrict__ slice_off,
                                                  const int32_t* __restrict__ slice_w, int32_t slices, int32_t begin,
                                                  int32_t end, Real alpha, Real beta, SellWindow win)
{
   __shared__ Real part[8][32];
   if (win.per_block > 0) {
      const bool taken =
         win.taken((int32_t)((int64_t)blockIdx.x * (8 / G) / win.per_block), cols, slice_off, slice_w, slices);
      // this kernel may run beside k_sell_window, whose rows are others, but ends after it
      if (blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
      if (taken) return;
   }
   const int wib = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int sub = wib % G;
   const int64_t slice = (int64_t)blockIdx.x * (8 / G) + wib / G;
   Real sum = 0;
   if (slice < slices) {
      const int64_t off = slice_off[slice] + lane;
      const int32_t w = slice_w[slice];
      int32_t k = sub;
      if (G == 1 && w <= 8) {
         // narrow slices (stencils): every slot's load issued at once
         int32_t c[8];
         Real v[8];
#pragma unroll
         for (int u = 0; u < 8; u++) {
            c[u] = -1;
            v[u] = Real(0);
            if (u < w) {
               c[u] = ld_stream(cols + off + (int64_t)kSellSlice * u);
               v[u] = ld_stream(vals + off + (int64_t)kSellSlice * u);
            }
         }
#pragma unroll
         for (int u = 0; u < 8; u++)
            if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
         k = w;
      }
      for (; k + 3 * G < w; k += 4 * G) {
         int32_t c[4];
         Real v[4];
#pragma unroll
         for (int u = 0; u < 4; u++) {
            c[u] = ld_stream(cols + off + (int64_t)kSellSlice * (k + u * G));
            v[u] = ld_stream(vals + off + (int64_t)kSellSlice * (k + u * G));
         }
#pragma unroll
         for (int u = 0; u < 4; u++)
            if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
      }
      for (; k < w; k += G) sum = fma_slot(cols, vals, x, off + (int64_t)kSellSlice * k, sum);
   }
   if (G == 1) {
      if (slice < slices) keep_range(y, slice * kSellSlice + lane, sum, alpha, beta, begin, end);
      return;
   }
   part[wib][lane] = sum;
   __syncthreads();
   if (sub == 0 && slice < slices) {
      Real s = 0;
#pragma unroll
      for (int q = 0; q < G; q++) s += part[wib + q][lane];
      keep_range(y, slice * kSellSlice + lane, s, alpha, beta, begin, end);
   }
}

// One warp per slice over a resident grid (G = 1): each warp walks the
// slices with the grid's warp count as stride and loads the next slice's
// offset and width before the current slice's entries, so the slice table
// is not a step of every slice's chain of dependent loads (on a 5-point
// operator the per-wave chain offset -> entries -> x made the full-grid
// launch 20% slower than Ellpack).
template <typename Real>
__global__ void __launch_bounds__(256) k_sell_walk(const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                                                   const Real* __restrict__ x, Real* __restrict__ y,
                                                   const int32_t* __restrict__ slice_off,
                                                   const int32_t* __restrict__ slice_w, int32_t slices, int32_t begin,
                                                   int32_t end, Real alpha, Real beta)
{
   const int lane = threadIdx.x & 31;
   const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
   int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   int32_t o = 0, w = 0;
   if (s < slices) {
      o = slice_off[s];
      w = slice_w[s];
   }
   for (; s < slices; s += nw) {
      const int64_t off = (int64_t)o + lane;
      const int32_t wc = w;
      if (s + nw < slices) {
         o = slice_off[s + nw];
         w = slice_w[s + nw];
      }
      Real sum = 0;
      int32_t k = 0;
      if (wc <= 8) {
         int32_t c[8];
         Real v[8];
#pragma unroll
         for (int u = 0; u < 8; u++) {
            c[u] = -1;
            v[u] = Real(0);
            if (u < wc) {
               c[u] = ld_stream(cols + off + (int64_t)kSellSlice * u);
               v[u] = ld_stream(vals + off + (int64_t)kSellSlice * u);
            }
         }
#pragma unroll
         for (int u = 0; u < 8; u++)
            if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
         k = wc;
      }
      for (; k + 3 < wc; k += 4) {
         int32_t c[4];
         Real v[4];
#pragma unroll
         for (int u = 0; u < 4; u++) {
            c[u] = ld_stream(cols + off + (int64_t)kSellSlice * (k + u));
            v[u] = ld_stream(vals + off + (int64_t)kSellSlice * (k + u));
         }
#pragma unroll
         for (int u = 0; u < 4; u++)
            if (c[u] >= 0) sum += v[u] * ld_gather(x + c[u]);
      }
      for (; k < wc; k++) sum = fma_slot(cols, vals, x, off + (int64_t)kSellSlice * k, sum);
      keep_range(y, s * kSellSlice + lane, sum, alpha, beta, begin, end);
   }
}

// Wide slices of a banded matrix: one block per SM with a contiguous run of
// slices keeps the x of its rows and of the columns around them in shared
// memory.  Columns that differ from lane to lane take the L1 cache one lookup a
// lane (27M of them, 96 us at one a cycle and SM), shared memory about 3.5
// cycles for 32.  FP32 residual at 1,000,003 rows of 9 to 45 entries in a band of
// 20,000: 102.9 us by two warps a slice, 81.9 so; its 370 MB with the padding take
// 57.
// Nothing is known of the columns beforehand, so a block first looks at some of
// its slots and leaves its run to k_sell_col, launched behind it, where too many
// lie outside: they want the L1 that the window takes, and 60% inside is where
// both take the same (FP64, 27 entries a row in a band of 20,000 at 2,000,003 rows,
// 62% inside: 201 us by a window, 229 by k_sell_col; in a band of 40,000 at 500,009
// rows, 48% inside: 78 and 72).  163 KB leave enough L1 for the columns outside:
// with 227 KB the same matrices took 209 and 88.
// k_sell_col's blocks look at their run too, a wave of them 1.8 us.  So the window's
// blocks let it start when they have their window, under their main loop (85.6 us
// for the residual after 93.9); and those that leave their run end at once, so that
// it finds the SMs empty and their L1 whole: random columns, 27 a row (FP64), at
// 500,009 and 1,000,003 rows 73.8 and 129.1 us by k_sell_col alone, 76.8 and 134.2
// behind the window's look; 138 and 169 when it starts earlier.
constexpr int kWindowThreads = 1024, kWindowWarps = kWindowThreads / 32, kWindowDepth = 8;
constexpr int kWindowBytes = 163 * 1024;
extern __shared__ __align__(16) unsigned char window_smem[];

template <typename Real>
__global__ void __launch_bounds__(kWindowThreads, 1)
   k_sell_window(const int32_t* __restrict__ cols, const Real* __restrict__ vals, const Real* __restrict__ x,
                 Real* __restrict__ y, const int32_t* __restrict__ slice_off, const int32_t* __restrict__ slice_w,
                 int32_t slices, SellWindow sw, int32_t begin, int32_t end, Real alpha, Real beta)
{
   Real* win = reinterpret_cast<Real*>(window_smem);
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   if (!sw.taken(blockIdx.x, cols, slice_off, slice_w, slices)) return;
   const int32_t s0 = (int32_t)blockIdx.x * sw.per_block;
   const int32_t s1 = (int32_t)imin64((int64_t)s0 + sw.per_block, slices);
   const int32_t lo = sw.lo(s0, s1);
   const uint32_t width = sw.width(lo);
   int32_t s = s0 + warp;
   int32_t o = 0, w = 0;
   if (s < s1) {
      o = slice_off[s];
      w = slice_w[s];
   }
   for (uint32_t j = threadIdx.x; j < width; j += kWindowThreads) win[j] = x[lo + j];
   __syncthreads();
   asm volatile("griddepcontrol.launch_dependents;");
   for (; s < s1; s += kWindowWarps) {
      const int32_t* C = cols + o + lane;
      const Real* V = vals + o + lane;
      const int32_t wc = w;
      if (s + kWindowWarps < s1) {
         o = slice_off[s + kWindowWarps];
         w = slice_w[s + kWindowWarps];
      }
      Real part[4] = {Real(0), Real(0), Real(0), Real(0)};  // as four warps a slice would sum
      for (int32_t k = 0; k < wc; k += kWindowDepth) {
         int32_t c[kWindowDepth];
         Real v[kWindowDepth];
#pragma unroll
         for (int u = 0; u < kWindowDepth; u++) {
            c[u] = -1;
            v[u] = Real(0);
            if (k + u < wc) {
               c[u] = ld_stream(C + (int64_t)kSellSlice * (k + u));
               v[u] = ld_stream(V + (int64_t)kSellSlice * (k + u));
            }
         }
#pragma unroll
         for (int u = 0; u < kWindowDepth; u++) {
            const uint32_t at = (uint32_t)(c[u] - lo);
            if (at < width)
               part[u & 3] += v[u] * win[at];
            else if (c[u] >= 0)
               part[u & 3] += v[u] * ld_gather(x + c[u]);
         }
      }
      const Real sum = ((part[0] + part[1]) + part[2]) + part[3];
      keep_range(y, (int64_t)s * kSellSlice + lane, sum, alpha, beta, begin, end);
   }
}

// k_sell_col.  Behind k_sell_window (win) it starts once that kernel's blocks have
// all looked at their runs, unless the stream is being captured.
template <typename Real, int G>
cudaError_t launch_sell_col(const tnlb_segments* seg, const int32_t* cols, const Real* vals, const Real* x, Real* y,
                            Real alpha, Real beta, int32_t begin, int32_t end, const SellWindow& win, cudaStream_t st)
{
   cudaLaunchConfig_t cfg{};
   cfg.gridDim = dim3(grid_for(seg->slices, 8 / G));
   cfg.blockDim = dim3(256);
   cfg.stream = st;
   cudaLaunchAttribute at{};
   at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
   at.val.programmaticStreamSerializationAllowed = 1;
   cfg.attrs = &at;
   if (win.per_block > 0) {
      cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
      const cudaError_t e = cudaStreamIsCapturing(st, &capture);
      if (e != cudaSuccess) return e;
      cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
   }
   return cudaLaunchKernelEx(&cfg, k_sell_col<Real, G>, cols, vals, x, y,
                             (const int32_t*)seg->slice_offsets.as<int32_t>(),
                             (const int32_t*)seg->slice_segment_sizes.as<int32_t>(), seg->slices, begin, end, alpha,
                             beta, win);
}

// Launches k_sell_window where it is expected to be the faster one; *out the runs
// that it may have taken (per_block 0: not launched).
template <typename Real>
void launch_window(const tnlb_segments* seg, int32_t columns, const int32_t* cols, const Real* vals, const Real* x,
                   Real* y, Real alpha, Real beta, int32_t begin, int32_t end, cudaStream_t st, SellWindow* out)
{
   int dev = 0, sms = 0;
   if (cudaGetDevice(&dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
      cudaGetLastError();
      return;
   }
   // at least two slices a warp, and a window of at least twice the block's rows
   const int32_t per_block = ((seg->slices + sms - 1) / sms + 7) / 8 * 8;
   const int32_t room = (int32_t)(kWindowBytes / sizeof(Real));
   if (per_block < 2 * kWindowWarps || (int64_t)per_block * kSellSlice * 2 > room) return;
   auto* k = k_sell_window<Real>;
   if (cudaFuncSetAttribute((const void*)k, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindowBytes) != cudaSuccess) {
      cudaGetLastError();
      return;
   }
   k<<<(seg->slices + per_block - 1) / per_block, kWindowThreads, (size_t)room * sizeof(Real), st>>>(
      cols, vals, x, y, seg->slice_offsets.as<int32_t>(), seg->slice_segment_sizes.as<int32_t>(), seg->slices,
      SellWindow{per_block, columns, room}, begin, end, alpha, beta);
   *out = SellWindow{per_block, columns, room};
}

template <typename Real, int G>
__global__ void k_sell_row(const int32_t* __restrict__ cols, const Real* __restrict__ vals, const Real* __restrict__ x,
                           Real* __restrict__ y, const int32_t* __restrict__ slice_off,
                           const int32_t* __restrict__ slice_w, int32_t begin, int32_t end, Real alpha, Real beta)
{
   const int64_t gid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   const int64_t row = begin + gid / G;
   const int lane = (int)(gid % G);
   Real sum = 0;
   if (row < end) {
      const int64_t s = row / kSellSlice;
      const int32_t w = slice_w[s];
      const int64_t base = slice_off[s] + (row % kSellSlice) * (int64_t)w;
      for (int32_t k = lane; k < w; k += G) sum = fma_slot(cols, vals, x, base + k, sum);
   }
   sum = group_sum<G>(sum);
   if (row < end && lane == 0) keep(y, (int32_t)row, sum, alpha, beta);
}

// ------------------------------------------------------ ChunkedEllpack

template <typename Real, bool ColMajor>
__global__ void __launch_bounds__(kChunksInSlice) k_chell(const int32_t* __restrict__ cols,
                                                          const Real* __restrict__ vals, const Real* __restrict__ x,
                                                          Real* __restrict__ y, const int32_t* __restrict__ sl_size,
                                                          const int32_t* __restrict__ sl_chunk,
                                                          const int32_t* __restrict__ sl_first,
                                                          const int32_t* __restrict__ sl_ptr,
                                                          const int32_t* __restrict__ seg_to_chunk, int32_t begin,
                                                          int32_t end, Real alpha, Real beta)
{
   __shared__ Real chunk_sum[kChunksInSlice];
   const int32_t s = blockIdx.x;
   const int c = threadIdx.x;
   const int64_t off = sl_ptr[s];
   const int32_t cs = sl_chunk[s];
   Real sum = 0;
   if (ColMajor) {
      for (int32_t k = 0; k < cs; k++) sum = fma_slot(cols, vals, x, off + c + (int64_t)kChunksInSlice * k, sum);
   }
   else {
      const int64_t b = off + (int64_t)c * cs;
      for (int32_t k = 0; k < cs; k++) sum = fma_slot(cols, vals, x, b + k, sum);
   }
   chunk_sum[c] = sum;
   __syncthreads();
   if (c < sl_size[s]) {
      const int32_t seg = sl_first[s] + c;
      int32_t ch = c == 0 ? 0 : seg_to_chunk[seg - 1];
      const int32_t last = seg_to_chunk[seg];
      Real r = 0;
      while (ch < last) r += chunk_sum[ch++];
      keep_range(y, seg, r, alpha, beta, begin, end);
   }
}

// Column-major slices, read by columns first.  A slice is 256 chunks wide and
// as tall as its longest chunk, so uneven rows leave most of it padding (34
// slots an entry for Zipf 1.73 row lengths at 700,001 rows: 1.5 GB of column
// indexes, 3.1 GB of values).  What bounds the product is reading the column
// indexes; the value of a padding slot is never fetched.  A thread takes four
// neighbouring chunks (one 16-byte word of columns) and every 4th slot row,
// kChellDepth rows at a time, and looks at their signs together: where all are
// padding it goes on at once.  Tall slices are cut over a cluster of Split
// blocks, whose partial sums the first one adds through shared memory, so that
// the tallest slice does not outlast the others.  1065 us by the block-per-slice
// kernel, 585 so.  Warps of 32 chunks (748 us) and the next words fetched before
// the last are used (640 us, 76 registers) were slower.
constexpr int kChellDepth = 4;
constexpr int64_t kChellTall = 64;
template <typename Real, int Split>
__global__ void __launch_bounds__(256) k_chell_cols(const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                                                    const Real* __restrict__ x, Real* __restrict__ y,
                                                    const int32_t* __restrict__ sl_size,
                                                    const int32_t* __restrict__ sl_chunk,
                                                    const int32_t* __restrict__ sl_first,
                                                    const int32_t* __restrict__ sl_ptr,
                                                    const int32_t* __restrict__ seg_to_chunk, int32_t begin,
                                                    int32_t end, Real alpha, Real beta)
{
   __shared__ Real part[4][kChunksInSlice];
   const int32_t s = blockIdx.x / Split;
   const int rank = (int)(blockIdx.x % Split);
   const int t = threadIdx.x, c = (t & 63) * 4;
   const int32_t cs = sl_chunk[s];
   const int32_t* C = cols + sl_ptr[s] + c;
   const Real* V = vals + sl_ptr[s] + c;
   Real sum[4] = {Real(0), Real(0), Real(0), Real(0)};
   constexpr int32_t kRows = 4 * Split;  // slot rows the cluster takes together
   for (int32_t k0 = rank * 4 + (t >> 6); k0 < cs; k0 += kRows * kChellDepth) {
      int4 q[kChellDepth];
      int32_t sign = -1;
#pragma unroll
      for (int u = 0; u < kChellDepth; u++) {
         const int32_t k = k0 + u * kRows;
         q[u] = k < cs ? ld_stream_v4(C + (int64_t)k * kChunksInSlice) : make_int4(-1, -1, -1, -1);
         sign &= q[u].x & q[u].y & q[u].z & q[u].w;
      }
      if (sign < 0) continue;
#pragma unroll
      for (int u = 0; u < kChellDepth; u++) {
         const Real* v = V + (int64_t)(k0 + u * kRows) * kChunksInSlice;
         const int32_t cc[4] = {q[u].x, q[u].y, q[u].z, q[u].w};
         Real vv[4], xx[4];
#pragma unroll
         for (int e = 0; e < 4; e++) {
            vv[e] = cc[e] >= 0 ? ld_stream(v + e) : Real(0);
            xx[e] = cc[e] >= 0 ? ld_gather(x + cc[e]) : Real(0);
         }
#pragma unroll
         for (int e = 0; e < 4; e++)
            if (cc[e] >= 0) sum[e] += vv[e] * xx[e];
      }
   }
#pragma unroll
   for (int e = 0; e < 4; e++) part[t >> 6][c + e] = sum[e];
   __syncthreads();
   Real total = ((part[0][t] + part[1][t]) + part[2][t]) + part[3][t];
   __syncthreads();
   part[0][t] = total;
   if constexpr (Split > 1) {
      auto cluster = cooperative_groups::this_cluster();
      cluster.sync();
      if (rank == 0) {
#pragma unroll
         for (int r = 1; r < Split; r++) total += cluster.map_shared_rank(&part[0][0], r)[t];
      }
      cluster.sync();
      if (rank != 0) return;
   }
   part[1][t] = total;
   __syncthreads();
   if (t < sl_size[s]) {
      const int32_t seg = sl_first[s] + t;
      int32_t ch = t == 0 ? 0 : seg_to_chunk[seg - 1];
      const int32_t last = seg_to_chunk[seg];
      Real r = 0;
      while (ch < last) r += part[1][ch++];
      keep_range(y, seg, r, alpha, beta, begin, end);
   }
}

template <typename Real, int Split>
cudaError_t launch_chell_cols(const tnlb_segments* seg, const int32_t* cols, const Real* vals, const Real* x, Real* y,
                              Real alpha, Real beta, int32_t begin, int32_t end, cudaStream_t st)
{
   cudaLaunchConfig_t cfg{};
   cfg.gridDim = dim3((unsigned)seg->ch_slices * Split);
   cfg.blockDim = dim3(256);
   cfg.stream = st;
   cudaLaunchAttribute at{};
   at.id = cudaLaunchAttributeClusterDimension;
   at.val.clusterDim.x = Split;
   at.val.clusterDim.y = at.val.clusterDim.z = 1;
   cfg.attrs = &at;
   cfg.numAttrs = Split > 1 ? 1 : 0;
   return cudaLaunchKernelEx(&cfg, k_chell_cols<Real, Split>, cols, vals, x, y,
                             (const int32_t*)seg->ch_slice_size.as<int32_t>(),
                             (const int32_t*)seg->ch_slice_chunk_size.as<int32_t>(),
                             (const int32_t*)seg->ch_slice_first.as<int32_t>(),
                             (const int32_t*)seg->ch_slice_pointer.as<int32_t>(),
                             (const int32_t*)seg->ch_segment_to_chunk.as<int32_t>(), begin, end, alpha, beta);
}

// ----------------------------------------------------------- BiEllpack

// Column-major strips: group g of a strip holds the h = 32 >> g widest rows
// (sorted positions 0..h-1) with w slots each, slot (k, r) at base + k h + r.
// All 32 lanes stride through the group's h w slots: lane l always meets
// row l & (h-1), so it keeps one partial sum, and the partials of a row are
// added across the lanes l, l + h, ... by log2(32/h) shuffles.  A strip with
// one dominant row (power-law matrices) thus spreads that row over the warp
// instead of leaving it to one lane.  Four slots per lane are loaded before
// any is used.
template <typename Real>
__global__ void k_biell_col(const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                            const Real* __restrict__ x, Real* __restrict__ y, const int32_t* __restrict__ perm,
                            const int32_t* __restrict__ gp, int32_t n, int32_t strips, int32_t begin, int32_t end,
                            Real alpha, Real beta)
{
   const int64_t strip = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const int lane = threadIdx.x & 31;  // sorted position in the strip
   if (strip >= strips) return;
   const int32_t* g = gp + strip * kBiGroups;
   Real sum = 0;
   int h = 32;
   for (int grp = 0; grp < kBiGroups; grp++, h >>= 1) {
      const int64_t base = g[grp];
      const int32_t size = g[grp + 1] - g[grp];
      if (size == 0) continue;  // warp-uniform
      Real part = 0;
      int32_t s = lane;
      for (; s + 96 < size; s += 128) {
         int32_t c[4];
         Real v[4];
#pragma unroll
         for (int u = 0; u < 4; u++) {
            c[u] = ld_stream(cols + base + s + 32 * u);
            v[u] = ld_stream(vals + base + s + 32 * u);
         }
#pragma unroll
         for (int u = 0; u < 4; u++)
            if (c[u] >= 0) part += v[u] * ld_gather(x + c[u]);
      }
      for (; s < size; s += 32) part = fma_slot(cols, vals, x, base + s, part);
      for (int o = 16; o >= h; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      if (lane < h) sum += part;
   }
   const int64_t row = strip * kBiStrip + lane;  // original row of this lane
   const int src = row < n ? perm[row] - (int32_t)(strip * kBiStrip) : 0;
   const Real mine = __shfl_sync(0xffffffffu, sum, src);
   if (row < n) keep_range(y, row, mine, alpha, beta, begin, end);
}

// Row-major strips: lane = sorted position walks its own w slots.
template <typename Real>
__global__ void k_biell_row(const int32_t* __restrict__ cols, const Real* __restrict__ vals,
                            const Real* __restrict__ x, Real* __restrict__ y, const int32_t* __restrict__ perm,
                            const int32_t* __restrict__ gp, int32_t n, int32_t strips, int32_t begin, int32_t end,
                            Real alpha, Real beta)
{
   const int64_t strip = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
   const int lane = threadIdx.x & 31;
   if (strip >= strips) return;
   const int32_t* g = gp + strip * kBiGroups;
   Real sum = 0;
   int h = 32;
   for (int grp = 0; grp < kBiGroups; grp++, h >>= 1) {
      const int64_t base = g[grp];
      const int32_t size = g[grp + 1] - g[grp];
      if (size == 0 || lane >= h) continue;
      const int32_t w = size / h;
      for (int32_t k = 0; k < w; k++) sum = fma_slot(cols, vals, x, base + (int64_t)lane * w + k, sum);
   }
   const int64_t row = strip * kBiStrip + lane;
   const int src = row < n ? perm[row] - (int32_t)(strip * kBiStrip) : 0;
   const Real mine = __shfl_sync(0xffffffffu, sum, src);
   if (row < n) keep_range(y, row, mine, alpha, beta, begin, end);
}

template <typename Real>
tnlb_status launch(const tnlb_segments* seg, const int32_t* cols, const Real* vals, int32_t columns, const Real* x,
                   Real* y, Real alpha, Real beta, int32_t begin, int32_t end, tnlb_kernel kernel, int32_t tps, cudaStream_t st,
                   int* launches)
{
   const bool col = seg->organization == TNLB_COLUMN_MAJOR;
   *launches = 0;
   if (end <= begin) return TNLB_OK;
   switch (seg->format) {
      case TNLB_ELLPACK: {
         if (col) {
            k_ell_col<Real><<<grid_for((int64_t)end - begin, 256), 256, 0, st>>>(
               cols, vals, x, y, seg->n, seg->segment_size, seg->aligned_size, begin, end, alpha, beta);
         }
         else {
            int G = tps > 0 ? tps : 1;
            if (kernel == TNLB_KERNEL_DEFAULT && tps <= 0) G = seg->segment_size >= 32 ? 32 : (seg->segment_size >= 8 ? 8 : 1);
            const int64_t th = ((int64_t)end - begin) * G;
            switch (G) {
               case 1: k_ell_row<Real, 1><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               case 2: k_ell_row<Real, 2><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               case 4: k_ell_row<Real, 4><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               case 8: k_ell_row<Real, 8><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               case 16: k_ell_row<Real, 16><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               case 32: k_ell_row<Real, 32><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, seg->segment_size, begin, end, alpha, beta); break;
               default: set_error("threads per segment must be 1..32 for row-major Ellpack"); return TNLB_ERR_INVALID_ARGUMENT;
            }
         }
         break;
      }
      case TNLB_SLICED_ELLPACK: {
         if (seg->slices == 0) return TNLB_OK;
         if (col) {
            int G = tps > 0 ? tps : 1;
            if (kernel == TNLB_KERNEL_DEFAULT && tps <= 0) {
               const int64_t mean_w = seg->storage / ((int64_t)seg->slices * kSellSlice);
               G = mean_w >= 256 ? 8 : (mean_w >= 64 ? 4 : (mean_w >= 16 ? 2 : 1));
            }
            // narrow slices are stencils, whose lanes gather neighbours
            SellWindow win{};
            if (kernel == TNLB_KERNEL_DEFAULT && tps <= 0 && G >= 2 && G <= 4) {
               launch_window<Real>(seg, columns, cols, vals, x, y, alpha, beta, begin, end, st, &win);
               TNLB_CHECK_LAUNCH();
               if (win.per_block > 0) *launches = 1;
            }
            const int32_t* so = seg->slice_offsets.as<int32_t>();
            const int32_t* sw = seg->slice_segment_sizes.as<int32_t>();
            switch (G) {
               case 1:
                  // FP64: the slice walk (5-point 1024^2: 18.1 -> 15.7 us);
                  // FP32 entries are half the bytes per slice and the
                  // full-grid launch measured 0.6 us faster there
                  if (sizeof(Real) == 8) {
                     auto* k = k_sell_walk<Real>;
                     const unsigned g = resident_grid((const void*)k, 256, (int64_t)seg->slices * 32, 1);
                     k<<<g, 256, 0, st>>>(cols, vals, x, y, so, sw, seg->slices, begin, end, alpha, beta);
                  }
                  else
                     TNLB_CUDA_TRY((launch_sell_col<Real, 1>(seg, cols, vals, x, y, alpha, beta, begin, end, win, st)));
                  break;
               case 2: TNLB_CUDA_TRY((launch_sell_col<Real, 2>(seg, cols, vals, x, y, alpha, beta, begin, end, win, st))); break;
               case 4: TNLB_CUDA_TRY((launch_sell_col<Real, 4>(seg, cols, vals, x, y, alpha, beta, begin, end, win, st))); break;
               case 8: TNLB_CUDA_TRY((launch_sell_col<Real, 8>(seg, cols, vals, x, y, alpha, beta, begin, end, win, st))); break;
               default: set_error("threads per segment must be 1, 2, 4 or 8 for column-major SlicedEllpack"); return TNLB_ERR_INVALID_ARGUMENT;
            }
         }
         else {
            const int G = tps > 0 ? tps : 8;
            const int64_t th = ((int64_t)end - begin) * G;
            const int32_t* so = seg->slice_offsets.as<int32_t>();
            const int32_t* sw = seg->slice_segment_sizes.as<int32_t>();
            switch (G) {
               case 1: k_sell_row<Real, 1><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               case 2: k_sell_row<Real, 2><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               case 4: k_sell_row<Real, 4><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               case 8: k_sell_row<Real, 8><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               case 16: k_sell_row<Real, 16><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               case 32: k_sell_row<Real, 32><<<grid_for(th, 256), 256, 0, st>>>(cols, vals, x, y, so, sw, begin, end, alpha, beta); break;
               default: set_error("threads per segment must be 1..32 for row-major SlicedEllpack"); return TNLB_ERR_INVALID_ARGUMENT;
            }
         }
         break;
      }
      case TNLB_CHUNKED_ELLPACK: {
         if (seg->ch_slices == 0) return TNLB_OK;
         // mean slots of a chunk: even rows fill their slices (36 slots for 9 to
         // 45 entries), and there one pass over columns and values together is
         // the better one; power-law rows, 1000 to 2,000,000 of them, 1.1 (FP32)
         // to 5.6 times as fast by columns first
         const int64_t tall = seg->storage / ((int64_t)seg->ch_slices * kChunksInSlice);
         if (col && tall >= kChellTall && aligned16(cols)) {
            TNLB_CUDA_TRY((launch_chell_cols<Real, 4>(seg, cols, vals, x, y, alpha, beta, begin, end, st)));
            break;
         }
         auto kern = col ? k_chell<Real, true> : k_chell<Real, false>;
         kern<<<seg->ch_slices, kChunksInSlice, 0, st>>>(
            cols, vals, x, y, seg->ch_slice_size.as<int32_t>(), seg->ch_slice_chunk_size.as<int32_t>(),
            seg->ch_slice_first.as<int32_t>(), seg->ch_slice_pointer.as<int32_t>(),
            seg->ch_segment_to_chunk.as<int32_t>(), begin, end, alpha, beta);
         break;
      }
      case TNLB_BIELLPACK: {
         if (seg->strips == 0) return TNLB_OK;
         auto kern = col ? k_biell_col<Real> : k_biell_row<Real>;
         kern<<<grid_for(seg->strips, 8), 256, 0, st>>>(cols, vals, x, y, seg->bi_perm.as<int32_t>(),
                                                         seg->bi_group_pointers.as<int32_t>(), seg->n, seg->strips,
                                                         begin, end, alpha, beta);
         break;
      }
      default: set_error("format has no Ellpack-family kernel"); return TNLB_ERR_INVALID_ARGUMENT;
   }
   TNLB_CHECK_LAUNCH();
   *launches += 1;
   return TNLB_OK;
}

}  // namespace

tnlb_status spmv_ell_family(const tnlb_segments* seg, tnlb_real real, const int32_t* cols, const void* vals,
                            int32_t columns, const void* x, void* y, double alpha, double beta, int32_t begin, int32_t end,
                            tnlb_kernel kernel, int32_t tps, cudaStream_t stream, int* launches)
{
   if (real == TNLB_F64)
      return launch<double>(seg, cols, (const double*)vals, columns, (const double*)x, (double*)y, alpha, beta, begin, end,
                            kernel, tps, stream, launches);
   return launch<float>(seg, cols, (const float*)vals, columns, (const float*)x, (float*)y, (float)alpha, (float)beta, begin,
                        end, kernel, tps, stream, launches);
}

}  // namespace tnlb
