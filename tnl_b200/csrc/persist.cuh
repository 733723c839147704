// persist.cuh -- CG and BiCGStab iterations in one resident kernel.
//
// An iteration of CG on a matrix that fits L2 is three short passes over a few
// vectors between two dot products; as separate launches each pass pays for
// its launch, its ramp and its tail, and every vector goes through memory.
// Here one block per SM (cooperative launch, all resident) owns a contiguous
// run of rows for the whole solve:
//  * the vectors that only the owner reads (r, A p, x, and what else fits) stay
//    in shared memory; only the vector a product gathers from is in global
//    memory, and the matrix comes from L2 where it fits;
//  * a dot product is a grid-wide exchange: every block posts its partial sum
//    with the number of the exchange in the same 8-byte words and polls the
//    slots of all others, so that the sum and the barrier are one round trip;
//  * every block forms the scalars from the same partials in the same order, so
//    all take the same branch.  Waits are bounded.
// The row arithmetic and its order are those of the product kernels.
#pragma once

#include <cfloat>

#include "internal.cuh"
#include "reduce.cuh"
#include "solver_state.cuh"

namespace tnlb {

// a thread holds two rows' slots: the wider, the fewer threads have registers
constexpr int persist_threads(int L) { return L > 8 ? 256 : L > 5 ? 512 : 1024; }
constexpr int kPersistMaxBlocks = 256;
constexpr int kPersistSums = 2;
constexpr int kPersistSpin = 1 << 22;  // polls of one wait, about 3 s

// ------------------------------------------------------------ the exchange

// slots[parity][sum][block]: the partial's two halves, each with the number of
// the exchange.  A slot is written again two exchanges later, when every block
// has read it.
struct PersistSync {
   ulonglong2* slots;  // [2 * kPersistSums * kPersistMaxBlocks], zero before the launch
   int32_t* err;
};
constexpr size_t kPersistSlotBytes = sizeof(ulonglong2) * 2 * kPersistSums * kPersistMaxBlocks;
inline PersistSync persist_sync(const DeviceBuffer& b)  // kPersistSlotBytes and an int32_t
{
   return {b.as<ulonglong2>(), reinterpret_cast<int32_t*>(b.as<unsigned char>() + kPersistSlotBytes)};
}

__device__ __forceinline__ void persist_post(ulonglong2* slot, double v, uint32_t epoch)
{
   const unsigned long long bits = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
   const unsigned long long lo = e | (bits & 0xffffffffull), hi = e | (bits >> 32);
   asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&slot->x), "l"(lo) : "memory");
   asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(&slot->y), "l"(hi) : "memory");
}

__device__ __forceinline__ bool persist_poll(const ulonglong2* slot, uint32_t epoch, double& v)
{
   unsigned long long lo, hi;
   asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(lo) : "l"(&slot->x) : "memory");
   asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(hi) : "l"(&slot->y) : "memory");
   v = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
   return (uint32_t)(lo >> 32) == epoch && (uint32_t)(hi >> 32) == epoch;
}

// Totals of K per-thread values over the grid, the same in every thread: the
// slots carry all that is exchanged, so no fence is needed.  K = 0 is a barrier:
// what any thread of the grid wrote before is visible after.  False (in every
// thread) when the wait ran out.
template <int K>
__device__ __forceinline__ bool persist_sum(const double* v, double* out, const PersistSync& g, uint32_t& epoch)
{
   constexpr int KS = K > 0 ? K : 1;
   __shared__ double s_warp[KS][32];
   __shared__ double s_all[KS][kPersistMaxBlocks];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
   const int G = (int)gridDim.x;
   const uint32_t e = ++epoch;
   ulonglong2* slots = g.slots + (size_t)(e & 1u) * kPersistSums * kPersistMaxBlocks;
   double w[KS];
#pragma unroll
   for (int k = 0; k < K; k++) {
      w[k] = warp_sum(v[k]);
      if (lane == 0) s_warp[k][warp] = w[k];
   }
   __syncthreads();
   if (warp == 0) {
#pragma unroll
      for (int k = 0; k < K; k++) w[k] = warp_sum(lane < warps ? s_warp[k][lane] : 0.0);
      if (K == 0) w[0] = 0.0;
      if (lane == 0) {
         if (K == 0) asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
         for (int k = 0; k < KS; k++) persist_post(slots + k * kPersistMaxBlocks + blockIdx.x, w[k], e);
      }
   }
   int bad = 0;
   for (int b = threadIdx.x; b < G; b += blockDim.x) {
#pragma unroll
      for (int k = 0; k < KS; k++) {
         double t = 0.0;
         int it = 0;
         while (!persist_poll(slots + k * kPersistMaxBlocks + b, e, t) && ++it < kPersistSpin) {}
         if (it >= kPersistSpin) bad = 1;
         if (K > 0) s_all[k][b] = t;
      }
   }
   if (K == 0 && threadIdx.x < G) asm volatile("fence.acq_rel.gpu;" ::: "memory");
   if (__syncthreads_or(bad)) {
      if (threadIdx.x == 0) atomicExch(g.err, 1);
      return false;
   }
#pragma unroll
   for (int k = 0; k < K; k++) {
      double t = 0.0;
      for (int b = lane; b < G; b += 32) t += s_all[k][b];
      out[k] = warp_sum(t);
   }
   return true;
}

// ------------------------------------------------------------------- rows

// A matrix whose rows hold at most L slots, one thread per row: slot k of row i
// is at base + k * step.
enum { kPersistCsr = 0, kPersistEll = 1, kPersistSell = 2 };
template <typename Real>
struct PersistRows {
   const int32_t* off;    // CSR row offsets, SlicedEllpack slice offsets
   const int32_t* width;  // SlicedEllpack slice widths
   const int32_t* cols;
   const Real* vals;
   int32_t ell_width, ell_row, ell_step;  // Ellpack: base = i * ell_row
   int32_t colmajor;                      // SlicedEllpack
};

template <typename Real, int Kind>
__device__ __forceinline__ void persist_extent(const PersistRows<Real>& A, int32_t i, int64_t& base, int32_t& step,
                                               int32_t& count)
{
   if (Kind == kPersistCsr) {
      const int32_t b = __ldg(A.off + i);
      base = b;
      step = 1;
      count = __ldg(A.off + i + 1) - b;
   }
   else if (Kind == kPersistEll) {
      base = (int64_t)i * A.ell_row;
      step = A.ell_step;
      count = A.ell_width;
   }
   else {
      const int32_t sl = i / kSellSlice, in = i % kSellSlice;
      count = __ldg(A.width + sl);
      base = __ldg(A.off + sl) + (A.colmajor ? in : (int64_t)in * count);
      step = A.colmajor ? kSellSlice : 1;
   }
}

// f(i, (A x)_i, x_i) for the rows first + threadIdx.x, + blockDim.x, ... < last,
// as a pipeline: while a row's x are gathered, the next row's slots and the
// extent of the one after are on their way.  x is written by other blocks
// between two calls: plain loads, never the read-only path.
template <typename Real, int Kind, int L, typename F>
__device__ __forceinline__ void persist_product(const PersistRows<Real>& A, const Real* x, int32_t first, int32_t last,
                                                F&& f)
{
   const int32_t stride = (int32_t)blockDim.x;
   int64_t base = 0;
   int32_t step = 0, count = 0;
   int32_t c[L];
   Real v[L];
   auto slots = [&]() {
#pragma unroll
      for (int k = 0; k < L; k++) {
         c[k] = -1;
         v[k] = Real(0);
         if (k < count) {
            c[k] = __ldg(A.cols + base + (int64_t)k * step);
            v[k] = __ldg(A.vals + base + (int64_t)k * step);
         }
      }
   };
   int32_t i = first + (int32_t)threadIdx.x;
   if (i >= last) return;
   persist_extent<Real, Kind>(A, i, base, step, count);
   slots();
   if (i + stride < last) persist_extent<Real, Kind>(A, i + stride, base, step, count);
   while (true) {
      const Real xi = x[i];
      Real xk[L], w[L];
      bool on[L];
#pragma unroll
      for (int k = 0; k < L; k++) {
         on[k] = c[k] >= 0;
         w[k] = v[k];
         xk[k] = on[k] ? x[c[k]] : Real(0);
      }
      const int32_t next = i + stride;
      if (next < last) slots();
      if (next < last && next + stride < last) persist_extent<Real, Kind>(A, next + stride, base, step, count);
      Real s = Real(0);
#pragma unroll
      for (int k = 0; k < L; k++)
         if (on[k]) s += w[k] * xk[k];
      f(i, s, xi);
      if (next >= last) break;
      i = next;
   }
}

// ----------------------------------------------------------------- kernels

// The owner's vectors, most used first: the first `kept` of them live in shared
// memory while the kernel runs, the others stay where they are.
template <typename Real, int N>
struct PersistVectors {
   Real* v[N];
   int32_t kept;
   int32_t rows;  // per block
};

extern __shared__ __align__(16) unsigned char persist_smem[];

// Pointers indexed by i - first; `load` says which vectors' values are read on entry.
template <typename Real, int N>
__device__ __forceinline__ void persist_enter(const PersistVectors<Real, N>& V, int32_t first, int32_t last,
                                              Real* (&p)[N], unsigned load)
{
#pragma unroll
   for (int q = 0; q < N; q++) {
      p[q] = V.v[q] ? V.v[q] + first : nullptr;
      if (q < V.kept && V.v[q]) {
         Real* s = reinterpret_cast<Real*>(persist_smem) + (size_t)q * V.rows;
         if (load >> q & 1u)
            for (int32_t j = threadIdx.x; j < last - first; j += blockDim.x) s[j] = p[q][j];
         p[q] = s;
      }
   }
}
template <typename Real, int N>
__device__ __forceinline__ void persist_leave(const PersistVectors<Real, N>& V, int32_t first, int32_t last,
                                              Real* const (&p)[N], unsigned store)
{
#pragma unroll
   for (int q = 0; q < N; q++)
      if (q < V.kept && V.v[q] && (store >> q & 1u))
         for (int32_t j = threadIdx.x; j < last - first; j += blockDim.x) V.v[q][first + j] = p[q][j];
}

// CG (CG.hpp:60-107) from the state that the solver's first steps leave: at most
// `cap` iterations or until S->done.  V: A p (then z), r, x, d; d null without
// a preconditioner.  Each thread touches only its own rows of V, so no barrier
// stands between the passes but the exchanges.
template <typename Real, int Kind, int L>
__global__ void __launch_bounds__(persist_threads(L), 1)
   k_cg_persist(const PersistRows<Real> A, PersistVectors<Real, 4> V, Real* p, int32_t n, DevState* S, PersistSync g,
                int32_t cap)
{
   const int32_t first = (int32_t)imin64((int64_t)blockIdx.x * V.rows, n);
   const int32_t last = (int32_t)imin64((int64_t)first + V.rows, n);
   Real* own[4];
   persist_enter(V, first, last, own, 0b1110u);
   Real *const Ap = own[0], *const r = own[1], *const x = own[2], *const d = own[3];
   DevState s = *S;
   uint32_t epoch = 0;
   for (int32_t turn = 0; turn < cap && !s.done; turn++) {
      double acc = 0.0, t;
      persist_product<Real, Kind, L>(A, p, first, last, [&](int32_t i, Real y, Real pi) {
         Ap[i - first] = y;
         acc += (double)y * (double)pi;
      });
      if (!persist_sum<1>(&acc, &t, g, epoch)) return;
      s.s2 = t;
      if (t == 0.0) {
         s.residue = 0.0;
         s.done = 1;
         s.flag = 1;
         break;
      }
      s.alpha = s.s1 / t;
      const Real alpha = (Real)s.alpha;
      acc = 0.0;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) {
         const int32_t j = i - first;
         x[j] += alpha * p[i];
         const Real ri = r[j] - alpha * Ap[j];
         r[j] = ri;
         Real zi = ri;
         if (d) zi = ri / d[j];
         Ap[j] = zi;
         acc += (double)ri * (double)zi;
      }
      if (!persist_sum<1>(&acc, &t, g, epoch)) return;
      s.s2 = s.s1;
      s.s1 = t;
      s.beta = (s.s2 == 0.0) ? 0.0 : s.s1 / s.s2;
      s.residue = sqrt(s.s1) / s.normb;
      next_iteration(s);
      if (s.done) break;
      const Real beta = (Real)s.beta;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) p[i] = Ap[i - first] + beta * p[i];
      if (!persist_sum<0>(nullptr, nullptr, g, epoch)) return;
   }
   persist_leave(V, first, last, own, 0b0110u);
   if (blockIdx.x == 0 && threadIdx.x == 0) *S = s;
}

// BiCGStab (BICGStab.hpp:72-120).  V: A p, r, s, A s, r_ast, x, d.  s.done = 2
// leaves an iteration before its update of p, for a restart by the host.
constexpr int32_t kPersistRestart = 2;

template <typename Real, int Kind, int L>
__global__ void __launch_bounds__(persist_threads(L), 1)
   k_bicg_persist(const PersistRows<Real> A, PersistVectors<Real, 6> V, Real* p, Real* sv, int32_t n, DevState* S,
                  PersistSync g, int32_t cap)
{
   const int32_t first = (int32_t)imin64((int64_t)blockIdx.x * V.rows, n);
   const int32_t last = (int32_t)imin64((int64_t)first + V.rows, n);
   Real* own[6];
   persist_enter(V, first, last, own, 0b111010u);
   Real *const Ap = own[0], *const r = own[1], *const As = own[2], *const ra = own[3], *const x = own[4],
               *const d = own[5];
   DevState s = *S;
   uint32_t epoch = 0;
   for (int32_t turn = 0; turn < cap; turn++) {
      const bool go = check_next(s);
      s.it++;
      if (!go) {
         s.done = 1;
         break;
      }
      double acc[2] = {0.0, 0.0}, t[2];
      persist_product<Real, Kind, L>(A, p, first, last, [&](int32_t i, Real y, Real) {
         const int32_t j = i - first;
         if (d) y = y / d[j];
         Ap[j] = y;
         acc[0] += (double)y * (double)ra[j];
      });
      if (!persist_sum<1>(acc, t, g, epoch)) return;
      s.alpha = s.rho / t[0];
      const Real alpha = (Real)s.alpha;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x)
         sv[i] = r[i - first] - alpha * Ap[i - first];
      if (!persist_sum<0>(nullptr, nullptr, g, epoch)) return;
      acc[0] = acc[1] = 0.0;
      persist_product<Real, Kind, L>(A, sv, first, last, [&](int32_t i, Real y, Real si) {
         const int32_t j = i - first;
         if (d) y = y / d[j];
         As[j] = y;
         acc[0] += (double)y * (double)si;
         acc[1] += (double)y * (double)y;
      });
      if (!persist_sum<2>(acc, t, g, epoch)) return;
      s.omega = t[0] / t[1];
      const Real omega = (Real)s.omega;
      acc[0] = acc[1] = 0.0;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) {
         const int32_t j = i - first;
         const Real si = sv[i];
         x[j] += alpha * p[i] + omega * si;
         const Real ri = si - omega * As[j];
         r[j] = ri;
         acc[0] += (double)ri * (double)ra[j];
         acc[1] += (double)ri * (double)ri;
      }
      if (!persist_sum<2>(acc, t, g, epoch)) return;
      s.rho_old = s.rho;
      s.rho = t[0];
      if (fabs(s.rho) < DBL_EPSILON * DBL_EPSILON * s.r_ast_sqnorm) {
         s.done = kPersistRestart;
         break;
      }
      s.residue = sqrt(t[1]) / s.normb;
      s.beta = (s.rho / s.rho_old) * (s.alpha / s.omega);
      const Real beta = (Real)s.beta, bo = (Real)(s.beta * s.omega);
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x)
         p[i] = r[i - first] + beta * p[i] - bo * Ap[i - first];
      if (!persist_sum<0>(nullptr, nullptr, g, epoch)) return;
   }
   persist_leave(V, first, last, own, 0b010011u);
   if (blockIdx.x == 0 && threadIdx.x == 0) *S = s;
}

// -------------------------------------------------------------------- host

// Whether the matrix has rows that one thread can take: the longest holds at
// most 16 slots.
inline bool persist_rows_fit(const tnlb_segments* seg)
{
   switch (seg->format) {
      case TNLB_CSR: return seg->max_row > 0 && seg->max_row <= 16;
      case TNLB_ELLPACK: return seg->segment_size > 0 && seg->segment_size <= 16;
      case TNLB_SLICED_ELLPACK: return seg->max_size > 0 && seg->max_size <= 16;
      default: return false;
   }
}

template <typename Real>
PersistRows<Real> persist_rows(const tnlb_segments* seg, const int32_t* cols, const Real* vals)
{
   PersistRows<Real> A{};
   const bool col = seg->organization == TNLB_COLUMN_MAJOR;
   A.cols = cols;
   A.vals = vals;
   A.colmajor = col;
   if (seg->format == TNLB_CSR) A.off = seg->offsets.as<int32_t>();
   if (seg->format == TNLB_SLICED_ELLPACK) {
      A.off = seg->slice_offsets.as<int32_t>();
      A.width = seg->slice_segment_sizes.as<int32_t>();
   }
   if (seg->format == TNLB_ELLPACK) {
      A.ell_width = seg->segment_size;
      A.ell_row = col ? 1 : seg->segment_size;
      A.ell_step = col ? seg->aligned_size : 1;
   }
   return A;
}

// Launch shape: one block per SM at most, at least kPersistMinRows rows each.
constexpr int32_t kPersistMinRows = 128;
struct PersistShape {
   int32_t blocks = 0, threads = 0, rows = 0, kept = 0;
   size_t smem = 0;
};

// False where the device cannot hold the grid.
inline bool persist_shape(const void* kernel, int32_t n, int vectors, size_t real, PersistShape& sh)
{
   int dev = 0, sms = 0, coop = 0, smem = 0, occ = 0;
   cudaFuncAttributes fa{};
   if (cudaGetDevice(&dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
       cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || !coop) {
      cudaGetLastError();
      return false;
   }
   const int64_t per = imax64(kPersistMinRows, (n + sms - 1) / sms);
   sh.rows = (int32_t)((per + 31) / 32 * 32);
   sh.blocks = (int32_t)((n + (int64_t)sh.rows - 1) / sh.rows);
   sh.threads = (int32_t)imin64(fa.maxThreadsPerBlock, sh.rows);
   const int64_t room = (int64_t)smem - (int64_t)fa.sharedSizeBytes;
   sh.kept = (int32_t)imin64(vectors, room / ((int64_t)sh.rows * (int64_t)real));
   sh.smem = (size_t)sh.kept * sh.rows * real;
   if (sh.blocks > kPersistMaxBlocks ||
       cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh.smem) != cudaSuccess ||
       cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, sh.threads, sh.smem) != cudaSuccess ||
       (int64_t)occ * sms < sh.blocks) {
      cudaGetLastError();
      return false;
   }
   return true;
}

template <typename Real, int Kind, template <typename, int, int> class K>
const void* persist_pick(int32_t longest)
{
   return longest <= 5 ? K<Real, Kind, 5>::get() : longest <= 8 ? K<Real, Kind, 8>::get() : K<Real, Kind, 16>::get();
}
template <typename Real, template <typename, int, int> class K>
const void* persist_pick(const tnlb_segments* seg)
{
   if (seg->format == TNLB_CSR) return persist_pick<Real, kPersistCsr, K>(seg->max_row);
   if (seg->format == TNLB_ELLPACK) return persist_pick<Real, kPersistEll, K>(seg->segment_size);
   return persist_pick<Real, kPersistSell, K>(seg->max_size);
}
template <typename Real, int Kind, int L>
struct CgPersistKernel {
   static const void* get() { return (const void*)k_cg_persist<Real, Kind, L>; }
};
template <typename Real, int Kind, int L>
struct BicgPersistKernel {
   static const void* get() { return (const void*)k_bicg_persist<Real, Kind, L>; }
};

}  // namespace tnlb
