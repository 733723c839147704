// persist.cu -- CG and BiCGStab iterations in one resident kernel.
//
// An iteration of CG on a matrix that fits L2 (persist_pays) is three short passes
// over a few vectors between two dot products; as separate launches each pass pays for
// its launch, its ramp and its tail, and every vector goes through memory.
// Here one block per SM (cooperative launch, all resident) owns a contiguous
// run of rows for the whole solve:
//  * the vectors that only the owner reads (r, A p, x, and what else fits) stay
//    in shared memory; only the vector a product gathers from is in global
//    memory, and the matrix comes from L2 where it fits;
//  * a dot product is a grid-wide exchange: every block posts its partial sum
//    with the number of the exchange in the same 8-byte words, block 0 takes
//    them and sends the total back the same way, so that the sum is also the
//    barrier;
//  * up to kClusterRows rows one cluster of 16 blocks does it all: gathers and
//    sums go through distributed shared memory and the barrier is the cluster's
//    (100 x 100: 9.0 us an iteration over the grid, 4.3 in the cluster);
//  * every block forms the scalars from the same totals, so all take the same
//    branch.  Waits are bounded.
// The row arithmetic and its order are those of the product kernels.
#include <cfloat>

#include "persist.cuh"
#include "reduce.cuh"

namespace tnlb {
namespace {

// A thread holds two rows' slots: the wider, the fewer threads have registers.
constexpr int persist_threads(int L) { return L > 8 ? 256 : L > 5 ? 512 : 1024; }
// Shared memory of a warp's staged CSR entries.
template <typename Real, int L>
constexpr int kPersistStage = 32 * L * (int)(sizeof(Real) + sizeof(int32_t));
constexpr int kPersistSpin = 1 << 22;  // polls of one wait, about 3 s

// ------------------------------------------------------------ the exchange

__device__ __forceinline__ void persist_post(ulonglong2* slot, double v, uint32_t epoch)
{
   const unsigned long long bits = (unsigned long long)__double_as_longlong(v), e = (unsigned long long)epoch << 32;
   const unsigned long long lo = e | (bits & 0xffffffffull), hi = e | (bits >> 32);
   asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(slot), "l"(lo), "l"(hi) : "memory");
}

// Waits for the slot's value of the exchange; false when the wait ran out.
__device__ __forceinline__ bool persist_take(const ulonglong2* slot, uint32_t epoch, double& v)
{
   for (int it = 0; it < kPersistSpin; it++) {
      unsigned long long lo, hi;
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo), "=l"(hi) : "l"(slot) : "memory");
      if ((uint32_t)(lo >> 32) == epoch && (uint32_t)(hi >> 32) == epoch) {
         v = __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
         return true;
      }
   }
   return false;
}
__device__ __forceinline__ void persist_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Totals of K per-thread values over the grid, the same in every thread: the
// slots carry all that is exchanged, so no fence is needed.  K = 0 is a barrier:
// what any thread of the grid wrote before is visible after.  False (in every
// thread) when a wait ran out.  Block 0 takes the partial sums of all and sends
// each block the total on a line of its own: with every block polling the slots
// of all others the polls queued up at their lines, 9000 cycles an exchange of
// 148 blocks.
struct PersistGrid {
   static constexpr bool kCluster = false;
   PersistSync g;
   uint32_t epoch;
   __host__ __device__ explicit PersistGrid(const PersistSync& s) : g(s), epoch(0) {}
   __device__ __forceinline__ void start() {}
   template <int K>
   __device__ __forceinline__ bool sum(const double* v, double* out);
};
template <int K>
__device__ __forceinline__ bool PersistGrid::sum(const double* v, double* out)
{
   constexpr int KS = K > 0 ? K : 1;
   __shared__ double s_warp[KS][32];
   __shared__ double s_total[2][KS];  // by parity: read before the next but one is written
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
   const int G = (int)gridDim.x;
   const uint32_t e = ++epoch;
   ulonglong2* in = g.slots + (size_t)(e & 1u) * kPersistSums * kPersistMaxBlocks;
   ulonglong2* to = g.slots + (size_t)2 * kPersistSums * kPersistMaxBlocks + (size_t)blockIdx.x * kPersistLine;
   double w[KS];
#pragma unroll
   for (int k = 0; k < K; k++) {
      w[k] = warp_sum(v[k]);
      if (lane == 0) s_warp[k][warp] = w[k];
   }
   __syncthreads();
   bool bad = false;
   if (blockIdx.x == 0) {
      // the sums of the others: a warp takes 32 blocks' slots
      __shared__ double s_part[KS][kPersistMaxBlocks / 32];
      if (warp == 0)
#pragma unroll
         for (int k = 0; k < K; k++) w[k] = warp_sum(lane < warps ? s_warp[k][lane] : 0.0);
      for (int b0 = warp * 32; b0 < G; b0 += warps * 32) {
         double t[KS];
#pragma unroll
         for (int k = 0; k < KS; k++) {
            t[k] = 0.0;
            const int b = b0 + lane;
            if (b == 0)
               t[k] = K > 0 ? w[k] : 0.0;
            else if (b < G)
               bad |= !persist_take(in + k * kPersistMaxBlocks + b, e, t[k]);
            t[k] = warp_sum(t[k]);
            if (lane == 0) s_part[k][b0 / 32] = t[k];
         }
      }
      if (K == 0) persist_fence();
      if (!__syncthreads_or(bad)) {
         double t[KS];
#pragma unroll
         for (int k = 0; k < KS; k++) {
            t[k] = 0.0;
            for (int q = 0; q * 32 < G; q++) t[k] += s_part[k][q];
            if (K > 0) out[k] = t[k];
         }
         if (K == 0) persist_fence();
         for (int b = threadIdx.x; b < G; b += blockDim.x)
#pragma unroll
            for (int k = 0; k < KS; k++)
               if (b > 0)
                  persist_post(g.slots + (size_t)2 * kPersistSums * kPersistMaxBlocks + (size_t)b * kPersistLine + k,
                               t[k], e);
         return true;
      }
      bad = true;
   }
   else {
      if (warp == 0) {
#pragma unroll
         for (int k = 0; k < K; k++) w[k] = warp_sum(lane < warps ? s_warp[k][lane] : 0.0);
         if (lane == 0) {
            if (K == 0) persist_fence();
#pragma unroll
            for (int k = 0; k < KS; k++) persist_post(in + k * kPersistMaxBlocks + blockIdx.x, K > 0 ? w[k] : 0.0, e);
#pragma unroll
            for (int k = 0; k < KS; k++) {
               double t = 0.0;
               bad |= !persist_take(to + k, e, t);
               s_total[e & 1u][k] = t;
            }
            if (K == 0) persist_fence();
         }
      }
      if (!__syncthreads_or(bad)) {
#pragma unroll
         for (int k = 0; k < K; k++) out[k] = s_total[e & 1u][k];
         return true;
      }
   }
   if (threadIdx.x == 0) atomicExch(g.err, 1);
   return false;
}

// The same over one cluster of blocks, for small systems: partial sums go
// straight to the other blocks' shared memory, and the barrier is the cluster's
// own, which also orders what was written to shared memory.
constexpr int kPersistCluster = 16;
struct PersistCluster {
   static constexpr bool kCluster = true;
   uint32_t turn;
   __host__ __device__ explicit PersistCluster(const PersistSync&) : turn(0) {}
   __device__ __forceinline__ void start() { barrier(); }
   __device__ __forceinline__ static void barrier()
   {
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
   }
   template <int K>
   __device__ __forceinline__ bool sum(const double* v, double* out)
   {
      if (K == 0) {
         barrier();
         return true;
      }
      constexpr int KS = K > 0 ? K : 1;
      __shared__ double s_warp[KS][32];
      // written again two turns later, when every block has read it
      __shared__ double s_all[2][KS][kPersistCluster];
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
      const uint32_t e = ++turn & 1u;
#pragma unroll
      for (int k = 0; k < K; k++) {
         const double w = warp_sum(v[k]);
         if (lane == 0) s_warp[k][warp] = w;
      }
      __syncthreads();
      if (warp == 0) {
#pragma unroll
         for (int k = 0; k < K; k++) {
            const double w = warp_sum(lane < warps ? s_warp[k][lane] : 0.0);
            if (lane < (int)gridDim.x) {
               uint32_t to;
               asm("mapa.shared::cluster.u32 %0, %1, %2;"
                   : "=r"(to)
                   : "r"((uint32_t)__cvta_generic_to_shared(&s_all[e][k][blockIdx.x])), "r"(lane));
               asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(to), "d"(w) : "memory");
            }
         }
      }
      barrier();
#pragma unroll
      for (int k = 0; k < K; k++) {
         double t = 0.0;
         for (int b = 0; b < (int)gridDim.x; b++) t += s_all[e][k][b];
         out[k] = t;
      }
      return true;
   }
};

// A vector that the products gather from: in global memory, or in a cluster
// each block's rows in its own shared memory.
template <typename Real, bool Cluster>
struct PersistGather {
   Real* v;  // of row 0
   __device__ __forceinline__ PersistGather(Real* global, Real*, int32_t, int32_t) : v(global) {}
   __device__ __forceinline__ Real at(int32_t c) const { return v[c]; }
   __device__ __forceinline__ Real& own(int32_t i) const { return v[i]; }
};
__device__ __forceinline__ double persist_remote(uint32_t a, double)
{
   double v;
   asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
   return v;
}
__device__ __forceinline__ float persist_remote(uint32_t a, float)
{
   float v;
   asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
   return v;
}
template <typename Real>
struct PersistGather<Real, true> {
   Real* s;  // of row `first`
   uint32_t base, rows, magic;
   int32_t first;
   __device__ __forceinline__ PersistGather(Real*, Real* shared, int32_t first_, int32_t rows_)
      : s(shared), base((uint32_t)__cvta_generic_to_shared(shared)), rows((uint32_t)rows_),
        magic(0xffffffffu / (uint32_t)rows_ + 1u), first(first_)
   {
   }
   __device__ __forceinline__ Real at(int32_t c) const
   {
      // c / rows, exact while c * rows < 2^32
      const uint32_t block = __umulhi((uint32_t)c, magic), a = base + ((uint32_t)c - block * rows) * sizeof(Real);
      uint32_t from;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(from) : "r"(a), "r"(block));
      return persist_remote(from, Real(0));
   }
   __device__ __forceinline__ Real& own(int32_t i) const { return s[i - first]; }
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
template <typename Real, int Kind, int L, typename X, typename F>
__device__ __forceinline__ void persist_product(const PersistRows<Real>& A, const X& x, int32_t first, int32_t last,
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
      const Real xi = x.own(i);
      Real xk[L], w[L];
      bool on[L];
#pragma unroll
      for (int k = 0; k < L; k++) {
         on[k] = c[k] >= 0;
         w[k] = v[k];
         xk[k] = on[k] ? x.at(c[k]) : Real(0);
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

// The same for CSR rows of more than 5 entries over the grid.  32 rows' entries
// are one contiguous run, but a lane that reads its own row touches a line of its
// own with every load.  So a warp reads the run together and its rows from
// `stage` in shared memory, while the next rows' run is on its way: 41 BiCGStab
// iterations on 95 x 96 x 97 (FP64, 7 entries) 2.88 ms after 3.10.  Five-entry
// rows gain nothing (201 CG iterations on 1024 x 1024 6.88 ms against 6.79).
template <typename Real, int L, typename X, typename F>
__device__ __forceinline__ void persist_product_csr(const PersistRows<Real>& A, const X& x, int32_t first, int32_t last,
                                                    unsigned char* stage, F&& f)
{
   const int lane = threadIdx.x & 31;
   const int32_t stride = (int32_t)blockDim.x;
   Real* sv = reinterpret_cast<Real*>(stage + (size_t)(threadIdx.x >> 5) * kPersistStage<Real, L>);
   int32_t* sc = reinterpret_cast<int32_t*>(sv + 32 * L);
   int32_t i = first + (int32_t)threadIdx.x;
   int32_t b = 0, e = 0, b1 = 0, e1 = 0, start = 0;  // this row's and the next's entries
   int32_t c[L];
   Real v[L];
   auto extent = [&](int32_t r, int32_t& from, int32_t& to) {
      from = r < last ? __ldg(A.off + r) : 0;
      to = r < last ? __ldg(A.off + r + 1) : 0;
   };
   auto fetch = [&](int32_t from, int32_t to) {
      start = __shfl_sync(0xffffffffu, from, 0);
      const int32_t end = (int32_t)__reduce_max_sync(0xffffffffu, (unsigned)to);
#pragma unroll
      for (int u = 0; u < L; u++) {
         const int32_t k = start + 32 * u + lane;
         c[u] = k < end ? ld_stream(A.cols + k) : -1;
         v[u] = k < end ? ld_stream(A.vals + k) : Real(0);
      }
   };
   if (i - lane >= last) return;
   extent(i, b, e);
   fetch(b, e);
   extent(i + stride, b1, e1);
   while (true) {
#pragma unroll
      for (int u = 0; u < L; u++) {
         sc[32 * u + lane] = c[u];
         sv[32 * u + lane] = v[u];
      }
      __syncwarp();
      const int32_t at = b - start, count = e - b;
      const bool more = i + stride - lane < last;  // the same in the whole warp
      if (more) fetch(b1, e1);
      Real xk[L], w[L];
      bool on[L];
#pragma unroll
      for (int k = 0; k < L; k++) {
         const int32_t ck = k < count ? sc[at + k] : -1;
         on[k] = ck >= 0;
         w[k] = k < count ? sv[at + k] : Real(0);
         xk[k] = on[k] ? x.at(ck) : Real(0);
      }
      b = b1;
      e = e1;
      if (more) extent(i + 2 * stride, b1, e1);
      Real s = Real(0);
#pragma unroll
      for (int k = 0; k < L; k++)
         if (on[k]) s += w[k] * xk[k];
      if (i < last) f(i, s, x.own(i));
      if (!more) break;
      i += stride;
      __syncwarp();
   }
}

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

// Where gathered vector q lies in a cluster's blocks, behind the owner's vectors;
// and its copy from (in) and to global memory, where the grid has it anyway.
template <typename Real, typename V>
__device__ __forceinline__ Real* persist_shared(const V& v, int q)
{
   return reinterpret_cast<Real*>(persist_smem) + (size_t)(v.kept + q) * v.rows;
}
template <typename Real>
__device__ __forceinline__ void persist_gathered(const PersistGather<Real, false>&, Real*, int32_t, int32_t, bool)
{
}
template <typename Real>
__device__ __forceinline__ void persist_gathered(const PersistGather<Real, true>& x, Real* global, int32_t first,
                                                 int32_t last, bool in)
{
   for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) {
      if (in)
         x.own(i) = global[i];
      else
         global[i] = x.own(i);
   }
}

// A product as the kernel's matrix and blocks take it.
template <typename Real, int Kind, int L, typename Sync, typename V, typename X, typename F>
__device__ __forceinline__ void persist_apply(const PersistRows<Real>& A, const V& v, const X& x, int32_t first,
                                              int32_t last, F&& f)
{
   if constexpr (Kind == kPersistCsr && L > 5 && !Sync::kCluster)
      persist_product_csr<Real, L>(A, x, first, last, persist_smem + (size_t)v.kept * v.rows * sizeof(Real), f);
   else
      persist_product<Real, Kind, L>(A, x, first, last, f);
}

// CG (CG.hpp:60-107) from the state that the solver's first steps leave: at most
// `cap` iterations or until S->done.  V: A p (then z), r, x, d; d null without
// a preconditioner.  Each thread touches only its own rows of V, so no barrier
// stands between the passes but the exchanges.
template <typename Real, int Kind, int L, typename Sync>
__global__ void __launch_bounds__(persist_threads(L), 1)
   k_cg_persist(const PersistRows<Real> A, PersistVectors<Real, 4> V, Real* p_global, int32_t n, DevState* S,
                PersistSync slots, int32_t cap)
{
   const int32_t first = (int32_t)imin64((int64_t)blockIdx.x * V.rows, n);
   const int32_t last = (int32_t)imin64((int64_t)first + V.rows, n);
   Real* own[4];
   persist_enter(V, first, last, own, 0b1110u);
   Real *const Ap = own[0], *const r = own[1], *const x = own[2], *const d = own[3];
   const PersistGather<Real, Sync::kCluster> p(p_global, persist_shared<Real>(V, 0), first, V.rows);
   persist_gathered(p, p_global, first, last, true);
   DevState s = *S;
   Sync g(slots);
   g.start();
   for (int32_t turn = 0; turn < cap && !s.done; turn++) {
      double acc = 0.0, t;
      persist_apply<Real, Kind, L, Sync>(A, V, p, first, last, [&](int32_t i, Real y, Real pi) {
         Ap[i - first] = y;
         acc += (double)y * (double)pi;
      });
      if (!g.template sum<1>(&acc, &t)) return;
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
         x[j] += alpha * p.own(i);
         const Real ri = r[j] - alpha * Ap[j];
         r[j] = ri;
         Real zi = ri;
         if (d) zi = ri / d[j];
         Ap[j] = zi;
         acc += (double)ri * (double)zi;
      }
      if (!g.template sum<1>(&acc, &t)) return;
      s.s2 = s.s1;
      s.s1 = t;
      s.beta = (s.s2 == 0.0) ? 0.0 : s.s1 / s.s2;
      s.residue = sqrt(s.s1) / s.normb;
      next_iteration(s);
      if (s.done) break;
      const Real beta = (Real)s.beta;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) p.own(i) = Ap[i - first] + beta * p.own(i);
      if (!g.template sum<0>(nullptr, nullptr)) return;
   }
   persist_leave(V, first, last, own, 0b0110u);
   persist_gathered(p, p_global, first, last, false);
   if (blockIdx.x == 0 && threadIdx.x == 0) *S = s;
}

// BiCGStab (BICGStab.hpp:72-120).  V: A p, r, A s, r_ast, x, d.

template <typename Real, int Kind, int L, typename Sync>
__global__ void __launch_bounds__(persist_threads(L), 1)
   k_bicg_persist(const PersistRows<Real> A, PersistVectors<Real, 6> V, Real* p_global, Real* s_global, int32_t n,
                  DevState* S, PersistSync slots, int32_t cap)
{
   const int32_t first = (int32_t)imin64((int64_t)blockIdx.x * V.rows, n);
   const int32_t last = (int32_t)imin64((int64_t)first + V.rows, n);
   Real* own[6];
   persist_enter(V, first, last, own, 0b111010u);
   Real *const Ap = own[0], *const r = own[1], *const As = own[2], *const ra = own[3], *const x = own[4],
               *const d = own[5];
   const PersistGather<Real, Sync::kCluster> p(p_global, persist_shared<Real>(V, 0), first, V.rows),
      sv(s_global, persist_shared<Real>(V, 1), first, V.rows);
   persist_gathered(p, p_global, first, last, true);
   DevState s = *S;
   Sync g(slots);
   g.start();
   for (int32_t turn = 0; turn < cap; turn++) {
      const bool go = check_next(s);
      s.it++;
      if (!go) {
         s.done = 1;
         break;
      }
      double acc[2] = {0.0, 0.0}, t[2];
      persist_apply<Real, Kind, L, Sync>(A, V, p, first, last, [&](int32_t i, Real y, Real) {
         const int32_t j = i - first;
         if (d) y = y / d[j];
         Ap[j] = y;
         acc[0] += (double)y * (double)ra[j];
      });
      if (!g.template sum<1>(acc, t)) return;
      s.alpha = s.rho / t[0];
      const Real alpha = (Real)s.alpha;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x)
         sv.own(i) = r[i - first] - alpha * Ap[i - first];
      if (!g.template sum<0>(nullptr, nullptr)) return;
      acc[0] = acc[1] = 0.0;
      persist_apply<Real, Kind, L, Sync>(A, V, sv, first, last, [&](int32_t i, Real y, Real si) {
         const int32_t j = i - first;
         if (d) y = y / d[j];
         As[j] = y;
         acc[0] += (double)y * (double)si;
         acc[1] += (double)y * (double)y;
      });
      if (!g.template sum<2>(acc, t)) return;
      s.omega = t[0] / t[1];
      const Real omega = (Real)s.omega;
      acc[0] = acc[1] = 0.0;
      for (int32_t i = first + (int32_t)threadIdx.x; i < last; i += blockDim.x) {
         const int32_t j = i - first;
         const Real si = sv.own(i);
         x[j] += alpha * p.own(i) + omega * si;
         const Real ri = si - omega * As[j];
         r[j] = ri;
         acc[0] += (double)ri * (double)ra[j];
         acc[1] += (double)ri * (double)ri;
      }
      if (!g.template sum<2>(acc, t)) return;
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
         p.own(i) = r[i - first] + beta * p.own(i) - bo * Ap[i - first];
      if (!g.template sum<0>(nullptr, nullptr)) return;
   }
   persist_leave(V, first, last, own, 0b010011u);
   persist_gathered(p, p_global, first, last, false);
   if (blockIdx.x == 0 && threadIdx.x == 0) *S = s;
}

// --------------------------------------------------------- Gram-Schmidt

__device__ __forceinline__ void persist_fetch(double* dst, const double* src)
{
   asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                : "memory");
}
__device__ __forceinline__ void persist_fetch(float* dst, const float* src)
{
   asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                : "memory");
}

// Modified Gram-Schmidt of w against the columns V_0 .. V_(cols-1), `passes`
// times (GMRES.hpp:497-547): h[l * 64 + k] = (w, V_k), w -= h V_k, then
// *norm = |w| and V_cols = w / |w|.  w and two columns stay in shared memory:
// each column is read once a pass, and the next one is on its way while the
// blocks exchange a dot product.  A launch for each of the steps, reading
// both columns and w and writing w, took 7.8 us at 1,024,000 rows; a step takes
// 4.5 here, most of it the exchange.
template <typename Real, typename Sync>
__global__ void __launch_bounds__(1024, 1)
   k_mgs_persist(Real* V, int64_t ld, const Real* w, int32_t cols, int32_t passes, int32_t rows, int32_t n, double* h,
                 double* norm, PersistSync slots)
{
   const int32_t first = (int32_t)imin64((int64_t)blockIdx.x * rows, n);
   const int32_t count = (int32_t)imin64(rows, n - first);
   Real* wl = reinterpret_cast<Real*>(persist_smem);
   Real* buf[2] = {wl + rows, wl + 2 * (size_t)rows};
   const int32_t steps = cols * passes;
   // a thread reads and writes its own entries only: no barrier guards the
   // buffers, only its own copies
   auto fetch = [&](int32_t t) {
      if (t >= steps) return;
      const Real* src = V + (int64_t)(t % cols) * ld + first;
      Real* dst = t & 1 ? buf[1] : buf[0];
      for (int32_t j = threadIdx.x; j < count; j += blockDim.x) persist_fetch(dst + j, src + j);
   };
   fetch(0);
   fetch(1);
   for (int32_t j = threadIdx.x; j < count; j += blockDim.x) wl[j] = w[first + j];
   Sync g(slots);
   g.start();
   double t = 0.0;
   for (int32_t q = 0; q <= steps; q++) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      const Real* v = q & 1 ? buf[1] : buf[0];
      const Real* before = q & 1 ? buf[0] : buf[1];
      const Real hq = (Real)t;
      double acc = 0.0;
      for (int32_t j = threadIdx.x; j < count; j += blockDim.x) {
         Real wi = wl[j];
         if (q > 0) {
            wi = wi - hq * before[j];
            wl[j] = wi;
         }
         acc += (double)wi * (double)(q < steps ? v[j] : wi);
      }
      if (q > 0) fetch(q + 1);
      if (!g.template sum<1>(&acc, &t)) return;
      if (blockIdx.x == 0 && threadIdx.x == 0 && q < steps) h[q / cols * 64 + q % cols] = t;
   }
   const double nw = sqrt(t);
   const Real scale = (Real)(1.0 / nw);
   Real* out = V + (int64_t)cols * ld + first;
   for (int32_t j = threadIdx.x; j < count; j += blockDim.x) out[j] = scale * wl[j];
   if (blockIdx.x == 0 && threadIdx.x == 0) *norm = nw;
}

// -------------------------------------------------------------------- host

// One block per SM at most, at least kPersistMinRows rows each; up to
// kClusterRows rows one cluster, all of whose vectors (the owner's and the
// `gathered` ones) have to fit shared memory.  `warp_stage`: bytes of a warp's
// staged entries.
// us an iteration of CG over the grid and in the cluster (FP64; BiCGStab and FP32
// alike unless stated): 5 slots 3000 rows 8.1 and 3.3, 20,000 8.4 and 5.9, 40,000
// 8.8 and 7.8; 7 slots 20,000 8.4 and 6.3, 40,000 8.9 and 8.6.  16 SMs read wide
// rows too slowly: 15 slots 10,000 rows 8.7 and 7.4, 14,000 8.4 and 9.0, 20,000 8.7
// and 10.8 (FP32 20,000 9.2 and 8.8).  30 GMRES steps (MGSR): 20,000 rows 3036 and
// 2610, 60,000 3117 and 3103.
constexpr int32_t kPersistMinRows = 128;
constexpr int64_t kClusterRows = 20000, kClusterWideRows = 12000;

bool persist_shape(const void* kernel, bool cluster, int64_t n, int vectors, int gathered, size_t real, int warp_stage,
                   PersistShape& sh)
{
   int dev = 0, sms = 0, coop = 0, smem = 0, occ = 0;
   cudaFuncAttributes fa{};
   sh = PersistShape{};
   if (n > INT32_MAX || cudaGetDevice(&dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
       cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || !coop) {
      cudaGetLastError();
      return false;
   }
   const int64_t blocks = cluster ? kPersistCluster : sms;
   const int64_t per = imax64(cluster ? 32 : kPersistMinRows, (n + blocks - 1) / blocks);
   sh.rows = (int32_t)((per + 31) / 32 * 32);
   sh.blocks = cluster ? kPersistCluster : (int32_t)((n + sh.rows - 1) / sh.rows);
   sh.cluster = cluster ? kPersistCluster : 0;
   sh.threads = (int32_t)imin64(fa.maxThreadsPerBlock, sh.rows);
   const int64_t stage = cluster ? 0 : (int64_t)warp_stage * (sh.threads / 32);
   const int64_t room = (int64_t)smem - (int64_t)fa.sharedSizeBytes - stage;
   sh.kept = (int32_t)imin64(vectors, room / ((int64_t)sh.rows * (int64_t)real));
   sh.smem = (size_t)(sh.kept + (cluster ? gathered : 0)) * sh.rows * real;
   const bool fits = (int64_t)sh.smem <= room;
   sh.smem += (size_t)stage;
   if (sh.blocks > kPersistMaxBlocks || !fits || (cluster && sh.kept < vectors) ||
       // the same value from every thread: the attribute is the kernel's, not the launch's
       cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem - (int)fa.sharedSizeBytes) !=
          cudaSuccess) {
      cudaGetLastError();
      return false;
   }
   if (cluster) {
      cudaLaunchConfig_t cfg{};
      cudaLaunchAttribute at{};
      cfg.gridDim = dim3(sh.blocks);
      cfg.blockDim = dim3(sh.threads);
      cfg.dynamicSmemBytes = sh.smem;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = kPersistCluster;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
          cudaOccupancyMaxActiveClusters(&occ, kernel, &cfg) != cudaSuccess || occ < 1) {
         cudaGetLastError();
         return false;
      }
   }
   else if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, sh.threads, sh.smem) != cudaSuccess ||
            (int64_t)occ * sms < sh.blocks) {
      cudaGetLastError();
      return false;
   }
   sh.kernel = kernel;
   return true;
}

int64_t l2_bytes()
{
   int dev = 0, bytes = 0;
   if (cudaGetDevice(&dev) != cudaSuccess ||
       cudaDeviceGetAttribute(&bytes, cudaDevAttrL2CacheSize, dev) != cudaSuccess)
      cudaGetLastError();
   return bytes;
}

// `pick(sync)`: the kernel for PersistGrid or PersistCluster.
template <typename Pick>
PersistShape persist_choose(Pick&& pick, int64_t n, int vectors, int gathered, size_t real, int warp_stage,
                            int64_t cluster_rows)
{
   PersistShape sh;
   if (n > cluster_rows || !persist_shape(pick(PersistCluster(PersistSync{})), true, n, vectors, gathered, real, 0, sh))
      persist_shape(pick(PersistGrid(PersistSync{})), false, n, vectors, gathered, real, warp_stage, sh);
   return sh;
}

#define TNLB_PERSIST_PICK(NAME, Real, Sync, Kind, longest)                                                     \
   ((longest) <= 5 ? (const void*)NAME<Real, Kind, 5, Sync>                                                    \
                   : (longest) <= 8 ? (const void*)NAME<Real, Kind, 8, Sync> : (const void*)NAME<Real, Kind, 16, Sync>)
#define TNLB_PERSIST_FORMAT(NAME, Real, Sync, seg)                                                             \
   ((seg)->format == TNLB_CSR       ? TNLB_PERSIST_PICK(NAME, Real, Sync, kPersistCsr, (seg)->max_row)         \
    : (seg)->format == TNLB_ELLPACK ? TNLB_PERSIST_PICK(NAME, Real, Sync, kPersistEll, (seg)->segment_size)    \
                                    : TNLB_PERSIST_PICK(NAME, Real, Sync, kPersistSell, (seg)->max_size))

template <typename Real>
int persist_stage(const tnlb_segments* seg)
{
   if (seg->format != TNLB_CSR || seg->max_row <= 5) return 0;
   return seg->max_row <= 8 ? kPersistStage<Real, 8> : kPersistStage<Real, 16>;
}

template <typename Real>
int64_t cluster_rows(const tnlb_segments* seg)
{
   return sizeof(Real) == 8 && persist_longest(seg) > 8 ? kClusterWideRows : kClusterRows;
}

}  // namespace

template <typename Real>
PersistShape persist_cg(const tnlb_segments* seg)
{
   if (!persist_pays(seg, sizeof(Real), false, l2_bytes())) return {};
   return persist_choose([&](auto sync) { return TNLB_PERSIST_FORMAT(k_cg_persist, Real, decltype(sync), seg); },
                         seg->n, 4, 1, sizeof(Real), persist_stage<Real>(seg), cluster_rows<Real>(seg));
}

template <typename Real>
PersistShape persist_bicgstab(const tnlb_segments* seg)
{
   if (!persist_pays(seg, sizeof(Real), true, l2_bytes())) return {};
   return persist_choose([&](auto sync) { return TNLB_PERSIST_FORMAT(k_bicg_persist, Real, decltype(sync), seg); },
                         seg->n, 6, 2, sizeof(Real), persist_stage<Real>(seg), cluster_rows<Real>(seg));
}

template <typename Real>
PersistShape persist_mgs(int64_t n)
{
   PersistShape sh = persist_choose([&](auto sync) { return (const void*)k_mgs_persist<Real, decltype(sync)>; }, n, 3,
                                    0, sizeof(Real), 0, kClusterRows);
   if (sh.kept < 3) sh.kernel = nullptr;
   return sh;
}

cudaError_t persist_launch(const PersistShape& sh, void** args, cudaStream_t st)
{
   if (sh.cluster == 0) return cudaLaunchCooperativeKernel(sh.kernel, dim3(sh.blocks), dim3(sh.threads), args, sh.smem, st);
   cudaLaunchConfig_t cfg{};
   cudaLaunchAttribute at{};
   cfg.gridDim = dim3(sh.blocks);
   cfg.blockDim = dim3(sh.threads);
   cfg.dynamicSmemBytes = sh.smem;
   cfg.stream = st;
   at.id = cudaLaunchAttributeClusterDimension;
   at.val.clusterDim.x = (unsigned)sh.cluster;
   at.val.clusterDim.y = at.val.clusterDim.z = 1;
   cfg.attrs = &at;
   cfg.numAttrs = 1;
   return cudaLaunchKernelExC(&cfg, sh.kernel, args);
}

template PersistShape persist_cg<double>(const tnlb_segments*);
template PersistShape persist_cg<float>(const tnlb_segments*);
template PersistShape persist_bicgstab<double>(const tnlb_segments*);
template PersistShape persist_bicgstab<float>(const tnlb_segments*);
template PersistShape persist_mgs<double>(int64_t);
template PersistShape persist_mgs<float>(int64_t);

}  // namespace tnlb
