// ilu_pipe.cuh -- triangular solves of the ILU factors as a pipeline of
// thread blocks (one kernel per triangle).
//
// A triangular solve is bound by its chain of dependency levels: a 2D grid
// in natural order has about 2N of them with at most N rows each, so what
// counts is the time from one level to the next.  One block walking the
// levels with x in global memory took 1.03 us a level, two solves of the
// 1000 x 1024 grid's FP64 factors 4.2 ms; here a level takes 0.21 us and
// they take 0.86 ms.
//  * The rows are cut into P contiguous parts, one block each (all resident:
//    cooperative launch).  A block walks its own rows level by level
//    ("steps" of at most kPipeStepRows rows), one row per thread.
//  * x of the block's last W rows stays in a shared-memory ring; an entry
//    whose column lies there costs one shared-memory read.
//  * Entries from other parts, or older than the ring, are "external": their
//    values are fetched a few steps ahead into the stage of the step that
//    needs them.  Each part publishes how many steps it has finished, and a
//    fetch waits until the part that owns the value has passed its step.  A
//    part thus runs behind the part it depends on by a fixed lag instead of
//    meeting it at a grid-wide barrier every level.
//  * A step's packed factor rows and right-hand side arrive by bulk copies
//    (cp.async.bulk) in one of S stages.  Each stage has its own producer
//    warp, so that S fetches of external values are in flight.  Consumer
//    warps only touch shared memory and wait on nothing but the step's
//    barrier; one warp watches the stages arrive, one releases them and one
//    publishes the progress.  With those duties on the consumer warps a level
//    took 0.47 us: every instruction on the chain costs its latency.
// Row arithmetic and order are those of the level-by-level kernels
// (separately rounded multiply and subtract, ascending columns, IEEE
// division), so results keep their bits.
//
// Every wait is bounded: it runs out when no part has finished a step for
// kPipePatience.  A part may lie behind a chain of others that solve one after
// the other for seconds, so polls counted from the start of a wait say nothing.
// A wait that runs out raises *err, which ends the others, and the host's
// *failed, which the caller reports.  The block then takes no further step,
// runs to its end and sets all its rows to NaN.
#pragma once

#include <algorithm>
#include <cmath>
#include <vector>

#include "band.cuh"
#include "internal.cuh"

namespace tnlb {

// Separately rounded arithmetic: no fused multiply-add, as on the Host.
template <typename Real>
__device__ __forceinline__ Real mul_rn(Real a, Real b);
template <>
__device__ __forceinline__ double mul_rn<double>(double a, double b)
{
   return __dmul_rn(a, b);
}
template <>
__device__ __forceinline__ float mul_rn<float>(float a, float b)
{
   return __fmul_rn(a, b);
}
template <typename Real>
__device__ __forceinline__ Real sub_rn(Real a, Real b);
template <>
__device__ __forceinline__ double sub_rn<double>(double a, double b)
{
   return __dsub_rn(a, b);
}
template <>
__device__ __forceinline__ float sub_rn<float>(float a, float b)
{
   return __fsub_rn(a, b);
}
template <typename Real>
__device__ __forceinline__ Real div_rn(Real a, Real b);
template <>
__device__ __forceinline__ double div_rn<double>(double a, double b)
{
   return __ddiv_rn(a, b);
}
template <>
__device__ __forceinline__ float div_rn<float>(float a, float b)
{
   return __fdiv_rn(a, b);
}

constexpr int32_t kPipeStepRows = 256;  // rows of a step = consumer threads, at most
constexpr int kPipeMaxStages = 12;
constexpr int kPipeMaxParts = 127;
constexpr int32_t kPipeWindow = 4096;   // ring entries; > (stages + 1) * step rows
constexpr uint32_t kPipeSmem = 200 * 1024;
constexpr int32_t kPipeMaxNeed = (1 << 24) - 1;
static_assert((kPipeMaxStages + 1) * kPipeStepRows < kPipeWindow, "an evicted ring entry must be finished");

// A part's step: packed positions [t0, t0 + rows), external entries
// [ext0, ext1).
struct PipeStep {
   int32_t t0, rows, ext0, ext1;
};
// External entry: index into the vector it is read from, and the part that
// owns it (top 8 bits) with the steps that part must have finished (0: the
// block's own, long finished).
struct PipeExt {
   int32_t idx;
   uint32_t need;
};

// Host plan of one triangle: the steps of the parts, in order, and the
// packed position of every row (each step starts at a multiple of 4).
struct PipePlan {
   int32_t parts = 1, chunk = 0, max_rows = 0, max_steps = 0;
   int64_t npad = 0;
   std::vector<PipeStep> steps;
   std::vector<int32_t> part_step;  // [parts + 1]
   std::vector<int32_t> rows_at;    // [npad], -1 in the padding
   std::vector<int32_t> pos, step;  // [n]: packed position, step (index into steps)
};

// Parts for n rows: a block's share costs time, and so does its lag behind
// its neighbour (2.2 us measured), which makes the best P grow like sqrt(n).
// FP64, us an application: 100 x 100 (n = 10^4) P = 1 104, 4 116, 8 138;
// 1000 x 1024 P = 1 2375, 4 1076, 8 939, 14 967, 20 997, 64 1275; 95 x 96 x
// 97 P = 4 1062, 8 707, 14 557, 20 514, 32 590; 192^3 P = 14 3379, 32 2176,
// 64 1946.  (By waits counted from their start; the parts taken here now take
// 105, 858 and 571.)
inline int32_t pipe_parts(int64_t n, int32_t sms)
{
   int32_t p = (int32_t)std::lround(std::sqrt((double)n / 5000.0));
   return std::max(1, std::min({p, sms, (int32_t)kPipeMaxParts}));
}

inline PipePlan pipe_plan(const std::vector<int32_t>& lev, int32_t max_level, int32_t parts)
{
   PipePlan P;
   const int32_t n = (int32_t)lev.size();
   P.parts = parts;
   P.chunk = (n + parts - 1) / parts;
   P.pos.resize(n);
   P.step.resize(n);
   P.part_step.push_back(0);
   std::vector<int32_t> cnt((size_t)max_level + 1), at((size_t)max_level + 1);
   int64_t t = 0;
   for (int32_t p = 0; p < parts; p++) {
      const int32_t r0 = (int32_t)std::min<int64_t>(n, (int64_t)p * P.chunk);
      const int32_t r1 = (int32_t)std::min<int64_t>(n, (int64_t)(p + 1) * P.chunk);
      int32_t lo = max_level + 1, hi = -1;
      for (int32_t i = r0; i < r1; i++) {
         lo = std::min(lo, lev[i]);
         hi = std::max(hi, lev[i]);
      }
      for (int32_t l = lo; l <= hi; l++) cnt[l] = 0;
      for (int32_t i = r0; i < r1; i++) cnt[lev[i]]++;
      // a level's rows in steps of kPipeStepRows; at[l] = its first step
      for (int32_t l = lo; l <= hi; l++) {
         at[l] = (int32_t)P.steps.size();
         for (int32_t c = cnt[l]; c > 0; c -= kPipeStepRows) {
            const int32_t rows = std::min(c, kPipeStepRows);
            P.steps.push_back({(int32_t)t, rows, 0, 0});
            P.max_rows = std::max(P.max_rows, rows);
            t += (rows + 3) / 4 * 4;
         }
         cnt[l] = 0;
      }
      for (int32_t i = r0; i < r1; i++) {
         const int32_t k = cnt[lev[i]]++;
         const int32_t s = at[lev[i]] + k / kPipeStepRows;
         P.step[i] = s;
         P.pos[i] = P.steps[s].t0 + k % kPipeStepRows;
      }
      P.part_step.push_back((int32_t)P.steps.size());
      P.max_steps = std::max(P.max_steps, P.part_step[p + 1] - P.part_step[p]);
   }
   P.npad = t;
   if (t > INT32_MAX) return P;  // positions past the index type: no plan
   P.rows_at.assign((size_t)P.npad, -1);
   for (int32_t i = 0; i < n; i++) P.rows_at[P.pos[i]] = i;
   return P;
}

// What a step takes at least, what each of its rows adds, and how long after a
// step another part's step that needs it can start (ns, measured).
constexpr double kPipeStepNs = 230.0, kPipeRowNs = 0.5, kPipeLagNs = 2200.0;

// Length of the plan's schedule: a step follows the one before it in its part
// and, by the lag, the steps of other parts that hold x of its entries
// [beg[i] + skip, end[i]).  Parts that depend on one another's last rows
// follow one another here as they do on the device.
inline double pipe_schedule_ns(const PipePlan& P, const std::vector<int32_t>& beg, const std::vector<int32_t>& end,
                               int32_t skip, const std::vector<int32_t>& cols, bool upper)
{
   const int64_t n = (int64_t)P.pos.size();
   std::vector<double> done(P.steps.size(), 0.0);  // first the earliest start, then the end
   double longest = 0.0;
   for (int32_t q = 0; q < P.parts; q++) {
      const int32_t p = upper ? P.parts - 1 - q : q;
      const int32_t r0 = (int32_t)std::min<int64_t>(n, (int64_t)p * P.chunk);
      const int32_t r1 = (int32_t)std::min<int64_t>(n, (int64_t)(p + 1) * P.chunk);
      for (int32_t i = r0; i < r1; i++)
         for (int32_t k = beg[i] + skip; k < end[i]; k++)
            if (cols[k] < r0 || cols[k] >= r1)
               done[P.step[i]] = std::max(done[P.step[i]], done[P.step[cols[k]]] + kPipeLagNs);
      double t = 0.0;
      for (int32_t s = P.part_step[p]; s < P.part_step[p + 1]; s++) {
         t = std::max(t, done[s]) + kPipeStepNs + kPipeRowNs * P.steps[s].rows;
         done[s] = t;
      }
      longest = std::max(longest, t);
   }
   return longest;
}

// The triangle's plan of `parts` parts and its length, or of one part where that
// takes no longer: where the parts have to follow one another.  level: row counts'
// prefix sums by level.
inline PipePlan pipe_choose(const std::vector<int32_t>& lev, const std::vector<int32_t>& level, int32_t parts,
                            const std::vector<int32_t>& beg, const std::vector<int32_t>& end, int32_t skip,
                            const std::vector<int32_t>& cols, bool upper, double* ns)
{
   double one = 0.0;
   for (size_t l = 0; l + 1 < level.size(); l++) {
      const int32_t rows = level[l + 1] - level[l];
      one += kPipeStepNs * ((rows + kPipeStepRows - 1) / kPipeStepRows) + kPipeRowNs * rows;
   }
   const int32_t max_level = (int32_t)level.size() - 2;
   if (parts > 1) {
      PipePlan P = pipe_plan(lev, max_level, parts);
      *ns = pipe_schedule_ns(P, beg, end, skip, cols, upper);
      if (*ns < one) return P;
   }
   *ns = one;
   return pipe_plan(lev, max_level, 1);
}

// A packed row: K values, the pivot (upper), K codes, where the result goes
// and its ring slot.  A code is the byte offset, in the block's shared
// memory, of the entry's x (in the ring or among the step's external
// values); -1 pads a row.  Rows are whole 16-byte words, read as such; 64
// and 128 bytes would put every second word of a warp's rows in the same
// banks.
template <typename Real, int K, bool Upper>
struct PipeRow {
   static constexpr int kValues = K + (Upper ? 1 : 0);
   static constexpr int kUsed = kValues * (int)sizeof(Real) + (K + 2) * 4;
   static constexpr int kWords = (kUsed + 15) / 16 + ((kUsed + 15) / 16 % 4 == 0 ? 1 : 0);
   static constexpr int kBytes = 16 * kWords;
   int4 w[kWords];
   __host__ __device__ int32_t word(int i) const
   {
      const int4 q = w[i / 4];
      return i % 4 == 0 ? q.x : i % 4 == 1 ? q.y : i % 4 == 2 ? q.z : q.w;
   }
   __device__ Real value(int k) const
   {
      if constexpr (sizeof(Real) == 8)
         return __hiloint2double(word(2 * k + 1), word(2 * k));
      else
         return __int_as_float(word(k));
   }
   static constexpr int kInts = kValues * (int)sizeof(Real) / 4;  // word of code 0
   __device__ int32_t code(int k) const { return word(kInts + k); }
   __device__ int32_t dst() const { return word(kInts + K); }
   __device__ int32_t slot() const { return word(kInts + K + 1); }  // byte offset in shared memory
};

// Shared memory: the ring, then the stages; a stage holds the step's row
// count, its packed rows, its right-hand side and its external values.
struct PipeLayout {
   int32_t stages, stage_bytes, in_off, ext_off;  // offsets within a stage
};
constexpr int32_t kPipeRows0 = 16;  // the packed rows' offset within a stage
// Row count of every stage once the block takes no further step.
constexpr int32_t kPipeNoRows = -1;

template <typename Real>
struct PipeArgs {
   const PipeStep* steps;
   const int32_t* part_step;
   const unsigned char* packed;  // position t's step at t0 * PipeRow::kBytes
   const Real* in;               // by packed position
   const PipeExt* ext;
   const Real* ext_src;  // what ext indexes
   Real* out;
   int32_t* progress;  // [parts * 32]: steps finished, one per 128 bytes
   int32_t* err;
   int32_t* failed;  // host memory
   PipeLayout lay;
   int32_t consumers;  // warps
};

__device__ __forceinline__ int32_t pipe_ld_acquire(const int32_t* p)
{
   int32_t v;
   asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
   return v;
}
__device__ __forceinline__ void pipe_st_release(int32_t* p, int32_t v)
{
   asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ double pipe_ld_relaxed(const double* p)
{
   double v;
   asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
   return v;
}
__device__ __forceinline__ float pipe_ld_relaxed(const float* p)
{
   float v;
   asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
   return v;
}

constexpr unsigned long long kPipePatience = 4000000000ull;  // ns
constexpr int kPipeLook = 1024;                              // polls between two looks around

// What a wait looks at while it lasts.
struct PipePatience {
   const int32_t* progress;
   int32_t *err, *failed;
   volatile int32_t* s_done;    // this block's steps finished
   volatile int32_t* s_failed;  // this block has given up
   uint32_t polls = 0, seen = 0;
   unsigned long long since = 0;

   // After a poll that found nothing: whether to go on.
   __device__ __forceinline__ bool more()
   {
      if ((++polls & 63) != 0) return true;
      return (polls & (kPipeLook - 1)) != 0 ? !*s_failed : look();
   }
   __device__ __forceinline__ bool look()
   {
      uint32_t now = (uint32_t)*s_done;
#pragma unroll 1
      for (int p = 0; p < (int)gridDim.x; p++) now += (uint32_t)pipe_ld_acquire(progress + p * 32);
      unsigned long long t;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
      if (polls == kPipeLook || now != seen) {
         seen = now;
         since = t;
      }
      if (!*s_failed && !pipe_ld_acquire(err) && t - since < kPipePatience) return true;
      *s_failed = 1;
      atomicExch(err, 1);
      asm volatile("st.relaxed.sys.global.s32 [%0], 1;" ::"l"(failed) : "memory");
      return false;
   }
};

// Waits until *flag >= need and returns *flag; -1 when the wait ran out here
// or elsewhere.
__device__ __forceinline__ int32_t pipe_wait(const int32_t* flag, int32_t need, PipePatience w)
{
   while (true) {
      const int32_t f = pipe_ld_acquire(flag);
      if (f >= need) return f;
      if (!w.more()) return -1;
   }
}

// Waits for the mbarrier's phase `parity`.
__device__ __forceinline__ bool pipe_bar_wait(uint64_t* bar, uint32_t parity, PipePatience w)
{
   while (!band_try(bar, parity))
      if (!w.more()) return false;
   return true;
}

template <typename Real, int K, bool Upper>
__global__ void __launch_bounds__((kPipeMaxStages + 3) * 32 + kPipeStepRows, 1) k_ilu_pipe(const PipeArgs<Real> a)
{
   using Row = PipeRow<Real, K, Upper>;
   constexpr int32_t kB = (int32_t)sizeof(Real);
   extern __shared__ __align__(128) unsigned char smem[];
   __shared__ __align__(8) uint64_t s_full[kPipeMaxStages], s_empty[kPipeMaxStages];
   __shared__ int32_t s_done;     // steps finished by the consumers
   __shared__ int32_t s_failed;   // a wait of this block ran out
   const int S = a.lay.stages, NC = a.consumers;
   const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
   const int part = blockIdx.x;
   const int32_t first = a.part_step[part], count = a.part_step[part + 1] - first;
   if (threadIdx.x == 0) {
      s_done = 0;
      s_failed = 0;
      for (int s = 0; s < S; s++) {
         *reinterpret_cast<int32_t*>(smem + (size_t)kPipeWindow * kB + (size_t)s * a.lay.stage_bytes) = 0;
         asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(band_smem(&s_full[s])) : "memory");
         asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(band_smem(&s_empty[s])) : "memory");
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   __syncthreads();
   if (count == 0) return;
   const PipePatience patience{a.progress, a.err, a.failed, &s_done, &s_failed};
   auto rows_of = [&](int s) {
      return reinterpret_cast<int32_t*>(smem + (size_t)kPipeWindow * kB + (size_t)s * a.lay.stage_bytes);
   };
   // the step barrier: consumers, the watcher and the keeper
   auto step_barrier = [&]() { asm volatile("bar.sync 1, %0;" ::"r"((NC + 2) * 32) : "memory"); };

   if (warp < NC) {
      // Consumers: thread c solves row c of every step.  The chain from one
      // step to the next is the gather from shared memory, the row's
      // arithmetic, the store to the ring and the barrier, and nothing
      // else: the next step's row is read while this one computes (the
      // watcher saw it arrive before the last barrier), and all waiting and
      // releasing of stages is done by other warps.
      const int32_t c = threadIdx.x;
      const unsigned char* const stages = smem + kPipeWindow * kB;
      const unsigned char* st = stages;  // of the step to load
      int32_t left = S;                  // stages before the first again
      struct Regs {
         Row row;
         Real x;
         bool active;
      } r0, r1;
      auto load = [&](Regs& r) {
         r.active = c < *reinterpret_cast<const int32_t*>(st);
         const int4* p = reinterpret_cast<const int4*>(st + kPipeRows0) + c * Row::kWords;
#pragma unroll
         for (int q = 0; q < Row::kWords; q++) r.row.w[q] = p[q];
         r.x = reinterpret_cast<const Real*>(st + a.lay.in_off)[c];
         st += a.lay.stage_bytes;
         if (--left == 0) {
            left = S;
            st = stages;
         }
      };
      auto step = [&](const Regs& cur, Regs& next, bool more) {
         Real xk[K];
         if (cur.active) {
#pragma unroll
            for (int k = 0; k < K; k++)
               xk[k] = cur.row.code(k) >= 0 ? *reinterpret_cast<const Real*>(smem + cur.row.code(k)) : Real(0);
         }
         if (more) load(next);
         if (cur.active) {
            Real xi = cur.x;
#pragma unroll
            for (int k = 0; k < K; k++)
               if (cur.row.code(k) >= 0) xi = sub_rn(xi, mul_rn(cur.row.value(k), xk[k]));
            if (Upper) xi = div_rn(xi, cur.row.value(K));
            *reinterpret_cast<Real*>(smem + cur.row.slot()) = xi;
            a.out[cur.row.dst()] = xi;
         }
         step_barrier();
      };
      step_barrier();
      load(r0);
      for (int32_t j = 0; j < count; j += 2) {
         step(r0, r1, j + 1 < count);
         if (j + 1 < count) step(r1, r0, j + 2 < count);
      }
   }
   else if (warp == NC) {
      // watcher: before step j starts, step j + 1 is there, or no stage has rows any more
      int s = 0;
      uint32_t parity = 0;
      bool ok = true;
      auto arrived = [&]() {
         if (ok && !pipe_bar_wait(&s_full[s], parity, patience)) {
            ok = false;
            for (int q = 0; q < S; q++) atomicExch(rows_of(q), kPipeNoRows);
         }
         if (++s == S) {
            s = 0;
            parity ^= 1u;
         }
         __syncwarp();
      };
      arrived();
      if (count > 1) arrived();
      step_barrier();
      for (int32_t j = 0; j < count; j++) {
         if (j + 2 < count) arrived();
         step_barrier();
      }
   }
   else if (warp == NC + 1) {
      // keeper: releases the stage of a finished step and counts the step
      int s = 0;
      step_barrier();
      for (int32_t j = 0; j < count; j++) {
         step_barrier();
         if (lane == 0) {
            band_arrive(&s_empty[s]);
            const int32_t d = j + 1;
            asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(band_smem(&s_done)), "r"(d) : "memory");
         }
         if (++s == S) s = 0;
         __syncwarp();
      }
   }
   else if (warp == NC + 2) {
      // publisher: the steps finished, made visible to the other blocks
      if (lane == 0 && gridDim.x > 1) {
         int32_t seen = 0;
         PipePatience w = patience;
         while (seen < count) {
            int32_t d;
            asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(d) : "r"(band_smem(&s_done)) : "memory");
            if (d > seen) {
               if (*const_cast<volatile int32_t*>(&s_failed)) break;  // steps after that hold no values
               pipe_st_release(a.progress + part * 32, d);
               seen = d;
            }
            else if (!w.more())
               break;
         }
      }
   }
   else {
      // Producers: warp NC + 3 + s fills stage s for steps s, s + S, ...
      // No lane spins on a barrier that another lane of its warp has still
      // to arrive on: the warp would starve that lane.
      constexpr int E = 8;  // external entries a lane has in flight
      const int s = warp - NC - 3;
      unsigned char* st = smem + (size_t)kPipeWindow * kB + (size_t)s * a.lay.stage_bytes;
      Real* ext = reinterpret_cast<Real*>(st + a.lay.ext_off);
      int32_t known_part = -1, known = 0;  // progress last read, and whose
      uint32_t parity = 1, filled = 1;
      int32_t rows = 0;  // as the stage's count says
      for (int32_t j = s; j < count; j += S) {
         const PipeStep d = a.steps[first + j];
         PipeExt e[E];
         auto entries = [&](int32_t k0) {
#pragma unroll
            for (int q = 0; q < E; q++) {
               const int32_t k = k0 + 32 * q + lane;
               if (k < d.ext1) e[q] = a.ext[k];
            }
         };
         entries(d.ext0);
         bool more = true;
         if (lane == 0) {
            more = j < S || pipe_bar_wait(&s_empty[s], parity, patience);
            more = more && atomicCAS(rows_of(s), rows, d.rows) == rows;
         }
         if (!__shfl_sync(0xffffffffu, (int)more, 0)) break;
         rows = d.rows;
         if (lane == 0) {
            const int rp = (d.rows + 3) & ~3;
            const uint32_t nb = (uint32_t)(rp * Row::kBytes), ni = (uint32_t)(rp * kB);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            band_expect(&s_full[s], nb + ni);
            band_copy(st + kPipeRows0, a.packed + (size_t)d.t0 * Row::kBytes, nb, &s_full[s]);
            band_copy(st + a.lay.in_off, a.in + d.t0, ni, &s_full[s]);
         }
         parity ^= 1u;
         __syncwarp();
         for (int32_t k0 = d.ext0; k0 < d.ext1; k0 += 32 * E) {
            if (k0 > d.ext0) entries(k0);
            Real v[E];
#pragma unroll
            for (int q = 0; q < E; q++) {
               if (k0 + 32 * q + lane >= d.ext1) continue;
               const int32_t need = (int32_t)(e[q].need & 0xffffffu), owner = (int32_t)(e[q].need >> 24);
               if (need > 0 && !(owner == known_part && known >= need)) {
                  known_part = owner;
                  known = pipe_wait(a.progress + owner * 32, need, patience);
               }
               v[q] = need == 0 || known >= need ? pipe_ld_relaxed(a.ext_src + e[q].idx) : (Real)NAN;
            }
#pragma unroll
            for (int q = 0; q < E; q++) {
               const int32_t k = k0 + 32 * q + lane;
               if (k < d.ext1) ext[k - d.ext0] = v[q];
            }
         }
         __syncwarp();
         if (lane == 0) band_arrive(&s_full[s]);
         __syncwarp();
         filled ^= 1u;
      }
      // the last copies have landed before the block ends, also where nobody waited for
      // them and a failure ends the other waits
      if (lane == 0 && s < count) band_wait(&s_full[s], filled);
   }
   __syncthreads();
   if (*const_cast<volatile int32_t*>(&s_failed))
      for (int32_t j = 0; j < count; j++) {
         const PipeStep d = a.steps[first + j];
         for (int32_t c = threadIdx.x; c < d.rows; c += blockDim.x)
            a.out[reinterpret_cast<const int32_t*>(a.packed + (size_t)(d.t0 + c) * Row::kBytes)[Row::kInts + K]] = (Real)NAN;
      }
}

// ----------------------------------------------------------------- set-up

// Entries of the factor rows as the plan sees them, one thread per packed
// position; column range of row i: [beg[i] + skip, end[i]).
struct PipeBuild {
   const int32_t *rows_at, *pos, *step, *beg, *end, *cols, *part_step;
   const PipeStep* steps;
   int32_t npad, chunk, skip;
};

// Whether an entry is read from the ring by a step that ends at position
// `send`: the owner is this part and its slot is not yet overwritten.
__host__ __device__ __forceinline__ bool pipe_in_ring(const PipeBuild& b, int32_t i, int32_t col, int32_t send)
{
   return col / b.chunk == i / b.chunk && b.pos[col] >= send - kPipeWindow;
}

static __global__ void k_pipe_count(PipeBuild b, int32_t* __restrict__ count)
{
   const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= b.npad) return;
   const int32_t i = b.rows_at[t];
   if (i < 0) return;
   const int32_t s = b.step[i], send = b.steps[s].t0 + b.steps[s].rows;
   int32_t e = 0;
   for (int32_t k = b.beg[i] + b.skip; k < b.end[i]; k++) e += pipe_in_ring(b, i, b.cols[k], send) ? 0 : 1;
   if (e) atomicAdd(count + s, e);
}

// Writes the packed rows and the external entries (`fill` starts at zero).
// dst_of: where a row's result goes (null: its row index), also what the
// external entries index.
template <typename Real, int K, bool Upper>
__global__ void k_pipe_emit(PipeBuild b, PipeLayout lay, const Real* __restrict__ lu,
                            const int32_t* __restrict__ dst_of, int32_t* __restrict__ fill,
                            unsigned char* __restrict__ packed, PipeExt* __restrict__ ext)
{
   using Row = PipeRow<Real, K, Upper>;
   const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= b.npad) return;
   const int32_t i = b.rows_at[t];
   if (i < 0) return;
   constexpr int32_t kB = (int32_t)sizeof(Real);
   const int32_t s = b.step[i], part = i / b.chunk;
   const PipeStep d = b.steps[s];
   const int32_t ext0 = kPipeWindow * kB + (s - b.part_step[part]) % lay.stages * lay.stage_bytes + lay.ext_off;
   Real* v = reinterpret_cast<Real*>(packed + (size_t)t * Row::kBytes);
   int32_t* q = reinterpret_cast<int32_t*>(v) + Row::kInts;
   const int32_t k0 = b.beg[i] + b.skip, k1 = b.end[i];
   for (int k = 0; k < K; k++) {
      int32_t code = -1;
      Real val = Real(0);
      if (k0 + k < k1) {
         const int32_t col = b.cols[k0 + k];
         val = lu[k0 + k];
         if (pipe_in_ring(b, i, col, d.t0 + d.rows))
            code = (b.pos[col] & (kPipeWindow - 1)) * kB;
         else {
            const int32_t slot = atomicAdd(fill + s, 1), owner = col / b.chunk;
            const int32_t need = owner == part ? 0 : b.step[col] - b.part_step[owner] + 1;
            code = ext0 + slot * kB;
            ext[d.ext0 + slot] = {dst_of ? dst_of[col] : col, ((uint32_t)owner << 24) | (uint32_t)need};
         }
      }
      v[k] = val;
      q[k] = code;
   }
   if (Upper) v[K] = b.beg[i] < b.end[i] ? lu[b.beg[i]] : Real(0);  // an empty U row: pivot 0
   q[K] = dst_of ? dst_of[i] : i;
   q[K + 1] = ((int32_t)t & (kPipeWindow - 1)) * kB;
}

// in[t] = b[row of t], and the progress of both triangles back to zero.
template <typename Real>
__global__ void k_pipe_start(const int32_t* __restrict__ rows_at, int32_t npad, const Real* __restrict__ b,
                             Real* __restrict__ in, int32_t* __restrict__ progress, int32_t nprogress)
{
   const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (t < nprogress) progress[t] = 0;
   if (t < npad) {
      const int32_t i = rows_at[t];
      in[t] = i >= 0 ? b[i] : Real(0);
   }
}

}  // namespace tnlb
