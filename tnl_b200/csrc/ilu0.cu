// ilu0.cu -- ILU(0) preconditioner on the GPU.
//
// The reference implements ILU(0) on the host only; its CUDA specialisation
// throws NotImplementedError (Solvers/Linear/Preconditioners/ILU0.h:121-143).
// Here the factorisation and both triangular solves run on the GPU,
// scheduled by dependency levels: row i of L depends on the rows j < i it
// references, row i of U on the rows j > i.  Levels are computed once on the
// host (one pass over the pattern in row order), rows of a level run in
// parallel, one kernel launch per level.  The solves of factors with many
// levels run as a pipeline of blocks, one launch per triangle
// (ilu_pipe.cuh); those with few, wide levels as launches per level captured
// once in a CUDA graph, runs of small levels sharing one single-block launch
// (a __syncthreads between levels).
//
// Arithmetic per row follows ILU0.hpp:59-118 (IKJ order, L_ik = A_ik/U_kk,
// then the updates of the rest of L_i and of U_i with U(k, j) looked up in
// row k of U, 0 if absent) and Utils/TriangularSolve.h:20-103 (ascending
// column order, unit-diagonal L), with separately rounded multiply and
// subtract, so the factors and the solves are bit-identical to the Host.
#include <algorithm>
#include <mutex>
#include <vector>

#include "ilu_pipe.cuh"
#include "internal.cuh"
#include "segview.cuh"

namespace tnlb {
namespace {

// One thread per row of the level.  lu holds A's values and is overwritten by
// the factors; lstart/ustart/uend delimit the L and U parts of each row.
template <typename Real>
__global__ void k_factor_level(const int32_t* __restrict__ rows, int32_t count, const int32_t* __restrict__ cols,
                               Real* __restrict__ lu, const int32_t* __restrict__ lstart,
                               const int32_t* __restrict__ ustart, const int32_t* __restrict__ uend)
{
   const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= count) return;
   const int32_t i = rows[t];
   const int32_t l0 = lstart[i], u0 = ustart[i], u1 = uend[i];
   for (int32_t ck = l0; ck < u0; ck++) {
      const int32_t k = cols[ck];
      const int32_t k0 = ustart[k], k1 = uend[k];
      // U(k,k): getElement searches row k of U; 0 if absent
      Real ukk = 0;
      for (int32_t q = k0; q < k1; q++)
         if (cols[q] == k) {
            ukk = lu[q];
            break;
         }
      const Real lik = div_rn(lu[ck], ukk);
      lu[ck] = lik;
      // remaining L entries and the U entries of row i, each minus L_ik*U(k,j)
      int32_t q = k0;
      for (int32_t cj = ck + 1; cj < u1; cj++) {
         const int32_t j = cols[cj];
         while (q < k1 && cols[q] < j) q++;
         const Real ukj = (q < k1 && cols[q] == j) ? lu[q] : Real(0);
         lu[cj] = sub_rn(lu[cj], mul_rn(lik, ukj));
      }
   }
}

// Forward substitution with unit-diagonal L for the rows of one level.
template <typename Real>
__global__ void k_lower_level(const int32_t* __restrict__ rows, int32_t count, const int32_t* __restrict__ cols,
                              const Real* __restrict__ lu, const int32_t* __restrict__ lstart,
                              const int32_t* __restrict__ ustart, const Real* __restrict__ b, Real* __restrict__ x)
{
   const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= count) return;
   const int32_t i = rows[t];
   Real xi = b[i];
   for (int32_t c = lstart[i]; c < ustart[i]; c++) xi = sub_rn(xi, mul_rn(lu[c], x[cols[c]]));
   x[i] = xi;
}

// Back substitution: x_i = (y_i - sum_{j>i} U_ij x_j) / U_ii (diagonal first in U_i).
template <typename Real>
__global__ void k_upper_level(const int32_t* __restrict__ rows, int32_t count, const int32_t* __restrict__ cols,
                              const Real* __restrict__ lu, const int32_t* __restrict__ ustart,
                              const int32_t* __restrict__ uend, Real* __restrict__ x)
{
   const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= count) return;
   const int32_t i = rows[t];
   const int32_t u0 = ustart[i];
   Real xi = x[i];
   for (int32_t c = u0 + 1; c < uend[i]; c++) xi = sub_rn(xi, mul_rn(lu[c], x[cols[c]]));
   x[i] = div_rn(xi, u0 < uend[i] ? lu[u0] : Real(0));  // an empty U row: pivot 0, as a padding slot
}

// Runs of consecutive small levels in ONE block: the block walks the levels
// in order, a __syncthreads between levels making each level's x visible to
// the next (the same block, so no grid-wide wait); the row arithmetic is
// that of k_lower_level / k_upper_level.
constexpr int kIluRunThreads = 1024;
constexpr int32_t kIluSmallLevel = 2048;

template <typename Real>
__global__ void __launch_bounds__(kIluRunThreads)
   k_lower_run(const int32_t* __restrict__ rows, const int32_t* __restrict__ lvl, int32_t l0, int32_t l1,
               const int32_t* __restrict__ cols, const Real* __restrict__ lu, const int32_t* __restrict__ lstart,
               const int32_t* __restrict__ ustart, const Real* __restrict__ b, Real* __restrict__ x)
{
   for (int32_t l = l0; l < l1; l++) {
      const int32_t s0 = lvl[l], s1 = lvl[l + 1];
      for (int32_t t = s0 + threadIdx.x; t < s1; t += blockDim.x) {
         const int32_t i = rows[t];
         Real xi = b[i];
         for (int32_t c = lstart[i]; c < ustart[i]; c++) xi = sub_rn(xi, mul_rn(lu[c], x[cols[c]]));
         x[i] = xi;
      }
      __syncthreads();
   }
}

template <typename Real>
__global__ void __launch_bounds__(kIluRunThreads)
   k_upper_run(const int32_t* __restrict__ rows, const int32_t* __restrict__ lvl, int32_t l0, int32_t l1,
               const int32_t* __restrict__ cols, const Real* __restrict__ lu, const int32_t* __restrict__ ustart,
               const int32_t* __restrict__ uend, Real* __restrict__ x)
{
   for (int32_t l = l0; l < l1; l++) {
      const int32_t s0 = lvl[l], s1 = lvl[l + 1];
      for (int32_t t = s0 + threadIdx.x; t < s1; t += blockDim.x) {
         const int32_t i = rows[t];
         const int32_t u0 = ustart[i];
         Real xi = x[i];
         for (int32_t c = u0 + 1; c < uend[i]; c++) xi = sub_rn(xi, mul_rn(lu[c], x[cols[c]]));
         x[i] = div_rn(xi, u0 < uend[i] ? lu[u0] : Real(0));
      }
      __syncthreads();
   }
}

// Level-ordered packed factors: position t of the level order (row
// rows[t]) holds its K (padded) L entries at pc/pv[t*K ..] (column -1 pads),
// and for U its off-diagonal entries plus the diagonal at dv[t]; the
// solve's input is permuted to the same order first (in[t] = b[rows[t]]).
// A row then needs one load of its own data and the gathers of x.
template <typename Real>
__global__ void k_permute(const int32_t* __restrict__ rows, int32_t n, const Real* __restrict__ src,
                          Real* __restrict__ dst)
{
   const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
   if (t < n) dst[t] = src[rows[t]];
}

template <typename Real>
__global__ void k_pack_vals(const int64_t* __restrict__ src, int64_t count, const Real* __restrict__ lu,
                            Real* __restrict__ dst)
{
   const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
   if (k < count) dst[k] = src[k] >= 0 ? lu[src[k]] : Real(0);
}

// Rows of one (large) level, packed: x_i = in_t - sum_j L_ij x_j.
template <typename Real, int K>
__global__ void k_lower_packed(int32_t t0, int32_t count, const int32_t* __restrict__ rows,
                               const int32_t* __restrict__ pc, const Real* __restrict__ pv,
                               const Real* __restrict__ in, Real* x)
{
   const int32_t t = t0 + blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= t0 + count) return;
   int32_t c[K];
   Real v[K];
#pragma unroll
   for (int j = 0; j < K; j++) {
      c[j] = pc[(int64_t)t * K + j];
      v[j] = pv[(int64_t)t * K + j];
   }
   const int32_t i = rows[t];
   Real xi = in[t];
#pragma unroll
   for (int j = 0; j < K; j++)
      if (c[j] >= 0) xi = sub_rn(xi, mul_rn(v[j], x[c[j]]));
   x[i] = xi;
}

// x_i = (in_t - sum_{j>i} U_ij x_j) / U_ii for the rows of one level, packed.
template <typename Real, int K>
__global__ void k_upper_packed(int32_t t0, int32_t count, const int32_t* __restrict__ rows,
                               const int32_t* __restrict__ pc, const Real* __restrict__ pv,
                               const Real* __restrict__ dv, const Real* __restrict__ in, Real* x)
{
   const int32_t t = t0 + blockIdx.x * blockDim.x + threadIdx.x;
   if (t >= t0 + count) return;
   int32_t c[K];
   Real v[K];
#pragma unroll
   for (int j = 0; j < K; j++) {
      c[j] = pc[(int64_t)t * K + j];
      v[j] = pv[(int64_t)t * K + j];
   }
   const int32_t i = rows[t];
   Real xi = in[t];
#pragma unroll
   for (int j = 0; j < K; j++)
      if (c[j] >= 0) xi = sub_rn(xi, mul_rn(v[j], x[c[j]]));
   x[i] = div_rn(xi, dv[t]);
}

// Runs of levels of at most kIluPipeThreads rows in one block, one row per
// thread per level, software-pipelined: the packed data and input of a
// thread's row in level l+1 (independent of x) are loaded while level l is
// solved, so after each __syncthreads only the gathers of x wait.
constexpr int kIluPipeThreads = 1024;
constexpr int32_t kIluPipeMaxLevels = 4096;

template <typename Real, int K, bool Upper>
__global__ void __launch_bounds__(kIluPipeThreads)
   k_solve_pipe(const int32_t* __restrict__ lvl, int32_t l0, int32_t l1, const int32_t* __restrict__ rows,
                const int32_t* __restrict__ pc, const Real* __restrict__ pv, const Real* __restrict__ dv,
                const Real* __restrict__ in, Real* x)
{
   __shared__ int32_t s_lvl[kIluPipeMaxLevels + 1];
   for (int32_t k = threadIdx.x; k <= l1 - l0; k += blockDim.x) s_lvl[k] = lvl[l0 + k];
   __syncthreads();
   int32_t i_n = -1, c_n[K];
   Real v_n[K], in_n = Real(0), d_n = Real(1);
   auto load = [&](int32_t l) {
      i_n = -1;
      if (l >= l1) return;
      const int32_t t = s_lvl[l - l0] + (int32_t)threadIdx.x;
      if (t >= s_lvl[l - l0 + 1]) return;
      i_n = rows[t];
      in_n = in[t];
      if (Upper) d_n = dv[t];
#pragma unroll
      for (int j = 0; j < K; j++) {
         c_n[j] = pc[(int64_t)t * K + j];
         v_n[j] = pv[(int64_t)t * K + j];
      }
   };
   load(l0);
   for (int32_t l = l0; l < l1; l++) {
      const int32_t i = i_n;
      int32_t c[K];
      Real v[K];
#pragma unroll
      for (int j = 0; j < K; j++) {
         c[j] = c_n[j];
         v[j] = v_n[j];
      }
      Real xi = in_n;
      const Real di = d_n;
      load(l + 1);
      if (i >= 0) {
#pragma unroll
         for (int j = 0; j < K; j++)
            if (c[j] >= 0) xi = sub_rn(xi, mul_rn(v[j], x[c[j]]));
         x[i] = Upper ? div_rn(xi, di) : xi;
      }
      __syncthreads();
   }
}

// One triangle's packed steps on the device.
template <typename Real>
struct PipeTri {
   int32_t K = 0, npad = 0, parts = 0, consumers = 0;
   PipeLayout lay{};
   DeviceBuffer steps, part_step, rows_at, packed, ext;

   template <bool Upper>
   static const void* kernel(int k)
   {
      switch (k) {
         case 1: return (const void*)k_ilu_pipe<Real, 1, Upper>;
         case 2: return (const void*)k_ilu_pipe<Real, 2, Upper>;
         case 3: return (const void*)k_ilu_pipe<Real, 3, Upper>;
         case 4: return (const void*)k_ilu_pipe<Real, 4, Upper>;
         default: return (const void*)k_ilu_pipe<Real, 8, Upper>;
      }
   }
   template <bool Upper>
   static int32_t row_size(int k)
   {
      switch (k) {
         case 1: return PipeRow<Real, 1, Upper>::kBytes;
         case 2: return PipeRow<Real, 2, Upper>::kBytes;
         case 3: return PipeRow<Real, 3, Upper>::kBytes;
         case 4: return PipeRow<Real, 4, Upper>::kBytes;
         default: return PipeRow<Real, 8, Upper>::kBytes;
      }
   }
   size_t smem() const { return (size_t)kPipeWindow * sizeof(Real) + (size_t)lay.stages * lay.stage_bytes; }

   // progress[parts * 32] is followed, at the same place for both
   // triangles, by the error word of the last (unused) part's slot.
   template <bool Upper>
   tnlb_status launch(const Real* in, Real* out, const Real* ext_src, int32_t* pr, int32_t* failed,
                      cudaStream_t st) const
   {
      PipeArgs<Real> a{steps.as<PipeStep>(), part_step.as<int32_t>(), packed.as<unsigned char>(), in,
                       ext.as<PipeExt>(), ext_src, out, pr, pr + kPipeMaxParts * 32, failed, lay, consumers};
      void* args[] = {&a};
      TNLB_CUDA_TRY(cudaLaunchCooperativeKernel(kernel<Upper>(K), dim3(parts), dim3(32 * (consumers + 3 + lay.stages)),
                                                args, smem(), st));
      return TNLB_OK;
   }

   // The packed triangle of `plan`, whose schedule takes `own_ns`; beg/end
   // delimit the entries of a row, `skip` of them not taken (U's pivot).  K
   // stays 0 when a step has more external entries than a stage holds, or the
   // plan is not worth it against `other_ns` of the level-by-level solve.
   template <bool Upper>
   tnlb_status build(PipePlan& plan, const PipeBuild& dev, int32_t k, const Real* lu, const int32_t* dst_of,
                     double own_ns, double other_ns, cudaStream_t st)
   {
      const int32_t ns = (int32_t)plan.steps.size();
      DeviceBuffer count;
      TNLB_TRY_STATUS(count.alloc(sizeof(int32_t) * (size_t)ns));
      TNLB_CUDA_TRY(cudaMemsetAsync(count.ptr, 0, sizeof(int32_t) * (size_t)ns, st));
      k_pipe_count<<<grid_for(plan.npad, 256), 256, 0, st>>>(dev, count.as<int32_t>());
      TNLB_CHECK_LAUNCH();
      std::vector<int32_t> ec(ns);
      TNLB_CUDA_TRY(cudaMemcpyAsync(ec.data(), count.ptr, sizeof(int32_t) * (size_t)ns, cudaMemcpyDeviceToHost, st));
      TNLB_CUDA_TRY(cudaStreamSynchronize(st));
      int64_t total = 0;
      int32_t emax = 0;
      for (int32_t s = 0; s < ns; s++) {
         plan.steps[s].ext0 = (int32_t)total;
         total += ec[s];
         plan.steps[s].ext1 = (int32_t)total;
         emax = std::max(emax, ec[s]);
      }
      // an external entry about 3 ns
      if (own_ns + 3.0 * (double)total / plan.parts >= other_ns ||
          (plan.parts > 1 && plan.max_steps >= kPipeMaxNeed))
         return TNLB_OK;
      const int32_t kk = k <= 4 ? std::max(k, 1) : 8;
      const int32_t row_bytes = row_size<Upper>(kk);
      consumers = (plan.max_rows + 31) / 32;
      // every consumer thread reads its row, also beyond a step's last
      lay.in_off = kPipeRows0 + consumers * 32 * row_bytes;
      lay.ext_off = lay.in_off + consumers * 32 * (int32_t)sizeof(Real);
      const int64_t bytes = (lay.ext_off + (int64_t)emax * (int64_t)sizeof(Real) + 127) / 128 * 128;
      const int64_t fit = ((int64_t)kPipeSmem - (int64_t)kPipeWindow * (int64_t)sizeof(Real)) / bytes;
      if (fit < 4) return TNLB_OK;
      lay.stages = (int32_t)std::min<int64_t>(fit, kPipeMaxStages);
      lay.stage_bytes = (int32_t)bytes;
      parts = plan.parts;
      npad = (int32_t)plan.npad;
      TNLB_TRY_STATUS(packed.alloc((size_t)npad * row_bytes));
      TNLB_TRY_STATUS(ext.alloc(sizeof(PipeExt) * (size_t)total));
      TNLB_CUDA_TRY(cudaMemcpyAsync(steps.ptr, plan.steps.data(), sizeof(PipeStep) * (size_t)ns,
                                    cudaMemcpyHostToDevice, st));
      TNLB_CUDA_TRY(cudaMemsetAsync(count.ptr, 0, sizeof(int32_t) * (size_t)ns, st));
      const unsigned g = grid_for(npad, 256);
      auto emit = [&](auto* kern) {
         kern<<<g, 256, 0, st>>>(dev, lay, lu, dst_of, count.as<int32_t>(), packed.as<unsigned char>(), ext.as<PipeExt>());
      };
      if (kk == 1) emit(k_pipe_emit<Real, 1, Upper>);
      else if (kk == 2) emit(k_pipe_emit<Real, 2, Upper>);
      else if (kk == 3) emit(k_pipe_emit<Real, 3, Upper>);
      else if (kk == 4) emit(k_pipe_emit<Real, 4, Upper>);
      else emit(k_pipe_emit<Real, 8, Upper>);
      TNLB_CHECK_LAUNCH();
      TNLB_CUDA_TRY(
         cudaFuncSetAttribute(kernel<Upper>(kk), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPipeSmem));
      TNLB_CUDA_TRY(cudaStreamSynchronize(st));
      K = kk;
      return TNLB_OK;
   }

   // The plan's steps and row order on the device, as k_pipe_count and
   // k_pipe_emit read them.
   tnlb_status upload(const PipePlan& plan, DeviceBuffer& pos, DeviceBuffer& step, cudaStream_t st)
   {
      const size_t n = plan.pos.size();
      auto put = [&](DeviceBuffer& d, const void* h, size_t bytes) -> tnlb_status {
         TNLB_TRY_STATUS(d.alloc(bytes));
         TNLB_CUDA_TRY(cudaMemcpyAsync(d.ptr, h, bytes, cudaMemcpyHostToDevice, st));
         return TNLB_OK;
      };
      TNLB_TRY_STATUS(put(steps, plan.steps.data(), sizeof(PipeStep) * plan.steps.size()));
      TNLB_TRY_STATUS(put(part_step, plan.part_step.data(), sizeof(int32_t) * plan.part_step.size()));
      TNLB_TRY_STATUS(put(rows_at, plan.rows_at.data(), sizeof(int32_t) * plan.rows_at.size()));
      TNLB_TRY_STATUS(put(pos, plan.pos.data(), sizeof(int32_t) * n));
      return put(step, plan.step.data(), sizeof(int32_t) * n);
   }
};

struct Ilu0Base {
   virtual ~Ilu0Base() = default;
   virtual tnlb_status apply(const void* b, void* x, cudaStream_t st) = 0;
   // Whether the applications that have finished on the device did so properly.
   virtual tnlb_status check() = 0;
   virtual void parts(int32_t* of) const = 0;  // of L's and U's pipelines
};

template <typename Real>
struct Ilu0 : Ilu0Base {
   int32_t n = 0;
   DeviceBuffer rp, cols, lu, lstart, ustart, uend, lrows, urows, tmp, dlptr, duptr;
   // packed level-ordered factors (when every row has <= 8 L and <= 8
   // off-diagonal U entries): strides kl / ku
   int kl = 0, ku = 0;
   DeviceBuffer lpc, lpv, upc, upv, udv, perm;
   bool pipe = false;  // whether the solves run as pipelines (ilu_pipe.cuh)
   PipeTri<Real> lpipe, upipe;
   DeviceBuffer lin, uin, progress;
   std::mutex order;
   cudaEvent_t done = nullptr;  // the last application
   int32_t* pipe_failed = nullptr;  // host memory that the pipeline's kernels write when a wait runs out
   std::vector<int32_t> lptr, uptr;  // level boundaries into lrows / urows
   cudaGraphExec_t exec = nullptr;
   const Real* g_b = nullptr;
   Real* g_x = nullptr;
   cudaStream_t cs = nullptr;

   ~Ilu0() override
   {
      if (exec) cudaGraphExecDestroy(exec);
      if (cs) cudaStreamDestroy(cs);
      if (done) cudaEventDestroy(done);
      if (pipe_failed) cudaFreeHost(pipe_failed);
   }

   template <int KL, int KU>
   void enqueue_packed(const Real* b, Real* x, cudaStream_t st)
   {
      Real* in = perm.as<Real>();
      const unsigned g = (unsigned)((n + 255) / 256);
      k_permute<Real><<<g, 256, 0, st>>>(lrows.as<int32_t>(), n, b, in);
      const int32_t nl = (int32_t)lptr.size() - 1;
      for (int32_t l = 0; l < nl;) {
         if (lptr[l + 1] - lptr[l] <= kIluPipeThreads) {
            int32_t e = l;
            while (e < nl && e - l < kIluPipeMaxLevels && lptr[e + 1] - lptr[e] <= kIluPipeThreads) e++;
            k_solve_pipe<Real, KL, false><<<1, kIluPipeThreads, 0, st>>>(
               dlptr.as<int32_t>(), l, e, lrows.as<int32_t>(), lpc.as<int32_t>(), lpv.as<Real>(), nullptr, in, x);
            l = e;
            continue;
         }
         const int32_t cnt = lptr[l + 1] - lptr[l];
         k_lower_packed<Real, KL><<<(cnt + 127) / 128, 128, 0, st>>>(lptr[l], cnt, lrows.as<int32_t>(),
                                                                     lpc.as<int32_t>(), lpv.as<Real>(), in, x);
         l++;
      }
      k_permute<Real><<<g, 256, 0, st>>>(urows.as<int32_t>(), n, x, in);
      const int32_t nu = (int32_t)uptr.size() - 1;
      for (int32_t l = 0; l < nu;) {
         if (uptr[l + 1] - uptr[l] <= kIluPipeThreads) {
            int32_t e = l;
            while (e < nu && e - l < kIluPipeMaxLevels && uptr[e + 1] - uptr[e] <= kIluPipeThreads) e++;
            k_solve_pipe<Real, KU, true><<<1, kIluPipeThreads, 0, st>>>(
               duptr.as<int32_t>(), l, e, urows.as<int32_t>(), upc.as<int32_t>(), upv.as<Real>(), udv.as<Real>(),
               in, x);
            l = e;
            continue;
         }
         const int32_t cnt = uptr[l + 1] - uptr[l];
         k_upper_packed<Real, KU><<<(cnt + 127) / 128, 128, 0, st>>>(uptr[l], cnt, urows.as<int32_t>(),
                                                                     upc.as<int32_t>(), upv.as<Real>(),
                                                                     udv.as<Real>(), in, x);
         l++;
      }
   }

   template <int KL>
   void enqueue_packed_u(const Real* b, Real* x, cudaStream_t st)
   {
      if (ku <= 1) enqueue_packed<KL, 1>(b, x, st);
      else if (ku <= 2) enqueue_packed<KL, 2>(b, x, st);
      else if (ku <= 4) enqueue_packed<KL, 4>(b, x, st);
      else enqueue_packed<KL, 8>(b, x, st);
   }

   // Levels in order.  Packed factors: runs of levels of at most
   // kIluPipeThreads rows go to one pipelined single-block launch, a larger
   // level to its own grid.  Otherwise (a row with more than 8 entries in L
   // or U): runs of levels of at most kIluSmallLevel rows in one
   // single-block launch, larger levels to their own grids.
   void enqueue(const Real* b, Real* x, cudaStream_t st)
   {
      if (kl > 0) {
         if (kl <= 1) enqueue_packed_u<1>(b, x, st);
         else if (kl <= 2) enqueue_packed_u<2>(b, x, st);
         else if (kl <= 4) enqueue_packed_u<4>(b, x, st);
         else enqueue_packed_u<8>(b, x, st);
         return;
      }
      const int32_t nl = (int32_t)lptr.size() - 1;
      for (int32_t l = 0; l < nl;) {
         if (lptr[l + 1] - lptr[l] <= kIluSmallLevel) {
            int32_t e = l;
            while (e < nl && lptr[e + 1] - lptr[e] <= kIluSmallLevel) e++;
            k_lower_run<Real><<<1, kIluRunThreads, 0, st>>>(lrows.as<int32_t>(), dlptr.as<int32_t>(), l, e,
                                                            cols.as<int32_t>(), lu.as<Real>(), lstart.as<int32_t>(),
                                                            ustart.as<int32_t>(), b, x);
            l = e;
            continue;
         }
         const int32_t cnt = lptr[l + 1] - lptr[l];
         k_lower_level<Real><<<(cnt + 127) / 128, 128, 0, st>>>(lrows.as<int32_t>() + lptr[l], cnt, cols.as<int32_t>(),
                                                               lu.as<Real>(), lstart.as<int32_t>(),
                                                               ustart.as<int32_t>(), b, x);
         l++;
      }
      const int32_t nu = (int32_t)uptr.size() - 1;
      for (int32_t l = 0; l < nu;) {
         if (uptr[l + 1] - uptr[l] <= kIluSmallLevel) {
            int32_t e = l;
            while (e < nu && uptr[e + 1] - uptr[e] <= kIluSmallLevel) e++;
            k_upper_run<Real><<<1, kIluRunThreads, 0, st>>>(urows.as<int32_t>(), duptr.as<int32_t>(), l, e,
                                                            cols.as<int32_t>(), lu.as<Real>(), ustart.as<int32_t>(),
                                                            uend.as<int32_t>(), x);
            l = e;
            continue;
         }
         const int32_t cnt = uptr[l + 1] - uptr[l];
         k_upper_level<Real><<<(cnt + 127) / 128, 128, 0, st>>>(urows.as<int32_t>() + uptr[l], cnt, cols.as<int32_t>(),
                                                               lu.as<Real>(), ustart.as<int32_t>(),
                                                               uend.as<int32_t>(), x);
         l++;
      }
   }

   // x = U^-1 L^-1 b: b to L's packed order, L's result straight to U's.
   tnlb_status apply_pipe(const Real* b, Real* x, cudaStream_t st)
   {
      int32_t* pr = progress.as<int32_t>();
      const int32_t flags = (kPipeMaxParts + 1) * 32;
      k_pipe_start<Real><<<grid_for(std::max(lpipe.npad, 2 * flags), 256), 256, 0, st>>>(
         lpipe.rows_at.template as<int32_t>(), lpipe.npad, b, lin.as<Real>(), pr, 2 * flags);
      TNLB_CHECK_LAUNCH();
      TNLB_TRY_STATUS((lpipe.template launch<false>(lin.as<Real>(), uin.as<Real>(), uin.as<Real>(), pr, pipe_failed, st)));
      return upipe.template launch<true>(uin.as<Real>(), x, x, pr + flags, pipe_failed, st);
   }

   void parts(int32_t* of) const override
   {
      of[0] = pipe ? lpipe.parts : 0;
      of[1] = pipe ? upipe.parts : 0;
   }

   tnlb_status check() override
   {
      if (!pipe_failed || !*(volatile int32_t*)pipe_failed) return TNLB_OK;
      *(volatile int32_t*)pipe_failed = 0;
      set_error("ILU solve: a wait between blocks ran out");
      return TNLB_ERR_CUDA;
   }

   // One application after the other, whichever streams and threads they come from:
   // they share the object's buffers, and the pipeline's progress words.
   tnlb_status apply(const void* bv, void* xv, cudaStream_t st) override
   {
      const Real* b = static_cast<const Real*>(bv);
      Real* x = static_cast<Real*>(xv);
      std::lock_guard<std::mutex> lock(order);
      if (done)
         TNLB_CUDA_TRY(cudaStreamWaitEvent(st, done, 0));
      else
         TNLB_CUDA_TRY(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
      TNLB_TRY_STATUS(pipe ? apply_pipe(b, x, st) : apply_levels(b, x, st));
      TNLB_CUDA_TRY(cudaEventRecord(done, st));
      return TNLB_OK;
   }

   tnlb_status apply_levels(const Real* b, Real* x, cudaStream_t st)
   {
      // Solves are replayed from a graph captured for fixed (b, x) buffers:
      // copy in/out of the graph's own buffers when the caller's differ.
      if (!exec) {
         TNLB_TRY_STATUS(tmp.alloc(sizeof(Real) * 2 * (size_t)(n > 0 ? n : 1)));
         g_b = tmp.as<Real>();
         g_x = tmp.as<Real>() + n;
         TNLB_CUDA_TRY(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
         cudaGraph_t graph = nullptr;
         TNLB_CUDA_TRY(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
         enqueue(g_b, g_x, cs);
         TNLB_CUDA_TRY(cudaStreamEndCapture(cs, &graph));
         cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
         cudaGraphDestroy(graph);
         TNLB_CUDA_TRY(e);
      }
      cudaEvent_t ev;
      TNLB_CUDA_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
      TNLB_CUDA_TRY(cudaMemcpyAsync((void*)g_b, b, sizeof(Real) * n, cudaMemcpyDeviceToDevice, st));
      TNLB_CUDA_TRY(cudaEventRecord(ev, st));
      TNLB_CUDA_TRY(cudaStreamWaitEvent(cs, ev, 0));
      TNLB_CUDA_TRY(cudaGraphLaunch(exec, cs));
      TNLB_CUDA_TRY(cudaEventRecord(ev, cs));
      TNLB_CUDA_TRY(cudaStreamWaitEvent(st, ev, 0));
      TNLB_CUDA_TRY(cudaMemcpyAsync(x, g_x, sizeof(Real) * n, cudaMemcpyDeviceToDevice, st));
      cudaEventDestroy(ev);
      return TNLB_OK;
   }
};

template <typename Real>
tnlb_status analyze_t(Ilu0<Real>* P, const std::vector<int32_t>& rp, const std::vector<int32_t>& cols, bool factorize,
                      cudaStream_t st);

template <typename Real>
tnlb_status create_t(const tnlb_segments* seg, const int32_t* cols_in, const Real* vals_in, cudaStream_t st,
                     Ilu0<Real>** out)
{
   const int32_t n = seg->n;
   auto* P = new Ilu0<Real>();
   P->n = n;
   // CSR copy of the matrix (rows in slot order, padding dropped)
   TNLB_TRY_STATUS(gather_csr(view_of(seg), sizeof(Real) == 8 ? TNLB_F64 : TNLB_F32, cols_in, vals_in, P->rp, P->cols,
                              P->lu, st));
   int64_t nnz = 0;
   {
      int32_t t = 0;
      TNLB_CUDA_TRY(cudaMemcpyAsync(&t, P->rp.template as<int32_t>() + n, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
      TNLB_CUDA_TRY(cudaStreamSynchronize(st));
      nnz = t;
   }
   // host analysis: L/U split and dependency levels
   std::vector<int32_t> rp(n + 1), cols(nnz);
   TNLB_CUDA_TRY(cudaMemcpyAsync(rp.data(), P->rp.ptr, sizeof(int32_t) * (n + 1), cudaMemcpyDeviceToHost, st));
   if (nnz) TNLB_CUDA_TRY(cudaMemcpyAsync(cols.data(), P->cols.ptr, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost, st));
   TNLB_CUDA_TRY(cudaStreamSynchronize(st));
   TNLB_TRY_STATUS(analyze_t(P, rp, cols, true, st));
   *out = P;
   return TNLB_OK;
}

// Factors given on the host (ILUT): row i holds its L entries (columns < i)
// then its U entries, the first U entry the pivot; the level analysis,
// packing and solves are those of ILU(0).
template <typename Real>
tnlb_status create_from_factors_t(int32_t n, const std::vector<int32_t>& rp, const std::vector<int32_t>& cols,
                                  const std::vector<Real>& lu, cudaStream_t st, Ilu0<Real>** out)
{
   auto* P = new Ilu0<Real>();
   P->n = n;
   const size_t nnz = (size_t)rp[n];
   TNLB_TRY_STATUS(P->rp.alloc(sizeof(int32_t) * ((size_t)n + 1)));
   TNLB_TRY_STATUS(P->cols.alloc(sizeof(int32_t) * (nnz ? nnz : 1)));
   TNLB_TRY_STATUS(P->lu.alloc(sizeof(Real) * (nnz ? nnz : 1)));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->rp.ptr, rp.data(), sizeof(int32_t) * ((size_t)n + 1), cudaMemcpyHostToDevice, st));
   if (nnz) {
      TNLB_CUDA_TRY(cudaMemcpyAsync(P->cols.ptr, cols.data(), sizeof(int32_t) * nnz, cudaMemcpyHostToDevice, st));
      TNLB_CUDA_TRY(cudaMemcpyAsync(P->lu.ptr, lu.data(), sizeof(Real) * nnz, cudaMemcpyHostToDevice, st));
   }
   TNLB_TRY_STATUS(analyze_t(P, rp, cols, false, st));
   *out = P;
   return TNLB_OK;
}

// The pipelined form of both triangular solves where it is expected to be
// faster than the level-by-level one, by times measured on 5- and 7-point
// grids: a level of at most kIluPipeThreads rows 1.0 us, a larger one 2.3 us
// plus its rows' 60 bytes at 3 TB/s.  Row i's entries: L [ls, us), U [us, ue)
// with the pivot first.
template <typename Real>
tnlb_status build_pipe(Ilu0<Real>* P, const std::vector<int32_t>& llev, const std::vector<int32_t>& ulev,
                       const std::vector<int32_t>& ls, const std::vector<int32_t>& us,
                       const std::vector<int32_t>& ue, const std::vector<int32_t>& hcols, int32_t ml, int32_t mu,
                       cudaStream_t st)
{
   auto level_ns = [](const std::vector<int32_t>& ptr) {
      double t = 0;
      for (size_t l = 0; l + 1 < ptr.size(); l++) {
         const int32_t rows = ptr[l + 1] - ptr[l];
         t += rows <= kIluPipeThreads ? 1000.0 : 2300.0 + 0.02 * rows;
      }
      return t;
   };
   int dev = 0, sms = 0;
   TNLB_CUDA_TRY(cudaGetDevice(&dev));
   TNLB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
   const int32_t parts = pipe_parts(P->n, sms);
   const double least = kPipeLagNs * parts + kPipeRowNs * P->n / parts;  // with no level at all
   if (least >= level_ns(P->lptr) || least >= level_ns(P->uptr)) return TNLB_OK;
   double l_ns = 0, u_ns = 0;
   PipePlan L = pipe_choose(llev, P->lptr, parts, ls, us, 0, hcols, false, &l_ns);
   PipePlan U = pipe_choose(ulev, P->uptr, parts, us, ue, 1, hcols, true, &u_ns);
   if (L.npad > INT32_MAX || U.npad > INT32_MAX) return TNLB_OK;
   DeviceBuffer lpos, lstep, upos, ustep;
   TNLB_TRY_STATUS(P->lpipe.upload(L, lpos, lstep, st));
   TNLB_TRY_STATUS(P->upipe.upload(U, upos, ustep, st));
   const int32_t* cols = P->cols.template as<int32_t>();
   auto i32 = [](const DeviceBuffer& d) { return d.as<int32_t>(); };
   const PipeBuild bl{i32(P->lpipe.rows_at), i32(lpos), i32(lstep), i32(P->lstart), i32(P->ustart), cols,
                      i32(P->lpipe.part_step), P->lpipe.steps.template as<PipeStep>(), (int32_t)L.npad, L.chunk, 0};
   const PipeBuild bu{i32(P->upipe.rows_at), i32(upos), i32(ustep), i32(P->ustart), i32(P->uend), cols,
                      i32(P->upipe.part_step), P->upipe.steps.template as<PipeStep>(), (int32_t)U.npad, U.chunk, 1};
   const Real* lu = P->lu.template as<Real>();
   TNLB_TRY_STATUS(P->upipe.template build<true>(U, bu, mu, lu, nullptr, u_ns, level_ns(P->uptr), st));
   if (P->upipe.K == 0) return TNLB_OK;
   TNLB_TRY_STATUS(P->lpipe.template build<false>(L, bl, ml, lu, i32(upos), l_ns, level_ns(P->lptr), st));
   if (P->lpipe.K == 0) return TNLB_OK;
   TNLB_TRY_STATUS(P->lin.alloc(sizeof(Real) * (size_t)L.npad));
   TNLB_TRY_STATUS(P->uin.alloc(sizeof(Real) * (size_t)U.npad));
   TNLB_TRY_STATUS(P->progress.alloc(sizeof(int32_t) * 2 * (kPipeMaxParts + 1) * 32));
   TNLB_CUDA_TRY(cudaHostAlloc((void**)&P->pipe_failed, sizeof(int32_t), cudaHostAllocMapped | cudaHostAllocPortable));
   *P->pipe_failed = 0;
   TNLB_CUDA_TRY(cudaMemsetAsync(P->uin.ptr, 0, sizeof(Real) * (size_t)U.npad, st));  // the padding is copied, not used
   TNLB_CUDA_TRY(cudaStreamSynchronize(st));
   P->pipe = true;
   return TNLB_OK;
}

// L/U split, dependency levels, level order and packed copies of the factors;
// with `factorize`, the ILU(0) factorisation of P->lu in place first.
template <typename Real>
tnlb_status analyze_t(Ilu0<Real>* P, const std::vector<int32_t>& rp, const std::vector<int32_t>& cols, bool factorize,
                      cudaStream_t st)
{
   const int32_t n = P->n;
   std::vector<int32_t> ls(n), us(n), ue(n), llev(n, 0), ulev(n, 0);
   int32_t lmax = 0, umax = 0;
   bool ordered = true;  // every off-diagonal entry of U lies right of its row
   for (int32_t i = 0; i < n; i++) {
      int32_t c = rp[i];
      // ILU0.hpp:35-55: columns < i -> L, i <= column < N -> U (sorted rows)
      ls[i] = c;
      while (c < rp[i + 1] && cols[c] < i) c++;
      us[i] = c;
      while (c < rp[i + 1] && cols[c] < n) c++;
      ue[i] = c;
      int32_t lv = 0;
      for (int32_t q = ls[i]; q < us[i]; q++) lv = std::max(lv, llev[cols[q]] + 1);
      llev[i] = lv;
      lmax = std::max(lmax, lv);
   }
   for (int32_t i = n - 1; i >= 0; i--) {
      int32_t lv = 0;
      for (int32_t q = us[i] + 1; q < ue[i]; q++) {
         lv = std::max(lv, ulev[cols[q]] + 1);
         ordered = ordered && cols[q] > i;
      }
      ulev[i] = lv;
      umax = std::max(umax, lv);
   }
   auto bucket = [&](const std::vector<int32_t>& lev, int32_t maxl, std::vector<int32_t>& ptr,
                     std::vector<int32_t>& rows) {
      ptr.assign(maxl + 2, 0);
      for (int32_t i = 0; i < n; i++) ptr[lev[i] + 1]++;
      for (int32_t l = 0; l <= maxl; l++) ptr[l + 1] += ptr[l];
      rows.resize(n);
      std::vector<int32_t> pos(ptr.begin(), ptr.end() - 1);
      for (int32_t i = 0; i < n; i++) rows[pos[lev[i]]++] = i;
   };
   std::vector<int32_t> lrows, urows;
   bucket(llev, n > 0 ? lmax : -1, P->lptr, lrows);
   bucket(ulev, n > 0 ? umax : -1, P->uptr, urows);
   TNLB_TRY_STATUS(P->lstart.alloc(sizeof(int32_t) * (n ? n : 1)));
   TNLB_TRY_STATUS(P->ustart.alloc(sizeof(int32_t) * (n ? n : 1)));
   TNLB_TRY_STATUS(P->uend.alloc(sizeof(int32_t) * (n ? n : 1)));
   TNLB_TRY_STATUS(P->lrows.alloc(sizeof(int32_t) * (n ? n : 1)));
   TNLB_TRY_STATUS(P->urows.alloc(sizeof(int32_t) * (n ? n : 1)));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->lstart.ptr, ls.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->ustart.ptr, us.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->uend.ptr, ue.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->lrows.ptr, lrows.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->urows.ptr, urows.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, st));
   TNLB_TRY_STATUS(P->dlptr.alloc(sizeof(int32_t) * P->lptr.size()));
   TNLB_TRY_STATUS(P->duptr.alloc(sizeof(int32_t) * P->uptr.size()));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->dlptr.ptr, P->lptr.data(), sizeof(int32_t) * P->lptr.size(), cudaMemcpyHostToDevice,
                                 st));
   TNLB_CUDA_TRY(cudaMemcpyAsync(P->duptr.ptr, P->uptr.data(), sizeof(int32_t) * P->uptr.size(), cudaMemcpyHostToDevice,
                                 st));
   // factorisation, level by level of L
   for (size_t l = 0; factorize && l + 1 < P->lptr.size(); l++) {
      const int32_t c = P->lptr[l + 1] - P->lptr[l];
      k_factor_level<Real><<<(c + 127) / 128, 128, 0, st>>>(P->lrows.template as<int32_t>() + P->lptr[l], c, P->cols.template as<int32_t>(),
                                                           P->lu.template as<Real>(), P->lstart.template as<int32_t>(),
                                                           P->ustart.template as<int32_t>(), P->uend.template as<int32_t>());
   }
   TNLB_CHECK_LAUNCH();
   // packed level-ordered copies of the factors
   int32_t ml = 0, mu = 0;
   for (int32_t i = 0; i < n; i++) {
      ml = std::max(ml, us[i] - ls[i]);
      mu = std::max(mu, ue[i] - us[i] - 1);
   }
   if (ml <= 8 && mu <= 8 && ordered) {
      const tnlb_status s = build_pipe(P, llev, ulev, ls, us, ue, cols, ml, mu, st);
      // its packed rows take up to four times a chain's: without room for them the levels do
      if (s != TNLB_OK && s != TNLB_ERR_OUT_OF_MEMORY) return s;
      if (s != TNLB_OK) {
         cudaGetLastError();
         clear_error();
      }
   }
   if (P->pipe) {
      for (DeviceBuffer* d : {&P->lrows, &P->urows, &P->dlptr, &P->duptr}) d->release();
      return TNLB_OK;
   }
   for (PipeTri<Real>* t : {&P->lpipe, &P->upipe})
      for (DeviceBuffer* d : {&t->steps, &t->part_step, &t->rows_at, &t->packed, &t->ext}) d->release();
   P->lin.release();
   P->uin.release();
   if (ml <= 8 && mu <= 8) {
      auto stride = [](int32_t m) { return m <= 1 ? 1 : m <= 2 ? 2 : m <= 4 ? 4 : 8; };
      const int kl = stride(ml), ku = stride(mu);
      std::vector<int32_t> lpc((size_t)n * kl, -1), upc((size_t)n * ku, -1);
      std::vector<int64_t> lsrc((size_t)n * kl, -1), usrc((size_t)n * ku, -1), dsrc(n, -1);
      for (int32_t t = 0; t < n; t++) {
         const int32_t i = lrows[t];
         for (int32_t j = 0; j < us[i] - ls[i]; j++) {
            lpc[(size_t)t * kl + j] = cols[ls[i] + j];
            lsrc[(size_t)t * kl + j] = ls[i] + j;
         }
         const int32_t r = urows[t];
         for (int32_t j = 0; j < ue[r] - us[r] - 1; j++) {
            upc[(size_t)t * ku + j] = cols[us[r] + 1 + j];
            usrc[(size_t)t * ku + j] = us[r] + 1 + j;
         }
         dsrc[t] = us[r] < ue[r] ? us[r] : -1;
      }
      DeviceBuffer src;
      TNLB_TRY_STATUS(src.alloc(sizeof(int64_t) * (size_t)n * std::max(kl, ku)));
      TNLB_TRY_STATUS(P->lpc.alloc(sizeof(int32_t) * (size_t)n * kl));
      TNLB_TRY_STATUS(P->upc.alloc(sizeof(int32_t) * (size_t)n * ku));
      TNLB_TRY_STATUS(P->lpv.alloc(sizeof(Real) * (size_t)n * kl));
      TNLB_TRY_STATUS(P->upv.alloc(sizeof(Real) * (size_t)n * ku));
      TNLB_TRY_STATUS(P->udv.alloc(sizeof(Real) * (size_t)n));
      TNLB_TRY_STATUS(P->perm.alloc(sizeof(Real) * (size_t)n));
      TNLB_CUDA_TRY(cudaMemcpyAsync(P->lpc.ptr, lpc.data(), sizeof(int32_t) * lpc.size(), cudaMemcpyHostToDevice, st));
      TNLB_CUDA_TRY(cudaMemcpyAsync(P->upc.ptr, upc.data(), sizeof(int32_t) * upc.size(), cudaMemcpyHostToDevice, st));
      // one staging buffer for the three gathers: synchronise between them
      auto pack = [&](const std::vector<int64_t>& h, DeviceBuffer& dst) -> tnlb_status {
         TNLB_CUDA_TRY(cudaMemcpyAsync(src.ptr, h.data(), sizeof(int64_t) * h.size(), cudaMemcpyHostToDevice, st));
         const int64_t cnt = (int64_t)h.size();
         k_pack_vals<Real><<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(src.as<int64_t>(), cnt,
                                                                          P->lu.template as<Real>(),
                                                                          dst.template as<Real>());
         TNLB_CHECK_LAUNCH();
         TNLB_CUDA_TRY(cudaStreamSynchronize(st));
         return TNLB_OK;
      };
      TNLB_TRY_STATUS(pack(lsrc, P->lpv));
      TNLB_TRY_STATUS(pack(usrc, P->upv));
      TNLB_TRY_STATUS(pack(dsrc, P->udv));
      P->kl = kl;
      P->ku = ku;
   }
   TNLB_CUDA_TRY(cudaStreamSynchronize(st));
   return TNLB_OK;
}

}  // namespace

tnlb_status ilu0_create(const tnlb_segments* seg, tnlb_real real, const int32_t* cols, const void* vals,
                        cudaStream_t st, void** out)
{
   TNLB_REQUIRE(seg->n > 0, TNLB_ERR_INVALID_ARGUMENT, "ILU0::update: the matrix is empty");
   if (real == TNLB_F64) {
      Ilu0<double>* p = nullptr;
      tnlb_status s = create_t<double>(seg, cols, (const double*)vals, st, &p);
      *out = static_cast<Ilu0Base*>(p);
      return s;
   }
   Ilu0<float>* p = nullptr;
   tnlb_status s = create_t<float>(seg, cols, (const float*)vals, st, &p);
   *out = static_cast<Ilu0Base*>(p);
   return s;
}

tnlb_status ilu_from_factors(tnlb_real real, int32_t n, const std::vector<int32_t>& rp,
                             const std::vector<int32_t>& cols, const void* lu, cudaStream_t st, void** out)
{
   if (real == TNLB_F64) {
      Ilu0<double>* p = nullptr;
      const double* v = static_cast<const double*>(lu);
      tnlb_status s = create_from_factors_t<double>(n, rp, cols, std::vector<double>(v, v + rp[n]), st, &p);
      *out = static_cast<Ilu0Base*>(p);
      return s;
   }
   Ilu0<float>* p = nullptr;
   const float* v = static_cast<const float*>(lu);
   tnlb_status s = create_from_factors_t<float>(n, rp, cols, std::vector<float>(v, v + rp[n]), st, &p);
   *out = static_cast<Ilu0Base*>(p);
   return s;
}

tnlb_status ilu0_apply(void* ilu, const void* b, void* x, cudaStream_t st)
{
   return static_cast<Ilu0Base*>(ilu)->apply(b, x, st);
}

tnlb_status ilu0_check(void* ilu) { return static_cast<Ilu0Base*>(ilu)->check(); }

void ilu0_parts(void* ilu, int32_t* parts) { static_cast<Ilu0Base*>(ilu)->parts(parts); }

void ilu0_destroy(void* ilu) { delete static_cast<Ilu0Base*>(ilu); }

// Factors for inspection: CSR pattern (rowptr n+1, cols nnz) and LU values
// (L strictly below the diagonal, U from the diagonal on), copied to the host.
tnlb_status ilu0_read(void* ilu, int32_t* h_rowptr, int32_t* h_cols, void* h_vals, int64_t capacity, int real_bytes)
{
   auto* b = static_cast<Ilu0Base*>(ilu);
   if (real_bytes == 8) {
      auto* p = dynamic_cast<Ilu0<double>*>(b);
      TNLB_REQUIRE(p, TNLB_ERR_INVALID_ARGUMENT, "real type mismatch");
      int32_t nnz = 0;
      TNLB_CUDA_TRY(cudaMemcpy(&nnz, p->rp.as<int32_t>() + p->n, sizeof(int32_t), cudaMemcpyDeviceToHost));
      TNLB_REQUIRE(capacity >= nnz, TNLB_ERR_INVALID_ARGUMENT, "buffer too small");
      TNLB_CUDA_TRY(cudaMemcpy(h_rowptr, p->rp.ptr, sizeof(int32_t) * (p->n + 1), cudaMemcpyDeviceToHost));
      TNLB_CUDA_TRY(cudaMemcpy(h_cols, p->cols.ptr, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost));
      TNLB_CUDA_TRY(cudaMemcpy(h_vals, p->lu.ptr, sizeof(double) * nnz, cudaMemcpyDeviceToHost));
      return TNLB_OK;
   }
   auto* p = dynamic_cast<Ilu0<float>*>(b);
   TNLB_REQUIRE(p, TNLB_ERR_INVALID_ARGUMENT, "real type mismatch");
   int32_t nnz = 0;
   TNLB_CUDA_TRY(cudaMemcpy(&nnz, p->rp.as<int32_t>() + p->n, sizeof(int32_t), cudaMemcpyDeviceToHost));
   TNLB_REQUIRE(capacity >= nnz, TNLB_ERR_INVALID_ARGUMENT, "buffer too small");
   TNLB_CUDA_TRY(cudaMemcpy(h_rowptr, p->rp.ptr, sizeof(int32_t) * (p->n + 1), cudaMemcpyDeviceToHost));
   TNLB_CUDA_TRY(cudaMemcpy(h_cols, p->cols.ptr, sizeof(int32_t) * nnz, cudaMemcpyDeviceToHost));
   TNLB_CUDA_TRY(cudaMemcpy(h_vals, p->lu.ptr, sizeof(float) * nnz, cudaMemcpyDeviceToHost));
   return TNLB_OK;
}

}  // namespace tnlb
