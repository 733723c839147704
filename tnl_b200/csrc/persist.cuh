// persist.cuh -- CG and BiCGStab iterations and Gram-Schmidt in one resident
// kernel (persist.cu): what the solvers need to launch them.
#pragma once

#include "internal.cuh"
#include "solver_state.cuh"

namespace tnlb {

constexpr int kPersistMaxBlocks = 256;
constexpr int kPersistSums = 2;

// slots[parity][sum][block]: the partial's two halves, each with the number of
// the exchange; a slot is written again two exchanges later, when its value has
// been used.  Behind them a line for each block, which takes the totals.
struct PersistSync {
   ulonglong2* slots;  // zero before the launch
   int32_t* err;
};
constexpr int kPersistLine = 8;  // 128 bytes
constexpr size_t kPersistSlotBytes = sizeof(ulonglong2) * kPersistMaxBlocks * (2 * kPersistSums + kPersistLine);
inline PersistSync persist_sync(const DeviceBuffer& b)  // kPersistSlotBytes and an int32_t
{
   return {b.as<ulonglong2>(), reinterpret_cast<int32_t*>(b.as<unsigned char>() + kPersistSlotBytes)};
}

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

// The owner's vectors, most used first: the first `kept` of them live in shared
// memory while the kernel runs, the others stay where they are.
template <typename Real, int N>
struct PersistVectors {
   Real* v[N];
   int32_t kept;
   int32_t rows;  // per block
};

// k_bicg_persist leaves an iteration with this in DevState::done before the
// update of p, for a restart by the host.
constexpr int32_t kPersistRestart = 2;

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

// Launch shape: `cluster` blocks (0: one block per SM at most) of `rows` rows.
struct PersistShape {
   const void* kernel = nullptr;
   int32_t blocks = 0, threads = 0, rows = 0, kept = 0, cluster = 0;
   size_t smem = 0;
};

// The kernel and its shape for n rows, a null kernel where the matrix has no
// such form or the device cannot hold the grid.
template <typename Real>
PersistShape persist_cg(const tnlb_segments* seg);
template <typename Real>
PersistShape persist_bicgstab(const tnlb_segments* seg);
// Gram-Schmidt: also null where a block's rows of three vectors do not fit its
// shared memory (1.3M rows in FP64).
template <typename Real>
PersistShape persist_mgs(int64_t n);
cudaError_t persist_launch(const PersistShape& sh, void** args, cudaStream_t st);

}  // namespace tnlb
