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

// Slots of the longest row; 0 for formats without a resident form.
inline int32_t persist_longest(const tnlb_segments* seg)
{
   switch (seg->format) {
      case TNLB_CSR: return seg->max_row;
      case TNLB_ELLPACK: return seg->segment_size;
      case TNLB_SLICED_ELLPACK: return seg->max_size;
      default: return 0;
   }
}

// Whether the resident kernel is the faster one: one thread can take the longest
// row (16 slots), and the matrix and the iteration's vectors are not too many
// bytes for the L2 cache.  Beyond that one block per SM has too few loads in
// flight, and the launches' full occupancy is the better one.  By multiples of
// the 126 MB: us an iteration, launches and resident, on matrices of 5, 7 and 15
// diagonals (FP64 unless stated):
//  * CG, 5 slots: 1.0M rows 37 and 31, 1.8M 0.82 to 0.93 of the launches' time,
//    3.0M 0.97 to 1.0, 4.2M 129 and 175; FP32 CSR 2.7M 0.98, 3.9M 1.11, but
//    Ellpack and SlicedEllpack 1.8M 0.70 to 0.74 and 2.3M 1.1;
//  * CG, 7 slots: 0.5M 21 and 19, 1.0M 0.90 to 1.0, 1.2M 0.84 to 1.20, 3.0M 109
//    and 172, 16.8M 541 and 1020; FP32 1.5M 0.94 to 0.97, 1.8M 1.14 to 1.24, but
//    CSR 0.5M 0.91 and 0.7M to 1.2M 1.02 to 1.10;
//  * CG, 15 slots: 0.5M 41 and 33, 0.7M 1.08 to 1.20, 4.2M 251 and 429; FP32 0.7M
//    0.87 to 0.94, 1.0M 0.97 to 1.36;
//  * BiCGStab, whose launches come with three host reads: 5 slots 4.2M 338 and 301,
//    16.8M 1085 and 972, FP32 6.3M 0.88 to 0.98, 9.1M 0.99 to 1.06; 7 slots 1.8M
//    0.74 to 0.78, 2.7M 0.99 to 1.06, 16.8M 1243 and 1797, FP32 2.3M 0.74 to 0.93,
//    3.3M 1.02 to 1.14; 15 slots 1.2M 0.74 to 1.0, 1.5M 1.0 to 1.16, FP32 1.2M 0.82
//    to 0.91, 1.8M 1.06 to 1.32.
inline bool persist_pays(const tnlb_segments* seg, size_t real, bool bicgstab, int64_t l2)
{
   const int32_t longest = persist_longest(seg);
   if (longest <= 0 || longest > 16) return false;
   const bool f64 = real == 8;
   double limit;
   if (bicgstab) {
      if (longest <= 5 && f64) return true;
      limit = longest <= 5 ? 4.0 : f64 ? 2.4 : 1.6;
   }
   else if (longest <= 5)
      limit = f64 || seg->format == TNLB_CSR ? 1.5 : 1.0;
   else if (longest <= 8)
      limit = f64 || seg->format != TNLB_CSR ? 1.0 : 0.4;
   else
      limit = 0.85;
   const int64_t bytes =
      seg->storage * (int64_t)(real + sizeof(int32_t)) + seg->n * (int64_t)(sizeof(int32_t) + (bicgstab ? 8 : 5) * real);
   return (double)bytes <= limit * (double)l2;
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

// The kernel and its shape for n rows, a null kernel where the launches are the
// faster ones or the device cannot hold the grid.
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
