// Host-only check of which systems take the resident CG and BiCGStab kernels
// (persist_pays, tnl_b200/csrc/persist.cuh): sizes measured on both routes, on
// either side of the line.  Prints "ok" or the first that differs.
#include <cstdio>

#include "persist.cuh"

namespace tnlb {
PoolUser::PoolUser() {}
PoolUser::~PoolUser() {}
bool pool_scope(cudaStream_t*) { return false; }
cudaError_t pool_alloc(void**, size_t, cudaStream_t) { return cudaErrorNotSupported; }
void set_error(const std::string&) {}
}  // namespace tnlb

int main()
{
   const struct {
      int32_t format;
      int64_t n;
      int32_t slots;
      size_t real;
      bool cg, bicgstab;
   } rows[] = {
      {TNLB_CSR, 10000, 5, 8, true, true},           {TNLB_CSR, 1048576, 5, 8, true, true},
      {TNLB_CSR, 1800000, 5, 8, true, true},         {TNLB_CSR, 4194304, 5, 8, false, true},
      {TNLB_CSR, 16777216, 5, 8, false, true},       {TNLB_CSR, 2700000, 5, 4, true, true},
      {TNLB_CSR, 4194304, 5, 4, false, true},        {TNLB_ELLPACK, 1800000, 5, 4, true, true},
      {TNLB_SLICED_ELLPACK, 2300000, 5, 4, false, true}, {TNLB_CSR, 16777216, 5, 4, false, false},
      {TNLB_CSR, 884640, 7, 4, false, true},         {TNLB_CSR, 500000, 7, 4, true, true},
      {TNLB_CSR, 884640, 7, 8, true, true},          {TNLB_CSR, 3000000, 7, 8, false, false},
      {TNLB_CSR, 16777216, 7, 8, false, false},      {TNLB_ELLPACK, 1500000, 7, 4, true, true},
      {TNLB_ELLPACK, 1800000, 7, 4, false, true},    {TNLB_CSR, 3900000, 7, 4, false, false},
      {TNLB_CSR, 500000, 15, 8, true, true},         {TNLB_SLICED_ELLPACK, 1000000, 15, 8, false, true},
      {TNLB_CSR, 1500000, 15, 8, false, false},      {TNLB_SLICED_ELLPACK, 700000, 15, 4, true, true},
      {TNLB_ELLPACK, 1000000, 15, 4, false, true},   {TNLB_CSR, 1800000, 15, 4, false, false},
      {TNLB_CSR, 1000, 17, 8, false, false},         {TNLB_CSR, 1000, 0, 8, false, false},
      {TNLB_ADAPTIVE_CSR, 1000, 5, 8, false, false}, {TNLB_CHUNKED_ELLPACK, 1000, 5, 8, false, false},
   };
   constexpr int64_t kL2 = 132644864;
   for (const auto& r : rows) {
      tnlb_segments seg;
      seg.format = r.format;
      seg.n = (int32_t)r.n;
      seg.storage = r.n * r.slots;
      seg.max_row = seg.segment_size = seg.max_size = r.slots;
      if (tnlb::persist_pays(&seg, r.real, false, kL2) != r.cg || tnlb::persist_pays(&seg, r.real, true, kL2) != r.bicgstab) {
         std::printf("format %d, %lld rows of %d slots, %zu bytes\n", r.format, (long long)r.n, r.slots, r.real);
         return 1;
      }
   }
   std::printf("ok\n");
   return 0;
}
