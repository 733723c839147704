// pool.cu -- the library's stream-ordered memory pool, one per device.
//
// cudaMallocAsync orders reuse between streams by itself, so that any thread
// may allocate and release on its own stream.  Reuse costs about 2 us a buffer
// where cudaMalloc and cudaFree of the solvers' vectors took 100 to 300 us
// each, mapping and unmapping their pages: 22.6 of the 52 ms of a
// mixed-precision FSAI-PCG solve at 2048 x 2048, 2.9 of the 12.2 ms of 200 CG
// iterations at 1024 x 1024.
#include <mutex>

#include "internal.cuh"

namespace tnlb {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mutex;
cudaMemPool_t g_pool[kMaxDevices] = {};
int64_t g_users = 0;

thread_local bool t_scope = false;
thread_local cudaStream_t t_stream = nullptr;

// A small cudaMalloc that is kept: the 2 MB block that the driver cuts small
// allocations from stays mapped with it.  Where a segments object was the only
// one, each of its index arrays cost 200 us to allocate and 160 us to free.
void* g_keeper[kMaxDevices] = {};

// The current device's pool, created at its first use (g_mutex held).
cudaError_t current_pool(cudaMemPool_t* pool)
{
   int dev = 0;
   cudaError_t e = cudaGetDevice(&dev);
   if (e != cudaSuccess) return e;
   if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
   if (!g_pool[dev]) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      cudaMemPool_t p = nullptr;
      e = cudaMemPoolCreate(&p, &props);
      uint64_t keep = kPoolKeep;
      if (e == cudaSuccess) e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
      if (e != cudaSuccess) return e;
      g_pool[dev] = p;
      if (cudaMalloc(&g_keeper[dev], 256) != cudaSuccess) cudaGetLastError();
   }
   *pool = g_pool[dev];
   return cudaSuccess;
}

}  // namespace

cudaError_t pool_alloc(void** ptr, size_t bytes, cudaStream_t st)
{
   cudaMemPool_t pool = nullptr;
   {
      std::lock_guard<std::mutex> lock(g_mutex);
      const cudaError_t e = current_pool(&pool);
      if (e != cudaSuccess) return e;
   }
   cudaError_t e = cudaMallocFromPoolAsync(ptr, bytes, pool, st);
   if (e == cudaErrorMemoryAllocation) {
      // what the pool keeps in pieces too small may make room for a whole
      cudaGetLastError();
      cudaStreamSynchronize(st);
      cudaMemPoolTrimTo(pool, 0);
      e = cudaMallocFromPoolAsync(ptr, bytes, pool, st);
   }
   return e;
}

PoolUser::PoolUser()
{
   std::lock_guard<std::mutex> lock(g_mutex);
   g_users++;
}

PoolUser::~PoolUser()
{
   std::lock_guard<std::mutex> lock(g_mutex);
   if (--g_users == 0)
      for (cudaMemPool_t p : g_pool)
         if (p) cudaMemPoolTrimTo(p, kPoolKeepIdle);
}

PoolScope::PoolScope(cudaStream_t st) : on(t_scope), before(t_stream)
{
   t_scope = true;
   t_stream = st;
}

PoolScope::~PoolScope()
{
   t_scope = on;
   t_stream = before;
}

bool pool_scope(cudaStream_t* st)
{
   *st = t_stream;
   return t_scope;
}

}  // namespace tnlb
