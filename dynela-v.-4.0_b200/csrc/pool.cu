// pool.cu - the pools of dnl_pool.h.
#include "dnl_pool.h"

#include <mutex>
#include <set>

namespace
{
constexpr int MAX_DEVICES = 128;
std::mutex g_mutex;
cudaMemPool_t g_pool[MAX_DEVICES];
bool g_asked[MAX_DEVICES];
std::set<void *> g_direct; // blocks of cudaMalloc

// The current device's pool, created at the first call; null where the device
// has none (plain cudaMalloc then).
cudaMemPool_t pool_of_device()
{
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES)
  {
    cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_asked[dev])
  {
    g_asked[dev] = true;
    int has = 0;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = DNL_POOL_KEEP;
    cudaMemPool_t p = nullptr;
    if (cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && has &&
        cudaMemPoolCreate(&p, &props) == cudaSuccess)
    {
      if (cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess)
        g_pool[dev] = p;
      else
        cudaMemPoolDestroy(p);
    }
    cudaGetLastError();
  }
  return g_pool[dev];
}
} // namespace

namespace
{
cudaError_t allocate(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t stream)
{
  return pool ? cudaMallocFromPoolAsync(p, bytes, pool, stream) : cudaMalloc(p, bytes);
}
} // namespace

cudaError_t dnl_pool_release(void)
{
  cudaMemPool_t pool = pool_of_device();
  if (!pool)
    return cudaSuccess;
  // (blocks are given back in the order of their streams' work)
  cudaError_t e = cudaDeviceSynchronize();
  return e == cudaSuccess ? cudaMemPoolTrimTo(pool, 0) : e;
}

cudaError_t dnl_pool_alloc(void **p, size_t bytes, cudaStream_t stream)
{
  *p = nullptr;
  if (bytes == 0)
    bytes = 1;
  cudaMemPool_t kept = pool_of_device(), pool = bytes <= DNL_POOL_LARGEST ? kept : nullptr;
  cudaError_t e = allocate(p, bytes, pool, stream);
  if (e == cudaErrorMemoryAllocation && kept)
  {
    // what the pool keeps may be what is missing
    cudaGetLastError();
    cudaStreamSynchronize(stream);
    cudaMemPoolTrimTo(kept, 0);
    e = allocate(p, bytes, pool, stream);
  }
  if (e != cudaSuccess || pool)
    return e;
  try
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    g_direct.insert(*p);
  }
  catch (...)
  {
    cudaFree(*p);
    *p = nullptr;
    return cudaErrorMemoryAllocation;
  }
  return cudaSuccess;
}

void dnl_pool_free(void *p, cudaStream_t stream)
{
  if (!p)
    return;
  bool direct;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    direct = g_direct.erase(p) > 0;
  }
  // (a pool's block is given back by cudaFree where the stream's device is not current)
  if (direct || cudaFreeAsync(p, stream) != cudaSuccess)
  {
    cudaGetLastError();
    cudaFree(p);
  }
}
