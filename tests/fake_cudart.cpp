// A CUDA runtime without a device, for tests of the engine's host code on the
// CPU: device memory is host memory, a launch is checked as the runtime checks
// it and written down, and no kernel runs.  Linked with the engine's objects
// in place of the CUDA runtime (test_host_runtime.py).
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace
{
struct Launch
{
  std::string kernel;
  dim3 grid, block;
  size_t smem;
  int device;
};
struct Stream
{
  int device;
  bool capturing = false;
  std::vector<Launch> captured;
};
struct Graph
{
  std::vector<Launch> launches;
};
struct Pool
{
  int device;
  size_t cached = 0; // given back to the pool and not to the device
};
struct Block
{
  size_t bytes;
  int device;
  Pool *pool;
};

int g_device = 0, g_devices = 2;
size_t g_limit = (size_t)1 << 40; // memory of a device
std::map<int, size_t> g_used;     // by device, with what its pools hold
std::map<void *, Block> g_blocks;
std::map<const void *, std::string> g_names;
std::map<std::pair<int, const void *>, int> g_smem; // opted-in dynamic shared memory
std::map<std::pair<int, const void *>, void *> g_symbols;
std::map<const void *, size_t> g_symbolBytes;
std::vector<Launch> g_log;
std::string g_refused; // launches of kernels with this in their name fail
cudaError_t g_last = cudaSuccess;
struct
{
  dim3 grid, block;
  size_t smem;
  cudaStream_t stream;
} g_call;

cudaError_t err(cudaError_t e)
{
  if (e != cudaSuccess)
    g_last = e;
  return e;
}

cudaError_t launch(const void *f, dim3 grid, dim3 block, size_t smem, cudaStream_t stream)
{
  Stream *s = (Stream *)stream;
  if (s && s->device != g_device)
    return err(cudaErrorInvalidResourceHandle);
  if (grid.x == 0 || grid.x > 0x7fffffffu || grid.y - 1u > 65534u || grid.z - 1u > 65534u ||
      block.x * block.y * block.z - 1u > 1023u)
    return err(cudaErrorInvalidConfiguration);
  auto it = g_smem.find({g_device, f});
  if (smem > (size_t)(it == g_smem.end() ? 48 << 10 : it->second))
    return err(cudaErrorInvalidValue);
  const std::string name = g_names.count(f) ? g_names[f] : "?";
  if (!g_refused.empty() && name.find(g_refused) != std::string::npos)
    return err(cudaErrorLaunchOutOfResources);
  const Launch l{name, grid, block, smem, g_device};
  (s && s->capturing ? s->captured : g_log).push_back(l);
  return cudaSuccess;
}

bool take(size_t bytes)
{
  if (g_used[g_device] + bytes > g_limit)
    return false;
  g_used[g_device] += bytes;
  return true;
}
} // namespace

extern "C" {

// ---- for the tests
void fake_reset(int devices, size_t limit)
{
  g_devices = devices;
  g_limit = limit;
  g_device = 0;
  g_log.clear();
  g_refused.clear();
  g_last = cudaSuccess;
}
void fake_set_device(int d) { g_device = d; }
void fake_set_limit(size_t limit) { g_limit = limit; }
size_t fake_used(int d) { return g_used[d]; }
void fake_refuse(const char *kernel) { g_refused = kernel; }
void fake_clear_log(void) { g_log.clear(); }
int fake_launches(void) { return (int)g_log.size(); }
const char *fake_launch(int i, int out[5])
{
  const Launch &l = g_log[i];
  out[0] = (int)l.grid.x;
  out[1] = (int)l.grid.y;
  out[2] = (int)l.block.x;
  out[3] = (int)l.smem;
  out[4] = l.device;
  return l.kernel.c_str();
}

// ---- devices and errors
cudaError_t cudaGetDeviceCount(int *n)
{
  *n = g_devices;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
  *d = g_device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 1;
  return cudaSuccess;
}
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "fake error"; }
cudaError_t cudaGetLastError(void)
{
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}

// ---- memory
static cudaError_t allocate(void **p, size_t bytes, Pool *pool)
{
  *p = nullptr;
  const size_t fromPool = pool ? std::min(bytes, pool->cached) : 0;
  if (!take(bytes - fromPool))
    return err(cudaErrorMemoryAllocation);
  if (pool)
    pool->cached -= fromPool;
  *p = calloc(bytes ? bytes : 1, 1);
  g_blocks[*p] = {bytes, g_device, pool};
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t bytes) { return allocate(p, bytes, nullptr); }
cudaError_t cudaFree(void *p)
{
  auto it = g_blocks.find(p);
  if (it == g_blocks.end())
    return p ? err(cudaErrorInvalidValue) : cudaSuccess;
  if (it->second.pool)
    it->second.pool->cached += it->second.bytes;
  else
    g_used[it->second.device] -= it->second.bytes;
  free(p);
  g_blocks.erase(it);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *pool, const cudaMemPoolProps *props)
{
  *pool = (cudaMemPool_t) new Pool{props->location.id};
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t pool)
{
  delete (Pool *)pool;
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t pool, cudaStream_t)
{
  return allocate(p, bytes, (Pool *)pool);
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t pool, size_t keep)
{
  Pool *q = (Pool *)pool;
  if (q->cached > keep)
  {
    g_used[q->device] -= q->cached - keep;
    q->cached = keep;
  }
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t)
{
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t)
{
  memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol)
{
  void *&a = g_symbols[{g_device, symbol}];
  if (!a)
    a = calloc(g_symbolBytes[symbol], 1);
  *p = a;
  return cudaSuccess;
}

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
  *s = (cudaStream_t) new Stream{g_device};
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
  delete (Stream *)s;
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e)
{
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e)
{
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t)
{
  *ms = 1.0f;
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode)
{
  if (((Stream *)s)->capturing)
    return err(cudaErrorIllegalState);
  ((Stream *)s)->capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g)
{
  Stream *q = (Stream *)s;
  if (!q->capturing)
    return err(cudaErrorIllegalState);
  Graph *o = new Graph{q->captured};
  q->captured.clear();
  q->capturing = false;
  *g = (cudaGraph_t)o;
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long)
{
  *x = (cudaGraphExec_t) new Graph(*(Graph *)g);
  return cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t)
{
  for (const Launch &l : ((Graph *)x)->launches)
    g_log.push_back(l);
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g)
{
  delete (Graph *)g;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x)
{
  delete (Graph *)x;
  return cudaSuccess;
}

// ---- kernels
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v)
{
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize)
    g_smem[{g_device, f}] = v;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int, size_t smem)
{
  auto it = g_smem.find({g_device, f});
  *n = smem > (size_t)(it == g_smem.end() ? 48 << 10 : it->second) ? 0 : 2;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int t, size_t smem, unsigned)
{
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, f, t, smem);
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **, size_t smem, cudaStream_t s)
{
  return launch(f, grid, block, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **)
{
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s)
{
  g_call = {grid, block, smem, s};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *s)
{
  *grid = g_call.grid;
  *block = g_call.block;
  *smem = g_call.smem;
  *(cudaStream_t *)s = g_call.stream;
  return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *)
{
  static void *h = nullptr;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *,
                            int *)
{
  g_names[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t bytes, int, int)
{
  g_symbolBytes[host] = bytes;
}
}
