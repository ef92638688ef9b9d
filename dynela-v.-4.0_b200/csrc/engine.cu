// engine.cu - host side of the B200 explicit-dynamics engine: model upload,
// node->slot CSR lists, the increment captured as a CUDA graph, the device-
// resident run loop, state access and the C ABI declared in include/dnlgpu.h.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "dnl_kernels.cuh"
#include "dnl_pool.h"
#include "dnl_steps.cuh"
#include "dnlgpu.h"

using namespace dnl;

namespace
{
char g_create_err[512] = "";

template <typename T> struct DBuf
{
  T *p = nullptr;
  size_t n = 0;
};
} // namespace

struct dnl_engine
{
  int device = 0;
  cudaStream_t stream = nullptr;
  int type = 0, npe = 0, dim = 0, precision = 0;
  int nInst = 0, nN = 0, nE = 0, nIP = 0, nIPpad = 0, nSpeed = 0, nFunc = 0;
  bool hasSpeed = false;
  DevModel M{};
  std::vector<void *> allocs;
  std::vector<int> elemBegin, nodeBegin;
  // the engine's node numbering (DNL_ORDER_*): empty when every instance keeps
  // the caller's; else intOf[caller's node] = engine's node and extOf the inverse
  std::vector<int> intOf, extOf;
  std::vector<int> nodeOrder; // per instance: DNL_ORDER_GIVEN or DNL_ORDER_RCM
  const int *dIntOf = nullptr;
  std::vector<Ctl> ctlInit;
  Ctl *hctl = nullptr; // host mirror of the control blocks
  double *denergy = nullptr, *denergyPart = nullptr; // of one call: [3], partials
  int kinBlocks = 0, pointBlocks = 0;                 // blocks of k_energy_parts for the largest instance
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graphExec = nullptr;
  // graphs of r < graphIncs increments (remExec[r]), for runs of a known
  // number of increments that is not a multiple of graphIncs
  cudaGraphExec_t remExec[64] = {};
  int remLaunches[64] = {};
  bool timing = false;
  double times[4] = {0, 0, 0, 0};
  long long launches = 0;
  int launchesPerStep = 0; // kernels of one graph replay
  int graphIncs = 8;        // increments per graph replay (dnl_engine_set_graph_increments)
  bool oneMat = false;      // one material in the whole engine: the element pass reads it from its parameters
  bool initialized = false;
  int nTiles = 0;
  int variant = 0;          // element-pass kernel variant (see kVariants)
  bool tuned = false;
  bool forced = false;      // a variant asked for by dnl_engine_set_variant and not chosen again by the autotuner
  // the build that runs increments in one cooperative launch (dnl_steps.cuh);
  // no kernel where the model is not run so
  StepsBuild steps;
  unsigned *stepsBar = nullptr;            // grid barrier
  unsigned long long *stepsPhase = nullptr; // [3] phase times (ns)
  double variantMs[DNL_NUM_VARIANTS] = {0};
  std::map<const void *, int> resident; // blocks per SM of the kernels asked so far (resident_blocks)
  int *derr = nullptr;      // bulk-copy wait failure flag
  int numSMs = 0;
  bool powerIteration = false;
  int piGrid = 0;
  int mode = DNL_MODE_PLAIN;          // element-pass mode (DNL_MODE_*)
  void *mlpImage = nullptr;           // learned-guess network image
  unsigned long long *dstats = nullptr; // Newton statistics [4] + harvest count
  // history items (dnl_engine_set_items): list, output offsets, values
  int nItems = 0;
  long long nValues = 0;
  int itemsKinetic = 0; // speed buffers whose kinetic energy an item asks for (bit 0 current, bit 1 previous)
  int4 *ditems = nullptr;
  long long *ditemOff = nullptr;
  double *dvalues = nullptr, *dkin = nullptr;
  void *itemMem = nullptr; // their allocation
  // read-back staging on the device, kept from call to call (grown on demand)
  void *dstage = nullptr;
  size_t stageBytes = 0;
  int *dslotInc = nullptr; // incidence of each force slot (node averages)
  size_t nSlotCap = 0;     // force slots allocated (fixed-stride or CSR layout)
  // history records kept on the device (dnl_engine_set_history)
  bool histOn = false;
  HistRing hist{};
  void *histMem = nullptr;
  std::vector<double> histHost; // records drained from the device, oldest first
  std::string err;
};

// error text of the entry points that have no handle (static_pass.cu)
void dnl_internal_set_error(const char *msg) { snprintf(g_create_err, sizeof(g_create_err), "%s", msg); }

namespace
{
int fail(dnl_engine *h, int code, const char *fmt, ...)
{
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (h)
    h->err = buf;
  else
    snprintf(g_create_err, sizeof(g_create_err), "%s", buf);
  return code;
}

#define CK(call)                                                                                                  \
  do                                                                                                              \
  {                                                                                                               \
    cudaError_t e_ = (call);                                                                                      \
    if (e_ != cudaSuccess)                                                                                        \
      return fail(h, DNL_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__);  \
  } while (0)

template <typename T> int dalloc(dnl_engine *h, T **p, size_t n)
{
  *p = nullptr;
  if (n == 0)
    n = 1;
  cudaError_t e = dnl_pool_alloc((void **)p, n * sizeof(T), h->stream);
  if (e != cudaSuccess)
    return fail(h, DNL_ERR_CUDA, "allocation of %zu bytes failed: %s", n * sizeof(T), cudaGetErrorString(e));
  h->allocs.push_back(*p);
  return DNL_OK;
}

template <typename T> int upload(dnl_engine *h, T **p, const std::vector<T> &v)
{
  int rc = dalloc(h, p, v.size());
  if (rc)
    return rc;
  if (!v.empty())
    CK(cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
  return DNL_OK;
}

int copy(dnl_engine *h, void *dst, const void *src, size_t bytes, cudaMemcpyKind kind)
{
  CK(cudaMemcpyAsync(dst, src, bytes, kind, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return DNL_OK;
}

// Device staging of the read-back entry points: allocated by the first call
// that needs it and kept (grown when a later call needs more), so that a
// read-back costs its kernel and its copy, not an allocation.
int staging(dnl_engine *h, size_t bytes, void **out)
{
  if (bytes > h->stageBytes)
  {
    if (h->dstage)
    {
      dnl_pool_free(h->dstage, h->stream);
      h->dstage = nullptr;
      h->stageBytes = 0;
    }
    CK(dnl_pool_alloc(&h->dstage, bytes, h->stream));
    h->stageBytes = bytes;
  }
  *out = h->dstage;
  return DNL_OK;
}

int npe_of(int type)
{
  return (type == DNL_ELQUA4NAX || type == DNL_ELQUA4N2D) ? 4 : (type == DNL_ELHEX8N3D ? 8 : 0);
}

int check_desc(const dnl_model_desc *d, int idx)
{
  if (!d)
    return fail(nullptr, DNL_ERR_ARG, "model %d: NULL description", idx);
  if (npe_of(d->elem_type) == 0)
    return fail(nullptr, DNL_ERR_ARG, "model %d: unknown element type %d", idx, d->elem_type);
  if (d->n_nodes <= 0 || d->n_elems <= 0 || !d->coords || !d->conn)
    return fail(nullptr, DNL_ERR_ARG, "model %d: empty mesh", idx);
  // before any of the caller's arrays is read: the engine indexes points and
  // node components with 32-bit integers
  if ((long long)d->n_elems * npe_of(d->elem_type) > 0x3fffffffLL || 3LL * d->n_nodes > 0x3fffffffLL)
    return fail(nullptr, DNL_ERR_ARG, "model %d: too large for 32-bit point indices (%d elements, %d nodes)", idx,
                d->n_elems, d->n_nodes);
  if (d->n_materials <= 0 || !d->materials)
    return fail(nullptr, DNL_ERR_ARG, "model %d: no material", idx);
  if (d->ts_method != DNL_TS_COURANT && d->ts_method != DNL_TS_POWER_ITERATION)
    return fail(nullptr, DNL_ERR_UNSUPPORTED, "model %d: unknown time-step method %d", idx, d->ts_method);
  if (d->stress_method != DNL_STRESS_NEWTON && d->stress_method != DNL_STRESS_DIRECT)
    return fail(nullptr, DNL_ERR_UNSUPPORTED, "model %d: unknown stress computation method %d", idx,
                d->stress_method);
  if (d->precision != DNL_PREC_FP64 && d->precision != DNL_PREC_MIXED)
    return fail(nullptr, DNL_ERR_ARG, "model %d: unknown precision %d", idx, d->precision);
  const int npe = npe_of(d->elem_type);
  // the range of the connectivity by a min / max pass (no early exit, so it
  // vectorises); the first entry out of range is looked for only when there is one
  const long nConn = (long)d->n_elems * npe;
  int32_t lo = INT32_MAX, hi = INT32_MIN;
  for (long k = 0; k < nConn; k++)
  {
    lo = std::min(lo, d->conn[k]);
    hi = std::max(hi, d->conn[k]);
  }
  if (lo < 0 || hi >= d->n_nodes)
    for (long k = 0; k < nConn; k++)
      if (d->conn[k] < 0 || d->conn[k] >= d->n_nodes)
        return fail(nullptr, DNL_ERR_ARG, "model %d: connectivity entry %ld = %d out of range", idx, k, d->conn[k]);
  if (d->elem_mat)
    for (int e = 0; e < d->n_elems; e++)
      if (d->elem_mat[e] < 0 || d->elem_mat[e] >= d->n_materials)
        return fail(nullptr, DNL_ERR_ARG, "model %d: material index of element %d out of range", idx, e);
  for (int f = 0; f < d->n_functions; f++)
    if (d->functions[f].n_points < 1 || !d->functions[f].x || !d->functions[f].y)
      return fail(nullptr, DNL_ERR_ARG, "model %d: empty function %d", idx, f);
  if (d->bc_code && d->bc_func)
    for (long k = 0; k < 3L * d->n_nodes; k++)
      if (d->bc_func[k] >= d->n_functions)
        return fail(nullptr, DNL_ERR_ARG, "model %d: function index out of range", idx);
  if (!(d->t_end > d->t_start))
    return fail(nullptr, DNL_ERR_ARG, "model %d: t_end must exceed t_start", idx);
  if (d->node_order != DNL_ORDER_GIVEN && d->node_order != DNL_ORDER_RCM && d->node_order != DNL_ORDER_AUTO)
    return fail(nullptr, DNL_ERR_ARG, "model %d: unknown node order %d", idx, d->node_order);
  return DNL_OK;
}

// The engine's numbering of one model's nodes: order[k] = the caller's node
// numbered k, or empty for the caller's numbering (DNL_ORDER_AUTO keeps it
// unless reverse Cuthill-McKee at least halves the mean element span).
std::vector<int> node_order_of(const dnl_model_desc *d, int npe)
{
  std::vector<int> order;
  if (d->node_order == DNL_ORDER_GIVEN)
    return order;
  order.resize(d->n_nodes);
  if (dnl_mesh_order_rcm(d->n_nodes, d->n_elems, npe, d->conn, order.data()) != DNL_OK)
    return {};
  if (d->node_order == DNL_ORDER_AUTO)
  {
    double given = 0.0, rcm = 0.0;
    if (dnl_mesh_span(d->n_nodes, d->n_elems, npe, d->conn, nullptr, &given) != DNL_OK ||
        dnl_mesh_span(d->n_nodes, d->n_elems, npe, d->conn, order.data(), &rcm) != DNL_OK || 2.0 * rcm > given)
      return {};
  }
  return order;
}


// ----------------------------------------------------------------- launches

// Element-pass variants the autotuner chooses from: plain (state loaded from
// global memory) or persistent with bulk-copy staging of each tile, each with
// its register budget (blocks of TILE threads per SM asked of the compiler).
struct Variant
{
  const char *name;
  int tma;  // 0 plain, 1 bulk-copy state, 2 fully staged, 3 bulk-copy state, a block per tile
  int minb; // blocks per SM of the register budget
  int pts;  // points (threads) per block
};
// each precision: a tile's state by one bulk copy, a block per tile (batches:
// blocks that walk over the tiles); FP32 a plain pass, FP64 the walking kernel
// for single models as well; then persistent staged tiles from the most
// blocks per SM (fewest registers, most spilled) to the fewest (no spills),
// then the fully staged kernel (node gathers one tile ahead as well),
// then plain blocks of half a tile (8 hexahedra) and of two tiles (32) at
// the register budgets of the 128-point ones; in FP32 also the plain passes
// at 48 registers (plain64/20, plain/10: 40 warps per SM, no more spilled
// than at 64 registers)
const Variant kVariantsF32[] = {{"once/6", 3, 6, 128},     {"plain/8", 0, 8, 128},    {"tma/4", 1, 4, 128},
                                {"plain64/20", 0, 20, 64},  {"tma/3", 1, 3, 128},      {"stage/4", 2, 4, 128},
                                {"stage/3", 2, 3, 128},     {"stage/2", 2, 2, 128},    {"plain64/12", 0, 12, 64},
                                {"plain64/16", 0, 16, 64},  {"plain/10", 0, 10, 128},  {"plain256/4", 0, 4, 256}};
const Variant kVariantsF64[] = {{"once/4", 3, 4, 128},     {"walk/4", 3, 4, 128},     {"tma/2", 1, 2, 128},
                                {"tma/3", 1, 3, 128},       {"plain/2", 0, 2, 128},    {"tma/1", 1, 1, 128},
                                {"stage/2", 2, 2, 128},     {"stage/1", 2, 1, 128},    {"plain64/8", 0, 8, 64},
                                {"plain64/6", 0, 6, 64},    {"plain256/2", 0, 2, 256}, {"plain256/1", 0, 1, 256}};
static_assert(sizeof(kVariantsF32) / sizeof(Variant) == DNL_NUM_VARIANTS, "variant list");
static_assert(sizeof(kVariantsF64) / sizeof(Variant) == DNL_NUM_VARIANTS, "variant list");
constexpr int kNumVariants = DNL_NUM_VARIANTS;

const Variant &variant_of(const dnl_engine *h, int v)
{
  return h->precision == DNL_PREC_MIXED ? kVariantsF32[v] : kVariantsF64[v];
}

// A kernel launched on the engine's stream; an error is this launch's own, and
// every caller returns it: a graph captured without one of its kernels would
// go on without it.
template <typename... P, typename... A>
int launch_attr(dnl_engine *h, cudaLaunchAttribute *at, void (*k)(P...), int grid, int block, size_t smem, A... args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = h->stream;
  cfg.attrs = at;
  cfg.numAttrs = at ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, args...);
  if (e == cudaSuccess)
  {
    h->launches++;
    return DNL_OK;
  }
  cudaGetLastError();
  return fail(h, DNL_ERR_CUDA, "kernel launch failed: %s", cudaGetErrorString(e));
}
template <typename... P, typename... A>
int launch(dnl_engine *h, void (*k)(P...), int grid, int block, size_t smem, A... args)
{
  return launch_attr(h, nullptr, k, grid, block, smem, args...);
}
// A kernel of the increment (element, nodal and Courant passes) launched with
// programmatic stream serialization (see pdl_wait); in the captured graph
// this is a programmatic edge.
template <typename... P, typename... A>
int launch_pdl(dnl_engine *h, void (*k)(P...), int grid, int block, size_t smem, A... args)
{
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  return launch_attr(h, &at, k, grid, block, smem, args...);
}

// Blocks per SM of a kernel of `threads` threads and `smem` bytes of dynamic
// shared memory, asked once per engine and kernel: the opt-in to more than
// 48 KB holds on the device where it was made, and the engines of a process
// may be on several.
int resident_blocks(dnl_engine *h, const void *kernel, int threads, size_t smem, int *blocks)
{
  auto it = h->resident.find(kernel);
  if (it == h->resident.end())
  {
    int n = 0;
    if (smem)
      CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, smem));
    it = h->resident.emplace(kernel, std::max(n, 1)).first;
  }
  *blocks = it->second;
  return DNL_OK;
}

template <typename R, int NPE, bool ONE, int MINB, int PTS = TILE> int launch_plain(dnl_engine *h)
{
  // work slots: a batch has up to nInst - 1 more slots than tiles (a tile
  // shared by two running instances is a slot of each); PTS / TILE slots per
  // block, or two blocks per slot
  const int slots = h->nTiles + h->nInst - 1;
  const int grid = PTS >= TILE ? (slots + PTS / TILE - 1) / (PTS / TILE) : 2 * slots;
  return launch_pdl(h, k_element<R, NPE, MINB, PTS, ONE>, grid, PTS, 0, h->M, h->nTiles);
}

template <typename R, int NPE, bool ONE, int MINB> int launch_tma(dnl_engine *h)
{
  const size_t smem = 2 * (DNL_IP_NREAD * TILE * sizeof(R) + TILE * sizeof(int)) + TILE * ElemShape<NPE>::template pass_row<R> * sizeof(R);
  int perSM = 0, rc = resident_blocks(h, (const void *)k_element_tma<R, NPE, MINB, ONE>, TILE, smem, &perSM);
  if (rc)
    return rc;
  const int grid = std::min(h->nTiles, perSM * h->numSMs);
  return launch_pdl(h, k_element_tma<R, NPE, MINB, ONE>, grid, TILE, smem, h->M, h->nTiles, h->derr);
}

template <typename R, int NPE, bool ONE, int MINB> int launch_stage(dnl_engine *h)
{
  const size_t smem = StageLayout<R, NPE>::BYTES;
  int perSM = 0, rc = resident_blocks(h, (const void *)k_element_stage<R, NPE, MINB, ONE>, TILE, smem, &perSM);
  if (rc)
    return rc;
  const int grid = std::min(h->nTiles, perSM * h->numSMs);
  return launch_pdl(h, k_element_stage<R, NPE, MINB, ONE>, grid, TILE, smem, h->M, h->nTiles, h->derr);
}

template <typename R, int NPE, bool ONE, bool LOOP, int MINB> int launch_once_t(dnl_engine *h)
{
  const size_t smem = DNL_IP_NREAD * TILE * sizeof(R) + TILE * ElemShape<NPE>::template pass_row<R> * sizeof(R);
  auto *k = k_element_once<R, NPE, MINB, ONE, LOOP>;
  int perSM = 0, rc = resident_blocks(h, (const void *)k, TILE, smem, &perSM);
  if (rc)
    return rc;
  const int slots = h->nTiles + h->nInst - 1; // see launch_plain
  return launch_pdl(h, k, LOOP ? std::min(slots, ONCE_BLOCKS * perSM * h->numSMs) : slots, TILE, smem, h->M, h->nTiles, h->derr);
}
// (a batch has a material per instance at least)
template <typename R, int NPE, bool ONE, int MINB> int launch_once(dnl_engine *h)
{
  if constexpr (!ONE)
    if (h->nInst > 1)
      return launch_once_t<R, NPE, false, true, MINB>(h);
  return launch_once_t<R, NPE, ONE, false, MINB>(h);
}

template <int NPE, int MODE> int launch_mode(dnl_engine *h)
{
  const size_t smem = MODE == MODE_GUESS ? mlp::SMEM_BYTES : 0;
  int perSM = 0, rc = resident_blocks(h, (const void *)k_element_mode<NPE, MODE>, TILE, smem, &perSM);
  if (rc)
    return rc;
  // the blocks resident on one SM must find their tensor-memory columns free
  if (MODE == MODE_GUESS && perSM * (int)mlp::TMEM_COLS > 512)
    return fail(h, DNL_ERR_CUDA, "guess kernel: %d blocks per SM exceed the tensor memory", perSM);
  const int grid = std::min(h->nTiles, perSM * h->numSMs);
  return launch(h, k_element_mode<NPE, MODE>, grid, TILE, smem, h->M, h->nTiles, h->derr);
}

template <int NPE> int launch_mode_any(dnl_engine *h)
{
  switch (h->mode)
  {
  case DNL_MODE_STATS: return launch_mode<NPE, MODE_STATS>(h);
  case DNL_MODE_HARVEST: return launch_mode<NPE, MODE_HARVEST>(h);
  default: return launch_mode<NPE, MODE_GUESS>(h);
  }
}

template <typename R, int NPE, bool ONE> int launch_variant(dnl_engine *h, int v)
{
  if constexpr (sizeof(R) == 4)
  {
    switch (v)
    {
    case 0: return launch_once<R, NPE, ONE, 6>(h);
    case 1: return launch_plain<R, NPE, ONE, 8>(h);
    case 2: return launch_tma<R, NPE, ONE, 4>(h);
    case 3: return launch_plain<R, NPE, ONE, 20, TILE / 2>(h);
    case 4: return launch_tma<R, NPE, ONE, 3>(h);
    case 5: return launch_stage<R, NPE, ONE, 4>(h);
    case 6: return launch_stage<R, NPE, ONE, 3>(h);
    case 7: return launch_stage<R, NPE, ONE, 2>(h);
    case 8: return launch_plain<R, NPE, ONE, 12, TILE / 2>(h);
    case 9: return launch_plain<R, NPE, ONE, 16, TILE / 2>(h);
    case 10: return launch_plain<R, NPE, ONE, 10>(h);
    default: return launch_plain<R, NPE, ONE, 4, 2 * TILE>(h);
    }
  }
  else
  {
    switch (v)
    {
    case 0: return launch_once<R, NPE, ONE, 4>(h);
    case 1: return launch_once_t<R, NPE, false, true, 4>(h);
    case 2: return launch_tma<R, NPE, ONE, 2>(h);
    case 3: return launch_tma<R, NPE, ONE, 3>(h);
    case 4: return launch_plain<R, NPE, ONE, 2>(h);
    case 5: return launch_tma<R, NPE, ONE, 1>(h);
    case 6: return launch_stage<R, NPE, ONE, 2>(h);
    case 7: return launch_stage<R, NPE, ONE, 1>(h);
    case 8: return launch_plain<R, NPE, ONE, 8, TILE / 2>(h);
    case 9: return launch_plain<R, NPE, ONE, 6, TILE / 2>(h);
    case 10: return launch_plain<R, NPE, ONE, 2, 2 * TILE>(h);
    default: return launch_plain<R, NPE, ONE, 1, 2 * TILE>(h);
    }
  }
}

int launch_element_any(dnl_engine *h, int mode)
{
  const int blocks = (int)(((long)h->nE * h->npe + TILE - 1) / TILE);
  if (mode == 1)
  {
    if (h->precision == DNL_PREC_MIXED)
    {
      if (h->npe == 8)
        return launch(h, k_element_start<float, 8>, blocks, TILE, 0, h->M);
      return launch(h, k_element_start<float, 4>, blocks, TILE, 0, h->M);
    }
    else
    {
      if (h->npe == 8)
        return launch(h, k_element_start<double, 8>, blocks, TILE, 0, h->M);
      return launch(h, k_element_start<double, 4>, blocks, TILE, 0, h->M);
    }
  }
  else
  {
    if (h->nInst > 1)
    {
      // the running instances of this increment, for the element, nodal and Courant passes
      if (int rc = launch(h, k_active_list, 1, 1024, 0, h->M, h->npe))
        return rc;
    }
    if (h->mode != DNL_MODE_PLAIN)
      return h->npe == 8 ? launch_mode_any<8>(h) : launch_mode_any<4>(h);
    else if (h->npe == 4)
    {
      // the axisymmetric models are small: one plain variant
      if (h->precision == DNL_PREC_MIXED)
        return h->oneMat ? launch_plain<float, 4, true, 6>(h) : launch_plain<float, 4, false, 6>(h);
      return h->oneMat ? launch_plain<double, 4, true, 4>(h) : launch_plain<double, 4, false, 4>(h);
    }
    else if (h->oneMat)
      return h->precision == DNL_PREC_MIXED ? launch_variant<float, 8, true>(h, h->variant)
                                            : launch_variant<double, 8, true>(h, h->variant);
    else
      return h->precision == DNL_PREC_MIXED ? launch_variant<float, 8, false>(h, h->variant)
                                            : launch_variant<double, 8, false>(h, h->variant);
  }
}

int launch_nodal(dnl_engine *h)
{
  const int threads = NODAL_THREADS;
  if (h->nInst > 1)
  {
    // a batch loops over its running instances' nodes
    const int blocks = std::min((h->nN + threads - 1) / threads, 16 * h->numSMs);
    if (h->precision == DNL_PREC_MIXED)
    {
      if (h->dim == 3)
        return launch(h, k_nodal_batch<float, 3>, blocks, threads, 0, h->M);
      return launch(h, k_nodal_batch<float, 2>, blocks, threads, 0, h->M);
    }
    else
    {
      if (h->dim == 3)
        return launch(h, k_nodal_batch<double, 3>, blocks, threads, 0, h->M);
      return launch(h, k_nodal_batch<double, 2>, blocks, threads, 0, h->M);
    }
  }
  else
  {
    // a thread per (node, component)
    const int blocks = (int)((3LL * h->nN + threads - 1) / threads);
    if (h->precision == DNL_PREC_MIXED)
    {
      if (h->dim == 3)
        return launch_pdl(h, k_nodal<float, 3>, blocks, threads, 0, h->M);
      return launch_pdl(h, k_nodal<float, 2>, blocks, threads, 0, h->M);
    }
    else
    {
      if (h->dim == 3)
        return launch_pdl(h, k_nodal<double, 3>, blocks, threads, 0, h->M);
      return launch_pdl(h, k_nodal<double, 2>, blocks, threads, 0, h->M);
    }
  }
}

int launch_courant(dnl_engine *h, int force)
{
  const int threads = 256, blocks = (h->nE + threads - 1) / threads;
  if (h->precision == DNL_PREC_MIXED)
  {
    if (h->npe == 8)
      return launch(h, k_courant<float, 8>, blocks, threads, 0, h->M, force);
    return launch(h, k_courant<float, 4>, blocks, threads, 0, h->M, force);
  }
  else
  {
    if (h->npe == 8)
      return launch(h, k_courant<double, 8>, blocks, threads, 0, h->M, force);
    return launch(h, k_courant<double, 4>, blocks, threads, 0, h->M, force);
  }
}

int launch_gather(dnl_engine *h, int what)
{
  const int threads = 256, blocks = (h->nN + threads - 1) / threads;
  if (h->precision == DNL_PREC_MIXED)
    return launch(h, k_gather<float>, blocks, threads, 0, h->M, what);
  return launch(h, k_gather<double>, blocks, threads, 0, h->M, what);
}

int launch_control(dnl_engine *h, int phase, double t_stop = 0.0, long long max_incs = 0)
{
  const int threads = 128, blocks = (h->nInst + threads - 1) / threads;
  return launch(h, k_control, blocks, threads, 0, h->M, phase, t_stop, max_incs);
}

int launch_bc_prep(dnl_engine *h)
{
  if (!h->hasSpeed)
    return DNL_OK;
  const int threads = 128, blocks = (h->nSpeed + threads - 1) / threads;
  return launch(h, k_bc_prep, blocks, threads, 0, h->M);
}

// Power-iteration time step: one cooperative launch (grid barriers inside).
int launch_pi(dnl_engine *h, int force)
{
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(h->piGrid);
  cfg.blockDim = dim3(TILE);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = h->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (h->npe == 8)
    CK(cudaLaunchKernelEx(&cfg, k_power_iteration<8>, h->M, force));
  else
    CK(cudaLaunchKernelEx(&cfg, k_power_iteration<4>, h->M, force));
  h->launches++;
  return DNL_OK;
}

int launch_timestep(dnl_engine *h, int force)
{
  return h->powerIteration ? launch_pi(h, force) : launch_courant(h, force);
}

// End of an increment: the time-step pass when due and the control update.
// With the Courant time step both run in one launch (k_courant_finish).
int launch_step_end(dnl_engine *h)
{
  if (h->powerIteration)
  {
    const int rc = launch_pi(h, 0);
    return rc ? rc : launch_control(h, CTL_FINISH);
  }
  const int threads = 256;
  const int blocks = std::max(1, std::min((h->nE + threads - 1) / threads, 2 * h->numSMs));
  if (h->precision == DNL_PREC_MIXED)
  {
    if (h->npe == 8)
      return launch_pdl(h, k_courant_finish<float, 8>, blocks, threads, 0, h->M);
    return launch_pdl(h, k_courant_finish<float, 4>, blocks, threads, 0, h->M);
  }
  else
  {
    if (h->npe == 8)
      return launch_pdl(h, k_courant_finish<double, 8>, blocks, threads, 0, h->M);
    return launch_pdl(h, k_courant_finish<double, 4>, blocks, threads, 0, h->M);
  }
}

// History records of the increment that just ended (single models with
// dnl_engine_set_history): one block after the end of the increment.
int launch_history(dnl_engine *h)
{
  if (!h->histOn)
    return DNL_OK;
  const int kin = h->itemsKinetic;
  if (h->precision == DNL_PREC_MIXED)
    return launch_pdl(h, k_history_ring<float>, 1, 256, 0, h->M, h->hist, (const int4 *)h->ditems,
                      (const long long *)h->ditemOff, h->nItems, (int)h->nValues, kin);
  return launch_pdl(h, k_history_ring<double>, 1, 256, 0, h->M, h->hist, (const int4 *)h->ditems,
                    (const long long *)h->ditemOff, h->nItems, (int)h->nValues, kin);
}

// The k_steps builds of the engine's precision, element, materials and time step method.
template <typename R> StepsBuild steps_build_of(const dnl_engine *h, int budget)
{
  if (h->npe == 8)
    return h->powerIteration ? steps_build<R, 8, true>(h->oneMat, budget) : steps_build<R, 8, false>(h->oneMat, budget);
  return h->powerIteration ? steps_build<R, 4, true>(h->oneMat, budget) : steps_build<R, 4, false>(h->oneMat, budget);
}

// Whether runs of this engine go through k_steps: a single model whose tiles all
// fit on the GPU at once at one of the register budgets (of 148 SMs, FP64: 444
// tiles, 7,104 hexahedra or 14,208 quadrilaterals; FP32: 592 tiles, 9,472 or
// 18,944).  Near the largest sizes the gain over graph replays is 13 to 17 %, at
// 25 tiles a quarter to a third (figures at k_steps); with more blocks per SM
// the element phase spills (FP64 at 128 registers, measured with the law's
// library calls: 23.3 against 20.4 us on 378 tiles).
void plan_steps(dnl_engine *h)
{
  h->steps = StepsBuild{};
  int coop = 0;
  if (h->nInst != 1 ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device) != cudaSuccess || !coop)
    return;
  for (int k = 0; k < STEPS_BUDGETS && !h->steps.kernel; k++)
  {
    const StepsBuild b = h->precision == DNL_PREC_MIXED ? steps_build_of<float>(h, k) : steps_build_of<double>(h, k);
    if (h->nTiles > b.minb * h->numSMs)
      continue; // the kernel stays unloaded
    int perSM = 0;
    if (cudaFuncSetAttribute(b.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b.smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, b.kernel, TILE, b.smem) != cudaSuccess)
    {
      cudaGetLastError();
      perSM = 0;
    }
    if (h->nTiles <= perSM * h->numSMs)
      h->steps = b;
  }
}

bool use_steps(const dnl_engine *h) { return h->steps.kernel && h->mode == DNL_MODE_PLAIN && !h->forced; }

// n increments at most (fewer when the model stops) in one launch.
int launch_steps(dnl_engine *h, int n, bool timed)
{
  StepsArgs a{};
  a.nIncs = n;
  a.bar = h->stepsBar;
  a.err = h->derr;
  a.pimax = h->stepsPhase + 4;
  a.phase = timed ? h->stepsPhase : nullptr;
  if (h->histOn)
  {
    a.histOn = 1;
    a.hist = h->hist;
    a.items = h->ditems;
    a.off = h->ditemOff;
    a.nItems = h->nItems;
    a.nValues = (int)h->nValues;
    a.kin = h->itemsKinetic;
  }
  CK(cudaMemsetAsync(h->stepsBar, 0, 4 * sizeof(unsigned long long), h->stream)); // and the maxima
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.gridDim = dim3(h->nTiles);
  cfg.blockDim = dim3(TILE);
  cfg.dynamicSmemBytes = h->steps.smem;
  cfg.stream = h->stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  void *args[] = {&h->M, &a};
  CK(cudaLaunchKernelExC(&cfg, h->steps.kernel, args));
  h->launches++;
  return DNL_OK;
}

template <typename R, int NPE> int launch_energies_t(dnl_engine *h, double *dst, const EnergyArgs &a, int n)
{
  k_energy_parts<R, NPE><<<(unsigned)a.blocks * n, 256, 0, h->stream>>>(h->M, h->denergyPart, a);
  k_energy_sum<<<n, 32, 0, h->stream>>>(h->denergyPart, dst, a);
  CK(cudaGetLastError());
  return DNL_OK;
}
// Energies of n instances from `first` on into dst [n][3]; points (one instance
// only: the room for the partials) false: the kinetic only.
int launch_energies(dnl_engine *h, double *dst, int speed_field, bool points, int first, int n)
{
  const int kin = h->kinBlocks, pts = points ? h->pointBlocks : 0;
  const EnergyArgs a{first, speed_field, kin, pts, std::max(kin, pts)};
  if (h->precision == DNL_PREC_MIXED)
    return h->npe == 8 ? launch_energies_t<float, 8>(h, dst, a, n) : launch_energies_t<float, 4>(h, dst, a, n);
  return h->npe == 8 ? launch_energies_t<double, 8>(h, dst, a, n) : launch_energies_t<double, 4>(h, dst, a, n);
}

// One increment: the kernels of the graph.
int enqueue_step(dnl_engine *h)
{
  int rc;
  if ((rc = launch_bc_prep(h)) || (rc = launch_element_any(h, 0)) || (rc = launch_nodal(h)) ||
      (rc = launch_step_end(h)))
    return rc;
  return launch_history(h);
}

// Increments of one k_steps launch: at 5 to 25 us each a launch lasts 2 to 13 ms.
constexpr int STEPS_CHUNK = 512;

// Graph replays a run issues between two looks at the device (about dflt
// increments): every increment can add a history record, so no more than the
// ring holds.
int poll_chunk(const dnl_engine *h, int dflt)
{
  const int incs = h->histOn ? std::min(dflt, h->hist.cap) : dflt;
  return std::max(1, incs / h->graphIncs);
}

// Records written on the device since the last look, appended on the host.
int drain_history(dnl_engine *h)
{
  if (!h->histOn)
    return DNL_OK;
  int cnt[2] = {0, 0}; // count, overflow (adjacent in the ring's memory)
  CK(cudaMemcpyAsync(cnt, h->hist.count, 2 * sizeof(int), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  if (cnt[1])
    return fail(h, DNL_ERR_ARG, "history ring overflow (capacity %d records)", h->hist.cap);
  if (cnt[0] > 0)
  {
    const size_t width = HIST_HEAD + (size_t)h->nValues, old = h->histHost.size();
    h->histHost.resize(old + width * cnt[0]);
    CK(cudaMemcpyAsync(h->histHost.data() + old, h->hist.rec, sizeof(double) * width * cnt[0],
                       cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemsetAsync(h->hist.count, 0, sizeof(int), h->stream));
    CK(cudaStreamSynchronize(h->stream));
  }
  return DNL_OK;
}

void drop_graph(dnl_engine *h)
{
  if (h->graphExec)
  {
    cudaGraphExecDestroy(h->graphExec);
    cudaGraphDestroy(h->graph);
    h->graphExec = nullptr;
    h->graph = nullptr;
  }
  for (auto &g : h->remExec)
    if (g)
    {
      cudaGraphExecDestroy(g);
      g = nullptr;
    }
}

// A graph of n increments, each kernel after the first waiting for the
// previous one by programmatic serialization, also across the increments'
// boundaries; increments past an instance's stop find it inactive and do
// nothing.  *launches: the kernels of one replay.  The graph is uploaded
// after instantiation, so that its first replay does not carry the upload.
int capture_steps(dnl_engine *h, int n, cudaGraph_t *graph, cudaGraphExec_t *exec, int *launches)
{
  long long before = h->launches;
  CK(cudaStreamBeginCapture(h->stream, cudaStreamCaptureModeThreadLocal));
  int rc = DNL_OK;
  for (int k = 0; k < n && !rc; k++)
    rc = enqueue_step(h);
  cudaError_t e = cudaStreamEndCapture(h->stream, graph);
  if (rc)
  {
    // (a capture that a launch has broken off gives no graph)
    if (e == cudaSuccess)
      cudaGraphDestroy(*graph);
    cudaGetLastError();
    *graph = nullptr;
    h->launches = before;
    return rc;
  }
  if (e != cudaSuccess)
    return fail(h, DNL_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(e));
  CK(cudaGraphInstantiate(exec, *graph, 0));
  // the executable graph goes to the device now, not at its first replay
  CK(cudaGraphUpload(*exec, h->stream));
  *launches = (int)(h->launches - before);
  h->launches = before;
  return DNL_OK;
}

int build_graph(dnl_engine *h)
{
  if (h->graphExec)
    return DNL_OK;
  return capture_steps(h, h->graphIncs, &h->graph, &h->graphExec, &h->launchesPerStep);
}

// The graph of r (1 <= r < graphIncs) increments: the end of a run of a known
// number of increments, so that no replay runs increments past it.
int build_rem_graph(dnl_engine *h, int r)
{
  if (h->remExec[r])
    return DNL_OK;
  cudaGraph_t g = nullptr;
  int rc = capture_steps(h, r, &g, &h->remExec[r], &h->remLaunches[r]);
  if (g)
    cudaGraphDestroy(g);
  return rc;
}

int sync_ctl(dnl_engine *h)
{
  CK(cudaMemcpyAsync(h->hctl, h->M.ctl, sizeof(Ctl) * h->nInst, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return DNL_OK;
}

int check_status(dnl_engine *h)
{
  int e = 0;
  if (cudaMemcpyAsync(&e, h->derr, sizeof(int), cudaMemcpyDeviceToHost, h->stream) == cudaSuccess &&
      cudaStreamSynchronize(h->stream) == cudaSuccess && e != 0)
    return fail(h, DNL_ERR_CUDA, "a bulk copy of the element pass or a grid barrier did not complete in time");
  for (int i = 0; i < h->nInst; i++)
    if (h->hctl[i].status != 0)
    {
      const char *what = h->hctl[i].status == DNL_ERR_NEG_JACOBIAN ? "negative Jacobian in element"
                                                                   : "radial return did not converge at point";
      return fail(h, h->hctl[i].status, "instance %d: %s %d (time %.6e)", i, what, h->hctl[i].bad, h->hctl[i].t);
    }
  return DNL_OK;
}

} // namespace

// =================================================================== C ABI

extern "C" {

int dnl_device_count(void)
{
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess)
  {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int dnl_release_memory(void)
{
  const cudaError_t e = dnl_pool_release();
  if (e == cudaSuccess)
    return DNL_OK;
  cudaGetLastError();
  return fail(nullptr, DNL_ERR_CUDA, "dnl_release_memory: %s", cudaGetErrorString(e));
}

const char *dnl_engine_last_error(const dnl_engine *h) { return h ? h->err.c_str() : g_create_err; }

int dnl_engine_batch_create(const dnl_model_desc *const *descs, int32_t n, dnl_engine **out)
{
  if (!out || !descs || n <= 0)
    return fail(nullptr, DNL_ERR_ARG, "invalid arguments");
  *out = nullptr;
  for (int i = 0; i < n; i++)
  {
    int rc = check_desc(descs[i], i);
    if (rc)
      return rc;
    if (descs[i]->elem_type != descs[0]->elem_type || descs[i]->precision != descs[0]->precision)
      return fail(nullptr, DNL_ERR_ARG, "all models of a batch share the element type and precision");
    if (n > 1 && descs[i]->ts_method == DNL_TS_POWER_ITERATION)
      return fail(nullptr, DNL_ERR_UNSUPPORTED, "the power-iteration time step is available for single models only");
  }
  if (dnl_device_count() == 0)
    return fail(nullptr, DNL_ERR_NO_DEVICE, "no CUDA device visible");

  dnl_engine *h = new dnl_engine;
  cudaGetDevice(&h->device);
  if (cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) != cudaSuccess)
  {
    delete h;
    return fail(nullptr, DNL_ERR_CUDA, "cudaStreamCreate failed");
  }
  h->type = descs[0]->elem_type;
  h->npe = npe_of(h->type);
  h->dim = h->npe == 8 ? 3 : 2;
  h->precision = descs[0]->precision;
  h->nInst = n;

  // ---- per instance (host, O(instances)): its first node, element, material
  // and function, the materials, the time functions and the control blocks;
  // the node and element arrays themselves are built on the device below
  std::vector<int4> base(n);
  std::vector<MatDev> mats;
  std::vector<double> fx, fy;
  std::vector<int> foff(1, 0);
  h->elemBegin.assign(1, 0);
  h->nodeBegin.assign(1, 0);
  long long nn = 0, ne = 0;
  bool anySpeed = false;
  for (int i = 0; i < n; i++)
  {
    const dnl_model_desc *d = descs[i];
    base[i] = make_int4((int)nn, (int)ne, (int)mats.size(), (int)foff.size() - 1);
    // an imposed speed other than zero (an imposed zero restrains the component)
    if (d->bc_code && d->bc_value && !anySpeed)
      for (long long k = 0; k < 3LL * d->n_nodes; k++)
        if (d->bc_code[k] == DNL_BC_SPEED && d->bc_value[k] != 0.0)
        {
          anySpeed = true;
          break;
        }
    for (int m = 0; m < d->n_materials; m++)
      mats.push_back(make_mat(d->materials[m]));
    for (int f = 0; f < d->n_functions; f++)
    {
      for (int p = 0; p < d->functions[f].n_points; p++)
      {
        fx.push_back(d->functions[f].x[p]);
        fy.push_back(d->functions[f].y[p]);
      }
      foff.push_back((int)fx.size());
    }
    Ctl c;
    memset(&c, 0, sizeof(c));
    double rb = (d->rho_b >= 0.0 && d->rho_b <= 1.0) ? d->rho_b : 0.8182;
    // Chung-Hulbert parameters (Explicit.C:86-104)
    c.alphaM = (2.0 * rb - 1.0) / (1.0 + rb);
    c.beta = (5.0 - 3.0 * rb) / ((1.0 + rb) * (1.0 + rb) * (2.0 - rb));
    c.gammaN = 1.5 - c.alphaM;
    c.omegaS = sqrt((12.0 * pow(1.0 + rb, 3) * (2.0 - rb)) / (10.0 + 15.0 * rb - rb * rb + pow(rb, 3) - pow(rb, 4)));
    c.safety = d->ts_safety > 0 ? d->ts_safety : 0.9;
    c.ts_freq = d->ts_freq > 0 ? d->ts_freq : 10;
    c.ts_method = d->ts_method;
    c.direct = d->stress_method == DNL_STRESS_DIRECT;
    c.plane = d->elem_type == DNL_ELQUA4N2D;
    c.t = d->t_start;
    c.t_end = d->t_end;
    c.t_stop = d->t_end;
    c.min_bits = INF_BITS;
    c.inc_stop = 0x7fffffffffffffffll;
    c.elem_begin = (int)ne;
    c.elem_end = (int)(ne + d->n_elems);
    c.node_begin = (int)nn;
    c.node_end = (int)(nn + d->n_nodes);
    h->ctlInit.push_back(c);
    nn += d->n_nodes;
    ne += d->n_elems;
    h->elemBegin.push_back((int)ne);
    h->nodeBegin.push_back((int)nn);
  }
  if (nn * 3 > 0x3fffffffLL || ne * h->npe > 0x3fffffffLL)
  {
    dnl_engine_destroy(h);
    return fail(nullptr, DNL_ERR_ARG, "model too large for 32-bit point indices");
  }
  h->nN = (int)nn;
  h->nE = (int)ne;
  h->nIP = h->nE * h->npe;
  // the engine's node numbering, instance by instance (within its node range)
  h->nodeOrder.assign(n, DNL_ORDER_GIVEN);
  for (int i = 0; i < n; i++)
  {
    const std::vector<int> order = node_order_of(descs[i], h->npe);
    if (order.empty())
      continue;
    if (h->intOf.empty())
    {
      h->intOf.resize(nn);
      h->extOf.resize(nn);
      for (int k = 0; k < (int)nn; k++)
        h->intOf[k] = h->extOf[k] = k;
    }
    h->nodeOrder[i] = DNL_ORDER_RCM;
    const int b = base[i].x;
    for (int k = 0; k < descs[i]->n_nodes; k++)
    {
      h->extOf[b + k] = b + order[k];
      h->intOf[b + order[k]] = b + k;
    }
  }
  const bool renum = !h->intOf.empty();
  h->nTiles = (h->nIP + TILE - 1) / TILE;
  h->nIPpad = h->nTiles * TILE;
  h->hasSpeed = anySpeed;
  h->nFunc = (int)foff.size() - 1;
  if (fx.empty())
  {
    fx.push_back(0.0);
    fy.push_back(0.0);
  }

  // ---- device memory of the model: one allocation, carved in 256-byte aligned parts
  const size_t rsz = h->precision == DNL_PREC_MIXED ? 4 : 8;
  const size_t nN = (size_t)h->nN, nI = (size_t)n, nIPpad = (size_t)h->nIPpad, nSp = anySpeed ? nN : 1;
  // energies: the blocks of k_energy_parts that have a node, a point of the
  // largest instance; partials of all instances' kinetic energies or one's three
  int mostNodes = 0, mostElems = 0;
  for (int i = 0; i < n; i++)
  {
    mostNodes = std::max(mostNodes, descs[i]->n_nodes);
    mostElems = std::max(mostElems, descs[i]->n_elems);
  }
  h->kinBlocks = std::min(KIN_GROUPS, (mostNodes + 255) / 256);
  h->pointBlocks = (int)std::min<long long>(ENERGY_BLOCKS, ((long long)mostElems * h->npe + 255) / 256);
  const size_t nPart = std::max((size_t)h->kinBlocks * nI, (size_t)h->kinBlocks + 2 * h->pointBlocks);
  // force slots: room for the fixed-stride layout (npe per node) or the CSR one
  const size_t nSlotCap = std::max((size_t)h->nIP, nN * h->npe);
  h->nSlotCap = nSlotCap;
  size_t total = 0;
  auto reserve = [&](size_t bytes) {
    const size_t o = total;
    total += (bytes + 255) / 256 * 256;
    return o;
  };
  const size_t o_eb = reserve(sizeof(int) * (nI + 1)), o_nb = reserve(sizeof(int) * (nI + 1)),
               o_conn = reserve(sizeof(int) * nIPpad), o_emat = reserve(sizeof(int) * (nIPpad / h->npe)),
               o_mat = reserve(sizeof(MatDev) * mats.size()), o_off = reserve(sizeof(int) * (nN + 1)),
               o_pos = reserve(sizeof(int) * nIPpad), o_bc = reserve(nN), o_bcval = reserve(sizeof(double4) * nSp),
               o_bcfun = reserve(sizeof(int4) * nSp), o_speed = reserve(sizeof(int) * nSp),
               o_fx = reserve(sizeof(double) * fx.size()), o_fy = reserve(sizeof(double) * fy.size()),
               o_foff = reserve(sizeof(int) * foff.size()), o_nodes = reserve(sizeof(double4) * nN * 9),
               o_mass = reserve(sizeof(double) * nN), o_ctl = reserve(sizeof(Ctl) * nI),
               o_perm = reserve(sizeof(int) * (renum ? nN : 1)),
               // zeroed at creation, from here to o_ip
               o_energy = reserve(sizeof(double) * (3 + nPart)), o_err = reserve(sizeof(int)),
               o_stats = reserve(sizeof(unsigned long long) * 5), o_done = reserve(sizeof(unsigned) * 2),
               o_steps = reserve(sizeof(unsigned long long) * 7),
               o_act = reserve(sizeof(int)), o_actlist = reserve(sizeof(int) * nI),
               o_acttile = reserve(sizeof(int) * (nI + 1)), o_actnode = reserve(sizeof(int) * (nI + 1)),
               o_actelem = reserve(sizeof(int) * (nI + 1)), o_due = reserve(sizeof(int)),
               o_duelist = reserve(sizeof(int) * nI), o_dueelem = reserve(sizeof(int) * (nI + 1)),
               o_ip = reserve((size_t)DNL_IP_NCOMP * nIPpad * rsz), o_slot = reserve(nSlotCap * 4 * rsz);
  char *A = nullptr;
  {
    cudaError_t e = dnl_pool_alloc((void **)&A, total, h->stream);
    if (e != cudaSuccess)
    {
      dnl_engine_destroy(h);
      return fail(nullptr, DNL_ERR_CUDA, "allocation of %zu bytes failed: %s", total, cudaGetErrorString(e));
    }
    h->allocs.push_back(A);
  }
  DevModel &M = h->M;
  M.nInst = h->nInst;
  M.nN = h->nN;
  M.nE = h->nE;
  M.nIP = h->nIP;
  M.nIPpad = h->nIPpad;
  M.nFunc = h->nFunc;
  M.inst_elem_begin = (const int *)(A + o_eb);
  M.inst_node_begin = (const int *)(A + o_nb);
  M.conn = (const int *)(A + o_conn);
  M.emat = (const int *)(A + o_emat);
  M.mat = (const MatDev *)(A + o_mat);
  h->oneMat = mats.size() == 1;
  M.one32 = mats[0].jc32;
  M.one64 = mats[0].jc64;
  M.one_rho0 = mats[0].rho0;
  M.csr_off = (const int *)(A + o_off);
  M.slot_pos = (const int *)(A + o_pos);
  M.bc = (const uint8_t *)(A + o_bc);
  M.bcval = (const double4 *)(A + o_bcval);
  M.bcfun = (const int4 *)(A + o_bcfun);
  M.speed_nodes = (const int *)(A + o_speed);
  M.fx = (const double *)(A + o_fx);
  M.fy = (const double *)(A + o_fy);
  M.foff = (const int *)(A + o_foff);
  double4 *nodes = (double4 *)(A + o_nodes);
  M.x = nodes;
  M.disp = nodes + nN;
  M.u[0] = nodes + 2 * nN;
  M.u[1] = nodes + 3 * nN;
  M.v[0] = nodes + 4 * nN;
  M.v[1] = nodes + 5 * nN;
  M.a[0] = nodes + 6 * nN;
  M.a[1] = nodes + 7 * nN;
  M.fout = nodes + 8 * nN;
  M.mass = (double *)(A + o_mass);
  M.ctl = (Ctl *)(A + o_ctl);
  h->dIntOf = renum ? (const int *)(A + o_perm) : nullptr;
  h->denergy = (double *)(A + o_energy);
  h->denergyPart = h->denergy + 3;
  h->derr = (int *)(A + o_err);
  h->dstats = (unsigned long long *)(A + o_stats);
  M.done_count = (unsigned *)(A + o_done);
  M.step_due = M.done_count + 1;
  h->stepsPhase = (unsigned long long *)(A + o_steps);
  h->stepsBar = (unsigned *)(h->stepsPhase + 3); // then the power iteration's three maxima
  M.act_count = (int *)(A + o_act);
  M.act_list = (int *)(A + o_actlist);
  M.act_tile_pre = (int *)(A + o_acttile);
  M.act_node_pre = (int *)(A + o_actnode);
  M.act_elem_pre = (int *)(A + o_actelem);
  M.due_count = (int *)(A + o_due);
  M.due_list = (int *)(A + o_duelist);
  M.due_elem_pre = (int *)(A + o_dueelem);
  M.ip = A + o_ip;
  M.slot = A + o_slot;
  M.stats = h->dstats;
  M.harvest_count = h->dstats + 4;
  M.harvest_stride = 1;
  M.guess_scope = DNL_GUESS_ALL;
  cudaDeviceGetAttribute(&h->numSMs, cudaDevAttrMultiProcessorCount, h->device);

  // ---- the caller's arrays as they come, into the read-back staging (reused later)
  size_t rtotal = 0;
  auto rreserve = [&](size_t bytes) {
    const size_t o = rtotal;
    rtotal += (bytes + 255) / 256 * 256;
    return o;
  };
  const int nScan = (h->nN + SCAN_BLOCK - 1) / SCAN_BLOCK;
  const size_t r_coords = rreserve(sizeof(double) * 3 * nN), r_vinit = rreserve(sizeof(double) * 3 * nN),
               r_bcval = rreserve(sizeof(double) * 3 * nN), r_bccode = rreserve(3 * nN),
               r_bcfun = rreserve(sizeof(int) * 3 * nN), r_conn = rreserve(sizeof(int) * (size_t)h->nIP),
               r_emat = rreserve(sizeof(int) * (size_t)h->nE), r_base = rreserve(sizeof(int4) * nI),
               r_count = rreserve(2 * sizeof(int)), r_cursor = rreserve(sizeof(int) * nN),
               r_list = rreserve(sizeof(int) * (size_t)h->nIP), r_sums = rreserve(sizeof(int) * (nScan + 1)),
               r_ext = rreserve(sizeof(int) * (renum ? nN : 1));
  char *Rw = nullptr;
  // a single model reserves the staging at its point state's size, so that
  // reading the state back later needs no allocation
  const size_t stateBytes = (size_t)DNL_IP_NCOMP * h->nIP * rsz;
  int rc = staging(h, n == 1 ? std::max(rtotal, stateBytes) : rtotal, (void **)&Rw);
  if (rc)
  {
    std::string e = h->err;
    dnl_engine_destroy(h);
    return fail(nullptr, rc, "%s", e.c_str());
  }
  BuildRaw R;
  R.coords = (const double *)(Rw + r_coords);
  R.vinit = (const double *)(Rw + r_vinit);
  R.bcval = (const double *)(Rw + r_bcval);
  R.bccode = (const int8_t *)(Rw + r_bccode);
  R.bcfun = (const int *)(Rw + r_bcfun);
  R.conn = (const int *)(Rw + r_conn);
  R.emat = (const int *)(Rw + r_emat);
  R.base = (const int4 *)(Rw + r_base);
  R.speedCount = (int *)(Rw + r_count);
  R.maxValence = R.speedCount + 1;
  R.cursor = (int *)(Rw + r_cursor);
  R.list = (int *)(Rw + r_list);
  R.blockSums = (int *)(Rw + r_sums);
  R.ext_of = renum ? (const int *)(Rw + r_ext) : nullptr;
  R.int_of = h->dIntOf;
  R.npe = h->npe;
  cudaError_t e = cudaSuccess;
  auto put = [&](size_t off, const void *src, size_t bytes) {
    if (e == cudaSuccess && bytes)
      e = cudaMemcpyAsync(Rw + off, src, bytes, cudaMemcpyHostToDevice, h->stream);
  };
  auto fill = [&](size_t off, int byte, size_t bytes) {
    if (e == cudaSuccess && bytes)
      e = cudaMemsetAsync(Rw + off, byte, bytes, h->stream);
  };
  for (int i = 0; i < n; i++)
  {
    const dnl_model_desc *d = descs[i];
    const size_t nb = (size_t)base[i].x, nni = (size_t)d->n_nodes, k3 = 3 * nb, n3 = 3 * nni;
    put(r_coords + sizeof(double) * k3, d->coords, sizeof(double) * n3);
    if (d->v_init)
      put(r_vinit + sizeof(double) * k3, d->v_init, sizeof(double) * n3);
    else
      fill(r_vinit + sizeof(double) * k3, 0, sizeof(double) * n3);
    if (d->bc_code)
      put(r_bccode + k3, d->bc_code, n3);
    else
      fill(r_bccode + k3, 0, n3);
    if (d->bc_value)
      put(r_bcval + sizeof(double) * k3, d->bc_value, sizeof(double) * n3);
    else
      fill(r_bcval + sizeof(double) * k3, 0, sizeof(double) * n3);
    if (d->bc_func)
      put(r_bcfun + sizeof(int) * k3, d->bc_func, sizeof(int) * n3);
    else
      fill(r_bcfun + sizeof(int) * k3, 0xff, sizeof(int) * n3); // -1: no function
    const size_t eb = (size_t)base[i].y;
    put(r_conn + sizeof(int) * eb * h->npe, d->conn, sizeof(int) * (size_t)d->n_elems * h->npe);
    if (d->elem_mat)
      put(r_emat + sizeof(int) * eb, d->elem_mat, sizeof(int) * (size_t)d->n_elems);
    else
      fill(r_emat + sizeof(int) * eb, 0, sizeof(int) * (size_t)d->n_elems);
  }
  put(r_base, base.data(), sizeof(int4) * nI);
  fill(r_count, 0, 2 * sizeof(int));
  if (renum)
  {
    put(r_ext, h->extOf.data(), sizeof(int) * nN);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(A + o_perm, h->intOf.data(), sizeof(int) * nN, cudaMemcpyHostToDevice, h->stream);
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_eb, h->elemBegin.data(), sizeof(int) * (nI + 1), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_nb, h->nodeBegin.data(), sizeof(int) * (nI + 1), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_mat, mats.data(), sizeof(MatDev) * mats.size(), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_fx, fx.data(), sizeof(double) * fx.size(), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_fy, fy.data(), sizeof(double) * fy.size(), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_foff, foff.data(), sizeof(int) * foff.size(), cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(A + o_ctl, h->ctlInit.data(), sizeof(Ctl) * nI, cudaMemcpyHostToDevice, h->stream);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(A + o_energy, 0, o_ip - o_energy, h->stream);
  if (e == cudaSuccess)
    e = cudaMemsetAsync(A + o_off, 0, sizeof(int) * (nN + 1), h->stream);
  if (e == cudaSuccess) // the padding slots of the fixed-stride layout stay zero
    e = cudaMemsetAsync(A + o_slot, 0, nSlotCap * 4 * rsz, h->stream);

  // ---- the model built on the device
  if (e == cudaSuccess)
  {
    const int tb = 256;
    k_build_nodes<<<(h->nN + tb - 1) / tb, tb, 0, h->stream>>>(M, R, anySpeed ? 1 : 0);
    k_build_elems<<<(h->nIPpad + tb - 1) / tb, tb, 0, h->stream>>>(M, R, h->nIPpad);
    int *offp = const_cast<int *>(M.csr_off) + 1;
    k_scan_blocks<<<nScan, SCAN_BLOCK, 0, h->stream>>>(offp, h->nN, R.blockSums);
    k_scan_sums<<<1, 32, 0, h->stream>>>(R.blockSums, nScan);
    k_scan_add<<<(h->nN + tb - 1) / tb, tb, 0, h->stream>>>(offp, h->nN, R.blockSums);
    k_slot_cursor<<<(h->nN + tb - 1) / tb, tb, 0, h->stream>>>(M, R);
    k_slot_fill<<<(h->nIP + tb - 1) / tb, tb, 0, h->stream>>>(M, R);
    k_slot_sort<<<(h->nN + tb - 1) / tb, tb, 0, h->stream>>>(M, R);
    k_slot_pos<<<(h->nN + tb - 1) / tb, tb, 0, h->stream>>>(M, R, h->npe);
    e = cudaGetLastError();
  }
  int counts[2] = {0, 0}; // nodes with an imposed speed, largest slot count of a node
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(counts, R.speedCount, 2 * sizeof(int), cudaMemcpyDeviceToHost, h->stream);
  if (e == cudaSuccess)
    e = cudaStreamSynchronize(h->stream);
  if (e != cudaSuccess)
  {
    dnl_engine_destroy(h);
    return fail(nullptr, DNL_ERR_CUDA, "model build failed: %s", cudaGetErrorString(e));
  }
  const int nSpeed = counts[0];
  h->nSpeed = nSpeed;
  M.nSpeed = nSpeed;
  // the layout k_slot_pos chose: npe slots per node when no node has more
  M.slotW = counts[1] <= h->npe ? h->npe : 0;
  // FP64 batches take the walking kernel under its own number, which also runs
  // a single model with the batch's arithmetic: with one material known at
  // compile time the FP64 build of variant 0 contracts differently.
  // 24 bars of 543,000 hexahedra together: 775.7 (stage/2) -> 689.9 us an increment,
  // 8 of 30,000: 68.5 -> 59.8.
  h->variant = h->nInst > 1 && h->precision == DNL_PREC_FP64 ? 1 : 0;
  h->powerIteration = (descs[0]->ts_method == DNL_TS_POWER_ITERATION);
  if (h->powerIteration)
  {
    // Model::computePowerIterationTimeStep start vector: linear from 1 to -1
    // over the degrees of freedom (Model.C:967-972)
    const int d = h->dim;
    const long ndof = (long)d * h->nN;
    std::vector<double> pv((size_t)3 * h->nN, 0.0);
    double prev = 1.0;
    for (long i = 0; i < ndof; i++)
    {
      const double val = (i == 0) ? 1.0 : prev - 2. / (ndof - 1);
      pv[3 * (i / d) + (i % d)] = val;
      prev = val;
    }
    int perSM = 0;
    if (h->npe == 8)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_power_iteration<8>, TILE, 0);
    else
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_power_iteration<4>, TILE, 0);
    const int tiles = (h->nIP + TILE - 1) / TILE;
    h->piGrid = std::max(1, std::min(tiles, std::max(perSM, 1) * h->numSMs));
    if ((rc = upload(h, &M.pv, pv)) || (rc = upload(h, &M.pv2, pv)) || (rc = dalloc(h, &M.pislot, h->nSlotCap)) ||
        (rc = dalloc(h, &M.blockmax, h->piGrid)))
    {
      std::string em = h->err;
      dnl_engine_destroy(h);
      snprintf(g_create_err, sizeof(g_create_err), "%s", em.c_str());
      return rc;
    }
    if (cudaStreamSynchronize(h->stream) != cudaSuccess)
    {
      dnl_engine_destroy(h);
      return fail(nullptr, DNL_ERR_CUDA, "upload failed");
    }
  }
  plan_steps(h);
  // host mirror of the control blocks (small: plain memory)
  h->hctl = new Ctl[h->nInst];
  *out = h;
  return DNL_OK;
}

int dnl_engine_create(const dnl_model_desc *desc, dnl_engine **out)
{
  const dnl_model_desc *d[1] = {desc};
  return dnl_engine_batch_create(d, 1, out);
}

namespace
{
void free_items(dnl_engine *h);
}

int dnl_engine_destroy(dnl_engine *h)
{
  if (!h)
    return DNL_OK;
  if (h->stream)
    cudaStreamSynchronize(h->stream);
  drop_graph(h);
  for (void *p : h->allocs)
    dnl_pool_free(p, h->stream);
  dnl_pool_free(h->dstage, h->stream);
  dnl_pool_free(h->histMem, h->stream);
  free_items(h);
  delete[] h->hctl;
  if (h->stream)
    cudaStreamDestroy(h->stream);
  delete h;
  return DNL_OK;
}

int dnl_engine_init(dnl_engine *h)
{
  if (!h)
    return DNL_ERR_ARG;
  // reference Jacobian, initial point state, element masses -> nodal lumped mass
  int rc;
  if ((rc = launch_element_any(h, 1)) || (rc = launch_gather(h, 0)))
    return rc;
  // Solver::computeTimeStep(true) (Explicit.C:156-158)
  if ((rc = launch_timestep(h, 1)) || (rc = launch_control(h, CTL_INIT_DT)))
    return rc;
  // first element pass at t_start (Explicit.C:161-181)
  if ((rc = launch_element_any(h, 0)) || (rc = launch_control(h, CTL_POST_INIT)))
    return rc;
  CK(cudaGetLastError());
  if ((rc = sync_ctl(h)))
    return rc;
  rc = check_status(h);
  if (rc)
    return rc;
  h->initialized = true;
  return DNL_OK;
}

int dnl_engine_run(dnl_engine *h, double t_pause, int64_t max_incs, int64_t *incs_done)
{
  if (!h)
    return DNL_ERR_ARG;
  if (!h->initialized)
    return fail(h, DNL_ERR_ARG, "dnl_engine_init must be called first");
  const bool steps = use_steps(h);
  const bool counted = !h->timing && max_incs > 0 && !h->histOn; // launches without polling
  const int rem = counted ? (int)(max_incs % h->graphIncs) : 0;
  int rc;
  if (!steps && ((rc = build_graph(h)) || (rem && (rc = build_rem_graph(h, rem)))))
    return rc;
  std::vector<long long> inc0(h->nInst);
  if ((rc = sync_ctl(h)))
    return rc;
  for (int i = 0; i < h->nInst; i++)
    inc0[i] = h->hctl[i].inc - ((h->hctl[i].prepared && h->hctl[i].active) ? 1 : 0);
  h->launches = 0;
  cudaEvent_t ev0, ev1;
  CK(cudaEventCreate(&ev0));
  CK(cudaEventCreate(&ev1));
  // reset the FP32 re-solve counters
  for (int i = 0; i < h->nInst; i++)
    CK(cudaMemsetAsync(&h->M.ctl[i].resolves, 0, sizeof(int), h->stream));
  CK(cudaEventRecord(ev0, h->stream));
  if ((rc = launch_control(h, CTL_LIMITS, t_pause, max_incs)))
    return rc;
  if (steps)
  {
    // STEPS_CHUNK increments a launch (less when the history ring holds
    // fewer), looking at the device after each unless their number is known
    if (h->timing)
      CK(cudaMemsetAsync(h->stepsPhase, 0, 3 * sizeof(unsigned long long), h->stream));
    const int chunk = h->histOn ? std::min(STEPS_CHUNK, h->hist.cap) : STEPS_CHUNK;
    for (int64_t s = 0;;)
    {
      const int n = max_incs > 0 ? (int)std::min<int64_t>(chunk, max_incs - s) : chunk;
      if ((rc = launch_steps(h, n, h->timing)))
        return rc;
      s += n;
      if (!counted)
      {
        if ((rc = sync_ctl(h)) || (rc = drain_history(h)))
          return rc;
        if (!h->hctl[0].active)
          break;
      }
      if (max_incs > 0 && s >= max_incs)
        break;
    }
    if (h->timing)
    {
      unsigned long long ns[3];
      CK(cudaMemcpyAsync(ns, h->stepsPhase, sizeof(ns), cudaMemcpyDeviceToHost, h->stream));
      CK(cudaStreamSynchronize(h->stream));
      for (int k = 0; k < 3; k++)
        h->times[k] = 1e-6 * (double)ns[k];
    }
  }
  else if (h->timing)
  {
    // kernel-by-kernel with events: per-phase device time.  A chunk of
    // increments is queued with its own events and read after one wait, so
    // that the kernels are already queued when their opening event completes
    // and each bracket holds device time only (waiting on every increment
    // would put the host's launch latency inside the brackets).
    // (increments, not graph replays: at most what the history ring holds)
    const int maxChunk = h->histOn ? std::max(1, std::min(64, h->hist.cap)) : 64;
    std::vector<cudaEvent_t> e(4 * (size_t)maxChunk);
    for (auto &ev : e)
      CK(cudaEventCreate(&ev));
    float acc[3] = {0, 0, 0};
    long long steps = 0;
    for (;;)
    {
      int queued = 0;
      for (int s = 0; s < maxChunk; s++)
      {
        cudaEvent_t *es = &e[4 * (size_t)s];
        if ((rc = launch_bc_prep(h)))
          break;
        CK(cudaEventRecord(es[0], h->stream));
        if ((rc = launch_element_any(h, 0)))
          break;
        CK(cudaEventRecord(es[1], h->stream));
        if ((rc = launch_nodal(h)))
          break;
        CK(cudaEventRecord(es[2], h->stream));
        if ((rc = launch_step_end(h)) || (rc = launch_history(h)))
          break;
        CK(cudaEventRecord(es[3], h->stream));
        queued++;
        if (max_incs > 0 && steps + queued >= max_incs)
          break;
      }
      if (rc)
        break;
      CK(cudaEventSynchronize(e[4 * (size_t)(queued - 1) + 3]));
      for (int s = 0; s < queued; s++)
      {
        const cudaEvent_t *es = &e[4 * (size_t)s];
        float t01, t12, t23;
        cudaEventElapsedTime(&t01, es[0], es[1]);
        cudaEventElapsedTime(&t12, es[1], es[2]);
        cudaEventElapsedTime(&t23, es[2], es[3]);
        acc[0] += t01;
        acc[1] += t12;
        acc[2] += t23;
      }
      steps += queued;
      if ((rc = sync_ctl(h)) || (rc = drain_history(h)))
        break;
      bool any = false;
      for (int i = 0; i < h->nInst; i++)
        any = any || h->hctl[i].active;
      if (!any || (max_incs > 0 && steps >= max_incs))
        break;
    }
    for (auto &ev : e)
      cudaEventDestroy(ev);
    if (rc)
      return rc;
    h->times[0] = acc[0];
    h->times[1] = acc[1];
    h->times[2] = acc[2];
  }
  else if (counted)
  {
    // known number of increments: replay the graph without polling, the last
    // rem increments by their own graph
    for (int64_t s = 0; s < max_incs / h->graphIncs; s++)
    {
      CK(cudaGraphLaunch(h->graphExec, h->stream));
      h->launches += h->launchesPerStep;
    }
    if (rem)
    {
      CK(cudaGraphLaunch(h->remExec[rem], h->stream));
      h->launches += h->remLaunches[rem];
    }
  }
  else
  {
    // until every instance stops (its end time, the pause time, or the
    // increment budget that CTL_LIMITS set), looking at the device every chunk
    const int chunk = poll_chunk(h, 64);
    for (;;)
    {
      for (int s = 0; s < chunk; s++)
      {
        CK(cudaGraphLaunch(h->graphExec, h->stream));
        h->launches += h->launchesPerStep;
      }
      if ((rc = sync_ctl(h)) || (rc = drain_history(h)))
        return rc;
      // an instance that fails stops alone; the others of a batch go on
      bool any = false;
      for (int i = 0; i < h->nInst; i++)
        any = any || h->hctl[i].active;
      if (!any)
        break;
    }
  }
  CK(cudaEventRecord(ev1, h->stream));
  CK(cudaEventSynchronize(ev1));
  float ms = 0;
  cudaEventElapsedTime(&ms, ev0, ev1);
  h->times[3] = ms;
  cudaEventDestroy(ev0);
  cudaEventDestroy(ev1);
  CK(cudaGetLastError());
  if ((rc = sync_ctl(h)))
    return rc;
  if (incs_done)
  {
    long long mx = 0;
    for (int i = 0; i < h->nInst; i++)
    {
      long long now = h->hctl[i].inc - ((h->hctl[i].prepared && h->hctl[i].active) ? 1 : 0);
      mx = std::max(mx, now - inc0[i]);
    }
    *incs_done = mx;
  }
  return check_status(h);
}

int dnl_engine_element_pass(dnl_engine *h, double time_step)
{
  if (!h)
    return DNL_ERR_ARG;
  if (!h->initialized)
    return fail(h, DNL_ERR_ARG, "dnl_engine_init must be called first");
  if (!(time_step > 0))
    return fail(h, DNL_ERR_ARG, "time step must be positive");
  // arm instance 0 with the given time step, run the element pass and assemble
  int rc = sync_ctl(h);
  if (rc)
    return rc;
  Ctl c = h->hctl[0];
  c.active = 1;
  c.prepared = 0;
  c.due = 0;
  c.dt_eff = time_step;
  c.t_new = c.t + time_step;
  for (int i = 1; i < h->nInst; i++)
  {
    Ctl ci = h->hctl[i];
    ci.active = 0;
    ci.prepared = 0;
    CK(cudaMemcpyAsync(&h->M.ctl[i], &ci, sizeof(Ctl), cudaMemcpyHostToDevice, h->stream));
  }
  CK(cudaMemcpyAsync(&h->M.ctl[0], &c, sizeof(Ctl), cudaMemcpyHostToDevice, h->stream));
  if ((rc = launch_element_any(h, 0)) || (rc = launch_gather(h, 1)) || (rc = launch_control(h, CTL_POST_INIT)))
    return rc;
  CK(cudaGetLastError());
  if ((rc = sync_ctl(h)))
    return rc;
  return check_status(h);
}

int dnl_engine_sizes(const dnl_engine *h, int32_t *ni, int32_t *nn, int32_t *ne, int32_t *nip)
{
  if (!h)
    return DNL_ERR_ARG;
  if (ni) *ni = h->nInst;
  if (nn) *nn = h->nN;
  if (ne) *ne = h->nE;
  if (nip) *nip = h->nIP;
  return DNL_OK;
}

int dnl_engine_instance_offsets(const dnl_engine *h, int32_t i, int32_t *node0, int32_t *elem0, int32_t *ip0)
{
  if (!h || i < 0 || i > h->nInst)
    return DNL_ERR_ARG;
  if (node0) *node0 = h->nodeBegin[i];
  if (elem0) *elem0 = h->elemBegin[i];
  if (ip0) *ip0 = h->elemBegin[i] * h->npe;
  return DNL_OK;
}

int dnl_engine_node_order(const dnl_engine *h, int32_t i, int32_t *order)
{
  if (!h || !order || i < 0 || i >= h->nInst)
    return DNL_ERR_ARG;
  *order = h->nodeOrder[i];
  return DNL_OK;
}

int dnl_engine_control(const dnl_engine *h, int32_t i, dnl_control *out)
{
  if (!h || !out || i < 0 || i >= h->nInst)
    return DNL_ERR_ARG;
  dnl_engine *hh = const_cast<dnl_engine *>(h);
  int rc = sync_ctl(hh);
  if (rc)
    return rc;
  const Ctl &c = h->hctl[i];
  out->time = c.t;
  out->time_step = (c.prepared && c.active) ? c.dt_eff : c.dt;
  out->t_end = c.t_end;
  out->increment = c.inc - ((c.prepared && c.active) ? 1 : 0);
  out->status = c.status;
  out->bad_index = c.bad;
  out->done = c.t >= c.t_end;
  out->fp64_resolves = c.resolves;
  out->last_time_step = (c.inc - ((c.prepared && c.active) ? 1 : 0)) > 0 ? c.dt_last : c.dt;
  return DNL_OK;
}

int dnl_engine_get_nodes(dnl_engine *h, int32_t field, double *out)
{
  if (!h || !out)
    return DNL_ERR_ARG;
  if (field < DNL_NODE_COORDS || field > DNL_NODE_ACCEL_PREV)
    return fail(h, DNL_ERR_ARG, "unknown nodal field %d", field);
  int rc;
  // the element slots hold the forces of the last element pass (of a run's
  // last increment, or of dnl_engine_element_pass): assemble them now, as
  // Model::computeInternalForces leaves them in Model::internalForces
  if (field == DNL_NODE_FORCE && (rc = launch_gather(h, 1)))
    return rc;
  // packed to [n][3] on the device (each instance on its own buffer parity),
  // then one copy into the caller's array
  const size_t bytes = sizeof(double) * 3 * (size_t)h->nN;
  void *st = nullptr;
  if ((rc = staging(h, bytes, &st)))
    return rc;
  k_nodes_out<<<(h->nN + 255) / 256, 256, 0, h->stream>>>(h->M, field, 0, h->nN, (double *)st, h->dIntOf);
  CK(cudaGetLastError());
  h->launches++;
  return copy(h, out, st, bytes, cudaMemcpyDeviceToHost);
}

int dnl_engine_set_nodes(dnl_engine *h, int32_t field, const double *in)
{
  if (!h || !in)
    return DNL_ERR_ARG;
  int rc = sync_ctl(h);
  if (rc)
    return rc;
  std::vector<double4> tmp(h->nN); // in the engine's numbering
  for (int i = 0; i < h->nN; i++)
    tmp[h->intOf.empty() ? i : h->intOf[i]] = make_double4(in[3 * i], in[3 * i + 1], in[3 * i + 2], 0.0);
  if (field == DNL_NODE_U || field == DNL_NODE_SPEED || field == DNL_NODE_ACCEL)
  {
    double4 **arr = field == DNL_NODE_U ? h->M.u : (field == DNL_NODE_SPEED ? h->M.v : h->M.a);
    // write into each instance's field0 buffer
    std::vector<double4> cur[2];
    for (int b = 0; b < 2; b++)
    {
      cur[b].resize(h->nN);
      { int rc_ = copy(h, cur[b].data(), arr[b], sizeof(double4) * h->nN, cudaMemcpyDeviceToHost); if (rc_) return rc_; }
    }
    for (int i = 0; i < h->nInst; i++)
      for (int k = h->nodeBegin[i]; k < h->nodeBegin[i + 1]; k++)
        cur[h->hctl[i].f0][k] = tmp[k];
    for (int b = 0; b < 2; b++)
      { int rc_ = copy(h, arr[b], cur[b].data(), sizeof(double4) * h->nN, cudaMemcpyHostToDevice); if (rc_) return rc_; }
    return DNL_OK;
  }
  double4 *dst = nullptr;
  switch (field)
  {
  case DNL_NODE_COORDS: dst = h->M.x; break;
  case DNL_NODE_DISP: dst = h->M.disp; break;
  default: return fail(h, DNL_ERR_ARG, "nodal field %d cannot be written", field);
  }
  { int rc_ = copy(h, dst, tmp.data(), sizeof(double4) * h->nN, cudaMemcpyHostToDevice); if (rc_) return rc_; }
  return DNL_OK;
}

int dnl_engine_get_ips(dnl_engine *h, double *out)
{
  if (!h || !out)
    return DNL_ERR_ARG;
  // the device reorders and widens a few components at a time into a staging
  // array, which is copied straight into the caller's array
  const size_t n = (size_t)h->nIP;
  const int group = 4;
  double *stage = nullptr;
  int rc = staging(h, sizeof(double) * n * group, (void **)&stage);
  if (rc)
    return rc;
  for (int c0 = 0; c0 < DNL_IP_NCOMP && rc == DNL_OK; c0 += group)
  {
    const int nc = std::min(group, DNL_IP_NCOMP - c0);
    const long long items = (long long)nc * (long long)n;
    const int threads = 256;
    const unsigned blocks = (unsigned)((items + threads - 1) / threads);
    if (h->precision == DNL_PREC_MIXED)
      k_ips_out<float><<<blocks, threads, 0, h->stream>>>(h->M, c0, nc, stage);
    else
      k_ips_out<double><<<blocks, threads, 0, h->stream>>>(h->M, c0, nc, stage);
    if (cudaGetLastError() != cudaSuccess)
      rc = fail(h, DNL_ERR_CUDA, "state read-back kernel failed");
    else
      rc = copy(h, out + (size_t)c0 * n, stage, sizeof(double) * n * nc, cudaMemcpyDeviceToHost);
  }
  return rc;
}

namespace
{
// Device side of dnl_engine_node_averages: n components into dst [n][nN].
int node_averages_dev(dnl_engine *h, const int32_t *comps, int n, double *dst)
{
  for (int k = 0; k < n; k++)
    if (!((comps[k] >= 0 && comps[k] < DNL_IP_NCOMP) || comps[k] == DNL_NODE_AVG_VON_MISES))
      return fail(h, DNL_ERR_ARG, "node average of unknown component %d", comps[k]);
  int rc;
  if (!h->dslotInc)
  {
    if ((rc = dalloc(h, &h->dslotInc, h->nSlotCap)))
      return rc;
    k_slot_incidence<<<(h->nIP + 255) / 256, 256, 0, h->stream>>>(h->M, h->dslotInc);
    h->launches++;
  }
  for (int b = 0; b < n; b += AvgComps::MAX)
  {
    AvgComps ac;
    ac.n = std::min(AvgComps::MAX, n - b);
    for (int k = 0; k < ac.n; k++)
      ac.c[k] = comps[b + k];
    const dim3 grid((h->nN + 127) / 128, (ac.n + AVG_GROUP - 1) / AVG_GROUP);
    double *o = dst + (size_t)b * h->nN;
    const bool f32 = h->precision == DNL_PREC_MIXED;
    if (h->npe == 8)
      f32 ? k_node_average<float, 8><<<grid, 128, 0, h->stream>>>(h->M, h->dslotInc, ac, o, h->dIntOf)
          : k_node_average<double, 8><<<grid, 128, 0, h->stream>>>(h->M, h->dslotInc, ac, o, h->dIntOf);
    else
      f32 ? k_node_average<float, 4><<<grid, 128, 0, h->stream>>>(h->M, h->dslotInc, ac, o, h->dIntOf)
          : k_node_average<double, 4><<<grid, 128, 0, h->stream>>>(h->M, h->dslotInc, ac, o, h->dIntOf);
    CK(cudaGetLastError());
    h->launches++;
  }
  return DNL_OK;
}

// The reference's VTK labels (Field.C:17-48) of the DNL_VTK_* fields, their kind
// (0 scalar, 1 vector, 2 tensor) and source: a nodal field DNL_NODE_* for
// the vectors (and the mass), a point-state component for the others.
struct VtkField
{
  const char *label;
  int kind;
  int node;  // DNL_NODE_* (current), or -1
  int prev;  // DNL_NODE_* read when prev = 1
  int comp;  // DNL_IP_* (first of 6 for a tensor) or DNL_NODE_AVG_VON_MISES, or -1
};
const VtkField kVtkFields[DNL_VTK_NFIELDS] = {
    {"coords", 1, DNL_NODE_COORDS, DNL_NODE_COORDS, -1},
    {"disp", 1, DNL_NODE_DISP, DNL_NODE_DISP, -1},
    {"dispInc", 1, DNL_NODE_U, DNL_NODE_U_PREV, -1},
    {"speed", 1, DNL_NODE_SPEED, DNL_NODE_SPEED_PREV, -1},
    {"speedInc", 1, DNL_NODE_ACCEL, DNL_NODE_ACCEL_PREV, -1},
    {"density", 0, -1, -1, DNL_IP_DENSITY},
    {"gamma", 0, -1, -1, DNL_IP_GAMMA},
    {"gammaCumulate", 0, -1, -1, DNL_IP_GAMMA_CUM},
    {"internalEnergy", 0, -1, -1, DNL_IP_EINT},
    {"plasticStrain", 0, -1, -1, DNL_IP_EPSP},
    {"plasticStrainRate", 0, -1, -1, DNL_IP_DEPSP},
    {"pressure", 0, -1, -1, DNL_IP_PRESSURE},
    {"T", 0, -1, -1, DNL_IP_T},
    {"vonMises", 0, -1, -1, DNL_NODE_AVG_VON_MISES},
    {"yield", 0, -1, -1, DNL_IP_YIELD},
    {"mass", 0, DNL_NODE_MASS, DNL_NODE_MASS, -1},
    {"PlasticStrain", 2, -1, -1, DNL_IP_PLASTIC_STRAIN},
    {"Strain", 2, -1, -1, DNL_IP_STRAIN},
    {"Stress", 2, -1, -1, DNL_IP_STRESS},
};

// Text output buffer: numbers printed as std::ostream prints a double by
// default (%g, 6 significant digits).
struct Text
{
  std::string s;
  char tmp[64];
  void num(double v)
  {
    const int k = snprintf(tmp, sizeof(tmp), "%g", v);
    s.append(tmp, (size_t)k);
  }
  void num(long v) { s += std::to_string(v); }
  void str(const char *t) { s += t; }
};
} // namespace

int dnl_engine_node_averages(dnl_engine *h, const int32_t *comps, int32_t n, double *out)
{
  if (!h || !comps || !out || n <= 0)
    return DNL_ERR_ARG;
  void *st = nullptr;
  int rc;
  if ((rc = staging(h, sizeof(double) * (size_t)n * h->nN, &st)) ||
      (rc = node_averages_dev(h, comps, n, (double *)st)))
    return rc;
  return copy(h, out, st, sizeof(double) * (size_t)n * h->nN, cudaMemcpyDeviceToHost);
}

int dnl_engine_write_vtk(dnl_engine *h, int32_t inst, const char *path, const char *title, const int32_t *fields,
                         int32_t n_fields, int32_t prev)
{
  if (!h || !path || (n_fields > 0 && !fields) || n_fields < 0)
    return DNL_ERR_ARG;
  if (inst < 0 || inst >= h->nInst)
    return fail(h, DNL_ERR_ARG, "instance %d out of range", inst);
  for (int k = 0; k < n_fields; k++)
    if (fields[k] < 0 || fields[k] >= DNL_VTK_NFIELDS)
      return fail(h, DNL_ERR_ARG, "unknown result field %d", fields[k]);
  int rc = sync_ctl(h);
  if (rc)
    return rc;
  const int n0 = h->nodeBegin[inst], nn = h->nodeBegin[inst + 1] - n0;
  const int e0 = h->elemBegin[inst], ne = h->elemBegin[inst + 1] - e0;
  // device columns: coordinates, then the nodal vectors, then the averages
  std::vector<int> nodeFields{DNL_NODE_COORDS};
  std::vector<int32_t> comps;
  std::vector<int> col(n_fields, -1); // first column (vector index or component index) of each field
  for (int k = 0; k < n_fields; k++)
  {
    const VtkField &f = kVtkFields[fields[k]];
    if (f.node >= 0)
    {
      col[k] = (int)nodeFields.size();
      nodeFields.push_back(prev ? f.prev : f.node);
    }
    else
    {
      col[k] = (int)comps.size();
      for (int c = 0; c < (f.kind == 2 ? 6 : 1); c++)
        comps.push_back(f.comp + c);
    }
  }
  const size_t vecBytes = sizeof(double) * 3 * (size_t)nn * nodeFields.size();
  const size_t avgBytes = sizeof(double) * (size_t)h->nN * comps.size();
  const size_t connBytes = sizeof(int) * (size_t)ne * h->npe;
  void *st = nullptr;
  if ((rc = staging(h, vecBytes + avgBytes + connBytes, &st)))
    return rc;
  double *dvec = (double *)st, *davg = (double *)((char *)st + vecBytes);
  for (size_t v = 0; v < nodeFields.size(); v++)
  {
    k_nodes_out<<<(nn + 255) / 256, 256, 0, h->stream>>>(h->M, nodeFields[v], n0, nn, dvec + v * 3 * (size_t)nn,
                                                         h->dIntOf);
    CK(cudaGetLastError());
    h->launches++;
  }
  if (!comps.empty() && (rc = node_averages_dev(h, comps.data(), (int)comps.size(), davg)))
    return rc;
  std::vector<double> vec(3 * (size_t)nn * nodeFields.size()), avg((size_t)h->nN * comps.size());
  std::vector<int> conn((size_t)ne * h->npe);
  CK(cudaMemcpyAsync(vec.data(), dvec, vecBytes, cudaMemcpyDeviceToHost, h->stream));
  if (!comps.empty())
    CK(cudaMemcpyAsync(avg.data(), davg, avgBytes, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaMemcpyAsync(conn.data(), h->M.conn + (size_t)e0 * h->npe, connBytes, cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));

  // VtkInterface::headerWrite / nodesWrite / elementsWrite / dataWrite
  Text o;
  o.s.reserve(64 * (size_t)nn * (1 + n_fields) + 32 * (size_t)ne);
  o.str("# vtk DataFile Version 4.0\n");
  o.str(title ? title : "");
  o.str("\nASCII\nDATASET UNSTRUCTURED_GRID\nFIELD FieldData 1\nTIME 1 1 double\n");
  o.num(h->hctl[inst].t);
  o.str("\nPOINTS ");
  o.num((long)nn);
  o.str(" float\n");
  for (int i = 0; i < nn; i++)
  {
    o.num(vec[3 * (size_t)i]);
    o.str(" ");
    o.num(vec[3 * (size_t)i + 1]);
    o.str(" ");
    o.num(vec[3 * (size_t)i + 2]);
    o.str("\n");
  }
  o.str("\nCELLS ");
  o.num((long)ne);
  o.str(" ");
  o.num((long)ne * (h->npe + 1));
  o.str("\n");
  for (int e = 0; e < ne; e++)
  {
    o.num((long)h->npe);
    o.str(" ");
    for (int j = 0; j < h->npe; j++)
    {
      const int c = conn[(size_t)e * h->npe + j];
      o.num((long)((h->extOf.empty() ? c : h->extOf[c]) - n0));
      o.str(" ");
    }
    o.str("\n");
  }
  o.str("\nCELL_TYPES ");
  o.num((long)ne);
  o.str("\n");
  const char *vtkType = h->npe == 8 ? "12\n" : "9\n"; // VTK_HEXAHEDRON, VTK_QUAD (ElementData vtkType)
  for (int e = 0; e < ne; e++)
    o.str(vtkType);
  o.str("\nPOINT_DATA ");
  o.num((long)nn);
  o.str("\n");
  for (int k = 0; k < n_fields; k++)
  {
    const VtkField &f = kVtkFields[fields[k]];
    if (f.kind == 1)
    {
      const double *v = vec.data() + (size_t)col[k] * 3 * nn;
      o.str("VECTORS ");
      o.str(f.label);
      o.str(" float\n");
      for (int i = 0; i < nn; i++)
      {
        o.num(v[3 * (size_t)i]);
        o.str(" ");
        o.num(v[3 * (size_t)i + 1]);
        o.str(" ");
        o.num(v[3 * (size_t)i + 2]);
        o.str("\n");
      }
    }
    else if (f.kind == 0)
    {
      o.str("SCALARS ");
      o.str(f.label);
      o.str(" float\nLOOKUP_TABLE default\n");
      for (int i = 0; i < nn; i++)
      {
        // the mass is a nodal vector (repeated on its components), the others node averages
        o.num(f.node >= 0 ? vec[(size_t)col[k] * 3 * nn + 3 * (size_t)i]
                          : avg[(size_t)col[k] * h->nN + n0 + i]);
        o.str("\n");
      }
    }
    else
    {
      o.str("TENSORS ");
      o.str(f.label);
      o.str(" float\n");
      static const int full[9] = {0, 1, 2, 1, 3, 4, 2, 4, 5}; // (i, j) -> xx, xy, xz, yy, yz, zz
      for (int i = 0; i < nn; i++)
        for (int c = 0; c < 9; c++)
        {
          o.num(avg[(size_t)(col[k] + full[c]) * h->nN + n0 + i]);
          o.str(c == 8 ? "\n" : " ");
        }
    }
  }
  o.str("\n");
  FILE *fp = fopen(path, "wb");
  if (!fp)
    return fail(h, DNL_ERR_ARG, "cannot open %s for writing", path);
  const size_t w = fwrite(o.s.data(), 1, o.s.size(), fp);
  const int cl = fclose(fp);
  if (w != o.s.size() || cl != 0)
    return fail(h, DNL_ERR_ARG, "writing %s failed", path);
  return DNL_OK;
}

int dnl_engine_get_ips_native(dnl_engine *h, void *out, int32_t word)
{
  if (!h || !out)
    return DNL_ERR_ARG;
  const int native = h->precision == DNL_PREC_MIXED ? 4 : 8;
  if (word != native)
    return fail(h, DNL_ERR_ARG, "the point state is kept in %d-byte words, not %d", native, word);
  const long long items = (long long)DNL_IP_NCOMP * h->nIP;
  const size_t bytes = (size_t)items * native;
  void *st = nullptr;
  int rc = staging(h, bytes, &st);
  if (rc)
    return rc;
  const unsigned blocks = (unsigned)((items + 255) / 256);
  if (native == 4)
    k_ips_out_native<float><<<blocks, 256, 0, h->stream>>>(h->M, (float *)st);
  else
    k_ips_out_native<double><<<blocks, 256, 0, h->stream>>>(h->M, (double *)st);
  CK(cudaGetLastError());
  h->launches++;
  return copy(h, out, st, bytes, cudaMemcpyDeviceToHost);
}

int dnl_engine_set_ips(dnl_engine *h, const double *in)
{
  if (!h || !in)
    return DNL_ERR_ARG;
  const size_t n = (size_t)h->nIP, total = (size_t)DNL_IP_NCOMP * h->nIPpad;
  if (h->precision == DNL_PREC_MIXED)
  {
    std::vector<float> tmp(total, 0.0f);
    for (int c = 0; c < DNL_IP_NCOMP; c++)
      for (size_t q = 0; q < n; q++)
        tmp[ip_index(c, (int)q)] = (float)in[c * n + q];
    return copy(h, h->M.ip, tmp.data(), total * sizeof(float), cudaMemcpyHostToDevice);
  }
  std::vector<double> tmp(total, 0.0);
  for (int c = 0; c < DNL_IP_NCOMP; c++)
    for (size_t q = 0; q < n; q++)
      tmp[ip_index(c, (int)q)] = in[c * n + q];
  return copy(h, h->M.ip, tmp.data(), total * sizeof(double), cudaMemcpyHostToDevice);
}

namespace
{
void free_items(dnl_engine *h)
{
  dnl_pool_free(h->itemMem, h->stream);
  h->itemMem = nullptr;
  h->ditems = nullptr;
  h->ditemOff = nullptr;
  h->dvalues = h->dkin = nullptr;
  h->nItems = 0;
  h->nValues = 0;
  h->itemsKinetic = 0;
}
} // namespace

int dnl_engine_set_items(dnl_engine *h, const dnl_item *items, int32_t n, int64_t *n_values)
{
  if (!h || n < 0 || (n > 0 && !items))
    return DNL_ERR_ARG;
  CK(cudaStreamSynchronize(h->stream));
  if (h->histOn)
  {
    // the records hold the items: a new list needs dnl_engine_set_history again
    drop_graph(h);
    h->histOn = false;
    h->histHost.clear();
  }
  free_items(h);
  std::vector<int4> it(n);
  std::vector<long long> off(n);
  long long total = 0;
  int kin = 0;
  for (int k = 0; k < n; k++)
  {
    const dnl_item &a = items[k];
    int width = 0;
    switch (a.kind)
    {
    case DNL_ITEM_NODE:
      if (a.index < 0 || a.index >= h->nN || a.field < DNL_NODE_COORDS || a.field > DNL_NODE_ACCEL_PREV)
        return fail(h, DNL_ERR_ARG, "item %d: node %d / field %d out of range", k, a.index, a.field);
      width = 3;
      break;
    case DNL_ITEM_POINT:
      if (a.index < 0 || a.index >= h->nIP)
        return fail(h, DNL_ERR_ARG, "item %d: integration point %d out of range", k, a.index);
      width = DNL_IP_NCOMP;
      break;
    case DNL_ITEM_KINETIC:
      if (a.index < 0 || a.index >= h->nInst || (a.field != DNL_NODE_SPEED && a.field != DNL_NODE_SPEED_PREV))
        return fail(h, DNL_ERR_ARG, "item %d: instance %d / speed field %d invalid", k, a.index, a.field);
      width = 1;
      kin |= a.field == DNL_NODE_SPEED ? 1 : 2;
      break;
    default:
      return fail(h, DNL_ERR_ARG, "item %d: unknown kind %d", k, a.kind);
    }
    const int idx = (a.kind == DNL_ITEM_NODE && !h->intOf.empty()) ? h->intOf[a.index] : a.index;
    it[k] = make_int4(a.kind, a.field, idx, 0);
    off[k] = total;
    total += width;
  }
  if (n > 0)
  {
    // one allocation: items, offsets, values, kinetic energies
    char *p = nullptr;
    CK(dnl_pool_alloc((void **)&p, (sizeof(int4) + sizeof(long long)) * n + sizeof(double) * (total + 6 * h->nInst),
                      h->stream));
    h->itemMem = p;
    h->ditems = (int4 *)p;
    h->ditemOff = (long long *)(h->ditems + n);
    h->dvalues = (double *)(h->ditemOff + n);
    h->dkin = h->dvalues + total;
    CK(cudaMemcpyAsync(h->ditems, it.data(), sizeof(int4) * n, cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->ditemOff, off.data(), sizeof(long long) * n, cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
  }
  h->nItems = n;
  h->nValues = total;
  h->itemsKinetic = kin;
  if (n_values)
    *n_values = total;
  return DNL_OK;
}

int dnl_engine_gather_items(dnl_engine *h, double *out)
{
  if (!h || (h->nItems > 0 && !out))
    return DNL_ERR_ARG;
  if (h->nItems == 0)
    return DNL_OK;
  int rc;
  if (h->itemsKinetic)
  {
    // energies of every instance on both speed fields: field0 then field1
    for (int f = 0; f < 2; f++)
      if ((h->itemsKinetic >> f) & 1)
        if ((rc = launch_energies(h, h->dkin + 3 * f * h->nInst, f, false, 0, h->nInst)))
          return rc;
  }
  const int threads = 128, blocks = (h->nItems + threads - 1) / threads;
  if (h->precision == DNL_PREC_MIXED)
    k_gather_items<float><<<blocks, threads, 0, h->stream>>>(h->M, h->ditems, h->ditemOff, h->nItems, h->dkin,
                                                                h->dvalues);
  else
    k_gather_items<double><<<blocks, threads, 0, h->stream>>>(h->M, h->ditems, h->ditemOff, h->nItems, h->dkin,
                                                                 h->dvalues);
  CK(cudaGetLastError());
  return copy(h, out, h->dvalues, sizeof(double) * h->nValues, cudaMemcpyDeviceToHost);
}

int dnl_engine_set_history(dnl_engine *h, const dnl_history_schedule *sched, int32_t n, int32_t capacity)
{
  if (!h || n < 0 || n > 64 || (n > 0 && !sched) || capacity < 0)
    return DNL_ERR_ARG;
  if (n > 0 && h->nInst != 1)
    return fail(h, DNL_ERR_UNSUPPORTED, "history records on the device are kept for single models");
  int rc = sync_ctl(h);
  if (rc)
    return rc;
  drop_graph(h); // the increment's graph gains or loses the history kernel
  h->histOn = false;
  h->histHost.clear();
  if (h->histMem)
  {
    dnl_pool_free(h->histMem, h->stream);
    h->histMem = nullptr;
  }
  if (n == 0)
    return DNL_OK;
  const int cap = capacity > 0 ? capacity : 64;
  const size_t width = HIST_HEAD + (size_t)h->nValues;
  // one allocation: count, overflow, last increment, the schedules, the records
  const size_t offLast = 16, offSched = 32, offRec = offSched + ((sizeof(double) * 3 * n + 255) / 256) * 256;
  const size_t bytes = offRec + sizeof(double) * width * cap;
  CK(dnl_pool_alloc(&h->histMem, bytes, h->stream));
  char *base = (char *)h->histMem;
  HistRing &H = h->hist;
  H.nSched = n;
  H.cap = cap;
  H.count = (int *)base;
  H.overflow = (int *)base + 1;
  H.last = (long long *)(base + offLast);
  H.start = (double *)(base + offSched);
  H.next = H.start + n;
  H.save = H.next + n;
  H.rec = (double *)(base + offRec);
  std::vector<double> tab(3 * (size_t)n);
  for (int j = 0; j < n; j++)
  {
    tab[j] = sched[j].start;
    tab[n + j] = sched[j].next;
    tab[2 * n + j] = sched[j].save;
  }
  const Ctl &c = h->hctl[0];
  const long long committed = c.inc - ((c.prepared && c.active) ? 1 : 0);
  CK(cudaMemsetAsync(base, 0, offSched, h->stream));
  CK(cudaMemcpyAsync(H.last, &committed, sizeof(long long), cudaMemcpyHostToDevice, h->stream));
  CK(cudaMemcpyAsync(H.start, tab.data(), sizeof(double) * 3 * n, cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->histOn = true;
  return DNL_OK;
}

int dnl_engine_history_records(dnl_engine *h, double *out, int64_t max_records, int64_t *n_records)
{
  if (!h || !n_records)
    return DNL_ERR_ARG;
  const size_t width = HIST_HEAD + (size_t)h->nValues;
  const int64_t pending = h->histOn ? (int64_t)(h->histHost.size() / width) : 0;
  if (!out)
  {
    *n_records = pending;
    return DNL_OK;
  }
  const int64_t k = std::max<int64_t>(0, std::min(pending, max_records));
  if (k > 0)
  {
    memcpy(out, h->histHost.data(), sizeof(double) * width * k);
    h->histHost.erase(h->histHost.begin(), h->histHost.begin() + (ptrdiff_t)(width * k));
  }
  *n_records = k;
  return DNL_OK;
}

int dnl_engine_energies(dnl_engine *h, int32_t i, double out[3])
{
  if (!h || !out || i < 0 || i >= h->nInst)
    return DNL_ERR_ARG;
  int rc = launch_energies(h, h->denergy, 0, true, i, 1);
  if (rc)
    return rc;
  CK(cudaMemcpyAsync(out, h->denergy, 3 * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  return DNL_OK;
}

// Element-pass autotuner: time every kernel variant over `steps` increments
// started from the same saved state, keep the fastest, and restore the state,
// so the simulation is left exactly where it was.
int dnl_engine_autotune(dnl_engine *h, int32_t steps)
{
  if (!h)
    return DNL_ERR_ARG;
  if (!h->initialized)
    return fail(h, DNL_ERR_ARG, "dnl_engine_init must be called first");
  if (steps <= 0)
    return DNL_OK;
  if (h->npe != 8) // one variant
  {
    h->forced = false;
    return DNL_OK;
  }
  const size_t rsz = h->precision == DNL_PREC_MIXED ? 4 : 8;
  const size_t ipBytes = (size_t)DNL_IP_NCOMP * h->nIPpad * rsz, nb = sizeof(double4) * h->nN;
  struct Saved
  {
    void *dst;
    const void *src;
    size_t bytes;
  };
  std::vector<Saved> parts = {{nullptr, h->M.ip, ipBytes},      {nullptr, h->M.x, nb},      {nullptr, h->M.disp, nb},
                              {nullptr, h->M.u[0], nb},        {nullptr, h->M.u[1], nb},   {nullptr, h->M.v[0], nb},
                              {nullptr, h->M.v[1], nb},        {nullptr, h->M.a[0], nb},   {nullptr, h->M.a[1], nb},
                              {nullptr, h->M.ctl, sizeof(Ctl) * h->nInst}};
  size_t total = 0;
  for (auto &p : parts)
    total += (p.bytes + 255) / 256 * 256;
  char *save = nullptr;
  if (dnl_pool_alloc((void **)&save, total, h->stream) != cudaSuccess)
    return fail(h, DNL_ERR_CUDA, "autotune: no room for the state snapshot (%zu bytes)", total);
  size_t off = 0;
  for (auto &p : parts)
  {
    p.dst = save + off;
    off += (p.bytes + 255) / 256 * 256;
    CK(cudaMemcpyAsync(p.dst, p.src, p.bytes, cudaMemcpyDeviceToDevice, h->stream));
  }
  cudaEvent_t e0, e1;
  CK(cudaEventCreate(&e0));
  CK(cudaEventCreate(&e1));
  const int before = h->variant;
  int best = before, rc = DNL_OK;
  double bestMs = 1e30;
  for (int v = 0; v < kNumVariants && !rc; v++)
  {
    if (h->nInst > 1 && (variant_of(h, v).tma == 0 || (v == 0 && h->precision == DNL_PREC_FP64)))
    {
      // plain variants are not offered to batches (see create), nor FP64's variant 0,
      // which is variant 1's kernel there
      h->variantMs[v] = -1.0;
      continue;
    }
    for (auto &p : parts)
      CK(cudaMemcpyAsync(const_cast<void *>(p.src), p.dst, p.bytes, cudaMemcpyDeviceToDevice, h->stream));
    h->variant = v;
    rc = launch_control(h, CTL_LIMITS, 1e300, steps);
    double ms = 0.0;
    for (int k = 0; k < steps && !rc; k++)
    {
      if ((rc = launch_bc_prep(h)))
        break;
      CK(cudaEventRecord(e0, h->stream));
      if ((rc = launch_element_any(h, 0)))
        break;
      CK(cudaEventRecord(e1, h->stream));
      if ((rc = launch_nodal(h)) || (rc = launch_step_end(h)))
        break;
      CK(cudaEventSynchronize(e1));
      float t = 0;
      cudaEventElapsedTime(&t, e0, e1);
      if (k > 0 || steps == 1)
        ms += t;
    }
    CK(cudaStreamSynchronize(h->stream));
    if (rc)
      break;
    CK(cudaGetLastError());
    ms /= (steps > 1 ? steps - 1 : 1);
    h->variantMs[v] = ms;
    if (ms < bestMs)
    {
      bestMs = ms;
      best = v;
    }
  }
  // Mixed single models: a variant by size when it is within 10 % of the fastest
  // trial.  The builds of 48 and 64 registers contract a multiply and an add
  // here and there that the others do not, which changes a last bit at a few
  // points in 10^5 and, through the halving exits of the return at first yield,
  // the plastic strain rate of single points by percents some hundred
  // increments later; a model's results should not depend on which of two
  // variants a few per cent apart won a trial of microseconds.  Below 16,000
  // hexahedra the pass of 80 registers (once/6), from there to 180,000 the plain
  // one of 48, because tuned models of these sizes have run so and keep their
  // results; above the fastest, which is once/6 (plate of 491,520: 206 against
  // 213 for the staged pass and 216 for the plain one).  What the rule costs, or
  // gives: us an increment over increments 100 to 600 of a bar, once/6 and
  // plain/10: 10,150 hexahedra 15.1 and 14.6, 14,025 15.9 and 16.6, 20,916 19.5
  // and 19.5, 45,760 30.7 and 30.9, 109,340 61.7 and 62.1, 153,600 83.4 and 84.2,
  // 226,800 124.8 and 126.2; in the first increments, where the trials are, once/6
  // is 3 to 6 % ahead on 39,900 to 153,600.  A batch is offered variants of one
  // arithmetic only and takes the fastest.
  if (h->nInst == 1 && h->precision == DNL_PREC_MIXED && h->nE < 180000)
  {
    const int prefer = h->nE < 16000 ? 0 : 10;
    if (h->variantMs[prefer] > 0.0 && h->variantMs[prefer] <= 1.1 * bestMs)
      best = prefer;
  }
  for (auto &p : parts)
    CK(cudaMemcpyAsync(const_cast<void *>(p.src), p.dst, p.bytes, cudaMemcpyDeviceToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  dnl_pool_free(save, h->stream);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  h->variant = rc ? before : best;
  if (rc)
    return rc;
  h->tuned = true;
  h->forced = false; // the engine's own choice again, cooperative increments among it
  drop_graph(h);
  return check_status(h);
}

int dnl_engine_variant(const dnl_engine *h, int32_t *variant, double ms[DNL_NUM_VARIANTS])
{
  if (!h)
    return DNL_ERR_ARG;
  if (variant)
    *variant = h->variant;
  if (ms)
    for (int v = 0; v < kNumVariants; v++)
      ms[v] = h->variantMs[v];
  return DNL_OK;
}

const char *dnl_variant_name(int32_t precision, int32_t variant)
{
  if (variant < 0 || variant >= kNumVariants || (precision != DNL_PREC_FP64 && precision != DNL_PREC_MIXED))
    return nullptr;
  return precision == DNL_PREC_MIXED ? kVariantsF32[variant].name : kVariantsF64[variant].name;
}

int dnl_engine_set_variant(dnl_engine *h, int32_t variant)
{
  if (!h || variant < 0 || variant >= kNumVariants)
    return DNL_ERR_ARG;
  h->variant = variant;
  h->forced = true;
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_set_timing(dnl_engine *h, int32_t on)
{
  if (!h)
    return DNL_ERR_ARG;
  h->timing = on != 0;
  return DNL_OK;
}

int dnl_engine_timings(const dnl_engine *h, double out[4])
{
  if (!h || !out)
    return DNL_ERR_ARG;
  for (int k = 0; k < 4; k++)
    out[k] = h->times[k];
  return DNL_OK;
}

int64_t dnl_engine_launch_count(const dnl_engine *h) { return h ? h->launches : 0; }

int dnl_engine_set_graph_increments(dnl_engine *h, int32_t n)
{
  if (!h || n < 1 || n > 64)
    return DNL_ERR_ARG;
  h->graphIncs = n;
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_set_mode(dnl_engine *h, int32_t mode)
{
  if (!h || mode < DNL_MODE_PLAIN || mode > DNL_MODE_GUESS)
    return DNL_ERR_ARG;
  if (mode != DNL_MODE_PLAIN && h->precision != DNL_PREC_MIXED)
    return fail(h, DNL_ERR_UNSUPPORTED, "element-pass modes run on the mixed-precision path");
  if (mode == DNL_MODE_GUESS && !h->mlpImage)
    return fail(h, DNL_ERR_ARG, "no guess network: call dnl_engine_set_guess_network first");
  if (mode == DNL_MODE_HARVEST && !h->M.harvest)
    return fail(h, DNL_ERR_ARG, "no harvest buffer: call dnl_engine_set_harvest first");
  h->mode = mode;
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_set_guess_network(dnl_engine *h, const dnl_mlp *net)
{
  if (!h || !net)
    return DNL_ERR_ARG;
  std::vector<unsigned char> img(mlp::IMAGE_BYTES);
  mlp::build_image(*net, img.data());
  if (!h->mlpImage)
  {
    int rc = dalloc(h, reinterpret_cast<unsigned char **>(&h->mlpImage), mlp::IMAGE_BYTES);
    if (rc)
      return rc;
  }
  CK(cudaMemcpyAsync(h->mlpImage, img.data(), mlp::IMAGE_BYTES, cudaMemcpyHostToDevice, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  h->M.mlp_image = h->mlpImage;
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_set_harvest(dnl_engine *h, float *d_pairs, int64_t capacity, int32_t stride)
{
  if (!h || (!d_pairs && capacity > 0) || capacity < 0 || stride < 1)
    return DNL_ERR_ARG;
  h->M.harvest = d_pairs;
  h->M.harvest_cap = capacity;
  h->M.harvest_stride = stride;
  CK(cudaMemsetAsync(h->dstats + 4, 0, sizeof(unsigned long long), h->stream));
  CK(cudaStreamSynchronize(h->stream));
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_harvest_count(dnl_engine *h, int64_t *count)
{
  if (!h || !count)
    return DNL_ERR_ARG;
  unsigned long long n = 0;
  CK(cudaMemcpyAsync(&n, h->dstats + 4, sizeof(n), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  *count = (int64_t)n;
  return DNL_OK;
}

int dnl_engine_set_guess_scope(dnl_engine *h, int32_t scope)
{
  if (!h || (scope != DNL_GUESS_ALL && scope != DNL_GUESS_FIRST_YIELD))
    return DNL_ERR_ARG;
  h->M.guess_scope = scope;
  drop_graph(h);
  return DNL_OK;
}

int dnl_engine_newton_stats(dnl_engine *h, int64_t out[4], int32_t reset)
{
  if (!h || !out)
    return DNL_ERR_ARG;
  unsigned long long v[4];
  CK(cudaMemcpyAsync(v, h->dstats, sizeof(v), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  for (int k = 0; k < 4; k++)
    out[k] = (int64_t)v[k];
  if (reset)
  {
    CK(cudaMemsetAsync(h->dstats, 0, sizeof(v), h->stream));
    CK(cudaStreamSynchronize(h->stream));
  }
  return DNL_OK;
}

} // extern "C"
