// dnl_steps.cuh - many increments of a single model in one cooperative launch.
//
// A small model's increment is a chain of latencies: three dependent kernels of
// a few microseconds each, of which the launch, the first loads of the control
// block and the drain of every grid are a good part.  Here the blocks stay
// resident and go from phase to phase through a grid barrier:
//
//   [imposed-speed nodes | barrier]
//   element phase  | barrier |  nodal phase  | barrier |
//   [time step when due: minima | barrier]  end of the increment, next one begun
//
// Every block holds its own copy of the control block in shared memory and
// advances it with the same arithmetic (finish_increment), so that no phase
// waits for a control block to be written and read back.
#pragma once

#include "dnl_kernels.cuh"

namespace dnl
{
// A build of k_steps: the kernel, its dynamic shared memory and the blocks per
// SM of its register budget.  The builds are translation units of their own
// (steps.cu): the first kernel that a process uses of a unit loads all of the
// unit's code.  A process's first engine, with all kernels in one unit, with
// two units of builds apart, with eight: 153,600 hexahedra, which use none of
// them, 55, 26, 26 ms; 800 quads 44 (two), 34 (eight).
struct StepsBuild
{
  const void *kernel = nullptr;
  size_t smem = 0;
  int minb = 0;
};
// the fewest blocks (most registers) first
constexpr int STEPS_BUDGETS = 2;
template <typename R, int NPE, bool PI> StepsBuild steps_build(bool one, int budget);
template <> StepsBuild steps_build<float, 4, false>(bool, int);
template <> StepsBuild steps_build<float, 4, true>(bool, int);
template <> StepsBuild steps_build<float, 8, false>(bool, int);
template <> StepsBuild steps_build<float, 8, true>(bool, int);
template <> StepsBuild steps_build<double, 4, false>(bool, int);
template <> StepsBuild steps_build<double, 4, true>(bool, int);
template <> StepsBuild steps_build<double, 8, false>(bool, int);
template <> StepsBuild steps_build<double, 8, true>(bool, int);
} // namespace dnl

namespace dnl
{
namespace
{

struct StepsArgs
{
  int nIncs;                // increments of this launch at most
  unsigned *bar;            // arrivals at the grid barrier, zero at launch
  int *err;
  unsigned long long *pimax; // [3] power iteration: max |v| of an iteration, zero at launch (double bits)
  unsigned long long *phase; // [3] ns spent in the element, nodal and time-step phases, or nullptr
  // history records (dnl_engine_set_history), histOn = 0: none
  int histOn, nItems, nValues, kin;
  HistRing hist;
  const int4 *items;
  const long long *off;
};

// Barrier of all the blocks of a cooperative launch: one arrival per block on
// a counter that only grows, and one polling thread per block.  The wait is
// bounded (about two seconds of SM clock); false when it gave up.
struct GridBarrier
{
  unsigned *count;
  unsigned target;
  int *err;
  int *gaveUp; // shared memory
  __device__ __forceinline__ bool sync()
  {
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0)
    {
      // release: the block's writes (ordered before by the block barrier) are visible to who sees the arrival
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
      const long long start = clock64();
      for (;;)
      {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
        if (v >= target)
          break;
        if (clock64() - start > (1ll << 32))
        {
          atomicExch(err, 1);
          *gaveUp = 1;
          break;
        }
      }
    }
    __syncthreads();
    return *gaveUp == 0;
  }
};

__device__ __forceinline__ unsigned long long global_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// I/O of a block whose tile's point state stays in shared memory over the
// increments of the launch (laid out as in global memory: run ip_slot(c) of
// TILE values).  When a Courant time step is due the densities go to global
// memory as well, where its pass reads them (the power iteration reads none).
template <typename R, bool ONE> struct ResidentIo
{
  using R4 = typename V4<R>::type;
  const DevModel &M;
  R *st;
  int t, q, f0, spos;
  bool density; // to global memory as well
  __device__ __forceinline__ double4 x(int n) const { return M.x[n]; }
  __device__ __forceinline__ double4 u(int n) const { return M.u[f0][n]; }
  __device__ __forceinline__ const MatDev &mat(int e) const { return M.mat[M.emat[e]]; }
  __device__ __forceinline__ const MatDev *matp(int e) const { return M.mat + M.emat[e]; }
  __device__ __forceinline__ JC<R, ONE> law(int e) const
  {
    JC<R, ONE> j;
    if constexpr (ONE)
      j.q = one_params<R>(M);
    else
      j.load(mat(e));
    return j;
  }
  __device__ __forceinline__ double rho0(int e) const
  {
    if constexpr (ONE)
      return M.one_rho0;
    else
      return mat(e).rho0;
  }
  __device__ __forceinline__ void put(int c, R v) const
  {
    st[ip_slot(c) * TILE + t] = v;
    if (c == DNL_IP_DENSITY && density)
      ipw<R>(M, c, q, v);
  }
  __device__ __forceinline__ void slot(const R4 &v) const { reinterpret_cast<R4 *>(M.slot)[spos] = v; }
  __device__ __forceinline__ const float *ip32() const { return reinterpret_cast<const float *>(st); }
  __device__ __forceinline__ int ip32_index() const { return t; }
  __device__ __forceinline__ void first_node(unsigned amask, int base, const double4 &X, const double4 &U,
                                             double4 &X0, double4 &U0) const
  {
    first_node_by_shuffle(amask, base, X, U, X0, U0);
  }
};

template <typename R, int NPE, bool PI> struct StepsLayout
{
  static constexpr uint32_t PASS_BYTES = TILE * ElemShape<NPE>::template pass_row<R> * sizeof(R);
  // the power iteration's transpose takes the same rows
  static constexpr int KV_ROW = NPE == 8 ? 25 : 9;
  static constexpr uint32_t KV_BYTES = PI ? TILE * KV_ROW * sizeof(double) : 0;
  static constexpr uint32_t ROW_BYTES = PASS_BYTES > KV_BYTES ? PASS_BYTES : KV_BYTES;
  static constexpr uint32_t STATE_BYTES = DNL_IP_NCOMP * TILE * sizeof(R);
  static_assert(ROW_BYTES % 16 == 0, "the state after the rows is 16-byte aligned");
};

// State of the power iteration between the time steps of a launch: iterations
// so far, which buffer holds the vector (M.pv or M.pv2), and the factor that
// normalises it.
struct PowerState
{
  unsigned it;
  int odd;
  double scale;
};

// k_power_iteration (same sums, same tests) inside the launch: per iteration an
// element phase and a node phase with a grid barrier after each; the largest
// |v| of an iteration collects in one of three words, of which the first block
// clears the next while no block reads it (k_power_iteration has every thread
// read a word per block).  800 axisymmetric quads with the time step at every
// increment, per increment, its own launch -> here: 35 -> 19 us (FP64), 24 ->
// 14 (mixed).  False when a barrier gave up.
template <typename R, int NPE>
__device__ __forceinline__ bool power_iteration(const DevModel &M, const StepsArgs &A, Ctl &c, GridBarrier &bar,
                                                PowerState &pi, double *rows, int t, int node, int spos)
{
  constexpr int DIM = ElemShape<NPE>::DIM, ROW = StepsLayout<R, NPE, true>::KV_ROW;
  const int lane = t & 31, g = t & (NPE - 1), base = lane & ~(NPE - 1);
  const int e = (blockIdx.x * TILE + t) / NPE;
  const bool act = e < M.nE;
  const unsigned amask = __ballot_sync(0xffffffffu, act);
  double fprev = c.pi_fmax, fmx = 0.0;
  for (int it = 1;; it++, pi.it++)
  {
    const double *v = pi.odd ? M.pv2 : M.pv;
    double *vn = pi.odd ? M.pv : M.pv2;
    if (act)
    {
      __syncwarp(amask); // the rows of the iteration before have been read
      M.pislot[spos] = element_Kv<NPE, ROW>(M, node, e, g, base, amask, c.plane != 0, v, pi.scale, rows + t * ROW,
                                            rows + (t - g) * ROW);
    }
    if (blockIdx.x == 0 && t == 0)
      A.pimax[(pi.it + 1) % 3] = 0ull;
    if (!bar.sync())
      return false;
    double lmax = 0.0;
    for (int k = blockIdx.x * TILE + t; k < 3 * M.nN; k += gridDim.x * TILE)
    {
      const int i = k / 3, cc = k % 3;
      double val = 0.0;
      if (cc < DIM)
      {
        const double *sl = reinterpret_cast<const double *>(M.pislot) + cc;
        const int kb = slot_begin(M, i), n = M.csr_off[i + 1] - M.csr_off[i];
        double acc = v[k] * pi.scale;
        for (int j0 = 0; j0 < n; j0 += NPE)
        {
          double y[NPE];
#pragma unroll
          for (int j = 0; j < NPE; j++)
            y[j] = j0 + j < n ? sl[4 * (size_t)(kb + j0 + j)] : 0.0;
#pragma unroll
          for (int j = 0; j < NPE; j++)
            if (j0 + j < n)
              acc += y[j];
        }
        val = acc / M.mass[i];
      }
      vn[k] = val;
      lmax = fmax(lmax, fabs(val));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
      lmax = fmax(lmax, __shfl_xor_sync(0xffffffffu, lmax, off));
    if (lane == 0)
      atomicMax(&A.pimax[pi.it % 3], (unsigned long long)__double_as_longlong(lmax));
    if (!bar.sync())
      return false;
    fmx = __longlong_as_double((long long)*(volatile unsigned long long *)&A.pimax[pi.it % 3]);
    const bool conv = fabs(fmx - fprev) / fmx < 1e-4;
    fprev = fmx;
    pi.scale = 1.0 / fmx;
    pi.odd ^= 1;
    if (conv || it > 1000)
    {
      pi.it++;
      if (t == 0)
      {
        if (conv)
        {
          c.pi_fmax = fmx;
          c.pi_omega = sqrt(fmx);
          c.pi_iters += it;
        }
        else
        {
          c.status = DNL_ERR_POWER_ITERATION;
          if (blockIdx.x == 0)
            raise_status(M.ctl, DNL_ERR_POWER_ITERATION, it);
        }
      }
      return true;
    }
  }
}

// One tile per block, its point state in shared memory from the first
// increment of the launch to the last.  Bound by latencies: in FP64 the element
// phase, 7.0 (800 quads) to 10.5 us (6,720 hexahedra) of an increment, most of it
// the return's serial chain (eval64); the nodal phase is 2.5 to 3.6 us, the time
// step and the end of the increment 0.8 to 1.1 on average, a barrier with the
// loads after it about 1 in each.  Per increment on the B200, increments 300 to
// 1,300 of an impact, kernel by kernel in graph replays -> here: 800 axisymmetric
// quads 14.4 -> 11.2 us (FP64) and 10.7 -> 7.3 (mixed), 7,747 plane quads 15.6 ->
// 12.7 and 11.0 -> 8.1, 6,048 hexahedra 18.0 -> 15.0 and 12.2 -> 9.6, 6,720 18.6 ->
// 15.4 (FP64), 8,960 13.1 -> 11.4 (mixed).
template <typename R, int NPE, int MINB, bool ONE, bool PI>
__global__ void __launch_bounds__(TILE, MINB) k_steps(DevModel M, StepsArgs A)
{
  constexpr int ROW = ElemShape<NPE>::template pass_row<R>;
  constexpr int DIM = ElemShape<NPE>::DIM;
  using L = StepsLayout<R, NPE, PI>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R *rows = reinterpret_cast<R *>(smem_raw);
  R *st = reinterpret_cast<R *>(smem_raw + L::ROW_BYTES);
  __shared__ Ctl c; // this block's control values
  __shared__ int gaveUp, hslot, hdue;
  __shared__ long long hlast;
  __shared__ double hsched[3][64], red[8 * KIN_GROUPS];
  const int t = threadIdx.x, lane = t & 31;
  if (t == 0)
  {
    c = *M.ctl;
    gaveUp = 0;
    if (A.histOn)
      hlast = *A.hist.last;
  }
  if (A.histOn)
    for (int j = t; j < A.hist.nSched; j += TILE)
    {
      hsched[0][j] = A.hist.start[j];
      hsched[1][j] = A.hist.next[j];
      hsched[2][j] = A.hist.save[j];
    }
  const int node = M.conn[blockIdx.x * TILE + t], spos = M.slot_pos[blockIdx.x * TILE + t];
  constexpr int NVEC = DNL_IP_NCOMP * TILE * sizeof(R) / sizeof(float4);
  float4 *tile = reinterpret_cast<float4 *>(reinterpret_cast<R *>(M.ip) + (size_t)blockIdx.x * DNL_IP_NCOMP * TILE);
  auto state_out = [&]() {
    for (int k = t; k < NVEC; k += TILE)
      tile[k] = reinterpret_cast<const float4 *>(st)[k];
  };
  for (int k = t; k < NVEC; k += TILE)
    reinterpret_cast<float4 *>(st)[k] = tile[k];
  __syncthreads();
  GridBarrier bar{A.bar, 0u, A.err, &gaveUp};
  const bool stamp = A.phase && blockIdx.x == 0 && t == 0;
  unsigned long long ns[3] = {0, 0, 0}, t0 = 0, t1 = 0;
  bool ok = true, reset_min = false;
  PowerState pi{0, 0, 1.0};
  int done = 0;
  for (; done < A.nIncs && c.active && ok; done++)
  {
    const bool due = c.due != 0; // the block's first thread rewrites c at the end of the increment
    if (M.nSpeed)
    {
      for (int k = blockIdx.x * TILE + t; k < M.nSpeed; k += gridDim.x * TILE)
        bc_prep_node(M, M.speed_nodes[k], &c);
      if (!(ok = bar.sync()))
        break;
    }
    if (stamp)
      t0 = global_ns();
    // ---- element phase.  The thread index passes through a register the
    // compiler knows nothing of, so that it does not keep what follows from it
    // (addresses, the signs of the shape functions) in registers over the whole
    // loop, where the nodal phase and the return have no room for them.
    int te = t;
    asm volatile("" : "+r"(te));
    const int g = te & (NPE - 1), base = te & 31 & ~(NPE - 1);
    const int q = blockIdx.x * TILE + te, e = q / NPE;
    const bool act = e < M.nE;
    const unsigned amask = __ballot_sync(0xffffffffu, act);
    if (act)
    {
      SharedTile<R> old{st, te};
      ResidentIo<R, ONE> io{M, st, te, q, c.f0, spos, !PI && due};
      element_update<R, NPE>(io, &c, M.ctl, q, e, g, base, amask, node, old, rows + te * ROW, rows + (te - g) * ROW);
    }
    if (!(ok = bar.sync()))
      break;
    if (stamp)
    {
      t1 = global_ns();
      ns[0] += t1 - t0;
    }
    // ---- nodal phase (and the status that the element phase may have raised)
    int status = 0;
    if (t == 0)
    {
      status = *(volatile int *)&M.ctl->status;
      if (reset_min && blockIdx.x == 0) // every block has read the last minimum
        *(volatile unsigned long long *)&M.ctl->min_bits = INF_BITS;
    }
    reset_min = false;
    for (int k = blockIdx.x * TILE + te; k < 3 * M.nN; k += gridDim.x * TILE)
      nodal_update<R, DIM>(M, k / 3, k % 3, &c);
    if (!(ok = bar.sync()))
      break;
    if (stamp)
    {
      t0 = global_ns();
      ns[1] += t0 - t1;
    }
    // ---- time step when due, end of the increment
    if constexpr (PI)
    {
      if (due)
      {
        if (!(ok = power_iteration<R, NPE>(M, A, c, bar, pi, reinterpret_cast<double *>(rows), te, node, spos)))
          break;
        if (t == 0 && c.status)
          status = c.status;
      }
    }
    else if (due)
    {
      const int nE32 = (M.nE + 31) & ~31;
      for (int e = blockIdx.x * TILE + t; e < nE32; e += gridDim.x * TILE)
        courant_warp<R, NPE>(M, e < M.nE ? e : M.nE - 1, lane, 0, e < M.nE, M.ctl);
      if (!(ok = bar.sync()))
        break;
      if (t == 0)
        c.min_bits = *(volatile unsigned long long *)&M.ctl->min_bits;
      reset_min = true;
    }
    if (t == 0)
    {
      c.status = status;
      finish_increment(c);
      hdue = 0;
      if (A.histOn)
      {
        const long long committed = c.inc - ((c.prepared && c.active) ? 1 : 0);
        if (committed != hlast)
        {
          hlast = committed;
          const unsigned long long mask = history_due(A.hist.nSched, c.t, hsched[0], hsched[1], hsched[2]);
          if (mask)
          {
            hdue = 1;
            hslot = blockIdx.x == 0 ? history_slot(A.hist, c, committed, mask, A.nValues) : -1;
          }
        }
      }
    }
    __syncthreads();
    if (hdue)
    {
      // a record: the point state where the first block reads it.  No block
      // goes on before the first has read the items: what follows changes them
      // ahead of its next barrier (the imposed-speed nodes' u, v and a by
      // bc_prep_node, the densities by the element phase when the time step is
      // due).
      state_out();
      if (!(ok = bar.sync()))
        break;
      if (blockIdx.x == 0 && hslot >= 0)
        history_items<R, TILE>(M, c, A.items, A.off, A.nItems, A.kin,
                               A.hist.rec + (size_t)hslot * (HIST_HEAD + A.nValues) + HIST_HEAD, red);
      if (!(ok = bar.sync()))
        break;
    }
    if (stamp)
      ns[2] += global_ns() - t0;
  }
  if (done)
    state_out();
  if (reset_min)
    bar.sync(); // every block has read the last minimum
  if constexpr (PI)
    if (pi.it)
    {
      // the normalised vector for the next launch (M.pv), by the threads that wrote it
      const double *v = pi.odd ? M.pv2 : M.pv;
      for (int k = blockIdx.x * TILE + t; k < 3 * M.nN; k += gridDim.x * TILE)
        M.pv[k] = v[k] * pi.scale;
    }
  if (blockIdx.x == 0 && t == 0 && done)
  {
    Ctl &G = *M.ctl; // status, bad and resolves are the global block's own
    G.t = c.t;
    G.dt = c.dt;
    G.dt_eff = c.dt_eff;
    G.t_new = c.t_new;
    G.inc = c.inc;
    G.active = c.active;
    G.prepared = c.prepared;
    G.due = c.due;
    G.f0 = c.f0;
    G.dt_last = c.dt_last;
    if (reset_min)
      G.min_bits = INF_BITS;
    G.pi_fmax = c.pi_fmax;
    G.pi_omega = c.pi_omega;
    G.pi_iters = c.pi_iters;
    if (A.histOn)
    {
      *A.hist.last = hlast;
      for (int j = 0; j < A.hist.nSched; j++)
        A.hist.next[j] = hsched[1][j];
    }
    if (stamp)
      for (int k = 0; k < 3; k++)
        A.phase[k] += ns[k];
  }
}

// A build of k_steps by register budget.
template <typename R, int NPE, bool ONE, bool PI, int MINB> StepsBuild steps_build_one()
{
  using L = StepsLayout<R, NPE, PI>;
  return {(const void *)k_steps<R, NPE, MINB, ONE, PI>, L::ROW_BYTES + L::STATE_BYTES, MINB};
}
template <typename R, int NPE, bool ONE, bool PI> StepsBuild steps_build_budget(int budget)
{
  // FP64: 255 and 168 registers a thread, FP32: 168 and 128 (no spill, a little)
  constexpr int B = sizeof(R) == 4 ? 3 : 2;
  return budget == 0 ? steps_build_one<R, NPE, ONE, PI, B>() : steps_build_one<R, NPE, ONE, PI, B + 1>();
}

} // namespace
} // namespace dnl
