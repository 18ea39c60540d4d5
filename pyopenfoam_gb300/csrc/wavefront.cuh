// Level-scheduled wavefronts in one cooperative launch.
//
// The DIC / DILU factorisations, the apply_full sweeps and the Gauss-Seidel
// sweeps visit the items (cells or faces) of a level schedule level by
// level; items of one level are independent, a level reads what earlier
// levels wrote.  Launching one kernel per level costs a launch and a drain
// per level (767 levels for DIC at 256^3).  Here all blocks are resident
// (cudaLaunchCooperativeKernel) and walk the levels together, separated by
// the bounded software grid barrier of barrier.cuh; values written by other
// blocks are read through L2 (__ldcg) by the item bodies.
//
// A barrier wait that runs out sets the barrier's fault word; every block
// that sees it overwrites the whole output with NaN (an invalid result is
// then visible downstream) and returns.  The host can read the fault word
// with gbf_wavefront_fault.
#pragma once

#include "barrier.cuh"

namespace gbf {

// body(i) for every item i of every level, in level order.  Returns false if
// a barrier wait ran out.
template <typename F>
__device__ __forceinline__ bool run_levels(GridBarrier* bar, const int32_t* __restrict__ level_ptr,
                                           int n_levels, F&& body,
                                           long long max_polls = kBarrierPolls) {
  const int stride = gridDim.x * blockDim.x;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  for (int lv = 0; lv < n_levels; ++lv) {
    const int start = __ldg(level_ptr + lv), end = __ldg(level_ptr + lv + 1);
    for (int i = start + tid; i < end; i += stride) body(i);
    if (lv + 1 < n_levels && !grid_barrier(bar, gridDim.x, max_polls)) return false;
  }
  return true;
}

// Every block that observed a barrier fault writes NaN over out[0, n).
__device__ __forceinline__ void poison(double* out, int n) {
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  for (int i = threadIdx.x; i < n; i += blockDim.x) out[i] = nan;
}

// Blocks of a cooperative wavefront launch: resident blocks of `kernel`,
// no more than needed for the largest level and at most `per_sm_max` per SM
// (fewer blocks make a cheaper barrier, more hide more latency of the
// items' dependent loads; a level larger than the grid is looped over).
// Measured on GB300: the Gauss-Seidel cell levels are fastest with two
// blocks per SM, the many small face levels (DILU, sweeps) with one.
// 0 when the device cannot launch cooperatively.
inline int wavefront_grid(const void* kernel, int block, long long max_level_items,
                          int per_sm_max) {
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!coop || sms <= 0) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) != cudaSuccess ||
      per_sm <= 0)
    return 0;
  long long g = (long long)(per_sm < per_sm_max ? per_sm : per_sm_max) * sms;
  const long long need = (max_level_items + block - 1) / block;
  if (g > need) g = need;
  return g < 1 ? 1 : (int)g;
}

// Zeroes the caller's barrier memory (gbf_wavefront_barrier_bytes) and
// launches `kernel` cooperatively on `grid` blocks of kBlock threads.
inline cudaError_t launch_wavefront(const void* kernel, int grid, void** args, void* barrier,
                                    cudaStream_t s) {
  static_assert(sizeof(GridBarrier) <= 64, "gbf_wavefront_barrier_bytes");
  cudaError_t e = cudaMemsetAsync(barrier, 0, sizeof(GridBarrier), s);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kBlock), args, 0, s);
}

// ---- dataflow walks (no barrier between levels) -----------------------------
//
// A step's inputs sit in slots of device memory that hold the empty marker
// until their producer stores them; a step polls only the slots it reads.
// The empty marker is the all-ones bit pattern (a NaN); a NaN result is
// stored as the canonical NaN so that it cannot read as empty.  Every wait
// is bounded: after max_polls passes a warp sets the barrier's fault word
// and returns, and the warps that see the fault word return too; the
// output kernel then writes NaN everywhere.
constexpr long long kFlowEmpty = -1LL;
constexpr long long kFlowPolls = 1LL << 22;  // passes of a warp, a trip through L2 each: > 3 s

__device__ __forceinline__ double ld_flow(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}

// v, a NaN as the canonical one (compared as integers: an FP64 instruction,
// a compare too, holds the warp for 64 clocks on GB300).
__device__ __forceinline__ double flow_value(double v) {
  const long long b = __double_as_longlong(v) & 0x7fffffffffffffffLL;
  return b > 0x7ff0000000000000LL ? __longlong_as_double(0x7ff8000000000000LL) : v;
}

__device__ __forceinline__ void st_flow(double* p, double v) {
  v = flow_value(v);
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v) : "memory");
}

__device__ __forceinline__ bool flow_empty(double v) {
  return __double_as_longlong(v) == kFlowEmpty;
}

// ---- block walks -------------------------------------------------------------
//
// A dataflow walk whose block b takes the cells [b per, (b+1) per) and keeps
// their slots in shared memory as well: a step whose inputs come from cells of
// its own block polls those (30 clocks) instead of a store's and a load's trip
// through L2 (together some 1500).  With cells numbered so that neighbours are
// mostly close -- any mesh numbering used in earnest -- most links of the chain
// from level to level stay inside a block.  Each block's items are in level
// order, 32 at a time round-robin to its warps; the warp holding the globally
// earliest unfinished item finds its inputs, as in the walk over the whole
// schedule: its block has begun every chunk before that one, and they are done.
constexpr int kWalkCellsMax = 24576;  // cells per block: 192 KB of slots

// The slots of one walk, as one block sees them.
template <bool LOCAL>
struct FlowSlots {
  double* g;       // all slots, in device memory
  double* own;     // this block's, in shared memory
  int c0, count;   // its cells

  // Where c's value is polled: a generic address, so that a warp's polls of
  // both kinds are one load instruction without a branch.
  __device__ __forceinline__ const double* at(int c) const {
    return LOCAL && (unsigned)(c - c0) < (unsigned)count ? own + (c - c0) : g + c;
  }
  static __device__ __forceinline__ double load(const double* p) {
    double v;
    asm volatile("ld.relaxed.gpu.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
  }
  // c is one of this block's cells when LOCAL
  __device__ __forceinline__ void store(int c, double v) const {
    v = flow_value(v);
    if (LOCAL) asm volatile("st.relaxed.gpu.f64 [%0], %1;" ::"l"(own + (c - c0)), "d"(v) : "memory");
    asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(g + c), "d"(v) : "memory");
  }
};

// Passes of a warp in a block walk over n cells.  A pass that polls shared
// memory alone takes some 165 ns, and the last block waits for all others: a
// chain of n cells, one a level, takes 728 ns a cell in the DIC walk and 884 in
// the Gauss-Seidel walk, some five passes.  Six times that, and a second for any
// system (kFlowPolls ran out on chains of about a million cells).  A bound in
// clocks, looked at every 64th pass, made the Gauss-Seidel sweep of 67x59x53
// cells 335 us instead of 305.
inline long long walk_polls(int n) { return (1LL << 23) + 32LL * n; }

// The items a warp takes: 32 at `first`, `stride` further on, up to `end`.
struct FlowRange {
  long long first, end, stride;
};

// Sets up a walk over `n` items (LOCAL: those of item_ptr[block] on, cells of
// `per` a block, with `dyn` the block's shared memory).
template <bool LOCAL>
__device__ __forceinline__ FlowRange flow_begin(FlowSlots<LOCAL>& slots, double* g, int n,
                                                const int32_t* __restrict__ item_ptr, int per,
                                                double* dyn) {
  slots.g = g;
  const int warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (!LOCAL)
    return FlowRange{32LL * (blockIdx.x * warps + warp), n, 32LL * gridDim.x * warps};
  slots.c0 = blockIdx.x * per;
  slots.count = n - slots.c0 < per ? n - slots.c0 : per;
  slots.own = dyn;
  for (int i = threadIdx.x; i < slots.count; i += blockDim.x)
    dyn[i] = __longlong_as_double(kFlowEmpty);
  __syncthreads();
  const long long b = __ldg(item_ptr + blockIdx.x);
  return FlowRange{b + 32 * warp, __ldg(item_ptr + blockIdx.x + 1), 32LL * warps};
}

// Launches a block walk: `n_blocks` resident blocks with `per` slots each.
inline cudaError_t launch_walk(const void* kernel, int n_blocks, int per, void** args,
                               void* barrier, cudaStream_t s) {
  const size_t dyn = sizeof(double) * (size_t)per;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(double) * kWalkCellsMax));
  if (e == cudaSuccess) e = cudaMemsetAsync(barrier, 0, sizeof(GridBarrier), s);
  if (e != cudaSuccess) return e;
  return cudaLaunchCooperativeKernel(kernel, dim3(n_blocks), dim3(kBlock), args, dyn, s);
}

// End of one pass over a chunk: true when every lane is done; false with
// *quit set when a wait ran out here or elsewhere.  SLEEP: whether the pass
// pauses (a walk that polls shared memory does not).
template <bool SLEEP = true>
__device__ __forceinline__ bool flow_pass_end(bool done, long long& polls, long long max_polls,
                                              GridBarrier* bar, bool* quit) {
  if (__all_sync(0xffffffffu, done)) return true;
  ++polls;
  if (polls > max_polls) {
    if ((threadIdx.x & 31) == 0) atomicExch(&bar->fault, 1);
    *quit = true;
    return false;
  }
  // one decision for the whole warp (polls is the same in every lane)
  if ((polls & 63) == 0 && __any_sync(0xffffffffu, *(volatile int*)&bar->fault != 0)) {
    *quit = true;
    return false;
  }
  // the pass is bound by the polls' L2 round trip: 0, 16 or 64 ns of sleep
  // measured the same on GB300 (DILU 128^3 2.61-2.62 ms), 256 ns 2 % slower
  if (SLEEP) __nanosleep(64);
  return false;
}

}  // namespace gbf
