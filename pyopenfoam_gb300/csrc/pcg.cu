// FP64 preconditioned conjugate gradient, PCGSolver._solve
// (solvers/pcg.py:97-187) with ResidualMonitor's convergence rules
// (solvers/residual.py:112-145).
//
// One iteration = three kernels; the scalars (alpha, beta, r.z, status,
// iteration, residual history) live in device memory and are produced by the
// last block of the reducing kernels, so the host never waits inside an
// iteration.  It reads the 64-byte status block every `check_every`
// iterations; kernels launched after convergence return immediately.
//
//   K_ap     : Ap = A p (bitwise reference Amul), partial p.Ap
//              last block: breakdown test |pAp| < 1e-30, alpha = rz / pAp
//   K_update : x = x + alpha p, r = r - alpha Ap, z = r / d,
//              partials r.r and r.z
//              last block: |r|, history, convergence, beta = rz'/rz
//   K_p      : p = z + beta p
//
// Element-wise arithmetic rounds exactly as the reference's torch ops
// (alpha*p rounded, then added; r / d by IEEE division); dot products are
// deterministic fixed-order trees with fused multiply-add accumulation.
//
// K_update is bound by the FP64 pipe (64 clocks of its SM quarter an
// instruction), so alpha p and the division run on the integer pipe
// (exact.cuh, the same bits; not alpha Ap as well: the two pipes are then
// about even) and r.r and r.z share one tree.  Whole solves with DIC, before
// and after: 120x110x100 72.2 -> 60.4 ms, 170x160x150 249.5 -> 173.1 ms (168.9
// with programmatic dependent launches), 90x80x70 in no order 47.7 -> 39.2 ms
// (732, 926 and 553 iterations).
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include "amul.cuh"
#include "barrier.cuh"
#include "exact.cuh"

namespace gbf {

struct PcgState {
  double rz, alpha, beta, res0, res, pAp;
  int iter, status, n_hist, pad;
  unsigned int ticket[4];
  GridBarrier bar;
};

struct PcgVecs {
  double *r, *z, *p, *Ap, *partials;
  PcgState* st;
};

__device__ __forceinline__ bool monitor_converged(double res, double res0, int iter,
                                                  const gbf_solve_params& P) {
  if (iter < P.min_iter) return false;
  if (res < P.tolerance) return true;
  if (res0 > 0.0 && res / res0 < P.rel_tol) return true;
  return false;
}

template <bool PREC>
__global__ void __launch_bounds__(kBlock)
    pcg_init_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                    const double* __restrict__ pd, const double* __restrict__ b,
                    const double* __restrict__ x, PcgVecs v, double* hist, gbf_solve_params P) {
  __shared__ double sh[2 * kBlock / 32];
  const int G = gridDim.x;
  double rr = 0.0, rz = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < L.n_cells; c += G * blockDim.x) {
    const double y = cell_amul<double, double, false>(L, coef, diag, x, c, __ldg(x + c));
    const double rc = __dsub_rn(__ldg(b + c), y);
    const double zc = PREC ? div_rn(rc, __ldg(pd + c)) : rc;
    v.r[c] = rc;
    v.z[c] = zc;
    v.p[c] = zc;
    rr = fma(rc, rc, rr);
    rz = fma(rc, zc, rz);
  }
  const SumPair sums = block_sum_two(rr, rz, sh);
  if (threadIdx.x == 0) {
    v.partials[blockIdx.x] = sums.a;
    v.partials[G + blockIdx.x] = sums.b;
  }
  if (last_block_done(&v.st->ticket[0])) {
    const SumPair total = reduce_partials_two(v.partials, v.partials + G, G, sh);
    const double trr = total.a, trz = total.b;
    if (threadIdx.x == 0) {
      PcgState* st = v.st;
      const double res = sqrt(trr);
      hist[0] = res;
      st->res0 = res;
      st->res = res;
      st->n_hist = 1;
      st->rz = trz;
      st->iter = 1;
      if (monitor_converged(res, res, 0, P))
        st->status = GBF_CONVERGED;
      else
        st->status = (P.max_iter < 1) ? GBF_MAX_ITER : GBF_RUNNING;
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(kBlock)
    pcg_ap_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                  PcgVecs v) {
  pdl_wait();
  pdl_launch_dependents();
  if (v.st->status != GBF_RUNNING) return;
  __shared__ double sh[2 * kBlock / 32];
  const int G = gridDim.x;
  const double* p = v.p;
  double acc = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < L.n_cells; c += G * blockDim.x) {
    const double pc = __ldg(p + c);
    const double y = cell_amul_k<KIND, double, double, false>(L, coef, diag, p, c, pc);
    v.Ap[c] = y;
    acc = fma(pc, y, acc);
  }
  acc = block_sum(acc, sh);
  if (threadIdx.x == 0) v.partials[blockIdx.x] = acc;
  if (last_block_done(&v.st->ticket[1])) {
    const double pAp = reduce_partials(v.partials, G, sh);
    if (threadIdx.x == 0) {
      PcgState* st = v.st;
      st->pAp = pAp;
      if (fabs(pAp) < 1e-30)
        st->status = GBF_BREAKDOWN;  // pcg.py:153-156: x returned as is
      else
        st->alpha = div_rn(st->rz, pAp);
    }
  }
}

template <bool PREC>
__global__ void __launch_bounds__(kBlock)
    pcg_update_kernel(int n, const double* __restrict__ pd, double* __restrict__ x, PcgVecs v,
                      double* hist, gbf_solve_params P) {
  pdl_wait();
  pdl_launch_dependents();
  if (v.st->status != GBF_RUNNING) return;
  __shared__ double sh[2 * kBlock / 32];
  const int G = gridDim.x;
  const double alpha = v.st->alpha;
  double rr = 0.0, rz = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += G * blockDim.x) {
    const double xc = __dadd_rn(x[c], mul_int(alpha, v.p[c]));
    const double rc = __dsub_rn(v.r[c], __dmul_rn(alpha, v.Ap[c]));
    const double zc = PREC ? div_rn(rc, __ldg(pd + c)) : rc;
    x[c] = xc;
    v.r[c] = rc;
    v.z[c] = zc;
    rr = fma(rc, rc, rr);
    rz = fma(rc, zc, rz);
  }
  const SumPair sums = block_sum_two(rr, rz, sh);
  if (threadIdx.x == 0) {
    v.partials[blockIdx.x] = sums.a;
    v.partials[G + blockIdx.x] = sums.b;
  }
  if (last_block_done(&v.st->ticket[2])) {
    const SumPair total = reduce_partials_two(v.partials, v.partials + G, G, sh);
    const double trr = total.a, trz = total.b;
    if (threadIdx.x == 0) {
      PcgState* st = v.st;
      const int it = st->iter;
      const double res = sqrt_rn(trr);
      hist[it] = res;
      st->res = res;
      st->n_hist = it + 1;
      if (monitor_converged(res, st->res0, it, P)) {
        st->status = GBF_CONVERGED;
      } else {
        st->beta = div_rn(trz, st->rz);
        st->rz = trz;
        st->iter = it + 1;
        if (it >= P.max_iter) st->status = GBF_MAX_ITER;
      }
    }
  }
}

__global__ void __launch_bounds__(kBlock) pcg_p_kernel(int n, PcgVecs v) {
  pdl_wait();
  pdl_launch_dependents();
  if (v.st->status != GBF_RUNNING) return;
  const double beta = v.st->beta;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    v.p[c] = __dadd_rn(v.z[c], __dmul_rn(beta, v.p[c]));
}

// ---------------------------------------------------------------------------
// Single-launch PCG for launch-bound (small and medium) systems.
//
// The three phases of an iteration run inside one cooperative launch whose
// blocks are all resident, separated by a grid barrier; every block reduces
// the per-block partials itself in the same fixed order, so all blocks hold
// the same scalars and take the same decisions without a further barrier.
// Same arithmetic per element and same ResidualMonitor rules as the
// three-kernel form.  Vectors that other blocks rewrite during the launch
// (p, and the partials) are read from L2 (__ldcg), never through L1.
//
// Every barrier wait is bounded: after kBarrierPolls polls (a few seconds)
// the block records a fault and returns; a block waiting at a barrier that
// sees the fault returns within 16 polls.  The host turns a fault into
// GBF_DEVICE_TIMEOUT.
// ---------------------------------------------------------------------------
// Its blocks per SM: the grid decides which cells share a partial sum, so it is
// fixed here and does not follow the register count of the day.
template <int KIND, bool PREC>
constexpr int kPersistentPerSM = !PREC ? 4 : KIND == kLayoutHex33 ? 2 : 3;

template <int KIND, bool PREC>
__global__ void __launch_bounds__(kBlock, (kPersistentPerSM<KIND, PREC>))
    pcg_persistent_kernel(gbf_layout L, const double* __restrict__ coef,
                          const double* __restrict__ diag, const double* __restrict__ pd,
                          const double* __restrict__ b, double* __restrict__ x, PcgVecs v,
                          double* hist, gbf_solve_params P) {
  __shared__ double sh[2 * kBlock / 32];
  const int G = gridDim.x, n = L.n_cells;
  const int c0 = blockIdx.x * blockDim.x + threadIdx.x, cs = G * blockDim.x;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  PcgState* st = v.st;
  GridBarrier* bar = &st->bar;
  double* partA = v.partials;       // p.Ap partials      [G]
  double* partB = v.partials + G;   // r.r, r.z partials  [2G]

  // r = b - A x, z = M^-1 r, p = z
  double rr = 0.0, rz = 0.0;
  for (int c = c0; c < n; c += cs) {
    const double y = cell_amul_k<KIND, double, double, false>(L, coef, diag, x, c, __ldg(x + c));
    const double rc = __dsub_rn(__ldg(b + c), y);
    const double zc = PREC ? div_rn(rc, __ldg(pd + c)) : rc;
    v.r[c] = rc;
    v.z[c] = zc;
    v.p[c] = zc;
    rr = fma(rc, rc, rr);
    rz = fma(rc, zc, rz);
  }
  const SumPair sums = block_sum_two(rr, rz, sh);
  if (threadIdx.x == 0) {
    partB[blockIdx.x] = sums.a;
    partB[G + blockIdx.x] = sums.b;
  }
  if (!grid_barrier(bar, G)) return;
  SumPair total = reduce_partials_two(partB, partB + G, G, sh);
  __shared__ double bc[2];
  if (threadIdx.x == 0) {
    bc[0] = total.a;
    bc[1] = total.b;
  }
  __syncthreads();
  const double res0 = sqrt(bc[0]);
  double rzv = bc[1], res = res0;
  int iter = 1, n_hist = 1;
  int status = monitor_converged(res0, res0, 0, P) ? GBF_CONVERGED
               : (P.max_iter < 1 ? GBF_MAX_ITER : GBF_RUNNING);
  if (lead) hist[0] = res0;

  for (int launched = 0; status == GBF_RUNNING && launched < P.max_iter; ++launched) {
    // Ap = A p, p.Ap
    double acc = 0.0;
    for (int c = c0; c < n; c += cs) {
      const double pc = __ldcg(v.p + c);
      const double y = cell_amul_k<KIND, double, double, false, true>(L, coef, diag, v.p, c, pc);
      v.Ap[c] = y;
      acc = fma(pc, y, acc);
    }
    acc = block_sum(acc, sh);
    if (threadIdx.x == 0) partA[blockIdx.x] = acc;
    if (!grid_barrier(bar, G)) return;
    const double s0 = reduce_partials(partA, G, sh);
    if (threadIdx.x == 0) bc[0] = s0;
    __syncthreads();
    const double pAp = bc[0];
    if (fabs(pAp) < 1e-30) {  // pcg.py:153-156: x returned as is
      status = GBF_BREAKDOWN;
      break;
    }
    const double alpha = rzv / pAp;
    // x += alpha p, r -= alpha Ap, z = M^-1 r, r.r, r.z
    rr = 0.0;
    rz = 0.0;
    for (int c = c0; c < n; c += cs) {
      const double xc = __dadd_rn(x[c], __dmul_rn(alpha, __ldcg(v.p + c)));
      const double rc = __dsub_rn(v.r[c], __dmul_rn(alpha, v.Ap[c]));
      const double zc = PREC ? div_rn(rc, __ldg(pd + c)) : rc;
      x[c] = xc;
      v.r[c] = rc;
      v.z[c] = zc;
      rr = fma(rc, rc, rr);
      rz = fma(rc, zc, rz);
    }
    const SumPair sums = block_sum_two(rr, rz, sh);
    if (threadIdx.x == 0) {
      partB[blockIdx.x] = sums.a;
      partB[G + blockIdx.x] = sums.b;
    }
    if (!grid_barrier(bar, G)) return;
    total = reduce_partials_two(partB, partB + G, G, sh);
    if (threadIdx.x == 0) {
      bc[0] = total.a;
      bc[1] = total.b;
    }
    __syncthreads();
    const int it = iter;
    res = sqrt(bc[0]);
    if (lead) hist[it] = res;
    n_hist = it + 1;
    if (monitor_converged(res, res0, it, P)) {
      status = GBF_CONVERGED;
      break;
    }
    const double beta = bc[1] / rzv;
    rzv = bc[1];
    iter = it + 1;
    if (it >= P.max_iter) {
      status = GBF_MAX_ITER;
      break;
    }
    // p = z + beta p
    for (int c = c0; c < n; c += cs) v.p[c] = __dadd_rn(v.z[c], __dmul_rn(beta, v.p[c]));
    if (!grid_barrier(bar, G)) return;
  }
  if (lead) {
    st->status = status;
    st->res = res;
    st->res0 = res0;
    st->n_hist = n_hist;
    st->iter = iter;
    st->rz = rzv;
  }
}

// ---------------------------------------------------------------------------
// The same solve for systems whose cells fit one per resident thread (hex 3+3
// layouts).  At 32^3 an iteration of pcg_persistent_kernel took 15.3 us, of
// which three grid barriers with a read of the partial sums behind each took
// about 6 and FP64 instructions -- 64 clocks each on the warp's SM quarter, two
// warps a quarter -- most of the rest.  Here:
//   * a thread keeps its cell's coefficients, x, r, z, p and its neighbours' p
//     in registers; p of the block's own cells is shared, p of the others'
//     is recomputed from their z (the same two roundings), so that an
//     iteration exchanges z and the partial sums only and needs two
//     grid-wide waits instead of three;
//   * a wait is the exchange of the values itself: z and the blocks' partial
//     sums travel as 16-byte words of a value and the number of its turn,
//     written and read whole, and whoever needs a value polls its word until
//     the turn is right (no counter, no second trip for the values, no fence
//     on the way, nothing to clear); a block's sums go into a copy for each
//     block, so no two blocks poll the same lines;
//   * two sums go through one tree (the halves of a warp), quotients run on
//     the integer pipe, convergence is one comparison of r.r with the smallest
//     r.r that is not converged, and x is updated while the sums travel.
// The partial sums are those of pcg_persistent_kernel, block by block and in
// its order, so x, the residuals and the decisions are its bits.  An iteration
// takes 8.6 us at 32^3 (15.3 before) and 14.2 us at 48 x 40 x 36 (23.3); of
// that some 3.3 and 6.4 us are FP64 instructions.  Tried on the way: sums
// behind a grid barrier's release and acquire, 11.3 and 20.5 us (a release
// store waits 2-5 us behind the other blocks' polls); empty-marker slots with
// a fence per iteration, 9.4 and 17.7 us; every block polling the same words
// instead of its own copy, 9.3 and 15.2 us.
//
// A word is written again two turns later.  Sums: a block publishes its sums of
// wait w + 2 after it has collected those of w + 1 of every block, and a block
// publishes those after it has read all of w.  z: a thread publishes that of
// iteration i + 2 after its block has collected p.Ap of that iteration, and a
// block publishes its part of it after its threads have read all z of i + 1.
// ---------------------------------------------------------------------------
constexpr int kSlotSets = 2;

// A value and the number of its turn.
struct __align__(16) TurnWord {
  double v;
  long long turn;
};

__device__ __forceinline__ void st_word(TurnWord* p, double v, long long turn) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(turn)
      : "memory");
}

__device__ __forceinline__ TurnWord ld_word(const TurnWord* p) {
  long long v, turn;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(v), "=l"(turn)
      : "l"(p)
      : "memory");
  return TurnWord{__longlong_as_double(v), turn};
}

// Resident blocks per SM the kernel is compiled for: it takes systems of up to
// 2 * 256 cells per SM (77824 on 152), for which pcg_persistent_kernel, with at
// least as many blocks resident, has a cell a thread too.
constexpr int kResidentPerSM = 2;
constexpr int kResidentMaxBlocks = 512;  // sizes the workspace

// The sums over the block of a and b, each the tree of block_sum: lanes 0-15 of
// a warp carry a, lanes 16-31 b, so each level is one addition for both.
// Threads from `count` on hold 0.0.  Valid in threads 0 (a) and 16 (b).
__device__ __forceinline__ double block_sum_pair(double a, double b, double* sh, int count) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const bool low = lane < 16;
  double v = 0.0;
  if (32 * wid < count) {
    v = __dadd_rn(low ? a : b, __shfl_xor_sync(0xffffffffu, low ? b : a, 16));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o, 16));
  }
  if ((lane & 15) == 0) sh[(low ? 0 : 8) + wid] = v;
  __syncthreads();
  if (wid == 0) {
    // the tree's first two levels add zeros, which turn -0.0 into +0.0
    v = first_term((lane & 15) < 8 ? sh[(low ? 0 : 8) + (lane & 7)] : 0.0);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o, 16));
  }
  return v;
}

// As above for one sum; valid in thread 0.
__device__ __forceinline__ double block_sum_one(double v, double* sh, int count) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (32 * wid < count) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  }
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = first_term(lane < 8 ? sh[lane] : 0.0);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
  }
  return v;
}

// One unsuccessful round of polls; false when the wait has run out.
__device__ __forceinline__ bool poll_again(long long& polls, long long most, int* fault) {
  ++polls;
  if (polls > most || ((polls & 63) == 0 && *(volatile int*)fault != 0)) {
    atomicExch(fault, 1);
    return false;
  }
  return true;
}

// a < b for a > 0, +0.0 or NaN and b >= +0.0 or NaN, on the integer pipe.
__device__ __forceinline__ bool less_nn(double a, double b) {
  const unsigned long long ua = (unsigned long long)__double_as_longlong(a);
  const unsigned long long ub = (unsigned long long)__double_as_longlong(b);
  return ua < ub && ub <= 0x7ff0000000000000ull;
}

// The smallest s >= 0 for which a monotone test holds, from a guess a few
// representable numbers away at most; NaN when it is not found there.
template <typename F>
__device__ __forceinline__ double first_where(double guess, F&& test) {
  long long g = __double_as_longlong(guess);
  for (int k = 0; k < 16 && !test(__longlong_as_double(g)); ++k) ++g;
  for (int k = 0; k < 32; ++k) {
    if (!test(__longlong_as_double(g))) return __longlong_as_double(0x7ff8000000000000LL);
    if (g == 0 || !test(__longlong_as_double(g - 1))) return __longlong_as_double(g);
    --g;
  }
  return __longlong_as_double(0x7ff8000000000000LL);
}

// The smallest r.r whose norm does not satisfy monitor_converged's two norm
// rules (sqrt and the division by res0 are monotone): 0 when none does, NaN
// when it lies outside the ordinary range, where the rules are applied as
// they stand.
__device__ double unconverged_rr(double res0, const gbf_solve_params& P) {
  const double nan = __longlong_as_double(0x7ff8000000000000LL);
  if (!(res0 < 1e140) || !(P.tolerance < 1e140) || !(P.rel_tol < 1e100)) return nan;
  double t = 0.0;  // the smallest norm that is not converged
  if (res0 > 0.0 && P.rel_tol > 0.0) {
    if (!(res0 > 1e-140) || !(P.rel_tol > 1e-100)) return nan;
    t = first_where(P.rel_tol * res0, [&](double r) { return !(r / res0 < P.rel_tol); });
  }
  if (P.tolerance > t) t = P.tolerance;
  if (!(t > 0.0)) return t;  // 0 or NaN
  if (!(t > 1e-140)) return nan;
  return first_where(t * t, [&](double s) { return !(sqrt(s) < t); });
}

template <bool PREC>
__global__ void __launch_bounds__(kBlock, kResidentPerSM)
    pcg_resident_kernel(gbf_layout L, const double* __restrict__ coef,
                        const double* __restrict__ diag, const double* __restrict__ pd,
                        const double* __restrict__ b, double* __restrict__ x_io, TurnWord* z_all,
                        TurnWord* slots, PcgState* st, double* hist, gbf_solve_params P,
                        long long max_polls) {
  __shared__ double sh[16], ps[kBlock], bc[2], sent[2];
  const int G = gridDim.x, n = L.n_cells, tid = threadIdx.x, blk = blockIdx.x;
  const int c0 = blk * kBlock, c = c0 + tid;
  const bool mine = c < n, lead = blk == 0 && tid == 0;
  int* fault = &st->bar.fault;

  // the cell's row: slot k at cell c + d[k] (bit k of `on`), inside the block (bit k of `in`)
  double a[6] = {}, pn[6] = {}, dc = 0.0, pdc = 1.0, x = 0.0, r = 0.0, z = 0.0, p = 0.0;
  int q[6] = {};
  unsigned on = 0, in = 0;
  if (mine) {
    const int s = c >> 5, lane = c & 31, base = 192 * s + lane;
    const int2* __restrict__ dm = reinterpret_cast<const int2*>(L.slot_dm) + 6 * s;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const int2 e = __ldg(dm + k);
      a[k] = __ldg(coef + base + 32 * k);
      if ((unsigned)e.y >> lane & 1u) {
        on |= 1u << k;
        q[k] = c + e.x;
        if ((unsigned)(q[k] - c0) < (unsigned)kBlock) in |= 1u << k;
      }
    }
    dc = __ldg(diag + c);
    if (PREC) pdc = __ldg(pd + c);
    x = x_io[c];
  }
  // (A v)[c] from v of the cell and of its neighbours: cell_amul_fixed's order
  auto row = [&](double vc, const double (&v)[6]) {
    double so = 0.0, sn = 0.0;
    double t = first_term(__dmul_rn(a[0], v[0]));
    so = (on & 1u) ? t : so;
#pragma unroll
    for (int k = 1; k < 3; ++k) {
      t = __dadd_rn(so, __dmul_rn(a[k], v[k]));
      so = (on >> k & 1u) ? t : so;
    }
    t = first_term(__dmul_rn(a[3], v[3]));
    sn = (on & 8u) ? t : sn;
#pragma unroll
    for (int k = 4; k < 6; ++k) {
      t = __dadd_rn(sn, __dmul_rn(a[k], v[k]));
      sn = (on >> k & 1u) ? t : sn;
    }
    return __dadd_rn(__dadd_rn(__dmul_rn(dc, vc), so), sn);
  };
  long long wait = 1;  // number of the grid-wide wait
  long long turn = 1;  // number of the z
  bool ok = true;
  auto z_of = [&](int q) { return z_all + (turn & 1) * (long long)n + q; };
  auto publish_z = [&] {
    if (mine) st_word(z_of(c), z, turn);
  };
  auto word = [&](int dest, int src, int which) {
    return slots + (((size_t)dest * 2 + (wait & 1)) * 2 + which) * G + src;
  };
  // Publishes the block's sums (in thread 0, the second in thread 16)
  auto publish = [&](double u, bool pair) {
    if (tid == 0) sent[0] = u;
    if (tid == 16) sent[1] = u;
    __syncthreads();
    for (int i = tid; i < G; i += kBlock) {
      st_word(word(i, blk, 0), sent[0], wait);
      if (pair) st_word(word(i, blk, 1), sent[1], wait);
    }
  };
  // Two words polled together, as far as wanted: values into v0, v1.
  auto poll_two = [&](const TurnWord* p0, bool want0, double& v0, const TurnWord* p1, bool want1,
                      double& v1, long long number) {
    long long polls = 0;
    while (want0 || want1) {
      TurnWord w0{0.0, 0}, w1{0.0, 0};
      if (want0) w0 = ld_word(p0);
      if (want1) w1 = ld_word(p1);
      if (want0 && w0.turn == number) v0 = w0.v, want0 = false;
      if (want1 && w1.turn == number) v1 = w1.v, want1 = false;
      if ((want0 || want1) && !poll_again(polls, max_polls, fault)) {
        ok = false;
        return;
      }
    }
  };
  // z of the neighbours in other blocks: slots 2 and 3 (the farthest ones of a
  // mesh in cell order) first, which most threads want
  auto gather = [&](double (&zq)[6]) {
    const unsigned far = on & ~in;
#pragma unroll
    for (int k = 2; k >= 0; --k)
      poll_two(z_of(q[k]), far >> k & 1u, zq[k], z_of(q[5 - k]), far >> (5 - k) & 1u, zq[5 - k],
               turn);
    ++turn;
  };
  // What this thread takes of all blocks' sums: those of blocks tid, tid + 256,
  // ..., reduce_partials' order.
  double got0 = 0.0, got1 = 0.0;
  auto collect = [&](bool pair) {
    got0 = got1 = 0.0;
    for (int i = tid; i < G; i += kBlock) {
      double w0 = 0.0, w1 = 0.0;
      poll_two(word(blk, i, 0), true, w0, word(blk, i, 1), pair, w1, wait);
      got0 = i == tid ? first_term(w0) : __dadd_rn(got0, w0);
      if (pair) got1 = i == tid ? first_term(w1) : __dadd_rn(got1, w1);
    }
    ++wait;
    return __syncthreads_and(ok) != 0;
  };

  // r = b - A x, z = M^-1 r, p = z
  {
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = (on >> k & 1u) ? __ldcg(x_io + q[k]) : 0.0;
    if (mine) {
      r = __dsub_rn(__ldg(b + c), row(x, v));
      z = PREC ? div_rn(r, pdc) : r;
      p = z;
    }
  }
  publish_z();
  double u = block_sum_pair(mine ? __fma_rn(r, r, 0.0) : 0.0, mine ? __fma_rn(r, z, 0.0) : 0.0,
                            sh, kBlock);
  publish(u, true);
  ps[tid] = p;
  gather(pn);
  if (!collect(true)) return;
  u = block_sum_pair(got0, got1, sh, G);
  if (tid == 0) bc[0] = u;
  if (tid == 16) bc[1] = u;
  __syncthreads();
  double rr = bc[0], rzv = bc[1];
  const double res0 = sqrt(rr);
  const double limit = unconverged_rr(res0, P);  // NaN: apply the rules
  auto converged = [&](double s, int iter) {
    if (iter < P.min_iter) return false;
    if (limit == limit && __double_as_longlong(s) >= 0) return less_nn(s, limit);
    return monitor_converged(sqrt(s), res0, iter, P);
  };
  int iter = 1, n_hist = 1;
  int status = converged(rr, 0) ? GBF_CONVERGED
               : (P.max_iter < 1 ? GBF_MAX_ITER : GBF_RUNNING);
  if (lead) hist[0] = res0;

  for (int launched = 0; status == GBF_RUNNING && launched < P.max_iter; ++launched) {
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] = (in >> k & 1u) ? ps[q[k] - c0] : pn[k];
    const double Ap = row(p, v);
    u = block_sum_one(mine ? __fma_rn(p, Ap, 0.0) : 0.0, sh, kBlock);
    publish(u, false);
    // (the root of an earlier r.r, while the sums travel)
    if (lead && launched > 0) hist[iter - 1] = sqrt_rn(rr);
    if (!collect(false)) return;
    u = block_sum_one(got0, sh, G);
    if (tid == 0) bc[0] = u;
    __syncthreads();
    const double pAp = bc[0];
    if (less_nn(fabs(pAp), 1e-30)) {
      status = GBF_BREAKDOWN;  // pcg.py:153-156: x returned as is
      break;
    }
    const double alpha = div_rn(rzv, pAp);
    r = __dsub_rn(r, __dmul_rn(alpha, Ap));
    z = (PREC && mine) ? div_rn(r, pdc) : r;
    publish_z();
    u = block_sum_pair(mine ? __fma_rn(r, r, 0.0) : 0.0, mine ? __fma_rn(r, z, 0.0) : 0.0, sh,
                       kBlock);
    publish(u, true);
    x = __dadd_rn(x, __dmul_rn(alpha, p));
    double zq[6] = {};
    gather(zq);
    if (!collect(true)) return;
    u = block_sum_pair(got0, got1, sh, G);
    if (tid == 0) bc[0] = u;
    if (tid == 16) bc[1] = u;
    __syncthreads();
    const int it = iter;
    rr = bc[0];
    n_hist = it + 1;
    if (converged(rr, it)) {
      status = GBF_CONVERGED;
      break;
    }
    const double beta = div_rn(bc[1], rzv);
    rzv = bc[1];
    iter = it + 1;
    if (it >= P.max_iter) {
      status = GBF_MAX_ITER;
      break;
    }
    p = __dadd_rn(z, __dmul_rn(beta, p));
    ps[tid] = p;
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if ((on & ~in) >> k & 1u) pn[k] = __dadd_rn(zq[k], __dmul_rn(beta, pn[k]));
    __syncthreads();
  }
  if (mine) x_io[c] = x;
  if (lead) {
    if (n_hist > 1) hist[n_hist - 1] = sqrt_rn(rr);
    st->status = status;
    st->res = sqrt_rn(rr);
    st->res0 = res0;
    st->n_hist = n_hist;
    st->iter = iter;
    st->rz = rzv;
  }
}

// Blocks of the single-launch PCG that can be resident at once (0 if the
// device cannot launch it cooperatively).
template <int KIND, bool PREC>
static int persistent_grid(int n) {
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!coop || sms <= 0) return 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pcg_persistent_kernel<KIND, PREC>,
                                                    kBlock, 0) != cudaSuccess || per_sm <= 0)
    return 0;
  if (per_sm > kPersistentPerSM<KIND, PREC>) per_sm = kPersistentPerSM<KIND, PREC>;
  long long g = (long long)per_sm * sms;
  const long long need = (n + kBlock - 1) / kBlock;
  if (g > need) g = need;
  if (g > kMaxGrid / 2) g = kMaxGrid / 2;  // partA + partB fit the partials buffer
  return g < 1 ? 1 : (int)g;
}

template <int KIND, bool PREC>
static cudaError_t launch_persistent(int grid, const gbf_layout* L, const double* coef,
                                     const double* diag, const double* pd, const double* b,
                                     double* x, PcgVecs v, double* hist,
                                     const gbf_solve_params* P, cudaStream_t s) {
  gbf_layout Lc = *L;
  gbf_solve_params Pc = *P;
  void* args[] = {&Lc, (void*)&coef, (void*)&diag, (void*)&pd, (void*)&b, &x, &v, &hist, &Pc};
  return cudaLaunchCooperativeKernel((const void*)pcg_persistent_kernel<KIND, PREC>,
                                     dim3(grid), dim3(kBlock), args, 0, s);
}

// Systems up to this many cells run the single-launch form under variant 0.
// Since the three kernels overlap their launches they are the faster form from
// about a million cells on hex layouts and throughout on general ones: an
// iteration with DIC, single launch and three kernels, hex 198360 cells 25.8 and
// 27.1 us, 499280 37.9 and 42.3, 1000000 64.0 and 64.6, 1560896 95.0 and 84.2,
// 2080768 123 and 103; renumbered 99360 30.2 and 27.5, 499280 73.6 and 63.0,
// 2080768 250 and 213.  The line is where it was because the forms sum over
// other cells: moving it moves the last bits of every solve in between.
constexpr int kPersistentMaxCells = 1 << 21;

// Whether pcg_resident_kernel takes the system: a hex 3+3 layout, one cell a
// resident thread.
template <bool PREC>
static bool resident_fits(const gbf_layout& L, bool hex) {
  int dev = 0, coop = 0, sms = 0, per_sm = 0;
  if (!hex || cudaGetDevice(&dev) != cudaSuccess) return false;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (!coop || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pcg_resident_kernel<PREC>,
                                                             kBlock, 0) != cudaSuccess)
    return false;
  if (per_sm > kResidentPerSM) per_sm = kResidentPerSM;
  if (L.n_cells > (long long)kResidentMaxBlocks * kBlock) return false;
  return L.n_cells <= (long long)per_sm * sms * kBlock;
}

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

}  // namespace gbf

using namespace gbf;

// r, z, p, Ap, the partial sums and the state.
static size_t pcg_base_bytes(int n) {
  return 4 * align256(sizeof(double) * (size_t)n) + align256(sizeof(double) * 2 * kMaxGrid) +
         align256(sizeof(PcgState));
}

// Bytes of pcg_resident_kernel's sum words on G blocks.
static size_t resident_bytes(long long G) {
  return align256((size_t)G * 2 * kSlotSets * G * sizeof(TurnWord));
}

// What a solve of n cells can use: grows with n, so that a workspace for the
// largest of several systems is one for each.  A system too large for the
// resident kernel needs no sum words, but asks for no less than the largest
// that is not.  Without a device there is no resident kernel.
extern "C" size_t gbf_pcg_workspace_bytes(int32_t n) {
  if (n < 0) return 0;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) {
    sms = 0;
    cudaGetLastError();  // no device: not an error of this query
  }
  long long most = (long long)kResidentPerSM * sms;
  if (most > kResidentMaxBlocks) most = kResidentMaxBlocks;
  const size_t base = pcg_base_bytes(n);
  const long long G = ((long long)n + kBlock - 1) / kBlock;
  if (G <= most) return base + resident_bytes(G);
  const size_t largest = pcg_base_bytes((int)(most * kBlock)) + resident_bytes(most);
  return base > largest ? base : largest;
}

extern "C" int gbf_pcg_solve_f64(const gbf_layout* L, const double* coef, const double* diag,
                                 const double* pd, const double* b, double* x, double* hist,
                                 const gbf_solve_params* P, gbf_solve_result* R, void* ws,
                                 size_t ws_bytes, void* stream) {
  ::gbf::NvtxScope nvtx_("gbf_pcg_solve_f64");
  int rc = check_layout(L);
  if (rc) return rc;
  GBF_REQUIRE(P && R, "pcg: NULL params/result");
  GBF_REQUIRE(P->max_iter >= 0, "pcg: negative max_iter");
  const int n = L->n_cells;
  memset(R, 0, sizeof(*R));
  if (n == 0) {
    // empty system: |r| = 0; converged iff 0 < tolerance (residual.py:137-140),
    // otherwise the first p.Ap = 0 is a breakdown (pcg.py:153)
    const bool conv = (0 >= P->min_iter) && (0.0 < P->tolerance);
    R->iterations = 1;
    R->status = conv ? GBF_CONVERGED : (P->max_iter < 1 ? GBF_MAX_ITER : GBF_BREAKDOWN);
    return GBF_OK;
  }
  GBF_REQUIRE(diag && b && x && hist && ws && (L->n_faces == 0 || coef), "pcg: NULL pointer");
  // the resident kernel's sum words are not required: without them the
  // multi-cell kernel runs, with the same bits
  GBF_REQUIRE(ws_bytes >= pcg_base_bytes(n), "pcg: workspace too small");
  cudaStream_t s = as_stream(stream);

  char* w = static_cast<char*>(ws);
  const size_t vb = align256(sizeof(double) * (size_t)n);
  PcgVecs v;
  v.r = reinterpret_cast<double*>(w);
  v.z = reinterpret_cast<double*>(w + vb);
  v.p = reinterpret_cast<double*>(w + 2 * vb);
  v.Ap = reinterpret_cast<double*>(w + 3 * vb);
  v.partials = reinterpret_cast<double*>(w + 4 * vb);
  v.st = reinterpret_cast<PcgState*>(w + 4 * vb + align256(sizeof(double) * 2 * kMaxGrid));

  GBF_REQUIRE(P->variant >= 0 && P->variant <= 2, "pcg: variant must be 0, 1 or 2");
  GBF_CHECK_CUDA(cudaMemsetAsync(v.st, 0, sizeof(PcgState), s));

  // single launch (variant 2, or variant 0 on a launch-bound system)
  if (P->variant == 2 || (P->variant == 0 && n <= kPersistentMaxCells)) {
    const bool hex = layout_kind(*L) == kLayoutHex33;
    const int Gr = (n + kBlock - 1) / kBlock;
    // its words are written and read whole, 16 bytes at a 16-byte boundary;
    // everything else in the workspace takes 8
    const bool resident =
        (pd ? resident_fits<true>(*L, hex) : resident_fits<false>(*L, hex)) &&
        ws_bytes >= pcg_base_bytes(n) + resident_bytes(Gr) &&
        reinterpret_cast<uintptr_t>(ws) % alignof(TurnWord) == 0;
    const int Gp = resident ? Gr
                   : hex ? (pd ? persistent_grid<kLayoutHex33, true>(n)
                             : persistent_grid<kLayoutHex33, false>(n))
                       : (pd ? persistent_grid<kLayoutGeneric, true>(n)
                             : persistent_grid<kLayoutGeneric, false>(n));
    if (Gp > 0) {
      cudaError_t e;
      if (resident) {
        // z words over r, z, p, Ap (32 bytes a cell), sum words behind
        TurnWord* zw = reinterpret_cast<TurnWord*>(w);
        TurnWord* sw = reinterpret_cast<TurnWord*>(w + pcg_base_bytes(n));
        GBF_CHECK_CUDA(cudaMemsetAsync(zw, 0, 2 * sizeof(TurnWord) * (size_t)n, s));
        GBF_CHECK_CUDA(cudaMemsetAsync(sw, 0, resident_bytes(Gp), s));
        gbf_layout Lc = *L;
        gbf_solve_params Pc = *P;
        long long polls = kBarrierPolls;
        void* args[] = {&Lc, (void*)&coef, (void*)&diag, (void*)&pd, (void*)&b, &x, &zw, &sw,
                        &v.st, &hist, &Pc, &polls};
        e = cudaLaunchCooperativeKernel(pd ? (const void*)pcg_resident_kernel<true>
                                           : (const void*)pcg_resident_kernel<false>,
                                        dim3(Gp), dim3(kBlock), args, 0, s);
      } else if (hex)
        e = pd ? launch_persistent<kLayoutHex33, true>(Gp, L, coef, diag, pd, b, x, v, hist, P, s)
               : launch_persistent<kLayoutHex33, false>(Gp, L, coef, diag, pd, b, x, v, hist, P,
                                                        s);
      else
        e = pd ? launch_persistent<kLayoutGeneric, true>(Gp, L, coef, diag, pd, b, x, v, hist, P,
                                                         s)
               : launch_persistent<kLayoutGeneric, false>(Gp, L, coef, diag, pd, b, x, v, hist,
                                                          P, s);
      GBF_CHECK_CUDA(e);
      PcgState hs;
      GBF_CHECK_CUDA(cudaMemcpyAsync(&hs, v.st, sizeof(hs), cudaMemcpyDeviceToHost, s));
      GBF_CHECK_CUDA(cudaStreamSynchronize(s));
      R->iterations = hs.n_hist;
      R->status = hs.bar.fault ? GBF_DEVICE_TIMEOUT
                               : (hs.status == GBF_RUNNING ? GBF_MAX_ITER : hs.status);
      R->final_residual = hs.res;
      R->initial_residual = hs.res0;
      R->launches = 1;
      return GBF_OK;
    }
    GBF_REQUIRE(P->variant != 2, "pcg: the device cannot run the single-launch form");
  }

  int G = reduction_grid();
  const int need = (n + kBlock - 1) / kBlock;
  if (G > need) G = need;
  if (pd)
    pcg_init_kernel<true><<<G, kBlock, 0, s>>>(*L, coef, diag, pd, b, x, v, hist, *P);
  else
    pcg_init_kernel<false><<<G, kBlock, 0, s>>>(*L, coef, diag, pd, b, x, v, hist, *P);
  GBF_CHECK_LAUNCH();

  const int chunk = P->check_every > 0 ? P->check_every : 32;
  PcgState hs;
  GBF_CHECK_CUDA(cudaMemcpyAsync(&hs, v.st, sizeof(hs), cudaMemcpyDeviceToHost, s));
  GBF_CHECK_CUDA(cudaStreamSynchronize(s));
  int launched = 0;
  while (hs.status == GBF_RUNNING && launched < P->max_iter) {
    for (int j = 0; j < chunk && launched < P->max_iter; ++j, ++launched) {
      const bool tb = timing_begin(kProbePcgAp, s);
      if (layout_kind(*L) == kLayoutHex33)
        launch_pdl(pcg_ap_kernel<kLayoutHex33>, G, kBlock, s, *L, coef, diag, v);
      else
        launch_pdl(pcg_ap_kernel<kLayoutGeneric>, G, kBlock, s, *L, coef, diag, v);
      if (tb) timing_end(kProbePcgAp, s);
      if (pd)
        launch_pdl(pcg_update_kernel<true>, G, kBlock, s, n, pd, x, v, hist, *P);
      else
        launch_pdl(pcg_update_kernel<false>, G, kBlock, s, n, pd, x, v, hist, *P);
      launch_pdl(pcg_p_kernel, G, kBlock, s, n, v);
    }
    GBF_CHECK_LAUNCH();
    GBF_CHECK_CUDA(cudaMemcpyAsync(&hs, v.st, sizeof(hs), cudaMemcpyDeviceToHost, s));
    GBF_CHECK_CUDA(cudaStreamSynchronize(s));
  }
  R->iterations = hs.n_hist;
  R->status = (hs.status == GBF_RUNNING) ? GBF_MAX_ITER : hs.status;
  R->final_residual = hs.res;
  R->initial_residual = hs.res0;
  R->launches = 1 + 3 * launched;
  return GBF_OK;
}

// Self-test of the cell-per-thread kernel's bounded waits, without a GPU fault:
// one block of a system of two, whose cell 255 has a face to cell 256 of the
// block that is not launched.  Nothing publishes that cell's z, so the wait
// runs out after 1000 polls (about a millisecond), the fault word is set, the
// block returns and x stays as it was.  result_h[0] = the fault word (1
// expected), [1] = 1 if x is unchanged.  Every index stays inside the buffers.
extern "C" int gbf_selftest_pcg_resident_fault(int32_t* result_h) {
  GBF_REQUIRE(result_h, "selftest: NULL pointer");
  int dev = 0, coop = 0;
  GBF_CHECK_CUDA(cudaGetDevice(&dev));
  GBF_CHECK_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  GBF_REQUIRE(coop, "selftest: the device has no cooperative launch");
  constexpr int n = 2 * kBlock, slices = n / 32;
  struct Buf {
    TurnWord z[2 * n], sums[2 * kSlotSets];
    double coef[192 * slices], diag[n], b[n], x[n], hist[2];
    int32_t dm[12 * slices];
    PcgState st;
  };
  Buf* h = static_cast<Buf*>(calloc(1, sizeof(Buf)));
  GBF_REQUIRE(h, "selftest: out of memory");
  for (int i = 0; i < n; ++i) h->diag[i] = 4.0, h->b[i] = h->x[i] = 1.0;
  const int last = kBlock / 32 - 1;  // slice of cell 255: its first slot, lane 31 alone
  h->dm[12 * last] = 1;
  h->dm[12 * last + 1] = (int32_t)0x80000000u;
  Buf* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(Buf));
  if (e == cudaSuccess) e = cudaMemcpy(d, h, sizeof(Buf), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    gbf_layout L;
    memset(&L, 0, sizeof(L));
    L.n_cells = n;
    L.slot_dm = d->dm;
    gbf_solve_params P;
    memset(&P, 0, sizeof(P));
    P.max_iter = 1;
    const double *coef = d->coef, *diag = d->diag, *pd = nullptr, *b = d->b;
    double *x = d->x, *hist = d->hist;
    TurnWord *z = d->z, *sums = d->sums;
    PcgState* st = &d->st;
    long long polls = 1000;
    void* args[] = {&L, (void*)&coef, (void*)&diag, (void*)&pd, (void*)&b, &x, &z, &sums,
                    &st, &hist, &P, &polls};
    e = cudaLaunchCooperativeKernel((const void*)pcg_resident_kernel<false>, dim3(1),
                                    dim3(kBlock), args, 0, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(h, d, sizeof(Buf), cudaMemcpyDeviceToHost);
  }
  if (d) cudaFree(d);
  int same = 1;
  for (int i = 0; i < n; ++i) same &= h->x[i] == 1.0 ? 1 : 0;
  result_h[0] = h->st.bar.fault;
  result_h[1] = same;
  free(h);
  GBF_CHECK_CUDA(e);
  return GBF_OK;
}

// ---------------------------------------------------------------------------
// gbf_pcg_solve_f64_noalloc: the FP64 PCG solve without a caller workspace.
//
// Who needs it: callers that cannot allocate device memory at the moment they
// solve.  Examples are real-time or embedded time loops that must never wait
// on the allocator or handle an out-of-memory error mid-step, host programs
// (a C, C++ or Fortran CFD code) whose device memory is owned by their own
// pool or runs under a fixed budget and which hand the solver only their own
// input and output buffers, and plugin hosts that expose no allocator to the
// library they load.  Such a caller keeps x, b, the matrix and the history
// buffer; everything else the solve needs (the four iteration vectors r, z,
// p, Ap, the per-block partial sums and the state block) lives in one
// file-scope device array of fixed size.
//
// Limits and rules:
//   * at most kNoAllocMaxCells (1,048,576) cells; larger systems are refused
//     with GBF_ERR_ARG -- use gbf_pcg_solve_f64 with a workspace for them;
//   * the array occupies 32.1 MiB on every GPU that loads the library, until
//     the process exits;
//   * it always runs the three-kernel-per-iteration form (variant 0 and 1
//     alike); variant 2, which demands the single cooperative launch, is
//     refused with GBF_ERR_ARG, as is any value outside 0..2;
//   * the solve cannot run inside a stream capture: between chunks of
//     iterations it copies the state block to the host and synchronises the
//     stream, which a capturing stream refuses;
//   * every call looks up the array's device address on the current device
//     (cudaGetSymbolAddress; no cache, so an address never outlives a
//     cudaDeviceReset that reloads the module); the first call on a device
//     loads the module there if it is not loaded yet;
//   * all calls share the one array, which keeps the previous call's
//     contents: the state block is cleared at the start of every call, and
//     calls whose work overlaps on the GPU (different streams, or different
//     host threads on one device) race on the array and must be serialised
//     by the caller;
//   * nothing here calls cudaMalloc, cudaFree or any allocating routine.
// ---------------------------------------------------------------------------
namespace gbf {

constexpr int kNoAllocMaxCells = 1 << 20;
constexpr size_t kNoAllocVecBytes = sizeof(double) * (size_t)kNoAllocMaxCells;  // 256-aligned
constexpr size_t kNoAllocPartialBytes = ((sizeof(double) * 2 * kMaxGrid) + 255) & ~(size_t)255;
constexpr size_t kNoAllocStateBytes = (sizeof(PcgState) + 255) & ~(size_t)255;
constexpr size_t kNoAllocBytes = 4 * kNoAllocVecBytes + kNoAllocPartialBytes + kNoAllocStateBytes;

static __device__ __align__(256) unsigned char g_pcg_noalloc_scratch[kNoAllocBytes];

// Device address of the scratch array on the current device, looked up on
// every call (a few microseconds of host time).
static int noalloc_scratch(void** out) {
  void* p = nullptr;
  GBF_CHECK_CUDA(cudaGetSymbolAddress(&p, g_pcg_noalloc_scratch));
  GBF_REQUIRE(p != nullptr, "pcg_noalloc: scratch address lookup returned NULL");
  *out = p;
  return GBF_OK;
}

}  // namespace gbf

extern "C" int gbf_pcg_solve_f64_noalloc(const gbf_layout* L, const double* coef,
                                         const double* diag, const double* pd, const double* b,
                                         double* x, double* hist, const gbf_solve_params* P,
                                         gbf_solve_result* R, void* stream) {
  ::gbf::NvtxScope nvtx_("gbf_pcg_solve_f64_noalloc");
  int rc = check_layout(L);
  if (rc) return rc;
  GBF_REQUIRE(P && R, "pcg_noalloc: NULL params/result");
  GBF_REQUIRE(P->max_iter >= 0, "pcg_noalloc: negative max_iter");
  GBF_REQUIRE(P->variant == 0 || P->variant == 1,
              "pcg_noalloc: variant must be 0 or 1 (this entry point always runs three kernels "
              "per iteration; the single-launch form, variant 2, needs gbf_pcg_solve_f64)");
  const int n = L->n_cells;
  GBF_REQUIRE(n <= kNoAllocMaxCells,
              "pcg_noalloc: %d cells exceed the fixed scratch limit of %d cells; use "
              "gbf_pcg_solve_f64 with a workspace",
              n, kNoAllocMaxCells);
  memset(R, 0, sizeof(*R));
  if (n == 0) {
    const bool conv = (0 >= P->min_iter) && (0.0 < P->tolerance);
    R->iterations = 1;
    R->status = conv ? GBF_CONVERGED : (P->max_iter < 1 ? GBF_MAX_ITER : GBF_BREAKDOWN);
    return GBF_OK;
  }
  GBF_REQUIRE(diag && b && x && hist && (L->n_faces == 0 || coef), "pcg_noalloc: NULL pointer");
  void* scratch = nullptr;
  rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  cudaStream_t s = as_stream(stream);

  char* w = static_cast<char*>(scratch);
  PcgVecs v;
  v.r = reinterpret_cast<double*>(w);
  v.z = reinterpret_cast<double*>(w + kNoAllocVecBytes);
  v.p = reinterpret_cast<double*>(w + 2 * kNoAllocVecBytes);
  v.Ap = reinterpret_cast<double*>(w + 3 * kNoAllocVecBytes);
  v.partials = reinterpret_cast<double*>(w + 4 * kNoAllocVecBytes);
  v.st = reinterpret_cast<PcgState*>(w + 4 * kNoAllocVecBytes + kNoAllocPartialBytes);

  int G = reduction_grid();
  const int need = (n + kBlock - 1) / kBlock;
  if (G > need) G = need;
  // the state block (status, scalars, reduction tickets) must start at zero
  GBF_CHECK_CUDA(cudaMemsetAsync(v.st, 0, sizeof(PcgState), s));
  if (pd)
    pcg_init_kernel<true><<<G, kBlock, 0, s>>>(*L, coef, diag, pd, b, x, v, hist, *P);
  else
    pcg_init_kernel<false><<<G, kBlock, 0, s>>>(*L, coef, diag, pd, b, x, v, hist, *P);
  GBF_CHECK_LAUNCH();

  const int chunk = P->check_every > 0 ? P->check_every : 32;
  PcgState hs;
  GBF_CHECK_CUDA(cudaMemcpyAsync(&hs, v.st, sizeof(hs), cudaMemcpyDeviceToHost, s));
  GBF_CHECK_CUDA(cudaStreamSynchronize(s));
  const bool hex = layout_kind(*L) == kLayoutHex33;
  int launched = 0;
  while (hs.status == GBF_RUNNING && launched < P->max_iter) {
    for (int j = 0; j < chunk && launched < P->max_iter; ++j, ++launched) {
      if (hex)
        launch_pdl(pcg_ap_kernel<kLayoutHex33>, G, kBlock, s, *L, coef, diag, v);
      else
        launch_pdl(pcg_ap_kernel<kLayoutGeneric>, G, kBlock, s, *L, coef, diag, v);
      if (pd)
        launch_pdl(pcg_update_kernel<true>, G, kBlock, s, n, pd, x, v, hist, *P);
      else
        launch_pdl(pcg_update_kernel<false>, G, kBlock, s, n, pd, x, v, hist, *P);
      launch_pdl(pcg_p_kernel, G, kBlock, s, n, v);
    }
    GBF_CHECK_LAUNCH();
    GBF_CHECK_CUDA(cudaMemcpyAsync(&hs, v.st, sizeof(hs), cudaMemcpyDeviceToHost, s));
    GBF_CHECK_CUDA(cudaStreamSynchronize(s));
  }
  R->iterations = hs.n_hist;
  R->status = (hs.status == GBF_RUNNING) ? GBF_MAX_ITER : hs.status;
  R->final_residual = hs.res;
  R->initial_residual = hs.res0;
  R->launches = 1 + 3 * launched;
  return GBF_OK;
}
