// Smoothers and the kernels of the host-driven smoothing solvers:
//   Gauss-Seidel sweeps       solvers/smooth_solver.py:134-187 (SmoothSolver,
//                             smoother "GaussSeidel"), solvers/smoothers.py:
//                             63-149 (GaussSeidelSmoother, forward+backward,
//                             relaxed)
//   residual r = b - A x      every smoother's and solver's residual
//   relaxation x += w s z     JacobiSmoother (smoothers.py:152-200), the
//                             DIC/DILU Richardson smoothers
//                             (smooth_solver.py:189-232, smoothers.py:203-260)
//   |r|_2                     the residual norm of the convergence checks
//
// Gauss-Seidel runs as a level-scheduled wavefront (one launch per level,
// gbf_gs_schedule): a cell's update reads the already-updated values of its
// lower-numbered neighbours (forward) and the old values of the others, as
// the reference's sequential cell loop does; no two neighbours share a level.
// Each row sum follows the reference's loop over faces in ascending face
// order (owner-side and neighbour-side slots merged by face index), one
// rounding per operation, so the sweep is bitwise the reference's.
#include <limits.h>
#include <math.h>

#include "amul.cuh"
#include "exact.cuh"
#include "wavefront.cuh"

namespace gbf {

// The row sum of cell c's update: dc * xc, then coef * x[col] over the
// cell's slots in ascending face order (owner-side and neighbour-side slots
// merged by face index), one rounding per operation.  fetch(col) gives the
// x value the update reads at col.
template <typename FETCH>
__device__ __forceinline__ double gs_row(const gbf_layout& L, const double* __restrict__ coef,
                                         double dc, double xc, int c, FETCH&& fetch) {
  double row = __dmul_rn(dc, xc);
  bool merged = false;
  if (L.n_faces > 0) {
    const CellSlots cs = cell_slots(L, c);
    if (cs.wo <= 4 && cs.wn <= 4) {
      // Every slot's face, coefficient and x value loaded at once; when the
      // cell's neighbour-side faces all precede its owner-side faces (always
      // on a mesh in upper-triangular face order), ascending face order is
      // the neighbour-side slots followed by the owner-side slots.
      int fk[8];
      double a[8], xv[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const bool use = k < 4 ? k < cs.wo : (k - 4) < cs.wn;
        const int slot_k = k < 4 ? k : cs.wo + (k - 4);
        const int slot = cs.base + 32 * slot_k;
        fk[k] = use ? __ldg(L.slot_face + slot) : -1;
        const int col = use ? slot_column(L, cs.e0 + slot_k, slot, c) : -1;
        a[k] = use ? __ldg(coef + slot) : 0.0;
        xv[k] = (use && col >= 0) ? fetch(col) : 0.0;
      }
      int max_nei = -1, min_own = INT_MAX;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (fk[k] >= 0 && fk[k] < min_own) min_own = fk[k];
        if (fk[4 + k] > max_nei) max_nei = fk[4 + k];
      }
      if (max_nei < min_own) {
#pragma unroll
        for (int k = 4; k < 8; ++k)
          if (fk[k] >= 0) row = __dadd_rn(row, __dmul_rn(a[k], xv[k]));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (fk[k] >= 0) row = __dadd_rn(row, __dmul_rn(a[k], xv[k]));
        merged = true;
      }
    }
  }
  if (L.n_faces > 0 && !merged) {
    const CellSlots cs = cell_slots(L, c);
    int i = 0, j = 0;
    while (true) {
      int fi = INT_MAX, fj = INT_MAX;
      while (i < cs.wo && (fi = __ldg(L.slot_face + cs.base + 32 * i)) < 0) ++i;
      if (i >= cs.wo) fi = INT_MAX;
      while (j < cs.wn && (fj = __ldg(L.slot_face + cs.base + 32 * (cs.wo + j))) < 0) ++j;
      if (j >= cs.wn) fj = INT_MAX;
      if (fi == INT_MAX && fj == INT_MAX) break;
      const int k = fi < fj ? i : cs.wo + j;
      const int slot = cs.base + 32 * k;
      const int col = slot_column(L, cs.e0 + k, slot, c);
      row = __dadd_rn(row, __dmul_rn(__ldg(coef + slot), fetch(col)));
      if (fi < fj)
        ++i;
      else
        ++j;
    }
  }
  return row;
}

// The updated value of cell c from its row sum (the value itself when the
// diagonal is too small to divide by, as in the reference).
template <bool RELAX>
__device__ __forceinline__ double gs_update(double row, double dx, double dc, double xc, double bc,
                                            double omega) {
  const double off = __dsub_rn(row, dx);  // dx = dc * xc, rounded
  if (!above_tiny(fabs(dc))) return xc;
  const double nv = div_rn(__dsub_rn(bc, off), dc);
  return RELAX ? __dadd_rn(xc, __dmul_rn(omega, __dsub_rn(nv, xc))) : nv;
}

template <bool RELAX>
__device__ __forceinline__ void gs_cell(const gbf_layout& L, const double* __restrict__ coef,
                                        const double* __restrict__ diag,
                                        const double* __restrict__ b, int c, double omega,
                                        double* x) {
  const double dc = __ldg(diag + c);
  const double xc = __ldcg(x + c);
  const double row = gs_row(L, coef, dc, xc, c, [&](int col) { return __ldcg(x + col); });
  if (above_tiny(fabs(dc)))
    x[c] = gs_update<RELAX>(row, __dmul_rn(dc, xc), dc, xc, __ldg(b + c), omega);
}

template <bool RELAX>
__global__ void __launch_bounds__(kBlock)
    gs_level_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                    const double* __restrict__ b, const int32_t* __restrict__ level_ptr,
                    const int32_t* __restrict__ level_cells, int level, double omega,
                    double* x) {
  const int start = __ldg(level_ptr + level);
  const int count = __ldg(level_ptr + level + 1) - start;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) gs_cell<RELAX>(L, coef, diag, b, __ldg(level_cells + start + t), omega, x);
}

// A whole Gauss-Seidel sweep in one cooperative launch (wavefront.cuh).
template <bool RELAX>
__global__ void __launch_bounds__(kBlock)
    gs_coop_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                   const double* __restrict__ b, const int32_t* __restrict__ level_ptr,
                   const int32_t* __restrict__ level_cells, int n_levels, double omega,
                   double* x, GridBarrier* bar) {
  if (!run_levels(bar, level_ptr, n_levels, [&](int i) {
        gs_cell<RELAX>(L, coef, diag, b, __ldg(level_cells + i), omega, x);
      }))
    poison(x, L.n_cells);
}

// A whole Gauss-Seidel sweep as a dataflow walk (wavefront.cuh): the cells
// of the level schedule in level order, dealt 32 at a time round-robin to
// the warps of one block per SM.  The sweep reads the old values from x_old
// (never written during the walk) and writes the new ones into the slots
// x_new (initialised to the empty marker); a cell polls only the new values
// it reads -- its neighbours swept before it (lower-numbered forward,
// higher-numbered backward), which are at earlier levels -- so the warp
// holding the earliest unfinished cell always finds its inputs.
//
// What bounds it is the chain from one level to the next: the store, its
// neighbour's poll, and the FP64 operations between them, 64 clocks each (a
// CUDA divide 560).  So everything that does not need a new value happens
// before the wait -- loads, the products with old values -- a pass only polls
// what is still missing, and the last arrival is followed by the products with
// new values, the row's additions and one integer-pipe division.  Repeating
// gs_row on every pass instead took 5.1 us a level
// (67 x 59 x 53 cells: 902 us a sweep, 274 us now).  The products, their order
// and the update are gs_cell's (gs_row, gs_update): the same bits.  Cells with
// more than four slots a side, and cells whose owner-side faces do not all
// follow their neighbour-side faces, repeat gs_row.
//
// The row sum of a cell from its first N slots a side, for the whole warp at
// once without branches (an FP64 instruction that no lane needs would hold the
// warp all the same): the waited-for side's products, then the terms in order.
template <int N>
__device__ __forceinline__ double gs_finish(double row, const double (&pn)[4],
                                            const double (&po)[4], const double (&v)[4],
                                            unsigned used, unsigned wait, bool reverse) {
  double t[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double c = reverse ? po[k] : pn[k], p = __dmul_rn(c, v[k]);
    t[k] = (wait >> k & 1u) ? p : c;
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double s = __dadd_rn(row, reverse ? pn[k] : t[k]);
    row = (used >> k & 1u) ? s : row;
  }
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double s = __dadd_rn(row, reverse ? t[k] : po[k]);
    row = (used >> k & 16u) ? s : row;
  }
  return row;
}

// LOCAL: a block walk (wavefront.cuh), cells in the order of block_ptr.
template <bool RELAX, bool LOCAL>
__global__ void __launch_bounds__(kBlock)
    gs_flow_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                   const double* __restrict__ b, const int32_t* __restrict__ cells,
                   const int32_t* __restrict__ block_ptr, int per, int reverse, double omega,
                   const double* __restrict__ x_old, double* x_new, GridBarrier* bar,
                   long long max_polls) {
  extern __shared__ double dyn[];
  FlowSlots<LOCAL> slots;
  const FlowRange range = flow_begin<LOCAL>(slots, x_new, L.n_cells, block_ptr, per, dyn);
  const int lane = threadIdx.x & 31;
  long long polls = 0;
  for (long long at = range.first; at < range.end; at += range.stride) {
    const long long i = at + lane;
    bool done = i >= range.end;
    int c = 0;
    double dc = 0.0, xc = 0.0, bc = 0.0;
    // pn, po: coefficients of the neighbour- and owner-side slots, of old
    // values already times the value; `from` where a new value is polled
    bool ordered = false;
    unsigned used = 0, wait = 0;  // bit k: neighbour-side slot k, 4 + k: owner-side slot k
    double pn[4] = {}, po[4] = {}, v[4] = {}, dx = 0.0;
    const double* from[4] = {};
    int wo = 0, wn = 0;
    if (!done) {
      c = __ldg(cells + i);
      dc = __ldg(diag + c);
      xc = __ldg(x_old + c);
      bc = __ldg(b + c);
      ordered = L.n_faces == 0;
      if (L.n_faces > 0) {
        const CellSlots cs = cell_slots(L, c);
        if (cs.wo <= 4 && cs.wn <= 4) {
          wo = cs.wo;
          wn = cs.wn;
          int fn[4], fo[4], qn[4], qo[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int so = cs.base + 32 * k, sn = cs.base + 32 * (wo + k);
            fo[k] = k < wo ? __ldg(L.slot_face + so) : -1;
            fn[k] = k < wn ? __ldg(L.slot_face + sn) : -1;
            qo[k] = k < wo ? slot_column(L, cs.e0 + k, so, c) : -1;
            qn[k] = k < wn ? slot_column(L, cs.e0 + wo + k, sn, c) : -1;
            po[k] = k < wo ? __ldg(coef + so) : 0.0;
            pn[k] = k < wn ? __ldg(coef + sn) : 0.0;
          }
          // forward sweeps wait on the neighbour side, backward on the owner side
          bool usual = true;
          int max_nei = -1, min_own = INT_MAX;
          double xo[4], xn[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool un = fn[k] >= 0 && qn[k] >= 0, uo = fo[k] >= 0 && qo[k] >= 0;
            if (un) used |= 1u << k, max_nei = fn[k];
            if (uo) used |= 16u << k, min_own = min_own < fo[k] ? min_own : fo[k];
            const bool nn = un && (reverse ? qn[k] > c : qn[k] < c);
            const bool no = uo && (reverse ? qo[k] > c : qo[k] < c);
            if (reverse ? nn : no) usual = false;
            if (reverse ? no : nn) {
              wait |= 1u << k;
              from[k] = slots.at(reverse ? qo[k] : qn[k]);
            }
            xn[k] = un && !nn ? __ldg(x_old + qn[k]) : 1.0;
            xo[k] = uo && !no ? __ldg(x_old + qo[k]) : 1.0;
          }
          ordered = usual && max_nei < min_own;
          if (ordered) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              if (reverse || !(wait >> k & 1u)) pn[k] = __dmul_rn(pn[k], xn[k]);
              if (!reverse || !(wait >> k & 1u)) po[k] = __dmul_rn(po[k], xo[k]);
            }
          } else {
            wait = 0;
          }
        }
      }
      dx = __dmul_rn(dc, xc);
    }
    unsigned left = wait;
    const int most_n = __reduce_max_sync(0xffffffffu, wn);
    const int most_o = __reduce_max_sync(0xffffffffu, wo);
    bool quit = false;
    for (;;) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (left >> k & 1u) v[k] = slots.load(from[k]);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if ((left >> k & 1u) && !flow_empty(v[k])) left &= ~(1u << k);
      bool finish = ordered && !done && left == 0;
      if (__any_sync(0xffffffffu, finish)) {
        const double row =
            most_n <= 3 && most_o <= 3
                ? gs_finish<3>(dx, pn, po, v, used, wait, reverse)
                : gs_finish<4>(dx, pn, po, v, used, wait, reverse);
        // a lane that does not finish divides 1 by 1: an empty slot's NaN would
        // take the whole warp through the division's slow path
        const double nv = gs_update<RELAX>(finish ? row : dx, dx, finish ? dc : 1.0, xc,
                                           finish ? bc : 1.0, omega);
        if (finish) {
          slots.store(c, nv);
          done = true;
        }
      }
      if (!ordered && !done) {
        bool missing = false;
        const double row = gs_row(L, coef, dc, xc, c, [&](int col) {
          if (reverse ? col > c : col < c) {
            const double w = slots.load(slots.at(col));
            missing |= flow_empty(w);
            return w;
          }
          return __ldg(x_old + col);
        });
        if (!missing) {
          slots.store(c, gs_update<RELAX>(row, dx, dc, xc, bc, omega));
          done = true;
        }
      }
      if (flow_pass_end<!LOCAL>(done, polls, max_polls, bar, &quit)) break;
      if (quit) return;
    }
  }
}

// x = the new values, or NaN everywhere if a wait of the walk ran out.
__global__ void gs_flow_out_kernel(int n, const GridBarrier* bar, const double* __restrict__ x_new,
                                   double* __restrict__ x) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) x[c] = bar->fault != 0 ? __longlong_as_double(0x7ff8000000000000LL) : x_new[c];
}

// r_c = b_c - (A x)_c, or with SWEEP one damped Jacobi sweep
// x_c + (omega / max(|diag_c|, 1e-30)) r_c: residual_kernel's and
// relax_kernel's operations in their order.
template <bool SWEEP>
__device__ __forceinline__ double row_result(double ax, double bc, double dc, double xc,
                                             double omega) {
  const double r = __dsub_rn(bc, ax);
  if (!SWEEP) return r;
  const double inv = div_rn(1.0, max_abs_tiny(dc));
  return __dadd_rn(xc, __dmul_rn(omega == 1.0 ? inv : __dmul_rn(omega, inv), r));
}

// row_result of every cell, a thread per cell: out is not x.  A hex level is
// bound by the FP64 pipe (16 operations a cell; 262144 cells: residual 8.9 us,
// sweep 11.3 us, against 8.9 + 1.8 us of a sweep as two kernels with a
// division per cell in the second).
template <int KIND, bool SWEEP>
__global__ void __launch_bounds__(kBlock)
    cell_rows_kernel(gbf_layout L, const double* __restrict__ coef, const double* __restrict__ diag,
                     const double* __restrict__ b, double omega, const double* __restrict__ x,
                     double* __restrict__ out) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < L.n_cells; c += gridDim.x * blockDim.x) {
    const double xc = __ldg(x + c);
    const double ax = cell_amul_k<KIND, double, double, false>(L, coef, diag, x, c, xc);
    out[c] = row_result<SWEEP>(ax, __ldg(b + c), SWEEP ? __ldg(diag + c) : 1.0, xc, omega);
  }
}

// The same on a small layout of any other kind (coarse multigrid levels,
// random numberings), a block per 32-cell slice.  A thread per cell walks its
// row of 10-25 slots through a chain of loads (offset entry, column, x) and of
// FP64 operations, each of which holds the warp's SM quarter for 64 clocks: 10
// us a level however small.  Here the block's warps take the slots in turn
// (products into shared memory), so all of the slice's loads are in flight
// together, and then one warp sums the owner side and another the neighbour
// side in slot order -- the products and the order of cell_amul, so its bits:
// 1148 cells 10.2 -> 3.6 us, 8094 cells 9.8 -> 3.8, 32768 cells 10.0 -> 5.0 us a
// sweep.
// The two summing warps differ from block to block, so that the sums do not
// all fall on the same quarter of an SM.
constexpr int kRowSlots = 32;  // slots of a slice held at a time

template <bool SWEEP, int kRowWarps>
__global__ void __launch_bounds__(32 * kRowWarps)
    slice_rows_kernel(gbf_layout L, const double* __restrict__ coef,
                      const double* __restrict__ diag, const double* __restrict__ b, double omega,
                      const double* __restrict__ x, double* __restrict__ out) {
  __shared__ double prod[kRowSlots][32];
  __shared__ unsigned have[kRowSlots];
  __shared__ double sum_n[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int s = blockIdx.x, c = 32 * s + lane;
  const unsigned turn = (blockIdx.x * 2654435761u >> 16) & (kRowWarps - 2);
  const bool owner_sum = warp == (int)turn, neighbour_sum = warp == (int)turn + 1;
  const CellSlots cs = cell_slots(L, 32 * s + lane);
  double xc = 0.0, bc = 0.0, dc = 1.0;
  if (owner_sum && c < L.n_cells) {
    xc = __ldg(x + c);
    bc = __ldg(b + c);
    dc = __ldg(diag + c);
  }
  const int W = cs.wo + cs.wn;
  double sum = 0.0;
  for (int k0 = 0; k0 < W; k0 += kRowSlots) {
    const int cnt = W - k0 < kRowSlots ? W - k0 : kRowSlots;
    int col[kRowSlots / kRowWarps];
    double a[kRowSlots / kRowWarps];
#pragma unroll
    for (int j = 0; j < kRowSlots / kRowWarps; ++j) {
      const int k = warp + kRowWarps * j;
      col[j] = k < cnt ? __ldg(L.slot_col + cs.base + 32 * (k0 + k)) : -1;
      a[j] = k < cnt ? __ldg(coef + cs.base + 32 * (k0 + k)) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < kRowSlots / kRowWarps; ++j) {
      const int k = warp + kRowWarps * j;
      if (k >= cnt) break;
      prod[k][lane] = __dmul_rn(a[j], col[j] >= 0 ? __ldg(x + col[j]) : 0.0);
      const unsigned m = __ballot_sync(0xffffffffu, col[j] >= 0);
      if (lane == 0) have[k] = m;
    }
    __syncthreads();
    if (owner_sum || neighbour_sum) {
      const int from = owner_sum ? 0 : (cs.wo > k0 ? cs.wo - k0 : 0);
      const int to = owner_sum ? (cs.wo - k0 < cnt ? cs.wo - k0 : cnt) : cnt;
#pragma unroll 4
      for (int k = from; k < to; ++k) {
        const double v = __dadd_rn(sum, prod[k][lane]);
        sum = ((have[k] >> lane) & 1u) ? v : sum;
      }
    }
    __syncthreads();
  }
  if (neighbour_sum) sum_n[lane] = sum;
  __syncthreads();
  if (owner_sum && c < L.n_cells) {
    double ax = __dmul_rn(dc, xc);
    if (L.n_faces > 0) ax = __dadd_rn(__dadd_rn(ax, sum), sum_n[lane]);
    out[c] = row_result<SWEEP>(ax, bc, dc, xc, omega);
  }
}

// Which of the kernels, by the slices an SM has.  Eight warps a slice while the
// device holds them all at once (eight blocks an SM), four above.  From
// kRowThreadSlices on the device is full with a thread per cell too, and the
// products need no trip through shared memory: residual of 91125 renumbered
// cells (18.7 slices an SM) 8.9 us against 8.8, of 74088 (15.2) 6.8 against 8.6,
// of 125000 11.4 against 9.9, of 2097152 166 against 123, of the first coarse
// level of 200^3 332 against 200.  Not on slices so wide that a thread per cell
// waits for the longest row of its warp: 250000 cells of a graph, slices of 20
// slots in the mean and 155 at most, 31 us against 88; up to kRowThreadWidth the
// two are within a fifth of each other (64^3 with 12 more neighbours a cell,
// renumbered, widest slice 32, 40 against 49; 128^3 so, 34, 324 against 291).
constexpr int kRowFewSlices = 8, kRowThreadSlices = 18;  // an SM
constexpr int kRowThreadWidth = 40;

template <bool SWEEP>
static int launch_rows(const gbf_layout* L, const double* coef, const double* diag,
                       const double* b, double omega, const double* x, double* out,
                       cudaStream_t s) {
  int32_t sms = 0;
  const int rc = gbf_device_sm_count(&sms);
  if (rc) return rc;
  if (layout_kind(*L) == kLayoutHex33) {
    const int grid = wave_grid(cell_rows_kernel<kLayoutHex33, SWEEP>, kBlock, L->n_cells);
    cell_rows_kernel<kLayoutHex33, SWEEP>
        <<<grid, kBlock, 0, s>>>(*L, coef, diag, b, omega, x, out);
  } else if (L->n_slices > (int64_t)kRowThreadSlices * sms && L->max_width <= kRowThreadWidth) {
    const int grid = wave_grid(cell_rows_kernel<kLayoutGeneric, SWEEP>, kBlock, L->n_cells);
    cell_rows_kernel<kLayoutGeneric, SWEEP>
        <<<grid, kBlock, 0, s>>>(*L, coef, diag, b, omega, x, out);
  } else if (L->n_slices <= (int64_t)kRowFewSlices * sms) {
    slice_rows_kernel<SWEEP, 8><<<L->n_slices, 256, 0, s>>>(*L, coef, diag, b, omega, x, out);
  } else {
    slice_rows_kernel<SWEEP, 4><<<L->n_slices, 128, 0, s>>>(*L, coef, diag, b, omega, x, out);
  }
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

// x += (omega * s_c) * z with s_c = 1 / max(|diag_c|, 1e-30), or
// x += omega * z without a diagonal.
__global__ void __launch_bounds__(kBlock)
    relax_kernel(int n, double omega, const double* __restrict__ diag,
                 const double* __restrict__ z, double* __restrict__ x) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  double s = omega;
  if (diag) {
    s = __dmul_rn(omega, div_rn(1.0, max_abs_tiny(__ldg(diag + c))));
  }
  x[c] = __dadd_rn(x[c], __dmul_rn(s, __ldg(z + c)));
}

// out = x + a * y (one rounding each); out may alias x or y.
__global__ void __launch_bounds__(kBlock)
    xpay_kernel(int n, const double* x, double a, const double* y, double* out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) out[c] = __dadd_rn(x[c], __dmul_rn(a, y[c]));
}

// DiagonalSolver: x = b / max(|d|, 1e-30), r = b - d * x.
__global__ void __launch_bounds__(kBlock)
    diagonal_solve_kernel(int n, const double* __restrict__ d, const double* __restrict__ b,
                          double* __restrict__ x, double* __restrict__ r) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const double dc = __ldg(d + c), a = fabs(dc), bc = __ldg(b + c);
  const double xc = __ddiv_rn(bc, a > 1e-30 ? a : 1e-30);
  x[c] = xc;
  r[c] = __dsub_rn(bc, __dmul_rn(dc, xc));
}

// FvMatrix.relax: diag /= a; source += ((1 - a) * diag) * field_old, with
// one_minus_a = 1 - a computed by the caller in double.
__global__ void __launch_bounds__(kBlock)
    fv_relax_kernel(int n, double a, double one_minus_a, double* __restrict__ diag,
                    double* __restrict__ source, const double* __restrict__ old) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  const double d = __ddiv_rn(diag[c], a);
  diag[c] = d;
  source[c] = __dadd_rn(source[c], __dmul_rn(__dmul_rn(one_minus_a, d), __ldg(old + c)));
}

constexpr int kNormBlocks = 1024;

__global__ void __launch_bounds__(kBlock)
    dot_partials_kernel(int n, const double* __restrict__ a, const double* __restrict__ b,
                        double* __restrict__ partials) {
  __shared__ double sh[kBlock / 32];
  double s = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
    s = __fma_rn(__ldg(a + c), __ldg(b + c), s);
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kBlock)
    sum_partials_kernel(int g, const double* __restrict__ partials, double* __restrict__ out) {
  __shared__ double sh[kBlock / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < g; i += blockDim.x) s = __dadd_rn(s, partials[i]);
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *out = s;
}

__global__ void __launch_bounds__(kBlock)
    sumsq_partials_kernel(int n, const double* __restrict__ r, double* __restrict__ partials) {
  __shared__ double sh[kBlock / 32];
  double s = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const double v = __ldg(r + c);
    s = __fma_rn(v, v, s);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

// r = b - A x and the per-block sums of r^2 in one pass, over the cells and in
// the order of sumsq_partials_kernel.
template <int KIND>
__global__ void __launch_bounds__(kBlock)
    residual_sumsq_kernel(gbf_layout L, const double* __restrict__ coef,
                          const double* __restrict__ diag, const double* __restrict__ b,
                          const double* __restrict__ x, double* __restrict__ r,
                          double* __restrict__ partials) {
  __shared__ double sh[kBlock / 32];
  double s = 0.0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < L.n_cells; c += gridDim.x * blockDim.x) {
    const double v = __dsub_rn(
        __ldg(b + c), cell_amul_k<KIND, double, double, false>(L, coef, diag, x, c, __ldg(x + c)));
    r[c] = v;
    s = __fma_rn(v, v, s);
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = s;
}

__global__ void __launch_bounds__(kBlock)
    sqrt_sum_kernel(int g, const double* __restrict__ partials, double* __restrict__ out) {
  __shared__ double sh[kBlock / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < g; i += blockDim.x) s = __dadd_rn(s, partials[i]);
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *out = sqrt(s);
}

}  // namespace gbf

using namespace gbf;

extern "C" int gbf_gauss_seidel_f64(const gbf_layout* L, const double* coef, const double* diag,
                                    const double* b, const int32_t* level_ptr,
                                    const int32_t* level_cells, const int32_t* level_ptr_h,
                                    int32_t n_levels, double omega, int32_t relax, double* x,
                                    void* barrier, void* stream) {
  ::gbf::NvtxScope nvtx_("gbf_gauss_seidel_f64");
  int rc = check_layout(L);
  if (rc) return rc;
  if (L->n_cells == 0) return GBF_OK;
  GBF_REQUIRE(diag && b && x && level_ptr && level_cells && level_ptr_h && n_levels >= 0 &&
                  (L->n_faces == 0 || coef),
              "gauss_seidel: NULL pointer or bad level count");
  cudaStream_t s = as_stream(stream);
  int max_level = 0;
  for (int l = 0; l < n_levels; ++l) {
    const int cnt = level_ptr_h[l + 1] - level_ptr_h[l];
    if (cnt > max_level) max_level = cnt;
  }
  const void* coop = relax ? (const void*)gs_coop_kernel<true> : (const void*)gs_coop_kernel<false>;
  const int gc = (barrier && n_levels > 0) ? wavefront_grid(coop, kBlock, max_level, 2) : 0;
  if (gc > 0) {
    gbf_layout Lc = *L;
    int nl = n_levels;
    GridBarrier* bar = static_cast<GridBarrier*>(barrier);
    void* args[] = {&Lc, (void*)&coef, (void*)&diag, (void*)&b, (void*)&level_ptr,
                    (void*)&level_cells, &nl, &omega, &x, &bar};
    GBF_CHECK_CUDA(launch_wavefront(coop, gc, args, barrier, s));
    return GBF_OK;
  }
  for (int l = 0; l < n_levels; ++l) {
    const int cnt = level_ptr_h[l + 1] - level_ptr_h[l];
    if (cnt <= 0) continue;
    const int grid = (cnt + kBlock - 1) / kBlock;
    if (relax)
      gs_level_kernel<true><<<grid, kBlock, 0, s>>>(*L, coef, diag, b, level_ptr, level_cells, l,
                                                    omega, x);
    else
      gs_level_kernel<false><<<grid, kBlock, 0, s>>>(*L, coef, diag, b, level_ptr, level_cells,
                                                     l, omega, x);
  }
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

// The walk over the whole level schedule (block_ptr NULL), or by blocks.
static int gauss_seidel_walk(const char* what, const gbf_layout* L, const double* coef,
                             const double* diag, const double* b, const int32_t* cells,
                             const int32_t* block_ptr, int32_t n_blocks, int32_t per,
                             int32_t reverse, double omega, int32_t relax, double* x,
                             double* scratch, void* barrier, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells;
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(diag && b && x && cells && scratch && barrier && (L->n_faces == 0 || coef),
              "%s: NULL pointer", what);
  GBF_REQUIRE(scratch != x, "%s: scratch must not be x", what);
  cudaStream_t s = as_stream(stream);
  GBF_CHECK_CUDA(cudaMemsetAsync(scratch, 0xff, sizeof(double) * (size_t)n, s));
  gbf_layout Lc = *L;
  int rev = reverse != 0;
  long long polls = block_ptr ? walk_polls(n) : kFlowPolls;
  GridBarrier* bar = static_cast<GridBarrier*>(barrier);
  const double* xo = x;
  void* args[] = {&Lc, (void*)&coef, (void*)&diag, (void*)&b, (void*)&cells, (void*)&block_ptr,
                  &per, &rev, &omega, (void*)&xo, &scratch, &bar, &polls};
  if (block_ptr) {
    const void* k = relax ? (const void*)gs_flow_kernel<true, true>
                          : (const void*)gs_flow_kernel<false, true>;
    GBF_CHECK_CUDA(launch_walk(k, n_blocks, per, args, barrier, s));
  } else {
    const void* k = relax ? (const void*)gs_flow_kernel<true, false>
                          : (const void*)gs_flow_kernel<false, false>;
    // one block per SM (the polling of warps ahead of the front slows it)
    const int grid = wavefront_grid(k, kBlock, n, 1);
    GBF_REQUIRE(grid > 0, "%s: the device cannot launch cooperative kernels", what);
    GBF_CHECK_CUDA(launch_wavefront(k, grid, args, barrier, s));
  }
  gs_flow_out_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(n, bar, scratch, x);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_gauss_seidel_flow_f64(const gbf_layout* L, const double* coef,
                                         const double* diag, const double* b,
                                         const int32_t* level_cells, int32_t reverse,
                                         double omega, int32_t relax, double* x, double* scratch,
                                         void* barrier, void* stream) {
  ::gbf::NvtxScope nvtx_("gbf_gauss_seidel_flow_f64");
  return gauss_seidel_walk("gauss_seidel_flow", L, coef, diag, b, level_cells, nullptr, 0, 0,
                           reverse, omega, relax, x, scratch, barrier, stream);
}

extern "C" int gbf_gauss_seidel_block_f64(const gbf_layout* L, const double* coef,
                                          const double* diag, const double* b,
                                          const int32_t* block_cells, const int32_t* block_ptr,
                                          int32_t n_blocks, int32_t per, int32_t reverse,
                                          double omega, int32_t relax, double* x, double* scratch,
                                          void* barrier, void* stream) {
  ::gbf::NvtxScope nvtx_("gbf_gauss_seidel_block_f64");
  GBF_REQUIRE(L && block_ptr, "gauss_seidel_block: NULL pointer");
  GBF_REQUIRE(n_blocks >= 1 && per >= 1 && per <= kWalkCellsMax &&
                  (long long)n_blocks * per >= L->n_cells &&
                  (long long)(n_blocks - 1) * per < (L->n_cells > 0 ? L->n_cells : 1),
              "gauss_seidel_block: %d blocks of %d cells do not cover %d cells", n_blocks, per,
              L->n_cells);
  return gauss_seidel_walk("gauss_seidel_block", L, coef, diag, b, block_cells, block_ptr,
                           n_blocks, per, reverse, omega, relax, x, scratch, barrier, stream);
}

extern "C" int gbf_residual_f64(const gbf_layout* L, const double* coef, const double* diag,
                                const double* b, const double* x, double* r, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  if (L->n_cells == 0) return GBF_OK;
  GBF_REQUIRE(diag && b && x && r && (L->n_faces == 0 || coef), "residual: NULL pointer");
  cudaStream_t s = as_stream(stream);
  return launch_rows<false>(L, coef, diag, b, 1.0, x, r, s);
}

extern "C" int gbf_jacobi_f64(const gbf_layout* L, const double* coef, const double* diag,
                              const double* b, double omega, int32_t n_sweeps, double* x,
                              double* scratch, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  GBF_REQUIRE(n_sweeps >= 0, "jacobi: negative n_sweeps");
  if (L->n_cells == 0 || n_sweeps == 0) return GBF_OK;
  GBF_REQUIRE(diag && b && x && scratch && scratch != x && (L->n_faces == 0 || coef),
              "jacobi: NULL pointer, or scratch is x");
  cudaStream_t s = as_stream(stream);
  double *from = x, *to = scratch;
  for (int k = 0; k < n_sweeps; ++k) {
    rc = launch_rows<true>(L, coef, diag, b, omega, from, to, s);
    if (rc) return rc;
    double* t = from;
    from = to;
    to = t;
  }
  if (from != x)  // an odd number of sweeps ends in the scratch
    GBF_CHECK_CUDA(cudaMemcpyAsync(x, from, sizeof(double) * (size_t)L->n_cells,
                                   cudaMemcpyDeviceToDevice, s));
  return GBF_OK;
}

extern "C" int gbf_residual_norm2_f64(const gbf_layout* L, const double* coef, const double* diag,
                                      const double* b, const double* x, double* r, double* out,
                                      void* workspace, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells;
  GBF_REQUIRE(out && workspace && (n == 0 || (diag && b && x && r)) && (L->n_faces == 0 || coef),
              "residual_norm2: NULL pointer");
  cudaStream_t s = as_stream(stream);
  int g = (n + kBlock - 1) / kBlock;
  g = g < 1 ? 1 : (g > kNormBlocks ? kNormBlocks : g);
  double* partials = static_cast<double*>(workspace);
  GBF_LAYOUT_DISPATCH(*L, K, residual_sumsq_kernel<K><<<g, kBlock, 0, s>>>(*L, coef, diag, b, x, r,
                                                                           partials));
  GBF_CHECK_LAUNCH();
  sqrt_sum_kernel<<<1, kBlock, 0, s>>>(g, partials, out);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_relax_f64(int32_t n, double omega, const double* diag, const double* z,
                             double* x, void* stream) {
  GBF_REQUIRE(n >= 0, "relax: negative n");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(z && x, "relax: NULL pointer");
  relax_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(n, omega, diag, z, x);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" size_t gbf_norm2_workspace_bytes(void) { return sizeof(double) * kNormBlocks; }

extern "C" int gbf_norm2_f64(int32_t n, const double* r, double* out, void* workspace,
                             void* stream) {
  GBF_REQUIRE(n >= 0 && out && workspace && (n == 0 || r), "norm2: bad arguments");
  cudaStream_t s = as_stream(stream);
  int g = (n + kBlock - 1) / kBlock;
  g = g < 1 ? 1 : (g > kNormBlocks ? kNormBlocks : g);
  double* partials = static_cast<double*>(workspace);
  sumsq_partials_kernel<<<g, kBlock, 0, s>>>(n, r, partials);
  sqrt_sum_kernel<<<1, kBlock, 0, s>>>(g, partials, out);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_xpay_f64(int32_t n, const double* x, double a, const double* y, double* out,
                            void* stream) {
  GBF_REQUIRE(n >= 0, "xpay: negative n");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(x && y && out, "xpay: NULL pointer");
  xpay_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(n, x, a, y, out);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_dot_f64(int32_t n, const double* a, const double* b, double* out,
                           void* workspace, void* stream) {
  GBF_REQUIRE(n >= 0 && out && workspace && (n == 0 || (a && b)), "dot: bad arguments");
  cudaStream_t s = as_stream(stream);
  int g = (n + kBlock - 1) / kBlock;
  g = g < 1 ? 1 : (g > kNormBlocks ? kNormBlocks : g);
  double* partials = static_cast<double*>(workspace);
  dot_partials_kernel<<<g, kBlock, 0, s>>>(n, a, b, partials);
  sum_partials_kernel<<<1, kBlock, 0, s>>>(g, partials, out);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_diagonal_solve_f64(int32_t n, const double* diag, const double* b, double* x,
                                      double* r, void* stream) {
  GBF_REQUIRE(n >= 0, "diagonal_solve: negative n");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(diag && b && x && r, "diagonal_solve: NULL pointer");
  diagonal_solve_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(n, diag, b,
                                                                                   x, r);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_fv_relax_f64(int32_t n, double a, double one_minus_a, double* diag,
                                double* source, const double* field_old, void* stream) {
  GBF_REQUIRE(n >= 0, "fv_relax: negative n");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(diag && source && field_old, "fv_relax: NULL pointer");
  fv_relax_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n, a, one_minus_a, diag, source, field_old);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}
