// GAMG transfer kernels (solvers/gamg.py:249-393): Galerkin-style coarse
// coefficients, restriction by aggregate sums and prolongation by
// injection.  The aggregation itself depends on the mesh topology only and
// is built once on the host (gbf_gamg_aggregate, gbf_gamg_coarse_faces); the
// kernels here run per matrix and per V-cycle.  Every sum runs over its
// members in ascending index order, as the reference's scatter_add and its
// Python face loop do, so the coarse matrices and transfers are bitwise the
// reference's.
#include "amul.cuh"
#include "exact.cuh"

namespace gbf {

// dst[C] = (0 + src[i0]) + src[i1] + ... over the fine cells i of aggregate
// C in ascending order (scatter_add of the fine vector onto the aggregates).
__global__ void __launch_bounds__(kBlock)
    gamg_restrict_kernel(int n_coarse, const int32_t* __restrict__ ptr,
                         const int32_t* __restrict__ members, const double* __restrict__ src,
                         double* __restrict__ dst) {
  const int C = blockIdx.x * blockDim.x + threadIdx.x;
  if (C >= n_coarse) return;
  double s = 0.0;
  for (int k = __ldg(ptr + C), e = __ldg(ptr + C + 1); k < e; ++k)
    s = __dadd_rn(s, __ldg(src + __ldg(members + k)));
  dst[C] = s;
}

// Coarse lower/upper: the first fine face's value, then += every later fine
// face of the same aggregate pair in face order.
__global__ void __launch_bounds__(kBlock)
    gamg_coarse_coeff_kernel(int n_cfaces, const int32_t* __restrict__ ptr,
                             const int32_t* __restrict__ faces, const double* __restrict__ lower,
                             const double* __restrict__ upper, double* __restrict__ clower,
                             double* __restrict__ cupper) {
  const int K = blockIdx.x * blockDim.x + threadIdx.x;
  if (K >= n_cfaces) return;
  const int b = __ldg(ptr + K), e = __ldg(ptr + K + 1);
  const int f0 = __ldg(faces + b);
  double sl = __ldg(lower + f0), su = __ldg(upper + f0);
  for (int k = b + 1; k < e; ++k) {
    const int f = __ldg(faces + k);
    sl = __dadd_rn(sl, __ldg(lower + f));
    su = __dadd_rn(su, __ldg(upper + f));
  }
  clower[K] = sl;
  cupper[K] = su;
}

// x[i] = x[i] + e[f2c[i]]
__global__ void __launch_bounds__(kBlock)
    gamg_prolong_add_kernel(int n_fine, const int32_t* __restrict__ f2c,
                            const double* __restrict__ e, double* __restrict__ x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_fine) return;
  x[i] = __dadd_rn(x[i], __ldg(e + __ldg(f2c + i)));
}

// Restriction and the coarse correction's zero start.
__global__ void __launch_bounds__(kBlock)
    gamg_restrict_start_kernel(int n_coarse, const int32_t* __restrict__ ptr,
                               const int32_t* __restrict__ members,
                               const double* __restrict__ src, double* __restrict__ dst,
                               double* __restrict__ coarse_x) {
  const int C = blockIdx.x * blockDim.x + threadIdx.x;
  if (C >= n_coarse) return;
  double s = 0.0;
  for (int k = __ldg(ptr + C), e = __ldg(ptr + C + 1); k < e; ++k)
    s = __dadd_rn(s, __ldg(src + __ldg(members + k)));
  dst[C] = s;
  coarse_x[C] = 0.0;
}

// ---------------------------------------------------------------------------
// The coarse end of the V-cycle in one launch: pre-smoothing, residual,
// restriction, ... down to the coarsest level, its sweeps, and back up, for
// the levels of at most kTailCells cells.  As launches this end is all latency:
// a level of 50 cells costs the same 2-4 us a launch as one of 30000, and the
// coarsest level alone takes 50 sweeps of two launches.
//
// One block, x, a second x and b of every level and the rows in shared memory.
// What bounds it is the FP64 unit of an SM quarter, which takes 64 clocks per
// warp instruction whether or not the instructions depend on each other: the
// products of all slots are dealt to all threads, and two threads per cell sum
// its owner and its neighbour side at the same time, so a sweep of a level of
// few slots costs (slots of the longer side) + 6 such instructions.
// (Larger levels do better as launches over more SMs: 1148 cells took 8.7 us a
// sweep on eight blocks of a cluster, 4 us as a launch.)  Operations and
// orders are those of the separate kernels.
// ---------------------------------------------------------------------------
constexpr int kTailCells = 256;               // largest level taken
constexpr int kTailBlock = 2 * kTailCells;
constexpr int kTailLevels = 12;               // kernel-parameter space
constexpr int kTailTotal = 2 * kTailCells;    // cells of all its levels together
constexpr int kTailRows = 8192;               // slots staged in shared memory

struct TailLevels {
  gbf_gamg_level lv[kTailLevels];
  int off[kTailLevels];  // where the level's x, second x and b begin
  int row[kTailLevels];  // where its staged rows begin, -1: not staged
  int n;
};

// x, second x and b; staged coefficients, products and columns
constexpr size_t kTailSmem = sizeof(double) * 3 * kTailTotal +
                             (2 * sizeof(double) + sizeof(int32_t)) * kTailRows;

// A level as one thread sees it.
struct TailCell {
  int n, c, side;       // cells; this pair's cell (c >= n: none); 0 owner side, 1 neighbour side
  int i0, cnt;          // first slot and slots of the side
  double dc, s;         // diagonal, 1 / max(|diagonal|, 1e-30)
  double *x, *y, *b;    // current x, the other one, right-hand side
  const double* rc;     // rows: staged, or the level's own arrays
  const int32_t* rq;
  double* prod;         // products of staged rows, NULL: not staged
  int n_slots;
};

// b - A x of the pair's cell, in its even thread: cell_amul's products and
// order.  Called by the whole block.
__device__ __forceinline__ double tail_residual(const TailCell& t) {
  const bool mine = t.c < t.n;
  double s = 0.0;
  if (t.prod) {  // the same in every thread
    for (int i = threadIdx.x; i < t.n_slots; i += kTailBlock) {
      const int q = t.rq[i];
      if (q >= 0) t.prod[i] = __dmul_rn(t.rc[i], t.x[q]);
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < t.cnt; ++k) {
      const int i = t.i0 + 32 * k;
      const double v = __dadd_rn(s, t.prod[i]);
      s = t.rq[i] >= 0 ? v : s;
    }
  } else {
    for (int k = 0; k < t.cnt; ++k) {
      const int q = __ldg(t.rq + t.i0 + 32 * k);
      if (q >= 0) s = __dadd_rn(s, __dmul_rn(__ldg(t.rc + t.i0 + 32 * k), t.x[q]));
    }
  }
  __syncwarp();
  const double sn = __shfl_down_sync(0xffffffffu, s, 1);
  if (!mine || t.side) return 0.0;
  const double ax = __dadd_rn(__dadd_rn(__dmul_rn(t.dc, t.x[t.c]), s), sn);
  return __dsub_rn(t.b[t.c], ax);
}

__device__ __forceinline__ void tail_sweeps(TailCell& t, int n_sweeps) {
  for (int k = 0; k < n_sweeps; ++k) {
    const double r = tail_residual(t);
    if (t.c < t.n && t.side == 0) t.y[t.c] = __dadd_rn(t.x[t.c], __dmul_rn(t.s, r));
    __syncthreads();
    double* p = t.x;
    t.x = t.y;
    t.y = p;
  }
}

__global__ void __launch_bounds__(kTailBlock)
    gamg_tail_kernel(const __grid_constant__ TailLevels T, int n_pre, int n_post, int n_coarsest,
                     const double* __restrict__ b_top, double* __restrict__ x_top) {
  extern __shared__ double sh[];
  const int tid = threadIdx.x, last = T.n - 1;
  double* stage_c = sh + 3 * kTailTotal;
  double* stage_p = stage_c + kTailRows;
  int32_t* stage_q = reinterpret_cast<int32_t*>(stage_p + kTailRows);

  // after k sweeps the current x is the first or the second of the two
  auto cell = [&](int l, int k) {
    const gbf_gamg_level& v = T.lv[l];
    TailCell t;
    t.n = v.layout.n_cells;
    t.c = tid >> 1;
    t.side = tid & 1;
    t.x = sh + T.off[l] + ((k & 1) ? t.n : 0);
    t.y = sh + T.off[l] + ((k & 1) ? 0 : t.n);
    t.b = sh + T.off[l] + 2 * t.n;
    t.rc = T.row[l] >= 0 ? stage_c + T.row[l] : v.coef;
    t.rq = T.row[l] >= 0 ? stage_q + T.row[l] : v.layout.slot_col;
    t.prod = T.row[l] >= 0 ? stage_p + T.row[l] : nullptr;
    t.n_slots = (int)v.layout.n_slots;
    t.i0 = t.cnt = 0;
    t.dc = t.s = 1.0;
    if (t.c < t.n) {
      t.dc = __ldg(v.diag + t.c);
      t.s = div_rn(1.0, max_abs_tiny(t.dc));  // omega = 1
      if (v.layout.n_faces > 0) {
        const CellSlots cs = cell_slots(v.layout, t.c);
        t.i0 = cs.base + (t.side ? 32 * cs.wo : 0);
        t.cnt = t.side ? cs.wn : cs.wo;
      }
    }
    return t;
  };

  {
    const int n = T.lv[0].layout.n_cells;
    if (tid < n) {
      sh[tid] = x_top[tid];
      sh[2 * n + tid] = __ldg(b_top + tid);
    }
  }
  for (int l = 0; l <= last; ++l) {
    if (T.row[l] < 0) continue;
    const gbf_gamg_level& v = T.lv[l];
    const int n = (int)v.layout.n_slots;
#pragma unroll 4
    for (int i = tid; i < n; i += kTailBlock) {
      stage_c[T.row[l] + i] = __ldg(v.coef + i);
      stage_q[T.row[l] + i] = __ldg(v.layout.slot_col + i);
    }
  }
  __syncthreads();

  for (int l = 0; l < last; ++l) {  // down
    const gbf_gamg_level& v = T.lv[l];
    TailCell t = cell(l, 0);
    tail_sweeps(t, n_pre);
    const double r = tail_residual(t);
    if (t.c < t.n && t.side == 0) t.y[t.c] = r;
    __syncthreads();
    const int nc = v.n_coarse;
    if (tid < nc) {
      double s = 0.0;
      for (int k = __ldg(v.agg_ptr + tid), e = __ldg(v.agg_ptr + tid + 1); k < e; ++k)
        s = __dadd_rn(s, t.y[__ldg(v.agg_cells + k)]);
      sh[T.off[l + 1] + tid] = 0.0;
      sh[T.off[l + 1] + 2 * nc + tid] = s;
    }
    __syncthreads();
  }
  TailCell t = cell(last, 0);
  tail_sweeps(t, n_coarsest);
  const double* e = t.x;
  for (int l = last - 1; l >= 0; --l) {  // up
    TailCell w = cell(l, n_pre);
    if (tid < w.n) w.x[tid] = __dadd_rn(w.x[tid], e[__ldg(T.lv[l].f2c + tid)]);
    __syncthreads();
    tail_sweeps(w, n_post);
    e = w.x;
  }
  if (tid < T.lv[0].layout.n_cells) x_top[tid] = e[tid];
}

}  // namespace gbf

using namespace gbf;

extern "C" int gbf_gamg_restrict_start_f64(int32_t n_coarse, const int32_t* agg_ptr,
                                           const int32_t* agg_cells, const double* fine,
                                           double* coarse_b, double* coarse_x, void* stream) {
  GBF_REQUIRE(n_coarse >= 0, "gamg_restrict_start: negative n_coarse");
  if (n_coarse == 0) return GBF_OK;
  GBF_REQUIRE(agg_ptr && agg_cells && fine && coarse_b && coarse_x,
              "gamg_restrict_start: NULL pointer");
  gamg_restrict_start_kernel<<<(n_coarse + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_coarse, agg_ptr, agg_cells, fine, coarse_b, coarse_x);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

// 1 when gbf_gamg_tail_f64 takes these levels (fine first): their number,
// the largest and all of them together fit the block's shared memory.
extern "C" int gbf_gamg_tail_fits(int32_t n_levels, const int32_t* n_cells) {
  if (n_levels < 1 || n_levels > kTailLevels || !n_cells) return 0;
  long long total = 0;
  for (int l = 0; l < n_levels; ++l) {
    if (n_cells[l] < 0 || n_cells[l] > kTailCells) return 0;
    total += n_cells[l];
  }
  return total <= kTailTotal ? 1 : 0;
}

extern "C" int gbf_gamg_tail_f64(const gbf_gamg_level* levels, int32_t n_levels,
                                 int32_t n_pre_smooth, int32_t n_post_smooth,
                                 int32_t n_coarsest_sweeps, const double* b, double* x,
                                 void* stream) {
  GBF_REQUIRE(levels && n_levels >= 1 && n_levels <= kTailLevels, "gamg_tail: bad level count");
  GBF_REQUIRE(n_pre_smooth >= 0 && n_post_smooth >= 0 && n_coarsest_sweeps >= 0,
              "gamg_tail: negative sweep count");
  int32_t sizes[kTailLevels];
  TailLevels T;
  for (int l = 0; l < n_levels; ++l) {
    const gbf_gamg_level& v = levels[l];
    int rc = check_layout(&v.layout);
    if (rc) return rc;
    const bool coarsest = l == n_levels - 1;
    GBF_REQUIRE(v.layout.n_cells == 0 || (v.diag && (v.layout.n_faces == 0 || v.coef)),
                "gamg_tail: NULL matrix");
    GBF_REQUIRE(coarsest || (v.agg_ptr && v.agg_cells && v.f2c &&
                             v.n_coarse == levels[l + 1].layout.n_cells),
                "gamg_tail: level %d does not match its coarse level", l);
    sizes[l] = v.layout.n_cells;
    T.lv[l] = v;
  }
  GBF_REQUIRE(gbf_gamg_tail_fits(n_levels, sizes), "gamg_tail: the levels are too large");
  if (sizes[0] == 0) return GBF_OK;
  GBF_REQUIRE(b && x, "gamg_tail: NULL pointer");
  T.n = n_levels;
  int off = 0;
  for (int l = 0; l < n_levels; ++l, off += 3 * sizes[l - 1]) T.off[l] = off;
  // rows are staged from the coarsest level up, as far as they fit
  long long rows = 0;
  for (int l = n_levels - 1; l >= 0; --l) {
    const gbf_layout& L = T.lv[l].layout;
    T.row[l] = -1;
    if (L.n_faces == 0 || rows + L.n_slots > kTailRows) continue;
    T.row[l] = (int)rows;
    rows += L.n_slots;
  }
  GBF_CHECK_CUDA(cudaFuncSetAttribute(gamg_tail_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kTailSmem));
  gamg_tail_kernel<<<1, kTailBlock, kTailSmem, as_stream(stream)>>>(
      T, n_pre_smooth, n_post_smooth, n_coarsest_sweeps, b, x);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_gamg_restrict_f64(int32_t n_coarse, const int32_t* agg_ptr,
                                     const int32_t* agg_cells, const double* fine,
                                     double* coarse, void* stream) {
  GBF_REQUIRE(n_coarse >= 0, "gamg_restrict: negative n_coarse");
  if (n_coarse == 0) return GBF_OK;
  GBF_REQUIRE(agg_ptr && agg_cells && fine && coarse, "gamg_restrict: NULL pointer");
  gamg_restrict_kernel<<<(n_coarse + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_coarse, agg_ptr, agg_cells, fine, coarse);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_gamg_coarse_coeffs_f64(int32_t n_cfaces, const int32_t* cf_ptr,
                                          const int32_t* cf_faces, const double* lower,
                                          const double* upper, double* coarse_lower,
                                          double* coarse_upper, void* stream) {
  GBF_REQUIRE(n_cfaces >= 0, "gamg_coarse_coeffs: negative n_cfaces");
  if (n_cfaces == 0) return GBF_OK;
  GBF_REQUIRE(cf_ptr && cf_faces && lower && upper && coarse_lower && coarse_upper,
              "gamg_coarse_coeffs: NULL pointer");
  gamg_coarse_coeff_kernel<<<(n_cfaces + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_cfaces, cf_ptr, cf_faces, lower, upper, coarse_lower, coarse_upper);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_gamg_prolong_add_f64(int32_t n_fine, const int32_t* f2c, const double* e,
                                        double* x, void* stream) {
  GBF_REQUIRE(n_fine >= 0, "gamg_prolong_add: negative n_fine");
  if (n_fine == 0) return GBF_OK;
  GBF_REQUIRE(f2c && e && x, "gamg_prolong_add: NULL pointer");
  gamg_prolong_add_kernel<<<(n_fine + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_fine, f2c, e, x);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}
