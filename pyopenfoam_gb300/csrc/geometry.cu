// Finite-volume mesh geometry on the GPU: face centres and area vectors,
// cell volumes and centres, interpolation weights and delta coefficients of
// a polyhedral mesh given as points + face-vertex lists + owner/neighbour.
//
// The formulas and their order of operations follow the reference's
// mesh/mesh_geometry.py:
//   face centre      = mean of the face's vertices            (:35-63)
//   face area vector = 1/2 sum_j v_j x v_{j+1}                (:66-108)
//   cell volume      = sum |tet(ref, fc, v_j, v_{j+1})| over the cell's
//                      faces, vertex order reversed on its neighbour-side
//                      faces; ref = mean of the cell's distinct vertices;
//                      centre = volume-weighted tet centroids  (:139-254)
//   weight           = |d_N| / (|d_P| + |d_N|), 1 on boundary   (:262-327)
//   delta            = 1 / |(C_N - C_P) . n_hat|, 0 on boundary (:330-395)
// with one thread per face or per cell instead of the reference's Python
// loops.  Every product and sum is explicitly rounded: face centres, area
// vectors are bitwise the reference's; cell volumes and centres (whose
// reference sums run over a Python set of vertex ids and a library dot
// product) agree to rounding.
//
// Nothing but arithmetic bounds these kernels: an FP64 instruction takes 64
// clocks of its SM quarter, so the products, quotients, roots and comparisons
// run on the integer pipe (exact.cuh, the same bits) beside the sums on the
// FP64 pipe, and an edge's vertex is moved to the cell's reference point once
// instead of twice.  64x48x40 hexahedra, before and after: cells 283 -> 175,
// faces 57 -> 32, interpolation 63 -> 18 us.
#include <math.h>

#include "common.cuh"
#include "exact.cuh"

namespace gbf {

constexpr int kMaxCellPoints = 64;

struct V3 {
  double x, y, z;
};

__device__ __forceinline__ V3 ld3(const double* __restrict__ p, int i) {
  return V3{__ldg(p + 3 * (size_t)i), __ldg(p + 3 * (size_t)i + 1), __ldg(p + 3 * (size_t)i + 2)};
}
__device__ __forceinline__ void st3(double* __restrict__ p, int i, V3 v) {
  p[3 * (size_t)i] = v.x;
  p[3 * (size_t)i + 1] = v.y;
  p[3 * (size_t)i + 2] = v.z;
}
__device__ __forceinline__ V3 add3(V3 a, V3 b) {
  return V3{__dadd_rn(a.x, b.x), __dadd_rn(a.y, b.y), __dadd_rn(a.z, b.z)};
}
__device__ __forceinline__ V3 sub3(V3 a, V3 b) {
  return V3{__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)};
}
__device__ __forceinline__ V3 scale3(V3 a, double s) {
  return V3{mul_int(a.x, s), mul_int(a.y, s), mul_int(a.z, s)};
}
__device__ __forceinline__ V3 div3(V3 a, double s) {
  return V3{div_rn(a.x, s), div_rn(a.y, s), div_rn(a.z, s)};
}
// a x b with each component rounded as fma(a_i, b_j, -(a_j b_i)), the
// rounding of ATen's CPU cross product (torch.linalg.cross).
__device__ __forceinline__ V3 cross3(V3 a, V3 b) {
  return V3{__fma_rn(a.y, b.z, -mul_int(a.z, b.y)),
            __fma_rn(a.z, b.x, -mul_int(a.x, b.z)),
            __fma_rn(a.x, b.y, -mul_int(a.y, b.x))};
}
__device__ __forceinline__ double dot3(V3 a, V3 b) {
  return __dadd_rn(__dadd_rn(mul_int(a.x, b.x), mul_int(a.y, b.y)), mul_int(a.z, b.z));
}
// |v| accumulated as sqrt(fma(z, z, fma(y, y, x*x))), the rounding of
// ATen's CPU p=2 norm over a length-3 row.
__device__ __forceinline__ double norm3(V3 v) {
  return sqrt_rn(__fma_rn(v.z, v.z, __fma_rn(v.y, v.y, mul_int(v.x, v.x))));
}

__global__ void __launch_bounds__(kBlock)
    face_geometry_kernel(int n_faces, const int32_t* __restrict__ face_ptr,
                         const int32_t* __restrict__ face_pts, const double* __restrict__ points,
                         double* __restrict__ centres, double* __restrict__ areas) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces) return;
  const int b = __ldg(face_ptr + f), nv = __ldg(face_ptr + f + 1) - b;
  V3 s{0.0, 0.0, 0.0};
  for (int j = 0; j < nv; ++j) s = add3(s, ld3(points, __ldg(face_pts + b + j)));
  st3(centres, f, div3(s, (double)nv));  // 0/0 = NaN for a face without vertices
  V3 a{0.0, 0.0, 0.0};
  if (nv >= 3) {
    V3 v0 = ld3(points, __ldg(face_pts + b));
    V3 vj = v0;
    for (int j = 0; j < nv; ++j) {
      const V3 vn = (j + 1 < nv) ? ld3(points, __ldg(face_pts + b + j + 1)) : v0;
      a = add3(a, cross3(vj, vn));
      vj = vn;
    }
    a = scale3(a, 0.5);
  }
  st3(areas, f, a);
}

// ---- cell -> face lists ------------------------------------------------------
// The order of the lists is the reference's visiting order: the owned faces
// ascending, then the neighboured ones (as ~face) ascending.  Five launches:
// counts, sums of 1024 counts, offsets, a fill in the order of arrival, and a
// ranking that puts every entry in its place.  An entry's rank is found by
// reading its cell's entries, one thread an entry: n loads of a line or two for
// a cell of n faces, so a cell with more than kRankMax faces is left to the
// host pass (status[1]).  64x48x40 hexahedra: 21 us, against 1360 us for the
// host pass and 750 us for its 32-bit copies of owner and neighbour.
constexpr unsigned int kRankMax = 4096;
constexpr int kScanCells = 1024;

// Faces whose cells lie outside [0, n_cells) are left out everywhere and the
// lowest is recorded in status[0] (0xffffffff: none).
__device__ __forceinline__ bool good_cell(int c, int n_cells) {
  return (unsigned int)c < (unsigned int)n_cells;
}

__global__ void __launch_bounds__(kBlock)
    list_count_kernel(int n_cells, int n_faces, int n_internal, const int64_t* __restrict__ owner,
                      const int64_t* __restrict__ neighbour, int32_t* __restrict__ own32,
                      int32_t* __restrict__ nei32, int32_t* __restrict__ count,
                      uint32_t* __restrict__ status) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces) return;
  const int o = (int)owner[f];
  own32[f] = o;
  bool good = good_cell(o, n_cells);
  if (good) atomicAdd(count + o, 1);
  if (f < n_internal) {
    const int m = (int)neighbour[f];
    nei32[f] = m;
    if (good_cell(m, n_cells))
      atomicAdd(count + m, 1);
    else
      good = false;
  }
  if (!good) atomicMin(status, (uint32_t)f);
}

__device__ __forceinline__ int block_sum_int(int v, int* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
#pragma unroll
  for (int w = 0; w < kBlock / 32; ++w) t += sh[w];
  return t;
}

__global__ void __launch_bounds__(kBlock)
    list_sums_kernel(int n_cells, const int32_t* __restrict__ count, int32_t* __restrict__ sums,
                     uint32_t* __restrict__ status) {
  __shared__ int sh[kBlock / 32];
  int v = 0, most = 0;
  for (int k = 0; k < kScanCells / kBlock; ++k) {
    const long long c = (long long)blockIdx.x * kScanCells + k * kBlock + threadIdx.x;
    const int n = c < n_cells ? count[c] : 0;
    v += n;
    most = max(most, n);
  }
  v = block_sum_int(v, sh);
  if (threadIdx.x == 0) sums[blockIdx.x] = v;
  most = __reduce_max_sync(0xffffffffu, most);
  if ((threadIdx.x & 31) == 0) atomicMin(status + 1, ~(uint32_t)most);
}

// cell_ptr, and in place of the counts the position of each cell's first entry.
__global__ void __launch_bounds__(kBlock)
    list_offsets_kernel(int n_cells, int32_t* __restrict__ count, const int32_t* __restrict__ sums,
                        int32_t* __restrict__ cell_ptr) {
  __shared__ int sh[kBlock / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int before = 0;
  for (int i = threadIdx.x; i < blockIdx.x; i += kBlock) before += sums[i];
  before = block_sum_int(before, sh);
  constexpr int K = kScanCells / kBlock;
  const long long c0 = (long long)blockIdx.x * kScanCells + K * threadIdx.x;
  int n[K], t = 0;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    n[k] = c0 + k < n_cells ? count[c0 + k] : 0;
    t += n[k];
  }
  int scan = t;  // inclusive over the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, scan, o);
    if (lane >= o) scan += up;
  }
  __syncthreads();  // sh: still read by the sum above
  if (lane == 31) sh[wid] = scan;
  __syncthreads();
  int at = before + scan - t;
  for (int w = 0; w < wid; ++w) at += sh[w];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if (c0 + k < n_cells) {
      cell_ptr[c0 + k] = at;
      count[c0 + k] = at;
      at += n[k];
      if (c0 + k == n_cells - 1) cell_ptr[n_cells] = at;
    }
  }
}

__global__ void __launch_bounds__(kBlock)
    list_fill_kernel(int n_cells, int n_faces, int n_internal, const int32_t* __restrict__ own32,
                     const int32_t* __restrict__ nei32, int32_t* __restrict__ at,
                     int32_t* __restrict__ entries) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces) return;
  const int o = own32[f];
  if (good_cell(o, n_cells)) entries[atomicAdd(at + o, 1)] = f;
  if (f < n_internal) {
    const int m = nei32[f];
    if (good_cell(m, n_cells)) entries[atomicAdd(at + m, 1)] = ~f;
  }
}

// Owned faces before neighboured ones, each ascending, as unsigned keys.
__device__ __forceinline__ uint32_t entry_key(int e) {
  return e >= 0 ? (uint32_t)e : ~(uint32_t)e | 0x80000000u;
}

__global__ void __launch_bounds__(kBlock)
    list_rank_kernel(int n_cells, int n_faces, int n_internal, const int32_t* __restrict__ own32,
                     const int32_t* __restrict__ nei32, const int32_t* __restrict__ cell_ptr,
                     const int32_t* __restrict__ entries, const uint32_t* __restrict__ status,
                     int32_t* __restrict__ cell_faces) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces || ~__ldg(status + 1) > kRankMax) return;
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    if (side == 1 && f >= n_internal) break;
    const int c = side == 0 ? own32[f] : nei32[f];
    if (!good_cell(c, n_cells)) continue;
    const int e = side == 0 ? f : ~f;
    const uint32_t key = entry_key(e);
    const int q0 = __ldg(cell_ptr + c), q1 = __ldg(cell_ptr + c + 1);
    int rank = 0;
    for (int q = q0; q < q1; ++q) rank += entry_key(__ldg(entries + q)) < key;
    cell_faces[q0 + rank] = e;
  }
}

// Vertex k of face f as seen from a cell: reversed order on the cell's
// neighbour-side faces (so that the face normal points out of the cell).
__device__ __forceinline__ int face_vertex(const int32_t* __restrict__ face_pts, int b, int nv,
                                           bool flip, int k) {
  return __ldg(face_pts + b + (flip ? nv - 1 - k : k));
}

__global__ void __launch_bounds__(128)
    cell_geometry_kernel(int n_cells, const int32_t* __restrict__ cell_ptr,
                         const int32_t* __restrict__ cell_faces,
                         const int32_t* __restrict__ face_ptr,
                         const int32_t* __restrict__ face_pts, const double* __restrict__ points,
                         const double* __restrict__ face_centres, double* __restrict__ volumes,
                         double* __restrict__ centres, int32_t* __restrict__ status) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n_cells) return;
  const int q0 = __ldg(cell_ptr + c), q1 = __ldg(cell_ptr + c + 1);
  if (q0 == q1) {  // a cell without faces keeps zero volume and centre
    volumes[c] = 0.0;
    st3(centres, c, V3{0.0, 0.0, 0.0});
    return;
  }
  // distinct vertices of the cell, ascending
  int pts[kMaxCellPoints];
  int np = 0;
  for (int q = q0; q < q1; ++q) {
    const int e = __ldg(cell_faces + q);
    const int f = e >= 0 ? e : ~e;
    const int b = __ldg(face_ptr + f), nv = __ldg(face_ptr + f + 1) - b;
    for (int k = 0; k < nv; ++k) {
      const int p = __ldg(face_pts + b + k);
      int i = 0;
      while (i < np && pts[i] < p) ++i;
      if (i < np && pts[i] == p) continue;
      if (np == kMaxCellPoints) {
        atomicExch(status, 1);
        volumes[c] = NAN;
        st3(centres, c, V3{NAN, NAN, NAN});
        return;
      }
      for (int j = np; j > i; --j) pts[j] = pts[j - 1];
      pts[i] = p;
      ++np;
    }
  }
  V3 ref{0.0, 0.0, 0.0};
  for (int i = 0; i < np; ++i) ref = add3(ref, ld3(points, pts[i]));
  ref = div3(ref, (double)np);

  double total = 0.0;
  V3 wc{0.0, 0.0, 0.0};
  for (int q = q0; q < q1; ++q) {
    const int e = __ldg(cell_faces + q);
    const bool flip = e < 0;
    const int f = flip ? ~e : e;
    const int b = __ldg(face_ptr + f), nv = __ldg(face_ptr + f + 1) - b;
    if (nv < 3) continue;
    const V3 fc = ld3(face_centres, f);
    const V3 bf = sub3(fc, ref);
    const V3 rf = add3(ref, fc);
    const V3 w0 = ld3(points, face_vertex(face_pts, b, nv, flip, 0));
    const V3 u0 = sub3(w0, ref);
    V3 wj = w0, uj = u0;
    for (int j = 0; j < nv; ++j) {
      V3 wn = w0, un = u0;
      if (j + 1 < nv) {
        wn = ld3(points, face_vertex(face_pts, b, nv, flip, j + 1));
        un = sub3(wn, ref);
      }
      const double av = fabs(div_rn(dot3(bf, cross3(uj, un)), 6.0));
      if (at_least(av, 1e-30)) {
        // a quarter is exact where a quotient by 4 is, and rounds as it does
        const V3 cen = scale3(add3(add3(rf, wj), wn), 0.25);
        total = __dadd_rn(total, av);
        wc = add3(wc, scale3(cen, av));
      }
      wj = wn;
      uj = un;
    }
  }
  if (fabs(total) > 1e-30) {
    volumes[c] = fabs(total);
    st3(centres, c, div3(wc, total));
  } else {  // degenerate cell: mean of its face centres
    V3 s{0.0, 0.0, 0.0};
    for (int q = q0; q < q1; ++q) {
      const int e = __ldg(cell_faces + q);
      s = add3(s, ld3(face_centres, e >= 0 ? e : ~e));
    }
    volumes[c] = 0.0;
    st3(centres, c, div3(s, (double)(q1 - q0)));
  }
}

__global__ void __launch_bounds__(kBlock)
    face_interp_kernel(int n_faces, int n_internal, const int32_t* __restrict__ owner,
                       const int32_t* __restrict__ neighbour,
                       const double* __restrict__ cell_centres,
                       const double* __restrict__ face_centres,
                       const double* __restrict__ face_areas, double* __restrict__ weights,
                       double* __restrict__ delta) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= n_faces) return;
  if (f >= n_internal) {
    weights[f] = 1.0;
    delta[f] = 0.0;
    return;
  }
  const V3 cp = ld3(cell_centres, __ldg(owner + f));
  const V3 cn = ld3(cell_centres, __ldg(neighbour + f));
  const V3 fc = ld3(face_centres, f);
  const double dP = norm3(sub3(fc, cp)), dN = norm3(sub3(fc, cn));
  const double den = __dadd_rn(dP, dN);
  weights[f] = div_rn(dN, above_tiny(den) ? den : 1.0);
  const V3 A = ld3(face_areas, f);
  const double am = norm3(A);
  const V3 nh = div3(A, above_tiny(am) ? am : 1.0);
  const double ddn = fabs(dot3(sub3(cn, cp), nh));
  delta[f] = div_rn(1.0, above_tiny(ddn) ? ddn : 1.0);
}

}  // namespace gbf

using namespace gbf;

extern "C" int gbf_face_geometry_f64(int32_t n_faces, const int32_t* face_ptr,
                                     const int32_t* face_pts, const double* points,
                                     double* face_centres, double* face_areas, void* stream) {
  GBF_REQUIRE(n_faces >= 0, "face_geometry: negative n_faces");
  if (n_faces == 0) return GBF_OK;
  GBF_REQUIRE(face_ptr && face_pts && points && face_centres && face_areas,
              "face_geometry: NULL pointer");
  face_geometry_kernel<<<(n_faces + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_faces, face_ptr, face_pts, points, face_centres, face_areas);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int64_t gbf_cell_faces_work_ints(int32_t n_cells, int32_t n_faces, int32_t n_internal) {
  return (int64_t)n_cells + (n_cells + kScanCells - 1) / kScanCells + n_faces + n_internal;
}

extern "C" int gbf_cell_faces_device(int32_t n_cells, int32_t n_faces, int32_t n_internal,
                                     const int64_t* owner, const int64_t* neighbour,
                                     int32_t* owner32, int32_t* neighbour32, int32_t* cell_ptr,
                                     int32_t* cell_faces, int32_t* work, uint32_t* status,
                                     void* stream) {
  GBF_REQUIRE(n_cells >= 1 && n_faces >= 1 && n_internal >= 0 && n_internal <= n_faces &&
                  (int64_t)n_faces + n_internal <= INT32_MAX,
              "cell_faces_device: bad counts");
  GBF_REQUIRE(owner && owner32 && cell_ptr && cell_faces && work && status &&
                  (n_internal == 0 || (neighbour && neighbour32)),
              "cell_faces_device: NULL pointer");
  cudaStream_t s = as_stream(stream);
  const int nb = (int)(((int64_t)n_cells + kScanCells - 1) / kScanCells);
  const int fb = (int)(((int64_t)n_faces + kBlock - 1) / kBlock);
  int32_t *count = work, *sums = work + n_cells, *entries = sums + nb;
  GBF_CHECK_CUDA(cudaMemsetAsync(count, 0, sizeof(int32_t) * (size_t)n_cells, s));
  GBF_CHECK_CUDA(cudaMemsetAsync(status, 0xff, 2 * sizeof(uint32_t), s));
  list_count_kernel<<<fb, kBlock, 0, s>>>(n_cells, n_faces, n_internal, owner, neighbour, owner32,
                                          neighbour32, count, status);
  list_sums_kernel<<<nb, kBlock, 0, s>>>(n_cells, count, sums, status);
  list_offsets_kernel<<<nb, kBlock, 0, s>>>(n_cells, count, sums, cell_ptr);
  list_fill_kernel<<<fb, kBlock, 0, s>>>(n_cells, n_faces, n_internal, owner32, neighbour32, count,
                                         entries);
  list_rank_kernel<<<fb, kBlock, 0, s>>>(n_cells, n_faces, n_internal, owner32, neighbour32,
                                         cell_ptr, entries, status, cell_faces);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_cell_geometry_f64(int32_t n_cells, const int32_t* cell_ptr,
                                     const int32_t* cell_faces, const int32_t* face_ptr,
                                     const int32_t* face_pts, const double* points,
                                     const double* face_centres, double* volumes,
                                     double* cell_centres, int32_t* status, void* stream) {
  GBF_REQUIRE(n_cells >= 0, "cell_geometry: negative n_cells");
  GBF_REQUIRE(status, "cell_geometry: NULL status");
  cudaStream_t s = as_stream(stream);
  GBF_CHECK_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), s));
  if (n_cells == 0) return GBF_OK;
  GBF_REQUIRE(cell_ptr && cell_faces && face_ptr && face_pts && points && face_centres &&
                  volumes && cell_centres,
              "cell_geometry: NULL pointer");
  cell_geometry_kernel<<<(n_cells + 127) / 128, 128, 0, s>>>(
      n_cells, cell_ptr, cell_faces, face_ptr, face_pts, points, face_centres, volumes,
      cell_centres, status);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_face_interp_f64(int32_t n_faces, int32_t n_internal, const int32_t* owner,
                                   const int32_t* neighbour, const double* cell_centres,
                                   const double* face_centres, const double* face_areas,
                                   double* weights, double* delta, void* stream) {
  GBF_REQUIRE(n_faces >= 0 && n_internal >= 0 && n_internal <= n_faces,
              "face_interp: bad face counts");
  if (n_faces == 0) return GBF_OK;
  GBF_REQUIRE(weights && delta && (n_internal == 0 || (owner && neighbour && cell_centres &&
                                                       face_centres && face_areas)),
              "face_interp: NULL pointer");
  face_interp_kernel<<<(n_faces + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_faces, n_internal, owner, neighbour, cell_centres, face_centres, face_areas, weights,
      delta);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}
