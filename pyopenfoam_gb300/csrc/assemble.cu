// Finite-volume assembly of the LDU coefficients:
//   fvm.laplacian (discretisation/operators.py:432-518) and
//   fvm.div with the upwind scheme (discretisation/operators.py:351-429).
//
// Face kernels write lower/upper in face order; cell kernels sum the
// diagonal with the same per-cell face order as the reference's
// scatter_add (owner-side faces ascending, then neighbour-side faces
// ascending, then boundary faces ascending), one rounding per operation, so
// the coefficients are bitwise identical to the reference's.
#include <math.h>

#include "common.cuh"
#include "exact.cuh"

namespace gbf {

// |S| of a face area vector as ATen's CPU p=2 norm over a length-3 row
// accumulates it: sqrt(fma(z, z, fma(y, y, x*x))).
__device__ __forceinline__ double face_smag(const double* __restrict__ a) {
  const double x = a[0], y = a[1], z = a[2];
  return sqrt_rn(__fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x))));
}

// Face diffusivity: constant, per face, or linearly interpolated from cells
// (LinearInterpolation.interpolate, interpolation.py:101-145:
//  w*phi_P + (1 - w)*phi_N on internal faces, phi_P on boundary faces).
struct DiffSpec {
  int mode;            // 0 constant, 1 per face, 2 per cell
  double value;        // mode 0
  const double* face;  // mode 1: [n_faces]
  const double* cell;  // mode 2: [n_cells]
  const double* w;     // mode 2: [n_faces] interpolation weights
};

__device__ __forceinline__ double face_D(const DiffSpec& D, int f, int p, int q, bool internal) {
  if (D.mode == 0) return D.value;
  if (D.mode == 1) return __ldg(D.face + f);
  const double dp = __ldg(D.cell + p);
  if (!internal) return dp;
  const double w = __ldg(D.w + f), v = __dsub_rn(1.0, w), dq = __ldg(D.cell + q);
  return __dadd_rn(mul_int(w, dp), mul_int(v, dq));
}

// (0 + sum over the cell's owner-side faces) + (sum over its neighbour-side
// faces, from 0) of own(f) / nei(f), faces in slot (= ascending) order.  The
// first term of a sum enters without an addition (first_term), and a sum that
// started at +0.0 is never -0.0, so adding it to 0.0 is the identity.  Up to
// four slots a side (hex and most polyhedral cells) have every face index and
// every face value of the cell in flight at once.
//
// M is the number of slots a side: an addition that no cell of the warp needs
// holds the FP64 pipe all the same, so slices of three (hex cells) have a body
// of their own; the widths are the slice's, so a warp takes one of them (497664
// hexahedra: lap_diag_kernel 25.7 -> 22.8 us, div_diag_kernel 18.3 -> 16.7 us;
// pressure_cell_kernel at 2097152, 105 -> 81 us).
template <int M, typename O, typename N>
__device__ __forceinline__ double few_face_sum(const gbf_layout& L, const CellSlots& cs, O&& own,
                                               N&& nei) {
  double so = 0.0, sn = 0.0, v[2 * M];
  int f[2 * M];
#pragma unroll
  for (int k = 0; k < M; ++k) {
    f[k] = k < cs.wo ? __ldg(L.slot_face + cs.base + 32 * k) : -1;
    f[M + k] = k < cs.wn ? __ldg(L.slot_face + cs.base + 32 * (cs.wo + k)) : -1;
  }
#pragma unroll
  for (int k = 0; k < M; ++k) {
    v[k] = f[k] >= 0 ? own(f[k]) : 0.0;
    v[M + k] = f[M + k] >= 0 ? nei(f[M + k]) : 0.0;
  }
  if (f[0] >= 0) so = first_term(v[0]);
  if (f[M] >= 0) sn = first_term(v[M]);
#pragma unroll
  for (int k = 1; k < M; ++k) {
    if (f[k] >= 0) so = __dadd_rn(so, v[k]);
    if (f[M + k] >= 0) sn = __dadd_rn(sn, v[M + k]);
  }
  return __dadd_rn(so, sn);
}

template <typename O, typename N>
__device__ __forceinline__ double cell_face_sum(const gbf_layout& L, int c, O&& own, N&& nei) {
  if (L.n_faces == 0) return 0.0;
  const CellSlots cs = cell_slots(L, c);
  if (cs.wo <= 3 && cs.wn <= 3) return few_face_sum<3>(L, cs, own, nei);
  if (cs.wo <= 4 && cs.wn <= 4) return few_face_sum<4>(L, cs, own, nei);
  double so = 0.0, sn = 0.0;
  for (int k = 0; k < cs.wo; ++k) {
    const int f = __ldg(L.slot_face + cs.base + 32 * k);
    if (f >= 0) so = __dadd_rn(so, own(f));
  }
  for (int k = 0; k < cs.wn; ++k) {
    const int f = __ldg(L.slot_face + cs.base + 32 * (cs.wo + k));
    if (f >= 0) sn = __dadd_rn(sn, nei(f));
  }
  return __dadd_rn(so, sn);
}

__global__ void __launch_bounds__(kBlock)
    lap_face_kernel(int nint, const int32_t* __restrict__ own, const int32_t* __restrict__ nei,
                    const double* __restrict__ areas, const double* __restrict__ delta,
                    DiffSpec D, const double* __restrict__ V, double* __restrict__ lower,
                    double* __restrict__ upper) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nint) return;
  const int p = __ldg(own + f), q = __ldg(nei + f);
  double c = __dmul_rn(face_D(D, f, p, q, true), face_smag(areas + 3 * (size_t)f));
  c = __dmul_rn(c, __ldg(delta + f));
  lower[f] = div_rn(-c, __ldg(V + p));
  upper[f] = div_rn(-c, __ldg(V + q));
}

// diag[c] = ((0 + sum_own c/V) + sum_nei c/V) + sum_bnd c_b/V, using
// c/V = -lower[f] (owner side) and -upper[f] (neighbour side) exactly.
__global__ void __launch_bounds__(kBlock)
    lap_diag_kernel(gbf_layout L, const double* __restrict__ lower,
                    const double* __restrict__ upper, const int32_t* __restrict__ bnd_ptr,
                    const int32_t* __restrict__ bnd_face, const double* __restrict__ areas,
                    const double* __restrict__ delta, DiffSpec D, const double* __restrict__ V,
                    int has_bnd, double* __restrict__ diag) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L.n_cells) return;
  double d = cell_face_sum(
      L, c, [&](int f) { return -__ldg(lower + f); }, [&](int f) { return -__ldg(upper + f); });
  if (has_bnd) {
    double sb = 0.0;
    const double vc = __ldg(V + c);
    for (int k = __ldg(bnd_ptr + c); k < __ldg(bnd_ptr + c + 1); ++k) {
      const int f = __ldg(bnd_face + k);
      double cb = __dmul_rn(face_D(D, f, c, c, false), face_smag(areas + 3 * (size_t)f));
      cb = __dmul_rn(cb, __ldg(delta + f));
      sb = __dadd_rn(sb, div_rn(cb, vc));
    }
    d = __dadd_rn(d, sb);
  }
  diag[c] = d;
}

// Upwind convection: F+ = F if F >= 0 else 0, F- = F if F < 0 else 0;
// lower = F-/V_P, upper = F+/V_N.
__global__ void __launch_bounds__(kBlock)
    div_face_kernel(int nint, const int32_t* __restrict__ own, const int32_t* __restrict__ nei,
                    const double* __restrict__ flux, const double* __restrict__ V,
                    double* __restrict__ lower, double* __restrict__ upper) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nint) return;
  const double F = __ldg(flux + f);
  const bool pos = not_negative(F);
  lower[f] = div_rn(pos ? 0.0 : F, __ldg(V + __ldg(own + f)));
  upper[f] = div_rn(pos ? F : 0.0, __ldg(V + __ldg(nei + f)));
}

// diag = (0 + sum_own (-F+)/V_P) + sum_nei |F-|/V_N
__global__ void __launch_bounds__(kBlock)
    div_diag_kernel(gbf_layout L, const double* __restrict__ flux, const double* __restrict__ V,
                    double* __restrict__ diag) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L.n_cells) return;
  const double vc = __ldg(V + c);
  diag[c] = cell_face_sum(
      L, c,
      [&](int f) {
        const double F = __ldg(flux + f);
        return div_rn(-(not_negative(F) ? F : 0.0), vc);
      },
      [&](int f) {
        const double F = __ldg(flux + f);
        return div_rn(fabs(not_negative(F) ? 0.0 : F), vc);
      });
}

// Linear-interpolation weights w = |d_N| / (|d_P| + |d_N|) of internal faces
// (weights.py:21-95), boundary faces 1; distances with the same fma norm.
__global__ void __launch_bounds__(kBlock)
    centre_weights_kernel(int nint, int nfaces, const int32_t* __restrict__ own,
                          const int32_t* __restrict__ nei, const double* __restrict__ cc,
                          const double* __restrict__ fc, double* __restrict__ w) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces) return;
  if (f >= nint) {
    w[f] = 1.0;
    return;
  }
  const int p = __ldg(own + f), q = __ldg(nei + f);
  double a[3], b[3];
  for (int k = 0; k < 3; ++k) {
    a[k] = __dsub_rn(__ldg(fc + 3 * (size_t)f + k), __ldg(cc + 3 * (size_t)p + k));
    b[k] = __dsub_rn(__ldg(fc + 3 * (size_t)f + k), __ldg(cc + 3 * (size_t)q + k));
  }
  const double dP = face_smag(a), dN = face_smag(b);
  const double den = __dadd_rn(dP, dN);
  w[f] = div_rn(dN, above_tiny(den) ? den : 1.0);
}

}  // namespace gbf

using namespace gbf;

static DiffSpec make_spec(int mode, double value, const double* Dface, const double* Dcell,
                          const double* w) {
  DiffSpec D;
  D.mode = mode;
  D.value = value;
  D.face = Dface;
  D.cell = Dcell;
  D.w = w;
  return D;
}

extern "C" int gbf_laplacian_assemble_f64(const gbf_layout* L, int32_t n_faces_total,
                                          const int32_t* owner_all, const int32_t* bnd_ptr,
                                          const int32_t* bnd_face, const double* face_areas,
                                          const double* delta, int32_t d_mode, double d_value,
                                          const double* d_face, const double* d_cell,
                                          const double* weights, const double* volumes,
                                          double* lower, double* upper, double* diag,
                                          void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells, nint = L->n_faces;
  GBF_REQUIRE(n_faces_total >= nint, "laplacian: n_faces_total < n_internal_faces");
  GBF_REQUIRE(d_mode >= 0 && d_mode <= 2, "laplacian: bad diffusivity mode %d", d_mode);
  GBF_REQUIRE(d_mode != 1 || d_face, "laplacian: per-face diffusivity is NULL");
  GBF_REQUIRE(d_mode != 2 || (d_cell && weights), "laplacian: per-cell diffusivity is NULL");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(diag && volumes && (n_faces_total == 0 || (face_areas && delta)),
              "laplacian: NULL pointer");
  const bool has_bnd = n_faces_total > nint;
  GBF_REQUIRE(!has_bnd || (bnd_ptr && bnd_face && owner_all), "laplacian: NULL boundary lists");
  const DiffSpec D = make_spec(d_mode, d_value, d_face, d_cell, weights);
  cudaStream_t s = as_stream(stream);
  if (nint > 0) {
    GBF_REQUIRE(lower && upper && L->owner && L->neighbour, "laplacian: NULL pointer");
    lap_face_kernel<<<(nint + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        nint, L->owner, L->neighbour, face_areas, delta, D, volumes, lower, upper);
    GBF_CHECK_LAUNCH();
  }
  lap_diag_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(
      *L, lower, upper, bnd_ptr, bnd_face, face_areas, delta, D, volumes, has_bnd ? 1 : 0, diag);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_div_upwind_assemble_f64(const gbf_layout* L, const double* flux,
                                           const double* volumes, double* lower, double* upper,
                                           double* diag, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells, nint = L->n_faces;
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(diag && volumes && (nint == 0 || (flux && lower && upper)),
              "div_upwind: NULL pointer");
  cudaStream_t s = as_stream(stream);
  if (nint > 0) {
    div_face_kernel<<<(nint + kBlock - 1) / kBlock, kBlock, 0, s>>>(nint, L->owner, L->neighbour,
                                                                    flux, volumes, lower, upper);
    GBF_CHECK_LAUNCH();
  }
  div_diag_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(*L, flux, volumes, diag);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_centre_weights_f64(int32_t n_internal, int32_t n_faces, const int32_t* owner,
                                      const int32_t* neighbour, const double* cell_centres,
                                      const double* face_centres, double* weights,
                                      void* stream) {
  GBF_REQUIRE(n_internal >= 0 && n_faces >= n_internal, "centre_weights: bad sizes");
  if (n_faces == 0) return GBF_OK;
  GBF_REQUIRE(weights && (n_internal == 0 || (owner && neighbour && cell_centres && face_centres)),
              "centre_weights: NULL pointer");
  centre_weights_kernel<<<(n_faces + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n_internal, n_faces, owner, neighbour, cell_centres, face_centres, weights);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

// ---------------------------------------------------------------------------
// Backward of the Laplacian assembly with respect to a per-face diffusivity.
// For an internal face c_f = D_f |S_f| delta_f enters lower_f = -c_f/V_P,
// upper_f = -c_f/V_N, diag_P += c_f/V_P, diag_N += c_f/V_N; a boundary face
// enters diag_P += c_f/V_P.  Hence
//   dL/dD_f = |S_f| delta_f ((g_diag_P - g_lower_f)/V_P + (g_diag_N - g_upper_f)/V_N)
//   dL/dD_b = |S_b| delta_b g_diag_P / V_P.
// One thread per face, no atomics.  (No reference counterpart as a kernel:
// the reference gets this from autograd through its torch ops.)
// ---------------------------------------------------------------------------
namespace gbf {
__global__ void __launch_bounds__(kBlock)
    lap_grad_gamma_kernel(int nint, int nfaces, const int32_t* __restrict__ own_all,
                          const int32_t* __restrict__ nei, const double* __restrict__ areas,
                          const double* __restrict__ delta, const double* __restrict__ V,
                          const double* __restrict__ gl, const double* __restrict__ gu,
                          const double* __restrict__ gd, double* __restrict__ gD) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces) return;
  const int p = __ldg(own_all + f);
  const double sd = face_smag(areas + 3 * (size_t)f) * __ldg(delta + f);
  double g = div_rn(__ldg(gd + p) - (f < nint ? __ldg(gl + f) : 0.0), __ldg(V + p));
  if (f < nint) {
    const int q = __ldg(nei + f);
    g += div_rn(__ldg(gd + q) - __ldg(gu + f), __ldg(V + q));
  }
  gD[f] = sd * g;
}

// DifferentiableLinearSolve.backward gradients
// (differentiable/linear_solver.py:139-149), reference rounding:
//   g_diag = (-lam)*x, g_lower_f = (-lam[own])*x[nei], g_upper_f = (-lam[nei])*x[own]
__global__ void __launch_bounds__(kBlock)
    dls_grad_kernel(int n, int nint, const int32_t* __restrict__ own,
                    const int32_t* __restrict__ nei, const double* __restrict__ lam,
                    const double* __restrict__ x, double* __restrict__ gd,
                    double* __restrict__ gl, double* __restrict__ gu) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) gd[i] = __dmul_rn(-__ldg(lam + i), __ldg(x + i));
  if (i < nint) {
    const int p = __ldg(own + i), q = __ldg(nei + i);
    gl[i] = __dmul_rn(-__ldg(lam + p), __ldg(x + q));
    gu[i] = __dmul_rn(-__ldg(lam + q), __ldg(x + p));
  }
}

// Fused adjoint face gradient of a Laplacian system A(D) x = b with respect
// to the per-face diffusivity, from the adjoint lam (A^T lam = dL/dx) and x:
// dL/dD_f = -lam^T (dA/dD_f) x
//         = |S| delta ((x_N - x_P)(lam_P/V_P - lam_N/V_N))   (internal)
//         = -|S| delta lam_P x_P / V_P                       (boundary)
// i.e. dls_grad followed by lap_grad_gamma without materialising the
// per-coefficient gradients.  `accumulate` adds into gD.
__global__ void __launch_bounds__(kBlock)
    adjoint_face_grad_kernel(int nint, int nfaces, const int32_t* __restrict__ own_all,
                             const int32_t* __restrict__ nei, const double* __restrict__ areas,
                             const double* __restrict__ delta, const double* __restrict__ V,
                             const double* __restrict__ lam, const double* __restrict__ x,
                             double scale, int accumulate, double* __restrict__ gD) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces) return;
  const int p = __ldg(own_all + f);
  const double sd = face_smag(areas + 3 * (size_t)f) * __ldg(delta + f);
  double g;
  if (f < nint) {
    const int q = __ldg(nei + f);
    g = (__ldg(x + q) - __ldg(x + p)) *
        (div_rn(__ldg(lam + p), __ldg(V + p)) - div_rn(__ldg(lam + q), __ldg(V + q)));
  } else {
    g = div_rn(-__ldg(lam + p) * __ldg(x + p), __ldg(V + p));
  }
  g = scale * sd * g;
  gD[f] = accumulate ? gD[f] + g : g;
}
}  // namespace gbf

extern "C" int gbf_laplacian_grad_gamma_f64(const gbf_layout* L, int32_t n_faces_total,
                                            const int32_t* owner_all, const double* face_areas,
                                            const double* delta, const double* volumes,
                                            const double* g_lower, const double* g_upper,
                                            const double* g_diag, double* g_gamma,
                                            void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  GBF_REQUIRE(n_faces_total >= L->n_faces, "laplacian_grad: n_faces_total < n_internal_faces");
  if (n_faces_total == 0) return GBF_OK;
  GBF_REQUIRE(owner_all && face_areas && delta && volumes && g_diag && g_gamma &&
                  (L->n_faces == 0 || (g_lower && g_upper && L->neighbour)),
              "laplacian_grad: NULL pointer");
  lap_grad_gamma_kernel<<<(n_faces_total + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      L->n_faces, n_faces_total, owner_all, L->neighbour, face_areas, delta, volumes, g_lower,
      g_upper, g_diag, g_gamma);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_dls_grads_f64(const gbf_layout* L, const double* lam, const double* x,
                                 double* g_diag, double* g_lower, double* g_upper, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells, nint = L->n_faces;
  const int m = n > nint ? n : nint;
  if (m == 0) return GBF_OK;
  GBF_REQUIRE(lam && x && g_diag && (nint == 0 || (g_lower && g_upper && L->owner)),
              "dls_grads: NULL pointer");
  dls_grad_kernel<<<(m + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      n, nint, L->owner, L->neighbour, lam, x, g_diag, g_lower, g_upper);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_adjoint_face_grad_f64(const gbf_layout* L, int32_t n_faces_total,
                                         const int32_t* owner_all, const double* face_areas,
                                         const double* delta, const double* volumes,
                                         const double* lam, const double* x, double scale,
                                         int32_t accumulate, double* g_gamma, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  GBF_REQUIRE(n_faces_total >= L->n_faces, "adjoint_face_grad: n_faces_total < n_internal");
  if (n_faces_total == 0) return GBF_OK;
  GBF_REQUIRE(owner_all && face_areas && delta && volumes && lam && x && g_gamma &&
                  (L->n_faces == 0 || L->neighbour),
              "adjoint_face_grad: NULL pointer");
  adjoint_face_grad_kernel<<<(n_faces_total + kBlock - 1) / kBlock, kBlock, 0,
                             as_stream(stream)>>>(L->n_faces, n_faces_total, owner_all,
                                                  L->neighbour, face_areas, delta, volumes, lam, x,
                                                  scale, accumulate, g_gamma);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

// ---------------------------------------------------------------------------
// DifferentiableLaplacian (differentiable/operators.py:409-643): the
// explicit Laplacian of a cell field and its backward.
//
// forward (:421-522), per cell c, faces in ascending order on each side:
//   flux_f = ((D_f * (phi_N - phi_P)) * |S_f|) * delta_f
//   lap = (0 + sum_own flux) + sum_nei (-flux)
//         [+ sum_bnd ((D_b * |S_b|) * delta_b) * phi_c]      (if boundary faces)
//   lap /= max(V_c, 1e-30)
// The phi-gradient of backward (:542-567) is the same operator applied to
// grad_output.  Each face flux is recomputed by both of its cells (same
// operands, same roundings), so the cell gather needs no scatter and no
// atomics.
// ---------------------------------------------------------------------------
namespace gbf {

__device__ __forceinline__ double clamp_volume(double v) {
  // v < 1e-30 on the integer pipe: every negative value, and the positive ones below 1e-30
  const long long b = __double_as_longlong(v), lo = __double_as_longlong(1e-30);
  const bool nan = (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
  return (b < lo && !nan) ? 1e-30 : v;
}

__global__ void __launch_bounds__(kBlock)
    explicit_lap_kernel(gbf_layout L, const int32_t* __restrict__ bnd_ptr,
                        const int32_t* __restrict__ bnd_face, const double* __restrict__ areas,
                        const double* __restrict__ delta, DiffSpec D,
                        const double* __restrict__ V, const double* __restrict__ phi,
                        int has_bnd, double* __restrict__ out) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L.n_cells) return;
  const double pc = __ldg(phi + c);
  double so = 0.0, sn = 0.0;
  if (L.n_faces > 0) {
    const CellSlots cs = cell_slots(L, c);
    for (int k = 0; k < cs.wo; ++k) {
      const int i = cs.base + 32 * k;
      const int f = __ldg(L.slot_face + i);
      if (f < 0) continue;
      const int q = __ldg(L.slot_col + i);
      double fl = __dmul_rn(face_D(D, f, c, q, true), __dsub_rn(__ldg(phi + q), pc));
      fl = mul_int(fl, face_smag(areas + 3 * (size_t)f));
      fl = mul_int(fl, __ldg(delta + f));
      so = __dadd_rn(so, fl);
    }
    for (int k = 0; k < cs.wn; ++k) {
      const int i = cs.base + 32 * (cs.wo + k);
      const int f = __ldg(L.slot_face + i);
      if (f < 0) continue;
      const int p = __ldg(L.slot_col + i);
      double fl = __dmul_rn(face_D(D, f, p, c, true), __dsub_rn(pc, __ldg(phi + p)));
      fl = mul_int(fl, face_smag(areas + 3 * (size_t)f));
      fl = mul_int(fl, __ldg(delta + f));
      sn = __dadd_rn(sn, -fl);
    }
  }
  double y = __dadd_rn(so, sn);
  if (has_bnd) {
    double sb = 0.0;
    for (int k = __ldg(bnd_ptr + c); k < __ldg(bnd_ptr + c + 1); ++k) {
      const int f = __ldg(bnd_face + k);
      double cb = __dmul_rn(face_D(D, f, c, c, false), face_smag(areas + 3 * (size_t)f));
      cb = __dmul_rn(cb, __ldg(delta + f));
      sb = __dadd_rn(sb, __dmul_rn(cb, pc));
    }
    y = __dadd_rn(y, sb);
  }
  out[c] = div_rn(y, clamp_volume(__ldg(V + c)));
}

// D-gradient per face (:570-600):
//   internal: (((g_P/V_P - g_N/V_N) * (phi_N - phi_P)) * |S|) * delta
//   boundary: (((g_P/V_P) * phi_P) * |S|) * delta
__global__ void __launch_bounds__(kBlock)
    explicit_lap_grad_d_kernel(int nint, int nfaces, const int32_t* __restrict__ own_all,
                               const int32_t* __restrict__ nei, const double* __restrict__ areas,
                               const double* __restrict__ delta, const double* __restrict__ V,
                               const double* __restrict__ phi, const double* __restrict__ g,
                               double* __restrict__ gface) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nfaces) return;
  const int p = __ldg(own_all + f);
  const double gp = div_rn(__ldg(g + p), clamp_volume(__ldg(V + p)));
  double a;
  if (f < nint) {
    const int q = __ldg(nei + f);
    const double gq = div_rn(__ldg(g + q), clamp_volume(__ldg(V + q)));
    a = __dmul_rn(__dsub_rn(gp, gq), __dsub_rn(__ldg(phi + q), __ldg(phi + p)));
  } else {
    a = __dmul_rn(gp, __ldg(phi + p));
  }
  a = __dmul_rn(a, face_smag(areas + 3 * (size_t)f));
  gface[f] = __dmul_rn(a, __ldg(delta + f));
}

// Per-cell D (:608-625): ((0 + sum_own gf*0.5) + sum_nei gf*0.5) [+ sum_bnd gf].
__global__ void __launch_bounds__(kBlock)
    face_grad_to_cells_kernel(gbf_layout L, const int32_t* __restrict__ bnd_ptr,
                              const int32_t* __restrict__ bnd_face,
                              const double* __restrict__ gface, int has_bnd,
                              double* __restrict__ gcell) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L.n_cells) return;
  double y = cell_face_sum(
      L, c, [&](int f) { return __dmul_rn(__ldg(gface + f), 0.5); },
      [&](int f) { return __dmul_rn(__ldg(gface + f), 0.5); });
  if (has_bnd) {
    double sb = 0.0;
    for (int k = __ldg(bnd_ptr + c); k < __ldg(bnd_ptr + c + 1); ++k)
      sb = __dadd_rn(sb, __ldg(gface + __ldg(bnd_face + k)));
    y = __dadd_rn(y, sb);
  }
  gcell[c] = y;
}

// Scalar D: the sum of the face gradients in one 1024-thread block, in a
// fixed order (strided per-thread sums, then the warp / block tree), so the
// result is reproducible run to run.
constexpr int kSumBlock = 1024;
__global__ void __launch_bounds__(kSumBlock)
    fixed_order_sum_kernel(int n, const double* __restrict__ a, double* __restrict__ out) {
  __shared__ double sh[kSumBlock / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += kSumBlock) s = __dadd_rn(s, __ldg(a + i));
  s = block_sum(s, sh);
  if (threadIdx.x == 0) *out = s;
}

}  // namespace gbf

extern "C" int gbf_explicit_laplacian_f64(const gbf_layout* L, int32_t n_faces_total,
                                          const int32_t* bnd_ptr, const int32_t* bnd_face,
                                          const double* face_areas, const double* delta,
                                          int32_t d_mode, double d_value, const double* d_face,
                                          const double* d_cell, const double* weights,
                                          const double* volumes, const double* phi, double* out,
                                          void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells, nint = L->n_faces;
  GBF_REQUIRE(n_faces_total >= nint, "explicit_laplacian: n_faces_total < n_internal_faces");
  GBF_REQUIRE(d_mode >= 0 && d_mode <= 2, "explicit_laplacian: bad diffusivity mode %d", d_mode);
  GBF_REQUIRE(d_mode != 1 || d_face, "explicit_laplacian: per-face diffusivity is NULL");
  GBF_REQUIRE(d_mode != 2 || (d_cell && (nint == 0 || weights)),
              "explicit_laplacian: per-cell diffusivity is NULL");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(volumes && phi && out && (n_faces_total == 0 || (face_areas && delta)),
              "explicit_laplacian: NULL pointer");
  const bool has_bnd = n_faces_total > nint;
  GBF_REQUIRE(!has_bnd || (bnd_ptr && bnd_face), "explicit_laplacian: NULL boundary lists");
  const DiffSpec D = make_spec(d_mode, d_value, d_face, d_cell, weights);
  explicit_lap_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, as_stream(stream)>>>(
      *L, bnd_ptr, bnd_face, face_areas, delta, D, volumes, phi, has_bnd ? 1 : 0, out);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}

extern "C" int gbf_explicit_laplacian_grad_d_f64(const gbf_layout* L, int32_t n_faces_total,
                                                 const int32_t* owner_all,
                                                 const int32_t* bnd_ptr, const int32_t* bnd_face,
                                                 const double* face_areas, const double* delta,
                                                 const double* volumes, const double* phi,
                                                 const double* g, double* g_face, double* g_cell,
                                                 double* g_sum, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int nint = L->n_faces;
  GBF_REQUIRE(n_faces_total >= nint, "explicit_laplacian_grad_d: n_faces_total < n_internal");
  cudaStream_t s = as_stream(stream);
  if (n_faces_total > 0) {
    GBF_REQUIRE(owner_all && face_areas && delta && volumes && phi && g && g_face &&
                    (nint == 0 || L->neighbour),
                "explicit_laplacian_grad_d: NULL pointer");
    explicit_lap_grad_d_kernel<<<(n_faces_total + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        nint, n_faces_total, owner_all, L->neighbour, face_areas, delta, volumes, phi, g, g_face);
    GBF_CHECK_LAUNCH();
  }
  const bool has_bnd = n_faces_total > nint;
  if (g_cell && L->n_cells > 0) {
    GBF_REQUIRE(!has_bnd || (bnd_ptr && bnd_face),
                "explicit_laplacian_grad_d: NULL boundary lists");
    face_grad_to_cells_kernel<<<(L->n_cells + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        *L, bnd_ptr, bnd_face, g_face, has_bnd ? 1 : 0, g_cell);
    GBF_CHECK_LAUNCH();
  }
  if (g_sum) {
    fixed_order_sum_kernel<<<1, kSumBlock, 0, s>>>(n_faces_total, g_face, g_sum);
    GBF_CHECK_LAUNCH();
  }
  return GBF_OK;
}

// ---------------------------------------------------------------------------
// Pressure equation (solvers/pressure_equation.py:49-148):
//   face_coeff = ((1/A_p)_f |S_f|) delta_f with (1/A_p)_f linearly
//   interpolated from 1/max(|A_p|, 1e-30) with the given face weights;
//   lower = -fc/V_P, upper = -fc/V_N; diag = (0 + sum_own fc/V_P) + sum_nei fc/V_N
//   (no boundary term); source = (((0 + sum_own -phi_f) + sum_nei phi_f)
//   [+ sum_bnd -phi_b]) / V.
// ---------------------------------------------------------------------------
namespace gbf {
// 1 / max(|A_p|, 1e-30) of every cell (pressure_equation.py:103-104; the clamp
// keeps NaN), which the faces interpolate.
__global__ void __launch_bounds__(kBlock)
    inv_diag_kernel(int n, const double* __restrict__ A, double* __restrict__ inv) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) inv[c] = div_rn(1.0, clamp_abs_min(__ldg(A + c)));
}

// The sums of pressure_cell_kernel for at most M slots a side (few_face_sum).
template <int M>
__device__ __forceinline__ void few_pressure_sums(const gbf_layout& L, const CellSlots& cs,
                                                  const double* __restrict__ lower,
                                                  const double* __restrict__ upper,
                                                  const double* __restrict__ phi, double& d,
                                                  double& y) {
  int f[2 * M];
  double v[2 * M], g[2 * M], vo = 0.0, vn = 0.0, go = 0.0, gn = 0.0;
#pragma unroll
  for (int k = 0; k < M; ++k) {
    f[k] = k < cs.wo ? __ldg(L.slot_face + cs.base + 32 * k) : -1;
    f[M + k] = k < cs.wn ? __ldg(L.slot_face + cs.base + 32 * (cs.wo + k)) : -1;
  }
#pragma unroll
  for (int k = 0; k < 2 * M; ++k) {
    v[k] = f[k] >= 0 ? -__ldg((k < M ? lower : upper) + f[k]) : 0.0;
    g[k] = f[k] >= 0 ? __ldg(phi + f[k]) : 0.0;
  }
  if (f[0] >= 0) vo = first_term(v[0]), go = first_term(-g[0]);
  if (f[M] >= 0) vn = first_term(v[M]), gn = first_term(g[M]);
#pragma unroll
  for (int k = 1; k < M; ++k) {
    if (f[k] >= 0) vo = __dadd_rn(vo, v[k]), go = __dsub_rn(go, g[k]);
    if (f[M + k] >= 0) vn = __dadd_rn(vn, v[M + k]), gn = __dadd_rn(gn, g[M + k]);
  }
  d = __dadd_rn(vo, vn);
  y = __dadd_rn(go, gn);
}

// diag and source in one pass over a cell's faces: one read of the face lists
// and all the face values of both sums in flight together (2097152 hexahedra:
// 81 us, against 63 + 56 us as two kernels).  Each sum is cell_face_sum's.
__global__ void __launch_bounds__(kBlock)
    pressure_cell_kernel(gbf_layout L, const double* __restrict__ lower,
                         const double* __restrict__ upper, const int32_t* __restrict__ bnd_ptr,
                         const int32_t* __restrict__ bnd_face, const double* __restrict__ phi,
                         const double* __restrict__ V, int has_bnd, double* __restrict__ diag,
                         double* __restrict__ src) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= L.n_cells) return;
  double d = 0.0, y = 0.0;
  if (L.n_faces > 0) {
    const CellSlots cs = cell_slots(L, c);
    if (cs.wo <= 3 && cs.wn <= 3) {
      few_pressure_sums<3>(L, cs, lower, upper, phi, d, y);
    } else if (cs.wo <= 4 && cs.wn <= 4) {
      few_pressure_sums<4>(L, cs, lower, upper, phi, d, y);
    } else {
      d = cell_face_sum(
          L, c, [&](int f) { return -__ldg(lower + f); },
          [&](int f) { return -__ldg(upper + f); });
      y = cell_face_sum(
          L, c, [&](int f) { return -__ldg(phi + f); }, [&](int f) { return __ldg(phi + f); });
    }
  }
  diag[c] = d;
  if (has_bnd) {
    double sb = 0.0;
    for (int k = __ldg(bnd_ptr + c); k < __ldg(bnd_ptr + c + 1); ++k)
      sb = __dadd_rn(sb, -__ldg(phi + __ldg(bnd_face + k)));
    y = __dadd_rn(y, sb);
  }
  src[c] = div_rn(y, __ldg(V + c));
}
}  // namespace gbf

extern "C" int gbf_pressure_assemble_f64(const gbf_layout* L, int32_t n_faces_total,
                                         const int32_t* bnd_ptr, const int32_t* bnd_face,
                                         const double* face_areas, const double* delta,
                                         const double* face_weights, const double* A_p,
                                         const double* volumes, const double* phiHbyA,
                                         double* lower, double* upper, double* diag,
                                         double* source, void* stream) {
  int rc = check_layout(L);
  if (rc) return rc;
  const int n = L->n_cells, nint = L->n_faces;
  GBF_REQUIRE(n_faces_total >= nint, "pressure_assemble: n_faces_total < n_internal_faces");
  if (n == 0) return GBF_OK;
  GBF_REQUIRE(A_p && volumes && diag && source && (n_faces_total == 0 || phiHbyA),
              "pressure_assemble: NULL pointer");
  const bool has_bnd = n_faces_total > nint;
  GBF_REQUIRE(!has_bnd || (bnd_ptr && bnd_face), "pressure_assemble: NULL boundary lists");
  // The inverse of A_p is formed once a cell, in diag until that is written,
  // and not twice a face: the face kernel is bound by the integer pipe, where
  // it divides (2097152 hexahedra: 151 us, now 11 + 126 us).
  const DiffSpec D = make_spec(2, 0.0, nullptr, diag, face_weights);
  cudaStream_t s = as_stream(stream);
  if (nint > 0) {
    GBF_REQUIRE(lower && upper && face_areas && delta && face_weights && L->owner &&
                    L->neighbour,
                "pressure_assemble: NULL pointer");
    inv_diag_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(n, A_p, diag);
    GBF_CHECK_LAUNCH();
    lap_face_kernel<<<(nint + kBlock - 1) / kBlock, kBlock, 0, s>>>(
        nint, L->owner, L->neighbour, face_areas, delta, D, volumes, lower, upper);
    GBF_CHECK_LAUNCH();
  }
  pressure_cell_kernel<<<(n + kBlock - 1) / kBlock, kBlock, 0, s>>>(
      *L, lower, upper, bnd_ptr, bnd_face, phiHbyA, volumes, has_bnd ? 1 : 0, diag, source);
  GBF_CHECK_LAUNCH();
  return GBF_OK;
}
