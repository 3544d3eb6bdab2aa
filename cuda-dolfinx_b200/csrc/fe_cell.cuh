// Coefficients and geometry of one affine tetrahedron, shared by the kernels
// that evaluate element tensors (fe_kernels.cu, fe_rows_vp2.cu).
#pragma once

#include <cuda_runtime.h>

#include "fe_internal.h"

namespace fe {
namespace {

struct CoefDev {
  int kind;            // fe_coeff_kind
  const double* v;     // DG0: [cells*ncomp]; P1: [nodes]
  const int32_t* map;  // P1: [cells*4]
  double c[3];         // constant
};

[[maybe_unused]] CoefDev to_dev(const Coefficient* c) {
  CoefDev d{};
  if (!c || c->kind < 0) {
    d.kind = FE_COEFF_CONSTANT;
    d.c[0] = d.c[1] = d.c[2] = 1.0;
    return d;
  }
  d.kind = c->kind;
  d.v = c->values;
  d.map = c->map ? c->map->dofs.p : nullptr;
  for (int i = 0; i < 3; ++i) d.c[i] = c->constant[i];
  return d;
}

// cellwise scalar value of a DG0 / constant coefficient
__device__ __forceinline__ double coef_cell(const CoefDev& k, int64_t c) {
  return k.kind == FE_COEFF_DG0 ? __ldg(k.v + c) : k.c[0];
}

// mean over the cell of a constant / DG0 / P1 coefficient (the exact factor of
// a P1 stiffness entry: the gradients are constant on the cell)
__device__ __forceinline__ double coef_mean(const CoefDev& k, int64_t c) {
  if (k.kind == FE_COEFF_P1) {
    const int4 m = __ldg(reinterpret_cast<const int4*>(k.map) + c);
    return 0.25 * ((__ldg(k.v + m.x) + __ldg(k.v + m.y)) + (__ldg(k.v + m.z) + __ldg(k.v + m.w)));
  }
  return coef_cell(k, c);
}

// ---------------------------------------------------------------------------
// Geometry of an affine tetrahedron: K = J^{-1}, |det J|
// ---------------------------------------------------------------------------
struct CellGeo {
  double K[3][3];
  double adet;
};

__device__ __forceinline__ void cell_geometry(const double* __restrict__ x, int4 v, CellGeo& g) {
  double x0[3], J[3][3];
  const int vv[3] = {v.y, v.z, v.w};
#pragma unroll
  for (int r = 0; r < 3; ++r) x0[r] = __ldg(x + 3 * (int64_t)v.x + r);
#pragma unroll
  for (int cc = 0; cc < 3; ++cc)
#pragma unroll
    for (int r = 0; r < 3; ++r) J[r][cc] = __ldg(x + 3 * (int64_t)vv[cc] + r) - x0[r];
  const double c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
  const double c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
  const double c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
  const double det = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
  const double id = 1.0 / det;
  g.K[0][0] = c00 * id;
  g.K[1][0] = c01 * id;
  g.K[2][0] = c02 * id;
  g.K[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) * id;
  g.K[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) * id;
  g.K[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) * id;
  g.K[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) * id;
  g.K[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) * id;
  g.K[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) * id;
  g.adet = fabs(det);
}

__device__ __forceinline__ int4 load_geom(const int32_t* __restrict__ geom, int64_t c) {
  return __ldg(reinterpret_cast<const int4*>(geom) + c);
}

// Ghat_s = adet * (K K^T)_s, s over (00,11,22,01,02,12)
__device__ __forceinline__ void ghat(const CellGeo& g, double G[6]) {
  const int pa[6] = {0, 1, 2, 0, 0, 1}, pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int s = 0; s < 6; ++s)
    G[s] = g.adet * (g.K[pa[s]][0] * g.K[pb[s]][0] + g.K[pa[s]][1] * g.K[pb[s]][1] +
                     g.K[pa[s]][2] * g.K[pb[s]][2]);
}

// P1 reference gradients dotted with K: grad phi_i = K^T ghat_i
__device__ __forceinline__ void p1_grads(const CellGeo& g, double G[4][3]) {
#pragma unroll
  for (int b = 0; b < 3; ++b) {
    G[1][b] = g.K[0][b];
    G[2][b] = g.K[1][b];
    G[3][b] = g.K[2][b];
    G[0][b] = -(g.K[0][b] + g.K[1][b] + g.K[2][b]);
  }
}

// W_ab[p][q] = |det| (mu (delta_ab (KK^T)_pq + K_pb K_qa) + lam K_pa K_qb), the
// geometric weights of component block (a, b) of the elasticity tensor
template <typename T>
__device__ __forceinline__ void elasticity_weights(const CellGeo& g, double lam, double mu, int a, int b,
                                                   T W[9]) {
#pragma unroll
  for (int p = 0; p < 3; ++p)
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      double kk = 0.0;
      if (a == b) kk = g.K[p][0] * g.K[q][0] + g.K[p][1] * g.K[q][1] + g.K[p][2] * g.K[q][2];
      W[p * 3 + q] = (T)(g.adet * (mu * (kk + g.K[p][b] * g.K[q][a]) + lam * g.K[p][a] * g.K[q][b]));
    }
}

}  // namespace
}  // namespace fe
