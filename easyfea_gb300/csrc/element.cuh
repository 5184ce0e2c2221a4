// Element-matrix building blocks shared by the assembly kernels: the
// Kelvin-Mandel B_p^T C product and its contraction with B_q.
#pragma once

#include "common.cuh"

namespace gfea {
namespace {

constexpr double kInvSqrt2 = 0.70710678118654752440;

template <typename T>
__device__ __forceinline__ void atomic_add_t(T* p, T v) { atomicAdd(p, v); }

// B_p^T C scaled by wJ: BtC[i][s] = wJ * sum_r B_p[r][i] C[r][s]
// (Kelvin-Mandel B of EasyFEA/FEM/_group_elem.py:1242-1312)
template <int D, typename R>
__device__ __forceinline__ void btc(const R (&g)[D], const R* C, R wJ, R (&out)[D][D == 2 ? 3 : 6]) {
  const R c = (R)kInvSqrt2;
  if constexpr (D == 2) {
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      out[0][s] = wJ * (g[0] * C[0 * 3 + s] + c * g[1] * C[2 * 3 + s]);
      out[1][s] = wJ * (g[1] * C[1 * 3 + s] + c * g[0] * C[2 * 3 + s]);
    }
  } else {
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      out[0][s] = wJ * (g[0] * C[0 * 6 + s] + c * (g[2] * C[4 * 6 + s] + g[1] * C[5 * 6 + s]));
      out[1][s] = wJ * (g[1] * C[1 * 6 + s] + c * (g[2] * C[3 * 6 + s] + g[0] * C[5 * 6 + s]));
      out[2][s] = wJ * (g[2] * C[2 * 6 + s] + c * (g[1] * C[3 * 6 + s] + g[0] * C[4 * 6 + s]));
    }
  }
}

// acc[i][j] += sum_s BtC[i][s] B_q[s][j]
template <int D, typename R>
__device__ __forceinline__ void btcb(const R (&BtC)[D][D == 2 ? 3 : 6], const R (&h)[D], R (&acc)[D][D]) {
  const R c = (R)kInvSqrt2;
  if constexpr (D == 2) {
    const R chx = c * h[0], chy = c * h[1];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      acc[i][0] += BtC[i][0] * h[0] + BtC[i][2] * chy;
      acc[i][1] += BtC[i][1] * h[1] + BtC[i][2] * chx;
    }
  } else {
    const R chx = c * h[0], chy = c * h[1], chz = c * h[2];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      acc[i][0] += BtC[i][0] * h[0] + BtC[i][4] * chz + BtC[i][5] * chy;
      acc[i][1] += BtC[i][1] * h[1] + BtC[i][3] * chz + BtC[i][5] * chx;
      acc[i][2] += BtC[i][2] * h[2] + BtC[i][3] * chy + BtC[i][4] * chx;
    }
  }
}

// Jacobian F[d][k] = sum_q dN_d(q) X_q[k] over the nodes q = h, h + S, ... of
// this lane, then over the S lanes that share the point (a butterfly).
//
// Products are rounded and added in the order of a butterfly over
// NextPow2(nPe) lanes, a node each, as the lane-per-node kernels sum them:
// far from the origin the rounding of F is ~1e-13 (coordinates of 120 on
// elements of 0.3), and on a mesh of equal elements it does not average out --
// another order moved the displacement of a slender 132,000-unknown bar by
// 2e-9, several times its solver error.
template <int ELEM, bool MASS, int S>
__device__ __forceinline__ void point_jacobian(const RefTables<ELEM, MASS>& ref, int g, int h, const double* x,
                                               double (&F)[Elem<ELEM>::dim][Elem<ELEM>::dim]) {
  constexpr int D = Elem<ELEM>::dim, nPe = Elem<ELEM>::nPe, NQ = NextPow2<nPe>::value / S;
#pragma unroll
  for (int d = 0; d < D; ++d)
#pragma unroll
    for (int k = 0; k < D; ++k) {
      double t[NQ];
#pragma unroll
      for (int j = 0; j < NQ; ++j) {
        const int q = h + S * j;
        t[j] = (S * j < nPe && q < nPe) ? __dmul_rn(ref.dN[g][d][q < nPe ? q : 0], x[(q < nPe ? q : 0) * D + k]) : 0.0;
      }
#pragma unroll
      for (int o = NQ / 2; o > 0; o >>= 1)
#pragma unroll
        for (int l = 0; l < o; ++l)
          if (S * (l + o) < nPe) t[l] = __dadd_rn(t[l], t[l + o]);
#pragma unroll
      for (int o = S / 2; o > 0; o >>= 1) t[0] = __dadd_rn(t[0], __shfl_xor_sync(0xffffffffu, t[0], o));
      F[d][k] = t[0];
    }
}

// Gradients of the element's shape functions at a point of Jacobian F:
// out(q, i, dN_q / dx_i) for the nodes q = h, h + S, ...; returns det F.  The
// expressions are lane_geometry's, for the reason given at point_jacobian.
template <int ELEM, bool MASS, int S, typename O>
__device__ __forceinline__ double point_gradients(const RefTables<ELEM, MASS>& ref, int g, int h,
                                                  const double (&F)[Elem<ELEM>::dim][Elem<ELEM>::dim], O out) {
  constexpr int D = Elem<ELEM>::dim, nPe = Elem<ELEM>::nPe;
  if constexpr (D == 3 && NextPow2<nPe>::value == 8) {
    const double a11 = F[0][0], a12 = F[0][1], a13 = F[0][2], a21 = F[1][0], a22 = F[1][1], a23 = F[1][2],
                 a31 = F[2][0], a32 = F[2][1], a33 = F[2][2];
    const double c11 = a22 * a33 - a32 * a23, c21 = -(a21 * a33 - a31 * a23), c31 = a21 * a32 - a31 * a22;
    const double det = a11 * c11 + a12 * c21 + a13 * c31;
    const double id = recip_newton(det);
    const double adj[3][3] = {{c11, -(a12 * a33 - a32 * a13), a12 * a23 - a22 * a13},
                              {c21, a11 * a33 - a31 * a13, -(a11 * a23 - a21 * a13)},
                              {c31, -(a11 * a32 - a31 * a12), a11 * a22 - a21 * a12}};
#pragma unroll
    for (int q0 = 0; q0 < nPe; q0 += S) {
      const int q = q0 + h;
      if (nPe % S == 0 || q < nPe) {
        const double d0 = ref.dN[g][0][q], d1 = ref.dN[g][1][q], d2 = ref.dN[g][2][q];
#pragma unroll
        for (int i = 0; i < 3; ++i) out(q, i, id * (adj[i][0] * d0 + adj[i][1] * d1 + adj[i][2] * d2));
      }
    }
    return det;
  } else {
    double iF[D][D];
    const double det = det_inv<D>(F, iF);
#pragma unroll
    for (int q0 = 0; q0 < nPe; q0 += S) {
      const int q = q0 + h;
      if (nPe % S == 0 || q < nPe) {
#pragma unroll
        for (int i = 0; i < D; ++i) {
          double v = 0;
#pragma unroll
          for (int d = 0; d < D; ++d) v += iF[i][d] * ref.dN[g][d][q];
          out(q, i, v);
        }
      }
    }
    return det;
  }
}

// Adjugate and determinant of the Jacobian F[d][k]: the gradient of a field
// with reference gradient e is adj e / det.
template <int D>
__device__ __forceinline__ double adjugate(const double (&F)[D][D], double (&adj)[D][D]) {
  static_assert(D == 2 || D == 3, "plane or solid elements");
  if constexpr (D == 2) {
    adj[0][0] = F[1][1];
    adj[0][1] = -F[0][1];
    adj[1][0] = -F[1][0];
    adj[1][1] = F[0][0];
    return F[0][0] * F[1][1] - F[1][0] * F[0][1];
  } else {
    adj[0][0] = F[1][1] * F[2][2] - F[2][1] * F[1][2];
    adj[0][1] = F[2][1] * F[0][2] - F[0][1] * F[2][2];
    adj[0][2] = F[0][1] * F[1][2] - F[1][1] * F[0][2];
    adj[1][0] = F[2][0] * F[1][2] - F[1][0] * F[2][2];
    adj[1][1] = F[0][0] * F[2][2] - F[2][0] * F[0][2];
    adj[1][2] = F[1][0] * F[0][2] - F[0][0] * F[1][2];
    adj[2][0] = F[1][0] * F[2][1] - F[2][0] * F[1][1];
    adj[2][1] = F[2][0] * F[0][1] - F[0][0] * F[2][1];
    adj[2][2] = F[0][0] * F[1][1] - F[1][0] * F[0][1];
    return F[0][0] * adj[0][0] + F[0][1] * adj[1][0] + F[0][2] * adj[2][0];
  }
}

// Kelvin-Mandel strain from the reference gradient E[d][k] of u, the adjugate
// and 1 / det.
template <int D>
__device__ __forceinline__ void strain_of_gradient(const double (&adj)[D][D], const double (&E)[D][D], double id,
                                                   double* eps) {
  auto grad = [&](int i, int k) {  // du_k / dx_i, times det
    double t = adj[i][0] * E[0][k];
#pragma unroll
    for (int d = 1; d < D; ++d) t += adj[i][d] * E[d][k];
    return t;
  };
  const double c = id * kInvSqrt2;
#pragma unroll
  for (int i = 0; i < D; ++i) eps[i] = id * grad(i, i);
  if constexpr (D == 2) {
    eps[2] = c * (grad(1, 0) + grad(0, 1));
  } else {
    eps[3] = c * (grad(2, 1) + grad(1, 2));
    eps[4] = c * (grad(2, 0) + grad(0, 2));
    eps[5] = c * (grad(1, 0) + grad(0, 1));
  }
}

}  // namespace
}  // namespace gfea
