// Rigid-body modes of the two-level preconditioner's coarse space, shared by
// the single-system PCG (solver.cu) and the batched PCG (batch.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "rowops.cuh"

namespace gfea {

template <int D>
struct Modes {
  static constexpr int nr = D == 1 ? 1 : (D == 2 ? 3 : 6);
};

// Rigid-body modes at one node (D x nr), rows of known DOFs zeroed.
// R holds exactly representable products of the float offsets, so the FP32
// and FP64 iterations apply the same modes.
template <int D, typename T = double>
__device__ __forceinline__ void node_modes(float4 o, const uint8_t* kn, T (&R)[D][Modes<D>::nr]) {
  if constexpr (D == 1) {
    R[0][0] = kn[0] ? T(0) : T(1);
  } else if constexpr (D == 2) {
    const T dx = o.x, dy = o.y;
    const T r0[3] = {1, 0, -dy}, r1[3] = {0, 1, dx};
    const bool k0 = kn[0], k1 = kn[1];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      R[0][m] = k0 ? T(0) : r0[m];
      R[1][m] = k1 ? T(0) : r1[m];
    }
  } else {
    const T dx = o.x, dy = o.y, dz = o.z;
    const T r0[6] = {1, 0, 0, 0, dz, -dy}, r1[6] = {0, 1, 0, -dz, 0, dx}, r2[6] = {0, 0, 1, dy, -dx, 0};
    const bool k0 = kn[0], k1 = kn[1], k2 = kn[2];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
      R[0][m] = k0 ? T(0) : r0[m];
      R[1][m] = k1 ? T(0) : r1[m];
      R[2][m] = k2 ? T(0) : r2[m];
    }
  }
}

// acc += R[:, m]^T x over the components x of a node at offset o (unmasked): the
// mode's non-zero products.
template <int D, typename T>
__host__ __device__ __forceinline__ void add_mode(DotAcc<T>& acc, int m, const T* o, const T* x) {
  if (D == 1 || m < D) {
    acc.add(x[m]);
  } else if constexpr (D == 2) {
    acc.add_prod(o[0], x[1]);
    acc.add_prod(-o[1], x[0]);
  } else if constexpr (D == 3) {
    const int a = m - 3, b = a == 2 ? 0 : a + 1, c = a == 0 ? 2 : a - 1;  // rotation about axis a
    acc.add_prod(o[b], x[c]);
    acc.add_prod(-o[c], x[b]);
  }
}

// Component k of R e at a node of offset o (unmasked; e: the coefficients of
// its aggregate's modes).
template <int D, typename T>
__device__ __forceinline__ T mode_row(int k, float4 o, const T* __restrict__ e) {
  if constexpr (D == 1) {
    return e[0];
  } else if constexpr (D == 2) {
    return k == 0 ? e[0] - (T)o.y * e[2] : e[1] + (T)o.x * e[2];
  } else {
    return k == 0   ? e[0] + ((T)o.z * e[4] - (T)o.y * e[5])
           : k == 1 ? e[1] + ((T)o.x * e[5] - (T)o.z * e[3])
                    : e[2] + ((T)o.y * e[3] - (T)o.x * e[4]);
  }
}

}  // namespace gfea
