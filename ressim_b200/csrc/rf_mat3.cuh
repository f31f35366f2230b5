// rf_mat3.cuh — 3x3 block helpers of the block ILU0 and the CPR weights.
#pragma once

#include <cmath>

#include "rf_ops.hpp"

namespace rf {

__device__ __forceinline__ void mat3_mul(const double* a, const double* b, double* c) {
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int k = 0; k < 3; ++k) c[3 * r + k] = a[3 * r] * b[k] + a[3 * r + 1] * b[3 + k] + a[3 * r + 2] * b[6 + k];
}
// 3x3 inverse by cofactors; fails only on an exactly zero determinant, then the diagonal
// reciprocal fallback (gmres_block_jacobi.rs:888-901) is used.
__host__ __device__ __forceinline__ void mat3_inverse_or_diag(const double* m, double* o) {
  const double m11 = m[0], m12 = m[1], m13 = m[2], m21 = m[3], m22 = m[4], m23 = m[5], m31 = m[6], m32 = m[7],
               m33 = m[8];
  const double c11 = m22 * m33 - m32 * m23;
  const double c21 = m21 * m33 - m31 * m23;
  const double c31 = m21 * m32 - m31 * m22;
  const double det = m11 * c11 - m12 * c21 + m13 * c31;
  if (det != 0.0) {
    o[0] = c11 / det;
    o[1] = (m13 * m32 - m33 * m12) / det;
    o[2] = (m12 * m23 - m22 * m13) / det;
    o[3] = -c21 / det;
    o[4] = (m11 * m33 - m31 * m13) / det;
    o[5] = (m13 * m21 - m23 * m11) / det;
    o[6] = c31 / det;
    o[7] = (m12 * m31 - m32 * m11) / det;
    o[8] = (m11 * m22 - m21 * m12) / det;
    return;
  }
  for (int k = 0; k < 9; ++k) o[k] = 0.0;
  for (int d = 0; d < 3; ++d) {
    const double v = m[4 * d];
    o[4 * d] = fabs(v) > kF64Eps ? 1.0 / v : 1.0;
  }
}

}  // namespace rf
