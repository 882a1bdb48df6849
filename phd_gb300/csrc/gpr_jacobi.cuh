// gpr_jacobi.cuh - small symmetric eigenproblems in registers.
#pragma once

#include "gpr_device.cuh"

namespace gpr {

// H = W diag(H) W^T by cyclic Jacobi rotations, H symmetric positive definite
// (its upper triangle is used, and holds the eigenvalues on the diagonal at
// the end).  A rotation's tangent only has to bring the entry down by a few
// digits, so it is taken in FP32 from the exact FP64 difference of the
// diagonal; cosine and sine are then formed in FP64, so each rotation is
// orthogonal to rounding, and the rotated entry keeps what is left of it.
// Entries below 6e-16 of the geometric mean of their diagonal, or below 2e-17 of
// the trace (a rounding of the largest entries), are skipped; the
// sweeps end when a whole sweep skipped (4 x 4 acoustic tensors: 3 - 5).  Returns
// false on a trace that is not positive and within 2^+-500, or without
// convergence.
template <int m> GPR_D bool jacobi_sym(double (&H)[m][m], double (&W)[m][m]) {
#pragma unroll
  for (int i = 0; i < m; i++)
#pragma unroll
    for (int j = 0; j < m; j++)
      W[i][j] = i == j ? 1.0 : 0.0;
  double tr = H[0][0];
#pragma unroll
  for (int i = 1; i < m; i++)
    tr += H[i][i];
  const int sh = fp_exponent(tr) - 1023;
  if (__double2hiint(tr) < 0 || sh < -500 || sh > 500)
    return false;
#pragma unroll 1
  for (int sweep = 0; sweep < 12; sweep++) {
    bool rotated = false;
#pragma unroll
    for (int p = 0; p < m - 1; p++)
#pragma unroll
      for (int q = p + 1; q < m; q++) {
        const float e = f32_scaled(H[p][q], sh);
        const float a = f32_scaled(H[p][p], sh), b = f32_scaled(H[q][q], sh);
        if (fabsf(e) <= 2e-17f || e * e <= 4e-31f * (a * b))
          continue;
        rotated = true;
        const float th = 0.5f * f32_scaled(H[q][q] - H[p][p], sh) * rcp32(e);
        const float tf = copysignf(rcp32(fabsf(th) + sqrt32(fmaf(th, th, 1.0f))), th);
        const double t = f64_scaled(tf, 0);
        const double c = rsqrt64(fma(t, t, 1.0)), s = c * t;
        const double u1 = fma(c, H[p][p], -(s * H[p][q])), u2 = fma(c, H[p][q], -(s * H[q][q]));
        const double u3 = fma(s, H[p][p], c * H[p][q]), u4 = fma(s, H[p][q], c * H[q][q]);
        H[p][p] = fma(c, u1, -(s * u2));
        H[p][q] = fma(s, u1, c * u2);
        H[q][q] = fma(s, u3, c * u4);
#pragma unroll
        for (int r = 0; r < m; r++) {
          if (r != p && r != q) {
            double &x = r < p ? H[r][p] : H[p][r], &y = r < q ? H[r][q] : H[q][r];
            const double xp = fma(c, x, -(s * y));
            y = fma(s, x, c * y);
            x = xp;
          }
          const double wp = fma(c, W[r][p], -(s * W[r][q]));
          W[r][q] = fma(s, W[r][p], c * W[r][q]);
          W[r][p] = wp;
        }
      }
    if (!rotated)
      return true;
  }
  return false;
}

}  // namespace gpr
