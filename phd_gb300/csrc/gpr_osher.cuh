// gpr_osher.cuh - Osher-Solomon and Roe dissipation on the device
// (solvers/fv/fluxes.cpp:22-64): D = sum_i w_i |M(q_i)| (qL - qR) over the
// Gauss nodes of the straight path q_i = qR + x_i (qL - qR) (Osher), or
// |sum_i w_i M(q_i)| (qL - qR) (Roe), with M = dF/dQ + B the system matrix
// (system/equations.cpp:169-176) and |M| = R |Lambda| R^-1 from its real
// nonsymmetric eigen-decomposition.
//
// The eigen-decomposition (Householder Hessenberg reduction, Francis
// double-shift QR with accumulated Schur vectors, eigenvectors by
// back-substitution on the quasi-triangular Schur form; Golub & Van Loan,
// Matrix Computations, Alg. 7.4.2, 7.5.1-7.5.2) exists in two forms: per
// thread with the matrices in local memory (the pointwise entry points), and
// per warp with the matrices in shared memory (the face kernel).  Eigenvalues
// closer than MULT_TOL ||T|| are treated as one semisimple eigenvalue (their
// Schur vectors stay independent eigenvectors), which is how the reference's
// Eigen solver behaves on the GPR system's 9-fold advection eigenvalue.
#pragma once

#include "gpr_jacobi.cuh"
#include "gpr_kernels.cuh"

namespace gpr {

constexpr double OSH_MULT_TOL = 1e-12;

// System matrix M = dF_x/dP dP/dQ + B_x (system/jacobians.cpp:10-152, equations.cpp:69-87, 169-176):
// row-major V x V into M (ld = V).
// dF_x/dP into F and dP/dQ into D (V x V row-major, zeroed by the caller).
template <bool TH, int V>
GPR_D void system_fd(const double *Q, const Prim<TH> &s, const DevPar &P, double *F, double *D) {
  constexpr int d = 0;
#define RF(i, j) F[(i) * V + (j)]
#define RD(i, j) D[(i) * V + (j)]
  const double r = s.r, ir = s.ir;
  const double E = Q[1] * ir;
  const double p = s.p;
  const double *v = s.v;
  const double *A = Q + 5;
  const EosRho &e = s.e;
  // dE/drho at fixed p and dE/dp (mg.cpp:141-170, eos.cpp)
  const double rG = r * e.G, irG2 = s.irG * s.irG;
  const double dnum = e.dpr * rG + (e.G + r * e.dG) * (p - e.pr);
  const double dedr = e.der - dnum * irG2;
  const double Ep = s.irG;
  double dC0 = 0.0;
  if (P.beta != 0.0) {
    double dcs2 = P.beta * ir * s.cs2;
    dC0 = (1.0 - P.beta / e.G) * dcs2 + P.beta / (e.G * e.G) * e.dG * s.cs2;
  }
  const double Er = dedr + 0.25 * dC0 * s.devGsq;
  const double vd = v[d], rvd = r * vd;
  double G[9];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      G[3 * i + j] = A[i] * A[j] + A[3 + i] * A[3 + j] + A[6 + i] * A[6 + j];
  const double *AG = s.AdG;
  RF(0, 0) = vd;
  RF(0, 2 + d) = r;
  RF(1, 0) = (E + r * Er) * vd;
  RF(1, 1) = (r * Ep + 1.0) * vd;
#pragma unroll
  for (int i = 0; i < 3; i++)
    RF(1, 2 + i) = r * vd * v[i];
  RF(1, 2 + d) += r * E + p;
#pragma unroll
  for (int i = 0; i < 3; i++)
    RF(2 + i, 0) = vd * v[i];
#pragma unroll
  for (int i = 2; i < 5; i++)
    RF(i, i) = rvd;
#pragma unroll
  for (int i = 0; i < 3; i++)
    RF(2 + i, 2 + d) += r * v[i];
  RF(2 + d, 1) = 1.0;
  {
    double sg[3];
    sigma_col<TH>(Q, s, d, sg);
    const double fr = (1.0 + P.beta) * ir;  // 1/rho + dcs2/drho / cs2
    const double sr[3] = {fr * sg[0], fr * sg[1], fr * sg[2]};
    const double C0 = P.beta == 0.0 ? s.cs2
                                    : (P.EOS == 1 ? (1.0 - P.beta / e.G) : P.C0f) * s.cs2;
    const double cs2 = s.cs2;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const int ind = i * 3 + j;
        double tmp = 0.0;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          // dsigma_k / dA_ij (state.cpp:58-71) with ii = d, jj = k
          double t = A[3 * i + d] * G[3 * k + j] + A[3 * i + k] * G[3 * d + j] -
                     2.0 / 3.0 * G[3 * d + k] * A[3 * i + j];
          if (d == j)
            t += AG[3 * i + k];
          if (k == j)
            t += AG[3 * i + d];
          const double dsA = -r * cs2 * t;
          RF(2 + k, 5 + ind) = -dsA;
          tmp -= v[k] * dsA;
        }
        RF(1, 5 + ind) = tmp;
      }
    RF(1, 0) -= sr[0] * v[0] + sr[1] * v[1] + sr[2] * v[2];
#pragma unroll
    for (int i = 0; i < 3; i++)
      RF(1, 2 + i) -= sg[i];
#pragma unroll
    for (int i = 0; i < 9; i++)
      RF(1, 5 + i) += rvd * (C0 * AG[i]);
#pragma unroll
    for (int i = 0; i < 3; i++)
      RF(2 + i, 0) -= sr[i];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      RF(5 + d, 2 + j) = A[j];
      RF(8 + d, 2 + j) = A[3 + j];
      RF(11 + d, 2 + j) = A[6 + j];
      RF(5 + d, 5 + j) = v[j];
      RF(8 + d, 8 + j) = v[j];
      RF(11 + d, 11 + j) = v[j];
    }
    // dP/dQ (equations.cpp:130-167)
#pragma unroll
    for (int i = 0; i < V; i++)
      RD(i, i) = 1.0;
    const double G_ = 1.0 / (r * Ep);
    double tmpu = (v[0] * v[0] + v[1] * v[1] + v[2] * v[2]) - (E + r * Er);
    if (TH)
      tmpu += P.calpha2 * (s.J[0] * s.J[0] + s.J[1] * s.J[1] + s.J[2] * s.J[2]);
    RD(1, 0) = G_ * tmpu;
    RD(1, 1) = G_;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      RD(1, 2 + i) = -G_ * v[i];
      RD(2 + i, 0) = -v[i] * ir;
    }
#pragma unroll
    for (int i = 2; i < 5; i++)
      RD(i, i) = ir;
#pragma unroll
    for (int i = 0; i < 9; i++)
      RD(1, 5 + i) = -G_ * r * (C0 * AG[i]);
  }
  if (TH) {
    const double ca2 = P.calpha2;
    const double T = s.T;
    const double Tr = -dnum * irG2 * P.icv;
    const double Tp = Ep * P.icv;
    const double *J = s.J;
    const double H[3] = {ca2 * Q[14] * ir, ca2 * Q[15] * ir, ca2 * Q[16] * ir};
    RF(1, 0) += Tr * H[d];
    RF(1, 1) += Tp * H[d];
#pragma unroll
    for (int i = 0; i < 3; i++)
      RF(1, 14 + i) = rvd * H[i];
    RF(1, 14 + d) += ca2 * T;
#pragma unroll
    for (int i = 0; i < 3; i++)
      RF(14 + i, 0) = v[d] * J[i];
    RF(14 + d, 0) += Tr;
    RF(14 + d, 1) = Tp;
#pragma unroll
    for (int i = 0; i < 3; i++)
      RF(14 + i, 2 + d) = r * J[i];
#pragma unroll
    for (int i = 14; i < 17; i++)
      RF(i, i) = rvd;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      RD(1, 14 + i) = -(1.0 / (r * Ep)) * (ca2 * Q[14 + i] * ir);
      RD(14 + i, 0) = -J[i] * ir;
    }
#pragma unroll
    for (int i = 14; i < 17; i++)
      RD(i, i) = ir;
  }
#undef RF
#undef RD
}

// M += the non-conservative block B_x (equations.cpp:69-87)
template <int V, int LSET> GPR_D void system_block(const double *v, double *M) {
  constexpr int d = 0;
#pragma unroll
  for (int i = 5; i < 14; i++)
    M[i * V + i] += v[d];
  // the level sets are advected: v_d on their diagonal (equations.cpp:85-86)
#pragma unroll
  for (int i = V - LSET; i < V; i++)
    M[i * V + i] += v[d];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    M[(5 + d) * V + 5 + i] -= v[i];
    M[(8 + d) * V + 8 + i] -= v[i];
    M[(11 + d) * V + 11 + i] -= v[i];
  }
}

template <bool TH, int V>
GPR_D void system_matrix(const double *Q, const Prim<TH> &s, const DevPar &P, double *M) {
  double F[V * V], D[V * V];
#pragma unroll 1
  for (int i = 0; i < V * V; i++) {
    F[i] = 0.0;
    D[i] = 0.0;
  }
  system_fd<TH, V>(Q, s, P, F, D);
#pragma unroll 1
  for (int i = 0; i < V; i++)
#pragma unroll 1
    for (int j = 0; j < V; j++) {
      double acc = 0.0;
#pragma unroll 1
      for (int k = 0; k < V; k++)
        acc += F[i * V + k] * D[k * V + j];
      M[i * V + j] = acc;
    }
  system_block<V, V - 14 - (TH ? 3 : 0)>(s.v, M);
}

// Householder reduction of H (n x n, ld n) to upper Hessenberg form,
// accumulating the transformations into Z.
template <int n> GPR_D void hess_reduce(double *H, double *Z) {
#pragma unroll 1
  for (int k = 0; k < n - 2; k++) {
    // no reflection when the column below the subdiagonal is zero to the
    // least normal number (Eigen's makeHouseholder rule, which the
    // reference's EigenSolver follows): a reflector built from subnormal
    // entries would divide by an underflowed norm
    double tail = 0.0;
#pragma unroll 1
    for (int i = k + 2; i < n; i++)
      tail += H[i * n + k] * H[i * n + k];
    if (tail <= DBL_MIN_NORMAL)
      continue;
    double alpha = 0.0;
#pragma unroll 1
    for (int i = k + 1; i < n; i++)
      alpha += H[i * n + k] * H[i * n + k];
    alpha = sqrt(alpha);
    if (alpha == 0.0)
      continue;
    const double x0 = H[(k + 1) * n + k];
    const double beta = x0 > 0 ? -alpha : alpha;
    double vv = (x0 - beta) * (x0 - beta);
#pragma unroll 1
    for (int i = k + 2; i < n; i++)
      vv += H[i * n + k] * H[i * n + k];
    if (vv == 0.0)
      continue;
    double v[n];
#pragma unroll 1
    for (int i = 0; i <= k; i++)
      v[i] = 0.0;
    v[k + 1] = x0 - beta;
#pragma unroll 1
    for (int i = k + 2; i < n; i++)
      v[i] = H[i * n + k];
    const double tau = 2.0 / vv;
#pragma unroll 1
    for (int j = 0; j < n; j++) {
      double s = 0.0;
#pragma unroll 1
      for (int i = k + 1; i < n; i++)
        s += v[i] * H[i * n + j];
      s *= tau;
#pragma unroll 1
      for (int i = k + 1; i < n; i++)
        H[i * n + j] -= s * v[i];
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double s = 0.0;
#pragma unroll 1
      for (int j = k + 1; j < n; j++)
        s += H[i * n + j] * v[j];
      s *= tau;
#pragma unroll 1
      for (int j = k + 1; j < n; j++)
        H[i * n + j] -= s * v[j];
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double s = 0.0;
#pragma unroll 1
      for (int j = k + 1; j < n; j++)
        s += Z[i * n + j] * v[j];
      s *= tau;
#pragma unroll 1
      for (int j = k + 1; j < n; j++)
        Z[i * n + j] -= s * v[j];
    }
#pragma unroll 1
    for (int i = k + 2; i < n; i++)
      H[i * n + k] = 0.0;
  }
}

// Francis double-shift QR on the upper Hessenberg H to real Schur form,
// transformations accumulated into Z; eigenvalues to (wr, wi).  Returns
// false if it does not converge within 60 n iterations.
template <int n> GPR_D bool hqr_schur(double *H, double *Z, double *wr, double *wi) {
  const double eps = 2.220446049250313e-16;
  double norm = 0.0;
#pragma unroll 1
  for (int i = 0; i < n; i++)
#pragma unroll 1
    for (int j = (i > 0 ? i - 1 : 0); j < n; j++)
      norm += fabs(H[i * n + j]);
  int hi = n - 1, iter = 0, total = 0;
  double exshift = 0.0;
  while (hi >= 0) {
    int l = hi;
    while (l > 0) {
      double s = fabs(H[(l - 1) * n + l - 1]) + fabs(H[l * n + l]);
      if (s == 0.0)
        s = norm;
      if (fabs(H[l * n + l - 1]) < eps * s)
        break;
      l--;
    }
    if (l == hi) {  // one root
      H[hi * n + hi] += exshift;
      wr[hi] = H[hi * n + hi];
      wi[hi] = 0.0;
      if (hi > 0)
        H[hi * n + hi - 1] = 0.0;
      hi--;
      iter = 0;
      continue;
    }
    double x = H[hi * n + hi];
    double y = H[(hi - 1) * n + hi - 1];
    double w = H[hi * n + hi - 1] * H[(hi - 1) * n + hi];
    if (l == hi - 1) {  // two roots
      if (hi >= 2)
        H[(hi - 1) * n + hi - 2] = 0.0;
      double p = 0.5 * (y - x);
      double q = p * p + w;
      // a complex pair with a rounding-level imaginary part is a real
      // double root (a semisimple eigenvalue split by rounding)
      if (q < 0.0 && sqrt(-q) <= OSH_MULT_TOL * norm)
        q = 0.0;
      double z = sqrt(fabs(q));
      H[hi * n + hi] = x + exshift;
      H[(hi - 1) * n + hi - 1] = y + exshift;
      x = H[hi * n + hi];
      if (q >= 0.0) {
        z = p >= 0 ? p + z : p - z;
        wr[hi - 1] = x + z;
        wr[hi] = z != 0.0 ? x - w / z : x + z;
        wi[hi - 1] = wi[hi] = 0.0;
        const double xx = H[hi * n + hi - 1];
        const double s = fabs(xx) + fabs(z);
        double pp = xx / s, qq = z / s;
        const double rr = sqrt(pp * pp + qq * qq);
        pp /= rr;
        qq /= rr;
#pragma unroll 1
        for (int j = hi - 1; j < n; j++) {
          const double a = H[(hi - 1) * n + j];
          H[(hi - 1) * n + j] = qq * a + pp * H[hi * n + j];
          H[hi * n + j] = qq * H[hi * n + j] - pp * a;
        }
#pragma unroll 1
        for (int i = 0; i <= hi; i++) {
          const double a = H[i * n + hi - 1];
          H[i * n + hi - 1] = qq * a + pp * H[i * n + hi];
          H[i * n + hi] = qq * H[i * n + hi] - pp * a;
        }
#pragma unroll 1
        for (int i = 0; i < n; i++) {
          const double a = Z[i * n + hi - 1];
          Z[i * n + hi - 1] = qq * a + pp * Z[i * n + hi];
          Z[i * n + hi] = qq * Z[i * n + hi] - pp * a;
        }
        H[hi * n + hi - 1] = 0.0;
      } else {
        wr[hi - 1] = wr[hi] = x + p;
        wi[hi - 1] = z;
        wi[hi] = -z;
      }
      hi -= 2;
      iter = 0;
      continue;
    }
    if (iter == 10 || iter == 20) {  // exceptional shift
      exshift += x;
#pragma unroll 1
      for (int i = 0; i <= hi; i++)
        H[i * n + i] -= x;
      const double s = fabs(H[hi * n + hi - 1]) + fabs(H[(hi - 1) * n + hi - 2]);
      x = y = 0.75 * s;
      w = -0.4375 * s * s;
    }
    iter++;
    total++;
    if (total > 60 * n)
      return false;
    int m = hi - 2;
    double p = 0, q = 0, r = 0, z;
    while (m >= l) {
      z = H[m * n + m];
      r = x - z;
      double s = y - z;
      p = (r * s - w) / H[(m + 1) * n + m] + H[m * n + m + 1];
      q = H[(m + 1) * n + m + 1] - z - r - s;
      r = H[(m + 2) * n + m + 1];
      s = fabs(p) + fabs(q) + fabs(r);
      p /= s;
      q /= s;
      r /= s;
      if (m == l)
        break;
      const double u = fabs(H[m * n + m - 1]) * (fabs(q) + fabs(r));
      const double vv =
          fabs(p) * (fabs(H[(m - 1) * n + m - 1]) + fabs(z) + fabs(H[(m + 1) * n + m + 1]));
      if (u < eps * vv)
        break;
      m--;
    }
#pragma unroll 1
    for (int i = m + 2; i <= hi; i++) {
      H[i * n + i - 2] = 0.0;
      if (i > m + 2)
        H[i * n + i - 3] = 0.0;
    }
#pragma unroll 1
    for (int k = m; k <= hi - 1; k++) {
      const bool notlast = (k != hi - 1);
      if (k != m) {
        p = H[k * n + k - 1];
        q = H[(k + 1) * n + k - 1];
        r = notlast ? H[(k + 2) * n + k - 1] : 0.0;
        x = fabs(p) + fabs(q) + fabs(r);
        if (x == 0.0)
          continue;
        p /= x;
        q /= x;
        r /= x;
      }
      double s = sqrt(p * p + q * q + r * r);
      if (p < 0)
        s = -s;
      if (k != m)
        H[k * n + k - 1] = -s * x;
      else if (l != m)
        H[k * n + k - 1] = -H[k * n + k - 1];
      p += s;
      x = p / s;
      y = q / s;
      z = r / s;
      q /= p;
      r /= p;
#pragma unroll 1
      for (int j = k; j < n; j++) {  // rows
        double pp = H[k * n + j] + q * H[(k + 1) * n + j];
        if (notlast) {
          pp += r * H[(k + 2) * n + j];
          H[(k + 2) * n + j] -= pp * z;
        }
        H[k * n + j] -= pp * x;
        H[(k + 1) * n + j] -= pp * y;
      }
      const int ihi = hi < k + 3 ? hi : k + 3;
#pragma unroll 1
      for (int i = 0; i <= ihi; i++) {  // columns
        double pp = x * H[i * n + k] + y * H[i * n + k + 1];
        if (notlast) {
          pp += z * H[i * n + k + 2];
          H[i * n + k + 2] -= pp * r;
        }
        H[i * n + k] -= pp;
        H[i * n + k + 1] -= pp * q;
      }
#pragma unroll 1
      for (int i = 0; i < n; i++) {
        double pp = x * Z[i * n + k] + y * Z[i * n + k + 1];
        if (notlast) {
          pp += z * Z[i * n + k + 2];
          Z[i * n + k + 2] -= pp * r;
        }
        Z[i * n + k] -= pp;
        Z[i * n + k + 1] -= pp * q;
      }
    }
  }
  return true;
}

// Eigenvectors (columns of Rr + i Ri, n x n row-major) from the real Schur
// form T and Schur vectors Z, by back-substitution per eigenvalue.
template <int n>
GPR_D void schur_vectors(const double *T, const double *Z, const double *wr, const double *wi,
                         double *Rr, double *Ri) {
  double norm = 0.0;
#pragma unroll 1
  for (int i = 0; i < n; i++)
#pragma unroll 1
    for (int j = i > 0 ? i - 1 : 0; j < n; j++)
      norm += fabs(T[i * n + j]);
#pragma unroll 1
  for (int k = 0; k < n; k++) {
    const double lr = wr[k], li = wi[k];
    double yr[n], yi[n];
#pragma unroll 1
    for (int i = 0; i < n; i++)
      yr[i] = yi[i] = 0.0;
    const bool blk2 = (k + 1 < n && T[(k + 1) * n + k] != 0.0);
    const bool blk1 = (k > 0 && T[k * n + k - 1] != 0.0);
    int top;
    if (!blk1 && !blk2) {
      yr[k] = 1.0;
      top = k;
    } else {
      const int b = blk2 ? k : k - 1;
      const double a11 = T[b * n + b] - lr, a12 = T[b * n + b + 1];
      const double a21 = T[(b + 1) * n + b];
      if (fabs(a12) >= fabs(a21)) {
        yr[b] = 1.0;
        yi[b] = 0.0;
        yr[b + 1] = -a11 / a12;
        yi[b + 1] = li / a12;
      } else {
        const double a22r = T[(b + 1) * n + b + 1] - lr;
        yr[b + 1] = 1.0;
        yi[b + 1] = 0.0;
        yr[b] = -a22r / a21;
        yi[b] = li / a21;
      }
      top = b + 1;
    }
    const int start = (blk1 || blk2) ? (blk2 ? k - 1 : k - 2) : k - 1;
#pragma unroll 1
    for (int i = start; i >= 0; i--) {
      const bool is2 = (i > 0 && T[i * n + i - 1] != 0.0);
      if (!is2) {
        double sr = 0.0, si = 0.0;
#pragma unroll 1
        for (int j = i + 1; j <= top; j++) {
          sr += T[i * n + j] * yr[j];
          si += T[i * n + j] * yi[j];
        }
        const double dr = T[i * n + i] - lr, di = -li;
        if (hypot(dr, di) <= OSH_MULT_TOL * norm) {
          yr[i] = yi[i] = 0.0;  // the same eigenvalue: independent Schur vector
          continue;
        }
        const double den = dr * dr + di * di;
        yr[i] = -(sr * dr + si * di) / den;
        yi[i] = -(si * dr - sr * di) / den;
      } else {
        const int a = i - 1;
        double s1r = 0, s1i = 0, s2r = 0, s2i = 0;
#pragma unroll 1
        for (int j = i + 1; j <= top; j++) {
          s1r += T[a * n + j] * yr[j];
          s1i += T[a * n + j] * yi[j];
          s2r += T[i * n + j] * yr[j];
          s2i += T[i * n + j] * yi[j];
        }
        const double m11r = T[a * n + a] - lr, m11i = -li;
        const double m12 = T[a * n + i], m21 = T[i * n + a];
        const double m22r = T[i * n + i] - lr, m22i = -li;
        const double detr = m11r * m22r - m11i * m22i - m12 * m21;
        const double deti = m11r * m22i + m11i * m22r;
        if (hypot(detr, deti) <= OSH_MULT_TOL * norm * OSH_MULT_TOL * norm) {
          yr[a] = yi[a] = yr[i] = yi[i] = 0.0;
          i--;
          continue;
        }
        const double den = detr * detr + deti * deti;
        const double nar = -(s1r * m22r - s1i * m22i) + m12 * s2r;
        const double nai = -(s1r * m22i + s1i * m22r) + m12 * s2i;
        const double nir = -(m11r * s2r - m11i * s2i) + m21 * s1r;
        const double nii = -(m11r * s2i + m11i * s2r) + m21 * s1i;
        yr[a] = (nar * detr + nai * deti) / den;
        yi[a] = (nai * detr - nar * deti) / den;
        yr[i] = (nir * detr + nii * deti) / den;
        yi[i] = (nii * detr - nir * deti) / den;
        i--;
      }
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double sr = 0.0, si = 0.0;
#pragma unroll 1
      for (int j = 0; j <= top; j++) {
        sr += Z[i * n + j] * yr[j];
        si += Z[i * n + j] * yi[j];
      }
      Rr[i * n + k] = sr;
      Ri[i * n + k] = si;
    }
  }
}

// Complex Gaussian elimination with partial pivoting: (Cr + i Ci) x = b for
// two right-hand sides b = (br + i bi)[2][n], overwritten by x.  Returns false
// if singular.
template <int n> GPR_D bool csolve_n(double *Cr, double *Ci, double *br, double *bi) {
#pragma unroll 1
  for (int c = 0; c < n; c++) {
    int p = c;
    double best = hypot(Cr[c * n + c], Ci[c * n + c]);
#pragma unroll 1
    for (int r = c + 1; r < n; r++) {
      const double a = hypot(Cr[r * n + c], Ci[r * n + c]);
      if (a > best) {
        best = a;
        p = r;
      }
    }
    if (best == 0.0)
      return false;
    if (p != c) {
      auto swap = [](double &x, double &y) {
        const double t = x;
        x = y;
        y = t;
      };
#pragma unroll 1
      for (int j = 0; j < n; j++) {
        swap(Cr[c * n + j], Cr[p * n + j]);
        swap(Ci[c * n + j], Ci[p * n + j]);
      }
#pragma unroll 1
      for (int h = 0; h < 2 * n; h += n) {
        swap(br[h + c], br[h + p]);
        swap(bi[h + c], bi[h + p]);
      }
    }
    const double pr = Cr[c * n + c], pi = Ci[c * n + c];
    const double den = pr * pr + pi * pi;
#pragma unroll 1
    for (int r = c + 1; r < n; r++) {
      const double ar = Cr[r * n + c], ai = Ci[r * n + c];
      const double fr = (ar * pr + ai * pi) / den, fi = (ai * pr - ar * pi) / den;
#pragma unroll 1
      for (int j = c; j < n; j++) {
        const double xr = Cr[c * n + j], xi = Ci[c * n + j];
        Cr[r * n + j] -= fr * xr - fi * xi;
        Ci[r * n + j] -= fr * xi + fi * xr;
      }
#pragma unroll 1
      for (int h = 0; h < 2 * n; h += n) {
        const double xr = br[h + c], xi = bi[h + c];
        br[h + r] -= fr * xr - fi * xi;
        bi[h + r] -= fr * xi + fi * xr;
      }
    }
  }
#pragma unroll 1
  for (int h = 0; h < 2 * n; h += n)
#pragma unroll 1
    for (int r = n - 1; r >= 0; r--) {
      double sr = br[h + r], si = bi[h + r];
#pragma unroll 1
      for (int j = r + 1; j < n; j++) {
        sr -= Cr[r * n + j] * br[h + j] - Ci[r * n + j] * bi[h + j];
        si -= Cr[r * n + j] * bi[h + j] + Ci[r * n + j] * br[h + j];
      }
      const double pr = Cr[r * n + r], pi = Ci[r * n + r];
      const double den = pr * pr + pi * pi;
      br[h + r] = (sr * pr + si * pi) / den;
      bi[h + r] = (si * pr - sr * pi) / den;
    }
  return true;
}

// The system matrix along x, or an average of it over states, leaves six
// distortion entries (A_k1, A_k2) and the level sets as they are but for the
// advection velocity vb on their diagonal:
//   M = [[C, B], [0, vb I]],   |M| (w, a) = (|C| w + g(C) B a, |vb| a),
// g(x) = (|x| - |vb|) / (x - vb), so only C is decomposed: 11 x 11 with heat
// conduction, else 8 x 8 (in place of 17 x 17 and 14 x 14: a quarter and a
// fifth of the work and of the local memory).  Entry r of the active part is
// state entry active_entry(r).
template <class L> constexpr int ACTIVE_N = L::THERMAL ? 11 : 8;
GPR_HD constexpr int active_entry(int r) {
  return r < 5 ? r : (r < 8 ? 5 + 3 * (r - 5) : 14 + (r - 8));
}
template <class L> GPR_HD constexpr bool passive_entry(int k) {
  return (k >= 5 && k < 14 && (k - 5) % 3 != 0) || k >= L::V - L::LSET;
}

// The largest passive entry of dq.
template <class L> GPR_D double max_passive(const double *dq) {
  double a = 0.0;
#pragma unroll
  for (int k = 5; k < L::V; k++)
    if (passive_entry<L>(k))
      a = fmax(a, fabs(dq[k]));
  return a;
}

// |l| and g(l) of one eigenvalue l = lr + i li.  For a real l of vb's sign g is
// that sign whatever l - vb (a semisimple l = vb included); where both vanish to
// rounding (tol) it would be the sign of a rounding error, and is 0, the mean
// of both.
GPR_D void abs_factors(double lr, double li, double vb, double tol, double &fa, double &gr,
                       double &gi) {
  gi = 0.0;
  fa = li == 0.0 ? fabs(lr) : hypot(lr, li);
  if (fa <= tol && fabs(vb) <= tol) {
    gr = 0.0;
    return;
  }
  if (li == 0.0) {
    if ((lr >= 0.0) == (vb >= 0.0))
      gr = vb >= 0.0 ? 1.0 : -1.0;
    else
      gr = (fa - fabs(vb)) / (lr - vb);
    return;
  }
  const double dr = lr - vb, den = dr * dr + li * li, num = fa - fabs(vb);
  gr = num * dr / den;
  gi = -num * li / den;
}

// C (ld n) and Ba of wt times the system matrix of q along x, added to C and
// Ba; returns wt v_x.  dF/dP and dP/dQ have a few nonzeros per row, known at
// compile time: the products are written for those (about 300 in place of
// V^3 = 4913).
template <class L>
GPR_D double system_active(const double *q, const double *a, double wt, const DevPar &P,
                           double *C, double *Ba) {
  constexpr int V = L::V, n = ACTIVE_N<L>;
  double F[V * V], D[V * V];
#pragma unroll
  for (int i = 0; i < V * V; i++)
    F[i] = D[i] = 0.0;
  Prim<L::THERMAL> s;
  prim<L::THERMAL>(q, P, s);
  system_fd<L::THERMAL, V>(q, s, P, F, D);
#pragma unroll
  for (int r = 0; r < n; r++) {
    const int R = active_entry(r);
    double ba = 0.0;
#pragma unroll
    for (int j = 0; j < V - L::LSET; j++) {
      // row R of dF/dP: entry 1 (pressure) for E, m_x and J_x only
      const bool press = R == 1 || R == 2 || R == 14;
      double x = j == 1 ? 0.0 : F[R * V + j] * D[j * V + j];
      if (press)
        x = fma(F[R * V + 1], D[V + j], x);
      if (j == 0) {
#pragma unroll
        for (int k = 2; k < 5; k++)
          x = fma(F[R * V + k], D[k * V], x);
        if (L::THERMAL) {
#pragma unroll
          for (int k = 14; k < 17; k++)
            x = fma(F[R * V + k], D[k * V], x);
        }
      }
      // B_x: v_x on the distortion's diagonal, -v_j in the x rows
      if (R >= 5 && R < 14) {
        if (j == R)
          x += s.v[0];
        if (j >= R && j < R + 3)
          x -= s.v[j - R];
      }
      if (passive_entry<L>(j)) {
        ba = fma(x, a[j], ba);
      } else {
        const int c = j < 5 ? j : (j < 14 ? 5 + (j - 5) / 3 : j - 6);
        C[r * n + c] = fma(wt, x, C[r * n + c]);
      }
    }
    Ba[r] = fma(wt, ba, Ba[r]);
  }
  return wt * s.v[0];
}

// How |M| dq by the active part ended.  Where an eigenvalue of C and vb both
// vanish and B a has a part along its eigenvector, |M| has two limits there
// (g = 1 and -1) that differ by that part.  No state's matrix has one (a state's
// v is semisimple), but Roe's average at a symmetric wall does: the path's
// velocities are v and -v, and the part is of the order of the jump.
enum AbsStatus { ABS_FAILED = 0, ABS_OK = 1, ABS_TWO_LIMITS = 2 };

// acc += w |M| dq for M given by C (n x n row-major, destroyed), Ba = B a (a the
// passive part of dq) and vb.  With a real spectrum the eigenvectors are Z Y, Y
// unit upper triangular (back-substitution on the Schur form), so R^-1 is Z^T
// and a triangular solve; complex eigenvalues take the complex elimination.
// strict: two limits are reported, with acc as it was, instead of their mean
// taken.
template <class L>
GPR_D AbsStatus abs_apply(double *C, const double *Ba, double vb, const double *dq, double w,
                          double *acc, bool strict = false) {
  constexpr int V = L::V, n = ACTIVE_N<L>;
  double Z[n * n], wr[n], wi[n], y[n];
#pragma unroll 1
  for (int i = 0; i < n * n; i++)
    Z[i] = (i % (n + 1) == 0) ? 1.0 : 0.0;
  hess_reduce<n>(C, Z);
  if (!hqr_schur<n>(C, Z, wr, wi))
    return ABS_FAILED;
  bool real = true;
#pragma unroll 1
  for (int k = 0; k < n; k++)
    real = real && wi[k] == 0.0;
  double dw[n];
#pragma unroll
  for (int r = 0; r < n; r++)
    dw[r] = dq[active_entry(r)];
  double norm = 0.0;
#pragma unroll 1
  for (int i = 0; i < n; i++)
#pragma unroll 1
    for (int j = i; j < n; j++)
      norm += fabs(C[i * n + j]);
  const double tol = OSH_MULT_TOL * norm;
  double part = tol * max_passive<L>(dq);  // of B a, above which two limits count
  if (!strict || fabs(vb) > tol)
    part = INFINITY;
  if (real) {
    double Y[n * n], c2[n];  // Y by columns
#pragma unroll 1
    for (int k = 0; k < n; k++) {
      double x1 = 0.0, x2 = 0.0;
#pragma unroll 1
      for (int i = 0; i < n; i++) {
        x1 += Z[i * n + k] * dw[i];
        x2 += Z[i * n + k] * Ba[i];
      }
      y[k] = x1;
      c2[k] = x2;
      Y[k * n + k] = 1.0;
#pragma unroll 1
      for (int i = k - 1; i >= 0; i--) {
        double sum = 0.0;
#pragma unroll 1
        for (int j = i + 1; j <= k; j++)
          sum += C[i * n + j] * Y[k * n + j];
        const double d = C[i * n + i] - wr[k];
        // the same eigenvalue: an independent Schur vector
        Y[k * n + i] = fabs(d) <= tol ? 0.0 : -sum / d;
      }
    }
#pragma unroll 1
    for (int k = n - 1; k >= 0; k--) {
#pragma unroll 1
      for (int i = 0; i < k; i++) {
        y[i] -= Y[k * n + i] * y[k];
        c2[i] -= Y[k * n + i] * c2[k];
      }
      if (fabs(wr[k]) <= tol && fabs(c2[k]) > part)
        return ABS_TWO_LIMITS;
      double fa, gr, gi;
      abs_factors(wr[k], 0.0, vb, tol, fa, gr, gi);
      y[k] = fa * y[k] + gr * c2[k];
    }
    // Y y (column by column, downwards in place), then Z
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double sum = y[i];
#pragma unroll 1
      for (int k = i + 1; k < n; k++)
        sum += Y[k * n + i] * y[k];
      y[i] = sum;
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double sum = 0.0;
#pragma unroll 1
      for (int k = 0; k < n; k++)
        sum += Z[i * n + k] * y[k];
      c2[i] = sum;
    }
#pragma unroll
    for (int r = 0; r < n; r++)
      acc[active_entry(r)] += w * c2[r];
  } else {
    double Rr[n * n], Ri[n * n], br[2 * n], bi[2 * n];
    schur_vectors<n>(C, Z, wr, wi, Rr, Ri);
    // C and Z are free: the elimination's copy of R
#pragma unroll 1
    for (int i = 0; i < n * n; i++) {
      C[i] = Rr[i];
      Z[i] = Ri[i];
    }
#pragma unroll 1
    for (int k = 0; k < n; k++) {
      br[k] = dw[k];
      br[n + k] = Ba[k];
      bi[k] = bi[n + k] = 0.0;
    }
    if (!csolve_n<n>(C, Z, br, bi))
      return ABS_FAILED;
#pragma unroll 1
    for (int k = 0; k < n; k++) {
      if (hypot(wr[k], wi[k]) <= tol && hypot(br[n + k], bi[n + k]) > part)
        return ABS_TWO_LIMITS;
      double fa, gr, gi;
      abs_factors(wr[k], wi[k], vb, tol, fa, gr, gi);
      const double xr = fa * br[k] + (gr * br[n + k] - gi * bi[n + k]);
      bi[k] = fa * bi[k] + (gr * bi[n + k] + gi * br[n + k]);
      br[k] = xr;
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double sum = 0.0;
#pragma unroll 1
      for (int k = 0; k < n; k++)
        sum += Rr[i * n + k] * br[k] - Ri[i * n + k] * bi[k];
      y[i] = sum;
    }
#pragma unroll
    for (int r = 0; r < n; r++)
      acc[active_entry(r)] += w * y[r];
  }
  const double av = w * fabs(vb);
#pragma unroll
  for (int k = 5; k < V; k++)
    if (passive_entry<L>(k))
      acc[k] = fma(av, dq[k], acc[k]);
  return ABS_OK;
}

// ---------------------------------------------------------------------------
// |M| of one state in closed form (Osher-Solomon).  In primitive variables (rho,
// p, v, A, J) the system matrix along x is v + N, where N couples only y =
// (v, J_x) with z = (rho, p, A): y' = Xi1 z, z' = Xi2 y (the energy equation's
// heat terms cancel but for h dJ_x).  So N^2 on y is the acoustic tensor Xi =
// Xi1 Xi2, the eigenvalues of M are v (nine-fold) and v +- c_k with c_k^2
// those of Xi, and for any eigenvectors
//   |M| (y, z) = (E(Xi) y + O(Xi) Xi1 z,  |v| z + Xi2 (K(Xi) Xi1 z + O(Xi) y)),
// E = max(c, |v|), O = sgn(v) min(c, |v|) / c, K = max(c - |v|, 0) / c^2.
// Along x the velocity block of Xi is symmetric and the heat row and column
// meet it at v_x only, so a diagonal scaling makes Xi symmetric and E, O, K
// follow from its 3 x 3 or 4 x 4 symmetric eigenproblem (Jacobi): about 1300
// FP64 instructions per path node in registers, where the 17 x 17
// eigen-decomposition with its vectors and complex solve takes about 1e5 in
// local memory.  An orthogonal decomposition has no loss at equal wave speeds.

// f += w |M(q)| dq along x.  Returns false, with f unchanged, where the form
// does not apply (wave speeds that are not real and positive, a heat coupling
// that no scaling makes symmetric): the caller then takes the general
// eigen-decomposition.
template <class L>
GPR_D bool abs_apply_acoustic(const double *q, const double *dq, double w, const DevPar &P,
                              double *f) {
  constexpr int V = L::V;
  constexpr bool TH = L::THERMAL;
  constexpr int m = TH ? 4 : 3;
  Prim<TH> s;
  prim<TH>(q, P, s);
  const double *A = q + 5;
  const double *dA = dq + 5;
  const EosRho &e = s.e;
  const double r = s.r, ir = s.ir, cs2 = s.cs2;
  const double rG = r * e.G, irG2 = s.irG * s.irG;
  double dnum = e.G * (s.p - e.pr);
  if (P.EOS != 0)
    dnum = e.dpr * rG + (e.G + r * e.dG) * (s.p - e.pr);
  double Er = e.der - dnum * irG2;
  double C0 = cs2;
  if (P.has_beta) {
    if (TH)
      return false;  // the impulse then couples to all of v
    const double dcs2 = P.beta * ir * cs2;
    Er += 0.25 * ((1.0 - P.beta / e.G) * dcs2 + P.beta / (e.G * e.G) * e.dG * cs2) * s.devGsq;
    C0 = (P.EOS == 1 ? (1.0 - P.beta / e.G) : P.C0f) * cs2;
  }
  const double c02 = (s.p * ir * ir - Er) * rG;
  const double eR = fma(q[1], ir, r * Er);  // d(rho E)/drho at fixed p, v, A, J
  const double rC0 = r * C0;
  // dq in primitive variables (dP/dQ, equations.cpp:130-167)
  const double rho = dq[0];
  double vp[3], Jp[3] = {0.0, 0.0, 0.0}, AGdA = 0.0;
  double pp = fma(-eR, rho, dq[1]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    vp[i] = fma(-s.v[i], rho, dq[2 + i]);
    pp = fma(-s.v[i], vp[i], pp);
    vp[i] *= ir;
  }
#pragma unroll
  for (int k = 0; k < 9; k++)
    AGdA = fma(s.AdG[k], dA[k], AGdA);
  pp = fma(-rC0, AGdA, pp);
  if (TH) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      Jp[i] = fma(-s.J[i], rho, dq[14 + i]);
      pp = fma(-P.calpha2 * s.J[i], Jp[i], pp);
      Jp[i] *= ir;
    }
  }
  pp *= e.G;
  // Xi1 z: (dp e_x - dsigma_x) / rho and dT / rho, with dsigma_x = (1 + beta)
  // sigma_x drho / rho - rho cs2 (dG devG + devG dG ... )(:,x), dG = dA^T A + A^T dA
  double y[m], a[m];
  {
    double dG[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const int i = k < 3 ? k : (k == 5 ? 1 : 0), j = k < 3 ? k : (k == 3 ? 1 : 2);
      double x = 0.0;
#pragma unroll
      for (int n = 0; n < 3; n++)
        x = fma(dA[3 * n + i], A[3 * n + j], fma(A[3 * n + i], dA[3 * n + j], x));
      dG[k] = x;
    }
    const double t3 = (s.G[0] + s.G[1] + s.G[2]) * (1.0 / 3.0);
    const double dt3 = (dG[0] + dG[1] + dG[2]) * (1.0 / 3.0);
    const double fr = P.b1 * rho * ir;
#pragma unroll
    for (int i = 0; i < 3; i++) {
      // S(i, x) = (G^2 - t3 G)(i, x): dS = dG G + G dG - dt3 G - t3 dG
      double x = fma(-dt3, sym3(s.G, i, 0), -(t3 * sym3(dG, i, 0)));
#pragma unroll
      for (int n = 0; n < 3; n++)
        x = fma(sym3(dG, i, n), sym3(s.G, n, 0), fma(sym3(s.G, i, n), sym3(dG, n, 0), x));
      a[i] = cs2 * fma(fr, sym3(s.S, i, 0), x);
      y[i] = vp[i];
    }
    a[0] = fma(ir, pp, a[0]);
  }
  // the acoustic tensor (max_abs_eigs, d = 0), symmetric after scaling the
  // impulse by del = sqrt(x30 / x03)
  double H[m][m], W[m][m];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double g3 = (1.0 / 3.0) * sym3(s.G, i, 0);
#pragma unroll
    for (int c = i; c < 3; c++) {
      double x = fma(s.G[0], sym3(s.G, i, c), fma(g3, sym3(s.G, c, 0), sym3(s.S, i, c)));
      if (i == 0)
        x = fma(c == 0 ? 2.0 * P.b1 : P.b1, sym3(s.S, 0, c), x);
      H[i][c] = cs2 * x;
    }
  }
  H[0][0] += c02;
  double h = 0.0, del = 1.0, idel = 1.0;
  if (TH) {
    h = P.calpha2 * s.T * e.G;
    const double rtp = s.irG * P.icv;
    const double dTr = -dnum * irG2 * P.icv;
    const double x03 = h * ir, x30 = fma(rtp, c02, dTr);
    const double pr = x03 * x30;
    if (!(pr > 0.0))
      return false;
    H[0][m - 1] = copysign(sqrt64(pr), x03);
    H[1][m - 1] = H[2][m - 1] = 0.0;
    H[m - 1][m - 1] = rtp * ir * h;
    del = fabs(H[0][m - 1] * rcp64(x03));
    idel = rcp64(del);
    y[m - 1] = Jp[0] * idel;
    a[m - 1] = ir * fma(rtp, pp, dTr * rho) * idel;
  }
  if (!jacobi_sym<m>(H, W))
    return false;
  bool pos = true;
#pragma unroll
  for (int k = 0; k < m; k++)
    pos = pos && H[k][k] > 0.0;
  if (!pos)
    return false;
  const double av = fabs(s.v[0]);
  double yo[m], wo[m];
#pragma unroll
  for (int i = 0; i < m; i++)
    yo[i] = wo[i] = 0.0;
#pragma unroll
  for (int k = 0; k < m; k++) {
    const double c = sqrt64(H[k][k]), ic = rcp64(c);
    const bool sub = c > av;
    const double E = sub ? c : av;
    const double O = sub ? s.v[0] * ic : copysign(1.0, s.v[0]);
    const double K = sub ? (c - av) * ic * ic : 0.0;
    double yk = 0.0, ak = 0.0;
#pragma unroll
    for (int i = 0; i < m; i++) {
      yk = fma(W[i][k], y[i], yk);
      ak = fma(W[i][k], a[i], ak);
    }
    const double ey = fma(E, yk, O * ak), ew = fma(K, ak, O * yk);
#pragma unroll
    for (int i = 0; i < m; i++) {
      yo[i] = fma(W[i][k], ey, yo[i]);
      wo[i] = fma(W[i][k], ew, wo[i]);
    }
  }
  // z: |v| z + Xi2 w, b = -beta sigma_x + rho c0^2 e_x
  const double rho_o = fma(r, wo[0], av * rho);
  double pw = r * c02 * wo[0];
  if (P.has_beta) {
    const double fb = P.beta * r * cs2;
#pragma unroll
    for (int i = 0; i < 3; i++)
      pw = fma(fb * sym3(s.S, i, 0), wo[i], pw);
  }
  if (TH)
    pw = fma(h * del, wo[m - 1], pw);
  const double p_o = fma(av, pp, pw);
  // back to conserved variables (dQ/dP)
  double en = fma(eR, rho_o, p_o * r * s.irG), AG = 0.0;
  f[0] = fma(w, rho_o, f[0]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double mi = fma(s.v[i], rho_o, r * yo[i]);
    en = fma(r * s.v[i], yo[i], en);
    f[2 + i] = fma(w, mi, f[2 + i]);
  }
#pragma unroll
  for (int k = 0; k < 9; k++) {
    double x = av * dA[k];
    if (k % 3 == 0) {
#pragma unroll
      for (int j = 0; j < 3; j++)
        x = fma(A[k + j], wo[j], x);
    }
    AG = fma(s.AdG[k], x, AG);
    f[5 + k] = fma(w, x, f[5 + k]);
  }
  en = fma(rC0, AG, en);
  if (TH) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const double Jo = i == 0 ? del * yo[m - 1] : av * Jp[i];
      en = fma(P.calpha2 * r * s.J[i], Jo, en);
      f[14 + i] = fma(w, fma(s.J[i], rho_o, r * Jo), f[14 + i]);
    }
  }
  f[1] = fma(w, en, f[1]);
#pragma unroll
  for (int k = V - L::LSET; k < V; k++)
    f[k] = fma(w * av, dq[k], f[k]);
  return true;
}

// f += w |M(q)| dq by the general eigen-decomposition (out of line: the
// callers' registers and code are those of the closed form).
template <class L>
__device__ __noinline__ bool abs_apply_general(const double *q, const double *dq, double w,
                                               const DevPar &P, double *f) {
  constexpr int n = ACTIVE_N<L>;
  double C[n * n], Ba[n];
#pragma unroll 1
  for (int i = 0; i < n * n; i++)
    C[i] = 0.0;
#pragma unroll
  for (int i = 0; i < n; i++)
    Ba[i] = 0.0;
  const double vb = system_active<L>(q, dq, 1.0, P, C, Ba);
  return abs_apply<L>(C, Ba, vb, dq, w, f) == ABS_OK;
}

// Eigen part of D_OSH along x into f (overwritten): sum_i w_i |M(q_i)| dq
// over the NQ Gauss nodes of the path qR -> qL; NaN if a general
// eigen-decomposition is needed and fails.
template <class L, int NQ>
GPR_D void osher_dissipation(const double *ql, const double *qr, const DevPar &P,
                             const double *nodes, const double *wts, double *f) {
  constexpr int V = L::V;
  double dq[V], q[V];
  bool flat = true;
#pragma unroll
  for (int k = 0; k < V; k++) {
    dq[k] = ql[k] - qr[k];
    f[k] = 0.0;
    flat = flat && (__double_as_longlong(dq[k]) << 1) == 0;
  }
  // qL = qR (a uniform region): |M| dq is exactly zero
  if (flat)
    return;
#pragma unroll 1
  for (int i = 0; i < NQ; i++) {
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = fma(nodes[i], dq[k], qr[k]);
    if (!abs_apply_acoustic<L>(q, dq, wts[i], P, f)) {
      double qm[V], dm[V], fm[V];
#pragma unroll
      for (int k = 0; k < V; k++) {
        qm[k] = q[k];
        dm[k] = dq[k];
        fm[k] = f[k];
      }
      const bool ok = abs_apply_general<L>(qm, dm, wts[i], P, fm);
#pragma unroll
      for (int k = 0; k < V; k++)
        f[k] = ok ? fm[k] : __longlong_as_double(0x7ff8000000000000ll);
    }
  }
}

// f = |M| dq for Roe's path average M by the decomposition of the whole V x V
// matrix, for the faces where the active part finds two limits: eigenvalues
// that agree to rounding take independent vectors (schur_vectors), which gives
// the value of the form before the active part was split off, and no mass flux
// through the wall but where the solver's own roundings tell such eigenvalues
// apart.  With heat conduction C has no zero eigenvalue there.
template <class L, int NQ>
__device__ __noinline__ bool roe_whole(const double *qr, const double *dq, const DevPar &P,
                                       const double *nodes, const double *wts, double *f) {
  constexpr int V = L::V;
  double M[V * V], Z[V * V], Rr[V * V], Ri[V * V], wr[V], wi[V], br[2 * V], bi[2 * V], q[V];
#pragma unroll 1
  for (int i = 0; i < V * V; i++)
    M[i] = 0.0;
#pragma unroll 1
  for (int n = 0; n < NQ; n++) {
#pragma unroll 1
    for (int k = 0; k < V; k++)
      q[k] = qr[k] + nodes[n] * dq[k];
#pragma unroll 1
    for (int i = 0; i < V * V; i++)
      Rr[i] = Ri[i] = 0.0;
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(q, P, s);
    system_fd<L::THERMAL, V>(q, s, P, Rr, Ri);
#pragma unroll 1
    for (int i = 0; i < V; i++)
#pragma unroll 1
      for (int j = 0; j < V; j++) {
        double x = 0.0;
#pragma unroll 1
        for (int k = 0; k < V; k++)
          x += Rr[i * V + k] * Ri[k * V + j];
        Z[i * V + j] = x;
      }
    system_block<V, L::LSET>(s.v, Z);
#pragma unroll 1
    for (int i = 0; i < V * V; i++)
      M[i] += wts[n] * Z[i];
  }
#pragma unroll 1
  for (int i = 0; i < V * V; i++)
    Z[i] = (i % (V + 1) == 0) ? 1.0 : 0.0;
  hess_reduce<V>(M, Z);
  if (!hqr_schur<V>(M, Z, wr, wi))
    return false;
  schur_vectors<V>(M, Z, wr, wi, Rr, Ri);
#pragma unroll 1
  for (int i = 0; i < V * V; i++) {
    M[i] = Rr[i];
    Z[i] = Ri[i];
  }
#pragma unroll 1
  for (int k = 0; k < V; k++) {
    br[k] = dq[k];
    br[V + k] = bi[k] = bi[V + k] = 0.0;
  }
  if (!csolve_n<V>(M, Z, br, bi))
    return false;
#pragma unroll 1
  for (int k = 0; k < V; k++) {
    const double a = hypot(wr[k], wi[k]);
    br[k] *= a;
    bi[k] *= a;
  }
#pragma unroll 1
  for (int i = 0; i < V; i++) {
    double x = 0.0;
#pragma unroll 1
    for (int k = 0; k < V; k++)
      x += Rr[i * V + k] * br[k] - Ri[i * V + k] * bi[k];
    f[i] = x;
  }
  return true;
}

// Eigen part of D_OSH (flux 2) / D_ROE (flux 1) at one interface into f
// (overwritten); NaN if the eigen-decomposition fails (fluxes.cpp:22-64).
// The path qR -> qL takes the scheme's NQ Gauss nodes (nodes, wts on [0, 1]).
template <class L, int NQ>
GPR_D void eig_dissipation_q(const double *ql, const double *qr, int flux, const DevPar &P,
                             const double *nodes, const double *wts, double *f) {
  constexpr int V = L::V;
  if (flux == GPR_FLUX_OSHER) {
    osher_dissipation<L, NQ>(ql, qr, P, nodes, wts, f);
    return;
  }
  constexpr int n = ACTIVE_N<L>;
  double dq[V], q[V], C[n * n], Ba[n];
  bool flat = true;
#pragma unroll
  for (int k = 0; k < V; k++) {
    dq[k] = ql[k] - qr[k];
    f[k] = 0.0;
    flat = flat && dq[k] == 0.0;
  }
  // qL = qR (a uniform region): |A| dq is exactly zero, whatever A's
  // eigen-decomposition
  if (flat)
    return;
#pragma unroll 1
  for (int i = 0; i < n * n; i++)
    C[i] = 0.0;
#pragma unroll
  for (int i = 0; i < n; i++)
    Ba[i] = 0.0;
  double vb = 0.0;
#pragma unroll 1
  for (int i = 0; i < NQ; i++) {
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = qr[k] + nodes[i] * dq[k];
    vb += system_active<L>(q, dq, wts[i], P, C, Ba);
  }
  const AbsStatus rc = abs_apply<L>(C, Ba, vb, dq, 1.0, f, !L::THERMAL);
  bool ok = rc == ABS_OK;
  if constexpr (!L::THERMAL) {
    if (rc == ABS_TWO_LIMITS) {
      double rm[V], dm[V], fm[V];
#pragma unroll
      for (int k = 0; k < V; k++) {
        rm[k] = qr[k];
        dm[k] = dq[k];
      }
      ok = roe_whole<L, NQ>(rm, dm, P, nodes, wts, fm);
#pragma unroll
      for (int k = 0; k < V; k++)
        f[k] = fm[k];
    }
  }
  if (!ok) {
#pragma unroll
    for (int k = 0; k < V; k++)
      f[k] = __longlong_as_double(0x7ff8000000000000ll);
  }
}

template <class L>
GPR_D void eig_dissipation(const double *ql, const double *qr, int flux, const DevPar &P,
                           const Consts &C, double *f) {
  eig_dissipation_q<L, NN>(ql, qr, flux, P, C.nodes, C.w, f);
}

GPR_HD constexpr int axis_swap_index(int a, int d) { return a == 0 ? d : (a == d ? 0 : a); }
// Index of state entry k with spatial axes 0 and d exchanged: velocity and
// thermal impulse components, and both indices of A (as the reference's
// rotate_tensors, system/multi/rotations.cpp:37-47).  The GPR system is
// invariant under this relabelling, so the system matrix along d is that
// along x of the relabelled state, relabelled back: exact, a permutation.
template <class L> GPR_HD constexpr int axis_swap(int k, int d) {
  if (d == 0)
    return k;
  if (k >= 2 && k < 5)
    return 2 + axis_swap_index(k - 2, d);
  if (k >= 5 && k < 14)
    return 5 + 3 * axis_swap_index((k - 5) / 3, d) + axis_swap_index((k - 5) % 3, d);
  if (L::THERMAL && k >= 14 && k < 17)
    return 14 + axis_swap_index(k - 14, d);
  return k;
}

// D_OSH / D_ROE along direction d (fluxes.cpp:22-64) through the x form.
template <class L, int NQ>
GPR_D void eig_dissipation_qd(const double *ql, const double *qr, int d, int flux,
                              const DevPar &P, const double *nodes, const double *wts,
                              double *f) {
  constexpr int V = L::V;
  if (d == 0) {
    eig_dissipation_q<L, NQ>(ql, qr, flux, P, nodes, wts, f);
    return;
  }
  double pl[V], pr[V], pf[V];
#pragma unroll
  for (int k = 0; k < V; k++) {
    pl[k] = ql[axis_swap<L>(k, d)];
    pr[k] = qr[axis_swap<L>(k, d)];
  }
  eig_dissipation_q<L, NQ>(pl, pr, flux, P, nodes, wts, pf);
#pragma unroll
  for (int k = 0; k < V; k++)
    f[k] = pf[axis_swap<L>(k, d)];
}
template <class L>
GPR_D void eig_dissipation_d(const double *ql, const double *qr, int d, int flux,
                             const DevPar &P, const Consts &C, double *f) {
  eig_dissipation_qd<L, NN>(ql, qr, d, flux, P, C.nodes, C.w, f);
}

// Interface terms for flux 1 / 2 along d: f = D + F(qL) + F(qR) and the path
// integral of B_d.
template <class L>
GPR_D void interface_point_eig(const double *ql, const double *qr, int flux, const DevPar &P,
                               const Consts &C, double *f, double *b, int d = 0) {
  constexpr int V = L::V;
  eig_dissipation_d<L>(ql, qr, d, flux, P, C, f);
  Prim<L::THERMAL> sl, sr;
  prim<L::THERMAL>(ql, P, sl);
  prim<L::THERMAL>(qr, P, sr);
  flux_add<L::THERMAL, V>(ql, sl, d, P, f);
  flux_add<L::THERMAL, V>(qr, sr, d, P, f);
  double dq[V];
#pragma unroll
  for (int k = 0; k < V; k++)
    dq[k] = qr[k] - ql[k];
  path_product<L, NN>(ql, dq, d, C.nodes, C.w, b);
}

// ---------------------------------------------------------------------------
// Warp-cooperative form: one warp per eigenproblem, matrices in shared
// memory.  The QR iteration's control flow (deflation tests, shifts) is
// evaluated identically by every lane from shared memory; the row, column
// and Schur-vector updates of each step are spread over the lanes; the
// eigenvectors are one lane each; the complex solve eliminates one row per
// lane.  The arithmetic of every element update is the serial one.

// Per-warp workspace.  H and Z are the active matrix and its Schur vectors;
// Rr and Ri hold dF/dP and dP/dQ before the eigen-decomposition, then the
// eigenvectors (Y in Rr for a real spectrum; for a complex one H and Z
// afterwards hold the copy that the complex solve factorises).
// Sized for the whole matrix where w_roe_whole may need it (m = V).
template <class L> struct EigWS {
  static constexpr int V = L::V, n = ACTIVE_N<L>, m = L::THERMAL ? n : V;
  double H[m * m], Z[m * m], Rr[V * V], Ri[V * V];
  double wr[m], wi[m], v[m], br[2 * m], bi[2 * m], Ba[n], vb;
  double q[V], ql[V], qr[V], dq[V], f[V];
};

GPR_D double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

template <int n> GPR_D void w_hess(double *H, double *Z, double *v, int lane) {
#pragma unroll 1
  for (int k = 0; k < n - 2; k++) {
    double tl = 0.0;  // the column below the subdiagonal (as hess_reduce)
    for (int i = k + 2 + lane; i < n; i += 32)
      tl += H[i * n + k] * H[i * n + k];
    if (warp_sum(tl) <= DBL_MIN_NORMAL)
      continue;
    double a2 = 0.0;
    for (int i = k + 1 + lane; i < n; i += 32)
      a2 += H[i * n + k] * H[i * n + k];
    const double alpha = sqrt(warp_sum(a2));
    if (alpha == 0.0)
      continue;
    const double x0 = H[(k + 1) * n + k];
    const double beta = x0 > 0 ? -alpha : alpha;
    double t2 = 0.0;
    for (int i = k + 2 + lane; i < n; i += 32)
      t2 += H[i * n + k] * H[i * n + k];
    const double vv = (x0 - beta) * (x0 - beta) + warp_sum(t2);
    if (vv == 0.0)
      continue;
    for (int i = lane; i < n; i += 32)
      v[i] = i <= k ? 0.0 : (i == k + 1 ? x0 - beta : H[i * n + k]);
    __syncwarp();
    const double tau = 2.0 / vv;
    for (int j = lane; j < n; j += 32) {  // (I - tau v v^T) H, column j
      double s = 0.0;
      for (int i = k + 1; i < n; i++)
        s += v[i] * H[i * n + j];
      s *= tau;
      for (int i = k + 1; i < n; i++)
        H[i * n + j] -= s * v[i];
    }
    __syncwarp();
    for (int i = lane; i < n; i += 32) {  // H (I - tau v v^T), row i; Z the same
      double s = 0.0;
      for (int j = k + 1; j < n; j++)
        s += H[i * n + j] * v[j];
      s *= tau;
      for (int j = k + 1; j < n; j++)
        H[i * n + j] -= s * v[j];
      double sz = 0.0;
      for (int j = k + 1; j < n; j++)
        sz += Z[i * n + j] * v[j];
      sz *= tau;
      for (int j = k + 1; j < n; j++)
        Z[i * n + j] -= sz * v[j];
    }
    __syncwarp();
    for (int i = k + 2 + lane; i < n; i += 32)
      H[i * n + k] = 0.0;
    __syncwarp();
  }
}

template <int n> GPR_D bool w_hqr(double *H, double *Z, double *wr, double *wi, int lane) {
  const double eps = 2.220446049250313e-16;
  double nrm = 0.0;
  for (int e = lane; e < n * n; e += 32) {
    int i = e / n, j = e % n;
    if (j >= i - 1)
      nrm += fabs(H[e]);
  }
  const double norm = warp_sum(nrm);
  int hi = n - 1, iter = 0, total = 0;
  double exshift = 0.0;
  while (hi >= 0) {
    int l = hi;
    while (l > 0) {
      double s = fabs(H[(l - 1) * n + l - 1]) + fabs(H[l * n + l]);
      if (s == 0.0)
        s = norm;
      if (fabs(H[l * n + l - 1]) < eps * s)
        break;
      l--;
    }
    if (l == hi) {
      __syncwarp();
      if (lane == 0) {
        H[hi * n + hi] += exshift;
        wr[hi] = H[hi * n + hi];
        wi[hi] = 0.0;
        if (hi > 0)
          H[hi * n + hi - 1] = 0.0;
      }
      __syncwarp();
      hi--;
      iter = 0;
      continue;
    }
    double x = H[hi * n + hi];
    double y = H[(hi - 1) * n + hi - 1];
    double w = H[hi * n + hi - 1] * H[(hi - 1) * n + hi];
    if (l == hi - 1) {
      double p = 0.5 * (y - x);
      double q = p * p + w;
      if (q < 0.0 && sqrt(-q) <= OSH_MULT_TOL * norm)
        q = 0.0;
      double z = sqrt(fabs(q));
      __syncwarp();
      if (lane == 0) {
        if (hi >= 2)
          H[(hi - 1) * n + hi - 2] = 0.0;
        H[hi * n + hi] = x + exshift;
        H[(hi - 1) * n + hi - 1] = y + exshift;
      }
      __syncwarp();
      x = H[hi * n + hi];
      if (q >= 0.0) {
        z = p >= 0 ? p + z : p - z;
        const double xx = H[hi * n + hi - 1];
        const double s = fabs(xx) + fabs(z);
        double pp = xx / s, qq = z / s;
        const double rr = sqrt(pp * pp + qq * qq);
        pp /= rr;
        qq /= rr;
        __syncwarp();
        if (lane == 0) {
          wr[hi - 1] = x + z;
          wr[hi] = z != 0.0 ? x - w / z : x + z;
          wi[hi - 1] = wi[hi] = 0.0;
        }
        for (int j = hi - 1 + lane; j < n; j += 32) {
          const double a = H[(hi - 1) * n + j];
          H[(hi - 1) * n + j] = qq * a + pp * H[hi * n + j];
          H[hi * n + j] = qq * H[hi * n + j] - pp * a;
        }
        __syncwarp();
        for (int i = lane; i <= hi; i += 32) {
          const double a = H[i * n + hi - 1];
          H[i * n + hi - 1] = qq * a + pp * H[i * n + hi];
          H[i * n + hi] = qq * H[i * n + hi] - pp * a;
        }
        for (int i = lane; i < n; i += 32) {
          const double a = Z[i * n + hi - 1];
          Z[i * n + hi - 1] = qq * a + pp * Z[i * n + hi];
          Z[i * n + hi] = qq * Z[i * n + hi] - pp * a;
        }
        __syncwarp();
        if (lane == 0)
          H[hi * n + hi - 1] = 0.0;
      } else if (lane == 0) {
        wr[hi - 1] = wr[hi] = x + p;
        wi[hi - 1] = z;
        wi[hi] = -z;
      }
      __syncwarp();
      hi -= 2;
      iter = 0;
      continue;
    }
    if (iter == 10 || iter == 20) {
      exshift += x;
      __syncwarp();
      for (int i = lane; i <= hi; i += 32)
        H[i * n + i] -= x;
      __syncwarp();
      const double s = fabs(H[hi * n + hi - 1]) + fabs(H[(hi - 1) * n + hi - 2]);
      x = y = 0.75 * s;
      w = -0.4375 * s * s;
    }
    iter++;
    total++;
    if (total > 60 * n)
      return false;
    // the scalar search runs on lane 0 and is broadcast (the other lanes
    // would only repeat it)
    int m = hi - 2;
    double p = 0, q = 0, r = 0, z;
    if (lane == 0) {
      while (m >= l) {
        z = H[m * n + m];
        r = x - z;
        double s = y - z;
        p = (r * s - w) / H[(m + 1) * n + m] + H[m * n + m + 1];
        q = H[(m + 1) * n + m + 1] - z - r - s;
        r = H[(m + 2) * n + m + 1];
        s = fabs(p) + fabs(q) + fabs(r);
        p /= s;
        q /= s;
        r /= s;
        if (m == l)
          break;
        const double u = fabs(H[m * n + m - 1]) * (fabs(q) + fabs(r));
        const double vv =
            fabs(p) * (fabs(H[(m - 1) * n + m - 1]) + fabs(z) + fabs(H[(m + 1) * n + m + 1]));
        if (u < eps * vv)
          break;
        m--;
      }
    }
    m = __shfl_sync(0xffffffffu, m, 0);
    p = __shfl_sync(0xffffffffu, p, 0);
    q = __shfl_sync(0xffffffffu, q, 0);
    r = __shfl_sync(0xffffffffu, r, 0);
    __syncwarp();
    for (int i = m + 2 + lane; i <= hi; i += 32) {
      H[i * n + i - 2] = 0.0;
      if (i > m + 2)
        H[i * n + i - 3] = 0.0;
    }
    __syncwarp();
#pragma unroll 1
    for (int k = m; k <= hi - 1; k++) {
      const bool notlast = (k != hi - 1);
      int skip = 0;
      __syncwarp();
      if (lane == 0) {
        if (k != m) {
          p = H[k * n + k - 1];
          q = H[(k + 1) * n + k - 1];
          r = notlast ? H[(k + 2) * n + k - 1] : 0.0;
          x = fabs(p) + fabs(q) + fabs(r);
          if (x == 0.0) {
            skip = 1;
          } else {
            p /= x;
            q /= x;
            r /= x;
          }
        }
        if (!skip) {
          double s = sqrt(p * p + q * q + r * r);
          if (p < 0)
            s = -s;
          if (k != m)
            H[k * n + k - 1] = -s * x;
          else if (l != m)
            H[k * n + k - 1] = -H[k * n + k - 1];
          p += s;
          x = p / s;
          y = q / s;
          z = r / s;
          q /= p;
          r /= p;
        }
      }
      skip = __shfl_sync(0xffffffffu, skip, 0);
      if (skip)
        continue;
      p = __shfl_sync(0xffffffffu, p, 0);
      q = __shfl_sync(0xffffffffu, q, 0);
      r = __shfl_sync(0xffffffffu, r, 0);
      x = __shfl_sync(0xffffffffu, x, 0);
      y = __shfl_sync(0xffffffffu, y, 0);
      z = __shfl_sync(0xffffffffu, z, 0);
      for (int j = k + lane; j < n; j += 32) {  // rows
        double pp = H[k * n + j] + q * H[(k + 1) * n + j];
        if (notlast) {
          pp += r * H[(k + 2) * n + j];
          H[(k + 2) * n + j] -= pp * z;
        }
        H[k * n + j] -= pp * x;
        H[(k + 1) * n + j] -= pp * y;
      }
      __syncwarp();
      const int ihi = hi < k + 3 ? hi : k + 3;
      for (int i = lane; i <= ihi; i += 32) {  // columns
        double pp = x * H[i * n + k] + y * H[i * n + k + 1];
        if (notlast) {
          pp += z * H[i * n + k + 2];
          H[i * n + k + 2] -= pp * r;
        }
        H[i * n + k] -= pp;
        H[i * n + k + 1] -= pp * q;
      }
      for (int i = lane; i < n; i += 32) {
        double pp = x * Z[i * n + k] + y * Z[i * n + k + 1];
        if (notlast) {
          pp += z * Z[i * n + k + 2];
          Z[i * n + k + 2] -= pp * r;
        }
        Z[i * n + k] -= pp;
        Z[i * n + k + 1] -= pp * q;
      }
      __syncwarp();
    }
  }
  return true;
}

// eigenvector k on lane k (k < n); T quasi-triangular Schur form, Z vectors
template <int n>
GPR_D void w_schur_vectors(const double *T, const double *Z, const double *wr,
                           const double *wi, double *Rr, double *Ri, int lane) {
  double nrm = 0.0;
  for (int e = lane; e < n * n; e += 32) {
    int i = e / n, j = e % n;
    if (j >= i - 1)
      nrm += fabs(T[e]);
  }
  const double norm = warp_sum(nrm);
  const int k = lane;
  if (k < n) {
    const double lr = wr[k], li = wi[k];
    double yr[n], yi[n];
#pragma unroll 1
    for (int i = 0; i < n; i++)
      yr[i] = yi[i] = 0.0;
    const bool blk2 = (k + 1 < n && T[(k + 1) * n + k] != 0.0);
    const bool blk1 = (k > 0 && T[k * n + k - 1] != 0.0);
    int top;
    if (!blk1 && !blk2) {
      yr[k] = 1.0;
      top = k;
    } else {
      const int b = blk2 ? k : k - 1;
      const double a11 = T[b * n + b] - lr, a12 = T[b * n + b + 1];
      const double a21 = T[(b + 1) * n + b];
      if (fabs(a12) >= fabs(a21)) {
        yr[b] = 1.0;
        yi[b] = 0.0;
        yr[b + 1] = -a11 / a12;
        yi[b + 1] = li / a12;
      } else {
        const double a22r = T[(b + 1) * n + b + 1] - lr;
        yr[b + 1] = 1.0;
        yi[b + 1] = 0.0;
        yr[b] = -a22r / a21;
        yi[b] = li / a21;
      }
      top = b + 1;
    }
    const int start = (blk1 || blk2) ? (blk2 ? k - 1 : k - 2) : k - 1;
#pragma unroll 1
    for (int i = start; i >= 0; i--) {
      const bool is2 = (i > 0 && T[i * n + i - 1] != 0.0);
      if (!is2) {
        double sr = 0.0, si = 0.0;
#pragma unroll 1
        for (int j = i + 1; j <= top; j++) {
          sr += T[i * n + j] * yr[j];
          si += T[i * n + j] * yi[j];
        }
        const double dr = T[i * n + i] - lr, di = -li;
        if (hypot(dr, di) <= OSH_MULT_TOL * norm) {
          yr[i] = yi[i] = 0.0;
          continue;
        }
        const double den = dr * dr + di * di;
        yr[i] = -(sr * dr + si * di) / den;
        yi[i] = -(si * dr - sr * di) / den;
      } else {
        const int a = i - 1;
        double s1r = 0, s1i = 0, s2r = 0, s2i = 0;
#pragma unroll 1
        for (int j = i + 1; j <= top; j++) {
          s1r += T[a * n + j] * yr[j];
          s1i += T[a * n + j] * yi[j];
          s2r += T[i * n + j] * yr[j];
          s2i += T[i * n + j] * yi[j];
        }
        const double m11r = T[a * n + a] - lr, m11i = -li;
        const double m12 = T[a * n + i], m21 = T[i * n + a];
        const double m22r = T[i * n + i] - lr, m22i = -li;
        const double detr = m11r * m22r - m11i * m22i - m12 * m21;
        const double deti = m11r * m22i + m11i * m22r;
        if (hypot(detr, deti) <= OSH_MULT_TOL * norm * OSH_MULT_TOL * norm) {
          yr[a] = yi[a] = yr[i] = yi[i] = 0.0;
          i--;
          continue;
        }
        const double den = detr * detr + deti * deti;
        const double nar = -(s1r * m22r - s1i * m22i) + m12 * s2r;
        const double nai = -(s1r * m22i + s1i * m22r) + m12 * s2i;
        const double nir = -(m11r * s2r - m11i * s2i) + m21 * s1r;
        const double nii = -(m11r * s2i + m11i * s2r) + m21 * s1i;
        yr[a] = (nar * detr + nai * deti) / den;
        yi[a] = (nai * detr - nar * deti) / den;
        yr[i] = (nir * detr + nii * deti) / den;
        yi[i] = (nii * detr - nir * deti) / den;
        i--;
      }
    }
#pragma unroll 1
    for (int i = 0; i < n; i++) {
      double sr = 0.0, si = 0.0;
#pragma unroll 1
      for (int j = 0; j <= top; j++) {
        sr += Z[i * n + j] * yr[j];
        si += Z[i * n + j] * yi[j];
      }
      Rr[i * n + k] = sr;
      Ri[i * n + k] = si;
    }
  }
  __syncwarp();
}

template <int n>
GPR_D bool w_csolve(double *Cr, double *Ci, double *br, double *bi, int lane) {
#pragma unroll 1
  for (int c = 0; c < n; c++) {
    double best = -1.0;
    int p = c;
    for (int r = c + lane; r < n; r += 32) {
      const double a = hypot(Cr[r * n + c], Ci[r * n + c]);
      if (a > best) {
        best = a;
        p = r;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int op = __shfl_xor_sync(0xffffffffu, p, o);
      if (ob > best || (ob == best && op < p)) {
        best = ob;
        p = op;
      }
    }
    if (best == 0.0)
      return false;
    __syncwarp();
    if (p != c) {
      for (int j = lane; j < n; j += 32) {
        double t = Cr[c * n + j];
        Cr[c * n + j] = Cr[p * n + j];
        Cr[p * n + j] = t;
        t = Ci[c * n + j];
        Ci[c * n + j] = Ci[p * n + j];
        Ci[p * n + j] = t;
      }
      if (lane < 2) {
        const int h = lane * n;
        double t = br[h + c];
        br[h + c] = br[h + p];
        br[h + p] = t;
        t = bi[h + c];
        bi[h + c] = bi[h + p];
        bi[h + p] = t;
      }
    }
    __syncwarp();
    const double pr = Cr[c * n + c], pi = Ci[c * n + c];
    const double den = pr * pr + pi * pi;
    for (int r = c + 1 + lane; r < n; r += 32) {
      const double ar = Cr[r * n + c], ai = Ci[r * n + c];
      const double fr = (ar * pr + ai * pi) / den, fi = (ai * pr - ar * pi) / den;
      for (int j = c; j < n; j++) {
        const double xr = Cr[c * n + j], xi = Ci[c * n + j];
        Cr[r * n + j] -= fr * xr - fi * xi;
        Ci[r * n + j] -= fr * xi + fi * xr;
      }
      for (int h = 0; h < 2 * n; h += n) {
        const double xr = br[h + c], xi = bi[h + c];
        br[h + r] -= fr * xr - fi * xi;
        bi[h + r] -= fr * xi + fi * xr;
      }
    }
    __syncwarp();
  }
  // back-substitution, one right-hand side per lane
  if (lane < 2) {
    const int h = lane * n;
#pragma unroll 1
    for (int r = n - 1; r >= 0; r--) {
      double sr = br[h + r], si = bi[h + r];
      for (int j = r + 1; j < n; j++) {
        sr -= Cr[r * n + j] * br[h + j] - Ci[r * n + j] * bi[h + j];
        si -= Cr[r * n + j] * bi[h + j] + Ci[r * n + j] * br[h + j];
      }
      const double pr = Cr[r * n + r], pi = Ci[r * n + r];
      const double den = pr * pr + pi * pi;
      br[h + r] = (sr * pr + si * pi) / den;
      bi[h + r] = (si * pr - sr * pi) / den;
    }
  }
  __syncwarp();
  return true;
}

// ws.f += w |M| ws.dq for M given by ws.H (C, destroyed), ws.Ba and ws.vb, as
// abs_apply.
template <class L>
GPR_D AbsStatus w_abs_apply(EigWS<L> &ws, double w, int lane, bool strict = false) {
  constexpr int V = L::V, n = ACTIVE_N<L>;
  for (int e = lane; e < n * n; e += 32)
    ws.Z[e] = (e % (n + 1) == 0) ? 1.0 : 0.0;
  __syncwarp();
  w_hess<n>(ws.H, ws.Z, ws.v, lane);
  if (!w_hqr<n>(ws.H, ws.Z, ws.wr, ws.wi, lane))
    return ABS_FAILED;
  __syncwarp();
  const bool real = __all_sync(0xffffffffu, lane >= n || ws.wi[lane < n ? lane : 0] == 0.0);
  double out = 0.0;  // entry `lane` of the active result
  double nrm = 0.0;
  for (int e = lane; e < n * n; e += 32)
    if (e % n >= e / n)
      nrm += fabs(ws.H[e]);
  const double tol = OSH_MULT_TOL * warp_sum(nrm);
  double part = tol * max_passive<L>(ws.dq);
  if (!strict || fabs(ws.vb) > tol)
    part = INFINITY;
  if (real) {
    double *Y = ws.Rr, *y = ws.br, *c2 = ws.br + n;  // Y by columns
    if (lane < n) {
      const int k = lane;
      double x1 = 0.0, x2 = 0.0;
      for (int i = 0; i < n; i++) {
        x1 += ws.Z[i * n + k] * ws.dq[active_entry(i)];
        x2 += ws.Z[i * n + k] * ws.Ba[i];
      }
      y[k] = x1;
      c2[k] = x2;
      Y[k * n + k] = 1.0;
      for (int i = k - 1; i >= 0; i--) {
        double sum = 0.0;
        for (int j = i + 1; j <= k; j++)
          sum += ws.H[i * n + j] * Y[k * n + j];
        const double d = ws.H[i * n + i] - ws.wr[k];
        Y[k * n + i] = fabs(d) <= tol ? 0.0 : -sum / d;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int k = n - 1; k > 0; k--) {
      if (lane < k) {
        y[lane] -= Y[k * n + lane] * y[k];
        c2[lane] -= Y[k * n + lane] * c2[k];
      }
      __syncwarp();
    }
    if (__any_sync(0xffffffffu,
                   lane < n && fabs(ws.wr[lane < n ? lane : 0]) <= tol && fabs(c2[lane < n ? lane : 0]) > part))
      return ABS_TWO_LIMITS;
    if (lane < n) {
      double fa, gr, gi;
      abs_factors(ws.wr[lane], 0.0, ws.vb, tol, fa, gr, gi);
      y[lane] = fa * y[lane] + gr * c2[lane];
    }
    __syncwarp();
    double sum = 0.0;
    if (lane < n)
      for (int k = lane; k < n; k++)
        sum += Y[k * n + lane] * y[k];
    if (lane < n)
      c2[lane] = sum;
    __syncwarp();
    if (lane < n)
      for (int k = 0; k < n; k++)
        out += ws.Z[lane * n + k] * c2[k];
  } else {
    w_schur_vectors<n>(ws.H, ws.Z, ws.wr, ws.wi, ws.Rr, ws.Ri, lane);
    double *Cr = ws.H, *Ci = ws.Z;
    for (int e = lane; e < n * n; e += 32) {
      Cr[e] = ws.Rr[e];
      Ci[e] = ws.Ri[e];
    }
    if (lane < n) {
      ws.br[lane] = ws.dq[active_entry(lane)];
      ws.br[n + lane] = ws.Ba[lane];
      ws.bi[lane] = ws.bi[n + lane] = 0.0;
    }
    __syncwarp();
    if (!w_csolve<n>(Cr, Ci, ws.br, ws.bi, lane))
      return ABS_FAILED;
    const int kl = lane < n ? lane : 0;
    if (__any_sync(0xffffffffu, lane < n && hypot(ws.wr[kl], ws.wi[kl]) <= tol &&
                                    hypot(ws.br[n + kl], ws.bi[n + kl]) > part))
      return ABS_TWO_LIMITS;
    if (lane < n) {
      double fa, gr, gi;
      abs_factors(ws.wr[lane], ws.wi[lane], ws.vb, tol, fa, gr, gi);
      const double b2r = ws.br[n + lane], b2i = ws.bi[n + lane];
      ws.br[lane] = fa * ws.br[lane] + (gr * b2r - gi * b2i);
      ws.bi[lane] = fa * ws.bi[lane] + (gr * b2i + gi * b2r);
    }
    __syncwarp();
    if (lane < n)
      for (int k = 0; k < n; k++)
        out += ws.Rr[lane * n + k] * ws.br[k] - ws.Ri[lane * n + k] * ws.bi[k];
  }
  if (lane < n)
    ws.f[active_entry(lane)] += w * out;
  for (int k = 5 + lane; k < V; k += 32)
    if (passive_entry<L>(k))
      ws.f[k] += w * fabs(ws.vb) * ws.dq[k];
  __syncwarp();
  return ABS_OK;
}

// wt times the system matrix of ws.q added to ws.H, ws.Ba and ws.vb (as
// system_active): F and D are built in ws.Rr / ws.Ri by lane 0, the products
// formed by all lanes.
template <class L> GPR_D void w_system_active(EigWS<L> &ws, double wt, const DevPar &P, int lane) {
  constexpr int V = L::V, n = ACTIVE_N<L>;
  for (int e = lane; e < V * V; e += 32) {
    ws.Rr[e] = 0.0;
    ws.Ri[e] = 0.0;
  }
  __syncwarp();
  if (lane == 0) {
    double q[V];
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = ws.q[k];
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(q, P, s);
    system_fd<L::THERMAL, V>(q, s, P, ws.Rr, ws.Ri);
    ws.v[0] = s.v[0];
    ws.v[1] = s.v[1];
    ws.v[2] = s.v[2];
  }
  __syncwarp();
  const double *F = ws.Rr, *D = ws.Ri;
  auto entry = [&](int R, int j) {  // M(R, j) of the active row R
    double x = F[R * V + 1] * D[V + j];
    if (j != 1)
      x += F[R * V + j] * D[j * V + j];
    if (j == 0) {
      for (int k = 2; k < 5; k++)
        x += F[R * V + k] * D[k * V];
      if (L::THERMAL)
        for (int k = 14; k < 17; k++)
          x += F[R * V + k] * D[k * V];
    }
    if (R >= 5 && R < 14) {
      if (j == R)
        x += ws.v[0];
      if (j >= R && j < R + 3)
        x -= ws.v[j - R];
    }
    return x;
  };
  for (int e = lane; e < n * n; e += 32)
    ws.H[e] += wt * entry(active_entry(e / n), active_entry(e % n));
  if (lane < n) {
    double ba = 0.0;
    for (int j = 5; j < 14; j++)
      if (passive_entry<L>(j))
        ba += entry(active_entry(lane), j) * ws.dq[j];
    ws.Ba[lane] += wt * ba;
  }
  if (lane == 0)
    ws.vb += wt * ws.v[0];
  __syncwarp();
}

// ws.f = |M| ws.dq by the whole matrix of Roe's path average, as roe_whole.
template <class L> GPR_D bool w_roe_whole(EigWS<L> &ws, const DevPar &P, const Consts &C, int lane) {
  constexpr int V = L::V;
  for (int e = lane; e < V * V; e += 32)
    ws.Z[e] = 0.0;
#pragma unroll 1
  for (int n = 0; n < NN; n++) {
    for (int k = lane; k < V; k += 32)
      ws.q[k] = ws.qr[k] + C.nodes[n] * ws.dq[k];
    for (int e = lane; e < V * V; e += 32)
      ws.Rr[e] = ws.Ri[e] = 0.0;
    __syncwarp();
    if (lane == 0) {
      double q[V];
#pragma unroll
      for (int k = 0; k < V; k++)
        q[k] = ws.q[k];
      Prim<L::THERMAL> s;
      prim<L::THERMAL>(q, P, s);
      system_fd<L::THERMAL, V>(q, s, P, ws.Rr, ws.Ri);
      ws.v[0] = s.v[0];
      ws.v[1] = s.v[1];
      ws.v[2] = s.v[2];
    }
    __syncwarp();
    for (int e = lane; e < V * V; e += 32) {
      const int i = e / V, j = e % V;
      double x = 0.0;
      for (int k = 0; k < V; k++)
        x += ws.Rr[i * V + k] * ws.Ri[k * V + j];
      ws.H[e] = x;
    }
    __syncwarp();
    if (lane == 0)
      system_block<V, L::LSET>(ws.v, ws.H);
    __syncwarp();
    for (int e = lane; e < V * V; e += 32)
      ws.Z[e] += C.w[n] * ws.H[e];
    __syncwarp();
  }
  for (int e = lane; e < V * V; e += 32) {
    ws.H[e] = ws.Z[e];
    ws.Z[e] = (e % (V + 1) == 0) ? 1.0 : 0.0;
  }
  __syncwarp();
  w_hess<V>(ws.H, ws.Z, ws.v, lane);
  if (!w_hqr<V>(ws.H, ws.Z, ws.wr, ws.wi, lane))
    return false;
  __syncwarp();
  w_schur_vectors<V>(ws.H, ws.Z, ws.wr, ws.wi, ws.Rr, ws.Ri, lane);
  for (int e = lane; e < V * V; e += 32) {
    ws.H[e] = ws.Rr[e];
    ws.Z[e] = ws.Ri[e];
  }
  if (lane < V) {
    ws.br[lane] = ws.dq[lane];
    ws.br[V + lane] = ws.bi[lane] = ws.bi[V + lane] = 0.0;
  }
  __syncwarp();
  if (!w_csolve<V>(ws.H, ws.Z, ws.br, ws.bi, lane))
    return false;
  if (lane < V) {
    const double a = hypot(ws.wr[lane], ws.wi[lane]);
    ws.br[lane] *= a;
    ws.bi[lane] *= a;
  }
  __syncwarp();
  if (lane < V) {
    double x = 0.0;
    for (int k = 0; k < V; k++)
      x += ws.Rr[lane * V + k] * ws.br[k] - ws.Ri[lane * V + k] * ws.bi[k];
    ws.f[lane] = x;
  }
  __syncwarp();
  return true;
}

// Osher interface terms at one point along D: f = D + F(qL) + F(qR), b = Bint.
template <class L, int D>
GPR_D void osher_point(const double *ql, const double *qr, const DevPar &P, const Consts &C,
                       double *f, double *b) {
  constexpr int V = L::V;
  eig_dissipation_qd<L, NN>(ql, qr, D, GPR_FLUX_OSHER, P, C.nodes, C.w, f);
  Prim<L::THERMAL> sl, sr;
  prim<L::THERMAL>(ql, P, sl);
  prim<L::THERMAL>(qr, P, sr);
  flux_add<L::THERMAL, V>(ql, sl, D, P, f);
  flux_add<L::THERMAL, V>(qr, sr, D, P, f);
  double dq[V];
#pragma unroll
  for (int k = 0; k < V; k++)
    dq[k] = qr[k] - ql[k];
  path_product<L, NN>(ql, dq, D, C.nodes, C.w, b);
}

// 2D faces with the Osher dissipation in closed form: the lanes, passes and
// in-place update of k_faces2d.
template <class L, int DIR>
__global__ void __launch_bounds__(128) k_faces2d_osher(
    double *__restrict__ fb, const double *__restrict__ qh, int nx, int ny,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double ih,
    int time_dg, DevPar P, Consts C, int parity) {
  constexpr int V = L::V;
  double f[V], b[V];
  faces2d_body<L, DIR>(fb, qh, nx, ny, mask, dt, dt_dev, ih, time_dg, C, parity, f, b,
                       [&](const double *ql, const double *qr) {
                         osher_point<L, DIR>(ql, qr, P, C, f, b);
                       });
}

// 1D faces with the Osher dissipation in closed form, one lane per (face,
// time node, side) as k_faces1d_split: side 0 (1) evaluates the flux of qL (qR)
// and path node 0 (1) of the dissipation and of Bint.  A face with a point the
// closed form declines gets OSHER_MARK in its first entry, and the
// warp-cooperative k_faces1d_eigw, launched next, evaluates the marked faces
// (on the device: whether there are any is not known to the host; the launch
// of blocks that return at once takes ~3 us).  The general routine per thread
// would give this kernel an 18 KB stack, which a caller that cannot let the
// device allocate must not meet.
constexpr unsigned long long OSHER_MARK = 0x7ff8000000000badull;
template <class L>
__global__ void __launch_bounds__(128) k_faces1d_osher(
    double *__restrict__ fb, const double *__restrict__ qh, long nface,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double idx,
    int time_dg, DevPar P, Consts C) {
  constexpr int V = L::V;
  static_assert(NN == 2, "two time nodes and two path nodes");
  if (dt_dev)
    dt = *dt_dev;
  const long face = (blockIdx.x * (long)blockDim.x + threadIdx.x) / 4;
  const int lq = threadIdx.x % 4, t = lq >> 1, side = lq & 1;
  const bool valid = face < nface;
  const long fi = valid ? face : 0;
  const bool on = valid && (mask == nullptr || (mask[fi] && mask[fi + 1]));
  const bool active = on && (time_dg || t == 0);
  const int nt = time_dg ? NN : 1, tt = time_dg ? t : 0;
  // each lane extrapolates its own side and takes the other from its partner
  const double *qs_ = qh + ((fi + side) * nt + tt) * NN * V;
  const double e0 = C.endv[1 - side][0], e1 = C.endv[1 - side][1];
  double qs[V], ql[V], qr[V], dq[V], f[V], b[V];
  bool flat = true;
#pragma unroll
  for (int k = 0; k < V; k++) {
    qs[k] = e0 * qs_[k] + e1 * qs_[V + k];
    const double o = __shfl_xor_sync(0xffffffffu, qs[k], 1);
    ql[k] = side ? o : qs[k];
    qr[k] = side ? qs[k] : o;
    dq[k] = ql[k] - qr[k];
    f[k] = 0.0;
    flat = flat && (__double_as_longlong(dq[k]) << 1) == 0;
  }
  bool ok = true;
  if (active && !flat) {
    double q[V];
    const double xn = C.nodes[side];
#pragma unroll
    for (int k = 0; k < V; k++)
      q[k] = fma(xn, dq[k], qr[k]);
    ok = abs_apply_acoustic<L>(q, dq, GAUSS_W, P, f);
  }
  {
#pragma unroll
    for (int k = 0; k < V; k++)
      dq[k] = -dq[k];
    Prim<L::THERMAL> s;
    prim<L::THERMAL>(qs, P, s);
    flux_add<L::THERMAL, V>(qs, s, 0, P, f);
    const double xn = C.nodes[side];
    const double wr = GAUSS_W * rcp64(fma(xn, dq[0], ql[0]));
    const double v[3] = {fma(xn, dq[2], ql[2]) * wr, fma(xn, dq[3], ql[3]) * wr,
                         fma(xn, dq[4], ql[4]) * wr};
    bdot<V, L::LSET>(v, dq, 0, b);
  }
  const double kk = dt * idx * (time_dg ? 0.5 * GAUSS_W : 0.5);
  face_reduce_store<V, 4>(b, f, kk, active, valid, lq, fb + fi * 2 * V);
  const unsigned lane = threadIdx.x & 31u;
  const bool bad = (__ballot_sync(0xffffffffu, !ok) >> (lane & ~3u)) & 0xfu;
  __syncwarp();
  // lane 0 of the face holds entry 0 after the reduction
  if (valid && bad && lq == 0)
    fb[fi * 2 * V] = __longlong_as_double((long long)OSHER_MARK);
}

// 1D faces with the Osher or Roe dissipation: one block per face, one warp
// per eigen-decomposition: warp w = t * NPATH + i handles time node t and,
// for Osher, path node i (NPATH = 2; Roe averages the path's matrices in one
// warp, NPATH = 1).  The contributions are summed in the serial order (path
// nodes, then time nodes); output as k_faces1d.  Roe's flux, and the Osher
// points that the closed form declines (marked != 0).
constexpr int EIG_WARPS = 4;

template <class L, bool BATCH = false>
__global__ void __launch_bounds__(32 * EIG_WARPS) k_faces1d_eigw(
    double *__restrict__ fb, const double *__restrict__ qh, long nface,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double dx,
    int time_dg, int flux, DevPar Pv, Consts C, Batch B, int marked) {
  constexpr int V = L::V;
  __shared__ EigWS<L> wsa[EIG_WARPS];
  __shared__ double part[NN][2][V];
  if (dt_dev)
    dt = *dt_dev;
  const int wid = threadIdx.x / 32, lane = threadIdx.x % 32;
  const long face = blockIdx.x;
  if (face >= nface)
    return;  // block-uniform
  // marked: only the faces k_faces1d_osher left (block-uniform: the block
  // writes the entry after its last barrier)
  if (marked &&
      (unsigned long long)__double_as_longlong(fb[face * 2 * V]) != OSHER_MARK)
    return;
  long fi = face;
  const int inst = BATCH ? B.inst_f[face] : 0;
  const DevPar &P = BATCH ? B.P[inst] : Pv;
  if (BATCH) {
    fi = B.off_b[inst] + (face - B.off_f[inst]);
    dt = B.clk[5 * inst + 1];
    dx = 1.0 / B.idx[inst];
  }
  const bool active = mask == nullptr || (mask[fi] && mask[fi + 1]);
  const int nt = time_dg ? NN : 1;
  const int npath = flux == GPR_FLUX_OSHER ? NN : 1;
  const int t = wid / npath, ip = wid % npath;
  const bool mine = active && t < nt;  // warp-uniform
  EigWS<L> &ws = wsa[wid];
  if (mine) {
    const double *ql_ = qh + (fi * nt + t) * NN * V;
    const double *qr_ = qh + ((fi + 1) * nt + t) * NN * V;
    for (int k = lane; k < V; k += 32) {
      ws.ql[k] = C.endv[1][0] * ql_[k] + C.endv[1][1] * ql_[V + k];
      ws.qr[k] = C.endv[0][0] * qr_[k] + C.endv[0][1] * qr_[V + k];
      ws.dq[k] = ws.ql[k] - ws.qr[k];
      ws.f[k] = 0.0;
    }
    __syncwarp();
    // qL = qR (a uniform region): |A| dq is exactly zero, whatever A's
    // eigen-decomposition; the dissipation stays zero without it
    bool flat = true;
    for (int k = lane; k < V; k += 32)
      flat = flat && ws.dq[k] == 0.0;
    flat = __all_sync(0xffffffffu, flat);
    bool ok = true;
    if (!flat) {
      // Osher: this warp's path node; Roe: the path-averaged matrix
      constexpr int n = ACTIVE_N<L>;
      for (int e = lane; e < n * n; e += 32)
        ws.H[e] = 0.0;
      if (lane < n)
        ws.Ba[lane] = 0.0;
      if (lane == 0)
        ws.vb = 0.0;
      const bool osher = flux == GPR_FLUX_OSHER;
#pragma unroll 1
      for (int i = osher ? ip : 0; i < (osher ? ip + 1 : NN); i++) {
        for (int k = lane; k < V; k += 32)
          ws.q[k] = ws.qr[k] + C.nodes[i] * ws.dq[k];
        __syncwarp();
        w_system_active<L>(ws, osher ? 1.0 : C.w[i], P, lane);
      }
      const AbsStatus rc =
          w_abs_apply<L>(ws, osher ? C.w[ip] : 1.0, lane, !osher && !L::THERMAL);
      ok = rc == ABS_OK;
      if constexpr (!L::THERMAL) {
        if (rc == ABS_TWO_LIMITS)
          ok = w_roe_whole<L>(ws, P, C, lane);
      }
    }
    if (!ok) {
      for (int k = lane; k < V; k += 32)
        ws.f[k] = __longlong_as_double(0x7ff8000000000000ll);
    }
  }
  __syncthreads();
  // warp t (path node 0) finishes time node t: D + F(qL) + F(qR) and Bint
  if (mine && ip == 0 && lane == 0) {
    double ql[V], qr[V], f[V], b[V], dq[V];
#pragma unroll
    for (int k = 0; k < V; k++) {
      ql[k] = ws.ql[k];
      qr[k] = ws.qr[k];
      double acc = 0.0;
      for (int i = 0; i < npath; i++)
        acc += wsa[t * npath + i].f[k];
      f[k] = acc;
    }
    Prim<L::THERMAL> sl, sr;
    prim<L::THERMAL>(ql, P, sl);
    prim<L::THERMAL>(qr, P, sr);
    flux_add<L::THERMAL, V>(ql, sl, 0, P, f);
    flux_add<L::THERMAL, V>(qr, sr, 0, P, f);
#pragma unroll
    for (int k = 0; k < V; k++) {
      dq[k] = qr[k] - ql[k];
      b[k] = 0.0;
    }
#pragma unroll
    for (int nn = 0; nn < NN; nn++) {
      const double rho = ql[0] + C.nodes[nn] * dq[0];
      const double ir = 1.0 / rho;
      const double v[3] = {(ql[2] + C.nodes[nn] * dq[2]) * ir, (ql[3] + C.nodes[nn] * dq[3]) * ir,
                           (ql[4] + C.nodes[nn] * dq[4]) * ir};
      double bd[V];
      bdot<V, L::LSET>(v, dq, 0, bd);
#pragma unroll
      for (int k = 0; k < V; k++)
        b[k] += C.w[nn] * bd[k];
    }
    const double kk = (time_dg ? dt * C.w[t] : dt) / (2.0 * dx);
#pragma unroll
    for (int k = 0; k < V; k++) {
      part[t][0][k] = kk * (b[k] + f[k]);
      part[t][1][k] = kk * (b[k] - f[k]);
    }
  }
  __syncthreads();
  if (wid == 0) {
    double *out = fb + face * 2 * V;
    for (int k = lane; k < V; k += 32) {
      double l = 0.0, r = 0.0;
      if (active) {
        l = part[0][0][k];
        r = part[0][1][k];
        if (nt == 2) {
          l += part[1][0][k];
          r += part[1][1][k];
        }
      }
      out[k] = l;
      out[V + k] = r;
    }
  }
}

// 2D Roe faces (and Osher's where its closed form does not hold): one thread
// per face quadrature point (time node t, transverse node s) of both directions
// (blockIdx.y): a point is one thread's serial chain, so the two directions side
// by side share one tail (fv_launcher, Roe: 64^2 4.75 to 3.34 ms, 160^2 21.0 to
// 19.2, 512^2 157.0 to 155.8).  The four points of a face lie in neighbouring
// lanes, which add kk (b + f) and kk (b - f) as (l0 + l1) + (l2 + l3) and write
// the sums to fb[dir][face][2][V]; terms kept per point in global memory would
// need 1088 bytes a face and direction at V = 17.
template <class L>
__global__ void __launch_bounds__(64) k_faces2d_eigp(
    double *__restrict__ fb, const double *__restrict__ qh, int nx, int ny,
    const uint8_t *__restrict__ mask, double dt, const double *__restrict__ dt_dev, double dx,
    double dy, int time_dg, int flux, DevPar P, Consts C) {
  constexpr int V = L::V;
  constexpr int NQ = NN * NN;
  static_assert(NQ == 4, "four quadrature points per 2D face");
  const int dir = blockIdx.y;
  if (dt_dev)
    dt = *dt_dev;
  const long gt = blockIdx.x * (long)blockDim.x + threadIdx.x;
  const long nf = (long)(nx + 1) * (ny + 1);
  const bool valid = gt < nf * NQ;
  const long fi = valid ? gt / NQ : 0;
  const int lq = (int)(gt % NQ), t = lq / NN, s = lq % NN;
  const int i = fi / (ny + 1), j = fi % (ny + 1);
  const long cb = (long)i * (ny + 2) + j;
  const long cn = dir == 0 ? cb + (ny + 2) : cb + 1;
  const bool geo = valid && (dir == 0 ? (j > 0) : (i > 0));
  const bool active = geo && (mask == nullptr || (mask[cb] && mask[cn])) && (time_dg || t == 0);
  double f[V], b[V], kk = 0.0;
  if (active) {
    const int nt = time_dg ? NN : 1, tt = time_dg ? t : 0;
    const double *q0 = qh + (cb * nt + tt) * NN * NN * V;
    const double *q1 = qh + (cn * nt + tt) * NN * NN * V;
    double ql[V], qr[V];
    const long o0 = dir == 0 ? (long)s * V : (long)s * NN * V;
    const long st = dir == 0 ? (long)NN * V : (long)V;
#pragma unroll
    for (int k = 0; k < V; k++) {
      ql[k] = C.endv[1][0] * q0[o0 + k] + C.endv[1][1] * q0[o0 + st + k];
      qr[k] = C.endv[0][0] * q1[o0 + k] + C.endv[0][1] * q1[o0 + st + k];
    }
    const double wt = time_dg ? dt * C.w[t] : dt;
    kk = wt / (2.0 * (dir == 0 ? dx : dy)) * C.w[s];
    interface_point_eig<L>(ql, qr, flux, P, C, f, b, dir);
  }
  __syncwarp();
  double *o = fb + (dir * nf + fi) * 2 * V;
#pragma unroll
  for (int h = 0; h < 2; h++)
#pragma unroll
    for (int k = 0; k < V; k++) {
      double x = active ? kk * (h == 0 ? b[k] + f[k] : b[k] - f[k]) : 0.0;
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      if (valid && lq == (h * V + k) % NQ)
        o[h * V + k] = x;
    }
}

}  // namespace gpr
