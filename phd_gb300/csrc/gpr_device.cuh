// gpr_device.cuh - device-side GPR (Godunov-Peshkov-Romenski) physics in FP64.
//
// Pointwise functions of one conserved state Q[V] (registers), restating the
// reference's system library (code/cpp/src/system/*.cpp) with the derived
// quantities of a state computed once (`Prim`) and shared by flux, source,
// the non-conservative product and the wave-speed bound, instead of being
// recomputed per call as the reference does (pressure() alone is evaluated
// 4-6 times per node there).  Every function cites the reference it restates.
//
// Layout of Q: [rho, rho E, rho v(3), A(3x3 row-major), rho J(3) if THERMAL,
// phi(LSET)].
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../include/gpr_gb300.h"

#define GPR_HD __host__ __device__ __forceinline__
#define GPR_D __device__ __forceinline__

#ifndef GPR_FASTMATH_PROVIDED  // a host build of this header brings its own
#include "gpr_fastmath.cuh"
#endif

namespace gpr {

// the least positive normal double (DBL_MIN)
constexpr double DBL_MIN_NORMAL = 2.2250738585072014e-308;

// Material parameters with the per-material constants the kernels need
// hoisted out of the per-node code (e.g. rho0 / (2 mu^(1/n)), 1/kappa).
struct DevPar {
  int EOS, flags;
  double rho0, ir0, Tref, cv, icv, pINF, Gamma0, c02, s, alpha, beta, gamma;
  double A, B, R1, R2;
  double b02, mu, tau0, sigmaY, n, calpha2, kappa, ikappa;
  double dp0, dp1, dp2;
  double th1c;   // rho0 / (2 mu^(1/n))          (sources.cpp:71)
  double tau1;   // 6 mu^(1/n) / (rho0 b02)      (analytic.cpp:62)
  double iG;     // 1/Gamma for the constant-Gamma EOS; 1/(Gamma0 rho0) for shock MG
  double C0f;    // 1 - beta/Gamma for the constant-Gamma EOS
  // Per-material products and tests, formed once on the host: in a kernel
  // each would be an FP64 instruction of every thread (a comparison too runs
  // on the FP64 pipe).
  double gm1;    // gamma - 1
  double b1;     // 1 + beta
  double b02q;   // b02 / 4
  double hca2;   // calpha2 / 2
  double ca2ik;  // calpha2 / kappa
  int has_beta, has_tref, has_dp;  // beta, Tref, dp not all zero
};

inline DevPar make_devpar(const gpr_par &p) {
  DevPar d;
  d.EOS = p.EOS;
  d.flags = p.flags;
  d.rho0 = p.rho0;
  d.ir0 = 1.0 / p.rho0;
  d.Tref = p.Tref;
  d.cv = p.cv;
  d.icv = 1.0 / p.cv;
  d.pINF = p.pINF;
  d.Gamma0 = p.Gamma0;
  d.c02 = p.c02;
  d.s = p.s;
  d.alpha = p.alpha;
  d.beta = p.beta;
  d.gamma = p.gamma;
  d.A = p.A;
  d.B = p.B;
  d.R1 = p.R1;
  d.R2 = p.R2;
  d.b02 = p.b02;
  d.mu = p.mu;
  d.tau0 = p.tau0;
  d.sigmaY = p.sigmaY;
  d.n = p.n;
  d.calpha2 = p.calpha2;
  d.kappa = p.kappa;
  d.ikappa = 1.0 / p.kappa;
  d.dp0 = p.dp[0];
  d.dp1 = p.dp[1];
  d.dp2 = p.dp[2];
  d.th1c = p.rho0 / (2.0 * pow(p.mu, 1.0 / p.n));
  d.tau1 = 6.0 * pow(p.mu, 1.0 / p.n) / (p.rho0 * p.b02);
  double G = p.EOS == 0 ? p.gamma - 1.0 : (p.EOS == 4 ? p.gamma : p.Gamma0);
  d.iG = p.EOS == 1 ? 1.0 / (p.Gamma0 * p.rho0) : 1.0 / G;
  d.C0f = 1.0 - p.beta / G;
  d.gm1 = p.gamma - 1.0;
  d.b1 = 1.0 + p.beta;
  d.b02q = 0.25 * p.b02;
  d.hca2 = 0.5 * p.calpha2;
  d.ca2ik = p.calpha2 * d.ikappa;
  // a NaN counts as present, as it does in the comparison x != 0
  d.has_beta = p.beta != 0.0;
  d.has_tref = p.Tref != 0.0;
  d.has_dp = p.dp[0] != 0.0 || p.dp[1] != 0.0 || p.dp[2] != 0.0;
  return d;
}

// ---------------------------------------------------------------------------
// Mie-Gruneisen EOS family (system/energy/mg.cpp:6-303).  EOS codes:
// 0 stiffened gas, 1 shock MG, 2 JWL, 3 Cochran-Chan, 4 Godunov-Romenski.

struct EosRho {  // density-only EOS quantities
  double G;      // Gamma_MG
  double dG;     // dGamma/drho
  double pr;     // p_ref
  double dpr;    // dp_ref/drho
  double er;     // e_ref
  double der;    // de_ref/drho
  double phi;    // integrating factor (only multiplied by Tref)
};

GPR_D EosRho eos_rho(double r, double ir, const DevPar &P) {
  EosRho e;
  switch (P.EOS) {
  case 0: {  // stiffened gas
    e.G = P.gm1;
    e.dG = 0.0;
    e.pr = -P.pINF;
    e.dpr = 0.0;
    e.er = P.pINF * ir;
    e.der = e.pr * ir * ir;
    e.phi = P.has_tref ? pow(r * P.ir0, P.gm1) : 0.0;
  } break;
  case 1: {  // shock Mie-Gruneisen
    e.G = P.Gamma0 * P.rho0 * ir;
    e.dG = -P.Gamma0 * P.rho0 * ir * ir;
    if (r > P.rho0) {
      double tmp = P.ir0 - P.s * (P.ir0 - ir);
      e.pr = P.c02 * (P.ir0 - ir) / (tmp * tmp);
      double t2 = P.s * (r - P.rho0) - r;
      e.dpr = P.c02 * P.rho0 * P.rho0 * (P.s * (P.rho0 - r) - r) / (t2 * t2 * t2);
      e.er = 0.5 * e.pr * (P.ir0 - ir);
      e.der = -(r - P.rho0) * P.rho0 * P.c02 / (t2 * t2 * t2);
    } else {
      e.pr = P.c02 * (r - P.rho0);
      e.dpr = P.c02;
      e.er = 0.0;
      e.der = 0.0;
    }
    e.phi = P.has_tref ? exp(P.Gamma0 * (1.0 - P.rho0 * ir)) : 0.0;
  } break;
  case 4: {  // Godunov-Romenski
    e.G = P.gamma;
    e.dG = 0.0;
    double tmp = pow(r * P.ir0, P.alpha);
    e.pr = P.c02 * r / P.alpha * (tmp - 1.0) * tmp;
    e.dpr = P.c02 / P.alpha * tmp * ((1.0 + P.alpha) * (tmp - 1.0) + P.alpha * tmp);
    e.er = P.c02 / (2.0 * P.alpha * P.alpha) * (tmp - 1.0) * (tmp - 1.0);
    e.der = e.pr * ir * ir;
    e.phi = P.has_tref ? pow(r * P.ir0, P.gamma) : 0.0;
  } break;
  case 2: {  // JWL
    e.G = P.Gamma0;
    e.dG = 0.0;
    double v_ = P.rho0 * ir;
    double e1 = exp(-P.R1 * v_), e2 = exp(-P.R2 * v_);
    e.pr = P.A * e1 + P.B * e2;
    e.dpr = v_ * ir * (P.A * P.R1 * e1 + P.B * P.R2 * e2);
    e.er = P.A / (P.rho0 * P.R1) * e1 + P.B / (P.rho0 * P.R2) * e2;
    e.der = e.pr * ir * ir;
    e.phi = P.has_tref ? pow(r * P.ir0, P.Gamma0) : 0.0;
  } break;
  default: {  // Cochran-Chan
    e.G = P.Gamma0;
    e.dG = 0.0;
    double v_ = P.rho0 * ir;
    double a1 = pow(v_, -P.R1), a2 = pow(v_, -P.R2);
    e.pr = P.A * a1 - P.B * a2;
    e.dpr = P.A * P.R1 * ir * a1 - P.B * P.R2 * ir * a2;
    e.er = -P.A / (P.rho0 * (1.0 - P.R1)) * (pow(v_, 1.0 - P.R1) - 1.0) +
           P.B / (P.rho0 * (1.0 - P.R2)) * (pow(v_, 1.0 - P.R2) - 1.0);
    e.der = e.pr * ir * ir;
    e.phi = P.has_tref ? pow(r * P.ir0, P.Gamma0) : 0.0;
  } break;
  }
  return e;
}

// ---------------------------------------------------------------------------
// Derived quantities of one state (variables/state.cpp, energy/eos.cpp,
// functions/matrices.cpp).  G = A^T A, devG = G - tr(G)/3 I.  |dev G|^2 is
// evaluated from A^T A; the reference's devGsq (matrices.cpp:16-26) uses the
// rows of A (A A^T), which has the same trace and Frobenius norm.
template <bool TH> struct Prim {
  double r, ir;          // rho, 1/rho
  double v[3];           // velocity
  double J[3];           // thermal impulse (TH)
  double AdG[9];         // A devG (row-major)
  double G[6];           // A^T A: 00, 11, 22, 01, 02, 12
  double S[6];           // devG A^T A (symmetric: the factors commute), same order
  double cs2;            // b02 (rho/rho0)^beta
  double devGsq;         // |dev G|^2
  double p, T;           // pressure, temperature
  double irG;            // 1 / (rho Gamma)
  EosRho e;
};

// entry (i, d) of a symmetric 3x3 matrix stored as 00, 11, 22, 01, 02, 12 (i a
// compile-time constant after unrolling; selects for a run-time d)
GPR_D double sym3(const double *m, int i, int d) {
  if (i == 0)
    return d == 0 ? m[0] : (d == 1 ? m[3] : m[4]);
  if (i == 1)
    return d == 0 ? m[3] : (d == 1 ? m[1] : m[5]);
  return d == 0 ? m[4] : (d == 1 ? m[5] : m[2]);
}

template <bool TH>
GPR_D void prim(const double *q, const DevPar &P, Prim<TH> &s) {
  s.r = q[0];
  s.ir = rcp64(s.r);
  s.v[0] = q[2] * s.ir;
  s.v[1] = q[3] * s.ir;
  s.v[2] = q[4] * s.ir;
  const double *A = q + 5;
  double G00 = A[0] * A[0] + A[3] * A[3] + A[6] * A[6];
  double G11 = A[1] * A[1] + A[4] * A[4] + A[7] * A[7];
  double G22 = A[2] * A[2] + A[5] * A[5] + A[8] * A[8];
  double G01 = A[0] * A[1] + A[3] * A[4] + A[6] * A[7];
  double G02 = A[0] * A[2] + A[3] * A[5] + A[6] * A[8];
  double G12 = A[1] * A[2] + A[4] * A[5] + A[7] * A[8];
  double t = (G00 + G11 + G22) * (1.0 / 3.0);
  double D00 = G00 - t, D11 = G11 - t, D22 = G22 - t;
  s.devGsq = D00 * D00 + D11 * D11 + D22 * D22 + 2.0 * (G01 * G01 + G02 * G02 + G12 * G12);
  s.G[0] = G00;
  s.G[1] = G11;
  s.G[2] = G22;
  s.G[3] = G01;
  s.G[4] = G02;
  s.G[5] = G12;
  s.S[0] = D00 * G00 + G01 * G01 + G02 * G02;
  s.S[1] = G01 * G01 + D11 * G11 + G12 * G12;
  s.S[2] = G02 * G02 + G12 * G12 + D22 * G22;
  s.S[3] = D00 * G01 + G01 * G11 + G02 * G12;
  s.S[4] = D00 * G02 + G01 * G12 + G02 * G22;
  s.S[5] = G01 * G02 + D11 * G12 + G12 * G22;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    double a0 = A[3 * i], a1 = A[3 * i + 1], a2 = A[3 * i + 2];
    s.AdG[3 * i + 0] = a0 * D00 + a1 * G01 + a2 * G02;
    s.AdG[3 * i + 1] = a0 * G01 + a1 * D11 + a2 * G12;
    s.AdG[3 * i + 2] = a0 * G02 + a1 * G12 + a2 * D22;
  }
  s.e = eos_rho(s.r, s.ir, P);
  s.cs2 = P.b02;
  // C_0 / 4 with C_0 = (1 - beta/Gamma) cs2 (shear.cpp:23-29); rho Gamma =
  // Gamma0 rho0 for shock MG
  double C0q = P.b02q;
  if (P.has_beta) {
    s.cs2 = P.b02 * pow(s.r * P.ir0, P.beta);
    C0q = 0.25 * ((P.EOS == 1 ? (1.0 - P.beta / s.e.G) : P.C0f) * s.cs2);
  }
  s.irG = P.EOS == 1 ? P.iG : s.ir * P.iG;
  double E1 = q[1] * s.ir - 0.5 * (s.v[0] * s.v[0] + s.v[1] * s.v[1] + s.v[2] * s.v[2]) -
              C0q * s.devGsq;
  if (TH) {
    s.J[0] = q[14] * s.ir;
    s.J[1] = q[15] * s.ir;
    s.J[2] = q[16] * s.ir;
    E1 -= P.hca2 * (s.J[0] * s.J[0] + s.J[1] * s.J[1] + s.J[2] * s.J[2]);
  }
  // pressure_mg (mg.cpp:126-131), temperature_mg (mg.cpp:133-139)
  double rG = s.r * s.e.G;
  s.p = (E1 - s.e.er) * rG + s.e.pr;
  s.T = (s.p - s.e.pr) * s.irG * P.icv;
  if (P.has_tref)
    s.T = s.e.phi * P.Tref + s.T;
}

// sigma column d: -rho cs2 (A devG)^T A(:,d) = -rho cs2 (devG A^T A)(:,d)
// (state.cpp:23-29)
template <bool TH>
GPR_D void sigma_col(const double *, const Prim<TH> &s, int d, double *sg) {
  double f = -s.r * s.cs2;
#pragma unroll
  for (int i = 0; i < 3; i++)
    sg[i] = f * sym3(s.S, i, d);
}

// ret += F_d(Q)   (equations.cpp:11-48)
template <bool TH, int V>
GPR_D void flux_add(const double *q, const Prim<TH> &s, int d, const DevPar &P, double *F) {
  double vd = s.v[d];
  double sg[3];
  sigma_col(q, s, d, sg);
  F[0] += q[2 + d];
  F[1] += vd * (q[1] + s.p) - (sg[0] * s.v[0] + sg[1] * s.v[1] + sg[2] * s.v[2]);
#pragma unroll
  for (int i = 0; i < 3; i++)
    F[2 + i] += vd * q[2 + i] - sg[i];
  F[2 + d] += s.p;
  const double *A = q + 5;
#pragma unroll
  for (int i = 0; i < 3; i++)
    F[5 + 3 * i + d] += A[3 * i] * s.v[0] + A[3 * i + 1] * s.v[1] + A[3 * i + 2] * s.v[2];
  if (TH) {
    F[1] += P.calpha2 * s.T * s.J[d];
#pragma unroll
    for (int i = 0; i < 3; i++)
      F[14 + i] += vd * q[14 + i];
    F[14 + d] += s.T;
  }
}

// Entries of F_d(Q) that can be nonzero (flux_add / flux_set write only
// these; the rest are exact zeros).
template <bool TH> __host__ __device__ constexpr bool flux_support(int k, int d) {
  return k < 5 || (k >= 5 && k < 14 && (k - 5) % 3 == d) || (TH && k >= 14 && k < 17);
}

// F = F_d(Q): flux_add into a zeroed array without the additions to zero
// (which the compiler must keep: 0.0 + x is not x for x = -0.0).
template <bool TH, int V>
GPR_D void flux_set(const double *q, const Prim<TH> &s, int d, const DevPar &P, double *F) {
#pragma unroll
  for (int k = 0; k < V; k++)
    F[k] = 0.0;
  double vd = s.v[d];
  double sg[3];
  sigma_col(q, s, d, sg);
  F[0] = q[2 + d];
  F[1] = vd * (q[1] + s.p) - (sg[0] * s.v[0] + sg[1] * s.v[1] + sg[2] * s.v[2]);
#pragma unroll
  for (int i = 0; i < 3; i++)
    F[2 + i] = vd * q[2 + i] - sg[i];
  F[2 + d] += s.p;
  const double *A = q + 5;
#pragma unroll
  for (int i = 0; i < 3; i++)
    F[5 + 3 * i + d] = A[3 * i] * s.v[0] + A[3 * i + 1] * s.v[1] + A[3 * i + 2] * s.v[2];
  if (TH) {
    F[1] += P.calpha2 * s.T * s.J[d];
#pragma unroll
    for (int i = 0; i < 3; i++)
      F[14 + i] = vd * q[14 + i];
    F[14 + d] += s.T;
  }
}

GPR_D double det3(const double *A) {
  return A[0] * (A[4] * A[8] - A[5] * A[7]) - A[1] * (A[3] * A[8] - A[5] * A[6]) +
         A[2] * (A[3] * A[7] - A[4] * A[6]);
}

// Sigma Frobenius-type norms used by the non-Newtonian relaxation rates.
template <bool TH>
GPR_D void sigma_full(const double *q, const Prim<TH> &s, double *sf) {
#pragma unroll
  for (int d = 0; d < 3; d++) {
    double c[3];
    sigma_col(q, s, d, c);
    sf[d] = c[0];
    sf[3 + d] = c[1];
    sf[6 + d] = c[2];
  }
}

// theta1inv (sources.cpp:13-81)
template <bool TH>
GPR_D double theta1inv(const double *q, const Prim<TH> &s, const DevPar &P) {
  const double A53 = pow53(det3(q + 5));  // det(A)^(5/3)
  int SOLID = P.flags & GPR_SOLID, PL = P.flags & GPR_POWER_LAW, BING = P.flags & GPR_BINGHAM;
  if (!SOLID && !BING && !PL)
    return A53 * P.th1c;
  double sf[9];
  sigma_full(q, s, sf);
  if (SOLID) {
    if (!PL)
      return 0.0;
    double a = sf[0] - sf[4], b = sf[4] - sf[8], c = sf[8] - sf[0];
    double sn = sqrt(0.5 * (a * a + b * b + c * c) + 3.0 * (sf[1] * sf[1] + sf[5] * sf[5] + sf[6] * sf[6]));
    sn = fmin(sn, 1e8);
    return 3.0 * A53 / (s.cs2 * P.tau0) * pow(sn / P.sigmaY, P.n);
  }
  double nn = 0.0;
#pragma unroll
  for (int i = 0; i < 9; i++)
    nn += sf[i] * sf[i];
  double sn = sqrt(nn) * 0.70710678118654752440;
  if (BING)
    return sn > P.sigmaY ? A53 * P.rho0 / (2.0 * P.mu) * (1.0 - P.sigmaY / sn) : 0.0;
  return A53 * P.th1c * pow(sn, (1.0 - P.n) / P.n);
}

// S(Q)   (equations.cpp:50-67)
template <bool TH, int V>
GPR_D void source(const double *q, const Prim<TH> &s, const DevPar &P, double *S,
                  double scale = 1.0) {
  // scale multiplies the result (through its scalar factors)
#pragma unroll
  for (int k = 0; k < V; k++)
    S[k] = 0.0;
  if (P.has_dp) {
    S[2] = P.dp0 * scale;
    S[3] = P.dp1 * scale;
    S[4] = P.dp2 * scale;
  }
  double f = -s.cs2 * theta1inv(q, s, P) * scale;
#pragma unroll
  for (int i = 0; i < 9; i++)
    S[5 + i] = s.AdG[i] * f;
  if (TH) {
    // -rho (calpha2 J) T / (kappa rho)
    double g = -P.ca2ik * s.T * scale;
#pragma unroll
    for (int i = 0; i < 3; i++)
      S[14 + i] = g * s.J[i];
  }
}

// B_d(Q) x   (equations.cpp:89-167); v = rho v / rho.
template <int V, int LSET>
GPR_D void bdot(const double *v, const double *x, int d, double *out) {
#pragma unroll
  for (int k = 0; k < 5; k++)
    out[k] = 0.0;
#pragma unroll
  for (int k = 14; k < V; k++)
    out[k] = 0.0;
  double v0 = v[0], v1 = v[1], v2 = v[2];
  if (d == 0) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      out[5 + 3 * r] = -v1 * x[6 + 3 * r] - v2 * x[7 + 3 * r];
      out[6 + 3 * r] = v0 * x[6 + 3 * r];
      out[7 + 3 * r] = v0 * x[7 + 3 * r];
    }
  } else if (d == 1) {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      out[5 + 3 * r] = v1 * x[5 + 3 * r];
      out[6 + 3 * r] = -v0 * x[5 + 3 * r] - v2 * x[7 + 3 * r];
      out[7 + 3 * r] = v1 * x[7 + 3 * r];
    }
  } else {
#pragma unroll
    for (int r = 0; r < 3; r++) {
      out[5 + 3 * r] = v2 * x[5 + 3 * r];
      out[6 + 3 * r] = v2 * x[6 + 3 * r];
      out[7 + 3 * r] = -v0 * x[5 + 3 * r] - v1 * x[6 + 3 * r];
    }
  }
  if (LSET > 0) {
    double vd = d == 0 ? v0 : (d == 1 ? v1 : v2);
#pragma unroll
    for (int i = 1; i <= LSET; i++)
      out[V - i] = vd * x[V - i];
  }
}

// ---------------------------------------------------------------------------
// Eigenvalues of a small real nonsymmetric matrix: Householder reduction to
// Hessenberg form, then Francis double-shift QR with deflation (Golub & Van
// Loan, Matrix Computations, Alg. 7.4.2, 7.5.1-7.5.2).  Returns the largest
// eigenvalue modulus (the reference calls Eigen's EigenSolver and takes
// max |lambda|, system/eig.cpp:73).  Returns NaN if it does not converge.
template <int n> GPR_D double max_abs_eig(double (&H)[n][n]) {
  const double eps = 2.220446049250313e-16;
  // Hessenberg reduction
#pragma unroll
  for (int k = 0; k < n - 2; k++) {
    double v[n];
    double alpha = 0.0, tail = 0.0;
#pragma unroll
    for (int i = 0; i < n; i++) {
      if (i > k)
        alpha += H[i][k] * H[i][k];
      if (i > k + 1)
        tail += H[i][k] * H[i][k];
    }
    alpha = sqrt(alpha);
    // no reflection when the column below the subdiagonal is zero to the
    // least normal number (Eigen's makeHouseholder rule): a reflector of
    // subnormal entries would divide by an underflowed norm
    if (alpha != 0.0 && tail > DBL_MIN_NORMAL) {
      double x0 = H[k + 1][k];
      double beta = x0 > 0 ? -alpha : alpha;
#pragma unroll
      for (int i = 0; i < n; i++)
        v[i] = i > k + 1 ? H[i][k] : 0.0;
      v[k + 1] = x0 - beta;
      double vv = 0.0;
#pragma unroll
      for (int i = 0; i < n; i++)
        vv += v[i] * v[i];
      if (vv != 0.0) {
        double tau = 2.0 / vv;
#pragma unroll
        for (int j = 0; j < n; j++) {
          double sacc = 0.0;
#pragma unroll
          for (int i = 0; i < n; i++)
            sacc += v[i] * H[i][j];
          sacc *= tau;
#pragma unroll
          for (int i = 0; i < n; i++)
            H[i][j] -= sacc * v[i];
        }
#pragma unroll
        for (int i = 0; i < n; i++) {
          double sacc = 0.0;
#pragma unroll
          for (int j = 0; j < n; j++)
            sacc += H[i][j] * v[j];
          sacc *= tau;
#pragma unroll
          for (int j = 0; j < n; j++)
            H[i][j] -= sacc * v[j];
        }
      }
    }
  }
  double norm = 0.0;
#pragma unroll
  for (int i = 0; i < n; i++)
#pragma unroll
    for (int j = 0; j < n; j++)
      if (j >= i - 1)
        norm += fabs(H[i][j]);
  double best = 0.0;
  int hi = n - 1, iter = 0, total = 0;
  double exshift = 0.0;
  while (hi >= 0) {
    int l = hi;
    while (l > 0) {
      double s = fabs(H[l - 1][l - 1]) + fabs(H[l][l]);
      if (s == 0.0)
        s = norm;
      if (fabs(H[l][l - 1]) < eps * s)
        break;
      l--;
    }
    if (l == hi) {
      best = fmax(best, fabs(H[hi][hi] + exshift));
      hi--;
      iter = 0;
      continue;
    }
    double x = H[hi][hi], y = H[hi - 1][hi - 1], w = H[hi][hi - 1] * H[hi - 1][hi];
    if (l == hi - 1) {
      double p = 0.5 * (y - x), q = p * p + w, z = sqrt(fabs(q));
      x += exshift;
      if (q >= 0.0) {
        z = p >= 0 ? p + z : p - z;
        best = fmax(best, fabs(x + z));
        best = fmax(best, fabs(z != 0.0 ? x - w / z : x + z));
      } else {
        best = fmax(best, hypot(x + p, z));
      }
      hi -= 2;
      iter = 0;
      continue;
    }
    if (iter == 10 || iter == 20) {
      exshift += x;
      for (int i = 0; i <= hi; i++)
        H[i][i] -= x;
      double s = fabs(H[hi][hi - 1]) + fabs(H[hi - 1][hi - 2]);
      x = y = 0.75 * s;
      w = -0.4375 * s * s;
    }
    iter++;
    if (++total > 30 * n)
      return nan("");
    int m = hi - 2;
    double p = 0, q = 0, r = 0, z;
    while (m >= l) {
      z = H[m][m];
      r = x - z;
      double s = y - z;
      p = (r * s - w) / H[m + 1][m] + H[m][m + 1];
      q = H[m + 1][m + 1] - z - r - s;
      r = H[m + 2][m + 1];
      s = fabs(p) + fabs(q) + fabs(r);
      p /= s;
      q /= s;
      r /= s;
      if (m == l)
        break;
      double u = fabs(H[m][m - 1]) * (fabs(q) + fabs(r));
      double vv = fabs(p) * (fabs(H[m - 1][m - 1]) + fabs(z) + fabs(H[m + 1][m + 1]));
      if (u < eps * vv)
        break;
      m--;
    }
    for (int i = m + 2; i <= hi; i++) {
      H[i][i - 2] = 0.0;
      if (i > m + 2)
        H[i][i - 3] = 0.0;
    }
    for (int k = m; k <= hi - 1; k++) {
      bool notlast = (k != hi - 1);
      if (k != m) {
        p = H[k][k - 1];
        q = H[k + 1][k - 1];
        r = notlast ? H[k + 2][k - 1] : 0.0;
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
        H[k][k - 1] = -s * x;
      else if (l != m)
        H[k][k - 1] = -H[k][k - 1];
      p += s;
      x = p / s;
      y = q / s;
      z = r / s;
      q /= p;
      r /= p;
      for (int j = k; j <= hi; j++) {
        double pp = H[k][j] + q * H[k + 1][j];
        if (notlast) {
          pp += r * H[k + 2][j];
          H[k + 2][j] -= pp * z;
        }
        H[k][j] -= pp * x;
        H[k + 1][j] -= pp * y;
      }
      int ihi = hi < k + 3 ? hi : k + 3;
      for (int i = l; i <= ihi; i++) {
        double pp = x * H[i][k] + y * H[i][k + 1];
        if (notlast) {
          pp += z * H[i][k + 2];
          H[i][k + 2] -= pp * r;
        }
        H[i][k] -= pp;
        H[i][k + 1] -= pp * q;
      }
    }
  }
  return best;
}

// Largest eigenvalue of a small real matrix whose spectrum is dominated by a
// simple, real, positive eigenvalue (the squared fastest wave speed of the
// thermo-acoustic tensor): characteristic polynomial by principal minors,
// Laguerre's iteration (cubically convergent, monotone from an upper bound
// for real-rooted polynomials) started at the infinity-norm bound, then a
// certificate: the polynomial deflated by (x - lambda) must have every root
// strictly inside |z| < (1 - 1e-9) lambda (Jury's criterion on the scaled
// quotient).  Returns false when the certificate fails (complex roots of
// larger modulus, a multiple largest root, no convergence); the caller then
// runs the QR iteration, so the result is max |eig| either way.
template <int m>
GPR_D bool max_eig_laguerre(const double (&X)[m][m], double &lam) {
  static_assert(m == 3 || m == 4, "3x3 or 4x4");
  double c1 = 0.0, c2 = 0.0, c3 = 0.0, c4 = 0.0;
#pragma unroll
  for (int i = 0; i < m; i++)
    c1 += X[i][i];
  if (m == 3) {
#pragma unroll
    for (int i = 0; i < m; i++)
#pragma unroll
      for (int j = i + 1; j < m; j++)
        c2 += X[i][i] * X[j][j] - X[i][j] * X[j][i];
    c3 = X[0][0] * (X[1][1] * X[2][2] - X[1][2] * X[2][1]) -
         X[0][1] * (X[1][0] * X[2][2] - X[1][2] * X[2][0]) +
         X[0][2] * (X[1][0] * X[2][1] - X[1][1] * X[2][0]);
  } else {
    // the 2x2 minors of rows (0, 1) and of rows (2, 3) give c2 (the two
    // principal ones), the four principal 3x3 minors (expanded along the
    // third row) and det X (Laplace along rows (0, 1))
    // (explicit fused multiply-adds: the same rounding in every kernel that
    // inlines this, whatever contraction the compiler would choose there)
    const int r2 = m == 4 ? 2 : 0, r3 = m == 4 ? 3 : 0;
    auto mn = [](double a, double b, double c, double d) { return fma(a, b, -(c * d)); };
    auto s = [&](int a, int b) { return mn(X[0][a], X[1][b], X[0][b], X[1][a]); };
    auto t = [&](int a, int b) { return mn(X[r2][a], X[r3][b], X[r2][b], X[r3][a]); };
    const double s01 = s(0, 1), s02 = s(0, 2), s12 = s(1, 2);
    const double s03 = s(0, 3), s13 = s(1, 3), s23 = s(2, 3);
    const double t01 = t(0, 1), t02 = t(0, 2), t12 = t(1, 2);
    const double t03 = t(0, 3), t13 = t(1, 3), t23 = t(2, 3);
    c2 = ((s01 + t23) + (mn(X[0][0], X[r2][r2], X[0][r2], X[r2][0]) +
                         mn(X[0][0], X[r3][r3], X[0][r3], X[r3][0]))) +
         (mn(X[1][1], X[r2][r2], X[1][r2], X[r2][1]) +
          mn(X[1][1], X[r3][r3], X[1][r3], X[r3][1]));
    auto e3 = [](double a, double sa, double b, double sb, double c, double sc) {
      return fma(c, sc, fma(a, sa, -(b * sb)));
    };
    c3 = (e3(X[r2][r2], s01, X[r2][1], s02, X[r2][0], s12) +
          e3(X[r3][r3], s01, X[r3][1], s03, X[r3][0], s13)) +
         (e3(X[0][0], t23, X[0][r2], t03, X[0][r3], t02) +
          e3(X[1][1], t23, X[1][r2], t13, X[1][r3], t12));
    c4 = (mn(s01, t23, s02, t13) + fma(s03, t12, s12 * t03)) - fma(s13, t02, -(s23 * t01));
  }
  // p(x) = x^m - c1 x^(m-1) + c2 x^(m-2) - c3 x^(m-3) [+ c4]
  double R = 0.0;
#pragma unroll
  for (int i = 0; i < m; i++) {
    double rs = 0.0;
#pragma unroll
    for (int j = 0; j < m; j++)
      rs += fabs(X[i][j]);
    R = fmax(R, rs);
  }
  const double Rs = R * (1.0 + 1e-12) + 1e-300;
  // Starting point in FP32: Laguerre on the scaled polynomial p(Rs y) / Rs^m
  // (O(1) coefficients, every root |y| <= 1) from y = 1 down to ~1e-4.  On
  // this GPU FP32 runs at full rate beside the FP64 pipe, so the FP64
  // iteration below, started just above that estimate, needs one or two
  // steps instead of ~5 from the bound.  A failed FP32 run (non-finite or out
  // of (0, 1]) leaves the start at the bound.
  double x = Rs;
  {
    // scaled coefficients in FP32 (a coefficient beyond the FP32 range makes
    // the start fail, and the FP64 iteration then starts at the bound)
    const float iR = 1.0f / (float)Rs;
    float cs[4];
    cs[0] = -(float)c1 * iR;
    cs[1] = ((float)c2 * iR) * iR;
    cs[2] = -(((float)c3 * iR) * iR) * iR;
    cs[3] = ((((float)c4 * iR) * iR) * iR) * iR;
    float y = 1.0f;
    for (int it = 0; it < 24; it++) {
      float p = 1.0f, dp = 0.0f, d2p = 0.0f;
#pragma unroll
      for (int k = 0; k < m; k++) {
        d2p = fmaf(d2p, y, 2.0f * dp);
        dp = fmaf(dp, y, p);
        p = fmaf(p, y, cs[k]);
      }
      if (p == 0.0f)
        break;
      float ip = 1.0f / p;
      float G = dp * ip;
      float H = fmaf(G, G, -(d2p * ip));
      float disc = fmaxf((m - 1) * fmaf((float)m, H, -(G * G)), 0.0f);
      float a = m / (G + copysignf(sqrtf(disc), G));
      y -= a;
      if (!(fabsf(a) > 1e-4f * fabsf(y)))
        break;
    }
    if (y > 0.0f && y <= 1.0f)
      x = fmin((double)y * (1.0 + 4e-6), 1.0) * Rs;
  }
  // without a real root above the other roots' real parts the steps wander
  bool found = false;
  for (int it = 0; it < 16; it++) {
    double p = 1.0, dp = 0.0, d2p = 0.0;
    const double cf[4] = {-c1, c2, -c3, c4};
#pragma unroll
    for (int k = 0; k < m; k++) {
      d2p = fma(d2p, x, 2.0 * dp);
      dp = fma(dp, x, p);
      p = fma(p, x, cf[k]);
    }
    found = p == 0.0;
    if (found)
      break;
    double ip = 1.0 / p;
    double G = dp * ip;
    double H = fma(G, G, -(d2p * ip));
    double disc = fmax((m - 1) * fma((double)m, H, -(G * G)), 0.0);
    double a = m / (G + copysign(sqrt(disc), G));
    x -= a;
    found = fabs(a) <= 1e-5 * fabs(x);  // cubic convergence: the error is now ~|a|^3
    if (found)
      break;
  }
  lam = x;
  if (!found || !(x > 0.0) || !(x <= R * (1.0 + 1e-9)))
    return false;
  // deflate and certify: all other roots strictly inside |z| < (1-1e-9) lam
  double l = x * (1.0 - 1e-9);
  double q2 = -c1 + x, q1 = fma(x, q2, c2);
  if (m == 3) {
    const double il = 1.0 / l;
    double a1 = q2 * il, a0 = q1 * il * il;
    return fabs(a0) < 1.0 && fabs(a1) < 1.0 + a0;
  }
  double q0 = fma(x, q1, -c3);
  const double il = 1.0 / l;
  double a2 = q2 * il, a1 = q1 * il * il, a0 = q0 * il * il * il;
  return (1.0 + a2 + a1 + a0 > 0.0) && (1.0 - a2 + a1 - a0 > 0.0) && fabs(a0) < 1.0 &&
         fabs(a0 * a0 - 1.0) > fabs(a0 * a2 - a1);
}

// The largest eigenvalue of the acoustic tensor by the general routines
// (Laguerre in FP64 with its certificate, then QR): for the states that
// top_root leaves (no real dominant root, or one within 1e-4 of another).
// Out of line: the callers' registers are not sized for it.
template <int m> __device__ __noinline__ double max_eig_general(const double *Xr) {
  double X[m][m], l2;
#pragma unroll
  for (int i = 0; i < m; i++)
#pragma unroll
    for (int c = 0; c < m; c++)
      X[i][c] = Xr[i * m + c];
  if (!max_eig_laguerre<m>(X, l2))
    l2 = max_abs_eig<m>(X);
  return l2;
}

// The largest root of x^m - c[0] x^(m-1) + c[1] x^(m-2) - ... when it is real,
// positive and simple (the squared fastest wave speed), with few FP64
// instructions: everything that only has to be near runs in FP32 on the
// polynomial scaled by a power of two (bit fields, no FP64 instruction), and
// FP64 evaluates the residual p(x) alone.
//  1. FP32: Laguerre's iteration from sqrt(c0^2 - 2 c1) (the 2-norm of a real
//     spectrum, at least its largest root) down to ~1e-6, and p' there.
//  2. FP32: certificate that p / (x - y) has its roots inside |z| < (1 - 1e-4)
//     y (Jury's criterion, margins ten times the FP32 rounding).
//  3. FP64: x <- x - p(x) / p'(y) with the FP32 derivative.  A step leaves the
//     error times ~1e-6 (the FP32 error of p' and its change over a 1e-6
//     interval); the ratio of two steps measures that factor, and the
//     iteration stops when the factor times the last step is below 2^-56 x (or
//     the step is at the rounding of p).
// Returns false when any of it fails; the caller takes the general routine.
// Against the previous FP64 Laguerre step with its FP64 certificate (two
// divisions and a root in each, and six FP64 <-> FP32 conversions, which run on
// the FP64 pipe) this issues about 13 FP64 instructions instead of about 110.
template <int m> GPR_D bool top_root(const double (&c)[m], double &lam) {
  const int hi = __double2hiint(c[0]);
  const int sh = ((hi >> 20) & 0x7ff) - 1022;
  if (hi < 0 || sh < -240 || sh > 240)
    return false;
  float a[m];  // coefficients of the scaled monic polynomial
#pragma unroll
  for (int k = 0; k < m; k++)
    a[k] = ((k & 1) ? 1.0f : -1.0f) * f32_scaled(c[k], (k + 1) * sh);
  const float b2 = fmaf(a[0], a[0], -2.0f * a[1]);
  float y = sqrt32(b2) * 1.00001f, dp = 0.0f;
  bool near = false;
#pragma unroll 1
  for (int it = 0; it < 12; it++) {
    float p = 1.0f, d2p = 0.0f;
    dp = 0.0f;
#pragma unroll
    for (int k = 0; k < m; k++) {
      d2p = fmaf(d2p, y, 2.0f * dp);
      dp = fmaf(dp, y, p);
      p = fmaf(p, y, a[k]);
    }
    if (near)  // p' at the accepted y
      break;
    // Laguerre's step m p / (p' + sqrt((m-1)^2 p'^2 - m (m-1) p p''))
    const float disc = fmaf((float)((m - 1) * (m - 1)) * dp, dp, -(float)(m * (m - 1)) * (p * d2p));
    const float st = (float)m * p * rcp32(dp + copysignf(sqrt32(fmaxf(disc, 0.0f)), dp));
    y -= st;
    near = fabsf(st) <= 1e-3f * y;
    if (!(y > 0.0f))
      return false;
  }
  if (!near)
    return false;
  // certificate on the quotient, scaled by l = (1 - 1e-4) y
  {
    const float il = 1.0001f * rcp32(y);
    const float q2 = a[0] + y, q1 = fmaf(y, q2, a[1]);
    bool in;
    if (m == 3) {
      const float a1 = q2 * il, a0 = q1 * il * il;
      in = fabsf(a0) < 1.0f - 1e-5f && fabsf(a1) < 1.0f + a0 - 1e-5f;
    } else {
      const float q0 = fmaf(y, q1, a[2]);
      const float a2 = q2 * il, a1 = q1 * il * il, a0 = q0 * il * il * il;
      in = 1.0f + a2 + a1 + a0 > 1e-5f && 1.0f - a2 + a1 - a0 > 1e-5f &&
           fabsf(a0) < 1.0f - 1e-5f && fabsf(a0 * a0 - 1.0f) > fabsf(a0 * a2 - a1) + 1e-5f;
    }
    if (!in)
      return false;
  }
  // p'(y) scales by 2^((m-1) sh)
  const double ip = f64_scaled(rcp32(dp), -(m - 1) * sh);
  double x = f64_scaled(y, sh);
  float prev = 0.0f;
#pragma unroll 1
  for (int it = 0; it < 8; it++) {
    double p = x - c[0];
#pragma unroll
    for (int k = 1; k < m; k++)
      p = fma(p, x, (k & 1) ? c[k] : -c[k]);
    const double st = p * ip;
    x -= st;
    const float s = fabsf(f32_scaled(st, sh));
    if (s * s <= 1.4e-17f * y * prev || s <= 2e-15f * y) {
      lam = x;
      return true;
    }
    prev = s;
  }
  return false;
}

// max |eigenvalue| of the GPR system in direction d (system/eig.cpp:8-77):
// |v_d| + sqrt(max |eig(Xi1 Xi2)|).  Xi1 (4x5) and Xi2 (5x4) are assembled
// implicitly: Xi = Xi1 Xi2 is formed directly from its nonzero blocks.  With
// G = A^T A and S = devG G (both symmetric), the distortion part of Xi's
// velocity block is (dsigma/dA A: state.cpp:43-56, A(:,d)^T A = G(d,:))
//   cs2 (S + e_d S(d,:) + G(:,d) G(d,:) / 3 + G(d,d) G),
// six entries and a row instead of two 3x3 products.
// Xo (m x m, row-major) and l2o, when given, receive Xi and its dominant
// eigenvalue (for the adjoint's wave-speed derivative).
template <bool TH>
GPR_D double max_abs_eigs(const double *q, const Prim<TH> &s, int d, const DevPar &P,
                          double *Xo = nullptr, double *l2o = nullptr) {
  const double r = s.r, ir = s.ir;
  const double cs2 = s.cs2;
  double Gd[3], Sd[3], X[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    Gd[i] = sym3(s.G, i, d);
    Sd[i] = sym3(s.S, i, d);
  }
  const double Gdd = d == 0 ? Gd[0] : (d == 1 ? Gd[1] : Gd[2]);
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const double g3 = (1.0 / 3.0) * Gd[i];
#pragma unroll
    for (int c = i; c < 3; c++)
      X[i][c] = fma(Gdd, sym3(s.G, i, c), fma(g3, Gd[c], sym3(s.S, i, c)));
  }
  // + e_d S(d,:), and with the reference's columns and rows 0: Xi1 column 0
  // (-dsigma/drho / rho, dsigma/drho = (1 + beta) sigma / rho) and Xi2 row 1
  // (b / rho with b = sigma - rho dsigma/drho + rho c0^2 e_d)
  const double b1 = P.b1;
  if (d == 0) {
    X[0][0] = fma(2.0 * b1, Sd[0], X[0][0]);
    X[0][1] = fma(b1, Sd[1], X[0][1]);
    X[0][2] = fma(b1, Sd[2], X[0][2]);
    X[1][0] = X[0][1];
    X[2][0] = X[0][2];
    X[2][1] = X[1][2];
  } else {
    X[1][0] = X[0][1];
    X[2][0] = X[0][2];
    X[2][1] = X[1][2];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      if (d == 1)
        X[1][c] += Sd[c];
      else
        X[2][c] += Sd[c];
    }
#pragma unroll
    for (int i = 0; i < 3; i++)
      X[i][0] = fma(b1, Sd[i], X[i][0]);
    if (P.has_beta) {
#pragma unroll
      for (int c = 0; c < 3; c++)
        X[0][c] = fma(P.beta, Sd[c], X[0][c]);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int c = 0; c < 3; c++)
      X[i][c] *= cs2;
  // c0^2 = (p/rho^2 - dE/drho) / dE/dp   (waves/speeds.cpp:8-18)
  const EosRho &e = s.e;
  const double rG = r * e.G, irG2 = s.irG * s.irG;
  double dnum = e.G * (s.p - e.pr);
  if (P.EOS != 0)
    dnum = e.dpr * rG + (e.G + r * e.dG) * (s.p - e.pr);
  double dEdr = e.der - dnum * irG2;
  if (P.has_beta) {
    const double dcs2 = P.beta * ir * cs2;
    const double dC0 = (1.0 - P.beta / e.G) * dcs2 + P.beta / (e.G * e.G) * e.dG * cs2;
    dEdr += 0.25 * dC0 * s.devGsq;
  }
  const double c02 = (s.p * ir * ir - dEdr) * rG;  // dE/dp = 1/(rho Gamma)
  if (d == 0)
    X[0][0] += c02;
  else if (d == 1)
    X[0][1] += c02;
  else
    X[0][2] += c02;
  // The heat-conduction row and column (TH): Xi couples the impulse to
  // velocity row 0 only (x03), and back through T's row (x3).
  double x03 = 0.0, x3[3] = {0.0, 0.0, 0.0}, x33 = 0.0;
  if (TH) {
    const double h = P.calpha2 * s.T * e.G;  // Xi2 row 1
    const double rtp = s.irG * P.icv;        // dT/dp
    x03 = h * ir;
    x33 = rtp * ir * h;
    const double dTr = -dnum * irG2 * P.icv;
    x3[0] = d == 0 ? fma(rtp, c02, dTr) : dTr;
    x3[1] = d == 1 ? rtp * c02 : 0.0;
    x3[2] = d == 2 ? rtp * c02 : 0.0;
    if (P.has_beta) {
      const double f = rtp * P.beta * cs2;
#pragma unroll
      for (int c = 0; c < 3; c++)
        x3[c] = fma(f, Sd[c], x3[c]);
    }
  }
  // The characteristic polynomial: that of the velocity block Y by its minors,
  // bordered: det(x - Xi) = (x - x33) chi_Y(x) - x03 x3 . adj(x - Y) e_0.
  // (explicit fused multiply-adds: the same rounding in every kernel)
  const double m12 = fma(X[1][1], X[2][2], -(X[1][2] * X[2][1]));
  const double n1 = fma(X[1][2], X[2][0], -(X[1][0] * X[2][2]));
  const double n2 = fma(X[1][0], X[2][1], -(X[2][0] * X[1][1]));
  const double m01 = fma(X[0][0], X[1][1], -(X[0][1] * X[1][0]));
  const double m02 = fma(X[0][0], X[2][2], -(X[0][2] * X[2][0]));
  const double s12 = X[1][1] + X[2][2];
  const double t1 = X[0][0] + s12, t2 = m12 + (m01 + m02);
  const double t3 = fma(X[0][2], n2, fma(X[0][1], n1, X[0][0] * m12));
  double l2;
  bool ok;
  if (TH) {
    double u2 = x3[0] * s12, u3 = x3[0] * m12;
    if (d != 0 || P.has_beta) {
      u2 = fma(-x3[2], X[2][0], fma(-x3[1], X[1][0], u2));
      u3 = fma(x3[2], n2, fma(x3[1], n1, u3));
    }
    const double c[4] = {t1 + x33, fma(-x03, x3[0], fma(x33, t1, t2)),
                         fma(-x03, u2, fma(x33, t2, t3)), fma(-x03, u3, x33 * t3)};
    ok = top_root<4>(c, l2);
  } else {
    const double c[3] = {t1, t2, t3};
    ok = top_root<3>(c, l2);
  }
  if (Xo || !ok) {
    constexpr int m = TH ? 4 : 3;
    double Xm[m * m];
#pragma unroll
    for (int i = 0; i < 3; i++) {
#pragma unroll
      for (int c = 0; c < 3; c++)
        Xm[i * m + c] = X[i][c];
      if (TH) {
        Xm[i * m + m - 1] = i == 0 ? x03 : 0.0;
        Xm[(m - 1) * m + i] = x3[i];
      }
    }
    if (TH)
      Xm[m * m - 1] = x33;
    if (!ok)
      l2 = max_eig_general<m>(Xm);
    if (Xo) {
#pragma unroll
      for (int k = 0; k < m * m; k++)
        Xo[k] = Xm[k];
    }
  }
  if (l2o)
    *l2o = l2;
  return sqrt64(l2) + fabs(s.v[d]);
}

}  // namespace gpr
