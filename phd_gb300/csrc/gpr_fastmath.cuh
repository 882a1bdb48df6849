// gpr_fastmath.cuh - FP64 reciprocal, square root and det^(5/3) with few
// FP64-pipe instructions, and conversions that use none.
//
// On GB300 every FP64 instruction (arithmetic, comparison, maximum, and the
// conversions to and from FP32) holds an SM's FP64 pipe for 16 - 19 cycles
// per warp, while integer, FP32 and special-function instructions take 0.25 -
// 2 beside it (measured: clock64 around 1024 instructions per thread of one
// block).  So an FP64 result is reached from a special-function start by one
// step of high order, and what needs no FP64 is done in integers.  In the same
// measurement 1/x takes 86 cycles per warp and SM, sqrt 143, cbrt 235; the
// forms below issue 3 (about 50 cycles), 5 (85) and 8 (140) FP64
// instructions.
//
// Each form tests its start's exponent and leaves zeros, infinities, NaNs,
// subnormals and the ends of the range to CUDA's own operation, so that the
// results there are the operators'.  That branch is a volatile instruction or
// an out-of-line call: as a plain expression it is evaluated on every call and
// selected afterwards (measured: 137 cycles per warp and SM for rcp64 against 51,
// sqrt64 229 against 86, pow53 277 against 140).
#pragma once

namespace gpr {

GPR_D int fp_exponent(double x) {  // biased exponent field
  return (__double2hiint(x) >> 20) & 0x7ff;
}

// 1 / b.  Start: the special-function reciprocal, within 2^-19.9 (measured
// over 2^25 mantissas); one third-order step of the geometric series,
// y (1 + e + e^2) with e = 1 - b y: truncation below 2^-59, and the final
// fused multiply-add rounds once.
GPR_D double rcp64(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  const double e = fma(-b, y, 1.0);
  double r = fma(y, fma(e, e, e), y);
  if ((unsigned)(fp_exponent(y) - 1) >= 0x7feu)
    asm volatile("rcp.rn.f64 %0, %1;" : "=d"(r) : "d"(b));
  return r;
}

// sqrt(x).  Start: the special-function reciprocal root y, within 2^-20
// (measured); one step of Goldschmidt's iteration g <- g + g (1/2 - g h) from
// g = x y, h = y / 2 (relative error below 2^-38), then the remainder form
// g + h (x - g^2) (Markstein), whose exact remainder leaves one rounding.
GPR_D double sqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  // y / 2 by the exponent field
  const double h = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
  double g = x * y;
  g = fma(g, fma(-g, h, 0.5), g);
  g = fma(fma(-g, g, x), h, g);
  // below 2^-900 the remainder would be subnormal
  if ((unsigned)((__double2hiint(x) >> 20) - 123) >= 0x7ffu - 123u)
    asm volatile("sqrt.rn.f64 %0, %1;" : "=d"(g) : "d"(x));
  return g;
}

// 1 / sqrt(x) for normal x well inside the range: one third-order step
// (Householder) from the special-function start, truncation below 2^-58.
GPR_D double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}

// x^(5/3) (sign of x), the distortion's det(A)^(5/3).  With y ~ |x|^(-1/3)
// from FP32 (of the mantissa times 2^(exponent mod 3): relative error below
// 2^-20), u = |x| y^2 and e = 1 - u y, |x|^(-1/3) = y (1 - e)^(-1/3) = y (1 +
// e/3 + 2 e^2/9 + O(e^3)): a third-order (Householder) step, truncation below
// 2^-61; the result is x^2 |x|^(-1/3).
static __device__ __noinline__ double pow53_general(double x) {
  const double cb = cbrt(x);
  return x * cb * cb;
}
// The start y ~ |x|^(-1/3) and the step's correction: |x|^(-1/3) = y + y p.
// The exponent of x is within 300 of 0.
GPR_D double icbrt_start(double x, double &p) {
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7ff;
  const int k = (ex - 1023 + 3000) / 3 - 1000;  // floor((ex - 1023) / 3)
  const int rem = ex - 1023 - 3 * k;
  const float m = __int_as_float(((127 + rem) << 23) | ((hi & 0xfffff) << 3) |
                                 (int)((unsigned)__double2loint(x) >> 29));
  const float s = exp2f(-0.33333333f * __log2f(m));  // in (1/2, 1]
  const unsigned sb = __float_as_uint(s);
  const double y = __hiloint2double((int)((sb >> 3) + ((1023 - 127 - k) << 20)), (int)(sb << 29));
  const double u = fabs(x) * (y * y);
  const double e = fma(-u, y, 1.0);
  p = e * fma(2.0 / 9.0, e, 1.0 / 3.0);
  return y;
}
GPR_D double pow53(double x) {
  const int ex = (__double2hiint(x) >> 20) & 0x7ff;
  if ((unsigned)(ex - 723) >= 600u)
    return pow53_general(x);
  double p;
  const double y = icbrt_start(x, p);
  const double w = (x * fabs(x)) * y;
  return fma(w, p, w);
}

// 2^(-sh) d in FP32 by the bit fields (truncated, not rounded); 0 below the
// FP32 range, a magnitude of at least 2^127 above it (infinities and NaNs
// included).
GPR_D float f32_scaled(double d, int sh) {
  const int hi = __double2hiint(d);
  const int field = (hi >> 20) & 0x7ff;
  int e = field - 896 - sh;  // FP32 exponent field
  e = e > 254 ? 254 : e;
  const unsigned m = ((hi & 0xfffffu) << 3) | ((unsigned)__double2loint(d) >> 29);
  const unsigned b = (e <= 0 || field == 0) ? 0u : ((unsigned)e << 23) | m;
  return __uint_as_float(b | (hi & 0x80000000u));
}
// 2^sh f in FP64 by the bit fields, f normal or zero
GPR_D double f64_scaled(float f, int sh) {
  const unsigned b = __float_as_uint(f);
  const unsigned m = b & 0x7fffffffu;
  const int hi = m ? (int)((m >> 3) + ((896 + sh) << 20)) : 0;
  return __hiloint2double(hi | (int)(b & 0x80000000u), m ? (int)(m << 29) : 0);
}

// approximate FP32 reciprocal and root (starts only)
GPR_D float rcp32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
GPR_D float sqrt32(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

}  // namespace gpr
