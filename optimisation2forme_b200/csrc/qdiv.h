// Correctly rounded FP64 quotients that share a divisor.
//
// The residual kernels divide many numerators by the same value (the cell
// volume V, the density rho): the reference computes each term as a/V with
// an IEEE division.  Here the reciprocal y = RN(1/b) is computed once, with
// an IEEE division, and each quotient is then obtained from y by
// multiply-add corrections (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1),
// 1990; the quotient theorem as stated in Muller et al., Handbook of
// Floating-Point Arithmetic, ch. 4):
//
//   q0 = RN(a*y)               within 1.5 ulp of a/b
//   r0 = RN(a - b*q0)          (fma)
//   q1 = RN(q0 + r0*y)         within 1/2 ulp + 2^-51 ulp of a/b, so
//   r1 = a - b*q1              is exact (fma), and
//   q  = RN(q1 + r1*y)         is RN(a/b) (Markstein's theorem: y is within
//                              1/2 ulp of 1/b and q1 within 1 ulp of a/b).
//
// The result is bit-identical to a/b, which keeps the FP64 residual
// bit-identical to the reference.  The theorem needs every intermediate in
// the normal range; outside it the plain division is used:
//   * the divisor: recip_for_div returns NaN unless 2^-500 <= |b| <= 2^500,
//     and a NaN y sends every quotient of that divisor to a/b;
//   * the quotient: unless 2^-400 <= |q0| <= 2^400 (so zeros, signed zeros,
//     infinities, NaNs and extreme magnitudes) the result is a/b.
// Within both ranges |a| lies in [2^-901, 2^901], so r0 and r1 are normal.
//
// The helpers are __host__ __device__ so that the CPU test
// (tests/qdiv_check.cpp) runs this very code against IEEE division.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define O2F_QDIV_FN __host__ __device__ __forceinline__
#else
#define O2F_QDIV_FN inline
#endif

namespace o2f {

// y for qdiv: RN(1/b), or NaN when b is outside [2^-500, 2^500].
O2F_QDIV_FN double recip_for_div(double b) {
  const double m = fabs(b);
  return (m >= 0x1p-500 && m <= 0x1p+500) ? 1.0 / b : NAN;
}

// The same from an already computed inv_b = RN(1/b).
O2F_QDIV_FN double recip_for_div(double b, double inv_b) {
  const double m = fabs(b);
  return (m >= 0x1p-500 && m <= 0x1p+500) ? inv_b : NAN;
}

// RN(a/b) given y = recip_for_div(b).
O2F_QDIV_FN double qdiv(double a, double b, double y) {
  const double q0 = a * y;
  const double m = fabs(q0);
  if (!(m >= 0x1p-400 && m <= 0x1p+400)) return a / b;
  const double r0 = fma(-b, q0, a);
  const double q1 = fma(r0, y, q0);
  const double r1 = fma(-b, q1, a);
  return fma(r1, y, q1);
}

// The same without the fallback, for loops that divide many numerators by
// one value: `ok` is cleared when the quotient is outside the range above,
// and the caller then recomputes with plain division.
O2F_QDIV_FN double qdiv_flag(double a, double b, double y, bool& ok) {
  const double q0 = a * y;
  const double m = fabs(q0);
  ok &= (m >= 0x1p-400) & (m <= 0x1p+400);
  const double r0 = fma(-b, q0, a);
  const double q1 = fma(r0, y, q0);
  const double r1 = fma(-b, q1, a);
  return fma(r1, y, q1);
}

// Without branches, for code that keeps many quotients in flight: the
// reciprocal comes from a seed by Newton's iteration and Markstein's final
// correction, and whatever leaves the range of the proofs above clears `ok`
// (the caller then recomputes with plain division).
//
// recip_seeded: y0 within 2^-18 of 1/b (relative).  Two Newton steps leave an
// error below one ulp, and RN(y + y * RN(1 - b*y)) is then RN(1/b) unless b's
// significand is all ones (Markstein 1990; Muller et al., ch. 4), which is
// excluded here.
O2F_QDIV_FN unsigned high_word(double x) {
#if defined(__CUDA_ARCH__)
  return (unsigned)__double2hiint(x);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &x, 8);
  return (unsigned)(u >> 32);
#endif
}
O2F_QDIV_FN unsigned low_word(double x) {
#if defined(__CUDA_ARCH__)
  return (unsigned)__double2loint(x);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &x, 8);
  return (unsigned)u;
#endif
}
// 2^-400 <= |x| < 2^400, by the exponent field.
O2F_QDIV_FN bool mid_range(double x) { return (high_word(x) & 0x7fffffffu) - 0x26f00000u < 0x32000000u; }
O2F_QDIV_FN bool is_zero(double x) { return ((high_word(x) & 0x7fffffffu) | low_word(x)) == 0u; }

O2F_QDIV_FN double recip_seeded(double b, double y0, bool& ok) {
  ok &= mid_range(b) & !(((high_word(b) & 0xfffffu) == 0xfffffu) & (low_word(b) == 0xffffffffu));
  const double y1 = fma(y0, fma(-b, y0, 1.0), y0);
  const double y2 = fma(y1, fma(-b, y1, 1.0), y1);
  return fma(y2, fma(-b, y2, 1.0), y2);
}

// RN(a/b) given y = RN(1/b); zero numerators included (with the quotient's sign).
O2F_QDIV_FN double quot(double a, double b, double y, bool& ok) {
  const double q0 = a * y;
  const bool zero = is_zero(a);
  ok &= mid_range(q0) | zero;
  const double r0 = fma(-b, q0, a);
  const double q1 = fma(r0, y, q0);
  const double r1 = fma(-b, q1, a);
  const double q = fma(r1, y, q1);
  return zero ? q0 : q;
}

// RN(sqrt(a)) for a > 0 from a seed y0 within 2^-18 of 1/sqrt(a) (relative):
// Goldschmidt's iteration on g = sqrt(a), h = 1/(2 sqrt(a)), then Markstein's
// correction g + h (a - g g), whose residual is exact (Muller et al., ch. 4).
O2F_QDIV_FN double sqrt_seeded(double a, double y0, bool& ok) {
  ok &= mid_range(a) & (high_word(a) < 0x80000000u);
  double g = a * y0, h = 0.5 * y0;
  double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  g = fma(h, fma(-g, g, a), g);
  return fma(h, fma(-g, g, a), g);
}

#if defined(__CUDACC__)
__device__ __forceinline__ double sqrt_fast(double a, bool& ok) {
  double y0;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(a));
  return sqrt_seeded(a, y0, ok);
}
__device__ __forceinline__ double recip_fast(double b, bool& ok) {
  double y0;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
  return recip_seeded(b, y0, ok);
}
__device__ __forceinline__ float recip_fast(float b, bool&) { return 1.0f / b; }
__device__ __forceinline__ float quot(float a, float, float y, bool&) { return a * y; }
#endif

// FP32 instantiations (the mixed-precision path, which is not bit-exact by
// design): one reciprocal per divisor, each quotient a multiplication
// (within 1.5 ulp of a/b).
O2F_QDIV_FN float recip_for_div(float b) { return 1.0f / b; }
O2F_QDIV_FN float recip_for_div(float, float inv_b) { return inv_b; }
O2F_QDIV_FN float qdiv(float a, float, float y) { return a * y; }
O2F_QDIV_FN float qdiv_flag(float a, float, float y, bool&) { return a * y; }

}  // namespace o2f
