// Quotients without a division, to the division's bits.  Nothing but integer
// and floating-point operations on doubles (tests/quotient_check.cpp compiles
// this file for the host).
#pragma once

namespace mfg {

// The forms below report an operand outside their window through the sign of
// an integer that is or-ed together over a cell's many divisions: a chain of
// predicates would cost their latency each (a cell's five quotients 206 cycles
// against 52 without them).
__device__ __forceinline__ int hi_mag(double a) { return __double2hiint(a) & 0x7FFFFFFF; }
// negative unless lo <= exponent of a <= hi (biased); a non-negative a's high
// word alone orders the exponents
__device__ __forceinline__ int outside_exp(double a, int lo, int hi) {
  const int m = hi_mag(a);
  return (m - (lo << 20)) | (((hi + 1) << 20) - 1 - m);
}

// Correctly rounded a / b from y = RN(1 / b), for a divisor known before the
// dividend (the LU-SGS diagonal, a cell's volume, a triangle's three nodes):
// the quotient's dependent chain is one product and four fused multiply-adds
// instead of a division.  Markstein's theorem (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990): for y within half an ulp of 1/b and q within one ulp of
// a/b, r = a - b q is exact and RN(q + r y) = RN(a / b).  q0 = RN(a near) is
// within two ulps; one correction step makes it faithful, the second rounds
// correctly.  `near` (a reciprocal within one ulp, or y) serves in the steps
// before the last.  A zero a is within the window: its steps give a zero, and
// the sign of every quotient is set to the division's.  bad turns negative for
// an a that is neither zero nor of an exponent in [-500, 500] (subnormals,
// overflow risks, non-finite values); b is the caller's to test, with the same
// bounds.  The caller then takes the division itself.
__device__ __forceinline__ double quot_near(double a, double b, double near, double y, int &bad) {
  const int w = outside_exp(a, 523, 1523);
  bad |= (hi_mag(a) | __double2loint(a)) == 0 ? 0 : w;
  const double q0 = __dmul_rn(a, near);
  const double r0 = __fma_rn(-b, q0, a);
  const double q1 = __fma_rn(r0, near, q0);
  const double r1 = __fma_rn(-b, q1, a);
  const double q = __fma_rn(r1, y, q1);
  const int sign = (__double2hiint(a) ^ __double2hiint(b)) & 0x80000000;
  return __hiloint2double((__double2hiint(q) & 0x7FFFFFFF) | sign, __double2loint(q));
}

// RN(1 / b) from an approximation y0 with e = 1 - b y0 of less than 2^-18: the
// geometric series 1 / b = y0 / (1 - e) = y0 (1 + e + e^2 + O(e^3)) leaves
// `near` within one ulp, and for such a reciprocal r = 1 - b near and RN(near +
// near r) round correctly (Markstein, as above) except when the significand of
// b is all ones.  bad turns negative for that significand and for an exponent
// outside [-500, 500].
__device__ __forceinline__ double rcp_rn_from(double b, double y0, double &near, int &bad) {
  const int ones = (__double2hiint(b) | 0xFFF00000) & __double2loint(b);
  bad |= outside_exp(b, 523, 1523) | (ones == -1 ? -1 : 0);
  const double e = __fma_rn(-b, y0, 1.0);
  near = __fma_rn(y0, __fma_rn(e, e, e), y0);
  const double r = __fma_rn(-b, near, 1.0);
  return __fma_rn(near, r, near);
}

}  // namespace mfg
