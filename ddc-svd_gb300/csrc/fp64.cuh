// fp64.cuh -- FP64 arithmetic of stages 2-4 in few instructions.
//
// GB300's FP64 pipe bounds the stages that use it: one FP64 instruction of a warp holds it
// for 64 cycles (19 per SM when four warps or more share the SM), against one
// for FP32 and integer instructions, and comparisons, fmin / fmax take a turn
// in it like an addition.  Measured per warp (one warp per scheduler): add,
// multiply, FMA 64-66 cycles, a compare and an add 176, a division 566, hypot
// 1059; the approximate reciprocal and the conversions to and from FP32 do not
// use the pipe (9 and 2 cycles).  So divisions are formed from the approximate
// reciprocal by one cubic Newton step (four FP64 instructions instead of
// about nine), values of known sign are compared through their bit patterns,
// and whatever does not need 53 bits is FP32.

#pragma once

namespace ddcsvd {

// a / x to about an ulp for normal x: with r ~ 1/x and e = 1 - x r,
// 1/x = r (1 + e + e^2 + ...); |e| < 2^-18, so e^3 is below rounding.  x = 0
// or subnormal gives NaN (callers fall back or had an infinity there before).
__device__ __forceinline__ double rcp_approx(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double quot(double a, double x) {
  const double r = rcp_approx(x);
  const double e = fma(-x, r, 1.0);
  const double y = fma(e, e, e);
  const double t = a * r;
  return fma(t, y, t);
}
// a / x rounded to nearest, as the division operator gives it, in six FP64
// instructions and a check: the reciprocal as above, q = a r, and the correction by
// the remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990).  r is not correctly rounded (|1 - x r| is at most
// 2^-53 (1 + 2^-6): half an ulp of rounding, and the seed's error, at most 2^-19.9,
// to the third power), so the corrected quotient can miss only where a / x lies within
// 2^-49 of an ulp of the midpoint of two doubles.  q is within 2.1 ulps of a / x,
// so its remainder is then x times 1/2 or 3/2 (or such a fraction of a
// neighbouring binade's ulp: a power of two, or three times one) of an ulp of q, to
// 2^-48: `sure` compares the 20 leading bits of the significands.  Some 2^-17 of the
// quotients are not sure (and those by powers of two, with d = 0); quot_rn leaves
// them, and operands beyond 2^+-500 (mid_range), to the operator.  The check costs
// the D&C and the vectors 1% (3000 columns 4.32 -> 4.36 ms, 2048 problems 11.44 -> 11.58).
__device__ __forceinline__ bool mid_range(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) - (523u << 20) <= (1000u << 20);
}
__device__ __forceinline__ double quot_mid(double a, double x, bool& sure) {
  double r = rcp_approx(x);
  const double e = fma(-x, r, 1.0);
  r = fma(r, fma(e, e, e), r);
  const double q = a * r, d = fma(-x, q, a);
  // leading bits of the significands of d, x and 3 x, from bit 31 down
  const unsigned hd = (unsigned)__double2hiint(d) << 12, hx = (unsigned)__double2hiint(x) << 12;
  const unsigned h3 = __float_as_uint(__uint_as_float(0x3f800000u | hx >> 9) * 1.5f) << 9;
  sure = hd - hx + (1u << 12) > (2u << 12) && hd - h3 + (2u << 12) > (4u << 12);
  return fma(d, r, q);
}
__device__ __forceinline__ double quot_rn(double a, double x) {
  bool sure;
  const double q = quot_mid(a, x, sure);
  return mid_range(a) && mid_range(x) && sure ? q : a / x;
}

// order of non-negative values = order of their bit patterns
__device__ __forceinline__ long long bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ long long abs_bits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }
// the order of any values (-0 and 0 equal) as integers
__device__ __forceinline__ long long order_bits(double x) {
  const long long b = bits(x);
  return (b << 1) == 0 ? 0 : b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// |x|'s bits for a maximum that ignores NaN, as fmax does
__device__ __forceinline__ long long max_bits(double x) {
  const long long b = abs_bits(x);
  return b <= 0x7ff0000000000000ll ? b : 0ll;
}

}  // namespace ddcsvd
