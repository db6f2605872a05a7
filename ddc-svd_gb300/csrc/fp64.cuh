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
// instructions: the reciprocal as above, q = a r, and the correction by the
// exact remainder (Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", 1990).  For operands within 2^+-500
// (mid_range); quot_rn leaves others to the operator.
__device__ __forceinline__ bool mid_range(double x) {
  return ((unsigned)__double2hiint(x) & 0x7ff00000u) - (523u << 20) <= (1000u << 20);
}
__device__ __forceinline__ double quot_mid(double a, double x) {
  double r = rcp_approx(x);
  const double e = fma(-x, r, 1.0);
  r = fma(r, fma(e, e, e), r);
  const double q = a * r;
  return fma(fma(-x, q, a), r, q);
}
__device__ __forceinline__ double quot_rn(double a, double x) {
  return mid_range(a) && mid_range(x) ? quot_mid(a, x) : a / x;
}

// order of non-negative values = order of their bit patterns
__device__ __forceinline__ long long bits(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ long long abs_bits(double x) { return __double_as_longlong(x) & 0x7fffffffffffffffll; }
// |x|'s bits for a maximum that ignores NaN, as fmax does
__device__ __forceinline__ long long max_bits(double x) {
  const long long b = abs_bits(x);
  return b <= 0x7ff0000000000000ll ? b : 0ll;
}

}  // namespace ddcsvd
