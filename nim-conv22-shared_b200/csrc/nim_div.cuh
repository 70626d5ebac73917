// Correctly rounded FP64 quotients in straight-line code, for the kernels
// whose divisions are their critical resource.
//
// An IEEE division compiles to its own branch (a slow path for extreme
// operands), so a kernel with a dozen of them runs them one after the other.
// Here the reciprocal of a divisor is refined once, every numerator over it
// takes five fused operations, and nothing branches: the quotients of a
// formula overlap.  The result is a / b rounded to nearest, bit for bit.
//
// Method: P. W. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Develop. 34 (1990) 111-119 (the
// final step q + r y with an exactly computed remainder r = a - b q).
//   y  = 1/b to a relative error below 2^-53 (1 + 2^-26): the documented
//        20-bit rcp.approx start, two Newton steps (2^-40, 2^-80), rounded
//   q0 = a y, then twice q <- q + (a - b q) y: after the first step q is
//        within (1/2 + 2^-51) ulp of Q = a/b, so the second adds an exact
//        remainder times y and forms Q to within 2^-54 (1 + 2^-25) ulp
//        before its one rounding.
// A quotient of two 53-bit numbers that is no 53-bit number itself lies at
// least 2^-54 (2/b') ulp from every midpoint of the format (b' in [1, 2) the
// significand of b: a - b m is a nonzero multiple of 2^-105 for a midpoint
// m).  With b' <= 2 - 2^-20 that is 2^-54 (1 + 2^-21): larger than the
// error, so the rounding is that of Q.  Divisors with b' above (and zero,
// subnormal, infinite or NaN ones) are div_ok's to refuse: the caller then
// divides.  Exponents must keep every intermediate normal: |b| and nonzero
// |a| within 2^+-480 are enough.
#pragma once
#include <cstdint>

namespace nim {

struct Recip {
  double b, y;
};
__device__ __forceinline__ Recip recip(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
  y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
  return {b, y};
}
// (the remainder as b q - a: with b > 0 that is +0 where the quotient is exact
// or a zero, and q - (+0) y leaves q as it is, -0 included; with b < 0 a +0
// numerator's quotient loses its sign)
__device__ __forceinline__ double quot(double a, const Recip &r) {
  double q = __dmul_rn(a, r.y);
  q = __fma_rn(-__fma_rn(r.b, q, -a), r.y, q);
  return __fma_rn(-__fma_rn(r.b, q, -a), r.y, q);
}
// b's exponent within +-E and its significand at most 2 - 2^-20
template <int E>
__device__ __forceinline__ bool div_ok(double b) {
  const uint32_t hi = (uint32_t)__double2hiint(b) & 0x7fffffffu;
  return (hi - ((1023u - E) << 20)) < ((2u * E) << 20) && (hi & 0xfffffu) != 0xfffffu;
}
// a's exponent within +-E, or a zero
template <int E>
__device__ __forceinline__ bool num_ok(double a) {
  const uint32_t hi = (uint32_t)__double2hiint(a) & 0x7fffffffu;
  return (hi - ((1023u - E) << 20)) < ((2u * E) << 20) || a == 0.0;
}

}  // namespace nim
