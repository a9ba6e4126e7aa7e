// float64 reciprocal and quotient with most of the work off the float64 pipe (device and
// host).
//
// A float64 operation costs 64 clocks of its pipe here and the compiler's division about
// nine of them (592 clocks measured).  The reciprocal is first formed to about 44 bits in
// float32 (a float32 reciprocal and one Newton step with the divisor split into two float32
// parts), which runs beside the float64 pipe; then
//   quotient    q0 = a r,  q = q0 + (a - b q0) r        (4 float64 operations with the seed's sum)
//   reciprocal  r + r (1 - b r)                         (3)
// Both last steps round once a value known to 2^-88, so the result is the correctly rounded
// one but for about one argument in 2^34 (Markstein's residual correction).  Divisors outside
// [2^-100, 2^70), negative or not finite, and nonzero dividends below 2^-600 or not finite take
// the compiler's division.
#pragma once

#include <math.h>

#include "fixdot.cuh"

namespace fx {

FX_HD float float_of_bits(uint32_t b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float f;
  memcpy(&f, &b, 4);
  return f;
#endif
}
FX_HD uint32_t bits_of_float(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t b;
  memcpy(&b, &f, 4);
  return b;
#endif
}
FX_HD float seed_rcp(float b) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
#else
  return 1.0f / b;
#endif
}
// a normal float32 (or zero, read as 2^-127) as float64, without a conversion instruction
FX_HD double widen(float f) {
  const uint32_t b = bits_of_float(f);
  const uint32_t hi = (((b & 0x7fffffffu) >> 3) + 0x38000000u) | (b & 0x80000000u);
  return from_bits((uint64_t)hi << 32 | (b << 29));
}

// positive, exponent inside [2^-100, 2^70): the float32 parts of b and 1 / b stay normal, what
// widen() adds to a zero correction (2^-127) is below 2^-57 of 1 / b
FX_HD bool plain_divisor(double b) { return (uint32_t)(bits_of(b) >> 32) - ((1023u - 100u) << 20) < (170u << 20); }

// 1 / b to about 2^-44 for a plain divisor; `r0` (tests) replaces the float32 seed
FX_HD double rcp44(double b, float r0) {
  const uint64_t u = bits_of(b);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u;
  const uint32_t top = (hi << 3 | lo >> 29) + 0x40000000u;  // exponent bias 1023 -> 127
  const uint32_t e = top & 0x7f800000u;
  // b = bh + bl: 24 significant bits, then the next 23
  const float bh = float_of_bits(top);
  const float one_ulp = float_of_bits(e - (23u << 23));
  const float bl = float_of_bits((e - (23u << 23)) | ((lo & 0x1fffffffu) >> 6)) - one_ulp;
  float t = fmaf(-bh, r0, 1.0f);
  t = fmaf(-bl, r0, t);
  return widen(r0) + widen(r0 * t);
}
FX_HD float seed_of(double b) {
  const uint64_t u = bits_of(b);
  return seed_rcp(float_of_bits((uint32_t)(u >> 29) + 0x40000000u));
}

FX_HD double rcp(double b) {
  if (!plain_divisor(b)) return 1.0 / b;
  const double r = rcp44(b, seed_of(b));
  return fma(r, fma(-b, r, 1.0), r);
}

FX_HD double quotient_from(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-b, q, a), r, q);
}
// whether a dividend keeps the residual a - b q exact and the quotient finite
FX_HD bool plain_dividend(double a) {
  return (((uint32_t)(bits_of(a) >> 32) & 0x7fffffffu) - ((1023u - 600u) << 20)) < (1400u << 20);
}
FX_HD double quotient(double a, double b) {
  if (!plain_divisor(b) || !plain_dividend(a)) return plain_divisor(b) && is_zero(a) ? a : a / b;
  return quotient_from(a, b, rcp44(b, seed_of(b)));
}

}  // namespace fx
