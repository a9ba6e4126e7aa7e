// Sums of float64 products on the integer pipes (device and host).
//
// This part issues float64 instructions at 2 per clock and SM, integer ones at about 100
// (32 x 32 -> 64-bit multiply-adds at about 35), and the two run side by side: a float64
// multiply-add takes the time of ~60 integer instructions.  The stencil sums of this path
// (TRiSK weights, advection coefficients, cell divergences) were bound by the float64 pipe
// with the integer pipes idle, so they are formed here in fixed point: every term is
// aligned to the largest one of its own sum, the sum is exact integer arithmetic, and the
// result is rounded once.  About 30 integer instructions a term instead of 64 clocks of the
// float64 pipe, and the float64 pipe is left to the rest of the kernel.
//
// Accuracy.  A value is 60 bits wide after alignment (53 significant), a weight 60 bits;
// of their product the low x low partial is dropped (a balanced split, so it is centred).
// A sum of n terms loses below (n + 1) 2^-55 of its largest term before it is rounded (2^-54.9
// the worst of 10 and 14 terms spread over 16 binades), and the one rounding adds at most 2^-53
// of the result.  Against a chain of n multiply-adds, which rounds n times, that is 0.4 to 0.65
// of its root mean square error and a third to a half of its worst.  Sums whose terms are
// exact and cancel exactly give zero.  Sums the format cannot hold (a non-finite or subnormal-range value, a total
// near the ends of the exponent range) are reported to the caller, which evaluates them in
// float64; values that are all zero sum to +0.
#pragma once

#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace fx {

constexpr uint32_t kExpMask = 0x7ff00000u;
constexpr uint32_t kBadWeight = 0x80000000u;  // exponent field of a weight the format refuses

FX_HD uint64_t bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  memcpy(&b, &x, 8);
  return b;
#endif
}
FX_HD double from_bits(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, 8);
  return x;
#endif
}
// tests of exact values on the integer side (a float64 compare costs a float64 slot)
FX_HD bool is_zero(double x) { return (bits_of(x) << 1) == 0u; }
FX_HD bool is_one(double x) { return bits_of(x) == 0x3ff0000000000000ull; }
FX_HD bool is_two(double x) { return bits_of(x) == 0x4000000000000000ull; }
// x / 2
FX_HD double half(double x) {
  const uint64_t b = bits_of(x);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
  return e - 2u < 2045u ? from_bits(b - ((uint64_t)1 << 52)) : 0.5 * x;  // e in [2, 2046]
}
FX_HD int clz64(uint64_t x) {  // x != 0
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return __builtin_clzll(x);
#endif
}
FX_HD uint32_t umax(uint32_t a, uint32_t b) { return a > b ? a : b; }
FX_HD uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }
FX_HD uint32_t umax_sum(uint32_t a, uint32_t b, uint32_t c) {  // max(a + b, c), one instruction
#ifdef __CUDA_ARCH__
  return __viaddmax_u32(a, b, c);
#else
  return umax(a + b, c);
#endif
}
FX_HD uint64_t shr64(uint64_t x, uint32_t d) {  // shifts past 63 give zero
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(d));
  return r;
#else
  return d > 63u ? 0u : x >> d;
#endif
}

// One weight: the 53-bit significand times 2^7 as hi 2^32 + lo with lo in [-2^31, 2^31),
// its exponent field in place, and the row the term gathers.
struct alignas(16) Weight {
  int32_t hi, lo;
  uint32_t e;
  int32_t row;
};

FX_HD Weight weight(double w, int32_t row) {
  const uint64_t b = bits_of(w);
  const uint32_t e = (uint32_t)(b >> 32) & kExpMask;
  Weight r{0, 0, 0u, row};
  if (e == 0u || e == kExpMask) {  // zero adds nothing; subnormal and non-finite are refused
    r.e = (b << 1) == 0u ? 0u : kBadWeight;
    return r;
  }
  int64_t m = (int64_t)(((b & 0xfffffffffffffull) | 0x10000000000000ull) << 7);
  m = (int64_t)b < 0 ? -m : m;
  r.lo = (int32_t)(uint32_t)(uint64_t)m;
  r.hi = (int32_t)((m - r.lo) >> 32);
  r.e = e;
  return r;
}

// significand << 7, moved right by d, with the sign of `sign_hi` (|result| < 2^60)
FX_HD int64_t aligned(uint32_t hi, uint32_t lo, uint32_t d, uint32_t sign_hi) {
  const uint64_t m = shr64((((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << 7, d);
  return (int32_t)sign_hi < 0 ? -(int64_t)m : (int64_t)m;
}

// +-(t + frac 2^-32) 2^(63 - e0 ... ): the float64 nearest to sign (t + frac / 2^32) 2^s, given
// as the biased exponent `be` that a t with its top bit at 2^63 would have
FX_HD double pack(uint64_t t, uint32_t frac, int be, bool neg) {
  if (t < 0x80000000ull) {  // a deep cancellation: the fraction becomes the low word
    t = (t << 32) | frac;
    frac = 0u;
    be -= 32;
    if (t == 0u) return 0.0;
  }
  const int n = clz64(t);
  t = (t << n) | (uint64_t)(n ? frac >> (32 - umin((uint32_t)n, 32u)) : 0u);
  // round half up in magnitude; a carry out of the significand runs into the exponent
  uint64_t b = ((uint64_t)(uint32_t)(be - n - 1) << 52) + (t >> 11) + ((t >> 10) & 1u);
  return from_bits(b | ((uint64_t)neg << 63));
}

// whether every value is a zero (an absent tracer, air at rest: sums that need no float64)
template <int N>
FX_HD bool all_zero(const double (&x)[N]) {
  uint64_t b = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) b |= bits_of(x[j]);
  return (b << 1) == 0u;
}

// sum_j w_j x_j over N terms (N <= 15; unused slots hold a zero weight and any finite x).
// False when the sum has to be evaluated in float64 (see above).
template <int N>
FX_HD bool dot(const double (&x)[N], const Weight* w, double* out) {
  static_assert(N <= 15, "the 64-bit partial sums hold 15 terms");
  uint32_t amax = 0u, emax = 0u, wmax = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint32_t a = (uint32_t)(bits_of(x[j]) >> 32) & kExpMask;
    amax = umax(amax, a);
    emax = umax_sum(a, w[j].e, emax);
    wmax = umax(wmax, w[j].e);
  }
  // emax - wmax >= 64 binades: zero and subnormal values fall out of the window by themselves
  if (amax == kExpMask || wmax >= kBadWeight || emax - wmax < (64u << 20) || (emax >> 20) - 1223u > 1837u) {
    *out = 0.0;
    return amax == 0u && wmax < kBadWeight && all_zero(x);
  }
  int64_t hh = 0, c1 = 0, c2 = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint64_t b = bits_of(x[j]);
    const uint32_t hi = (uint32_t)(b >> 32);
    const int64_t m = aligned(hi, (uint32_t)b, (emax - ((hi & kExpMask) + w[j].e)) >> 20, hi);
    const int32_t ml = (int32_t)(uint32_t)(uint64_t)m;
    const int32_t mh = (int32_t)(uint32_t)((uint64_t)m >> 32) + (int32_t)((uint32_t)ml >> 31);
    hh += (int64_t)mh * w[j].hi;
    c1 += (int64_t)mh * w[j].lo;
    c2 += (int64_t)ml * w[j].hi;
  }
  // total = (t + frac / 2^32) 2^64 2^(emax - 2164)
  const int64_t c = (c1 >> 1) + (c2 >> 1);
  int64_t t = hh + (c >> 31);
  uint32_t frac = (uint32_t)c << 1;
  const bool neg = t < 0;
  if (neg) {
    t = ~t + (frac == 0u ? 1 : 0);
    frac = 0u - frac;
  }
  *out = pack((uint64_t)t, frac, (int)(emax >> 20) - 1014, neg);
  return true;
}

// sum_j s_j x_j over N <= 8 terms, s_j = +-1 given as the sign bit (bit 31) of sgn[j]; a slot
// that is not used holds x = 0.  False as for dot().
template <int N>
FX_HD bool sum(const double (&x)[N], const uint32_t (&sgn)[N], double* out) {
  static_assert(N <= 8, "the 64-bit sum holds 8 terms");
  uint32_t amax = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) amax = umax(amax, (uint32_t)(bits_of(x[j]) >> 32) & kExpMask);
  if ((amax >> 20) - 128u > 1912u) {
    *out = 0.0;
    return amax == 0u && all_zero(x);
  }
  int64_t t = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint64_t b = bits_of(x[j]);
    const uint32_t hi = (uint32_t)(b >> 32);
    t += aligned(hi, (uint32_t)b, (amax - (hi & kExpMask)) >> 20, hi ^ sgn[j]);
  }
  const bool neg = t < 0;
  *out = pack(neg ? 0u - (uint64_t)t : (uint64_t)t, 0u, (int)(amax >> 20) + 4, neg);
  return true;
}

// The positive and the negative part of the terms s_j x_j, *pos = sum of the positive ones and
// *neg = minus the sum of the negative ones, from one alignment.  False as for dot().
template <int N>
FX_HD bool sum_parts(const double (&x)[N], const uint32_t (&sgn)[N], double* pos, double* neg) {
  static_assert(N <= 8, "the 64-bit sum holds 8 terms");
  uint32_t amax = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) amax = umax(amax, (uint32_t)(bits_of(x[j]) >> 32) & kExpMask);
  if ((amax >> 20) - 128u > 1912u) {
    *pos = *neg = 0.0;
    return amax == 0u && all_zero(x);
  }
  uint64_t p = 0u, q = 0u;
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const uint64_t b = bits_of(x[j]);
    const uint32_t hi = (uint32_t)(b >> 32);
    const uint64_t t = (uint64_t)aligned(hi, (uint32_t)b, (amax - (hi & kExpMask)) >> 20, 0u);
    if ((int32_t)(hi ^ sgn[j]) < 0) q += t;
    else p += t;
  }
  *pos = pack(p, 0u, (int)(amax >> 20) + 4, false);
  *neg = pack(q, 0u, (int)(amax >> 20) + 4, false);
  return true;
}

FX_HD bool is_finite(double x) { return ((uint32_t)(bits_of(x) >> 32) & kExpMask) != kExpMask; }
// x where x > 0, else +0 (NaN gives 0)
FX_HD double positive(double x) { return bits_of(x) - 1u < 0x7ff0000000000000ull ? x : 0.0; }
// min(max(x, 0), 1), NaN gives 0
FX_HD double clamp01(double x) {
  const uint64_t b = bits_of(positive(x));
  return from_bits(b < 0x3ff0000000000000ull ? b : 0x3ff0000000000000ull);
}
// the smaller of two values in [0, inf]
FX_HD double min_nonneg(double a, double b) { return bits_of(a) < bits_of(b) ? a : b; }
// float64 order as integer order (negative values mirrored)
FX_HD int64_t order_key(double x) {
  const int64_t b = (int64_t)bits_of(x);
  return b ^ (int64_t)((uint64_t)(b >> 63) >> 1);
}
FX_HD double from_order_key(int64_t k) { return from_bits((uint64_t)(k ^ (int64_t)((uint64_t)(k >> 63) >> 1))); }

}  // namespace fx
