// pow_exner_fx(x, y): pow_exner (pow_exner.cuh) in fixed point on the integer pipes, for the
// float64 step, whose other kernels leave those pipes idle while the float64 pipe, on which
// pow_exner takes ~130 operations, bounds them: the recovery of the last RK stage at 40962 x 55
// 538 -> 126 us (84 us without the Exner function).
//
// Method (the table-driven reduction of Tang, ACM TOMS 15 (1989) 144 and 16 (1990) 378, with a
// short reciprocal so that the reduced argument is exact):
//   x = 2^e m, m in [1, 2);  n / 2^11 close to 1 / m from the table, u = m n / 2^11 - 1 exactly,
//   |u| < 2^-9.9;
//   log2 x = e - log2(n / 2^11) + u / ln 2 - u^2 (1/2 - u/3 + ... + u^5/7) / ln 2,
//   the linear term and the table on 96 fraction bits;
//   z = y log2 x = k + j / 1024 + t, 0 <= t < 2^-10;
//   x^y = 2^k 2^(j/1024) (1 + r + r^2 (1/2 + r/6 + ... + r^4/720)), r = t ln 2.
// The error before the one rounding is below 2^-72 of the result (2.5 units of 2^-74: the
// truncations of t, r and the sum), so the result is correctly rounded except within 2^-19
// units in the last place of a rounding boundary, as pow_exner's.  Arguments outside
// (normal positive x, 2^-20 <= |y| < 16, result normal) take pow_exner.
//
// Compiles for the device and, for its tests, for the host; both give the same bits (integer
// arithmetic only).
#pragma once

#include "pow_exner.cuh"

#ifdef __CUDACC__
#define MPASG_POWFX_TABLE static __device__ const
#else
#define MPASG_POWFX_TABLE static const
#endif

namespace mpasg_pow {
namespace powfx {

struct alignas(16) Entry {
  uint64_t a;
  uint32_t b, c;
};

#include "pow_fx_tables.inc"

MPASG_POW_HD Entry entry(const Entry* p) {
#ifdef __CUDA_ARCH__
  const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
  return {(uint64_t)v.y << 32 | v.x, v.z, v.w};
#else
  return *p;
#endif
}
MPASG_POW_HD uint64_t mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}

struct U128 {
  uint64_t hi, lo;
};
MPASG_POW_HD U128 add(U128 a, U128 b) {
  const uint64_t lo = a.lo + b.lo;
  return {a.hi + b.hi + (lo < b.lo ? 1u : 0u), lo};
}
MPASG_POW_HD U128 neg(U128 a) { return {~a.hi + (a.lo == 0 ? 1u : 0u), (uint64_t)0 - a.lo}; }

// log2 of 2^e M 2^-52 (M with its leading bit) on 96 fraction bits, two's complement
MPASG_POW_HD U128 log2_fixed(uint64_t M, int e) {
  const Entry t = entry(kPowFxLog + ((M >> 42) & 1023));
  const uint64_t U = M * t.b - ((uint64_t)1 << 63);  // u on 63 fraction bits, signed
  const bool minus = (int64_t)U < 0;
  // u / ln 2: 126 fraction bits, of which 96 are kept
  const uint64_t ph = mulhi(U, kPowFxInvLn2) - (minus ? kPowFxInvLn2 : 0), pl = U * kPowFxInvLn2;
  const U128 lin = {(uint64_t)((int64_t)ph >> 30), ph << 34 | pl >> 30};
  // u^2 (1/2 - u/3 + ...) / ln 2: |u| on 72 fraction bits, the bracket on 64 (from u^3 on, 32)
  const uint64_t A = (minus ? (uint64_t)0 - U : U) << 9;
  const uint32_t a = (uint32_t)(A >> 32);  // 40 fraction bits
  const uint32_t p7 = (uint32_t)((uint64_t)a * kPowFxC7 >> 40);
  const uint32_t h6 = minus ? kPowFxC6 + p7 : kPowFxC6 - p7;
  const uint32_t p6 = (uint32_t)((uint64_t)a * h6 >> 40);
  const uint32_t h5 = minus ? kPowFxC5 + p6 : kPowFxC5 - p6;
  const uint64_t p5 = (uint64_t)a * h5 >> 8;
  const uint64_t h4 = minus ? kPowFxC4 + p5 : kPowFxC4 - p5;
  const uint64_t p4 = mulhi(A, h4) >> 8;
  const uint64_t h3 = minus ? kPowFxC3 + p4 : kPowFxC3 - p4;
  const uint64_t p3 = mulhi(A, h3) >> 8;
  const uint64_t h2 = minus ? kPowFxC2 + p3 : kPowFxC2 - p3;
  const uint64_t w = mulhi(mulhi(A, A), h2);  // 80 fraction bits
  const U128 whole = {((uint64_t)(int64_t)e << 32) + t.c, t.a};
  return add(add(whole, lin), neg({w >> 48, w << 16}));
}

// mantissa of 2^f for the fraction f of z (96 fraction bits), on 52 bits, rounded (2^53 for 2)
MPASG_POW_HD uint64_t exp2_mantissa(U128 z) {
  const Entry t = entry(kPowFxExp + ((z.hi >> 22) & 1023));
  const uint64_t T = (z.hi & ((1u << 22) - 1u)) << 42 | z.lo >> 22;  // 74 fraction bits
  const uint64_t r = mulhi(T, kPowFxLn2) + (T != 0 ? 1u : 0u);       // centres the truncations
  const uint32_t rs = (uint32_t)(r >> 32);                           // 42 fraction bits
  const uint32_t h5 = kPowFxD5 + (uint32_t)((uint64_t)rs * kPowFxD6 >> 42);
  const uint64_t h4 = kPowFxD4 + ((uint64_t)rs * h5 >> 10);
  const uint64_t h3 = kPowFxD3 + (mulhi(r, h4) >> 10);
  const uint64_t h2 = ((uint64_t)1 << 63) + (mulhi(r, h3) >> 10);
  const uint64_t q = r + ((mulhi(mulhi(r, r), h2) + 512) >> 10);
  // table (95 fraction bits) + table q (137)
  const uint64_t ph = mulhi(t.a, q), pl = t.a * q;
  const U128 R = add({t.a >> 32, t.a << 32 | t.b}, {ph >> 42, ph << 22 | pl >> 42});
  const uint64_t mant = R.hi << 21 | R.lo >> 43, rest = R.lo & (((uint64_t)1 << 43) - 1), half = (uint64_t)1 << 42;
  return mant + ((rest > half || (rest == half && (mant & 1))) ? 1u : 0u);
}

}  // namespace powfx

#ifdef __CUDACC__
static __device__ __noinline__
#else
inline
#endif
double pow_exner_slow(double x, double y) { return pow_exner(x, y); }

MPASG_POW_HD double pow_exner_fx(double x, double y) {
  const uint64_t bx = (uint64_t)bits_of(x), by = (uint64_t)bits_of(y);
  const uint32_t hx = (uint32_t)(bx >> 52);                  // sign and exponent
  const int ey = (int)((uint32_t)(by >> 52) & 0x7ffu) - 1023;
  if (hx - 1u >= 2046u || ey < -20 || ey > 3) return pow_exner_slow(x, y);
  const uint64_t one = (uint64_t)1 << 52;
  powfx::U128 L = powfx::log2_fixed((bx & (one - 1)) | one, (int)hx - 1023);
  bool minus = (int64_t)L.hi < 0;
  if (minus) L = powfx::neg(L);
  // |z| = |L| |y|: the top 128 bits of L times y's significand on 63 fraction bits, then 2^(ey + 1)
  const uint64_t Y = ((by & (one - 1)) | one) << 11;
  powfx::U128 z = powfx::add({powfx::mulhi(L.hi, Y), L.hi * Y}, {0, powfx::mulhi(L.lo, Y)});
  const int s = ey + 1;
  if (s > 0) z = {z.hi << s | z.lo >> (64 - s), z.lo << s};
  else if (s < 0) z = {z.hi >> -s, z.hi << (64 + s) | z.lo >> -s};
  if (by >> 63) minus = !minus;
  if (minus) z = powfx::neg(z);
  const int k = (int)((int64_t)z.hi >> 32);
  if (k < -1000 || k > 1000) return pow_exner_slow(x, y);
  return from_bits((int64_t)(((uint64_t)(k + 1022) << 52) + powfx::exp2_mantissa(z)));
}

}  // namespace mpasg_pow
