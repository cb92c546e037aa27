// Positive floating-point numbers with 64-bit mantissas on the integer
// pipes: products, reciprocals, square roots, exp and log for the column
// physics (internal header).
//
// The FP64 pipe of this GPU takes 64 cycles for one warp instruction, the
// integer and FP32 pipes one or two.  A product of two 64-bit mantissas is
// three 32 x 32 -> 64 bit multiply-adds and a few additions, so arithmetic
// of this kind is several times faster than FP64 instructions, runs beside
// them, and keeps 62 or more significant bits where FP64 keeps 53.
//
// A UF is m 2^(e-63), m > 0.  "Normalised" means that m's top bit is set;
// a product of normalised numbers lacks at most one leading bit, and each
// further unnormalised product one more.  rcp, sqrt and log take normalised
// arguments.  No exponent is checked: callers bound their inputs and take
// FP64 arithmetic outside the bounds.
//
// Methods: the reciprocal and the square root start from the FP32
// special-function unit's 23 bits and make one cubic step; exp and log are
// the table-driven methods of P. T. P. Tang (ACM TOMS 15 (1989) and 16
// (1990)) in fixed point with 256-entry tables (gen_fx_tables.py).
#pragma once

#include <cuda_runtime.h>

#include "fx_tables.cuh"

namespace dccm {
namespace fx {

typedef unsigned long long u64;
struct UF {
  u64 m;
  int e;
};

// Constant as a UF (exact), at compile time or on the host.
__host__ __device__ constexpr UF uf(double v) {
  int e = 0;
  while (v >= 2.0) v *= 0.5, ++e;
  while (v < 1.0) v *= 2.0, --e;
  return {(u64)(v * 4503599627370496.0) << 11, e};
}

// floor(a b 2^-64), or one less (the product of the low words is left out)
__device__ __forceinline__ u64 mulhi(u64 a, u64 b) {
  const unsigned al = (unsigned)a, ah = (unsigned)(a >> 32), bl = (unsigned)b, bh = (unsigned)(b >> 32);
  const u64 p = (u64)ah * bl;
  const u64 q = (u64)al * bh + (unsigned)p;
  return (u64)ah * bh + (p >> 32) + (q >> 32);
}
__device__ __forceinline__ UF mul(UF a, UF b) { return {mulhi(a.m, b.m), a.e + b.e + 1}; }
// m's upper word must not be zero
__device__ __forceinline__ UF norm(UF a) {
  const int z = __clz((int)(a.m >> 32));
  return {a.m << z, a.e - z};
}

// Positive normal double.
__device__ __forceinline__ UF from_double(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
  return {((u64)mh << 32) | (lo << 11), (int)((hi >> 20) & 0x7FFu) - 1023};
}
// Nearest double (ties away from zero); the exponent must be in the normal range.
__device__ __forceinline__ double to_double(UF a) {
  a = norm(a);
  const u64 r = (a.m >> 11) + ((unsigned)a.m >> 10 & 1u);  // 53 bits, or 2^53
  return __hiloint2double((int)((unsigned)(r >> 32) + ((unsigned)(a.e + 1022) << 20)), (int)(unsigned)r);
}

// 1 / a, a normalised; m of the result in [2^62, 2^63].
__device__ __forceinline__ UF rcp(UF a) {
  const unsigned ah = (unsigned)(a.m >> 32), al = (unsigned)a.m;
  float f;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(f) : "f"(__uint_as_float(0x3F800000u | (ah >> 8 & 0x7FFFFFu))));
  // y ~ 1 / D in 2^-31 units, D = m 2^-63 in [1, 2), f in (1/2, 1]
  const unsigned y = (min(__float_as_uint(f), 0x3F7FFFFFu) << 7 & 0x3FFFFFFFu) | 0x40000000u;
  // err = 1 - D y in 2^-62 units (below 2^-21)
  const u64 t = (u64)ah * y + ((u64)al * y >> 32);
  const long long err = (long long)((1ull << 62) - t);
  const int e32 = (int)(err >> 10);  // 2^-52
  const long long g = err + (((long long)e32 * e32 >> 32) >> 10);  // err + err^2
  // y + y g, 2^-63 units: y g 2^-30 by words of g
  const u64 p = (u64)y * (unsigned)g;
  const long long c = (long long)(p >> 30) + (((long long)(int)y * (int)(g >> 32)) << 2);
  return {((u64)y << 32) + (u64)c, -a.e};
}

// sqrt(a), a normalised.
__device__ __forceinline__ UF sqrt(UF a) {
  const bool odd = a.e & 1;
  const u64 X = odd ? a.m : a.m >> 1;  // D / 4 in 2^-64 units, D in [1, 4), a = D 2^(e - odd)
  const unsigned xh = (unsigned)(X >> 32), xl = (unsigned)X;
  float f;
  // D as FP32 (truncated): exponent 0 or 1
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(f)
      : "f"(__uint_as_float((odd ? 0x40000000u : 0x3F800000u) | ((unsigned)(a.m >> 40) & 0x7FFFFFu))));
  // r ~ 1 / sqrt(D) in 2^-31 units, f in (1/2, 1]
  const unsigned r = (min(__float_as_uint(f), 0x3F7FFFFFu) << 7 & 0x3FFFFFFFu) | 0x40000000u;
  const u64 r2 = (u64)r * r;                                 // 1 / D in 2^-62 units, exact
  const long long err = (long long)((1ull << 62) - mulhi(X, r2 << 2));  // 1 - D r^2 in 2^-62 units
  const int e32 = (int)(err >> 10);                          // 2^-52
  const long long e2 = ((long long)e32 * e32 >> 32) >> 10;   // err^2
  const long long g = (err >> 1) + (e2 * 3 >> 3);            // err / 2 + 3 err^2 / 8
  const u64 s = ((u64)xh * r + ((u64)xl * r >> 32)) << 1;     // D r in 2^-62 units, below 2^63
  // s g, by words of both
  const unsigned sh = (unsigned)(s >> 32), sl = (unsigned)s;
  const u64 p = (u64)sh * (unsigned)g;
  const long long c = (long long)(p >> 30) + (((long long)(int)sh * (int)(g >> 32)) << 2) +
                      ((long long)(int)(g >> 12) * (int)(sl >> 1) >> 49);
  return {s + (u64)c, (odd ? a.e - 1 : a.e) / 2 + 1};
}

// 1 + a (any m > 0)
__device__ __forceinline__ UF one_plus(UF a) {
  if (a.e < 0) return {(1ull << 63) + (a.e < -63 ? 0ull : a.m >> -a.e), 0};
  const u64 one = a.e > 63 ? 0ull : (1ull << 63) >> a.e;
  return {(a.m >> 1) + (one >> 1), a.e + 1};
}

// a + b + c, rounded down at 2^-61 of the largest term; normalised.
__device__ __forceinline__ UF sum3(UF a, UF b, UF c) {
  const int e = max(max(a.e, b.e), c.e) + 2;
  return norm({(a.m >> min(e - a.e, 63)) + (b.m >> min(e - b.e, 63)) + (c.m >> min(e - c.e, 63)), e});
}
// a - b into r (normalised, rounded at 2^-62 of the larger one); false unless
// positive.
__device__ __forceinline__ bool sub(UF a, UF b, UF &r) {
  const int e = max(a.e, b.e) + 1;
  const long long s = (long long)(a.m >> min(e - a.e, 63)) - (long long)(b.m >> min(e - b.e, 63));
  const int z = __clzll(s);
  r = {(u64)s << (z & 63), e - z};
  return s > 0;
}

// e^x for x in 2^-58 units, |x| < 32.
__device__ __forceinline__ UF exp_fix(long long x) {
  // n = floor(256 x / ln 2), at most a little below it, so that the rest r >= 0
  const int xh = (int)(x >> 32);  // 2^-26
  const int n = ((int)((long long)xh * EXP_INV >> 32) - 4) >> 16;
  const u64 r = (u64)(x - (((long long)n * EXP_STEP_H << 20) + ((long long)n * EXP_STEP_L >> 12)));  // < 2^-8.5
  const unsigned r40 = (unsigned)(r >> 18), r32 = r40 >> 8;
  // w = 1/6 + r/24 + r^2/120, u = r w, p = r + r^2/2 + r^2 u
  const unsigned w = 715827883u + __umulhi(r32, 178956971u + __umulhi(r32, 35791394u));
  const unsigned u = (unsigned)((u64)r40 * w >> 32);  // 2^-40
  const u64 rr = r << 14, s = mulhi(rr, rr);          // r^2, 2^-80
  const u64 p = (r << 12) + (s >> 11) + ((u64)(unsigned)(s >> 32) * u >> 18);  // 2^-70
  const u64 T = __ldg(EXP2_256 + (n & 255));
  return {T + (mulhi(T, p << 1) >> 7), (n >> 8) + 1};
}

// ln a in 2^-57 units, a normalised and >= 1.
__device__ __forceinline__ u64 log_fix(UF a) {
  const unsigned j = (unsigned)(a.m >> 55) & 255u;
  const ulonglong2 T = __ldg(LOG_256 + j);
  const u64 f = (a.m & ((1ull << 55) - 1)) << 8;  // D - F, 2^-71
  const u64 u = mulhi(f, T.x);                    // (D - F) / F < 2^-8, 2^-70
  const u64 v = u << 2;                           // 2^-72
  const u64 s = mulhi(v, v);                      // u^2, 2^-80
  const unsigned u32 = (unsigned)(v >> 40);       // 2^-32
  // u^3 (1/3 - u/4 + u^2/5 - u^3/6 + u^4/7)
  const unsigned w =
      1431655765u - __umulhi(u32, 1073741824u - __umulhi(u32, 858993459u - __umulhi(u32, 715827883u - __umulhi(u32, 613566757u))));
  const unsigned u3 = (unsigned)((u64)(unsigned)(v >> 32) * (unsigned)(s >> 32) >> 32);  // 2^-56
  const u64 l = u - (s >> 11) + ((u64)u3 * w >> 18);                                    // log(1 + u), 2^-70
  return (u64)(unsigned)a.e * LN2_57 + T.y + (l >> 13);
}

// 1 / x for a double: nearly correctly rounded where x and 1 / x are
// comfortably normal, the exact division elsewhere.
__device__ __forceinline__ double rcp_d(double x) {
  const unsigned hi = (unsigned)__double2hiint(x);
  const unsigned ef = hi >> 20 & 0x7FFu;
  if (ef - 16u >= 2016u) return 1.0 / x;
  const double y = to_double(rcp(from_double(x)));
  return __hiloint2double(__double2hiint(y) | (int)(hi & 0x80000000u), __double2loint(y));
}

// x c for a double x and a constant c > 0, given as a UF within 2^+-100 and
// as a double; c's UF {0, 0} or an x far from 1 takes the FP64 product.
__device__ __forceinline__ double scale_d(double x, UF c, double cd) {
  const unsigned hi = (unsigned)__double2hiint(x);
  if ((hi >> 20 & 0x7FFu) - 128u >= 1790u || c.m == 0) return x * cd;
  const double y = to_double(mul(from_double(x), c));
  return __hiloint2double(__double2hiint(y) | (int)(hi & 0x80000000u), __double2loint(y));
}

}  // namespace fx
}  // namespace dccm
