// Signed 9-bit digits of FP64 values, the operand form of the FP64 Legendre
// contractions on the tensor cores (internal header).
//
// A vector of doubles with largest biased exponent E (all |a| < 2^(E-1022))
// is written in fixed point, Q = a 2^(1084-E) (|Q| <= 2^62, the 53-bit
// mantissas exact down to 2^-9 of the vector's largest binade and rounded
// at 2^-62 of it below), and Q in seven balanced digits of 9 bits,
//   a = 2^(E-1030) sum_{i=1..7} d_i 2^(-9 (i-1)),  |d_i| <= 256,
// every one a BF16 number exactly.  Products of digits are integers of at
// most 2^16, so FP32 accumulation of up to 2^24 / 2^16 of them is exact.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dccm {

constexpr int DG_SLICES = 7;

// Biased exponent field of the larger magnitude, as the vector's scale:
// reduce the magnitudes' high words with max, then shift.
__device__ __forceinline__ unsigned dg_mag(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }
__device__ __forceinline__ int dg_exp(unsigned maxmag) {
  const int e = (int)(maxmag >> 20);
  return e < 1 ? 1 : e;
}

// Q of x for scale exponent E, with half of each lower digit's range added
// so that the digits come off as plain bit fields.
__device__ __forceinline__ unsigned long long dg_fixed(double x, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ef = (int)(b >> 52) & 0x7FF;
  const unsigned long long mant = (b & 0xFFFFFFFFFFFFFull) | (ef ? 0x10000000000000ull : 0ull);
  const int sh = 9 + (ef ? ef : 1) - E;  // <= 9
  unsigned long long q;
  if (sh >= 0) q = mant << sh;
  else q = sh < -60 ? 0ull : ((mant >> (-sh - 1)) + 1ull) >> 1;
  if ((long long)b < 0) q = 0ull - q;
  constexpr unsigned long long BIAS =
      256ull * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) + (1ull << 45));
  return q + BIAS;
}

// Digit i = 1..7 of a biased Q as an FP32 number (low 16 bits zero: BF16 exact).
template <int i> __device__ __forceinline__ float dg_digit(unsigned long long q) {
  if constexpr (i == 1) {
    const unsigned u = (unsigned)((int)(q >> 32) >> 22) & 1023u;  // signed, -256 .. 256 (mod 1024)
    return __uint_as_float(0x4B000000u | ((u + 512u) & 1023u)) - 8389120.f;
  } else {
    const unsigned u = (unsigned)(q >> (9 * (7 - i))) & 511u;
    return __uint_as_float(0x4B000000u | u) - 8388864.f;
  }
}

// Digit i of two values as one BF16 pair (a in the low half).
template <int i> __device__ __forceinline__ unsigned dg_pair(unsigned long long a, unsigned long long b) {
  return __byte_perm(__float_as_uint(dg_digit<i>(a)), __float_as_uint(dg_digit<i>(b)), 0x7632);
}

// The seven slices of eight values of one row (consecutive along K): one
// 16-byte store per slice, slices `stride` bytes apart.
template <int i = 1>
__device__ __forceinline__ void dg_store8(unsigned char *dst, size_t stride, const unsigned long long (&q)[8]) {
  *reinterpret_cast<uint4 *>(dst) =
      make_uint4(dg_pair<i>(q[0], q[1]), dg_pair<i>(q[2], q[3]), dg_pair<i>(q[4], q[5]), dg_pair<i>(q[6], q[7]));
  if constexpr (i < DG_SLICES) dg_store8<i + 1>(dst + stride, stride, q);
}

// 96-bit two's complement sum of drained accumulators.
struct Dg96 {
  unsigned w0, w1, w2;
};

// x += vh 2^36 + vl
__device__ __forceinline__ void dg_add(Dg96 &x, long long vh, long long vl) {
  const unsigned h0 = (unsigned)vh << 4, h1 = (unsigned)(vh >> 28);
  const unsigned l0 = (unsigned)vl, l1 = (unsigned)(vl >> 32), l2 = (unsigned)((int)l1 >> 31);
  asm("{\n\t.reg .u32 a, b;\n\t"
      "add.cc.u32 a, %4, %6;\n\t"
      "addc.u32 b, %5, %7;\n\t"
      "add.cc.u32 %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, a;\n\t"
      "addc.u32 %2, %2, b;\n\t}"
      : "+r"(x.w0), "+r"(x.w1), "+r"(x.w2)
      : "r"(l0), "r"(l1), "r"(l2), "r"(h0), "r"(h1));
}
__device__ __forceinline__ Dg96 dg_sum(const Dg96 &x, const Dg96 &y) {
  Dg96 r;
  asm("add.cc.u32 %0, %3, %6;\n\taddc.cc.u32 %1, %4, %7;\n\taddc.u32 %2, %5, %8;"
      : "=&r"(r.w0), "=&r"(r.w1), "=r"(r.w2)
      : "r"(x.w0), "r"(x.w1), "r"(x.w2), "r"(y.w0), "r"(y.w1), "r"(y.w2));
  return r;
}
__device__ __forceinline__ Dg96 dg_diff(const Dg96 &x, const Dg96 &y) {
  Dg96 r;
  asm("sub.cc.u32 %0, %3, %6;\n\tsubc.cc.u32 %1, %4, %7;\n\tsubc.u32 %2, %5, %8;"
      : "=&r"(r.w0), "=&r"(r.w1), "=r"(r.w2)
      : "r"(x.w0), "r"(x.w1), "r"(x.w2), "r"(y.w0), "r"(y.w1), "r"(y.w2));
  return r;
}

// x 2^ex as the nearest double (ties away from zero; bits below the top 64
// of x are dropped, 2^-11 of the result's last place).
__device__ __forceinline__ double dg_to_double(Dg96 x, int ex) {
  const unsigned sgn = x.w2 & 0x80000000u;
  if (sgn) x = dg_diff(Dg96{0, 0, 0}, x);
  int be = ex + 95 + 1023;  // biased exponent of bit 95
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (x.w2 == 0) {
      x.w2 = x.w1;
      x.w1 = x.w0;
      x.w0 = 0;
      be -= 32;
    }
  if (x.w2 == 0) return 0.0;
  const int z = __clz((int)x.w2);
  be -= z;
  const unsigned mh = __funnelshift_l(x.w1, x.w2, z), ml = __funnelshift_l(x.w0, x.w1, z);
  const unsigned long long mant = ((((unsigned long long)mh << 32) | ml) >> 11) + ((ml >> 10) & 1u);  // 53 bits, or 2^53
  if ((unsigned)(be - 1) >= 2045u) {  // subnormal result or overflow
    const double r = ldexp((double)mant, be - 1075);
    return sgn ? -r : r;
  }
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + mant;
  return __longlong_as_double((long long)(bits | ((unsigned long long)sgn << 32)));
}

}  // namespace dccm
