// Signed 9-bit digits of FP64 values, the operand form of the FP64 Legendre
// contractions on the tensor cores (internal header).
//
// A vector of doubles with largest biased exponent E (all |a| < 2^(E-1022))
// is written in fixed point, Q = a 2^(1084-E) (|Q| <= 2^62, the 53-bit
// mantissas exact down to 2^-9 of the vector's largest binade and rounded
// at 2^-62 of it below), and Q in seven balanced digits of 9 bits,
//   a = 2^(E-1030) sum_{i=1..7} d_i 2^(-9 (i-1)),  |d_i| <= 256,
// every one an FP16 number exactly.  Products of digits are integers of at
// most 2^16, so FP32 accumulation of them is exact up to a sum of 2^24.
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

// Q of x for scale exponent E (at least that of the vector; 0 for an x beyond
// it), with 256 added to every digit so that they come off as plain bit fields.
__device__ __forceinline__ unsigned long long dg_fixed(double x, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ef = (int)(b >> 52) & 0x7FF;
  // the 53-bit mantissa at bits 10 .. 62, moved down by E - ef + 1, rounded
  const unsigned long long m = ((b << 10) & 0x3FFFFFFFFFFFFC00ull) | (ef ? 1ull << 62 : 0ull);
  const unsigned r = min((unsigned)(E - max(ef, 1)), 63u);  // at 63 nothing is left
  const unsigned long long q = ((m >> r) + 1ull) >> 1;
  constexpr unsigned long long BIAS =
      256ull * (1ull + (1ull << 9) + (1ull << 18) + (1ull << 27) + (1ull << 36) + (1ull << 45) + (1ull << 54));
  const unsigned long long s = (unsigned long long)((long long)b >> 63);
  return (q ^ s) + (BIAS - s);
}

__device__ __forceinline__ unsigned sub_f16x2(unsigned a, unsigned b) {
  unsigned r;
  asm("sub.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// The digits in bits 0 .. 8 (FIELD 0), 9 .. 17 (1) or 0 .. 9 (2, the leading
// digit) of two words as a pair of FP16 integers (a in the low half): the
// fields become the low mantissa bits of 1024 + u, or one bit higher of 512 +
// u, and the subtraction is exact.
template <int FIELD> __device__ __forceinline__ unsigned dg_pair(unsigned a, unsigned b) {
  if constexpr (FIELD == 1) return sub_f16x2((__byte_perm(a, b, 0x6521) & 0x03FE03FEu) | 0x60006000u, 0x62006200u);
  const unsigned mask = FIELD == 0 ? 0x01FF01FFu : 0x03FF03FFu;
  return sub_f16x2((__byte_perm(a, b, 0x5410) & mask) | 0x64006400u, 0x65006500u);
}

// The seven slices of eight values of one row (consecutive along K): one
// 16-byte store per slice, slices `stride` bytes apart.
__device__ __forceinline__ void dg_store8(unsigned char *dst, size_t stride, const unsigned long long (&q)[8]) {
  unsigned w[8];
  auto put = [&](int i, auto pair) {
    *reinterpret_cast<uint4 *>(dst + i * stride) =
        make_uint4(pair(w[0], w[1]), pair(w[2], w[3]), pair(w[4], w[5]), pair(w[6], w[7]));
  };
  auto low = [](unsigned a, unsigned b) { return dg_pair<0>(a, b); };
  auto high = [](unsigned a, unsigned b) { return dg_pair<1>(a, b); };
  auto top = [](unsigned a, unsigned b) { return dg_pair<2>(a, b); };
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = (unsigned)(q[e] >> 54);
  put(0, top);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = (unsigned)(q[e] >> 36);
  put(1, high);
  put(2, low);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = (unsigned)(q[e] >> 18);
  put(3, high);
  put(4, low);
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = (unsigned)q[e];
  put(5, high);
  put(6, low);
}

// Sum of drained accumulators (levels s = 2 .. 8 of digit products, 2 .. 5
// integers below 2^24): t in units of level 6 (2^18 level-8 units), the rest below in
// FP32 (its 24 bits reach 2^-61 of the largest product).
// 1.01 K 2^52 < 2^62 for K products: K < 1,000.
struct DgSum {
  long long t;
  float l;
};
// Conversions to integers are the limit here (one warp instruction in eight
// cycles), so levels 4 and 6 hand their multiples of 512 to the level above
// in FP32, exactly, and only what is left, |.| <= 256, goes to the level
// below: three conversions in place of five.
__device__ __forceinline__ void dg_accumulate(DgSum &x, const unsigned (&r)[DG_SLICES]) {
  constexpr float M = 1.5f * 4294967296.f;  // 2^32: rounds to multiples of 512
  float v[DG_SLICES];
#pragma unroll
  for (int s = 0; s < DG_SLICES; ++s) v[s] = __uint_as_float(r[s]);
  const float h2 = __fadd_rn(__fadd_rn(v[2], M), -M), h4 = __fadd_rn(__fadd_rn(v[4], M), -M);
  const float l2 = __fadd_rn(v[2], -h2), l4 = __fadd_rn(v[4], -h4);
  const int i0 = __float2int_rn(v[0]);
  const int i1 = __float2int_rn(fmaf(h2, 1.f / 512.f, v[1]));
  const int i3 = __float2int_rn(fmaf(l2, 512.f, fmaf(h4, 1.f / 512.f, v[3])));
  x.t += (long long)i3 * (1 << 9);
  x.t += (long long)i1 * (1 << 27);
  x.t += (long long)i0 << 36;
  x.l = fmaf(l4, 262144.f, fmaf(v[5], 512.f, x.l)) + v[6];
}
// x 2^k in whole level-6 units, 0 <= k <= 10 and x 2^k within range
__device__ __forceinline__ long long dg_sum_fixed(const DgSum &x, int k) {
  return (x.t << k) + __float2int_rn(x.l * __int_as_float((k + 109) << 23));  // l 2^(k - 18)
}

// q 2^ex as the nearest double (ties away from zero).
__device__ __forceinline__ double fixed_to_double(long long q, int ex) {
  const long long s = q >> 63;
  unsigned long long m = (unsigned long long)((q ^ s) - s);
  const int z = __clzll((long long)m);
  if (m == 0) return 0.0;
  m <<= z;
  const unsigned long long mant = (m >> 11) + ((unsigned)m >> 10 & 1u);  // 53 bits, or 2^53
  const int be = ex + 63 - z + 1023;
  if ((unsigned)(be - 1) >= 2045u) {  // subnormal result or overflow
    if (be < -60) return __longlong_as_double((long long)((unsigned long long)s << 63));
    const double r = ldexp((double)mant, be - 1075);
    return s ? -r : r;
  }
  return __longlong_as_double((long long)((((unsigned long long)(unsigned)(be - 1) << 52) + mant) |
                                          ((unsigned long long)s << 63)));
}

// The same where every result is normal or zero: FIXED_EX_MIN <= ex <=
// FIXED_EX_MAX (no branch).
constexpr int FIXED_EX_MIN = -1022, FIXED_EX_MAX = 959;
__device__ __forceinline__ double fixed_to_double_normal(long long q, int ex) {
  const long long s = q >> 63;
  unsigned long long m = (unsigned long long)((q ^ s) - s);
  const int z = __clzll((long long)(m | 1));
  m <<= z;
  const unsigned long long mant = (m >> 11) + ((unsigned)m >> 10 & 1u);
  const unsigned hi = (unsigned)(mant >> 32) + ((unsigned)(ex + 1085 - z) << 20) + (unsigned)(s << 31);
  return __hiloint2double(q ? (int)hi : 0, (int)(unsigned)mant);
}

}  // namespace dccm
