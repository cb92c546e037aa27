// Longitude FFT of the FP64 path, in 64-bit block fixed point on the
// integer pipes.
//
// The FP64 pipe of this GPU issues one warp instruction in 64 cycles, and a
// 1024-point transform of a row pair takes about 36,000 FP64 operations (a
// shared-memory Stockham transform in FP64 ran T341 x 192 field-levels in
// 5.2 ms either way, T85 x 128 in 131 / 147 us).  In fixed point an addition
// is two integer instructions and is exact, and a product with a 62-bit
// twiddle takes three 32 x 32 -> 64 bit multiply-adds, all on full-rate
// pipes.
//
// Rows pair up as in fft.cu: z = g(jn) + i g(js), one complex transform of
// length I = R1 R2 (R3) by T = I / R1 threads.  A row pair has one scale:
//   forward  the largest magnitude of the pair sits at 2^CB; every pass
//            of radix R is followed by its twiddles times 2^-ceil(log2 R)
//            (12: times 2/3 2^-3), so nothing overflows (|Z| <= sum |z|) and
//            a pass rounds once, below 2^-53 of the row's r.m.s. for
//            noise-like rows and below 2^-52 for a single value;
//   inverse  every partial sum of the transform is bounded by the sum S of
//            the input magnitudes, so the inputs are scaled with S at 2^62
//            and no pass scales: roundings are a few 2^-62 S.
// Both are below the rounding errors of an FP64 transform (about 2.5e-16 of
// the r.m.s.; measured errors of the whole transforms fell, see the tests).
// A row pair that holds an infinity or NaN comes out NaN.
//
// Passes are in place: forward decimation in frequency (radix-R DFT in
// registers over stride N / R, twiddles), leaving frequency f = p1 + R1 p2 +
// R1 R2 p3 at position p1 N1 + p2 N2 + p3; inverse the same passes
// mirrored, from that order to natural order.  Positions are padded by one
// in every last radix and one in every N1, so that the passes' 16-byte
// accesses and the reads by frequency are free of bank conflicts.  A CTA
// takes BB field-levels of one latitude pair, so that F and G are read and
// written in runs of 16 BB bytes.
#include <math.h>
#include <string.h>

#include "digits.cuh"
#include "sht_plan.cuh"

namespace dccm {
namespace sht {
namespace f64 {

struct C64 {
  long long x, y;
};
__device__ __forceinline__ C64 operator+(C64 a, C64 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ C64 operator-(C64 a, C64 b) { return {a.x - b.x, a.y - b.y}; }
// a times SG i
template <int SG> __device__ __forceinline__ C64 muli(C64 a) {
  return SG > 0 ? C64{-a.y, a.x} : C64{a.y, -a.x};
}

// z w for a twiddle in 64-bit fixed point, w = (x 2^32 + y, z 2^32 + w) with
// signed low words: (z W) >> (32 + SH), rounded to nearest.  The product of
// the two low words (below 2^-2 of the result's last place) is left out.
template <int SH> __device__ __forceinline__ C64 twmul(C64 a, int4 w) {
  const int xl = (int)a.x, xh = (int)(a.x >> 32) + ((unsigned)xl >> 31);
  const int yl = (int)a.y, yh = (int)(a.y >> 32) + ((unsigned)yl >> 31);
  const int ns = -w.z, nt = -w.w;
  constexpr long long HALF = 1ll << (SH - 1);
  long long m = (long long)xh * w.y + HALF;
  m += (long long)xl * w.x;
  m += (long long)yh * nt;
  m += (long long)yl * ns;
  long long r = (m >> 32) + (long long)xh * w.x;
  r += (long long)yh * ns;
  long long n = (long long)xh * w.w + HALF;
  n += (long long)xl * w.z;
  n += (long long)yh * w.y;
  n += (long long)yl * w.x;
  long long s = (n >> 32) + (long long)xh * w.z;
  s += (long long)yh * w.x;
  if constexpr (SH == 32) return {r, s};
  else return {(r << (32 - SH)) | ((unsigned)m >> SH), (s << (32 - SH)) | ((unsigned)n >> SH)};
}
// x c for a constant |c| <= 1 given as (hi, lo) words of c 2^62
__device__ __forceinline__ long long cmulr(long long x, int ch, int cl) {
  const int xl = (int)x, xh = (int)(x >> 32) + ((unsigned)xl >> 31);
  long long m = (long long)xh * cl + (1ll << 29);
  m += (long long)xl * ch;
  const long long r = (m >> 32) + (long long)xh * ch;
  return (r << 2) | ((unsigned)m >> 30);
}

// cos(pi/4), cos(pi/8), sin(pi/8), sin(pi/3) times 2^62 as a signed low word
// and the rest
#define DCCM_FX(name, v)                                            \
  constexpr int name##_L = (int)(unsigned)((unsigned long long)(v)); \
  constexpr int name##_H = (int)(((v) + 0x80000000ll) >> 32)
DCCM_FX(RH, 3260954456333195553ll);
DCCM_FX(C8, 4260642322793532497ll);
DCCM_FX(S8, 1764815834521887442ll);
DCCM_FX(Q3, 3993837246235628775ll);
#undef DCCM_FX

__device__ __forceinline__ C64 mulc(C64 a, int ch, int cl, int sh, int sl) { return twmul<30>(a, make_int4(ch, cl, sh, sl)); }
// a e^{SG i pi/4}, a e^{SG 3 i pi/4}
template <int SG> __device__ __forceinline__ C64 rot1(C64 a) {
  const C64 b = SG > 0 ? C64{a.x - a.y, a.x + a.y} : C64{a.x + a.y, a.y - a.x};
  return {cmulr(b.x, RH_H, RH_L), cmulr(b.y, RH_H, RH_L)};
}
template <int SG> __device__ __forceinline__ C64 rot3(C64 a) { return muli<SG>(rot1<SG>(a)); }

template <int SG> __device__ __forceinline__ void dft4(C64 &a, C64 &b, C64 &c, C64 &d) {
  const C64 s0 = a + c, d0 = a - c, s1 = b + d, d1 = muli<SG>(b - d);
  a = s0 + s1;
  b = d0 + d1;
  c = s0 - s1;
  d = d0 - d1;
}
template <int SG> __device__ __forceinline__ void dft3(C64 &a, C64 &b, C64 &c) {
  const C64 t = b + c, u = muli<SG>(b - c);
  const C64 m = {a.x - (t.x >> 1), a.y - (t.y >> 1)};
  const C64 q = {cmulr(u.x, Q3_H, Q3_L), cmulr(u.y, Q3_H, Q3_L)};
  a = a + t;
  b = m + q;
  c = m - q;
}

// v[p] = sum_q v[q] e^{SG 2 pi i p q / R}
template <int SG, int R> __device__ __forceinline__ void dft(C64 (&v)[R]) {
  if constexpr (R == 4) {
    dft4<SG>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {  // 2 x 4: even and odd q, then radix 2 over them
    dft4<SG>(v[0], v[2], v[4], v[6]);
    dft4<SG>(v[1], v[3], v[5], v[7]);
    const C64 o1 = rot1<SG>(v[3]), o2 = muli<SG>(v[5]), o3 = rot3<SG>(v[7]);
    const C64 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = e0 + o0;
    v[4] = e0 - o0;
    v[1] = e1 + o1;
    v[5] = e1 - o1;
    v[2] = e2 + o2;
    v[6] = e2 - o2;
    v[3] = e3 + o3;
    v[7] = e3 - o3;
  } else if constexpr (R == 16) {  // 4 x 4
#pragma unroll
    for (int q = 0; q < 4; ++q) dft4<SG>(v[q], v[q + 4], v[q + 8], v[q + 12]);
    // v[q + 4 a]: twiddle e^{SG 2 pi i a q / 16}
    const int S = SG;
    v[5] = mulc(v[5], C8_H, C8_L, S * S8_H, S * S8_L);
    v[6] = rot1<SG>(v[6]);
    v[7] = mulc(v[7], S8_H, S8_L, S * C8_H, S * C8_L);
    v[9] = rot1<SG>(v[9]);
    v[10] = muli<SG>(v[10]);
    v[11] = rot3<SG>(v[11]);
    v[13] = mulc(v[13], S8_H, S8_L, S * C8_H, S * C8_L);
    v[14] = rot3<SG>(v[14]);
    v[15] = mulc(v[15], -C8_H, -C8_L, -S * S8_H, -S * S8_L);
#pragma unroll
    for (int a = 0; a < 4; ++a) dft4<SG>(v[4 * a], v[4 * a + 1], v[4 * a + 2], v[4 * a + 3]);
    // output p = a + 4 b is at v[4 a + b]
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = a + 1; b < 4; ++b) {
        const C64 t = v[4 * a + b];
        v[4 * a + b] = v[4 * b + a];
        v[4 * b + a] = t;
      }
  } else {  // R == 12: coprime factors 3 x 4 (Good's mapping), no twiddles
    static_assert(R == 12);
    C64 u[3][4];
    // q = 4 a + 3 b (mod 12)
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) u[a][b] = v[(4 * a + 3 * b) % 12];
#pragma unroll
    for (int b = 0; b < 4; ++b) dft3<SG>(u[0][b], u[1][b], u[2][b]);
#pragma unroll
    for (int a = 0; a < 3; ++a) dft4<SG>(u[a][0], u[a][1], u[a][2], u[a][3]);
    // p = A (mod 3), B (mod 4) with e^{2 pi i p (4 a + 3 b) / 12} = e^{2 pi i p a / 3} e^{2 pi i p b / 4}
#pragma unroll
    for (int p = 0; p < 12; ++p) v[p] = u[p % 3][p % 4];
  }
}

constexpr int clog2(int r) { return r <= 1 ? 0 : r <= 2 ? 1 : r <= 4 ? 2 : r <= 8 ? 3 : 4; }

template <int I_, int R1_, int R2_, int R3_> struct Shape {
  static constexpr int I = I_, R1 = R1_, R2 = R2_, R3 = R3_;
  static constexpr int N1 = I / R1, N2 = N1 / R2;  // N2 = R3
  static constexpr int T = N1;                     // threads a row pair
  static constexpr int RL = R3 > 1 ? R3 : R2;      // last radix
  // forward: bits that a pass scales down by (R1 = 12: with the 2/3 of 1/I)
  static constexpr int S1 = R1 == 12 ? 3 : clog2(R1), S2 = R3 > 1 ? clog2(R2) : 0;
  // forward: components of the input at most (1 - 2^-53) 2^CB, so that R1 2^(CB +
  // 1/2) and the fold of four results of the last pass, 4 RL (1 - 2^-53) 2^CB
  // and a few units of rounding, stay below 2^63
  static constexpr int CB = 61 - clog2(RL) < 58 ? 61 - clog2(RL) : 58;
  static constexpr int THREADS = T >= 64 ? 256 : 128;
  static constexpr int BB = THREADS / T;
  // CTAs of an SM: eight points a thread fit 80 registers, 12 or 16 take 128
  static constexpr int MINB = (R1 == 8 && R3 > 1 ? 768 : 512) / THREADS;
  static __host__ __device__ constexpr int at(int a) { return a + a / RL + (R3 > 1 ? a / N1 : 0); }
  // stride of the row pairs' buffers, 2 (mod 8) 16-byte units
  static constexpr int LD = (at(I - 1) + 1 + 7) / 8 * 8 + 2;
  static constexpr int TW = (R1 - 1) * N1 + (R3 > 1 ? (R2 - 1) * N2 : 0);  // twiddles of a direction
  static __device__ __forceinline__ int pos(int f) {                       // position of frequency f
    const int p1 = f % R1, r = f / R1;
    return at(p1 * N1 + (r % R2) * N2 + r / R2);
  }
};

// lanes of this thread's row pair (T <= 32)
template <int T> __device__ __forceinline__ unsigned group_mask() {
  if constexpr (T >= 32) return 0xffffffffu;
  else return ((1u << T) - 1u) << (threadIdx.x % 32 / T * T);
}
template <int T> __device__ __forceinline__ void group_sync(int g) {
  if constexpr (T <= 32) __syncwarp(group_mask<T>());
  else asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "n"(T) : "memory");
}

__device__ __forceinline__ unsigned mag(double x) { return (unsigned)__double2hiint(x) & 0x7FFFFFFFu; }

// x 2^k as an integer, k = sh + 1075 - (exponent of the row), given as
// r = 10 - (shift of the 53-bit mantissa): (mantissa 2^10) >> (r - ef), rounded.
__device__ __forceinline__ long long to_fixed(double x, int rbase) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int ef = (int)(b >> 52) & 0x7FF;
  const unsigned long long m = ((b << 10) & 0x3FFFFFFFFFFFFC00ull) | (ef ? 1ull << 62 : 0ull);
  int r = rbase - (ef ? ef : 1);
  r = r > 64 ? 64 : r;  // at 64 nothing is left
  const long long q = (long long)(((m >> (r - 1)) + 1) >> 1);
  return (long long)b < 0 ? -q : q;
}

// One in-place pass over the buffer of a row pair: DFTs of radix R over
// stride NS within blocks of R NS.  SG < 0: DFT, then twiddles (scaled);
// SG > 0: twiddles, then DFT.
template <class Sh, int SG, int R, int NS, int SHIFT>
__device__ __forceinline__ void pass(C64 *z, const int4 *__restrict__ tw, int t) {
#pragma unroll
  for (int d0 = 0; d0 < Sh::I / R; d0 += Sh::T) {
    const int d = d0 + t;
    if ((Sh::I / R) % Sh::T != 0 && d >= Sh::I / R) break;
    const int k = d % NS, base = (d / NS) * (R * NS) + k;
    C64 v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = z[Sh::at(base + q * NS)];
    if (NS > 1 && SG > 0) {
#pragma unroll
      for (int q = 1; q < R; ++q) v[q] = twmul<SHIFT>(v[q], __ldg(tw + (q - 1) * NS + k));
    }
    dft<SG, R>(v);
    if (NS > 1 && SG < 0) {
      // the p = 0 output has twiddle 1: the same scaling by a rounded shift
      constexpr int s = clog2(R);
      v[0] = {(v[0].x + (1ll << (s - 1))) >> s, (v[0].y + (1ll << (s - 1))) >> s};
#pragma unroll
      for (int p = 1; p < R; ++p) v[p] = twmul<SHIFT>(v[p], __ldg(tw + (p - 1) * NS + k));
    }
#pragma unroll
    for (int p = 0; p < R; ++p) z[Sh::at(base + p * NS)] = v[p];
  }
}

template <class Sh>
__global__ void __launch_bounds__(Sh::THREADS, Sh::MINB)
fft_forward_kernel(int N, int J, int batch, const double *__restrict__ grid, double *__restrict__ G,
                   const int4 *__restrict__ tw, int4 w0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C64 *buf = reinterpret_cast<C64 *>(smem_raw);
  __shared__ unsigned smx[Sh::BB][2];
  __shared__ int sE[Sh::BB];
  const int Jh = J / 2, jj = blockIdx.x % Jh, jn = Jh + jj, js = Jh - 1 - jj;
  const int b0 = blockIdx.x / Jh * Sh::BB, nb = min(Sh::BB, batch - b0);
  const int g = threadIdx.x / Sh::T, t = threadIdx.x % Sh::T;  // row pair, thread of it
  C64 *z = buf + (size_t)g * Sh::LD;
  pdl_wait();
  pdl_trigger();
  if (g < nb) {
    const double *gn = grid + ((int64_t)(b0 + g) * J + jn) * Sh::I + t;
    const double *gs = grid + ((int64_t)(b0 + g) * J + js) * Sh::I + t;
    double a[Sh::R1], b[Sh::R1];
#pragma unroll
    for (int q = 0; q < Sh::R1; ++q) {
      a[q] = __ldg(gn + q * Sh::N1);
      b[q] = __ldg(gs + q * Sh::N1);
    }
    unsigned mx = 0;
#pragma unroll
    for (int q = 0; q < Sh::R1; ++q) mx = max(mx, max(mag(a[q]), mag(b[q])));
#pragma unroll
    for (int o = (Sh::T < 32 ? Sh::T : 32) / 2; o > 0; o >>= 1)
      mx = max(mx, __shfl_xor_sync(group_mask<Sh::T>(), mx, o));
    if constexpr (Sh::T > 32) {
      if (t % 32 == 0) smx[g][t / 32] = mx;
      group_sync<Sh::T>(g);
      mx = max(smx[g][0], smx[g][1]);
    }
    const int E = max((int)(mx >> 20), 1);
    if (t == 0) sE[g] = E;
    // |x| < 2^(E - 1022) -> 2^CB: the mantissa moves by CB - 53 + ef - E
    const int rb = 10 - (Sh::CB - 53) + E;
    C64 v[Sh::R1];
#pragma unroll
    for (int q = 0; q < Sh::R1; ++q) v[q] = {to_fixed(a[q], rb), to_fixed(b[q], rb)};
    dft<-1, Sh::R1>(v);
    v[0] = twmul<32>(v[0], w0);
#pragma unroll
    for (int p = 1; p < Sh::R1; ++p) v[p] = twmul<32>(v[p], __ldg(tw + (p - 1) * Sh::N1 + t));
#pragma unroll
    for (int p = 0; p < Sh::R1; ++p) z[Sh::at(p * Sh::N1 + t)] = v[p];
    group_sync<Sh::T>(g);
    pass<Sh, -1, Sh::R2, Sh::N2, 32>(z, tw + (Sh::R1 - 1) * Sh::N1, t);
    if constexpr (Sh::R3 > 1) {
      group_sync<Sh::T>(g);
      pass<Sh, -1, Sh::R3, 1, 32>(z, nullptr, t);
    }
  }
  __syncthreads();
  // results: E = A + B, O = A - B of the rows' spectra A, B, field-levels fastest
  constexpr bool THREE = Sh::I % 3 == 0;  // the twiddles carry 2/3
  const int bl = threadIdx.x % Sh::BB;
  if (bl >= nb) return;
  const C64 *zb = buf + (size_t)bl * Sh::LD;
  const int E = sE[bl];
  // value = q 2^ex: row scale, pass scalings, the halves of A and B, and 1/I
  constexpr int LI = THREE ? clog2(Sh::I / 96) + 5 + 1 : clog2(Sh::I / 64) + 6;
  const int ex = E - 1022 - Sh::CB + Sh::S1 + Sh::S2 - 1 - LI;
  const int64_t C2B = 2LL * batch;
  double2 *out = reinterpret_cast<double2 *>(G + (int64_t)jj * C2B + 2 * (b0 + bl));
  const int64_t pst = (int64_t)Jh * batch;  // one parity of one m, in double2
  const double nan = __longlong_as_double(0x7FF8000000000000ll);
  const bool normal = E < 2047 && ex >= FIXED_EX_MIN && ex <= FIXED_EX_MAX;
  for (int m = threadIdx.x / Sh::BB; m <= N; m += Sh::T) {
    const C64 a = zb[Sh::pos(m)], c = zb[Sh::pos(m ? Sh::I - m : 0)];
    // 2A = (a.x + c.x, a.y - c.y), 2B = (a.y + c.y, c.x - a.x)
    const long long ar = a.x + c.x, ai = a.y - c.y, br = a.y + c.y, bi = c.x - a.x;
    double2 e, o;
    if (normal) {
      e = make_double2(fixed_to_double_normal(ar + br, ex), fixed_to_double_normal(ai + bi, ex));
      o = make_double2(fixed_to_double_normal(ar - br, ex), fixed_to_double_normal(ai - bi, ex));
    } else {  // results that may be subnormal or infinite, or NaN
      e = make_double2(fixed_to_double(ar + br, ex), fixed_to_double(ai + bi, ex));
      o = make_double2(fixed_to_double(ar - br, ex), fixed_to_double(ai - bi, ex));
      if (E >= 2047) e = o = make_double2(nan, nan);
    }
    if (m == 0) e.y = o.y = 0.0;
    out[(int64_t)(2 * m) * pst] = e;
    out[(int64_t)(2 * m + 1) * pst] = o;
  }
}

template <class Sh>
__global__ void __launch_bounds__(Sh::THREADS, Sh::MINB)
fft_inverse_kernel(int N, int J, int batch, const double *__restrict__ F, double *__restrict__ grid,
                   const int4 *__restrict__ tw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C64 *buf = reinterpret_cast<C64 *>(smem_raw);
  __shared__ unsigned smx[Sh::BB], ssum[Sh::BB];
  const int Jh = J / 2, jj = blockIdx.x % Jh, jn = Jh + jj, js = Jh - 1 - jj;
  const int b0 = blockIdx.x / Jh * Sh::BB, nb = min(Sh::BB, batch - b0);
  if (threadIdx.x < Sh::BB) smx[threadIdx.x] = ssum[threadIdx.x] = 0;
  __syncthreads();
  pdl_wait();
  pdl_trigger();
  // Fourier coefficients (m, field-level), field-levels fastest
  constexpr int KI = Sh::R1 / 2;  // N + 1 <= I / 2
  const int bl = threadIdx.x % Sh::BB, m0 = threadIdx.x / Sh::BB;
  const int64_t C2B = 2LL * batch;
  C64 *zb = buf + (size_t)bl * Sh::LD;
  double2 a[KI], b[KI];
#pragma unroll
  for (int i = 0; i < KI; ++i) {
    const int m = m0 + i * Sh::T;
    a[i] = b[i] = make_double2(0.0, 0.0);
    if (bl < nb && m <= N) {
      const double *f = F + (int64_t)m * J * C2B + 2 * (b0 + bl);
      a[i] = __ldg(reinterpret_cast<const double2 *>(f + jn * C2B));
      b[i] = __ldg(reinterpret_cast<const double2 *>(f + js * C2B));
      if (m == 0) a[i].y = b[i].y = 0.0;
    }
  }
  // their bits wait in the positions of m and I - m (frequencies above N hold
  // zeros, the same in either form; I / 2, never used as N < I / 2, stands in
  // for m = 0's).  The two passes over them are loops: with the values in
  // registers and both unrolled the kernel outgrew the instruction cache (3.5
  // of 8 cycles an instruction waited for code; T85 x 128 took 48 us, now 34,
  // T42 x 104 15, now 12)
  unsigned mx = 0;
#pragma unroll
  for (int i = 0; i < KI; ++i) {
    const int m = m0 + i * Sh::T;
    mx = max(max(mx, max(mag(a[i].x), mag(a[i].y))), max(mag(b[i].x), mag(b[i].y)));
    zb[Sh::pos(m)] = {__double_as_longlong(a[i].x), __double_as_longlong(a[i].y)};
    zb[Sh::pos(m ? Sh::I - m : Sh::I / 2)] = {__double_as_longlong(b[i].x), __double_as_longlong(b[i].y)};
  }
  atomicMax(&smx[bl], mx);
  __syncthreads();
  const int E = max((int)(smx[bl] >> 20), 1);
  // sum of the magnitudes in units of 2^(E - 1022 - 20), rounded up: each as
  // FP32 relative to 2^(E - 1023) (20 bits of its mantissa), a thread's sum
  // with a margin above those and the sums' rounding errors
  const int nm = (N + Sh::T) / Sh::T;  // m0 + i T <= N needs i < nm
  const int hb = (E - 127) * (1 << 20);
  auto rel = [&](long long x) {
    return __int_as_float(max(((int)(x >> 32) & 0x7FFFFFFF) - hb, 0) << 3);
  };
  float sum = 0.f;
#pragma unroll 2
  for (int i = 0; i < nm; ++i) {
    const int m = m0 + i * Sh::T;
    const C64 u = zb[Sh::pos(m)], w = zb[Sh::pos(m ? Sh::I - m : Sh::I / 2)];
    sum += (rel(u.x) + rel(u.y)) + (rel(w.x) + rel(w.y));
  }
  atomicAdd(&ssum[bl], __float2uint_ru(sum * (524288.f + 8.f)) + 1u);
  __syncthreads();
  // sum of |Re Z| + |Im Z| over all frequencies < 2^(nbit + 1) units -> 2^62:
  // the mantissa moves by ef - E + 28 - nbit
  const int nbit = 32 - __clz((int)ssum[bl]);
  const int rb = 10 - (28 - nbit) + E;
#pragma unroll 2
  for (int i = 0; i < nm; ++i) {
    const int m = m0 + i * Sh::T;
    C64 &zm = zb[Sh::pos(m)], &zi = zb[Sh::pos(m ? Sh::I - m : Sh::I / 2)];
    const C64 u = zm, w = zi;
    const long long ar = to_fixed(__longlong_as_double(u.x), rb), ai = to_fixed(__longlong_as_double(u.y), rb);
    const long long br = to_fixed(__longlong_as_double(w.x), rb), bi = to_fixed(__longlong_as_double(w.y), rb);
    zm = {ar - bi, ai + br};
    zi = m ? C64{ar + bi, br - ai} : C64{0, 0};
  }
  __syncthreads();
  const int g = threadIdx.x / Sh::T, t = threadIdx.x % Sh::T;
  if (g >= nb) return;
  C64 *z = buf + (size_t)g * Sh::LD;
  if constexpr (Sh::R3 > 1) {
    pass<Sh, 1, Sh::R3, 1, 30>(z, nullptr, t);
    group_sync<Sh::T>(g);
  }
  pass<Sh, 1, Sh::R2, Sh::N2, 30>(z, tw + (Sh::R1 - 1) * Sh::N1, t);
  group_sync<Sh::T>(g);
  C64 v[Sh::R1];
#pragma unroll
  for (int q = 0; q < Sh::R1; ++q) v[q] = z[Sh::at(q * Sh::N1 + t)];
#pragma unroll
  for (int q = 1; q < Sh::R1; ++q) v[q] = twmul<30>(v[q], __ldg(tw + (q - 1) * Sh::N1 + t));
  dft<1, Sh::R1>(v);
  const int Eg = max((int)(smx[g] >> 20), 1);
  const int ex = Eg - 1075 - (28 - (32 - __clz((int)ssum[g])));
  double *gn = grid + ((int64_t)(b0 + g) * J + jn) * Sh::I + t;
  double *gs = grid + ((int64_t)(b0 + g) * J + js) * Sh::I + t;
  if (Eg < 2047 && ex >= FIXED_EX_MIN && ex <= FIXED_EX_MAX) {
#pragma unroll
    for (int p = 0; p < Sh::R1; ++p) {
      gn[p * Sh::N1] = fixed_to_double_normal(v[p].x, ex);
      gs[p * Sh::N1] = fixed_to_double_normal(v[p].y, ex);
    }
  } else {  // results that may be subnormal or infinite, or NaN
    const double nan = __longlong_as_double(0x7FF8000000000000ll);
#pragma unroll
    for (int p = 0; p < Sh::R1; ++p) z[Sh::at(p * Sh::N1 + t)] = v[p];
#pragma unroll 1
    for (int p = 0; p < Sh::R1; ++p) {
      const C64 u = z[Sh::at(p * Sh::N1 + t)];
      gn[p * Sh::N1] = Eg >= 2047 ? nan : fixed_to_double(u.x, ex);
      gs[p * Sh::N1] = Eg >= 2047 ? nan : fixed_to_double(u.y, ex);
    }
  }
}

// ------------------------------------------------------------------ host
// cos and sin of pi x / 4, 0 <= x <= 1 (x = num / den), as integers times
// 2^62, by Taylor series in 128-bit integers (error below 2^-61: the same
// table on every host).
static void octant(unsigned num, unsigned den, long long &c, long long &s) {
  typedef unsigned __int128 u128;
  // pi / 4 in 2^-96 units
  const u128 PI4 = ((u128)0xC90FDAA2ull << 64) | 0x2168C234C4C6628Bull;
  const u128 th = PI4 * num / den;  // num < 2^11: no overflow below 2^128
  const unsigned long long x = (unsigned long long)(th >> 32) + (unsigned long long)((th >> 31) & 1);  // 2^-64 units
  auto mul = [](unsigned long long a, unsigned long long b) { return (unsigned long long)(((u128)a * b + (1ull << 63)) >> 64); };
  const unsigned long long x2 = mul(x, x);
  // terms 1 - x^2/2 + ... and x - x^3/6 + ..., summed signed in 128 bits
  __int128 cs = (__int128)1 << 64, sn = x;
  unsigned long long tc = 0, ts = x;
  for (int k = 1; k <= 14; ++k) {
    tc = k == 1 ? x2 / 2 : mul(tc, x2) / (unsigned)((2 * k - 1) * (2 * k));
    ts = mul(ts, x2) / (unsigned)((2 * k) * (2 * k + 1));
    cs += (k & 1) ? -(__int128)tc : (__int128)tc;
    sn += (k & 1) ? -(__int128)ts : (__int128)ts;
  }
  c = (long long)((cs + 2) >> 2);
  s = (long long)((sn + 2) >> 2);
}
// e^{2 pi i t / I} times 2^62, from cos and sin of the first octant's I / 8 + 1
// angles (I is a multiple of 32).
struct Roots {
  int I;
  std::vector<long long> c, s;
  explicit Roots(int n) : I(n), c(n / 8 + 1), s(n / 8 + 1) {
    for (int k = 0; k <= n / 8; ++k) octant((unsigned)(8 * k), (unsigned)n, c[k], s[k]);
  }
  void get(int t, long long &x, long long &y) const {
    const int o = 8 * t / I, r = t - o * (I / 8);  // octant, remainder in 1/I of the circle
    long long a, b;
    if (o & 1) b = c[I / 8 - r], a = s[I / 8 - r];  // the octant's mirror image
    else a = c[r], b = s[r];
    switch (o / 2) {  // quadrant
      case 0: x = a; y = b; break;
      case 1: x = -b; y = a; break;
      case 2: x = -a; y = -b; break;
      default: x = b; y = -a; break;
    }
  }
};
static int4 words(long long c, long long s) {
  auto hi = [](long long v) { return (int)((v + 0x80000000ll) >> 32); };
  auto lo = [](long long v) {
    const int l = (int)(unsigned)(unsigned long long)v;
    return l == (int)0x80000000 ? l + 1 : l;  // its negative has to fit
  };
  return make_int4(hi(c), lo(c), hi(s), lo(s));
}
// v 2^-k, times 2/3 if three, rounded
static long long scaled(long long v, int k, bool three) {
  __int128 x = (__int128)v * (three ? 2 : 1);
  const __int128 d = ((__int128)1 << k) * (three ? 3 : 1);
  return (long long)(x >= 0 ? (x + d / 2) / d : -((-x + d / 2) / d));
}

// Three passes of eight points a thread where they can be had (us inverse /
// forward, against two of 16 or 16 first): T42 x 8 8.9 / 8.2 (9.9 / 10.2), T85 x
// 8 9.8 / 8.2 (11.9 / 10.2), T170 x 64 59 / 53 (67 / 55).  1024 points keep 16
// first, as four passes would be needed; 192 = 12 x 4 x 4 was no faster.
template <class F> static int with_shape(int I, F &&f) {
  switch (I) {
    case 64: return f(Shape<64, 8, 8, 1>());
    case 96: return f(Shape<96, 12, 8, 1>());
    case 128: return f(Shape<128, 8, 4, 4>());
    case 192: return f(Shape<192, 12, 16, 1>());
    case 256: return f(Shape<256, 8, 8, 4>());
    case 384: return f(Shape<384, 12, 8, 4>());
    case 512: return f(Shape<512, 8, 8, 8>());
    case 768: return f(Shape<768, 12, 8, 8>());
    case 1024: return f(Shape<1024, 16, 8, 8>());
    default: return DCCM_ERR_UNSUPPORTED;
  }
}

}  // namespace f64

// Twiddles of both directions: forward entries e^{-i theta} 2^(64 - s), such
// that twmul<32> scales by 2^-s, s = ceil(log2 R) (and by 2/3 in the first
// pass of lengths with a factor 3, the odd part of 1/I); inverse entries e^{+i
// theta} 2^62 for twmul<30>.
int build_fft_f64(Plan &P, std::vector<int4> &h) {
  using namespace f64;
  return with_shape(P.I, [&](auto sh) {
    using Sh = decltype(sh);
    h.assign(2 * Sh::TW + 1, int4());
    const bool three = Sh::I % 3 == 0;
    const Roots roots(Sh::I);
    for (int dir = 0; dir < 2; ++dir) {
      int4 *w = h.data() + dir * Sh::TW;
      auto fill = [&](int R, int NS, int scale, bool th) {
        for (int p = 1; p < R; ++p)
          for (int k = 0; k < NS; ++k) {
            long long c, s;
            roots.get(p * k * (Sh::I / (R * NS)), c, s);  // p k < R NS
            if (dir == 0) *w++ = words(scaled(c, scale - 2, th), scaled(-s, scale - 2, th));
            else *w++ = words(c, s);
          }
      };
      fill(Sh::R1, Sh::N1, Sh::S1, three);
      if (Sh::R3 > 1) fill(Sh::R2, Sh::N2, Sh::S2, false);
    }
    // the first pass's twiddle 1, scaled
    h[2 * Sh::TW] = words(scaled(1ll << 62, Sh::S1 - 2, three), 0);
    return DCCM_OK;
  });
}

int fft_inverse_f64(const Plan &P, int batch, const double *F, double *grid, cudaStream_t s) {
  if (batch <= 0) return DCCM_OK;
  return f64::with_shape(P.I, [&](auto sh) {
    using Sh = decltype(sh);
    const size_t smem = (size_t)Sh::BB * Sh::LD * sizeof(f64::C64);
    DCCM_CUDA(cudaFuncSetAttribute(f64::fft_inverse_kernel<Sh>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    DCCM_CUDA(launch_pdl(f64::fft_inverse_kernel<Sh>, dim3((unsigned)P.Jh * ((batch + Sh::BB - 1) / Sh::BB)), dim3(Sh::THREADS), smem,
                         s, P.N, P.J, batch, F, grid, P.d_twfx + Sh::TW));
    return DCCM_OK;
  });
}

int fft_forward_f64(const Plan &P, int batch, const double *grid, double *G, cudaStream_t s) {
  if (batch <= 0) return DCCM_OK;
  return f64::with_shape(P.I, [&](auto sh) {
    using Sh = decltype(sh);
    const size_t smem = (size_t)Sh::BB * Sh::LD * sizeof(f64::C64);
    DCCM_CUDA(cudaFuncSetAttribute(f64::fft_forward_kernel<Sh>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    DCCM_CUDA(launch_pdl(f64::fft_forward_kernel<Sh>, dim3((unsigned)P.Jh * ((batch + Sh::BB - 1) / Sh::BB)), dim3(Sh::THREADS), smem,
                         s, P.N, P.J, batch, grid, G, P.d_twfx, P.twfx0));
    return DCCM_OK;
  });
}

}  // namespace sht
}  // namespace dccm
