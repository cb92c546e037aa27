// FP64 Legendre transforms on the 5th-generation tensor cores (tcgen05),
// exact products of integer digits with the accuracy of FP64 arithmetic.
//
// The FP64 pipe of this GPU does one FMA for every 64 of the FP32 pipe
// (1.05 TFLOP/s measured), and the contraction took 80 % of the plain FP64
// transforms as an FP64 FMA loop (T341 x 192 field-levels: synthesis 10.4
// ms, analysis 13.5 ms; T85 x 128: 209 and 340 us; with the kernels below
// 0.53, 0.61 ms, 39 and 35 us, packs included).  Here every operand is
// split into seven 9-bit digits (digits.cuh: the scheme of K. Ozaki, T.
// Ogita, S. Oishi, S. Rump, "Error-free transformations of matrix
// multiplication", Numer. Algorithms 59 (2012), with integer digits), and
// the products d_i(a) d_j(b) of equal weight, s = i + j = 2 .. 8, are
// summed in one FP32 accumulator per s: integers below 2^24, so the sums
// are exact.  28 MMAs take the place of an FP64 FMA; the products left out
// (s >= 9) are below 2^-60 of (largest |a|) (largest |b|).  Errors are thus
// relative to the largest product of a contraction (one m, parity and
// field-level; synthesis: of the row of the table), where they are well under
// the rounding errors of an FP64 sum; a result far smaller than that has fewer
// correct digits than an FP64 sum of its own products would give it.
//
// Exactness: an accumulator takes at most 96 values of K (DG_KB chunks) before
// it is drained, so levels s = 2 and 3 (one and two products of at most 2^16 a
// value) stay within 2^24 whatever the tables, and levels 4 and 5 whatever the
// data, by the digits that the tables have (0.94 of 2^24 at most; with 128
// values level 5 could reach 1.2: a unit of it is 2^-43 of the largest product.
// A drain more an item of the T341 analysis: 2,597 -> 2,612 us both ways); from
// level 6 on (below 2^-52 of the largest product) a rounding would not be seen.
//
// As the mixed path (legendre_tc.cu) the contractions run per zonal
// wavenumber m and parity p (n - m even / odd), folded by equatorial symmetry:
//   inverse  D_p[c][jj] = sum_k S_p[c][k] Pbar_p[jj][k],
//            F(jn) = D_0 + D_1, F(js) = D_0 - D_1 (added as integers);
//   forward  D_p[c][k]  = sum_jj X_p[c][jj] ((w/2) Pbar)_p[k][jj],
//            X and the table with a power of two per latitude (dg_fwd_scales).
//
// Both operands lie in global memory as the shared-memory image of a tile
// (K-major rows of 32 values = 64 bytes, 64-byte swizzle), so that a stage
// is filled by a few untiled bulk copies:
//   A  [ct][chunk][7][128 rows c][32], written by the pack kernels, chunk =
//      32 values of K of one (m, p);
//   B  [m][p][nt][q][7][rows][32], built once per plan.
// The digit slices of B lie one after the other in the image, so one MMA
// multiplies slice i of A with several consecutive slices j of B (N = rows
// x slices, up to 256 columns), whose results fall into consecutive
// accumulators s = i + j: a slice of A is read from shared memory once for
// all of them.
//
// What bounds it at T341 x 192: the packs take 100 and 240 us (the analysis
// pack moves 1.5 GB), the rest is shared memory: a K step of 16 reads 28 KB of
// A's slices and 28 KB of B's for its 7 MMAs of 32 to 224 columns and is
// written 35 KB by the copies, 710 cycles at 128 bytes a cycle against 450 of
// MMAs at the peak rate; clock stamps show the MMAs of two steps issued in
// 1,360 cycles, and 2,000 with the drains beside them.  TN = 64 (half the
// reads of A, but one accumulator set, whose drains the MMAs then wait for)
// is 3 % slower there and 16 % at T85.  At T85 and below an item is latency:
// the loads 0.7 us, a chunk's MMAs 0.6, draining a set 0.8, the results 2-3.
//
// A work item is (m, 128 columns c, TN rows of N).  Warp 0 copies, warp 1
// allocates TMEM and issues the MMAs, warps 2-17 drain the accumulators
// (7 TMEM columns an output, integer arithmetic, one store).  Every wait is
// bounded, as in legendre_tc.cu.
#include <math.h>
#include <string.h>

#include "digits.cuh"
#include "sht_plan.cuh"
#include "tcgen05.cuh"

namespace dccm {
namespace sht {

constexpr int DG_CHUNK = 32;                                   // K of a stage
constexpr int DG_KB = 3;                                       // chunks an accumulator takes (96 values of K)
constexpr int DG_ROW = 2 * DG_CHUNK;                           // bytes of a K-major row of a chunk
constexpr int DG_A_SLICE = 128 * DG_ROW;                       // 8 KB
constexpr int DG_A_BYTES = DG_SLICES * DG_A_SLICE;             // 56 KB
constexpr int DG_EPI_WARPS = 16;
constexpr int DG_THREADS = 64 + 32 * DG_EPI_WARPS;
constexpr size_t DG_WORK_CAP = (size_t)4 << 30;                // A images of one launch
constexpr int TN = 32;                                         // rows of N an item
constexpr int DG_B_BYTES = DG_SLICES * TN * DG_ROW;
constexpr int DG_STAGE = DG_A_BYTES + DG_B_BYTES;              // 70 KB
constexpr int DG_NSTAGE = 3;
constexpr int DG_NONFINITE = 8192;                             // forward: scale exponent of a column with an infinity or NaN
constexpr int DG_NACC = 2;                                     // accumulator sets (7 TN TMEM columns each)
constexpr int DG_SMEM = 1024 + DG_NSTAGE * DG_STAGE + 256;

struct DgMInfo {
  long long tab[2];  // first table tile of (m, p), bytes
  int ch[2];         // first A chunk of (m, p)
  int nq[2];         // K chunks
  int kv[2];         // valid K
  int nv[2];         // valid N
  int nr[2];         // N rounded up to 16
  long long eb[2];   // first row-scale entry: inverse eb[0] + jj; forward idx(m, m) (entry idx(m, n))
};

struct DgArgs {
  int N, Jh, batch;
  int c0;            // first column of this launch
  int nct;           // column tiles
  int nitems;        // items per column tile
  int nchunk;        // A chunks per column tile
  int ldea;          // row length of ea
  int enan;          // scale exponent from which an operand was not finite
  long long ncoef;
  const DgMInfo *mi;
  const int2 *items;           // (m, nt)
  const unsigned char *A, *B;
  const int *ea;               // scale exponents of A: inverse [m][c], forward [2m+p][c]
  const short *eb;             // scale exponents of the table rows
  double *out;                 // F or spectra
  int *err;
  unsigned long long wait_ns;
  int withhold;
};

__device__ __forceinline__ uint64_t dg_desc(uint32_t addr) {
  // K-major, 64-byte swizzle, 8-row groups 512 bytes apart
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)4 << 61);
}

// byte offset of 16-byte unit u (8 values of K) of row r in a swizzled slice
__host__ __device__ __forceinline__ int dg_unit(int r, int u) { return r * DG_ROW + ((u ^ ((r >> 1) & 3)) << 4); }

// The MMAs of one stage, ks K steps of 16, for a tile of NTW rows of N: slice
// i of A with as many consecutive slices j of B as 256 columns hold, into
// accumulators i + j.  Descriptors by constant offsets from the stage's two:
// with them built anew for each MMA the issuing thread was the limit (T341 x
// 192 with loads and epilogue taken out: synthesis 250, analysis 298 us).
template <int NTW>
__device__ __forceinline__ void dg_mma(uint32_t acc, uint64_t da, uint64_t db, int ks, int first) {
  constexpr int PER = 256 / NTW;
  for (int kk = 0; kk < ks; ++kk) {
#pragma unroll
    for (int i = 0; i < DG_SLICES; ++i)
#pragma unroll
      for (int j = 0; j < DG_SLICES - i; j += PER) {
        const int n = DG_SLICES - i - j < PER ? DG_SLICES - i - j : PER;
        mma_bf16(acc + (i + j) * NTW, da + (i * DG_A_SLICE >> 4), db + (j * NTW * DG_ROW >> 4),
                 idesc_f16kind(n * NTW, 0, 0), i ? 1 : first);
      }
    first = 1;
    da += 2;  // 32 bytes
    db += 2;
  }
}

__device__ __forceinline__ int dg_item(int k) {  // as cta_item: rounds in alternating directions
  const int G = (int)gridDim.x, b = (int)blockIdx.x;
  return (k & 1) ? (k + 1) * G - 1 - b : k * G + b;
}

__device__ __noinline__ double dg_double_any(long long q, int ex) { return fixed_to_double(q, ex); }

// Bits, at most 10, that the sums S (and those in any) can be shifted up by to
// stay below 2^62: the lower levels (DgSum::l, below 2^31 then) still come on
// top, and carry a sum that lies just below a power of two over it.
template <int EC> __device__ __forceinline__ int dg_room(const DgSum (&S)[EC], unsigned &any) {
#pragma unroll
  for (int x = 0; x < EC; ++x) {
    const int hi = (int)(S[x].t >> 32);
    any |= (unsigned)(hi ^ (hi >> 31));
  }
  return min(__clz((int)any) - 2, 10);
}

// The integer pipes limit this part (16 results a thread of the inverse took
// 7,400 cycles with a range branch each and the scales loaded at the end: half
// of an item's epilogue; T85 x 128 both ways 120 -> 111 us without them).
// put(x, conv) for x < EC, where conv(q, x) is the double of q units of 2^-up
// at level 6, given the scale exponents of the table's rows: without branches
// where all results are normal.
template <int EC, class Put>
__device__ __forceinline__ void dg_results(const int (&eb)[EC], int E, int up, int enan, Put put) {
  const int e0 = E - 1022 - 52 - up;
  bool normal = E < enan;
#pragma unroll
  for (int x = 0; x < EC; ++x) normal = normal && e0 + eb[x] >= FIXED_EX_MIN && e0 + eb[x] <= FIXED_EX_MAX;
  if (normal) {
#pragma unroll
    for (int x = 0; x < EC; ++x) put(x, [&](long long q, int k) { return fixed_to_double_normal(q, e0 + eb[k]); });
  } else {  // rows of the table near the poles at large m, extreme or non-finite operands
#pragma unroll
    for (int x = 0; x < EC; ++x)
      put(x, [&](long long q, int k) {
        return E < enan ? dg_double_any(q, e0 + eb[k]) : __longlong_as_double(0x7FF8000000000000ll);
      });
  }
}

// A CTA's items in order, with the table entries of the current one in
// registers: they are loaded an item ahead (the first before the wait for the
// kernel before, a chain of loads of 1 us), their place in the list two ahead.
// Read through the table at each use, that is anew after every wait and copy,
// T341 x 192 took 3 % longer.
struct DgWalk {
  int k, it, ct, m, nt;
  DgMInfo mi;
  int2 next, after;
  DgMInfo minext;

  __device__ __forceinline__ static int2 entry(const DgArgs &a, int it) {
    return it < a.nct * a.nitems ? __ldg(a.items + it / a.nct) : make_int2(0, 0);
  }
  __device__ __forceinline__ explicit DgWalk(const DgArgs &a) : k(-1), next(entry(a, dg_item(0))), after(entry(a, dg_item(1))) {
    minext = a.mi[next.x];
  }
  // the next item, if there is one
  __device__ __forceinline__ bool step(const DgArgs &a) {
    it = dg_item(++k);
    if (it >= a.nct * a.nitems) return false;
    ct = it % a.nct;
    m = next.x;
    nt = next.y;
    mi = minext;
    next = after;
    after = entry(a, dg_item(k + 2));
    minext = a.mi[next.x];
    return true;
  }
};

// position of Re (im = 0) or Im s_n^m in SPML's real layout of a field-level
__device__ __forceinline__ long long wa_at(int n, int m, int im) { return (long long)n * (n + 1) + (im ? -m : m); }

// WA: forward results in SPML's real layout.
template <int DIR, bool WA>
__global__ void __launch_bounds__(DG_THREADS, 1) legendre_dg_kernel(const __grid_constant__ DgArgs a) {
  constexpr int NSTAGE = DG_NSTAGE, NACC = DG_NACC;
  extern __shared__ __align__(1024) unsigned char smem_dyn[];
  unsigned char *stage = reinterpret_cast<unsigned char *>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = reinterpret_cast<uint64_t *>(stage + NSTAGE * DG_STAGE);
  uint64_t *full = bars, *empty = bars + NSTAGE, *accf = bars + 2 * NSTAGE, *acce = accf + NACC;
  uint64_t *drain = bars + 15;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 16);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 17);

  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < NACC; ++s) {
      mbar_init(&accf[s], 1);
      mbar_init(&acce[s], 32 * DG_EPI_WARPS);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  DgWalk w(a);  // (tables: nothing that the kernel before writes)
  pdl_wait();
  pdl_trigger();

  if (warp == 0) {
    // -------------------------------------------------------- copies
    if (lane == 0 && !a.withhold) {
      int g = 0;
      bool ok = true;
      while (ok && w.step(a)) {
        const int ct = w.ct, nt = w.nt;
        const DgMInfo &mi = w.mi;
        // rows of the column tile that hold data (whole groups of 8)
        const int rows = min(128, ((2 * a.batch - a.c0 - ct * 128) + 7) & ~7);
        for (int p = 0; p < 2 && ok; ++p) {
          const int nr = p ? mi.nr[1] : mi.nr[0], nq = p ? mi.nq[1] : mi.nq[0];
          if (nt * TN >= nr) continue;
          const int ntw = min(TN, nr - nt * TN);
          const uint32_t bb = (uint32_t)(DG_SLICES * DG_ROW * ntw);
          const unsigned char *Bt = a.B + (p ? mi.tab[1] : mi.tab[0]) + (long long)nt * TN * nq * (DG_SLICES * DG_ROW);
          const unsigned char *At = a.A + ((long long)ct * a.nchunk + (p ? mi.ch[1] : mi.ch[0])) * DG_A_BYTES;
          for (int q = 0; q < nq; ++q, ++g) {
            const int s = g % NSTAGE;
            if (!mbar_wait(&empty[s], ((g / NSTAGE) & 1) ^ 1, a.err, abort_flag, 1, a.wait_ns)) { ok = false; break; }
            unsigned char *As = stage + s * DG_STAGE;
            const unsigned char *Ag = At + (long long)q * DG_A_BYTES;
            mbar_arrive_tx(&full[s], (uint32_t)(DG_SLICES * DG_ROW * rows) + bb);
            bulk_load(As + DG_A_BYTES, Bt + (long long)q * bb, bb, &full[s]);
            if (rows == 128) {
              bulk_load(As, Ag, DG_A_BYTES, &full[s]);
            } else {
              for (int i = 0; i < DG_SLICES; ++i)
                bulk_load(As + i * DG_A_SLICE, Ag + i * DG_A_SLICE, (uint32_t)(rows * DG_ROW), &full[s]);
            }
          }
        }
      }
      if (!ok) {  // let the copies in flight land before the CTA's shared memory goes
        for (int h = g > NSTAGE ? g - NSTAGE : 0; h < g; ++h)
          mbar_wait_bounded(&full[h % NSTAGE], (h / NSTAGE) & 1, nullptr, 0);
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA
    if (lane == 0) {
      int g = 0, seg = 0;
      bool ok = true;
      while (ok && w.step(a)) {
        const int nt = w.nt;
        const DgMInfo &mi = w.mi;
        for (int p = 0; p < 2 && ok; ++p) {
          const int nr = p ? mi.nr[1] : mi.nr[0], nq = p ? mi.nq[1] : mi.nq[0], kv = p ? mi.kv[1] : mi.kv[0];
          if (nt * TN >= nr) continue;
          const int ntw = min(TN, nr - nt * TN);
          for (int q0 = 0; q0 < nq && ok; q0 += DG_KB, ++seg) {
            const int set = seg % NACC;
            if (!mbar_wait(&acce[set], ((seg / NACC) & 1) ^ 1, a.err, abort_flag, 2, a.wait_ns)) { ok = false; break; }
            tc_fence_after();
            const uint32_t acc = tmem + set * 256;
            int first = 0;  // 0 until the accumulators have been written
            for (int q = q0; q < min(nq, q0 + DG_KB); ++q, ++g) {
              const int s = g % NSTAGE;
              if (!mbar_wait(&full[s], (g / NSTAGE) & 1, a.err, abort_flag, 3, a.wait_ns)) { ok = false; break; }
              tc_fence_after();
              const uint32_t As = smem_u32(stage + s * DG_STAGE);
              const uint64_t da = dg_desc(As), db = dg_desc(As + DG_A_BYTES);
              const int ks = min(2, (kv - q * DG_CHUNK + 15) / 16);
              if (ntw == TN) dg_mma<TN>(acc, da, db, ks, first);
              else dg_mma<16>(acc, da, db, ks, first);
              first = 1;
              mma_commit(&empty[s]);
            }
            if (ok) mma_commit(&accf[set]);
          }
        }
      }
      if (!ok) {  // MMAs in flight end before the TMEM is freed
        mma_commit(drain);
        mbar_wait_bounded(drain, 0, nullptr, 0);
      }
    }
    __syncwarp();
  } else {
    // ----------------------------------------------------- epilogue
    // four warps a TMEM lane quarter, each with TN / 4 columns
    constexpr int EC = TN / 4;
    const int quad = warp & 3, j0 = ((warp - 2) >> 2) * EC;
    const int row = quad * 32 + lane;
    const int C2B = 2 * a.batch;
    int seg = 0;
    bool dead = false;
    while (!dead && w.step(a)) {
      const int ct = w.ct, m = w.m, nt = w.nt;
      const DgMInfo &mi = w.mi;
      const int c = a.c0 + ct * 128 + row;
      const bool live = c < C2B;
      const int r0 = nt * TN + j0;  // first row of the table
      // inverse: both parities' sums; forward: the current parity's
      DgSum sum[DIR == 0 ? 2 : 1][EC];
      int E = 0, ex[EC];  // scale exponents of A's column and the table's rows
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        DgSum(&S)[EC] = sum[DIR == 0 ? p : 0];
#pragma unroll
        for (int x = 0; x < EC; ++x) S[x] = DgSum{0, 0.f};
        if (nt * TN >= mi.nr[p]) continue;
        const int ntw = min(TN, mi.nr[p] - nt * TN);
        const int nx = live ? mi.nv[p] - r0 : 0;  // columns k of the tile with a result
        // loaded ahead of the sums they scale
        if ((DIR == 1 || p == 0) && nx > 0) {
          E = a.ea[(long long)(DIR == 0 ? m : 2 * m + p) * a.ldea + c];
          // forward: n = m + p + 2 (r0 + x)
          const short *eb = a.eb + mi.eb[p] + (DIR == 0 ? r0 : p + 2 * r0);
#pragma unroll
          for (int x = 0; x < EC; ++x) ex[x] = x < nx ? eb[DIR == 0 ? x : 2 * x] : 0;
        }
        for (int q0 = 0; q0 < mi.nq[p]; q0 += DG_KB, ++seg) {
          const int set = seg % NACC;
          if (!mbar_wait(&accf[set], (seg / NACC) & 1, a.err, abort_flag, 4, a.wait_ns)) {
            dead = true;
            break;
          }
          tc_fence_after();
          const uint32_t tb = tmem + ((uint32_t)(quad * 32) << 16) + set * 256 + j0;
          if (j0 < ntw) {
#pragma unroll
            for (int h = 0; h < EC; h += 4) {
              uint32_t v[DG_SLICES][4];
#pragma unroll
              for (int s = 0; s < DG_SLICES; ++s) tmem_ld4_nw(tb + s * ntw + h, v[s]);
              tmem_wait_ld();
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const uint32_t w7[DG_SLICES] = {v[0][x], v[1][x], v[2][x], v[3][x], v[4][x], v[5][x], v[6][x]};
                dg_accumulate(S[h + x], w7);
              }
            }
          }
          tc_fence_before();
          mbar_arrive(&acce[set]);
        }
        if (dead) break;
        if (DIR == 1 && nx > 0) {
          double *dst = a.out + ((long long)(c >> 1) * a.ncoef + mi.eb[p] + p + 2 * r0) * 2 + (c & 1);
          const bool zero = m == 0 && (c & 1);
          const int nn = m + p + 2 * r0;  // n of the first result
          if constexpr (WA) dst = a.out + (long long)(c >> 1) * (a.N + 1) * (a.N + 1) + wa_at(nn, m, c & 1);
          unsigned any = 0;
          const int up = dg_room(S, any);
          dg_results<EC>(ex, E, up, a.enan, [&](int x, auto conv) {
            const double v = conv(dg_sum_fixed(S[x], up), x);
            if constexpr (WA) {
              // n (n + 1) grows by 2 x (2 nn + 1 + 2 x) over 2 x degrees
              if (x < nx && !zero) dst[2 * x * (2 * nn + 1 + 2 * x)] = v;
            } else if (x < nx) {
              dst[4 * x] = zero ? 0.0 : v;
            }
          });
        }
      }
      if (DIR == 0 && !dead && live && r0 < a.Jh) {
        double *Fn = a.out + ((long long)m * 2 * a.Jh + a.Jh + r0) * C2B + c;      // latitude Jh + jj
        double *Fs = a.out + ((long long)m * 2 * a.Jh + a.Jh - 1 - r0) * C2B + c;  // its mirror
        unsigned any = 0;
        dg_room(sum[0], any);
        const int up = dg_room(sum[DIR == 0], any) - 1;  // for e + o and e - o
        dg_results<EC>(ex, E, up, a.enan, [&](int x, auto conv) {
          const long long e = dg_sum_fixed(sum[0][x], up), o = dg_sum_fixed(sum[DIR == 0][x], up);
          const double n = conv(e + o, x), s = conv(e - o, x);
          if (r0 + x < a.Jh) {
            Fn[(long long)x * C2B] = n;
            Fs[-(long long)x * C2B] = s;
          }
        });
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

// ------------------------------------------------------------------ packs
// Spectra -> A images.  G lanes handle one (m, field-level b): they find the
// largest magnitude of its coefficients n = m .. N (one scale for both
// parities and for re and im), then write the digits; a lane takes 8
// coefficients of one parity (n0 + p, n0 + p + 2, ...).  Whole chunks are
// written, zeros past the last coefficient.
// Where the spectra lie: complex numbers read as 16-byte pairs, the same at an
// address that is a multiple of 8 bytes only, SPML's real layout (spml.cu).
enum SpecLayout { SPEC_PAIRS, SPEC_DOUBLES, SPEC_WA };
template <int G, SpecLayout LAY>
__global__ void __launch_bounds__(256)
dg_pack_spec(const DgMInfo *__restrict__ mi_, int N, long long ncoef, const double *__restrict__ spec, int b0, int nb,
             int nchunk, unsigned char *__restrict__ A, int *__restrict__ ea, int ldea) {
  const int m = blockIdx.y;
  const int nq0 = mi_[m].nq[0], nq1 = mi_[m].nq[1], ch0 = mi_[m].ch[0], ch1 = mi_[m].ch[1];
  asm volatile("" ::"r"(nq0 + nq1 + ch0 + ch1));  // plan constants: loaded before the wait
  pdl_wait();
  pdl_trigger();
  const int gl = threadIdx.x % G;
  const int bl = blockIdx.x * (256 / G) + threadIdx.x / G;  // field-level of this launch
  const bool live = bl < nb;
  const int b = b0 + (live ? bl : 0);
  const double *src = spec + 2 * ((long long)b * ncoef + idx_mn(N, m, m));
  const double *wa = spec + (long long)b * (N + 1) * (N + 1);
  auto coefficient = [&](int n) {
    if constexpr (LAY == SPEC_WA) return make_double2(__ldg(wa + wa_at(n, m, 0)), m ? __ldg(wa + wa_at(n, m, 1)) : 0.0);
    else if constexpr (LAY == SPEC_DOUBLES) return make_double2(__ldg(src + 2 * (n - m)), __ldg(src + 2 * (n - m) + 1));
    else return __ldg(reinterpret_cast<const double2 *>(src) + (n - m));
  };
  // Im s_n^0 does not enter the synthesis, whatever it holds: not the scale
  // either (its digits are then any, and its column is not read)
  const unsigned im_mag = m ? 0x7FFFFFFFu : 0u;
  const int nu = 4 * max(nq0, nq1);  // units of 8 a parity, both parities side by side
  unsigned mx = 0;
  double2 v[8];
  for (int t = gl; t < 2 * nu; t += G) {
    const int n0 = m + 16 * (t >> 1) + (t & 1);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[e] = live && n0 + 2 * e <= N ? coefficient(n0 + 2 * e) : make_double2(0.0, 0.0);
      mx = max(mx, max(dg_mag(v[e].x), (unsigned)__double2hiint(v[e].y) & im_mag));
    }
  }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (!live) return;
  const int E = dg_exp(mx);
  const int c = 2 * bl;  // column within this launch
  const int ct = c / 128, row = c % 128;
  if (gl == 0) *reinterpret_cast<int2 *>(ea + (long long)m * ldea + 2 * b) = make_int2(E, E);
  const bool keep = 2 * nu <= G;  // the values are still in registers
  for (int t = gl; t < 2 * nu; t += G) {
    const int p = t & 1, u = t >> 1;
    if (u >= 4 * (p ? nq1 : nq0)) continue;
    const int n0 = m + 16 * u + p;
    if (!keep) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = n0 + 2 * e <= N ? coefficient(n0 + 2 * e) : make_double2(0.0, 0.0);
    }
    unsigned char *img = A + ((long long)ct * nchunk + (p ? ch1 : ch0) + (u >> 2)) * DG_A_BYTES;
    unsigned long long q[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) q[e] = dg_fixed(v[e].x, E);
    dg_store8(img + dg_unit(row, u & 3), DG_A_SLICE, q);
#pragma unroll
    for (int e = 0; e < 8; ++e) q[e] = dg_fixed(v[e].y, E);
    dg_store8(img + dg_unit(row + 1, u & 3), DG_A_SLICE, q);
  }
}

// Exponents of a lane's eight latitudes, times 2^20 (of the high words' unit).
__device__ __forceinline__ void dg_factors(const int *ec, int (&f)[8]) {
  const int4 a = __ldg(reinterpret_cast<const int4 *>(ec)), b = __ldg(reinterpret_cast<const int4 *>(ec) + 1);
  f[0] = a.x, f[1] = a.y, f[2] = a.z, f[3] = a.w, f[4] = b.x, f[5] = b.y, f[6] = b.z, f[7] = b.w;
}
// Folded Fourier coefficients G[m][p][jj][c] -> A images, every latitude times
// its factor 2^ec (dg_fwd_scales), one scale per (m, p, c).  A warp takes 8
// columns x 4 units of 8 latitudes (one chunk): its loads are 64-byte runs along
// c, its stores whole rows of an image.  WQ warps share the chunks of 8 columns.
template <int WQ>
__global__ void __launch_bounds__(256, 4)
dg_pack_four(const DgMInfo *__restrict__ mi_, int Jh, int C2B, int c0, int nc, const double *__restrict__ Gf, int nchunk,
             unsigned char *__restrict__ A, int *__restrict__ ea, int ldea, int guard, const int *__restrict__ ec_,
             int ldec) {
  __shared__ int smx[8][8];
  const int mp = blockIdx.y, m = mp >> 1, p = mp & 1;
  const int nv = mi_[m].nv[p], nq = mi_[m].nq[p], ch = mi_[m].ch[p];
  asm volatile("" ::"r"(nv + nq + ch));  // plan constants: loaded before the wait
  pdl_wait();
  pdl_trigger();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int c8 = lane & 7, u = lane >> 3;
  const int cl = (blockIdx.x * (8 / WQ) + warp / WQ) * 8 + c8;
  const bool live = cl < nc;
  if (nv <= 0) return;  // this parity has no coefficient (uniform over the block)
  const double *src = Gf + (long long)mp * Jh * C2B + c0 + (live ? cl : 0);
  const int *ec = ec_ + (long long)mp * ldec;
  double v[8];
  int f[8];  // (loaded again for the digits: eight registers fewer meanwhile)
  int mx = 1 << 20;  // exponents are at most 0: enough for zeros and subnormals
  unsigned any = 0;
  for (int q = warp % WQ; q < nq; q += WQ) {
    const int j0 = q * DG_CHUNK + 8 * u;
    dg_factors(ec + j0, f);
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = live && j0 + e < Jh ? __ldg(src + (long long)(j0 + e) * C2B) : 0.0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      any = max(any, dg_mag(v[e]));
      mx = max(mx, (int)dg_mag(v[e]) + f[e]);
    }
  }
  mx = any < 0x7FF00000u ? mx >> 20 : DG_NONFINITE;
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
  mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
  if (WQ > 1) {
    if (u == 0) smx[warp][c8] = mx;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < WQ; ++k) mx = max(mx, smx[warp / WQ * WQ + k][c8]);
  }
  if (!live) return;
  const int E = mx + guard;
  if (u == 0 && warp % WQ == 0) ea[(long long)mp * ldea + c0 + cl] = E;
  const int ct = cl / 128, row = cl % 128;
  const bool keep = nq <= WQ;
  for (int q = warp % WQ; q < nq; q += WQ) {
    const int j0 = q * DG_CHUNK + 8 * u;
    dg_factors(ec + j0, f);
    if (!keep) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = j0 + e < Jh ? __ldg(src + (long long)(j0 + e) * C2B) : 0.0;
    }
    unsigned char *img = A + ((long long)ct * nchunk + ch + q) * DG_A_BYTES;
    unsigned long long qv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) qv[e] = dg_fixed(v[e], E - (f[e] >> 20));
    dg_store8(img + dg_unit(row, u), DG_A_SLICE, qv);
  }
}

// ------------------------------------------------------------------ tables
// Inverse: scale exponent of every table row (m, jj) over all n.  The stored
// value is E - 1022: the row's entries are below 2^eb.  One warp per row.
__global__ void dg_inv_scales(int N, int Jh, const double *__restrict__ pnm, long long nrows, short *__restrict__ eb) {
  const long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= nrows) return;
  unsigned mx = 0;
  const int m = (int)(r / Jh), jj = (int)(r % Jh);
  for (int n = m + lane; n <= N; n += 32) mx = max(mx, dg_mag(pnm[idx_mn(N, m, n) * Jh + jj]));
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (lane == 0) eb[r] = (short)(dg_exp(mx) - 1022);
}

// Forward: factors 2^ec of the latitudes, 2^-ec of them on the table, such
// that every latitude's largest entry of (w/2) Pbar over the degrees of one (m, p)
// lies in [2^7, 2^8) (ec < 0: entries are at most sqrt(2 N + 1) / 2); then the scale exponent of every row (m, n) over the
// latitudes.  Towards the poles the entries of large m fall by hundreds of orders
// of magnitude, and the Fourier coefficients need not: without the factors the
// largest coefficient set the scale although its products count for nothing, and
// a field non-zero near the poles alone lost whole wavenumbers (T85: from m =
// 40 on).  With them the scale is that of the largest product of the (m, p); the
// analysis pack does two integer instructions a value more for them (T341 x 192
// both ways 2,577 -> 2,590 us, T85 x 128 106.9 -> 107.5).
// Block (m, p); ec[(2 m + p) ldec + jj] times 2^20, zero past the last latitude.
__global__ void __launch_bounds__(256)
dg_fwd_scales(const DgMInfo *__restrict__ mi_, int N, int Jh, const double *__restrict__ pnm, const double *__restrict__ w,
              int *__restrict__ ec_, int ldec, short *__restrict__ eb) {
  const int mp = blockIdx.x, m = mp >> 1, p = mp & 1;
  const int nv = mi_[m].nv[p];
  int *ec = ec_ + (long long)mp * ldec;
  const double *tab = pnm + (idx_mn(N, m, m) + p) * Jh;  // row k (n = m + p + 2 k) at 2 k Jh
  for (int jj = threadIdx.x; jj < ldec; jj += blockDim.x) {
    unsigned mx = 0;
    if (jj < Jh)
      for (int k = 0; k < nv; ++k) mx = max(mx, dg_mag((0.5 * w[Jh + jj]) * tab[2LL * k * Jh + jj]));
    ec[jj] = jj < Jh && nv > 0 ? (dg_exp(mx) - 1030) * (1 << 20) : 0;
  }
  __syncthreads();
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  for (int k = warp; k < nv; k += blockDim.x / 32) {
    int mx = -4096;
    for (int jj = lane; jj < Jh; jj += 32) mx = max(mx, dg_exp(dg_mag((0.5 * w[Jh + jj]) * tab[2LL * k * Jh + jj])) - (ec[jj] >> 20));
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) eb[mi_[m].eb[p] + p + 2 * k] = (short)(mx - 1022);
  }
}

// Table tiles: thread = (m, p, row of N, unit of 8 along K).
__global__ void __launch_bounds__(256)
dg_build(int dir, int N, int Jh, const DgMInfo *__restrict__ mi_, const double *__restrict__ pnm,
         const double *__restrict__ w, const short *__restrict__ eb, const int *__restrict__ ec, int ldec,
         unsigned char *__restrict__ B) {
  const int m = blockIdx.y, p = blockIdx.z;
  const DgMInfo &mi = mi_[m];
  const int nu = 4 * mi.nq[p];
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < mi.nr[p] * nu; t += gridDim.x * blockDim.x) {
    // neighbouring threads along the table's contiguous latitude index
    const int r = dir == 0 ? t % mi.nr[p] : t / nu, ug = dir == 0 ? t / mi.nr[p] : t % nu;
    unsigned long long q[8];
    int E = 1;
    if (r < mi.nv[p]) E = eb[dir == 0 ? mi.eb[0] + r : mi.eb[p] + p + 2 * r] + 1022;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int k = 8 * ug + e;
      double x = 0.0;
      int Ek = 1;
      if (r < mi.nv[p] && k < mi.kv[p]) {
        if (dir == 0) x = pnm[idx_mn(N, m, m + p + 2 * k) * Jh + r];
        else x = (0.5 * w[Jh + k]) * pnm[idx_mn(N, m, m + p + 2 * r) * Jh + k];
        Ek = dir == 0 ? E : E + (ec[(2 * m + p) * ldec + k] >> 20);
      }
      q[e] = dg_fixed(x, Ek);
    }
    const int nt = r / TN, ntw = min(TN, mi.nr[p] - nt * TN);
    unsigned char *tile = B + mi.tab[p] +
                          ((long long)nt * TN * mi.nq[p] + (long long)(ug >> 2) * ntw) * (DG_SLICES * DG_ROW);
    dg_store8(tile + dg_unit(r % TN, ug & 3), (size_t)ntw * DG_ROW, q);
  }
}

// ------------------------------------------------------------------ host

// One direction's metadata; tab: bytes of its tiles.
static void plan_dir(const Plan &P, int dir, DgTable &T, std::vector<DgMInfo> &mi, std::vector<int2> &items,
                     long long &tab) {
  const int N = P.N, Jh = P.Jh;
  mi.resize(N + 1);
  tab = 0;
  int ch = 0;
  for (int m = 0; m <= N; ++m) {
    DgMInfo &M = mi[m];
    int nrmax = 0;
    for (int p = 0; p < 2; ++p) {
      const int cnt = count_np(N, m, p);
      M.kv[p] = cnt > 0 ? (dir == 0 ? cnt : Jh) : 0;
      M.nv[p] = cnt > 0 ? (dir == 0 ? Jh : cnt) : 0;
      M.nq[p] = (M.kv[p] + DG_CHUNK - 1) / DG_CHUNK;
      M.nr[p] = (M.nv[p] + 15) / 16 * 16;
      M.tab[p] = tab;
      M.ch[p] = ch;
      M.eb[p] = dir == 0 ? (long long)m * Jh : idx_mn(N, m, m);
      tab += (long long)M.nr[p] * M.nq[p] * (DG_SLICES * DG_ROW);
      ch += M.nq[p];
      nrmax = M.nr[p] > nrmax ? M.nr[p] : nrmax;
    }
    for (int nt = 0; nt * TN < nrmax; ++nt) items.push_back(make_int2(m, nt));
  }
  T.nchunk = ch;
  // keep the 64-bit sums of (inverse: two parities of) K products in range (DgSum)
  const int K = dir == 0 ? 2 * count_np(N, 0, 0) : Jh;
  while (K >> T.guard > 512) ++T.guard;
  T.nitems = (int)items.size();
}

// Tables of both directions and the A images.  The images of one launch are
// bounded (DG_WORK_CAP); a larger batch takes several launches.
int build_digits(Plan &P) {
  // set here and not by the first launch of a process: it holds for the
  // device and context that the plan is made in
  for (auto kernel : {legendre_dg_kernel<0, false>, legendre_dg_kernel<1, false>, legendre_dg_kernel<1, true>})
    DCCM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DG_SMEM));
  DgTable *T[2] = {&P.dinv, &P.dfwd};
  std::vector<DgMInfo> mi[2];
  std::vector<int2> items[2];
  long long tab[2];
  // one allocation: metadata and items of both directions (one copy), row
  // scales, tiles
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const long long nrows[2] = {(long long)(P.N + 1) * P.Jh, (long long)P.ncoef};
  const int ldec = (P.Jh + DG_CHUNK - 1) / DG_CHUNK * DG_CHUNK;
  size_t at_mi[2], at_it[2], at_eb[2], at_tab[2], at_ec, at = 0;
  for (int d = 0; d < 2; ++d) {
    plan_dir(P, d, *T[d], mi[d], items[d], tab[d]);
    at_mi[d] = at;
    at_it[d] = at + mi[d].size() * sizeof(DgMInfo);
    at = up(at_it[d] + items[d].size() * sizeof(int2));
  }
  std::vector<unsigned char> &h = P.h_dg;
  h.assign(at, 0);
  for (int d = 0; d < 2; ++d) {
    memcpy(h.data() + at_mi[d], mi[d].data(), mi[d].size() * sizeof(DgMInfo));
    memcpy(h.data() + at_it[d], items[d].data(), items[d].size() * sizeof(int2));
    at_eb[d] = at;
    at_tab[d] = at + up((size_t)nrows[d] * sizeof(short));
    at = up(at_tab[d] + (size_t)tab[d]);
  }
  at_ec = at;
  at += (size_t)2 * (P.N + 1) * ldec * sizeof(int);
  DCCM_CUDA(cudaMalloc(&P.d_dgmem, at));
  unsigned char *base = (unsigned char *)P.d_dgmem;
  DCCM_CUDA(cudaMemcpyAsync(base, h.data(), h.size(), cudaMemcpyHostToDevice));
  for (int d = 0; d < 2; ++d) {
    T[d]->d_mi = base + at_mi[d];
    T[d]->d_items = (int2 *)(base + at_it[d]);
    T[d]->d_eb = (short *)(base + at_eb[d]);
    T[d]->d_tab = base + at_tab[d];
    T[d]->d_ec = d == 0 ? nullptr : (int *)(base + at_ec);
    if (d == 0)
      dg_inv_scales<<<(unsigned)((nrows[d] + 7) / 8), 256>>>(P.N, P.Jh, P.d_pnm, nrows[d], T[d]->d_eb);
    else
      dg_fwd_scales<<<2 * (P.N + 1), 256>>>((const DgMInfo *)T[d]->d_mi, P.N, P.Jh, P.d_pnm, P.d_w, T[d]->d_ec, ldec,
                                            T[d]->d_eb);
    DCCM_LAUNCH_CHECK();
    dg_build<<<dim3(16, P.N + 1, 2), 256>>>(d, P.N, P.Jh, (const DgMInfo *)T[d]->d_mi, P.d_pnm, P.d_w, T[d]->d_eb,
                                            T[d]->d_ec, ldec, (unsigned char *)T[d]->d_tab);
    DCCM_LAUNCH_CHECK();
  }
  const int nch = P.dinv.nchunk > P.dfwd.nchunk ? P.dinv.nchunk : P.dfwd.nchunk;
  const size_t per = (size_t)nch * DG_A_BYTES;
  const int nct = (2 * P.max_batch + 127) / 128;
  size_t cap = DG_WORK_CAP / per;
  if (cap < 1) cap = 1;
  P.dg_ct = (size_t)nct < cap ? nct : (int)cap;
  P.dg_ldea = 2 * P.max_batch;
  const size_t dig = per * P.dg_ct;
  DCCM_CUDA(cudaMalloc(&P.d_dig, dig + (size_t)2 * (P.N + 1) * P.dg_ldea * sizeof(int)));
  P.d_ea = (int *)((unsigned char *)P.d_dig + dig);
  return DCCM_OK;
}

template <int DIR, bool WA> static int launch_kernel(const DgArgs &a, int items, cudaStream_t s) {
  const int ctas = sm_count();
  DCCM_CUDA(launch_pdl(legendre_dg_kernel<DIR, WA>, dim3(items < ctas ? items : ctas), dim3(DG_THREADS), (size_t)DG_SMEM, s,
                       a));
  return DCCM_OK;
}

static int launch_dg(Plan &P, int dir, int batch, int c0, int nct, double *out, bool wa, cudaStream_t s) {
  const DgTable &T = dir == 0 ? P.dinv : P.dfwd;
  DgArgs a;
  a.N = P.N;
  a.Jh = P.Jh;
  a.batch = batch;
  a.c0 = c0;
  a.nct = nct;
  a.nitems = T.nitems;
  a.nchunk = T.nchunk;
  a.ldea = P.dg_ldea;
  a.enan = dir == 0 ? 2047 : DG_NONFINITE;
  a.ncoef = P.ncoef;
  a.mi = (const DgMInfo *)T.d_mi;
  a.items = T.d_items;
  a.A = (const unsigned char *)P.d_dig;
  a.B = (const unsigned char *)T.d_tab;
  a.ea = P.d_ea;
  a.eb = T.d_eb;
  a.out = out;
  a.err = P.d_err;
  a.wait_ns = tunables().wait_limit_ms > 0 ? 1000000ull * (unsigned long long)tunables().wait_limit_ms : WAIT_LIMIT_NS;
  a.withhold = tunables().tc_withhold_loads;
  const int items = nct * T.nitems;
  if (dir == 0) return launch_kernel<0, false>(a, items, s);
  return wa ? launch_kernel<1, true>(a, items, s) : launch_kernel<1, false>(a, items, s);
}

int legendre_inv_f64(Plan &P, int batch, const double *spec, double *F, cudaStream_t s, bool wa) {
  const int nct = (2 * batch + 127) / 128;
  const DgMInfo *mi = (const DgMInfo *)P.dinv.d_mi;
  for (int t = 0; t < nct; t += P.dg_ct) {
    const int k = nct - t < P.dg_ct ? nct - t : P.dg_ct;
    const int b0 = 64 * t, nb = batch - b0 < 64 * k ? batch - b0 : 64 * k;
    auto pack = [&](auto kernel, int g) {
      return launch_pdl(kernel, dim3((nb + 256 / g - 1) / (256 / g), P.N + 1), dim3(256), 0, s, mi, P.N, (long long)P.ncoef,
                        spec, b0, nb, P.dinv.nchunk, (unsigned char *)P.d_dig, P.d_ea, P.dg_ldea);
    };
    // lanes a (m, field-level): 2 units of 8 for every 16 coefficients; any
    // number does for spectra at an odd multiple of 8 bytes
    if (wa)
      DCCM_CUDA(P.N < 64 ? pack(dg_pack_spec<8, SPEC_WA>, 8) : P.N < 128 ? pack(dg_pack_spec<16, SPEC_WA>, 16)
                                                                          : pack(dg_pack_spec<32, SPEC_WA>, 32));
    else if (!pairs_aligned(spec))
      DCCM_CUDA(pack(dg_pack_spec<32, SPEC_DOUBLES>, 32));
    else
      DCCM_CUDA(P.N < 64 ? pack(dg_pack_spec<8, SPEC_PAIRS>, 8) : P.N < 128 ? pack(dg_pack_spec<16, SPEC_PAIRS>, 16)
                                                                             : pack(dg_pack_spec<32, SPEC_PAIRS>, 32));
    DCCM_TRY(launch_dg(P, 0, batch, 128 * t, k, F, false, s));
  }
  return DCCM_OK;
}

int legendre_fwd_f64(Plan &P, int batch, const double *G, double *spec, cudaStream_t s, bool wa) {
  const int nct = (2 * batch + 127) / 128;
  const int nq = (P.Jh + DG_CHUNK - 1) / DG_CHUNK;
  const DgMInfo *mi = (const DgMInfo *)P.dfwd.d_mi;
  for (int t = 0; t < nct; t += P.dg_ct) {
    const int k = nct - t < P.dg_ct ? nct - t : P.dg_ct;
    const int c0 = 128 * t, nc = 2 * batch - c0 < 128 * k ? 2 * batch - c0 : 128 * k;
    auto pack = [&](auto kernel, int wq) {
      const int per = 8 * (8 / wq);
      return launch_pdl(kernel, dim3((nc + per - 1) / per, 2 * (P.N + 1)), dim3(256), 0, s, mi, P.Jh, 2 * batch, c0, nc, G,
                        P.dfwd.nchunk, (unsigned char *)P.d_dig, P.d_ea, P.dg_ldea, P.dfwd.guard,
                        (const int *)P.dfwd.d_ec, nq * DG_CHUNK);
    };
    DCCM_CUDA(nq <= 1 ? pack(dg_pack_four<1>, 1) : nq <= 2 ? pack(dg_pack_four<2>, 2)
              : nq <= 4 ? pack(dg_pack_four<4>, 4) : pack(dg_pack_four<8>, 8));
    DCCM_TRY(launch_dg(P, 1, batch, c0, k, spec, wa, s));
  }
  return DCCM_OK;
}

}  // namespace sht
}  // namespace dccm
