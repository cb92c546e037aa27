// Implicit surface coupling of the vertical diffusion (the producer of the
// bulk-flux kernel's ImplCplCoef1/2 and the consumer of its DelVarImplCPL):
//   forward   SfcImplicitCoupling_VDiffForward
//             (atm/dcpam_sfc_implicit_coupling_mod.f90:72-378) with
//             Solve_TriDiagSystem_Forward (:380-405);
//   backward  SfcImplicitCoupling_VDiffBackward (:25-70) with
//             Solve_TriDiagSystem_Backward (:407-420).
// One thread per atmosphere column and system (momentum, temperature, each
// tracer); every array is the reference's (i, j, k[, n]) layout with the
// columns flattened, so consecutive threads touch consecutive addresses at
// every level.  The forward sweep builds each level's row and eliminates it
// in the same pass from the model top down, so the matrices that the
// reference keeps as module state for the backward sweep are written once
// and never re-read.
//
// FP64 accuracy throughout.  The FP64 pipe is the scarce one on this GPU
// (1/64 of FP32), so reciprocals and products of positive numbers run with
// 64-bit mantissas on the integer pipes (fx64.cuh; zeros, infinities and
// out-of-range values take FP64 divisions), one reciprocal per level and
// matrix serves every right-hand side (the momentum matrix serves U and V,
// the tracer matrix every tracer), the mass term uses 1 / (g 2 dt), and each
// level's full Exner function is inverted once.  Results agree with the reference's operation order to
// rounding (the tests hold 1e-13).  Level 1
// of the eliminated systems divides by the zero sub-diagonal the reference
// sets at k = 1 (:199, :237, :272), as the reference does: the coupler
// replaces U, V, T and the vapour tracer there with the surface solution
// before the backward sweep (atm/dccm_atm_mod.f90:832-835).
#include <algorithm>
#include <new>

#include "common.cuh"
#include "fx64.cuh"
#include "nvtx.cuh"

struct dccm_implcpl {
  int ncol = 0, kmax = 0, ncmax = 0, ih2o = 1;
  dccm_implcpl_consts k;
  // kmax x ncol each: the diagonals M(k,0) of UV, Temp and QMix after the
  // forward sweep (M(k,-1) is then 1 and M(k,1) 0), and that sweep's shared
  // factors G, 1/Exner_f and the mass term
  double *d_mtx = nullptr;
  dccm::DevBuf stage;       // host entry points
  cudaStream_t stream = nullptr;
};

namespace dccm {
namespace implcpl {

struct Fwd {
  const double *MomX, *MomY, *Heat, *QFlx, *P, *Ef, *Eh, *Tv, *Z, *Kv, *Kt, *Kq;
  double *DU, *DV, *DT, *DQ, *C1, *C2;
  double *mtx;  // M(k,0) of UV, Temp and QMix
  double *G, *IEF, *Mass;  // per (level, column) factors shared by the systems (geo_kernel)
  long long ncol;
  int kmax, ncmax, ih2o;
  double Grav, CpDry, GasR, inv_g2dt;
  fx::UF uCp, uGasR;  // CpDry and GasR for the integer arithmetic
  bool fast;          // both positive and within 2^+-100
};

// One thread per (column, system): blockIdx.y 0 = momentum (U and V share
// the matrix), 1 = temperature, 2 + t = tracer t (each tracer thread
// eliminates the tracer matrix; tracer 0 stores it).  A single pass from
// the model top down builds each level's row (:188-308) and eliminates it
// at once (:380-405), carrying the eliminated M(k+1,0) and right-hand sides
// of the level above; the eliminated matrix and tendencies are written
// once.  The next level's inputs are fetched while one is eliminated.
//
// With the couplings' magnitudes l = -M(k,-1), u = -M(k,1) and a = -M(k+1,0),
// all positive in an ordinary column, the elimination
//   M(k,0) <- (M(k,0) M(k+1,0) - M(k,1)) / (M(k,-1) M(k+1,0)), and the same
//   of the right-hand side,
// is, with c = u / a,
//   a <- (M(k,0) - c) / l,   r <- (c r - b) / l
// (with q = 1 / a carried: c = u q, q <- l / (M(k,0) - c)): products and reciprocals of positive numbers, which run with 64-bit
// mantissas on the integer pipes (fx64.cuh), and a few signed sums in FP64.
// The top and bottom rows, and rows where a coupling is zero, negative, not
// finite or beyond 2^+-100, take the reference's form in FP64: each column by
// its own values, so that its results do not depend on the columns beside it.
// FP64 was the sweeps' limit (67 operations a column and level forward, 21
// backward; now 12 and 8): with these, forward sweeps of 32,768 columns x 32
// levels took 95 us (174 in FP64), backward 35 (71); with one column in seven
// without diffusion aloft forward 216 (218 with every row in FP64), 2,048 x 16
// 36 (34).  What is left is the sum of three pipes' work (the ALU's about as long as
// FP64's).  The level after the current one is always being fetched: 95 -> 75
// us, 131,072 x 48 397 -> 324, against two levels fetched together ahead of
// their use (five CTAs an SM at 102 registers or four at 128).  The backward
// sweep fetches LVB ahead in the same way (FP64 pipe 66 % busy; with eight
// unrolled and one copy of the code for each matrix a quarter of its cycles
// waited for instructions: 131,072 x 48 172 -> 150 us); its CTAs are single
// warps, so that its three kinds of block spread evenly (32,768 x 32 35 us with
// 128 threads, 33 with 64, 31 with 32; 2,048 x 16 10.3 and 8.3).
constexpr int GL = 2;   // levels a thread of geo_kernel
constexpr int LVB = 2;  // backward sweep: levels fetched ahead

// positive, exponent field in [lo, hi]
__device__ __forceinline__ bool pos_in(double x, unsigned lo, unsigned hi) {
  return ((unsigned)__double2hiint(x) >> 20) - lo <= hi - lo;
}
// -x by the sign bit (a negation that stays a value of its own costs a DADD)
__device__ __forceinline__ double negd(double x) {
  return __hiloint2double(__double2hiint(x) ^ (int)0x80000000, __double2loint(x));
}
__device__ __forceinline__ bool usual(double x) { return pos_in(x, 923, 1123); }

// The factors every system's row uses, once per (level, column) instead of
// once per system: G(j) = P_h(j) / (R Tv_h(j) (z(j+1) - z(j))) at half level
// j = 1..kmax-1 (the transfer coefficient of :182-195 is K(j) G(j)), the
// reciprocal Exner function 1 / Exner_f(j) at full level j (0-based index,
// the temperature rows of :222-260), and the mass term of that level's row.
// A thread takes GL levels of a column (131,072 x 48: forward sweep 333 us with
// one, 324 with two, 326 with four, which has too few threads at 8,192).
__global__ void __launch_bounds__(256) geo_kernel(const Fwd a) {
  pdl_trigger();
  const long long n = a.ncol, K = a.kmax;
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const int j0 = (int)(t / n) * GL;
  const long long c = t % n;
  if (j0 >= K) return;
  double P[GL + 1], Z[GL + 1], Tv[GL], Ef[GL];
#pragma unroll
  for (int i = 0; i <= GL; ++i) {
    const int j = j0 + i;
    P[i] = j <= K ? a.P[c + n * j] : 1.0;
    Z[i] = j >= 1 && j <= K ? a.Z[c + n * (j - 1)] : 0.0;  // full level j - 1
    if (i < GL) {
      Tv[i] = j >= 1 && j < K ? a.Tv[c + n * j] : 1.0;
      Ef[i] = j < K ? a.Ef[c + n * j] : 1.0;
    }
  }
#pragma unroll
  for (int i = 0; i < GL; ++i) {
    const int j = j0 + i;
    if (j >= K) break;
    const long long o = c + n * j;
    a.Mass[o] = (P[i] - P[i + 1]) * a.inv_g2dt;
    a.IEF[o] = fx::rcp_d(Ef[i]);
    if (j >= 1) {
      const double dz = Z[i + 1] - Z[i];
      double g;
      if (a.fast && usual(P[i]) && usual(Tv[i]) && usual(dz)) {
        using namespace fx;
        const UF d = mul(mul(from_double(Tv[i]), a.uGasR), from_double(dz));
        g = to_double(mul(from_double(P[i]), rcp(norm(d))));
      } else {
        g = P[i] * fx::rcp_d(a.GasR * Tv[i] * dz);
      }
      a.G[o] = g;
    }
  }
}

// Row k eliminated as the reference does, in FP64 (top: the row at the model
// top).  A call of its own, so that its FP64 operations are not issued,
// predicated off, on the rows that do not take it.
struct Row {
  double m0, r[2];
};
static __device__ __noinline__ Row eliminate_fp64(bool top, double mm, double m0, double mp, double m0p, double b0,
                                                  double b1, double rp0, double rp1) {
  Row w;
  const double inv = fx::rcp_d(top ? mm : mm * m0p);
  w.m0 = top ? m0 * inv : (m0 * m0p - mp) * inv;
  w.r[0] = top ? b0 * inv : (b0 * m0p - mp * rp0) * inv;
  w.r[1] = top ? b1 * inv : (b1 * m0p - mp * rp1) * inv;
  return w;
}

template <int SYS>
__device__ __forceinline__ void forward_column(const Fwd &a, long long c, int tracer) {
  using fx::UF;
  constexpr int NR = SYS == 0 ? 2 : 1;
  const long long n = a.ncol;
  const int K = a.kmax;
  const double *__restrict__ Kd = SYS == 0 ? a.Kv : (SYS == 1 ? a.Kt : a.Kq);
  const double *__restrict__ fl[NR];
  double *__restrict__ out[NR];
  if constexpr (SYS == 0) {
    fl[0] = a.MomX;
    fl[1] = a.MomY;
    out[0] = a.DU;
    out[1] = a.DV;
  } else if constexpr (SYS == 1) {
    fl[0] = a.Heat;
    out[0] = a.DT;
  } else {
    fl[0] = a.QFlx + n * (long long)(K + 1) * tracer;
    out[0] = a.DQ + n * (long long)K * tracer;
  }
  double *mat = a.mtx + SYS * n * K;
  const bool store_mat = SYS != 2 || tracer == 0;
  // values at level k carried from the previous (upper) iteration
  double flk[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) flk[r] = fl[r][c + n * K];
  double Kdk = 0.0, Gk = 0.0, Ehk = 0.0;  // of half level k (0 at the top)
  double ief_k1 = 0.0, ief_k = SYS == 1 ? a.IEF[c + n * (K - 1)] : 0.0;
  double m0p = 0.0, rp[NR] = {}, m0_2 = 0.0, r_2[NR], c2[NR], tc1 = 0.0, dfadt1 = 0.0, dfadt2 = 0.0;
  // the integer forms: the transfer coefficient of half level k (SYS 1: times
  // Cp Exner_h), 1 / a
  UF upU{1ull << 63, 0}, qU{1ull << 63, 0};
  bool upv = false, qv = false;
  bool efv = SYS == 1 && usual(ief_k);  // full level k's Exner function
  // half level k-1 and full level k-1 of the coming level k
  double Mn = 0.0, Gn = 0.0, Kdn = 0.0, Ehn = 0.0, Iefn = 0.0, fln[NR];
  auto fetch = [&](int k) {
    if (k < 1) return;
    Mn = a.Mass[c + n * (k - 1)];
    if (k > 1) {
      Gn = a.G[c + n * (k - 1)];
      Kdn = Kd[c + n * (k - 1)];
      if (SYS == 1) {
        Ehn = a.Eh[c + n * (k - 1)];
        Iefn = a.IEF[c + n * (k - 2)];
      }
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) fln[r] = fl[r][c + n * (k - 1)];
  };
  fetch(K);
#pragma unroll 1
  for (int k = K; k >= 1; --k) {
    const double Mm = Mn, Gm = Gn, Kdm = Kdn, Ehm = Ehn;
    double flm[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) flm[r] = fln[r];
    const double ief_km = SYS == 1 && k > 1 ? Iefn : 0.0;
    fetch(k - 1);
    // transfer coefficient of half level k-1 (SYS 1: times Cp Exner_h)
    UF lowU{1ull << 63, 0};
    const bool efm = SYS == 1 && usual(ief_km);
    bool lv = false;
    if (k > 1) {
      // every factor of the two couplings across this half level: M(k,-1) and
      // M(k-1,1) hold the Exner functions of both its full levels
      lv = a.fast && usual(Kdm) && usual(Gm);
      if (SYS == 1) lv = lv && usual(Ehm) && efv && efm;
      lowU = fx::mul(fx::from_double(Kdm), fx::from_double(Gm));
      if (SYS == 1) lowU = fx::mul(fx::mul(lowU, a.uCp), fx::from_double(Ehm));
      lowU = fx::norm(lowU);
    }
    double b[NR], re[NR], m0e;
#pragma unroll
    for (int r = 0; r < NR; ++r) b[r] = flm[r] - flk[r];
    bool done = false;
    if (lv && upv && qv && usual(Mm)) {
      // row k: its diagonal mass + l' + u', the couplings l and u (SYS 1: the
      // couplings with their own level's Exner function, l' and u' with k's)
      UF mU = fx::from_double(Mm), l = lowU, u = upU, l0 = lowU, u0 = upU;
      if (SYS == 1) {
        const UF ik = fx::from_double(ief_k);
        mU = fx::mul(mU, a.uCp);
        l0 = fx::mul(lowU, ik);
        u0 = fx::mul(upU, ik);
        l = fx::norm(fx::mul(lowU, fx::from_double(ief_km)));
        u = fx::mul(upU, fx::from_double(ief_k1));
      }
      const UF cU = fx::mul(u, qU);
      UF dU;
      if (fx::sub(fx::sum3(mU, l0, u0), cU, dU)) {
        const UF iU = fx::rcp(l);
        qU = fx::mul(l, fx::rcp(dU));
        const double il = fx::to_double(iU), cc = fx::to_double(cU);
        m0e = negd(fx::to_double(fx::mul(dU, iU)));
#pragma unroll
        for (int r = 0; r < NR; ++r) re[r] = fma(cc, rp[r], -b[r]) * il;
        done = true;
      }
    }
    if (!done) {
      // row k as the reference builds (:182-256) and eliminates it; +0
      // where it assigns 0
      const double tkm = k > 1 ? Kdm * Gm : 0.0, tck = Kdk * Gk;
      double mm, m0, mp;
      if constexpr (SYS != 1) {
        m0 = Mm + tkm + tck;
        mm = k > 1 ? -tkm : 0.0;
        mp = k < K ? -tck : 0.0;
        if (k == 1) tc1 = tck;
      } else {
        const double ehm = k > 1 ? a.CpDry * Ehm * tkm : 0.0, ehk = a.CpDry * Ehk * tck;
        m0 = a.CpDry * Mm + ehm * ief_k + ehk * ief_k;
        mm = k > 1 ? -(ehm * ief_km) : 0.0;
        mp = k < K ? -(ehk * ief_k1) : 0.0;
        if (k == 1) {
          dfadt1 = ehk * ief_k;  // DFADT1 = Cp Exner_h(1) TTC(1) / Exner_f(1)
          dfadt2 = mp;           // DFADT2 = -Cp Exner_h(1) TTC(1) / Exner_f(2)
        }
      }
      const Row w = eliminate_fp64(k == K, mm, m0, mp, m0p, b[0], b[NR - 1], rp[0], rp[NR - 1]);
      m0e = w.m0;
      re[0] = w.r[0];
      if (NR == 2) re[NR - 1] = w.r[1];
      qU = fx::rcp(fx::from_double(negd(m0e)));
    }
    qv = pos_in(negd(m0e), 723, 1323);
    upU = lowU;
    upv = lv;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      if (k == 1) c2[r] = b[r];  // ImplCplCoef2 starts from the level-1 divergence (:310-313)
      out[r][c + n * (k - 1)] = re[r];
      rp[r] = re[r];
      if (k == 2) r_2[r] = re[r];
      flk[r] = flm[r];
    }
    if (store_mat) mat[c + n * (k - 1)] = m0e;
    if (k == 2) m0_2 = m0e;
    m0p = m0e;
    ief_k1 = ief_k;
    ief_k = ief_km;
    efv = efm;
    if (k > 1) {
      Kdk = Kdm;
      Gk = Gm;
      if (SYS == 1) Ehk = Ehm;
    }
  }
  // coupling coefficients (:342-375); DFADUV1 = -DFADUV2 = TC(1)
  const double Tmp = a.Mass[c];
  const double i2 = fx::rcp_d(m0_2);
  if constexpr (SYS == 0) {
    const double cu = Tmp + tc1 + tc1 * i2;
    a.C1[c + n * 0] = cu;
    a.C2[c + n * 0] = c2[0] + tc1 * r_2[0] * i2;
    a.C1[c + n * 1] = cu;
    a.C2[c + n * 1] = c2[1] + tc1 * r_2[1] * i2;
  } else if constexpr (SYS == 1) {
    a.C1[c + n * 2] = a.CpDry * Tmp + dfadt1 - dfadt2 * i2;
    a.C2[c + n * 2] = c2[0] - dfadt2 * r_2[0] * i2;
  } else {
    if (tracer == a.ih2o - 1) {
      a.C1[c + n * 3] = Tmp + tc1 + tc1 * i2;
      a.C2[c + n * 3] = c2[0] + tc1 * r_2[0] * i2;
    }
  }
}

__global__ void __launch_bounds__(128, 4) forward_kernel(const Fwd a) {
  pdl_wait();
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= a.ncol) return;
  if (blockIdx.y == 0) forward_column<0>(a, c, 0);
  else if (blockIdx.y == 1) forward_column<1>(a, c, 0);
  else forward_column<2>(a, c, blockIdx.y - 2);
}

// Back substitution (:407-420) and the division by 2 dt (:53-61), one
// thread per (column, matrix): blockIdx.y 0 = momentum (U and V), 1 =
// temperature, 2 = the tracers; one reciprocal of M(k,0) per level serves
// every right-hand side of the matrix, and the next LVB levels are fetched
// while the chains run through the current ones.  M(k,-1) is 1 after the forward sweep and is
// not read; the reciprocals and the products with 1 / (2 dt) run on the
// integer pipes.
struct Bwd {
  const double *mtx;  // M(k,0) of UV, Temp and QMix
  double *DU, *DV, *DT, *DQ;
  long long ncol;
  int kmax, ncmax;
  double inv_2dt;
  fx::UF u2dt;  // inv_2dt
};

template <int NR>
__device__ __forceinline__ void backward_chains(const double *__restrict__ mat, double *x0, double *x1, long long c,
                                                long long n, int K, double inv_2dt, fx::UF u2dt) {
  double *x[2] = {x0, x1};
  double v[NR];
  double xs[LVB][NR], m0[LVB];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LVB; ++i)
      if (k0 + i <= K) {
        const long long o = c + n * (k0 + i - 1);
#pragma unroll
        for (int r = 0; r < NR; ++r) xs[i][r] = x[r][o];
        m0[i] = mat[o];
      }
  };
#pragma unroll
  for (int r = 0; r < NR; ++r) v[r] = x[r][c];
  load(2);
#pragma unroll
  for (int r = 0; r < NR; ++r) x[r][c] = fx::scale_d(v[r], u2dt, inv_2dt);
#pragma unroll 1
  for (int k0 = 2; k0 <= K; k0 += LVB) {
    double ys[LVB][NR], p0[LVB];
#pragma unroll
    for (int i = 0; i < LVB; ++i) {
      p0[i] = m0[i];
#pragma unroll
      for (int r = 0; r < NR; ++r) ys[i][r] = xs[i][r];
    }
    load(k0 + LVB);
#pragma unroll
    for (int i = 0; i < LVB; ++i) {
      if (k0 + i > K) break;
      const long long o = c + n * (k0 + i - 1);
      const double im = fx::rcp_d(p0[i]);
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        v[r] = (ys[i][r] - v[r]) * im;
        x[r][o] = fx::scale_d(v[r], u2dt, inv_2dt);
      }
    }
  }
}

__global__ void __launch_bounds__(32, 32) backward_kernel(const Bwd a) {
  const long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (c >= a.ncol) return;
  const long long n = a.ncol;
  const int K = a.kmax, y = blockIdx.y;
  const double *mat = a.mtx + y * n * K;
  // tracers in pairs (one reciprocal per level for both)
  const int nx = y == 0 ? 2 : y == 1 ? 1 : a.ncmax;
  for (int t = 0; t < nx; t += 2) {
    double *x0 = y == 0 ? a.DU : y == 1 ? a.DT : a.DQ + n * (long long)K * t;
    double *x1 = y == 0 ? a.DV : x0 + n * (long long)K;
    if (t + 1 < nx) backward_chains<2>(mat, x0, x1, c, n, K, a.inv_2dt, a.u2dt);
    else backward_chains<1>(mat, x0, nullptr, c, n, K, a.inv_2dt, a.u2dt);
  }
}

}  // namespace implcpl
}  // namespace dccm

using namespace dccm;

extern "C" int dccm_implcpl_create(int ncol, int kmax, int ncmax, int index_h2ovap,
                                   const dccm_implcpl_consts *consts, dccm_implcpl **plan) {
  DCCM_NVTX_FUNC();
  if (!plan || !consts) return DCCM_ERR_INVALID_ARG;
  *plan = nullptr;
  if (ncol < 1 || kmax < 2 || ncmax < 1 || index_h2ovap < 1 || index_h2ovap > ncmax) return DCCM_ERR_INVALID_ARG;
  if (!(consts->Grav > 0.0) || !(consts->DelTime > 0.0)) return DCCM_ERR_INVALID_ARG;
  dccm_implcpl *p = new (std::nothrow) dccm_implcpl();
  if (!p) return DCCM_ERR_NOMEM;
  p->ncol = ncol;
  p->kmax = kmax;
  p->ncmax = ncmax;
  p->ih2o = index_h2ovap;
  p->k = *consts;
  const cudaError_t e = cudaMalloc(&p->d_mtx, (size_t)6 * kmax * ncol * sizeof(double));
  if (e != cudaSuccess) {
    set_cuda_error(e);
    delete p;
    return DCCM_ERR_CUDA;
  }
  *plan = p;
  return DCCM_OK;
}

extern "C" int dccm_implcpl_destroy(dccm_implcpl *p) {
  DCCM_NVTX_FUNC();
  if (!p) return DCCM_OK;
  if (p->d_mtx) cudaFree(p->d_mtx);
  p->stage.release();
  if (p->stream) cudaStreamDestroy(p->stream);
  delete p;
  return DCCM_OK;
}

static size_t mstride(const dccm_implcpl *p) { return (size_t)p->kmax * p->ncol; }

// A constant the integer arithmetic takes: positive, within 2^+-100.
static bool ordinary(double x) { return x > 0x1p-100 && x < 0x1p100; }

extern "C" int dccm_implcpl_forward_dev(dccm_implcpl *p, const dccm_implcpl_forward_args *a, void *stream) {
  DCCM_NVTX_FUNC();
  if (!p || !a) return DCCM_ERR_INVALID_ARG;
  const void *need[] = {a->xyr_MomFluxX, a->xyr_MomFluxY, a->xyr_HeatFlux, a->xyrf_QMixFlux, a->xyr_Press,
                        a->xyz_Exner, a->xyr_Exner, a->xyr_VirTemp, a->xyz_Height, a->xyr_VelDiffCoef,
                        a->xyr_TempDiffCoef, a->xyr_QMixDiffCoef, a->xyz_DUDt, a->xyz_DVDt, a->xyz_DTempDt,
                        a->xyzf_DQMixDt, a->xya_ImplCplCoef1, a->xya_ImplCplCoef2};
  for (const void *q : need)
    if (!q) return DCCM_ERR_INVALID_ARG;
  implcpl::Fwd f;
  f.MomX = a->xyr_MomFluxX;
  f.MomY = a->xyr_MomFluxY;
  f.Heat = a->xyr_HeatFlux;
  f.QFlx = a->xyrf_QMixFlux;
  f.P = a->xyr_Press;
  f.Ef = a->xyz_Exner;
  f.Eh = a->xyr_Exner;
  f.Tv = a->xyr_VirTemp;
  f.Z = a->xyz_Height;
  f.Kv = a->xyr_VelDiffCoef;
  f.Kt = a->xyr_TempDiffCoef;
  f.Kq = a->xyr_QMixDiffCoef;
  f.DU = a->xyz_DUDt;
  f.DV = a->xyz_DVDt;
  f.DT = a->xyz_DTempDt;
  f.DQ = a->xyzf_DQMixDt;
  f.C1 = a->xya_ImplCplCoef1;
  f.C2 = a->xya_ImplCplCoef2;
  f.mtx = p->d_mtx;
  f.ncol = p->ncol;
  f.kmax = p->kmax;
  f.ncmax = p->ncmax;
  f.ih2o = p->ih2o;
  f.Grav = p->k.Grav;
  f.CpDry = p->k.CpDry;
  f.GasR = p->k.GasRDry;
  f.inv_g2dt = 1.0 / (p->k.Grav * (2.0 * p->k.DelTime));
  f.G = p->d_mtx + 3 * mstride(p);
  f.IEF = f.G + mstride(p);
  f.Mass = f.IEF + mstride(p);
  f.fast = ordinary(f.CpDry) && ordinary(f.GasR);
  f.uCp = fx::uf(f.fast ? f.CpDry : 1.0);
  f.uGasR = fx::uf(f.fast ? f.GasR : 1.0);
  const long long nk = (long long)p->ncol * ((p->kmax + implcpl::GL - 1) / implcpl::GL);
  implcpl::geo_kernel<<<(unsigned)((nk + 255) / 256), 256, 0, as_stream(stream)>>>(f);
  DCCM_LAUNCH_CHECK();
  const int threads = 128;
  DCCM_CUDA(launch_dependent(implcpl::forward_kernel, dim3((unsigned)((p->ncol + threads - 1) / threads), 2 + p->ncmax),
                             dim3(threads), 0, as_stream(stream), f));
  return DCCM_OK;
}

extern "C" int dccm_implcpl_backward_dev(dccm_implcpl *p, double *xyz_DUDt, double *xyz_DVDt,
                                         double *xyz_DTempDt, double *xyzf_DQMixDt, void *stream) {
  DCCM_NVTX_FUNC();
  if (!p || !xyz_DUDt || !xyz_DVDt || !xyz_DTempDt || !xyzf_DQMixDt) return DCCM_ERR_INVALID_ARG;
  implcpl::Bwd b;
  b.mtx = p->d_mtx;
  b.DU = xyz_DUDt;
  b.DV = xyz_DVDt;
  b.DT = xyz_DTempDt;
  b.DQ = xyzf_DQMixDt;
  b.ncol = p->ncol;
  b.kmax = p->kmax;
  b.ncmax = p->ncmax;
  b.inv_2dt = 1.0 / (2.0 * p->k.DelTime);
  // an exponent that sends every product to the FP64 form where 1 / (2 dt) is not ordinary
  b.u2dt = ordinary(b.inv_2dt) ? fx::uf(b.inv_2dt) : fx::UF{0, 0};
  const int threads = 32;
  implcpl::backward_kernel<<<dim3((unsigned)((p->ncol + threads - 1) / threads), 3), threads, 0,
                             as_stream(stream)>>>(b);
  DCCM_LAUNCH_CHECK();
  return DCCM_OK;
}

extern "C" int dccm_implcpl_info(const dccm_implcpl *p, int *ncol, int *kmax, int *ncmax) {
  if (!p) return DCCM_ERR_INVALID_ARG;
  if (ncol) *ncol = (int)p->ncol;
  if (kmax) *kmax = p->kmax;
  if (ncmax) *ncmax = p->ncmax;
  return DCCM_OK;
}

// Host entry points: stage through the plan's device buffer.
static int host_stream(dccm_implcpl *p) {
  if (!p->stream) DCCM_CUDA(cudaStreamCreateWithFlags(&p->stream, cudaStreamNonBlocking));
  return DCCM_OK;
}

extern "C" int dccm_implcpl_forward(dccm_implcpl *p, const dccm_implcpl_forward_args *a) {
  DCCM_NVTX_FUNC();
  if (!p || !a) return DCCM_ERR_INVALID_ARG;
  DCCM_TRY(host_stream(p));
  const size_t n = p->ncol, K = p->kmax, nc = p->ncmax;
  const size_t half = n * (K + 1), full = n * K;
  // inputs: 9 half-level arrays, 2 full-level, tracer fluxes; outputs: 3 full,
  // tracer tendencies, 2 x 4 coefficients
  const size_t tot = 9 * half + 2 * full + nc * half + 3 * full + nc * full + 8 * n;
  DCCM_TRY(p->stage.ensure(tot * sizeof(double)));
  double *d = static_cast<double *>(p->stage.ptr);
  const double *hin[] = {a->xyr_MomFluxX, a->xyr_MomFluxY, a->xyr_HeatFlux, a->xyr_Press, a->xyr_Exner,
                         a->xyr_VirTemp, a->xyr_VelDiffCoef, a->xyr_TempDiffCoef, a->xyr_QMixDiffCoef};
  for (const double *q : hin)
    if (!q) return DCCM_ERR_INVALID_ARG;
  if (!a->xyz_Exner || !a->xyz_Height || !a->xyrf_QMixFlux || !a->xyz_DUDt || !a->xyz_DVDt ||
      !a->xyz_DTempDt || !a->xyzf_DQMixDt || !a->xya_ImplCplCoef1 || !a->xya_ImplCplCoef2)
    return DCCM_ERR_INVALID_ARG;
  double *dh[9];
  size_t off = 0;
  for (int i = 0; i < 9; ++i, off += half) {
    dh[i] = d + off;
    DCCM_CUDA(cudaMemcpyAsync(dh[i], hin[i], half * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  }
  double *dEf = d + off;
  off += full;
  double *dZ = d + off;
  off += full;
  double *dQF = d + off;
  off += nc * half;
  DCCM_CUDA(cudaMemcpyAsync(dEf, a->xyz_Exner, full * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(dZ, a->xyz_Height, full * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(dQF, a->xyrf_QMixFlux, nc * half * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  dccm_implcpl_forward_args g;
  g.xyr_MomFluxX = dh[0];
  g.xyr_MomFluxY = dh[1];
  g.xyr_HeatFlux = dh[2];
  g.xyr_Press = dh[3];
  g.xyr_Exner = dh[4];
  g.xyr_VirTemp = dh[5];
  g.xyr_VelDiffCoef = dh[6];
  g.xyr_TempDiffCoef = dh[7];
  g.xyr_QMixDiffCoef = dh[8];
  g.xyz_Exner = dEf;
  g.xyz_Height = dZ;
  g.xyrf_QMixFlux = dQF;
  g.xyz_DUDt = d + off;
  off += full;
  g.xyz_DVDt = d + off;
  off += full;
  g.xyz_DTempDt = d + off;
  off += full;
  g.xyzf_DQMixDt = d + off;
  off += nc * full;
  g.xya_ImplCplCoef1 = d + off;
  off += 4 * n;
  g.xya_ImplCplCoef2 = d + off;
  DCCM_TRY(dccm_implcpl_forward_dev(p, &g, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xyz_DUDt, g.xyz_DUDt, full * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xyz_DVDt, g.xyz_DVDt, full * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xyz_DTempDt, g.xyz_DTempDt, full * sizeof(double), cudaMemcpyDeviceToHost,
                            p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xyzf_DQMixDt, g.xyzf_DQMixDt, nc * full * sizeof(double), cudaMemcpyDeviceToHost,
                            p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xya_ImplCplCoef1, g.xya_ImplCplCoef1, 4 * n * sizeof(double),
                            cudaMemcpyDeviceToHost, p->stream));
  DCCM_CUDA(cudaMemcpyAsync(a->xya_ImplCplCoef2, g.xya_ImplCplCoef2, 4 * n * sizeof(double),
                            cudaMemcpyDeviceToHost, p->stream));
  DCCM_CUDA(cudaStreamSynchronize(p->stream));
  return DCCM_OK;
}

extern "C" int dccm_implcpl_backward(dccm_implcpl *p, double *xyz_DUDt, double *xyz_DVDt, double *xyz_DTempDt,
                                     double *xyzf_DQMixDt) {
  DCCM_NVTX_FUNC();
  if (!p || !xyz_DUDt || !xyz_DVDt || !xyz_DTempDt || !xyzf_DQMixDt) return DCCM_ERR_INVALID_ARG;
  DCCM_TRY(host_stream(p));
  const size_t full = (size_t)p->ncol * p->kmax, nc = p->ncmax;
  DCCM_TRY(p->stage.ensure((3 + nc) * full * sizeof(double)));
  double *d = static_cast<double *>(p->stage.ptr);
  double *h[4] = {xyz_DUDt, xyz_DVDt, xyz_DTempDt, xyzf_DQMixDt};
  const size_t len[4] = {full, full, full, nc * full};
  double *dv[4];
  size_t off = 0;
  for (int i = 0; i < 4; ++i) {
    dv[i] = d + off;
    off += len[i];
    DCCM_CUDA(cudaMemcpyAsync(dv[i], h[i], len[i] * sizeof(double), cudaMemcpyHostToDevice, p->stream));
  }
  DCCM_TRY(dccm_implcpl_backward_dev(p, dv[0], dv[1], dv[2], dv[3], p->stream));
  for (int i = 0; i < 4; ++i)
    DCCM_CUDA(cudaMemcpyAsync(h[i], dv[i], len[i] * sizeof(double), cudaMemcpyDeviceToHost, p->stream));
  DCCM_CUDA(cudaStreamSynchronize(p->stream));
  return DCCM_OK;
}

extern "C" int dccm_implcpl_matrices(dccm_implcpl *p, double *uv, double *temp, double *qmix) {
  DCCM_NVTX_FUNC();
  if (!p) return DCCM_ERR_INVALID_ARG;
  double *h[3] = {uv, temp, qmix};
  const size_t n = mstride(p);
  for (int i = 0; i < 3; ++i)
    if (h[i]) {
      DCCM_CUDA(cudaMemcpy(h[i] + n, p->d_mtx + i * n, n * sizeof(double), cudaMemcpyDeviceToHost));
      std::fill(h[i], h[i] + n, 1.0);
      std::fill(h[i] + 2 * n, h[i] + 3 * n, 0.0);
    }
  return DCCM_OK;
}
