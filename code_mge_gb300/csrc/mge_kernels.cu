// mge_kernels.cu -- sm_103a kernels of code_mge's multigrid Runge-Kutta cycle.
//
// GB300 executes FP64 at 1/58 of its FP32 rate (about 0.6 TFMA/s against
// 6.8 TB/s of HBM), so an all-FP64 JST stage is bound by FP64 issue, not by
// memory.  The stage is therefore split so that every per-cell and per-face
// quantity is evaluated exactly once (the reference re-evaluates each cell
// flux for both faces), with the intermediates kept in HBM/L2:
//
//   k_prep     per cell: 1/rho, rho*E+p, the cell flux F(w).s for i/j/k
//              (ceflux, eflux.f90:133-155) and the pressure sensors
//              (dflux.f90:71-76,131-136,188-193)
//   k_face_*   per face: averaged convective flux (eflux.f90:42-98) and the
//              blended 2nd/4th-difference dissipation (dflux.f90:82-112)
//   k_rec_*    per cut-cell record: the efluxb/dfluxb face replacements
//   k_combine  per cell: dw, fw, forcing, blanking, time-step scaling and,
//              without smoothing, the update + depvars (euler.f90:127-399)
//   k_irs_*    implicit residual smoothing lines (psmoo.f90:171-237)
//   k_update   the state after smoothing and depvars (euler.f90:375-399)
//   k_bcond    boundary conditions and the records' solid states
//
// Arithmetic follows the reference expression by expression.  The plain path
// is compiled with --fmad=false (no contraction); divisions by a quantity
// whose reciprocal is already known use Markstein's correction
// (q0 = a*y, r = fma(-q0,b,a), q = fma(r,y,q0) with y = RN(1/b)), which
// returns the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34,
// 1990), so results stay bit-identical to IEEE a/b at a third of its cost.
#include <cmath>
#include <cstdio>
#include <cstdlib>

#include <cooperative_groups.h>
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "exact_ops.cuh"
#include "fast_pow.cuh"
#include "mge_internal.h"
#include "soft_fp64.cuh"

namespace cg = cooperative_groups;

// The file is compiled once per part, in parallel: 0 the launchers on FP64
// blocks (and what belongs to no precision), 1 those on FP32 blocks, 2 the
// launches over several cases.
#ifndef MGE_PART
#error "compile with -DMGE_PART=0, 1 and 2"
#endif

namespace mge {

// --------------------------------------------------------------- helpers
// a * b, for doubles on the integer pipes (soft_fp64.cuh: the same bits as
// the FP64 multiply), so that a kernel bound by the FP64 issue rate can move
// some of its independent products off the FP64 pipe
__device__ __forceinline__ double smul(double a, double b) { return soft::mul(a, b); }
__device__ __forceinline__ float smul(float a, float b) { return a * b; }
// a / b, for doubles on the integer pipes (the same bits as the FP64
// division, which costs about ten FP64 instructions)
__device__ __forceinline__ double sdiv(double a, double b) { return soft::div(a, b); }
__device__ __forceinline__ float sdiv(float a, float b) { return a / b; }
__device__ __forceinline__ double mdiv(double a, double b, double y) {
  double q = a * y;
  double r = fma(-q, b, a);
  return fma(r, y, q);
}
__device__ __forceinline__ float mdiv(float a, float b, float y) {
  float q = a * y;
  float r = fmaf(-q, b, a);
  return fmaf(r, y, q);
}
// mdiv with its first product on the integer pipes (smul, below): the same
// quotient
__device__ __forceinline__ double smul(double a, double b);
__device__ __forceinline__ double smdiv(double a, double b, double y) {
  double q = smul(a, y);
  double r = fma(-q, b, a);
  return fma(r, y, q);
}
__device__ __forceinline__ float smdiv(float a, float b, float y) { return mdiv(a, b, y); }
// the same by choice: S takes the integer pipes.  They win where a kernel is
// bound by the FP64 rate; a level of few cells is bound by the latency of its
// dependent chains, and there the plain operations are the shorter ones (a
// product 32 cycles against about 100).  The bits are the same either way.
template <bool S, typename T> __device__ __forceinline__ T pmul(T a, T b) {
  if constexpr (S) return smul(a, b); else return a * b;
}
template <bool S, typename T> __device__ __forceinline__ T pdiv(T a, T b) {
  if constexpr (S) return sdiv(a, b); else return a / b;
}
template <bool S, typename T> __device__ __forceinline__ T pmdiv(T a, T b, T y) {
  if constexpr (S) return smdiv(a, b, y); else return mdiv(a, b, y);
}
// Quotients by one divisor b: a/b and (a*w)/b, each operation rounded.  With the
// integer pipes nothing is left on the FP64 pipe (soft::mulquot_normal); without,
// one reciprocal and Markstein's quotient.  The same bits as the divisions; a
// divisor that is zero or infinite, an infinite dividend and a quotient that
// overflows give NaN in both, as mdiv does (the time step stops there).
template <bool S, typename T> struct SharedDiv {
  T b, y;
  __device__ __forceinline__ explicit SharedDiv(T d) : b(d), y(pdiv<S>(T(1), d)) {}
  __device__ __forceinline__ T quot(T a) const { return pmdiv<S>(a, b, y); }
  __device__ __forceinline__ T mulquot(T a, T w) const { return pmdiv<S>(pmul<S>(a, w), b, y); }
};
// out of line, for what lies outside the normal range
static __device__ __noinline__ double mdiv_of(double a, double b) { return mdiv(a, b, 1.0 / b); }
static __device__ __noinline__ double muldiv_of(double a, double w, double b) { return mdiv(a * w, b, 1.0 / b); }
template <> struct SharedDiv<true, double> {
  double b;
  soft::Recip r;
  __device__ __forceinline__ explicit SharedDiv(double d) : b(d), r(soft::recip(d)) {}
  __device__ __forceinline__ double quot(double a) const {
    double q;
    return soft::quot_normal(a, r, q) ? q : mdiv_of(a, b);
  }
  __device__ __forceinline__ double mulquot(double a, double w) const {
    double q;
    return soft::mulquot_normal(a, w, r, q) ? q : muldiv_of(a, w, b);
  }
};
// cell (or face) t of a box of nx by ny by any number of cells, counted from
// (i0, i0, i0).  A block's scratch alone holds 64 fields, so its cells number
// fewer than 2^31 on any device and 32-bit divisions suffice (a 64-bit one
// costs about ten times as much).
__device__ __forceinline__ void cell_of(long long t, int nx, int ny, int i0, int& i, int& j, int& k) {
  const unsigned u = (unsigned)t, q = u / (unsigned)nx, r = q / (unsigned)ny;
  i = i0 + (int)(u - q * (unsigned)nx);
  j = i0 + (int)(q - r * (unsigned)ny);
  k = i0 + (int)r;
}
// reciprocals the host prepares once, RN(1/x) of the divisor x in the
// block's precision, so that mdiv gives the correctly rounded quotient
__device__ __forceinline__ double rcp_gm1(const PhysParams& P, double) { return P.rgm1; }
__device__ __forceinline__ float rcp_gm1(const PhysParams& P, float) { return P.rgm1f; }
__device__ __forceinline__ double rcp_gamma(const PhysParams& P, double) { return P.rgamma; }
__device__ __forceinline__ float rcp_gamma(const PhysParams& P, float) { return P.rgammaf; }
__device__ __forceinline__ double rcp_h(const DevBlock<double>& b, int d) { return b.rh[d]; }
__device__ __forceinline__ float rcp_h(const DevBlock<float>& b, int d) { return b.rhf[d]; }
__device__ __forceinline__ double rcp_4h(const DevBlock<double>& b, int d) { return b.r4h[d]; }
__device__ __forceinline__ float rcp_4h(const DevBlock<float>& b, int d) { return b.r4hf[d]; }
__device__ __forceinline__ double rcp_vol(const DevBlock<double>& b) { return b.rvol; }
__device__ __forceinline__ float rcp_vol(const DevBlock<float>& b) { return b.rvolf; }
// the line-sweep pivots in the sweep's precision (the FP32 sweeps read the
// single-precision tables: no conversion per cell)
__device__ __forceinline__ double irs_e1(const IrsTables& t, int q, double) { return t.e1[q]; }
__device__ __forceinline__ float irs_e1(const IrsTables& t, int q, float) { return t.e1f[q]; }
__device__ __forceinline__ double irs_e1r(const IrsTables& t, int q, double) { return t.e1r[q]; }
__device__ __forceinline__ float irs_e1r(const IrsTables& t, int q, float) { return t.e1rf[q]; }
// x / e1[q] as fma(x, e1r, x*e1l), with e1r + e1l = 1/e1 to twice the precision: one
// dependent operation fewer than Markstein's quotient.  The host has checked that
// it rounds as the division for every finite x whose products and quotient are
// normal numbers (IrsTables::quick).  An infinite x gives infinity or NaN by the
// sign of e1l, where mdiv gives NaN; the residual norm counts both as NaN.
template <bool SC> __device__ __forceinline__ double irs_quick(double x, double e1r, double e1l) {
  return fma(x, e1r, SC ? smul(x, e1l) : x * e1l);
}
__device__ __forceinline__ double irs_e2(const IrsTables& t, int q, double) { return t.e2[q]; }
__device__ __forceinline__ float irs_e2(const IrsTables& t, int q, float) { return t.e2f[q]; }
template <typename T> __device__ __forceinline__ T fdimT(T a, T b) { return a > b ? a - b : T(0); }
template <typename T> __device__ __forceinline__ T fmaxT(T a, T b) { return a > b ? a : b; }
template <typename T> __device__ __forceinline__ T fminT(T a, T b) { return a < b ? a : b; }

// depvars_one, depvars.f90:48-49
template <bool S = true, typename T = double> __device__ __forceinline__ T depvars(T gamma, const T* w) {
  // the products on the integer pipes and the halving as an exponent step:
  // the same bits as 0.5*(w1*w1 + w2*w2 + w3*w3)/w0 and (gamma-1)*dim(w4, qq)
  T qq = pdiv<S>(mulhalf(pmul<S>(w[1], w[1]) + pmul<S>(w[2], w[2]) + pmul<S>(w[3], w[3])), w[0]);
  return pmul<S>(gamma - T(1), fdimT(w[4], qq));
}

struct Idx {
  int i, j, k;
};
__device__ __forceinline__ long long cidx(int Pi, int Pj, int i, int j, int k) {
  return (long long)i + (long long)Pi * ((long long)j + (long long)Pj * (long long)k);
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

// --------------------------------------------------------------- timestep (timestep.f90:39-115)
// TC is the arithmetic precision (FP64 in the plain path, FP32 in the mixed one).
template <typename T, typename TC, bool S, bool SAVE>
__device__ __forceinline__ unsigned long long body_timestep(const DevBlock<T>& b, const PhysParams& P, unsigned* err,
                                                            long long t) {
  const int nxl = b.nx, nyl = b.ny;
  unsigned long long mine = ~0ull;  // bits of this cell's vdtim for the global minimum
  int i, j, k;
  cell_of(t, nxl, nyl, 2, i, j, k);
  const long long N = b.N;
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  const TC gamma = (TC)P.gamma;
  TC w0 = (TC)b.w[c], w1 = (TC)b.w[N + c], w2 = (TC)b.w[2 * N + c], w3 = (TC)b.w[3 * N + c];
  if (SAVE) {
#pragma unroll
    for (int v = 0; v < 5; v++) b.wn[v * N + c] = b.w[v * N + c];
  }
  TC pc = (TC)b.p[c];
  const SharedDiv<S, TC> rho(w0);
  TC cc = rho.mulquot(gamma, pc);
  if (cc < TC(0) || cc != cc) {  // timestep.f90:45-48
    atomicCAS(err, 0u, (unsigned)ERR_NEGPRESS);  // the first stop in launch order wins
    return mine;
  }
  cc = sqrt(fmaxT(cc, TC(0)));
  TC uu = rho.quot(w1), uv = rho.quot(w2), uw = rho.quot(w3);
  // face vectors are axis-aligned: |u.s| = |u_d s_d|, |s| precomputed
  TC ri = fabs(pmul<S>(uu, (TC)b.s[0])) + pmul<S>(cc, (TC)b.sqrt_ds[0]);
  TC rj = fabs(pmul<S>(uv, (TC)b.s[1])) + pmul<S>(cc, (TC)b.sqrt_ds[1]);
  TC rk = fabs(pmul<S>(uw, (TC)b.s[2])) + pmul<S>(cc, (TC)b.sqrt_ds[2]);
  TC lsum = ri + rj + rk;
  TC fict;
  if (P.eqn_ns) {  // viscous spectral radii, timestep.f90:141-178
    const TC fmue = pdiv<S>((TC)P.viscl, (TC)P.prlmean);
    const TC f1 = pdiv<S>(pdiv<S>(TC(4), w0), TC(3));
    const TC f2 = pdiv<S>(gamma, w0);
    const TC fac = fmaxT(f1, f2);
    const TC dtv = pdiv<S>(fac * fmue, (TC)b.vol);
    const TC s0 = (TC)b.s[0], s1 = (TC)b.s[1], s2 = (TC)b.s[2];
    TC rvi = dtv * (s0 * s0), rvj = dtv * (s1 * s1), rvk = dtv * (s2 * s2);
    fict = pdiv<S>((TC)b.vol, lsum + (TC)P.cfac * (rvi + rvj + rvk));
  } else {
    fict = pdiv<S>((TC)b.vol, lsum);
  }
  const TC plim = TC(0.001);
  TC pip = (TC)b.p[c + 1], pim = (TC)b.p[c - 1];
  TC pjp = (TC)b.p[c + b.Pi], pjm = (TC)b.p[c - b.Pi];
  long long pl = (long long)b.Pi * b.Pj;
  TC pkp = (TC)b.p[c + pl], pkm = (TC)b.p[c - pl];
  TC p2 = mul2(pc);
  TC dpi = fabs(pdiv<S>(pip - p2 + pim, pip + p2 + pim + plim));
  TC dpj = fabs(pdiv<S>(pjp - p2 + pjm, pjp + p2 + pjm + plim));
  TC dpk = fabs(pdiv<S>(pkp - p2 + pkm, pkp + p2 + pkm + plim));
  TC r = pdiv<S>(TC(1), TC(1) + fminT((TC)P.dimcfl, mul2(dpi + dpj + dpk)));
  if (P.unsteady) {  // timestep.f90:85-99,180-190: at most 2*dtstep/(3*cfl)
    const TC dtime = (TC(2) * (TC)P.dtstep) / (TC(3) * (TC)P.cfl);
    fict = fict < dtime ? fict : dtime;
  }
  TC vd = pmul<S>(fict, r);
  double vdd = (double)vd;
  if (vdd >= 0.0) mine = (unsigned long long)__double_as_longlong(vdd);
  if (b.blank[c] == 0) {  // timestep.f90:212-223
    b.vdtim[c] = T(0);
    b.lam[c] = T(0);
  } else {
    b.vdtim[c] = (T)vd;
    b.lam[c] = (T)lsum;
  }
  if (b.eps && P.smoo > 0.0) {
    // coefficients of the psmoo variant, timestep.f90:286-309; the radii of
    // blanked cells are zero there (timestep.f90:212-223), so their ratios
    // are 0/0 and the NaN-ignoring min/max give eps = smoo
    const bool bl = b.blank[c] == 0;
    const TC zi = bl ? TC(0) : ri, zj = bl ? TC(0) : rj, zk = bl ? TC(0) : rk;
    const TC smoo = (TC)P.smoo;
    const TC cflrat = sqrt(TC(1) + TC(4) * smoo);
    auto coef = [&](TC ra, TC rb, TC rc) -> TC {  // ra: this direction's radius
      TC reval = rb / ra + rc / ra;
      TC q = cflrat / (TC(1) + TC(0.0625) * reval);
      TC ex = TC(0.25) * (q * q - TC(1));
      ex = fmin(smoo, ex);
      return fmax(TC(0), ex);
    };
    b.eps[c] = (T)coef(zi, zj, zk);
    b.eps[N + c] = (T)coef(zj, zk, zi);
    b.eps[2 * N + c] = (T)coef(zk, zi, zj);
  }
  return mine;
}

// minimum over the calling block (vdtim >= 0, so the IEEE bit patterns order
// like the values), valid in thread 0; every thread of the block must call it
__device__ __forceinline__ unsigned long long block_min(unsigned long long mine) {
  __shared__ unsigned long long smin[32];
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long q = __shfl_down_sync(0xffffffffu, mine, o);
    mine = q < mine ? q : mine;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) smin[wid] = mine;
  __syncthreads();
  if (wid == 0) {
    mine = (lane < (int)(blockDim.x >> 5)) ? smin[lane] : ~0ull;
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long q = __shfl_down_sync(0xffffffffu, mine, o);
      mine = q < mine ? q : mine;
    }
  }
  return mine;
}
// dtim = min(10, every block's minimum): the blocks meet in dtim[1] (bits) and
// count themselves in dtim[2]; the last of nblocks writes dtim[0] and leaves the
// other two as it found them (~0 and 0), so no launch has to reset them
__device__ __forceinline__ void block_min_dtim(unsigned long long mine, double* dtim, int nblocks) {
  mine = block_min(mine);
  if (threadIdx.x != 0) return;
  unsigned long long* run = (unsigned long long*)(dtim + 1);
  unsigned* count = (unsigned*)(dtim + 2);
  if (mine != ~0ull) atomicMin(run, mine);
  __threadfence();
  if (atomicAdd(count, 1u) == (unsigned)nblocks - 1) {
    __threadfence();
    const unsigned long long m = atomicExch(run, ~0ull), ten = (unsigned long long)__double_as_longlong(10.0);
    *count = 0u;
    *dtim = __longlong_as_double((long long)(m < ten ? m : ten));
  }
}

// SAVE: wn = w as well (euler.f90:80-83), from the values the cell has loaded
template <typename T, typename TC, bool S, bool SAVE>
__global__ void k_timestep(DevBlock<T> b, PhysParams P, unsigned* err) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long mine = ~0ull;
  if (t < (long long)b.nx * b.ny * b.nz) mine = body_timestep<T, TC, S, SAVE>(b, P, err, t);
  block_min_dtim(mine, b.dtim, gridDim.x);  // global dtim (timestep.f90:112), kept even when vt = 0
}

// --------------------------------------------------------------- stage: per-cell pass
// Box [1..ie]x[1..je]x[1..ke]: every cell whose flux or sensor a face needs.
template <bool S, typename T>
__device__ __forceinline__ T van_albada(T a, T b, T e2);

// FAST: the contracted form of the mixed precision's finest level (JST
// central scheme, Euler): the cell flux takes the velocity q = (w_d s)/rho
// once and multiplies, F(v) = q w(v), instead of rounding each product
// before its division.  The result is the same quantity to an FP64 rounding
// or two, not the reference's bit pattern.
template <typename T, bool FAST = false, bool S = true>
__device__ __forceinline__ void body_prep(const DevBlock<T>& b, const PhysParams& P, int dissip_on, long long t) {
  const int ex = b.ie, ey = b.je;  // count = ie (cells 1..ie)
  int i, j, k;
  cell_of(t, ex, ey, 1, i, j, k);
  const long long N = b.N;
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  T w[5];
#pragma unroll
  for (int v = 0; v < 5; v++) w[v] = b.w[v * N + c];
  T p = b.p[c];
  T y = pdiv<S>(T(1), w[0]);
  T Hc = w[4] + p;
  b.H[c] = Hc;
  if (P.eqn_ns && dissip_on) {  // velocity and temperature, zero in solid cells (euler.f90:140-154)
    const bool solid = b.blank[c] == 0;
#pragma unroll
    for (int a = 0; a < 3; a++) b.vt[a * N + c] = solid ? T(0) : mdiv(w[1 + a], w[0], y);
    b.vt[3 * N + c] = solid ? T(0) : pdiv<S>(p, w[0] * (T)P.gas_const);
  }
  // the MUSCL Roe faces take their central flux from the reconstructed
  // states, not from the cell fluxes
  if (FAST) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const T s = (T)b.s[d];
      const T f0 = pmul<S>(w[1 + d], s);
      const T q = pmul<S>(f0, y);
      T f1 = pmul<S>(q, w[1]), f2 = pmul<S>(q, w[2]), f3 = pmul<S>(q, w[3]);
      if (d == 0) f1 = fma(p, s, f1);
      if (d == 1) f2 = fma(p, s, f2);
      if (d == 2) f3 = fma(p, s, f3);
      T* F = b.F + (long long)(d * 5) * N + c;
      F[0] = f0;
      F[N] = f1;
      F[2 * N] = f2;
      F[3 * N] = f3;
      F[4 * N] = pmul<S>(q, Hc);
    }
  } else if (P.distype != 2) {
#pragma unroll
    for (int d = 0; d < 3; d++) {
      // the products of this FP64-bound pass go to the integer pipes (smul);
      // the fused steps of the quotients stay on the FP64 pipe
      T s = (T)b.s[d];
      T f0 = pmul<S>(w[1 + d], s);  // sum(w(2:4)*ss) with the two zero components dropped
      T f1 = pmdiv<S>(pmul<S>(f0, w[1]), w[0], y);
      T f2 = pmdiv<S>(pmul<S>(f0, w[2]), w[0], y);
      T f3 = pmdiv<S>(pmul<S>(f0, w[3]), w[0], y);
      if (d == 0) f1 = f1 + pmul<S>(p, s);
      if (d == 1) f2 = f2 + pmul<S>(p, s);
      if (d == 2) f3 = f3 + pmul<S>(p, s);
      T f4 = pmdiv<S>(pmul<S>(f0, Hc), w[0], y);
      T* F = b.F + (long long)(d * 5) * N + c;
      F[0] = f0;
      F[N] = f1;
      F[2 * N] = f2;
      F[3 * N] = f3;
      F[4 * N] = f4;
    }
  }
  if (dissip_on && P.distype == 0) {
    // the differences the dissipation faces take (dflux.f90:95-99), once per
    // cell instead of once per face; the neighbour's enthalpy is formed
    // again with the same addition
    const long long sts[3] = {1, (long long)b.Pi, (long long)b.Pi * b.Pj};
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const long long cn = c - sts[d];
      T* Dl = b.dlt + (long long)(d * 5) * N + c;
#pragma unroll
      for (int v = 0; v < 4; v++) Dl[v * N] = w[v] - b.w[v * N + cn];
      Dl[4 * N] = Hc - (b.w[4 * N + cn] + b.p[cn]);
    }
  }
  if (dissip_on && P.distype == 0) {  // the pressure sensors of the JST faces
    const long long pl = (long long)b.Pi * b.Pj;
    // i: abs(p(i-1) +2p(i) +p(i+1)), dflux.f90:71-76
    {
      T pm = b.p[c - 1], pp = b.p[c + 1], p2 = mul2(p);
      T pb = fabs(pm + p2 + pp);
      b.fp[c] = (pb > T(0)) ? pdiv<S>(fabs(pm - p2 + pp), pb) : T(0);
    }
    // j: abs(p(j+1) +2p(j) +p(j-1)), dflux.f90:131-136
    {
      T pm = b.p[c - b.Pi], pp = b.p[c + b.Pi], p2 = mul2(p);
      T pb = fabs(pp + p2 + pm);
      b.fp[N + c] = (pb > T(0)) ? pdiv<S>(fabs(pp - p2 + pm), pb) : T(0);
    }
    // k: abs(p(k-1) +2p(k) +p(k+1)), dflux.f90:188-193
    {
      T pm = b.p[c - pl], pp = b.p[c + pl], p2 = mul2(p);
      T pb = fabs(pm + p2 + pp);
      b.fp[2 * N + c] = (pb > T(0)) ? pdiv<S>(fabs(pm - p2 + pp), pb) : T(0);
    }
  }
}

// One direction of the prep pass for the central scheme of the Euler
// equations: the cell flux, the differences and the sensor along D, at the
// cells a face along D reads (tangential indices physical).  Three times the
// threads of body_prep with a third of its chain each, for the levels that
// leave most of the chip idle.
template <typename T, bool FAST, bool S, int D>
__device__ __forceinline__ void body_prep_dir(const DevBlock<T>& b, const PhysParams& P, int dissip_on, int t) {
  const int n0 = b.nx + (D == 0 ? 2 : 0), n1 = b.ny + (D == 1 ? 2 : 0), n2 = b.nz + (D == 2 ? 2 : 0);
  if (t >= n0 * n1 * n2) return;
  int i, j, k;
  cell_of(t, n0, n1, 2, i, j, k);
  if (D == 0) i -= 1;
  if (D == 1) j -= 1;
  if (D == 2) k -= 1;
  const long long N = b.N, st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  T w[5], wn[5], p = b.p[c], pm = T(0), pp = T(0);
#pragma unroll
  for (int v = 0; v < 5; v++) w[v] = b.w[v * N + c];
  if (dissip_on) {
#pragma unroll
    for (int v = 0; v < 5; v++) wn[v] = b.w[v * N + c - st];
    pm = b.p[c - st], pp = b.p[c + st];
  }
  const T y = pdiv<S>(T(1), w[0]), Hc = w[4] + p;
  const T s = (T)b.s[D];
  const T f0 = pmul<S>(w[1 + D], s);
  T f[5];
  f[0] = f0;
  if (FAST) {
    const T q = pmul<S>(f0, y);
#pragma unroll
    for (int v = 1; v < 4; v++) f[v] = v == 1 + D ? fma(p, s, pmul<S>(q, w[v])) : pmul<S>(q, w[v]);
    f[4] = pmul<S>(q, Hc);
  } else {
#pragma unroll
    for (int v = 1; v < 4; v++) {
      f[v] = pmdiv<S>(pmul<S>(f0, w[v]), w[0], y);
      if (v == 1 + D) f[v] = f[v] + pmul<S>(p, s);
    }
    f[4] = pmdiv<S>(pmul<S>(f0, Hc), w[0], y);
  }
  T* F = b.F + (long long)(D * 5) * N + c;
#pragma unroll
  for (int v = 0; v < 5; v++) F[v * N] = f[v];
  if (!dissip_on) return;
  T* Dl = b.dlt + (long long)(D * 5) * N + c;
#pragma unroll
  for (int v = 0; v < 4; v++) Dl[v * N] = w[v] - wn[v];
  Dl[4 * N] = Hc - (wn[4] + pm);
  const T p2 = mul2(p);
  const T pb = D == 1 ? fabs(pp + p2 + pm) : fabs(pm + p2 + pp);
  const T pa = D == 1 ? fabs(pp - p2 + pm) : fabs(pm - p2 + pp);
  b.fp[D * N + c] = (pb > T(0)) ? pdiv<S>(pa, pb) : T(0);
}

// dflux_matrix, dflux.f90:283-339, with general face vector ss
template <typename T>
__device__ __noinline__ void dflux_matrix(T gamma, const T* u1, const T* u2, const T* dw, const T* ss, T* ff) {
  T gam1 = gamma - T(1), epsn = T(1), epsl = T(1);
  T rr = T(0.5) * (u1[0] + u2[0]);
  T us[3];
  for (int q = 0; q < 3; q++) us[q] = T(0.5) * (u1[q + 1] + u2[q + 1]) / rr;
  T ee = T(0.5) * (u1[4] + u2[4]) / rr;
  T qq = T(0.5) * (us[0] * us[0] + us[1] * us[1] + us[2] * us[2]);
  T c2 = gamma * gam1 * (ee - qq);
  T hh = c2 / gam1 + qq;
  T sss = ss[0] * ss[0] + ss[1] * ss[1] + ss[2] * ss[2];
  T cs = sqrt(c2 * sss);
  T qn = ss[0] * us[0] + ss[1] * us[1] + ss[2] * us[2];
  T e0 = fabs(qn) + cs;
  T e1 = fmaxT(epsn * e0, (T)fabs(qn + cs));
  T e2 = fmaxT(epsn * e0, (T)fabs(qn - cs));
  T e3 = fmaxT(epsl * e0, (T)fabs(qn));
  T s1 = T(0.5) * (e1 + e2), s2 = T(0.5) * (e1 - e2), s3 = e3;
  T ak1 = (s1 - s3) / c2 * gam1;
  T ak2 = s2 / cs;
  T ak3 = c2 / gam1 / sss;
  T d0 = dw[0], d1 = dw[1], d2 = dw[2], d3 = dw[3], d4 = dw[4];
  T vd = qq * d0 - us[0] * d1 - us[1] * d2 - us[2] * d3 + d4;
  T qd = qn * d0 - ss[0] * d1 - ss[1] * d2 - ss[2] * d3;
  ff[0] = ak1 * vd - ak2 * qd + s3 * d0;
  ff[1] = ak1 * (us[0] * vd - ss[0] * ak3 * qd) + ak2 * (gam1 * ss[0] * vd - us[0] * qd) + s3 * d1;
  ff[2] = ak1 * (us[1] * vd - ss[1] * ak3 * qd) + ak2 * (gam1 * ss[1] * vd - us[1] * qd) + s3 * d2;
  ff[3] = ak1 * (us[2] * vd - ss[2] * ak3 * qd) + ak2 * (gam1 * ss[2] * vd - us[2] * qd) + s3 * d3;
  ff[4] = ak1 * (hh * vd - qn * ak3 * qd) + ak2 * (gam1 * qn * vd - hh * qd) + s3 * d4;
}


// --------------------------------------------------------------- Roe, MUSCL and viscous faces
// (the reference's roepak/viscpak sources are not in its tree; these follow
// the published methods, as the oracle does: Roe 1981 with Harten's entropy
// fix, MUSCL with the van Albada limiter, central-gradient laminar stresses)
template <bool S, typename T>
__device__ __forceinline__ T van_albada(T a, T b, T e2) {
  // smooth form, no cut-off at a*b <= 0: with e2 > 0 a cut-off would make the
  // slope jump by up to b/3 when a changes sign.  Both differences zero (a
  // uniform stretch) and e2 > 0: the numerator is e2*a + e2*b, a zero with
  // the sign of a + b, and so is the quotient
  if (a == T(0) && b == T(0) && e2 > T(0)) return a + b;
  const T aa = pmul<S>(a, a), bb = pmul<S>(b, b);
  return pdiv<S>(pmul<S>(bb + e2, a) + pmul<S>(aa + e2, b), aa + bb + mul2(e2));
}

// yl, yr: RN(1/wl[0]) and RN(1/wr[0]); every quotient below that shares a
// divisor takes one reciprocal and mdiv, which rounds as the division does
template <typename T, bool S>
__device__ __forceinline__ void roe_diss_inl(const PhysParams& P, int d, T area, const T* wl, T pl, const T* wr, T pr,
                                             T yl, T yr, T* out) {
  const T g = (T)P.gamma;
  T ul[3], ur[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    ul[a] = pmdiv<S>(wl[1 + a], wl[0], yl);
    ur[a] = pmdiv<S>(wr[1 + a], wr[0], yr);
  }
  const T hl = pmdiv<S>(wl[4] + pl, wl[0], yl), hr = pmdiv<S>(wr[4] + pr, wr[0], yr);
  const T rt = sqrt(pmdiv<S>(wr[0], wl[0], yl));
  const T rh = pmul<S>(rt, wl[0]);
  const T den = T(1) + rt, yden = pdiv<S>(T(1), den);
  T uh[3];
#pragma unroll
  for (int a = 0; a < 3; a++) uh[a] = pmdiv<S>(ul[a] + pmul<S>(rt, ur[a]), den, yden);
  const T hh = pmdiv<S>(hl + pmul<S>(rt, hr), den, yden);
  const T q2 = pmul<S>(uh[0], uh[0]) + pmul<S>(uh[1], uh[1]) + pmul<S>(uh[2], uh[2]);
  const T c2 = pmul<S>(g - T(1), hh - mulhalf(q2));
  const T ch = sqrt(fmaxT(c2, (T)1e-300));
  const T un = d == 0 ? uh[0] : (d == 1 ? uh[1] : uh[2]);
  const T dr = wr[0] - wl[0], dp = pr - pl;
  T du[3];
#pragma unroll
  for (int a = 0; a < 3; a++) du[a] = ur[a] - ul[a];
  const T dun = d == 0 ? du[0] : (d == 1 ? du[1] : du[2]);
  const T delta = pmul<S>((T)P.epsentr, fabs(un) + ch);
  auto fix = [&](T lam) {
    const T a = fabs(lam);
    return (a < delta && delta > T(0)) ? pdiv<S>(pmul<S>(lam, lam) + pmul<S>(delta, delta), mul2(delta)) : a;
  };
  const T l1 = fix(un - ch), l2 = fix(un), l5 = fix(un + ch);
  const T c22 = mul2(c2), yc22 = pdiv<S>(T(1), c22);
  const T rcd = pmul<S>(pmul<S>(rh, ch), dun);
  const T a1 = pmdiv<S>(dp - rcd, c22, yc22);
  const T a2 = dr - pdiv<S>(dp, c2);
  const T a5 = pmdiv<S>(dp + rcd, c22, yc22);
  const T w1 = pmul<S>(l1, a1), w5 = pmul<S>(l5, a5);
  T sh[3];
#pragma unroll
  for (int a = 0; a < 3; a++) sh[a] = pmul<S>(rh, du[a] - (a == d ? dun : T(0)));
  T res[5];
  res[0] = w1 + pmul<S>(l2, a2) + w5;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const T k1 = uh[a] - (a == d ? ch : T(0)), k5 = uh[a] + (a == d ? ch : T(0));
    res[1 + a] = pmul<S>(w1, k1) + pmul<S>(l2, pmul<S>(a2, uh[a]) + sh[a]) + pmul<S>(w5, k5);
  }
  const T cu = pmul<S>(ch, un);
  const T en = pmul<S>(mulhalf(a2), q2) + (pmul<S>(uh[0], sh[0]) + pmul<S>(uh[1], sh[1]) + pmul<S>(uh[2], sh[2]));
  res[4] = pmul<S>(w1, hh - cu) + pmul<S>(l2, en) + pmul<S>(w5, hh + cu);
  const T ha = mulhalf(area);
#pragma unroll
  for (int v = 0; v < 5; v++) out[v] = pmul<S>(ha, res[v]);
}

template <typename T, bool S>
__device__ __noinline__ void roe_diss(const PhysParams& P, int d, T area, const T* wl, T pl, const T* wr, T pr, T yl, T yr,
                                      T* out) {
  roe_diss_inl<T, S>(P, d, area, wl, pl, wr, pr, yl, yr, out);
}

// face q (between q-1 and q) along D at cell c: cell states, MUSCL when order 2
template <typename T, int D>
__device__ __noinline__ void face_states(const DevBlock<T>& b, const PhysParams& P, long long c, int q, int order, T* wl, T* pl,
                            T* wr, T* pr) {
  const long long N = b.N;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  for (int v = 0; v < 5; v++) {
    wl[v] = b.w[v * N + c - st];
    wr[v] = b.w[v * N + c];
  }
  *pl = b.p[c - st];
  *pr = b.p[c];
  if (order < 2) return;
  const int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
  if (q - 2 < 0 || q + 1 > lq + 2) return;
  if (b.blank[c - 2 * st] == 0 || b.blank[c - st] == 0 || b.blank[c] == 0 || b.blank[c + st] == 0) return;
  T qv[4][5];  // primitive (rho,u,v,w,p) at q-2..q+1
  for (int o = 0; o < 4; o++) {
    long long co = c + (o - 2) * st;
    T r = b.w[co], yr = sdiv(T(1), r);
    qv[o][0] = r;
    for (int a = 0; a < 3; a++) qv[o][1 + a] = mdiv(b.w[(1 + a) * N + co], r, yr);
    qv[o][4] = b.p[co];
  }
  T L[5], R[5];
  for (int kq = 0; kq < 5; kq++) {
    T dm = qv[1][kq] - qv[0][kq], d0 = qv[2][kq] - qv[1][kq], dp = qv[3][kq] - qv[2][kq];
    T e2 = (T)P.lim_e2[kq];
    L[kq] = qv[1][kq] + T(0.5) * van_albada<true>(dm, d0, e2);
    R[kq] = qv[2][kq] - T(0.5) * van_albada<true>(d0, dp, e2);
  }
  if (L[0] <= T(0) || R[0] <= T(0) || L[4] <= T(0) || R[4] <= T(0)) return;
  const T gm1 = (T)P.gamma - T(1), rg = rcp_gm1(P, T(0));
  wl[0] = L[0];
  wr[0] = R[0];
  for (int a = 0; a < 3; a++) {
    wl[1 + a] = L[0] * L[1 + a];
    wr[1 + a] = R[0] * R[1 + a];
  }
  wl[4] = mdiv(L[4], gm1, rg) + T(0.5) * L[0] * (L[1] * L[1] + L[2] * L[2] + L[3] * L[3]);
  wr[4] = mdiv(R[4], gm1, rg) + T(0.5) * R[0] * (R[1] * R[1] + R[2] * R[2] + R[3] * R[3]);
  *pl = L[4];
  *pr = R[4];
}

// y = RN(1/w[0])
// face_states in the MUSCL form from the per-cell velocities (F[0..2]) and
// limited slopes (dlt) of k_prim and the prep pass: the same values, with each
// quotient and slope formed once per cell instead of once per face
template <typename T, int D, bool S>
__device__ __forceinline__ void face_states_pre(const DevBlock<T>& b, const PhysParams& P, long long c, int q, T* wl, T* pl,
                                             T* wr, T* pr) {
  const long long N = b.N;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long cm = c - st;
  for (int v = 0; v < 5; v++) {
    wl[v] = b.w[v * N + cm];
    wr[v] = b.w[v * N + c];
  }
  *pl = b.p[cm];
  *pr = b.p[c];
  const int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
  if (q - 2 < 0 || q + 1 > lq + 2) return;
  if (b.blank[c - 2 * st] == 0 || b.blank[cm] == 0 || b.blank[c] == 0 || b.blank[c + st] == 0) return;
  const T* sl = b.dlt + (long long)(D * 5) * N;
  T L[5], R[5];
  L[0] = wl[0] + mulhalf(sl[cm]);
  R[0] = wr[0] - mulhalf(sl[c]);
  for (int a = 0; a < 3; a++) {
    L[1 + a] = b.F[(long long)a * N + cm] + mulhalf(sl[(long long)(1 + a) * N + cm]);
    R[1 + a] = b.F[(long long)a * N + c] - mulhalf(sl[(long long)(1 + a) * N + c]);
  }
  L[4] = *pl + mulhalf(sl[4 * N + cm]);
  R[4] = *pr - mulhalf(sl[4 * N + c]);
  if (L[0] <= T(0) || R[0] <= T(0) || L[4] <= T(0) || R[4] <= T(0)) return;
  const T gm1 = (T)P.gamma - T(1), rg = rcp_gm1(P, T(0));
  wl[0] = L[0];
  wr[0] = R[0];
  for (int a = 0; a < 3; a++) {
    wl[1 + a] = pmul<S>(L[0], L[1 + a]);
    wr[1 + a] = pmul<S>(R[0], R[1 + a]);
  }
  wl[4] = pmdiv<S>(L[4], gm1, rg) +
          pmul<S>(mulhalf(L[0]), pmul<S>(L[1], L[1]) + pmul<S>(L[2], L[2]) + pmul<S>(L[3], L[3]));
  wr[4] = pmdiv<S>(R[4], gm1, rg) +
          pmul<S>(mulhalf(R[0]), pmul<S>(R[1], R[1]) + pmul<S>(R[2], R[2]) + pmul<S>(R[3], R[3]));
  *pl = L[4];
  *pr = R[4];
}

template <bool S, typename T>
__device__ __forceinline__ void ceflux_gen(int D, const T* w, T p, T s, T y, T* f) {
  T f0 = pmul<S>(w[1 + D], s);
  f[0] = f0;
  f[1] = pmdiv<S>(pmul<S>(f0, w[1]), w[0], y);
  f[2] = pmdiv<S>(pmul<S>(f0, w[2]), w[0], y);
  f[3] = pmdiv<S>(pmul<S>(f0, w[3]), w[0], y);
  f[1 + D] = f[1 + D] + pmul<S>(p, s);
  f[4] = pmdiv<S>(pmul<S>(f0, w[4] + p), w[0], y);
}

// laminar viscous flux through face q along D (at cell c), times S
template <typename T, int D, bool S>
__device__ __forceinline__ void visc_face_inl(const DevBlock<T>& b, const PhysParams& P, long long c, T area, T* out) {
  const long long N = b.N;
  const long long st[3] = {1, (long long)b.Pi, (long long)b.Pi * b.Pj};
  const long long cl = c - st[D];
  const double h[3] = {b.hx, b.hy, b.hz};
  T g[4][3];
  for (int a = 0; a < 4; a++) {
    const T* f = b.vt + (long long)a * N;
    for (int t = 0; t < 3; t++) {
      if (t == D)
        g[a][t] = pmdiv<S>(f[c] - f[cl], (T)h[D], rcp_h(b, D));
      else
        g[a][t] = pmdiv<S>((f[c + st[t]] - f[c - st[t]]) + (f[cl + st[t]] - f[cl - st[t]]), T(4) * (T)h[t],
                       rcp_4h(b, t));
    }
  }
  const T mu = (T)P.viscl, kt = (T)P.kt;
  T div = g[0][0] + g[1][1] + g[2][2];
  T tau[3];
  for (int a = 0; a < 3; a++)
    tau[a] = pmul<S>(mu, g[a][D] + g[D][a]) - (a == D ? pmul<S>((T(2) / T(3)) * mu, div) : T(0));
  T uf[3];
  for (int a = 0; a < 3; a++) uf[a] = mulhalf(b.vt[a * N + cl] + b.vt[a * N + c]);
  out[0] = T(0);
  for (int a = 0; a < 3; a++) out[1 + a] = pmul<S>(area, tau[a]);
  out[4] = pmul<S>(area, (pmul<S>(uf[0], tau[0]) + pmul<S>(uf[1], tau[1]) + pmul<S>(uf[2], tau[2])) + pmul<S>(kt, g[3][D]));
}

template <typename T, int D, bool S>
__device__ __noinline__ void visc_face(const DevBlock<T>& b, const PhysParams& P, long long c, T area, T* out) {
  visc_face_inl<T, D, S>(b, P, c, area, out);
}

// --------------------------------------------------------------- stage: per-face pass
// Thread (i,j,k) in [2..ie]x[2..je]x[2..ke] owns the lower face of cell
// (i,j,k) in each direction whose tangential indices are physical.
// SCH: FACE_CENTRAL or FACE_ROE when the launch knows the scheme (each then
// gets its own register allocation), FACE_ANY to test P.distype; FACE_JST:
// the central scheme with scalar dissipation and no viscous flux, without
// the registers the matrix dissipation and the viscous face would take.
enum { FACE_CENTRAL = 0, FACE_ROE = 1, FACE_ANY = 2, FACE_JST = 3 };
template <typename T, int D, int SCH, bool S>
__device__ __forceinline__ void face_dir(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd, int i, int j,
                                         int k) {
  const long long N = b.N;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  const int q = D == 0 ? i : (D == 1 ? j : k);      // face between q-1 and q
  const int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
  const int eq = lq + 1, bq = lq + 2;
  T* E = b.efs + (long long)(D * 5) * N;
  if (SCH != FACE_JST && P.eqn_ns && dissip_on) {  // viscous face flux, blended like the dissipation
    T o[5];
    if (SCH == FACE_ROE)
      visc_face_inl<T, D, S>(b, P, c, (T)fabs(b.s[D]), o);
    else
      visc_face<T, D, S>(b, P, c, (T)fabs(b.s[D]), o);
    T* V = b.vfs + (long long)(D * 5) * N;
#pragma unroll
    for (int v = 0; v < 5; v++) V[v * N + c] = pmul<S>(cd, o[v]);
  }
  const bool roe = SCH == FACE_ROE || (SCH == FACE_ANY && P.distype != 0);
  if (roe) {  // Roe: central part of the (reconstructed) states, upwind part into dfs
    T wl[5], wr[5], pl, pr;
    if (SCH == FACE_ROE && P.distype == 2)
      face_states_pre<T, D, S>(b, P, c, q, wl, &pl, wr, &pr);
    else
      face_states<T, D>(b, P, c, q, P.distype == 2 ? 2 : 1, wl, &pl, wr, &pr);
    const T yl = pdiv<S>(T(1), wl[0]), yr = pdiv<S>(T(1), wr[0]);
    if (P.distype == 2) {
      T f1[5], f2[5];
      ceflux_gen<S, T>(D, wr, pr, (T)b.s[D], yr, f1);
      ceflux_gen<S, T>(D, wl, pl, (T)b.s[D], yl, f2);
#pragma unroll
      for (int v = 0; v < 5; v++) E[v * N + c] = mulhalf(f1[v] + f2[v]);
    } else {
      const T* F = b.F + (long long)(D * 5) * N;
#pragma unroll
      for (int v = 0; v < 5; v++) E[v * N + c] = mulhalf(F[v * N + c] + F[v * N + c - st]);
    }
    if (!dissip_on) return;
    T o[5];
    if (SCH == FACE_ROE)
      roe_diss_inl<T, S>(P, D, (T)fabs(b.s[D]), wl, pl, wr, pr, yl, yr, o);
    else
      roe_diss<T, S>(P, D, (T)fabs(b.s[D]), wl, pl, wr, pr, yl, yr, o);
    T* Df = b.dfs + (long long)(D * 5) * N;
#pragma unroll
    for (int v = 0; v < 5; v++) Df[v * N + c] = pmul<S>(cd, o[v]);
    return;
  }
  // convective: efs(q) = 0.5*(F(q) + F(q-1))
  const T* F = b.F + (long long)(D * 5) * N;
#pragma unroll
  for (int v = 0; v < 5; v++) E[v * N + c] = mulhalf(F[v * N + c] + F[v * N + c - st]);
  if (!dissip_on) return;
  // dissipation face q (dflux.f90:87-111)
  const T* fpd = b.fp + (long long)D * N;
  T f_m2 = (q - 2 == 0) ? T(0) : fpd[c - 2 * st];
  T f_m1 = fpd[c - st];
  T f_0 = fpd[c];
  T f_p1 = (q + 1 == bq) ? T(0) : fpd[c + st];
  // the sensors are >= +0: their maximum and the comparison below are taken
  // on the bit patterns (exact_ops.cuh)
  T ep = max_nonneg(max_nonneg(max_nonneg(f_m2, f_m1), f_0), f_p1);
  // lambda at ghost cells equals the adjacent physical cell (timestep.f90:227-282)
  long long cm = (q - 1 < 2) ? c : c - st;
  long long cp = (q > lq) ? c - st : c;
  T lam = mulhalf(b.lam[cm] + b.lam[cp]);
  T dis2 = (T)P.vis2 * ep;
  T dis4 = (T)P.vis4;
  dis4 = gt_nonneg(dis4, dis2) ? dis4 - dis2 : T(0);
  dis2 = dis2 * cd;
  dis4 = dis4 * cd;
  // diw(q) = w(q)-w(q-1), formed once per cell by the prep pass;
  // diw(1) = diw(2); diw(ib) = diw(ie)
  const T* Dl = b.dlt + (long long)(D * 5) * N;
  T out[5];
#pragma unroll
  for (int v = 0; v < 5; v++) {
    T d0 = Dl[v * N + c];
    T dm = (q - 1 == 1) ? d0 : Dl[v * N + c - st];
    T dp = (q + 1 == bq) ? d0 : Dl[v * N + c + st];
    T t3 = dp - mul2(d0) + dm;
    out[v] = pmul<S>(dis2, d0) - pmul<S>(dis4, t3);
  }
  if (SCH == FACE_JST || !P.matrix) {
#pragma unroll
    for (int v = 0; v < 5; v++) out[v] = pmul<S>(out[v], lam);
  } else {
    T ss[3] = {T(0), T(0), T(0)};
    ss[D] = (T)b.s[D];
    T ff[5], wq1[5], wq2[5];  // w at q-1 and q, enthalpy in slot 4
#pragma unroll
    for (int v = 0; v < 4; v++) {
      wq1[v] = b.w[v * N + c - st];
      wq2[v] = b.w[v * N + c];
    }
    wq1[4] = b.H[c - st];
    wq2[4] = b.H[c];
    dflux_matrix((T)P.gamma, wq1, wq2, out, ss, ff);
#pragma unroll
    for (int v = 0; v < 5; v++) out[v] = ff[v];
  }
  T* Df = b.dfs + (long long)(D * 5) * N;
#pragma unroll
  for (int v = 0; v < 5; v++) Df[v * N + c] = out[v];
  (void)eq;
}

template <typename T, int SCH = FACE_ANY, bool S = true>
__device__ __forceinline__ void body_face(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd, long long t) {
  const int ex = b.ie - 1, ey = b.je - 1;  // 2..ie
  int i, j, k;
  cell_of(t, ex, ey, 2, i, j, k);
  bool jp = j <= b.jl, kp = k <= b.kl, ip = i <= b.il;
  if (jp && kp) face_dir<T, 0, SCH, S>(b, P, dissip_on, cd, i, j, k);
  if (ip && kp) face_dir<T, 1, SCH, S>(b, P, dissip_on, cd, i, j, k);
  if (ip && jp) face_dir<T, 2, SCH, S>(b, P, dissip_on, cd, i, j, k);
}

// The contracted form's dissipation face (scalar JST, dflux.f90:87-112): the
// combine pass forms the convective part from the cell fluxes, so only dfs is
// written.  The face's coefficients take lambda once, dis2*lambda and
// dis4*lambda, and each variable is one product and two multiply-adds.
template <typename T, int D, bool S>
__device__ __forceinline__ void face_diss_fast(const DevBlock<T>& b, const PhysParams& P, T cd, int i, int j, int k) {
  const long long N = b.N;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  const int q = D == 0 ? i : (D == 1 ? j : k);
  const int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
  const int bq = lq + 2;
  const T* fpd = b.fp + (long long)D * N;
  const T f_m2 = (q - 2 == 0) ? T(0) : fpd[c - 2 * st];
  const T f_p1 = (q + 1 == bq) ? T(0) : fpd[c + st];
  const T ep = max_nonneg(max_nonneg(max_nonneg(f_m2, fpd[c - st]), fpd[c]), f_p1);
  const long long cm = (q - 1 < 2) ? c : c - st;
  const long long cp = (q > lq) ? c - st : c;
  const T lam = mulhalf(b.lam[cm] + b.lam[cp]);
  const T dis2 = pmul<S>((T)P.vis2, ep);
  const T dis4 = gt_nonneg((T)P.vis4, dis2) ? (T)P.vis4 - dis2 : T(0);
  const T a2 = pmul<S>(pmul<S>(dis2, cd), lam), a4 = pmul<S>(pmul<S>(dis4, cd), lam);
  const T* Dl = b.dlt + (long long)(D * 5) * N;
  T* Df = b.dfs + (long long)(D * 5) * N;
#pragma unroll
  for (int v = 0; v < 5; v++) {
    const T d0 = Dl[v * N + c];
    const T dm = (q - 1 == 1) ? d0 : Dl[v * N + c - st];
    const T dp = (q + 1 == bq) ? d0 : Dl[v * N + c + st];
    const T t3 = fma(T(-2), d0, dp + dm);
    Df[v * N + c] = fma(a2, d0, -pmul<S>(a4, t3));
  }
}

// One direction of the face pass, at the faces along D between physical lines
// of cells; FAST: the contracted form's dissipation faces
template <typename T, bool FAST, bool S, int D, int SCH = FACE_JST>
__device__ __forceinline__ void body_face_split(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd, int t) {
  const int n0 = b.nx + (D == 0), n1 = b.ny + (D == 1), n2 = b.nz + (D == 2);
  if (t >= n0 * n1 * n2) return;
  int i, j, k;
  cell_of(t, n0, n1, 2, i, j, k);
  if (FAST)
    face_diss_fast<T, D, S>(b, P, cd, i, j, k);
  else
    face_dir<T, D, SCH, S>(b, P, dissip_on, cd, i, j, k);
}

// The split passes as one range of items: three rows, one per direction, each
// of whole 256-thread blocks (e = 2: prep, 1: faces)
template <typename T>
__host__ __device__ __forceinline__ long long split_row(const DevBlock<T>& b, int e) {
  const long long x = (long long)(b.nx + e) * b.ny * b.nz, y = (long long)b.nx * (b.ny + e) * b.nz,
                  z = (long long)b.nx * b.ny * (b.nz + e);
  const long long m = x > y ? (x > z ? x : z) : (y > z ? y : z);
  return (m + 255) / 256 * 256;
}
template <typename T> long long split_items_t(const DevBlock<T>& b, int e) { return 3 * split_row(b, e); }
template <typename T, bool FAST, bool S>
__device__ __forceinline__ void body_prep_rows(const DevBlock<T>& b, const PhysParams& P, int dissip_on, long long t) {
  const long long row = split_row(b, 2);
  if (t < row) body_prep_dir<T, FAST, S, 0>(b, P, dissip_on, (int)t);
  else if (t < 2 * row) body_prep_dir<T, FAST, S, 1>(b, P, dissip_on, (int)(t - row));
  else if (t < 3 * row) body_prep_dir<T, FAST, S, 2>(b, P, dissip_on, (int)(t - 2 * row));
}
template <typename T, bool FAST, bool S>
__device__ __forceinline__ void body_face_rows(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd,
                                               long long t) {
  const long long row = split_row(b, 1);
  if (t < row) body_face_split<T, FAST, S, 0>(b, P, dissip_on, cd, (int)t);
  else if (t < 2 * row) body_face_split<T, FAST, S, 1>(b, P, dissip_on, cd, (int)(t - row));
  else if (t < 3 * row) body_face_split<T, FAST, S, 2>(b, P, dissip_on, cd, (int)(t - 2 * row));
}

// --------------------------------------------------------------- stage: cut-cell record terms
// A record's corrections take dense face fluxes out and wall fluxes in.  The
// wall side depends only on the state (w, p, H, lambda, wsol, psol), not on
// this stage's face fluxes, so the record pass (rec_wall_terms) runs beside
// the face pass, and the combine pass takes the dense side from efs/dfs/vfs
// itself.  rec_wall holds per record (25 values):
//   [0,5)   efluxb first addend, [5,10) second addend (efluxb.f90:72-110)
//   [10,15) viscous wall stress term (NS)
//   [15,20) dfluxb Z0: fs1 - fs2 (JST) or the Roe wall flux
//   [20,25) dfluxb fs1 (solid on the + side) or fs2 (solid on the - side)
// With X the dense differences, dfluxb.f90 applies fw(t) = fw(t) - X and then
// fw(t) = fw(t) + Z at the cut cell (X0, Z0) and at its neighbour (X1, Z1).
template <typename T>
__device__ __forceinline__ void ceflux_axis(int D, const T* w, T p, T s, T* f) {
  T f0 = w[1 + D] * s;
  T y = T(1) / w[0];
  f[0] = f0;
  f[1] = mdiv(f0 * w[1], w[0], y);
  f[2] = mdiv(f0 * w[2], w[0], y);
  f[3] = mdiv(f0 * w[3], w[0], y);
  f[1 + D] = f[1 + D] + p * s;
  f[4] = mdiv(f0 * (w[4] + p), w[0], y);
}

template <typename T>
__device__ void rec_wall_terms(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd, unsigned* err, int m) {
  T* W = b.rec_wall + 25LL * m;
  const long long N = b.N;
  const int* ri = b.rec_i + 8 * m;
  int i = ri[0], j = ri[1], k = ri[2], id = ri[3], zz = ri[4];
  int D = zz - 1;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  T s = (T)b.s[D];
  T wc[5];
  for (int v = 0; v < 5; v++) wc[v] = b.w[v * N + c];
  if (fabs(wc[0]) < T(1.0e-8)) atomicCAS(err, 0u, (unsigned)ERR_ZERORHO);
  T psol = b.rec_psol[m];
  T wsol[5];
  for (int v = 0; v < 5; v++) wsol[v] = b.rec_wsol[5 * m + v];
  // efluxb.f90:66-110
  T f1[5], f2[5], f3[5];
  ceflux_axis<T>(D, wc, b.p[c], s, f1);
  ceflux_axis<T>(D, wsol, psol, s, f2);
  const bool plus = (id >= 4);  // solid on the + side
  long long cn = plus ? c - st : c + st;
  T wnb[5];
  for (int v = 0; v < 5; v++) wnb[v] = b.w[v * N + cn];
  ceflux_axis<T>(D, wnb, b.p[cn], s, f3);
  for (int v = 0; v < 5; v++) {
    T fs = T(0.5) * (f1[v] + f2[v]);
    T fa = T(0.5) * (f1[v] + f3[v]);
    W[v] = plus ? fa : fs;
    W[5 + v] = plus ? fs : fa;
  }
  if (!dissip_on) return;
  if (P.eqn_ns) {  // no-slip adiabatic wall face: normal gradients to the mirror state only
    T u[3], ug[3], qbv[3] = {(T)b.rec_qb[3 * m], (T)b.rec_qb[3 * m + 1], (T)b.rec_qb[3 * m + 2]};
    const double hh[3] = {b.hx, b.hy, b.hz};
    for (int a = 0; a < 3; a++) {
      u[a] = wc[1 + a] / wc[0];
      ug[a] = T(2) * qbv[a] - u[a];
    }
    const T mu = (T)P.viscl, S = (T)fabs(b.s[D]);
    T o[5];
    T tau[3];
    for (int a = 0; a < 3; a++) {
      T gn = plus ? (ug[a] - u[a]) / (T)hh[D] : (u[a] - ug[a]) / (T)hh[D];
      tau[a] = (a == D) ? (T(4) / T(3)) * mu * gn : mu * gn;
    }
    o[0] = T(0);
    for (int a = 0; a < 3; a++) o[1 + a] = S * tau[a];
    o[4] = S * (qbv[0] * tau[0] + qbv[1] * tau[1] + qbv[2] * tau[2]);
    for (int v = 0; v < 5; v++) W[10 + v] = plus ? -(cd * o[v]) : cd * o[v];
  }
  if (P.distype != 0) {  // Roe: the wall face's upwind flux taken to the ghost state
    T o[5];
    const T S = (T)fabs(b.s[D]);
    const T yc = T(1) / wc[0], ys = T(1) / wsol[0];
    if (plus)
      roe_diss<T, false>(P, D, S, wc, b.p[c], wsol, psol, yc, ys, o);
    else
      roe_diss<T, false>(P, D, S, wsol, psol, wc, b.p[c], ys, yc, o);
    for (int v = 0; v < 5; v++) W[15 + v] = plus ? -(cd * o[v]) : cd * o[v];
    return;
  }
  // dfluxb.f90:29-423; w(:,5) is the enthalpy here
  wsol[4] = wsol[4] + psol;
  auto pp = [&](int a) -> T { return b.p[c + a * st]; };
  // the enthalpy formed here with the prep pass's addition: a record at the
  // block's edge reaches the outer ghost layer, where the prep pass forms no H
  auto ww = [&](int a, int v) -> T {
    const long long q = c + a * st;
    return v < 4 ? b.w[v * N + q] : b.w[4 * N + q] + b.p[q];
  };
  auto lamc = [&](int a) -> T {
    // lambda with the ghost-copy rule of timestep.f90:227-282 along the record axis
    int q = (D == 0 ? i : (D == 1 ? j : k)) + a;
    int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
    int qq = q < 2 ? 2 : (q > lq ? lq : q);
    return b.lam[c + (long long)(qq - (q - a)) * st];
  };
  const int pos = D == 0 ? i : (D == 1 ? j : k);
  const int lim = D == 0 ? b.ib : (D == 1 ? b.jb : b.kb);
  T fp[3], ep, lam, dis2, dis4;
  T fs1[5], fs2[5], diw[3][5];
  T ssv[3] = {T(0), T(0), T(0)};
  ssv[D] = s;
  auto setdis = [&]() {
    dis2 = (T)P.vis2 * ep;
    dis4 = (T)P.vis4;
    dis4 = fdimT(dis4, dis2);
    dis2 = dis2 * cd;
    dis4 = dis4 * cd;
  };
  if (plus) {
    if (D == 0) {
      fp[0] = fabs(pp(-2) - T(2) * pp(-1) + pp(0)) / fabs(pp(-2) + T(2) * pp(-1) + pp(0));
      fp[1] = fabs(pp(-1) - T(2) * pp(0) + psol) / fabs(pp(-1) + T(2) * pp(0) + psol);
    } else {
      fp[0] = fabs(pp(0) - T(2) * pp(-1) + pp(-2)) / fabs(pp(0) + T(2) * pp(-1) + pp(-2));
      fp[1] = fabs(psol - T(2) * pp(0) + pp(-1)) / fabs(psol + T(2) * pp(0) + pp(-1));
    }
    ep = fmaxT(fp[0], fp[1]);
    lam = lamc(0);
    setdis();
    for (int v = 0; v < 5; v++) {
      diw[0][v] = ww(0, v) - ww(-1, v);
      diw[1][v] = wsol[v] - ww(0, v);
      diw[2][v] = diw[1][v];
      fs2[v] = diw[2][v] - T(2) * diw[1][v] + diw[0][v];
      fs2[v] = dis2 * diw[1][v] - dis4 * fs2[v];
    }
    if (!P.matrix) {
      for (int v = 0; v < 5; v++) fs2[v] = fs2[v] * lam;
    } else {
      T wcv[5], tmp[5];
      for (int v = 0; v < 5; v++) wcv[v] = ww(0, v);
      dflux_matrix((T)P.gamma, wcv, wsol, fs2, ssv, tmp);
      for (int v = 0; v < 5; v++) fs2[v] = tmp[v];
    }
    if (pos - 3 >= 0)
      fp[2] = fabs(pp(-1) - T(2) * pp(-2) + pp(-3)) / fabs(pp(-1) + T(2) * pp(-2) + pp(-3));
    else
      fp[2] = T(0);
    ep = fmaxT(fmaxT(fp[0], fp[1]), fp[2]);
    lam = T(0.5) * (lamc(-1) + lamc(0));
    setdis();
    for (int v = 0; v < 5; v++) {
      diw[0][v] = ww(-1, v) - ww(-2, v);
      diw[1][v] = ww(0, v) - ww(-1, v);
      diw[2][v] = wsol[v] - ww(0, v);
      fs1[v] = diw[2][v] - T(2) * diw[1][v] + diw[0][v];
      fs1[v] = dis2 * diw[1][v] - dis4 * fs1[v];
    }
    if (!P.matrix) {
      for (int v = 0; v < 5; v++) fs1[v] = fs1[v] * lam;
    } else {
      T wa[5], wcv[5], tmp[5];
      for (int v = 0; v < 5; v++) {
        wa[v] = ww(-1, v);
        wcv[v] = ww(0, v);
      }
      dflux_matrix((T)P.gamma, wa, wcv, fs1, ssv, tmp);
      for (int v = 0; v < 5; v++) fs1[v] = tmp[v];
    }
    for (int v = 0; v < 5; v++) {
      W[15 + v] = fs1[v] - fs2[v];
      W[20 + v] = fs1[v];
    }
  } else {
    fp[0] = fabs(pp(1) - T(2) * pp(0) + psol) / fabs(pp(1) + T(2) * pp(0) + psol);
    fp[1] = fabs(pp(2) - T(2) * pp(1) + pp(0)) / fabs(pp(2) + T(2) * pp(1) + pp(0));
    if (pos + 3 <= lim)
      fp[2] = fabs(pp(3) - T(2) * pp(2) + pp(1)) / fabs(pp(3) + T(2) * pp(2) + pp(1));
    else
      fp[2] = T(0);
    ep = fmaxT(fmaxT(fp[0], fp[1]), fp[2]);
    lam = T(0.5) * (lamc(0) + lamc(1));
    setdis();
    for (int v = 0; v < 5; v++) {
      diw[0][v] = ww(0, v) - wsol[v];
      diw[1][v] = ww(1, v) - ww(0, v);
      diw[2][v] = ww(2, v) - ww(1, v);
      fs2[v] = diw[2][v] - T(2) * diw[1][v] + diw[0][v];
      fs2[v] = dis2 * diw[1][v] - dis4 * fs2[v];
    }
    if (!P.matrix) {
      for (int v = 0; v < 5; v++) fs2[v] = fs2[v] * lam;
    } else {
      T wcv[5], wbv[5], tmp[5];
      for (int v = 0; v < 5; v++) {
        wcv[v] = ww(0, v);
        wbv[v] = ww(1, v);
      }
      dflux_matrix((T)P.gamma, wcv, wbv, fs2, ssv, tmp);
      for (int v = 0; v < 5; v++) fs2[v] = tmp[v];
    }
    ep = fmaxT(fp[0], fp[1]);
    lam = lamc(0);
    setdis();
    for (int v = 0; v < 5; v++) {
      diw[1][v] = ww(0, v) - wsol[v];
      diw[0][v] = diw[1][v];
      diw[2][v] = ww(1, v) - ww(0, v);
      fs1[v] = diw[2][v] - T(2) * diw[1][v] + diw[0][v];
      fs1[v] = dis2 * diw[1][v] - dis4 * fs1[v];
    }
    if (!P.matrix) {
      for (int v = 0; v < 5; v++) fs1[v] = fs1[v] * lam;
    } else {
      T wcv[5], tmp[5];
      for (int v = 0; v < 5; v++) wcv[v] = ww(0, v);
      dflux_matrix((T)P.gamma, wsol, wcv, fs1, ssv, tmp);
      for (int v = 0; v < 5; v++) fs1[v] = tmp[v];
    }
    for (int v = 0; v < 5; v++) {
      W[15 + v] = fs1[v] - fs2[v];
      W[20 + v] = fs2[v];
    }
  }
}

template <typename T>
__global__ void k_rec_wall(const __grid_constant__ DevBlock<T> b, const __grid_constant__ PhysParams P, int dissip_on,
                           T cd, unsigned* err) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < b.nmir) rec_wall_terms(b, P, dissip_on, cd, err, m);
}

__host__ __device__ __forceinline__ int pad32(int n) { return (n + 31) & ~31; }
template <typename T> __host__ __device__ __forceinline__ int rec_lane_items(const DevBlock<T>& b) {
  return pad32(8 * b.nmir);
}
// the scheme of the split passes and of rec_wall_lanes
__host__ __device__ __forceinline__ bool split_scheme(const PhysParams& P) {
  return P.distype == 0 && !P.eqn_ns && !P.matrix;
}

// rec_wall_terms for the central scheme with scalar dissipation of the Euler
// equations, eight lanes a record: lane v < 5 forms variable v, and the six
// divisions (three sensors, three reciprocals of densities) go to six lanes.
// One thread a record ran 3,000 instructions in a row, 20 us by events on any
// level; this takes 9.  Same operations, same order, same bits.  Every lane of
// a warp calls it.
template <typename T>
__device__ __forceinline__ void rec_wall_lanes(const DevBlock<T>& b, const PhysParams& P, int dissip_on, T cd,
                                               unsigned* err, int t) {
  const int lane = t & 7;
  const bool own = (t >> 3) < b.nmir;
  const int m = own ? t >> 3 : b.nmir - 1;
  const int v = lane < 5 ? lane : 4;
  const long long N = b.N;
  const int* ri = b.rec_i + 8 * m;
  const int D = ri[4] - 1;
  const long long st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, ri[0], ri[1], ri[2]);
  const bool plus = ri[3] >= 4;  // solid on the + side
  const int es = plus ? -1 : 1;  // along the axis, away from the wall
  const long long e = es * st;
  const T s = D == 0 ? (T)b.s[0] : (D == 1 ? (T)b.s[1] : (T)b.s[2]);
  const int pos = D == 0 ? ri[0] : (D == 1 ? ri[1] : ri[2]);
  const int lim = D == 0 ? b.ib : (D == 1 ? b.jb : b.kb);
  const bool third = plus ? pos - 3 >= 0 : pos + 3 <= lim;
  const T* wv = b.w + v * N + c;
  const T w0 = wv[0], w1 = wv[e], w2 = wv[2 * e], ws = b.rec_wsol[5 * m + v], psol = b.rec_psol[m];
  const T p0 = b.p[c], p1 = b.p[c + e], p2 = b.p[c + 2 * e], p3 = third ? b.p[c + 3 * e] : T(0);
  const int lq = D == 0 ? b.il : (D == 1 ? b.jl : b.kl);
  const int q1 = pos + es < 2 ? 2 : (pos + es > lq ? lq : pos + es);  // the ghost-copy rule of timestep.f90:227-282
  const T lam0 = b.lam[c], lam1 = b.lam[c + (long long)(q1 - pos) * st];
  auto from = [&](T x, int l) { return __shfl_sync(0xffffffffu, x, l, 8); };
  // a division a lane: the sensors beside the wall, one cell on and two cells
  // on, in the argument order of dfluxb.f90's three axes; then 1/rho at the
  // cut cell, the solid state and the neighbour
  const bool fwd = plus && D != 0;
  const T r0 = from(w0, 0), rs = from(ws, 0), r1 = from(w1, 0);
  T num = T(1), den = lane == 3 ? r0 : (lane == 4 ? rs : r1);
  if (lane < 3) {
    const T x = lane == 0 ? (fwd ? psol : p1) : (lane == 1 ? (fwd ? p0 : p2) : (plus ? p1 : p3));
    const T y = lane == 0 ? p0 : (lane == 1 ? p1 : p2);
    const T z = lane == 0 ? (fwd ? p1 : psol) : (lane == 1 ? (fwd ? p2 : p0) : (plus ? p3 : p1));
    num = fabs(x - T(2) * y + z);
    den = fabs(x + T(2) * y + z);
  }
  const T quot = num / den;
  const T s0 = from(quot, 0), s1 = from(quot, 1), sq = from(quot, 2), s2 = third ? sq : T(0);
  const T y0 = from(quot, 3), ys = from(quot, 4), y1 = from(quot, 5);
  // ceflux of the three states (efluxb.f90:66-110)
  auto flux = [&](T x, T p, T rho, T y) -> T {
    const T f0 = from(x, 1 + D) * s;
    const T q = lane == 4 ? f0 * (x + p) : f0 * x;
    T f = lane == 0 ? f0 : mdiv(q, rho, y);
    if (lane == 1 + D) f = f + p * s;
    return f;
  };
  const T f1 = flux(w0, p0, r0, y0), f2 = flux(ws, psol, rs, ys), f3 = flux(w1, p1, r1, y1);
  const T fs = T(0.5) * (f1 + f2), fa = T(0.5) * (f1 + f3);
  T* W = b.rec_wall + 25LL * m;
  const bool put = own && lane < 5;
  if (put) {
    W[v] = plus ? fa : fs;
    W[5 + v] = plus ? fs : fa;
  }
  if (own && lane == 0 && fabs(w0) < T(1.0e-8)) atomicCAS(err, 0u, (unsigned)ERR_ZERORHO);
  if (!dissip_on) return;
  // dfluxb.f90:29-423; the fifth variable is the enthalpy
  const T W0 = lane == 4 ? w0 + p0 : w0, W1 = lane == 4 ? w1 + p1 : w1, W2 = lane == 4 ? w2 + p2 : w2;
  const T Ws = lane == 4 ? ws + psol : ws;
  const T A = plus ? s1 : s0, B = plus ? s0 : s1;
  const T near = fmaxT(A, B);
  auto face = [&](T ep, T lam, T x2, T x1, T x0) -> T {
    T dis2 = (T)P.vis2 * ep;
    T dis4 = fdimT((T)P.vis4, dis2);
    dis2 = dis2 * cd;
    dis4 = dis4 * cd;
    const T f = x2 - T(2) * x1 + x0;
    return (dis2 * x1 - dis4 * f) * lam;
  };
  const T dw = plus ? Ws - W0 : W0 - Ws, d1 = plus ? W0 - W1 : W1 - W0, d2 = plus ? W1 - W2 : W2 - W1;
  const T wall = face(near, lam0, plus ? dw : d1, dw, plus ? d1 : dw);
  const T next = face(fmaxT(near, s2), T(0.5) * (plus ? lam1 + lam0 : lam0 + lam1), plus ? dw : d2, d1, plus ? d2 : dw);
  if (put) {
    W[15 + v] = plus ? next - wall : wall - next;
    W[20 + v] = next;
  }
}
template <typename T>
__global__ void k_rec_lanes(DevBlock<T> b, PhysParams P, int dissip_on, T cd, unsigned* err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < rec_lane_items(b)) rec_wall_lanes(b, P, dissip_on, cd, err, t);
}

// the record's geometry: cell, axis stride, solid side
template <typename T>
__device__ __forceinline__ void rec_geom(const DevBlock<T>& b, int m, long long& c, long long& st, int& D, bool& plus) {
  const int* ri = b.rec_i + 8 * m;
  D = ri[4] - 1;
  st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  c = cidx(b.Pi, b.Pj, ri[0], ri[1], ri[2]);
  plus = ri[3] >= 4;
}

// --------------------------------------------------------------- stage: combine + update
// euler.f90:320-331,387-391: the unsteady mode's factor lam = 1 + 3*de/(2*dtstep)
// with de = fn*vdtim (or fn*dtim), dividing the coarse-level residual and the
// finest level's update
template <typename T>
__device__ __forceinline__ T unsteady_lam(const DevBlock<T>& b, const PhysParams& P, const StageArgs& A, long long c) {
  const T vd = A.vt ? (T)(*b.dtim) : b.vdtim[c];
  const T de = (T)A.fn * vd;
  return T(1) + ((de * T(3)) / T(2)) / (T)P.dtstep;
}

// The cut-cell records act here in record order on the cell they touch: the
// dense face pair out, the wall pair in, from this stage's face fluxes and
// the record pass's wall terms (rec_wall_terms).
//
// FAST (the contracted form, JST central scheme): the convective part of dw
// is the central difference of the cell fluxes, efs(q) - efs(q+1) =
// 0.5*(F(q-1) - F(q+1)) in each direction, so no convective face pass runs;
// a record's dense face pair takes the same difference.
template <typename T, bool FAST = false, bool S = true>
__device__ __forceinline__ void body_combine(const DevBlock<T>& b, const PhysParams& P, const StageArgs& A,
                                             unsigned* err, long long t) {
  const int nxl = b.nx, nyl = b.ny;
  int i, j, k;
  cell_of(t, nxl, nyl, 2, i, j, k);
  const long long N = b.N;
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  const long long sj = b.Pi, sk = (long long)b.Pi * b.Pj;
  const int tg = b.cutmap[c];
  T dwv[5], fwv[5];
  if (FAST) {
    const T* Fx = b.F;
    const T* Fy = b.F + 5 * N;
    const T* Fz = b.F + 10 * N;
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const T a = (Fx[v * N + c - 1] - Fx[v * N + c + 1]) + (Fy[v * N + c - sj] - Fy[v * N + c + sj]);
      dwv[v] = mulhalf(a + (Fz[v * N + c - sk] - Fz[v * N + c + sk]));
    }
  } else {
    const T* Ex = b.efs;
    const T* Ey = b.efs + 5 * N;
    const T* Ez = b.efs + 10 * N;
#pragma unroll
    for (int v = 0; v < 5; v++) {
      T a = Ex[v * N + c] - Ex[v * N + c + 1];
      a = a + Ey[v * N + c] - Ey[v * N + c + sj];
      a = a + Ez[v * N + c] - Ez[v * N + c + sk];
      dwv[v] = a;
    }
  }
  // fw: blending and dissipation (euler.f90:127-135, dflux.f90:116-238)
  const T fac = T(1) - (T)A.cd;
  if (A.dissip_on) {
    const T* Dx = b.dfs;
    const T* Dy = b.dfs + 5 * N;
    const T* Dz = b.dfs + 10 * N;
    T vis[5];
#pragma unroll
    for (int v = 0; v < 5; v++) vis[v] = A.scale_fw ? pmul<S>(b.fw[v * N + c], fac) : T(0);
    if (P.eqn_ns) {  // viscous faces, then the viscous wall faces in record order
      const T* Vx = b.vfs;
      const T* Vy = b.vfs + 5 * N;
      const T* Vz = b.vfs + 10 * N;
#pragma unroll
      for (int v = 0; v < 5; v++) {
        T a = vis[v];
        a = a + (Vx[v * N + c] - Vx[v * N + c + 1]);
        a = a + (Vy[v * N + c] - Vy[v * N + c + sj]);
        a = a + (Vz[v * N + c] - Vz[v * N + c + sk]);
        vis[v] = a;
      }
      if (tg >= 0) {
        for (int o = b.tgt_off[tg]; o < b.tgt_off[tg + 1]; o++) {
          const int op = b.tgt_ops[o];
          if (op & 1) continue;
          const int m = op >> 1;
          long long cm, st;
          int D;
          bool plus;
          rec_geom(b, m, cm, st, D, plus);
          const T* V = b.vfs + (long long)(D * 5) * N;
          const T* Wm = b.rec_wall + 25LL * m;
          const long long qn = plus ? cm + st : cm;  // the wall face's upper cell
#pragma unroll
          for (int v = 0; v < 5; v++) {
            const T x = plus ? -V[v * N + qn] : V[v * N + qn];
            vis[v] = vis[v] - x;
            vis[v] = vis[v] + Wm[10 + v];
          }
        }
      }
    }
    if (FAST) {
#pragma unroll
      for (int v = 0; v < 5; v++) {
        const T a = (Dx[v * N + c] - Dx[v * N + c + 1]) + (Dy[v * N + c] - Dy[v * N + c + sj]);
        const T d = a + (Dz[v * N + c] - Dz[v * N + c + sk]);
        fwv[v] = A.scale_fw ? fma(b.fw[v * N + c], fac, d) : d;
      }
    } else {
#pragma unroll
      for (int v = 0; v < 5; v++) {
        T a = vis[v];
        a = a + (Dx[v * N + c] - Dx[v * N + c + 1]);
        a = a + (Dy[v * N + c] - Dy[v * N + c + sj]);
        a = a + (Dz[v * N + c] - Dz[v * N + c + sk]);
        fwv[v] = a;
      }
    }
  } else {
#pragma unroll
    for (int v = 0; v < 5; v++) fwv[v] = A.scale_fw ? pmul<S>(b.fw[v * N + c], fac) : T(0);
  }
  if (tg >= 0) {
    // cut-cell wall faces, this cell's records in record order: efluxb on dw
    // (efluxb.f90:72-110) and dfluxb on fw (dfluxb.f90:47-420)
    for (int o = b.tgt_off[tg]; o < b.tgt_off[tg + 1]; o++) {
      const int op = b.tgt_ops[o];
      const int m = op >> 1;
      long long cm, st;
      int D;
      bool plus;
      rec_geom(b, m, cm, st, D, plus);
      const T* Wm = b.rec_wall + 25LL * m;
      if (!(op & 1)) {  // efluxb on the cut cell: the dense face pair out, the wall pair in
        const T* E = b.efs + (long long)(D * 5) * N;
        const T* Fd = b.F + (long long)(D * 5) * N;
#pragma unroll
        for (int v = 0; v < 5; v++) {
          const T x = FAST ? mulhalf(Fd[v * N + cm - st] - Fd[v * N + cm + st]) : E[v * N + cm] - E[v * N + cm + st];
          dwv[v] = dwv[v] - x;
          dwv[v] = dwv[v] + Wm[v] - Wm[5 + v];
        }
      }
      if (A.dissip_on) {
        const T* Dd = b.dfs + (long long)(D * 5) * N;
        auto dd = [&](int a, int v) -> T { return Dd[v * N + cm + a * st]; };
#pragma unroll
        for (int v = 0; v < 5; v++) {
          T x, z;
          if (P.distype != 0) {  // Roe wall: the dense face out, the ghost-state flux in (neighbour: zeros)
            const long long qn = plus ? cm + st : cm;
            x = (op & 1) ? T(0) : (plus ? -Dd[v * N + qn] : Dd[v * N + qn]);
            z = (op & 1) ? T(0) : Wm[15 + v];
          } else if (!(op & 1)) {  // dfluxb X0, Z0
            x = dd(0, v) - dd(1, v);
            z = Wm[15 + v];
          } else if (plus) {  // dfluxb X1, Z1, solid on the + side
            x = dd(-1, v) - dd(0, v);
            z = dd(-1, v) - Wm[20 + v];
          } else {  // solid on the - side
            x = dd(1, v) - dd(2, v);
            z = Wm[20 + v] - dd(2, v);
          }
          fwv[v] = fwv[v] - x;
          fwv[v] = fwv[v] + z;
        }
      }
    }
  }
  if (A.dissip_on || A.scale_fw || A.m == 1) {  // the first stage starts fw
#pragma unroll
    for (int v = 0; v < 5; v++) b.fw[v * N + c] = fwv[v];
  }
#pragma unroll
  for (int v = 0; v < 5; v++) dwv[v] = dwv[v] + fwv[v];
  if (A.tmode) {  // euler.f90:249-275: BDF2, or the first step's (halved) BDF1
    const T f = (T(0.5) * (T)b.vol) / (T)P.dtstep;
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const T wv = b.w[v * N + c], w1 = b.w1[v * N + c];
      const T d = A.tmode == 2 ? (T(3) * wv - T(4) * w1) + b.w2[v * N + c] : wv - w1;
      dwv[v] = dwv[v] + f * d;
    }
  }
  if (A.forcing) {  // euler.f90:294-318
#pragma unroll
    for (int v = 0; v < 5; v++) {
      T q;
      if (A.first_forcing) {
        q = T(0);
        if (b.marker[c] == 1) q = T(1) * b.wr[v * N + c] - dwv[v];
        b.qf[v * N + c] = q;
      } else {
        q = b.qf[v * N + c];
      }
      dwv[v] = dwv[v] + q;
    }
    if (P.unsteady) {
      const T lam = unsteady_lam(b, P, A, c), rl = T(1) / lam;
#pragma unroll
      for (int v = 0; v < 5; v++) dwv[v] = mdiv(dwv[v], lam, rl);
    }
  }
  if (FAST) {
    if (b.blank[c] == 0)
#pragma unroll
      for (int v = 0; v < 5; v++) dwv[v] = T(0);
  } else if (b.blank[c] == 0) {
    // dw * blank: x * 1 is x itself, so only blanked cells multiply (by 0)
#pragma unroll
    for (int v = 0; v < 5; v++) dwv[v] = dwv[v] * T(0);
  }
  if (A.lres) {
#pragma unroll
    for (int v = 0; v < 5; v++) b.dw[v * N + c] = dwv[v];
    return;
  }
  // time-step scaling, euler.f90:364-372: de = fn*vdtim/cellvolume
  T vd = A.vt ? (T)(*b.dtim) : b.vdtim[c];
  T de = FAST ? ((T)A.fn * vd) * rcp_vol(b) : pmdiv<S>(pmul<S>((T)A.fn, vd), (T)b.vol, rcp_vol(b));
#pragma unroll
  for (int v = 0; v < 5; v++) dwv[v] = pmul<S>(de, dwv[v]);
  if (A.irs) {
#pragma unroll
    for (int v = 0; v < 5; v++) b.dw[v * N + c] = dwv[v];
    return;
  }
  // update, euler.f90:381-399 (steady: lam = 1, and dw/1 is dw)
  T wv[5];
  if (P.unsteady && !A.forcing) {
    const T lam = unsteady_lam(b, P, A, c), rl = T(1) / lam;
#pragma unroll
    for (int v = 0; v < 5; v++) wv[v] = b.wn[v * N + c] - mdiv(dwv[v], lam, rl);
  } else {
#pragma unroll
    for (int v = 0; v < 5; v++) wv[v] = b.wn[v * N + c] - dwv[v];
  }
#pragma unroll
  for (int v = 0; v < 5; v++) {
    b.w[v * N + c] = wv[v];
    b.dw[v * N + c] = dwv[v];
  }
  b.p[c] = depvars<S>((T)P.gamma, wv);
}

// --------------------------------------------------------------- implicit residual smoothing
// psmoo_old (psmoo.f90:97-242): constant-coefficient Thomas sweeps along i,
// then j, then k, skipping blanked cells without re-factoring the pivots.
// One thread per (line, variable); consecutive threads walk consecutive
// lines of one variable, so the j- and k-sweeps are coalesced.  TC is the
// arithmetic precision.
template <typename T, int D>
__device__ __forceinline__ long long irs_lines(const DevBlock<T>& b) {
  return D == 0 ? (long long)b.ny * b.nz : (D == 1 ? (long long)b.nx * b.nz : (long long)b.nx * b.ny);
}

template <typename T, int D>
__device__ __forceinline__ void line_of(const DevBlock<T>& b, long long ln, long long& c0, long long& st, int& l) {
  if (D == 0) {
    int j = 2 + (int)((unsigned)ln % (unsigned)b.ny), k = 2 + (int)((unsigned)ln / (unsigned)b.ny);
    c0 = cidx(b.Pi, b.Pj, 0, j, k);
    st = 1;
    l = b.il;
  } else if (D == 1) {
    int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), k = 2 + (int)((unsigned)ln / (unsigned)b.nx);
    c0 = cidx(b.Pi, b.Pj, i, 0, k);
    st = b.Pi;
    l = b.jl;
  } else {
    int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), j = 2 + (int)((unsigned)ln / (unsigned)b.nx);
    c0 = cidx(b.Pi, b.Pj, i, j, 0);
    st = (long long)b.Pi * b.Pj;
    l = b.kl;
  }
}

// the variable of (line, variable) item t: t / lines, which is 0..4
__device__ __forceinline__ int line_var(long long t, long long lines) {
  return (t >= lines) + (t >= 2 * lines) + (t >= 3 * lines) + (t >= 4 * lines);
}

// two neighbouring cells of an i line, the first at an even offset of a field
// whose planes and rows are even (irs_pairs)
template <typename T, typename TC>
__device__ __forceinline__ void irs_load2(const T* d, const uint8_t* bl, int q, TC& x0, TC& x1, unsigned char& b0,
                                          unsigned char& b1) {
  static_assert(std::is_same<T, double>::value, "pairs are of FP64 values");
  const double2 x = *reinterpret_cast<const double2*>(d + q);
  const uchar2 b = *reinterpret_cast<const uchar2*>(bl + q);
  x0 = x.x;
  x1 = x.y;
  b0 = b.x;
  b1 = b.y;
}
template <typename T>
__device__ __forceinline__ void irs_store2(T* d, int q, double x0, double x1) {
  *reinterpret_cast<double2*>(d + q) = make_double2(x0, x1);
}
// whether every even cell of every i line lies on a 16-byte boundary of dw and
// a 2-byte one of blank
template <typename T>
inline bool irs_pairs(const DevBlock<T>& b) {
  return b.Pi % 2 == 0 && b.N % 2 == 0 && (uintptr_t)b.dw % 16 == 0 && (uintptr_t)b.blank % 2 == 0;
}

// SC: the products of the forward and backward steps on the integer pipes.
// That lengthens the serial chain of each line, so it pays only where many
// lines run at once and the sweep is bound by the FP64 rate; with few lines
// (coarse levels, slabs) the chain's latency bounds it and the FP64 forms
// are faster.
// QK: the quotient in two operations (irs_quick).
// Every FP64 warp instruction takes 64 cycles of its scheduler, dependent or
// not, whatever its active lanes, so a row costs 64 cycles an operation however
// few the lines: 5 operations forward and 2 back with Markstein's quotient, 4 and
// 2 with the short one, and every instruction around them adds to the chain.
// A blanked row therefore keeps its value by a select, not a branch.  With the
// short quotient, select and longer chunks, i and j sweeps: 512x512x2 202 and
// 199 -> 162 and 151 us, 256x256x2 97 and 99 -> 79 and 78, 96^3 98 and 82 -> 90 and
// 70, 192^3 569 and 381 -> 544 and 324.
// PAIR (i lines of FP64 values, irs_pairs): whole chunks start at an even cell and
// move two cells an access.  The lanes of a warp are on 32 lines, so an access
// takes 32 cycles of the L1 however wide it is, six a row against
// six FP64 operations of 16.  192^3 544 -> 391 us (j, whose lanes are side by side, 325),
// 96^3 91 -> 73, 48^3 23.0 -> 22.6.
template <typename T, typename TC, int D, bool SC = false, bool QK = false, int K = 8, bool PAIR = false>
__device__ __forceinline__ void body_irs(const DevBlock<T>& b, const IrsTables& tb, TC bb, long long t) {
  const long long lines = irs_lines<T, D>(b);
  const int v = line_var(t, lines);
  const long long ln = t - (long long)v * lines;
  long long c0, st;
  int l;
  line_of<T, D>(b, ln, c0, st, l);
  T* d = b.dw + (long long)v * b.N + c0;
  const uint8_t* bl = b.blank + c0;
  TC prev;
  {
    TC x = (TC)d[2 * st];
    if (bl[2 * st] != 0) {
      if constexpr (QK)
        x = irs_quick<false>(x, tb.e1r[2], tb.e1l[2]);
      else
        x = x / irs_e1(tb, 2, TC(0));
      d[2 * st] = (T)x;
    }
    prev = x;
  }
  // The recurrence is serial, its loads are not: each chunk of K cells is
  // loaded before any of it is solved, so one memory latency is paid per
  // chunk instead of per cell.  Every cell is read once and written once
  // after its own read, so the order of results is unchanged.
  constexpr bool tables_first = !(SC && D > 0);
  auto forward = [&](int q0, auto whole) {
    TC xb[K], pb[K], rb[K];
    unsigned char bk[K];
    // the tables with the chunk: behind the stores below they are loaded row
    // by row, which the i sweep's strided lines and a warp alone on its
    // scheduler wait for; many warps would rather have the registers
    auto tables = [&](int u) {
      if constexpr (QK)
        pb[u] = tb.e1l[q0 + u];
      else
        pb[u] = irs_e1(tb, q0 + u, TC(0));
      rb[u] = irs_e1r(tb, q0 + u, TC(0));
    };
    constexpr bool pair = PAIR && decltype(whole)::value;
#pragma unroll
    for (int u = 0; u < K; u++)
      if (decltype(whole)::value || q0 + u <= l) {
        if constexpr (pair) {
          if (u % 2 == 0) irs_load2(d, bl, q0 + u, xb[u], xb[u + 1], bk[u], bk[u + 1]);
        } else {
          xb[u] = (TC)d[(q0 + u) * st];
          bk[u] = bl[(q0 + u) * st];
        }
        if (tables_first) tables(u);
      }
    TC half = 0;
#pragma unroll
    for (int u = 0; u < K; u++)
      if (decltype(whole)::value || q0 + u <= l) {
        if (!tables_first) tables(u);
        const TC z = xb[u] - (SC ? smul(bb, prev) : bb * prev);
        TC x;
        if constexpr (QK)
          x = irs_quick<SC>(z, rb[u], pb[u]);
        else
          x = SC ? smdiv(z, pb[u], rb[u]) : mdiv(z, pb[u], rb[u]);
        prev = bk[u] != 0 ? x : xb[u];
        if constexpr (pair) {  // a blanked cell gets its own value back
          if (u % 2 == 0)
            half = prev;
          else
            irs_store2(d, q0 + u - 1, half, prev);
        } else if (bk[u] != 0) {
          d[(q0 + u) * st] = (T)x;
        }
      }
  };
  auto one = [&](int q) {  // forward at the one cell q
    const TC z0 = (TC)d[q * st];
    TC p1;
    if constexpr (QK)
      p1 = tb.e1l[q];
    else
      p1 = irs_e1(tb, q, TC(0));
    const TC r1 = irs_e1r(tb, q, TC(0));
    const TC z = z0 - (SC ? smul(bb, prev) : bb * prev);
    TC x;
    if constexpr (QK)
      x = irs_quick<SC>(z, r1, p1);
    else
      x = SC ? smdiv(z, p1, r1) : mdiv(z, p1, r1);
    prev = bl[q * st] != 0 ? x : z0;
    if (bl[q * st] != 0) d[q * st] = (T)x;
  };
  int q0 = 3;
  if (PAIR && l >= 3) one(q0++);
  for (; q0 + K - 1 <= l; q0 += K) forward(q0, std::true_type{});
  if (q0 <= l) forward(q0, std::false_type{});
  auto backward = [&](int q0, auto whole) {
    TC xb[K], pb[K];
    unsigned char bk[K];
    constexpr bool pair = PAIR && decltype(whole)::value;
#pragma unroll
    for (int u = 0; u < K; u++)
      if (decltype(whole)::value || q0 - u >= 2) {
        if constexpr (pair) {
          if (u % 2 == 0) irs_load2(d, bl, q0 - u - 1, xb[u + 1], xb[u], bk[u + 1], bk[u]);
        } else {
          xb[u] = (TC)d[(q0 - u) * st];
          bk[u] = bl[(q0 - u) * st];
        }
        pb[u] = irs_e2(tb, q0 - u, TC(0));
      }
    TC half = 0;
#pragma unroll
    for (int u = 0; u < K; u++)
      if (decltype(whole)::value || q0 - u >= 2) {
        const TC x = xb[u] - (SC ? smul(pb[u], prev) : pb[u] * prev);
        prev = bk[u] != 0 ? x : xb[u];
        if constexpr (pair) {
          if (u % 2 == 0)
            half = prev;
          else
            irs_store2(d, q0 - u, prev, half);
        } else if (bk[u] != 0) {
          d[(q0 - u) * st] = (T)x;
        }
      }
  };
  q0 = l - 1;
  if (PAIR && q0 % 2 == 0 && q0 >= 2) {  // down to an odd cell
    const TC z0 = (TC)d[q0 * st], e2 = irs_e2(tb, q0, TC(0));
    const TC x = z0 - (SC ? smul(e2, prev) : e2 * prev);
    prev = bl[q0 * st] != 0 ? x : z0;
    if (bl[q0 * st] != 0) d[q0 * st] = (T)x;
    q0--;
  }
  for (; q0 - K + 1 >= 2; q0 -= K) backward(q0, std::true_type{});
  if (q0 >= 2) backward(q0, std::false_type{});
}

// The FP32 sweeps of the mixed form's finest level, whose storage is FP64.
// body_irs<double, float, D> converts every value on its way in and out of
// each sweep, and on this part those conversions issue at the FP64 rate.
// Here the i sweep reads dw and leaves its results in an FP32 copy (in the
// stage scratch, free after the residual pass); the j sweep works in the
// copy; the k sweep writes its results back to dw.  A float stored as double
// and read back is the same float, so every value is the one body_irs gives;
// blanked cells keep their dw, as there.
template <typename TS, typename TO, int D>
__device__ __forceinline__ void body_irs_mixed(const DevBlock<double>& b, const IrsTables& tb, float bb,
                                               const TS* src, float* mid, TO* out, long long t) {
  constexpr bool fill = !std::is_same<TS, float>::value;  // the i sweep: every cell into the copy
  constexpr bool back = !std::is_same<TO, float>::value;  // the k sweep: results back to dw
  const long long lines = irs_lines<double, D>(b);
  const int v = line_var(t, lines);
  const long long ln = t - (long long)v * lines;
  long long c0, st;
  int l;
  if (D == 0) {
    int j = 2 + (int)((unsigned)ln % (unsigned)b.ny), k = 2 + (int)((unsigned)ln / (unsigned)b.ny);
    c0 = cidx(b.Pi, b.Pj, 0, j, k);
    st = 1;
    l = b.il;
  } else if (D == 1) {
    int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), k = 2 + (int)((unsigned)ln / (unsigned)b.nx);
    c0 = cidx(b.Pi, b.Pj, i, 0, k);
    st = b.Pi;
    l = b.jl;
  } else {
    int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), j = 2 + (int)((unsigned)ln / (unsigned)b.nx);
    c0 = cidx(b.Pi, b.Pj, i, j, 0);
    st = (long long)b.Pi * b.Pj;
    l = b.kl;
  }
  const TS* s = src + (long long)v * b.N;
  float* m = mid + (long long)v * b.N;
  TO* o = out + (long long)v * b.N;
  float prev;
  {
    const long long c = c0 + 2 * st;
    float x = (float)s[c];
    if (b.blank[c] != 0) {
      x = x / irs_e1(tb, 2, 0.0f);
      m[c] = x;
    } else if (fill) {
      m[c] = x;
    }
    prev = x;
  }
  constexpr int K = 8;
  float xb[K], pb[K], rb[K];
  unsigned char bk[K];
  for (int q0 = 3; q0 <= l; q0 += K) {
#pragma unroll
    for (int u = 0; u < K; u++)
      if (q0 + u <= l) {
        const long long c = c0 + (q0 + u) * st;
        xb[u] = (float)s[c];
        bk[u] = b.blank[c];
        pb[u] = irs_e1(tb, q0 + u, 0.0f);
        rb[u] = irs_e1r(tb, q0 + u, 0.0f);
      }
#pragma unroll
    for (int u = 0; u < K; u++)
      if (q0 + u <= l) {
        const float x = mdiv(xb[u] - bb * prev, pb[u], rb[u]);
        prev = bk[u] != 0 ? x : xb[u];
        if (fill || bk[u] != 0) m[c0 + (q0 + u) * st] = prev;
      }
  }
  // the backward pass does not revisit row l: its forward result is final
  if (back && b.blank[c0 + l * st] != 0) o[c0 + l * st] = (TO)prev;
  for (int q0 = l - 1; q0 >= 2; q0 -= K) {
#pragma unroll
    for (int u = 0; u < K; u++)
      if (q0 - u >= 2) {
        const long long c = c0 + (q0 - u) * st;
        xb[u] = m[c];
        bk[u] = b.blank[c];
        pb[u] = irs_e2(tb, q0 - u, 0.0f);
      }
#pragma unroll
    for (int u = 0; u < K; u++)
      if (q0 - u >= 2) {
        const float x = xb[u] - pb[u] * prev;
        prev = bk[u] != 0 ? x : xb[u];
        if (bk[u] != 0) o[c0 + (q0 - u) * st] = (TO)x;
      }
  }
}

// The mixed form's i sweep with one warp per (line, variable).  A psmoo_old
// row is an affine map of the row before it, x(q) = a(q) x(q-1) + c(q):
// forward a = -bb/e1(q), c = dw(q)/e1(q) on unblanked rows and a = 0,
// c = dw(q) on blanked ones (the row keeps its value, and the next row
// takes it as its predecessor); backward a = -e2(q), c = x(q) on unblanked
// rows.  Each lane composes the maps of K consecutive rows, a warp scan of
// the composed maps gives every lane the value entering its rows, and the
// lane applies its maps in order.  Loads and stores of a warp cover one
// contiguous line.  FP32 arithmetic: on the FP64 residual of the mixed
// form's finest level, the result going to the FP32 copy the j and k sweeps
// continue on; or on an FP32 level's residual, in place (every row of the
// line, blanked rows with their unsmoothed value).
template <int K, typename T = double>
__global__ void __launch_bounds__(256) k_irs_scan_i(DevBlock<T> b, IrsTables tb, float bb, float* cp) {
  const long long lines = (long long)b.ny * b.nz;
  const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (wid >= 5 * lines) return;  // uniform over the warp
  const int v = line_var(wid, lines);
  const long long ln = wid - (long long)v * lines;
  const int j = 2 + (int)((unsigned)ln % (unsigned)b.ny), k = 2 + (int)((unsigned)ln / (unsigned)b.ny);
  const long long c0 = cidx(b.Pi, b.Pj, 0, j, k);
  const int l = b.il;
  const T* src = b.dw + (long long)v * b.N + c0;  // read whole into registers before any write
  float* dst = cp + (long long)v * b.N + c0;
  const uint8_t* bl = b.blank + c0;
  const int q0 = 2 + lane * K;
  float x[K];
  unsigned bk = 0;
  // forward: the lane's maps, composed in row order
  float ca = 1.f, cc = 0.f;
#pragma unroll
  for (int u = 0; u < K; u++) {
    const int q = q0 + u;
    if (q <= l) {
      const float d = (float)src[q];
      float a = 0.f, c = d;
      if (bl[q] != 0) {
        bk |= 1u << u;
        const float r = irs_e1r(tb, q, 0.0f);
        a = q == 2 ? 0.f : -bb * r;
        c = d * r;
      }
      x[u] = c;
      ca = a * ca;
      cc = fmaf(a, cc, c);
    } else {
      x[u] = 0.f;
    }
  }
  // inclusive scan over the lanes in row order, then the value entering
  // this lane's first row (row 2's map ignores its input: a = 0)
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float pa = __shfl_up_sync(0xffffffffu, ca, off), pc = __shfl_up_sync(0xffffffffu, cc, off);
    if (lane >= off) {
      cc = fmaf(ca, pc, cc);
      ca = ca * pa;
    }
  }
  float prev = __shfl_up_sync(0xffffffffu, cc, 1);
  if (lane == 0) prev = 0.f;
#pragma unroll
  for (int u = 0; u < K; u++) {
    const int q = q0 + u;
    if (q <= l && q > 2 && (bk >> u & 1u)) x[u] = fmaf(-bb * irs_e1r(tb, q, 0.0f), prev, x[u]);
    if (q <= l) prev = x[u];
  }
  // backward: rows l-1 down to 2; row l keeps its forward value
  ca = 1.f;
  cc = 0.f;
#pragma unroll
  for (int u = K - 1; u >= 0; u--) {
    const int q = q0 + u;
    if (q <= l) {
      const float a = (q < l && (bk >> u & 1u)) ? -irs_e2(tb, q, 0.0f) : 0.f;
      ca = a * ca;
      cc = fmaf(a, cc, x[u]);
    }
  }
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const float pa = __shfl_down_sync(0xffffffffu, ca, off), pc = __shfl_down_sync(0xffffffffu, cc, off);
    if (lane + off < 32) {
      cc = fmaf(ca, pc, cc);
      ca = ca * pa;
    }
  }
  prev = __shfl_down_sync(0xffffffffu, cc, 1);
  if (lane == 31) prev = 0.f;
#pragma unroll
  for (int u = K - 1; u >= 0; u--) {
    const int q = q0 + u;
    if (q <= l) {
      if (q < l && (bk >> u & 1u)) x[u] = fmaf(-irs_e2(tb, q, 0.0f), prev, x[u]);
      prev = x[u];
      dst[q] = x[u];
    }
  }
}

// the rows a lane of k_irs_scan_i takes for a line of len rows (0: none fits)
inline int irs_scan_k(int len) {
  const int need = (len + 31) / 32;
  const int ks[] = {2, 4, 6, 8, 12, 16};
  for (int q : ks)
    if (need <= q) return q;
  return 0;
}

template <typename TS, typename TO, int D>
__global__ void k_irs_mixed(DevBlock<double> b, IrsTables tb, float bb, const TS* src, float* mid, TO* out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 5 * irs_lines<double, D>(b)) body_irs_mixed<TS, TO, D>(b, tb, bb, src, mid, out, t);
}

// Shared-memory variant of body_irs: a block stages LT whole lines of one
// variable (and their blanking) in shared memory with coalesced loads, each
// of its first LT threads runs the reference's sweep on one line there, and
// the block writes the lines back coalesced.  Arithmetic and order per line
// are those of body_irs.
// Loads from src and stores to dst (both dw, except for the FP32 copy of the
// mixed form's i sweep: dw in, the copy out, every cell of the tile written)
template <typename T, typename TC, int D, int LT, typename TS, typename TO>
__device__ __forceinline__ void body_irs_smem(const DevBlock<T>& b, const IrsTables& tb, TC bb, const TS* src,
                                              TO* dst) {
  extern __shared__ unsigned char smem_raw[];
  const long long lines = irs_lines<T, D>(b);
  const long long ntile = (lines + LT - 1) / LT;
  const int v = (int)(blockIdx.x / ntile);
  const long long tile = blockIdx.x - (long long)v * ntile;
  const long long l0 = tile * LT;
  const int nl = (int)min((long long)LT, lines - l0);
  const int l = (D == 0) ? b.il : (D == 1 ? b.jl : b.kl);   // rows 2..l
  const int len = l - 1;
  const int S = (D == 0) ? (len | 1) : LT;                  // odd row stride for line-major tiles
  TC* x = (TC*)smem_raw;
  unsigned char* bl = smem_raw + sizeof(TC) * (size_t)LT * (len + 1);
  const TS* d = src + (long long)v * b.N;
  TO* dout = dst + (long long)v * b.N;
  const long long N = b.N;
  (void)N;
  // element (line r, row q) of the tile -> global cell
  auto cell = [&](int r, int q) -> long long {
    long long ln = l0 + r;
    if (D == 0) {
      int j = 2 + (int)((unsigned)ln % (unsigned)b.ny), k = 2 + (int)((unsigned)ln / (unsigned)b.ny);
      return cidx(b.Pi, b.Pj, 2 + q, j, k);
    } else if (D == 1) {
      int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), k = 2 + (int)((unsigned)ln / (unsigned)b.nx);
      return cidx(b.Pi, b.Pj, i, 2 + q, k);
    } else {
      int i = 2 + (int)((unsigned)ln % (unsigned)b.nx), j = 2 + (int)((unsigned)ln / (unsigned)b.nx);
      return cidx(b.Pi, b.Pj, i, j, 2 + q);
    }
  };
  auto sidx = [&](int r, int q) -> int { return D == 0 ? r * S + q : q * LT + r; };
  const int tot = nl * len;
  for (int e = threadIdx.x; e < LT * len; e += blockDim.x) {
    int r, q;
    if (D == 0) { r = e / len; q = e - r * len; } else { q = e / LT; r = e - q * LT; }
    if (r < nl) {
      long long c = cell(r, q);
      x[sidx(r, q)] = (TC)d[c];
      bl[sidx(r, q)] = b.blank[c];
    }
  }
  __syncthreads();
  const int r = threadIdx.x;
  if (r < nl) {
    TC prev;
    {
      TC xv = x[sidx(r, 0)];
      if (bl[sidx(r, 0)] != 0) {
        xv = xv / irs_e1(tb, 2, TC(0));
        x[sidx(r, 0)] = xv;
      }
      prev = xv;
    }
    for (int q = 1; q < len; q++) {
      TC xv = x[sidx(r, q)];
      if (bl[sidx(r, q)] != 0) {
        xv = mdiv(xv - bb * prev, irs_e1(tb, q + 2, TC(0)), irs_e1r(tb, q + 2, TC(0)));
        x[sidx(r, q)] = xv;
      }
      prev = xv;
    }
    for (int q = len - 2; q >= 0; q--) {
      TC xv = x[sidx(r, q)];
      if (bl[sidx(r, q)] != 0) {
        xv = xv - irs_e2(tb, q + 2, TC(0)) * prev;
        x[sidx(r, q)] = xv;
      }
      prev = xv;
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < LT * len; e += blockDim.x) {
    int rr, q;
    if (D == 0) { rr = e / len; q = e - rr * len; } else { q = e / LT; rr = e - q * LT; }
    if (rr < nl) dout[cell(rr, q)] = (TO)x[sidx(rr, q)];
  }
  (void)tot;
}

template <typename T, typename TC, int D, int LT>
__global__ void __launch_bounds__(LT) k_irs_smem(DevBlock<T> b, IrsTables tb, TC bb) {
  body_irs_smem<T, TC, D, LT>(b, tb, bb, (const T*)b.dw, b.dw);
}

// the mixed form's i sweep in shared-memory tiles: dw in, the FP32 copy out
template <int LT>
__global__ void __launch_bounds__(LT) k_irs_smem_fill(DevBlock<double> b, IrsTables tb, float bb, float* cp) {
  body_irs_smem<double, float, 0, LT>(b, tb, bb, (const double*)b.dw, cp);
}

template <typename TC, int LT>
size_t irs_smem_bytes(int len) {
  return sizeof(TC) * (size_t)LT * (len + 1) + (size_t)LT * (len + 1);
}

// update after smoothing, euler.f90:381-399 (steady: lam = 1)
// --------------------------------------------------------------- psmoo + progon3 (irs_variant 1)
// psmoo.f90:1-95 with progon3.f90:41-60: per-cell coefficients eps from the
// time step, aa = 1+2eps, bb = cc = -eps with the end couplings zeroed
// (psmoo.f90:49-50), solved by progon3's forward/backward recurrences.  One
// thread per line carries all five variables: the coefficient recurrences v
// and w do not depend on the variable and are formed once.  The recurrences
// pass through the stage scratch F, dead between the residual pass and the
// next stage: slot q of a line holds progon3's v(q), w(q), u(q,1:5) on the
// way forward and s(q-1), t(q-1,1:5) on the way back.
template <typename T, typename TC, int D>
__device__ __noinline__ void body_psmoo_line(const DevBlock<T>& b, long long ln) {
  const long long N = b.N;
  long long c0, st;
  int l;
  line_of<T, D>(b, ln, c0, st, l);
  const T* eps = b.eps + (long long)D * N;
  T* Sv = b.F;          // v forward, s backward
  T* Sw = b.F + N;      // w forward
  T* Su = b.F + 2 * N;  // u(1:5) forward, t(1:5) backward
  // forward: equation i = 1..n sits at cell q = i+1 = 2..l (n = l-1)
  TC v = TC(0), w = TC(1), u[5];
#pragma unroll
  for (int x = 0; x < 5; x++) u[x] = TC(0);
  for (int q = 2; q <= l; q++) {
    const long long c = c0 + q * st;
    const TC e = (TC)eps[c];
    const TC a = TC(1) + TC(2) * e;
    const TC bq = (q == l) ? TC(0) : -e;
    const TC cq = (q == 2) ? TC(0) : -e;
    const TC z = TC(1) / (a + cq * v);
    v = -bq * z;
#pragma unroll
    for (int x = 0; x < 5; x++) u[x] = (-cq * u[x] + (TC)b.dw[x * N + c]) * z;
    w = -cq * w * z;
    if (q < l) {  // v(n+1), w(n+1), u(n+1) are never read back
      Sv[c] = (T)v;
      Sw[c] = (T)w;
#pragma unroll
      for (int x = 0; x < 5; x++) Su[x * N + c] = (T)u[x];
    }
  }
  // backward: s(i) = v(i+1) s(i+1) + w(i+1), t likewise, i = n-1..1, read
  // from slot i+1 and stored back there; s(n-1), t(n-1) are kept for x(n)
  // (zero when n = 1, progon3's s(0), t(0))
  TC s = TC(1), t[5], shi = TC(0), thi[5];
#pragma unroll
  for (int x = 0; x < 5; x++) t[x] = thi[x] = TC(0);
  for (int q = l - 1; q >= 2; q--) {
    const long long c = c0 + q * st;
    const TC vv = (TC)Sv[c], ww = (TC)Sw[c];
    s = vv * s + ww;
#pragma unroll
    for (int x = 0; x < 5; x++) t[x] = vv * t[x] + (TC)Su[x * N + c];
    Sv[c] = (T)s;
#pragma unroll
    for (int x = 0; x < 5; x++) Su[x * N + c] = (T)t[x];
    if (q == l - 1) {
      shi = s;
#pragma unroll
      for (int x = 0; x < 5; x++) thi[x] = t[x];
    }
  }
  // x(n) at cell l, then x(i) = s(i) x(n) + t(i) at cells 2..l-1
  const long long cl = c0 + l * st;
  const TC el = (TC)eps[cl];
  const TC an = TC(1) + TC(2) * el, bn = TC(0), cn = (l == 2) ? TC(0) : -el;
  const TC den = an + bn * s + cn * shi;
  TC xn[5];
#pragma unroll
  for (int x = 0; x < 5; x++) xn[x] = ((TC)b.dw[x * N + cl] - bn * t[x] - cn * thi[x]) / den;
  for (int q = 2; q <= l - 1; q++) {
    const long long c = c0 + q * st;
    const TC sv = (TC)Sv[c];
#pragma unroll
    for (int x = 0; x < 5; x++) b.dw[x * N + c] = (T)(sv * xn[x] + (TC)Su[x * N + c]);
  }
#pragma unroll
  for (int x = 0; x < 5; x++) b.dw[x * N + cl] = (T)xn[x];
}

template <typename T, typename TC, int D>
__global__ void k_psmoo_line(DevBlock<T> b) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < irs_lines<T, D>(b)) body_psmoo_line<T, TC, D>(b, t);
}

template <typename T, bool S = true>
__device__ __forceinline__ void body_update(const DevBlock<T>& b, const PhysParams& P, const StageArgs& A,
                                            long long t) {
  int i, j, k;
  cell_of(t, b.nx, b.ny, 2, i, j, k);
  const long long N = b.N;
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  T wv[5];
  if (P.unsteady && !A.forcing) {
    const T lam = unsteady_lam(b, P, A, c), rl = T(1) / lam;
#pragma unroll
    for (int v = 0; v < 5; v++) wv[v] = b.wn[v * N + c] - mdiv(b.dw[v * N + c], lam, rl);
  } else {
#pragma unroll
    for (int v = 0; v < 5; v++) wv[v] = b.wn[v * N + c] - b.dw[v * N + c];
  }
#pragma unroll
  for (int v = 0; v < 5; v++) b.w[v * N + c] = wv[v];
  b.p[c] = depvars<S>((T)P.gamma, wv);
}

// --------------------------------------------------------------- bc_cutcell (bc_cutcell.f90:40-268)
// Eight lanes a record: lane q fetches cloud cell q's place and weight, lane v
// sums variable v over the cloud (lane 5 the pressure) in the cloud's order with
// its eight loads in flight together, and lanes 0-2 divide the normal's
// components.  One thread a record walked the cloud 48 loads in a row, 20-34 us
// by events; this takes 10 by itself and nothing beside the face ghosts.  All
// eight entries are loaded: those past the cloud, and all of an empty one, hold
// the record's own cell (mge_add_block).  Every lane of a warp calls it.
template <typename T>
__device__ __forceinline__ void cutcell_lanes(const DevBlock<T>& b, const PhysParams& P, unsigned* err, int t) {
  const int lane = t & 7, v = lane < 5 ? lane : 0;
  const int mm = t >> 3, m = mm < b.nmir ? mm : b.nmir - 1;
  const bool own = mm < b.nmir && mm <= b.m0;  // after the first empty cloud the reference returns
  const bool empty = m == b.m0;
  T* ws = b.rec_wsol + 5LL * m;
  const long long N = b.N;
  const int ncl = b.rec_i[8 * m + 5];
  auto from = [&](T x, int l) { return __shfl_sync(0xffffffffu, x, l, 8); };
  const int* ijk = b.rec_cloud + (8 * m + lane) * 3;
  const int cl = (int)cidx(b.Pi, b.Pj, ijk[0], ijk[1], ijk[2]);
  const T cf = (T)b.rec_coef[8 * m + lane];
  const T* src = lane == 5 ? b.p : b.w + v * N;
  T x[8];
#pragma unroll
  for (int q = 0; q < 8; q++) x[q] = src[__shfl_sync(0xffffffffu, cl, q, 8)];
  T sum = T(0);
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const T a = from(cf, q);
    if (q < ncl) sum = sum + a * x[q];
  }
  T nv[3] = {(T)b.rec_nvec[3 * m], (T)b.rec_nvec[3 * m + 1], (T)b.rec_nvec[3 * m + 2]};
  const T qb[3] = {(T)b.rec_qb[3 * m], (T)b.rec_qb[3 * m + 1], (T)b.rec_qb[3 * m + 2]};
  const T nn = sqrt(nv[0] * nv[0] + nv[1] * nv[1] + nv[2] * nv[2]);
  const T nq = (lane == 0 ? nv[0] : (lane == 1 ? nv[1] : nv[2])) / nn;
#pragma unroll
  for (int q = 0; q < 3; q++) nv[q] = from(nq, q);
  T wsol[5];
#pragma unroll
  for (int q = 0; q < 5; q++) wsol[q] = from(sum, q);
  const T psol = from(sum, 5);
  if (!P.eqn_ns) {
    const T qn = T(2) * (nv[0] * (wsol[1] - wsol[0] * qb[0]) + nv[1] * (wsol[2] - wsol[0] * qb[1]) +
                         nv[2] * (wsol[3] - wsol[0] * qb[2]));
#pragma unroll
    for (int q = 0; q < 3; q++) wsol[1 + q] = wsol[1 + q] - qn * nv[q];
  } else {
#pragma unroll
    for (int q = 0; q < 3; q++) wsol[1 + q] = T(2) * qb[q] * wsol[0] - wsol[1 + q];
  }
  wsol[4] = psol / ((T)P.gamma - T(1)) +
            T(0.5) * (wsol[1] * wsol[1] + wsol[2] * wsol[2] + wsol[3] * wsol[3]) / wsol[0];
  bool nan = false;
#pragma unroll
  for (int q = 0; q < 5; q++) nan |= (wsol[q] != wsol[q]);
  if (!own) return;
  if (nan && !empty && !P.eqn_ns && lane == 0) atomicCAS(err, 0u, (unsigned)ERR_NAN);
  // an empty cloud: this record is zeroed
  const T r = lane == 0 ? wsol[0] : (lane == 1 ? wsol[1] : (lane == 2 ? wsol[2] : (lane == 3 ? wsol[3] : wsol[4])));
  if (lane < 5) ws[lane] = empty ? T(0) : r;
  if (lane == 5) b.rec_psol[m] = empty ? T(0) : psol;
}

// --------------------------------------------------------------- face boundary conditions
// the far field's powers: the short forms for gamma = 1.4 in FP64 (fast_pow.cuh)
__device__ __forceinline__ double pow_gm(const PhysParams& P, double x, double gm) {
  if (P.gamma14) return pow_5_2(x, P.pow_dm);
  return pow(x, gm);
}
__device__ __forceinline__ float pow_gm(const PhysParams&, float x, float gm) { return pow(x, gm); }
__device__ __forceinline__ double pow_gamma(const PhysParams& P, double x, double gamma) {
  if (P.gamma14) return pow_7_5(x, P.pow_dg);
  return pow(x, gamma);
}
__device__ __forceinline__ float pow_gamma(const PhysParams&, float x, float gamma) { return pow(x, gamma); }

template <typename T> struct CellState {
  T w[5];
  T p;
};
template <typename T>
__device__ __forceinline__ CellState<T> load_cell(const DevBlock<T>& b, long long c) {
  CellState<T> s;
#pragma unroll
  for (int v = 0; v < 5; v++) s.w[v] = b.w[v * b.N + c];
  s.p = b.p[c];
  return s;
}
template <typename T>
__device__ __forceinline__ void store_cell(const DevBlock<T>& b, long long c, const CellState<T>& s) {
#pragma unroll
  for (int v = 0; v < 5; v++) b.w[v * b.N + c] = s.w[v];
  b.p[c] = s.p;
}

// bc_far.f90:42-284: the ghost state of a far-field face from the state s of
// the cell it is taken from, in place; false (s unchanged) when the normal
// velocity is NaN.  Inflow and outflow differ only in the entropy and in the
// tangential velocities, so both run the same chain; the quotients by the
// cell's density share one reciprocal, those by gamma-1 and gamma take the
// host's (mdiv: the same roundings as the divisions).
template <typename T>
__device__ __forceinline__ bool far_state(const DevBlock<T>& b, const PhysParams& P, int face, CellState<T>& s) {
  const int ax = (face - 1) % 3;
  const T gamma = (T)P.gamma, gm = (T)P.gm;
  const T fn0 = (T)b.fnv[face - 1][0], fn1 = (T)b.fnv[face - 1][1], fn2 = (T)b.fnv[face - 1][2];
  const T fnn = ax == 0 ? fn0 : (ax == 1 ? fn1 : fn2);
  const T y0 = T(1) / s.w[0], gm1 = gamma - T(1), rg1 = rcp_gm1(P, T(0)), rgam = rcp_gamma(P, T(0));
  const T vel_norm = mdiv(s.w[1] * fn0 + s.w[2] * fn1 + s.w[3] * fn2, s.w[0], y0);
  if (vel_norm != vel_norm) return false;
  const bool in = vel_norm <= T(0);
  const T rmi = (T)P.u0[ax] * fnn - mdiv(T(2) * (T)P.c0, gm1, rg1);
  T vv[3];
#pragma unroll
  for (int a = 0; a < 3; a++) vv[a] = mdiv(s.w[1 + a], s.w[0], y0);
  const T un = ax == 0 ? vv[0] : (ax == 1 ? vv[1] : vv[2]);
  const T ce = sqrt(mdiv(gamma * s.p, s.w[0], y0));
  const T rpo = un * fnn + mdiv(T(2) * ce, gm1, rg1);
  const T vn = T(0.5) * (rpo + rmi) * fnn;
  const T ci = T(0.25) * (gamma - T(1)) * (rpo - rmi);
  const T cc = mdiv(ci * ci, gamma, rgam);
  const T si = in ? (T)P.si_far : pow_gamma(P, s.w[0], gamma) / s.p;
  const T rho = pow_gm(P, si * cc, gm);
  const T pr = rho * cc;
#pragma unroll
  for (int a = 0; a < 3; a++) vv[a] = a == ax ? vn : (in ? (T)P.u0[a] : vv[a]);
  s.w[0] = rho;
  s.w[1] = rho * vv[0];
  s.w[2] = rho * vv[1];
  s.w[3] = rho * vv[2];
  s.w[4] = pr * gm + T(0.5) * rho * (vv[0] * vv[0] + vv[1] * vv[1] + vv[2] * vv[2]);
  s.p = pr;
  return true;
}
// the coordinate along a face's axis that its ghost coordinate q takes its
// state from; inner: the source of the inner layer, whatever q's layer
__device__ __forceinline__ int bc_source(int kind, bool low, int l, int q, bool inner) {
  const int lay = inner ? 0 : (low ? 1 - q : q - (l + 1));  // 0: next to the physical cells
  if (kind == -60) return low ? l - lay : 2 + lay;
  const int off = kind == -20 ? 0 : lay;  // both far-field layers take the first cell's state
  return low ? 2 + off : l - off;
}

// bcond.f90:16-42 applies the faces 1..6 one after the other over their
// whole tangential range, so a later face overwrites the edge and corner
// ghosts of an earlier one and reads what the earlier one wrote.  A ghost
// cell's final state is therefore that of its last writer, the
// highest-numbered face (with a boundary condition) whose axis is a ghost
// axis of the cell, applied to a cell with one ghost axis fewer.  The first
// launch forms the cells with one ghost axis; ghost_state follows the writers
// of an edge or corner cell down to such a cell (at most two of them) and
// applies them on the way back.
template <typename T>
__device__ __forceinline__ int ghost_writer(const DevBlock<T>& b, int i, int j, int k) {
  if (((i < 2) | (i > b.il)) + ((j < 2) | (j > b.jl)) + ((k < 2) | (k > b.kl)) < 2) return 0;
  if (k > b.kl && b.bctype[5] != 0) return 6;
  if (j > b.jl && b.bctype[4] != 0) return 5;
  if (i > b.il && b.bctype[3] != 0) return 4;
  if (k < 2 && b.bctype[2] != 0) return 3;
  if (j < 2 && b.bctype[1] != 0) return 2;
  if (i < 2 && b.bctype[0] != 0) return 1;
  return 0;
}
// moves (i, j, k) to the cell face f takes its state from; true when the
// pressure comes from another one (bc_wall.f90 gives both layers the pressure
// of the first physical cell), whose coordinate along the axis is then srp
template <typename T>
__device__ __forceinline__ bool ghost_source(const DevBlock<T>& b, int f, int& i, int& j, int& k, int& srp) {
  const int ax = (f - 1) % 3, kind = b.bctype[f - 1];
  const int l = ax == 0 ? b.il : (ax == 1 ? b.jl : b.kl), g = ax == 0 ? i : (ax == 1 ? j : k);
  const int src = bc_source(kind, f <= 3, l, g, false);
  if (ax == 0) i = src;
  else if (ax == 1) j = src;
  else k = src;
  srp = bc_source(kind, f <= 3, l, g, true);
  return kind == -80 && srp != src;
}
template <typename T>
__device__ __forceinline__ void ghost_apply(const DevBlock<T>& b, const PhysParams& P, int f, CellState<T>& s) {
  const int ax = (f - 1) % 3, kind = b.bctype[f - 1];
  if (kind == -20) {
    // a NaN normal velocity passes the state on: it has already stopped the run
    far_state(b, P, f, s);
  } else if (kind != -60) {
#pragma unroll
    for (int a = 0; a < 3; a++)
      if (kind == -80 || a == ax) s.w[1 + a] = -s.w[1 + a];
  }
}
// with walls among the faces: the pressure may follow another chain of cells
template <typename T, int DEPTH>
__device__ __noinline__ void ghost_state_wall(const DevBlock<T>& b, const PhysParams& P, int i, int j, int k,
                                              CellState<T>& s) {
  const int f = DEPTH > 0 ? ghost_writer(b, i, j, k) : 0;
  if (!f) {
    s = load_cell(b, cidx(b.Pi, b.Pj, i, j, k));
    return;
  }
  if constexpr (DEPTH > 0) {
    int srp;
    const bool other = ghost_source(b, f, i, j, k, srp);
    ghost_state_wall<T, DEPTH - 1>(b, P, i, j, k, s);
    ghost_apply(b, P, f, s);
    if (other) {
      const int ax = (f - 1) % 3;
      CellState<T> q;
      ghost_state_wall<T, DEPTH - 1>(b, P, ax == 0 ? srp : i, ax == 1 ? srp : j, ax == 2 ? srp : k, q);
      s.p = q.p;
    }
  }
}
// the state an edge or corner ghost takes from the faces; false when no face
// writes the cell (s is then what is stored there)
template <typename T>
__device__ __forceinline__ bool ghost_state(const DevBlock<T>& b, const PhysParams& P, int i, int j, int k,
                                            CellState<T>& s) {
  const int f0 = ghost_writer(b, i, j, k);
  bool wall = false;
#pragma unroll
  for (int q = 0; q < 6; q++) wall |= b.bctype[q] == -80;
  if (wall) {  // the same for every lane
    ghost_state_wall<T, 2>(b, P, i, j, k, s);
    return f0 != 0;
  }
  int srp, f1 = 0;
  if (f0) {
    ghost_source(b, f0, i, j, k, srp);
    f1 = ghost_writer(b, i, j, k);
    if (f1) ghost_source(b, f1, i, j, k, srp);
  }
  s = load_cell(b, cidx(b.Pi, b.Pj, i, j, k));
  // one copy of the far field's chain, its lanes together: calls from the
  // levels of a recursion ran them apart and cost three times as much
#pragma unroll 1
  for (int q = 0; q < 2; q++) {
    const int f = q == 0 ? f1 : f0;
    if (f) ghost_apply(b, P, f, s);
  }
  return f0 != 0;
}

// Every face carries a boundary condition: all ghosts follow from physical
// cells, and the edge and corner ghosts, the corner cells of bc_corner.f90
// included, take one launch after the face ghosts'.  Otherwise some ghosts
// keep what another routine put there (bc_embed, bc_overlap), and the corner
// cells, which overwrite such ghosts, run as a launch of their own.
template <typename T>
__host__ __device__ __forceinline__ bool bc_whole(const DevBlock<T>& b) {
  return b.bctype[0] && b.bctype[1] && b.bctype[2] && b.bctype[3] && b.bctype[4] && b.bctype[5];
}
// work items, in whole warps: the face ghosts (an item writes both layers);
// the ghost cells with two or three ghost axes (without the corner cells when
// those share the launch); the corner cells, four lanes each
template <typename T>
__host__ __device__ __forceinline__ int bc_n1(const DevBlock<T>& b) {
  return pad32(2 * (b.ny * b.nz + b.nx * b.nz + b.nx * b.ny));
}
template <typename T>
__host__ __device__ __forceinline__ int bc_n2(const DevBlock<T>& b) {
  return pad32(bc_whole(b) ? 12 * (b.nx + b.ny + b.nz) + 48 : 16 * (b.nx + b.ny + b.nz) + 64);
}
template <typename T>
__host__ __device__ __forceinline__ int bc_n3(const DevBlock<T>& b) {
  return pad32(4 * (4 * b.nz + 4 * b.ny + 4 * (b.nx + 2) + 8));
}
template <typename T> long long bc_items_t(const DevBlock<T>& b, int part) {
  if (part == 0) return (long long)bc_n1(b) + (b.cut_beside ? rec_lane_items(b) : 0);
  if (part == 1) return (long long)bc_n2(b) + (bc_whole(b) ? bc_n3(b) : 0);
  return bc_whole(b) ? 0 : bc_n3(b);
}

// the face ghosts whose two tangential coordinates are physical
template <typename T>
__device__ __forceinline__ void body_bc_face(const DevBlock<T>& b, const PhysParams& P, int t) {
  const int sz[3] = {b.ny * b.nz, b.nx * b.nz, b.nx * b.ny};
  int face = 1;
#pragma unroll
  for (int q = 0; q < 5; q++)
    if (face == q + 1 && t >= sz[q % 3]) {
      t -= sz[q % 3];
      face = q + 2;
    }
  const int ax = (face - 1) % 3, kind = b.bctype[face - 1];
  if (kind == 0 || t >= sz[ax]) return;
  const int na = ax == 0 ? b.ny : b.nx;
  const int t1 = 2 + t % na, t2 = 2 + t / na;
  const int l = ax == 0 ? b.il : (ax == 1 ? b.jl : b.kl);
  auto at = [&](int q) -> long long {
    return ax == 0 ? cidx(b.Pi, b.Pj, q, t1, t2) : (ax == 1 ? cidx(b.Pi, b.Pj, t1, q, t2) : cidx(b.Pi, b.Pj, t1, t2, q));
  };
  const bool low = face <= 3;
  const int g1 = low ? 1 : l + 1, g2 = low ? 0 : l + 2;
  const long long d1 = at(g1), d2 = at(g2);
  CellState<T> s1 = load_cell(b, at(bc_source(kind, low, l, g1, false))), s2;
  if (kind == -20) {
    if (far_state(b, P, face, s1))
      s2 = s1;
    else
      s1 = s2 = load_cell(b, d1);  // NaN normal velocity: the second layer copies the first as it stands
  } else {
    s2 = load_cell(b, at(bc_source(kind, low, l, g2, false)));
#pragma unroll
    for (int a = 0; a < 3; a++)
      if (kind == -80 || (kind == -50 && a == ax)) {
        s1.w[1 + a] = -s1.w[1 + a];
        s2.w[1 + a] = -s2.w[1 + a];
      }
    if (kind == -80) s2.p = s1.p;
  }
  store_cell(b, d1, s1);
  store_cell(b, d2, s2);
}

// the ghost coordinate of a side (0 low, 1 high) and layer (0 inner)
__device__ __forceinline__ int ghost_coord(int l, int side, int lay) { return side ? l + 1 + lay : 1 - lay; }

// the ghost cells with two or three ghost axes
template <typename T>
__device__ __forceinline__ void body_bc_edge(const DevBlock<T>& b, const PhysParams& P, int t) {
  const bool all = !bc_whole(b);  // with the corner cells' own ghost states
  const int nc = all ? 16 : 12;
  int i, j, k;
  auto combo = [&](int q, int la, int lb, int& ca, int& cb) {
    const int m = q % 3;
    const int s = all ? q >> 2 : q / 3, l1 = all ? q & 1 : (m >= 1), l2 = all ? (q >> 1) & 1 : (m != 1);
    ca = ghost_coord(la, s & 1, l1);
    cb = ghost_coord(lb, s >> 1, l2);
  };
  if (t < nc * b.nz) {
    combo(t / b.nz, b.il, b.jl, i, j);
    k = 2 + t % b.nz;
  } else if ((t -= nc * b.nz) < nc * b.ny) {
    combo(t / b.ny, b.il, b.kl, i, k);
    j = 2 + t % b.ny;
  } else if ((t -= nc * b.ny) < nc * b.nx) {
    combo(t / b.nx, b.jl, b.kl, j, k);
    i = 2 + t % b.nx;
  } else if ((t -= nc * b.nx) < 4 * nc) {
    const int e = t & 3;
    i = ghost_coord(b.il, e & 1, e >> 1);
    combo(t >> 2, b.jl, b.kl, j, k);
  } else {
    i = j = k = 2;  // padding: a physical cell, not written
  }
  CellState<T> s;
  if (ghost_state(b, P, i, j, k, s)) store_cell(b, cidx(b.Pi, b.Pj, i, j, k), s);
}

// The corner cells of bc_corner.f90:23-157, after the faces: the inner edges
// along k and j (k, j physical) from the two face ghosts beside them and the
// physical cell, then those along i over the whole range, then the eight
// corners from three such edge cells.  Four lanes share a cell: each takes
// one of its terms, and lane 0 adds them up.  A corner's edge cells are formed
// again from the face ghosts instead of waiting for the lanes that own them.
// (0..ib, je, 1) is bc_corner.f90:120 as written, (x + a) - a; the corner
// groups there also write the edge cell they read, because where the corner
// cells run by themselves its ghost state is what is stored.
// Every lane of a warp calls it.
template <typename T>
__device__ __forceinline__ void body_bc_corner(const DevBlock<T>& b, const PhysParams& P, int t) {
  const int g0 = t >> 2, lane = t & 3;
  const int il = b.il, jl = b.jl, kl = b.kl, ie = b.ie, je = b.je, ke = b.ke;
  const int n0 = 4 * b.nz, n1 = 4 * b.ny, n2 = 4 * (b.nx + 2);
  int g = g0, kind = -1;  // 0: three-term edge, 1: (x + a) - a, 2: corner
  int i = 2, j = 2, k = 2, ii = 2, jj = 2, kk = 2;  // the cell and the physical coordinates beside it
  int a0 = 2, a1 = 2, a2 = 2;                       // this lane's term
  if (g < n0) {
    const int e = g / b.nz;
    k = kk = 2 + g % b.nz;
    i = e & 1 ? ie : 1, ii = e & 1 ? il : 2;
    j = e >> 1 ? je : 1, jj = e >> 1 ? jl : 2;
    kind = 0;
    a0 = lane == 1 ? i : ii, a1 = lane == 0 ? j : jj, a2 = k;
  } else if ((g -= n0) < n1) {
    const int e = g / b.ny;
    j = jj = 2 + g % b.ny;
    i = e & 1 ? ie : 1, ii = e & 1 ? il : 2;
    k = e >> 1 ? ke : 1, kk = e >> 1 ? kl : 2;
    kind = 0;
    a0 = lane == 1 ? i : ii, a1 = j, a2 = lane == 0 ? k : kk;
  } else if ((g -= n1) < n2) {
    const int e = g / (b.nx + 2), q = g % (b.nx + 2);
    i = ii = q == 0 ? 0 : (q <= b.nx ? 1 + q : b.ib);
    j = e & 1 ? je : 1, jj = e & 1 ? jl : 2;
    k = e >> 1 ? ke : 1, kk = e >> 1 ? kl : 2;
    kind = e == 1 ? 1 : 0;
    a0 = i;
    a1 = lane == (kind == 1 ? 0 : 1) ? j : jj;
    a2 = lane == 0 ? k : kk;
    // the cells next to a corner of that edge are written by the corner's group
    if (kind == 1 && (i == 2 || i == il)) kind = -1;
  } else if ((g -= n2) < 8) {
    i = g & 1 ? ie : 1, ii = g & 1 ? il : 2;
    j = (g >> 1) & 1 ? je : 1, jj = (g >> 1) & 1 ? jl : 2;
    k = g >> 2 ? ke : 1, kk = g >> 2 ? kl : 2;
    kind = 2;
    a0 = lane == 2 ? i : ii;
    a1 = lane == 1 || lane == 3 ? j : jj;
    a2 = lane == 0 || lane == 3 ? k : kk;
    if (lane == 3 && !(j == je && k == 1)) a1 = jj, a2 = kk;  // only that edge's own state is a term
  }
  CellState<T> s;
  if (kind < 0 || (kind < 2 && lane == 3)) a0 = a1 = a2 = 2;  // no term: a physical cell
  if (bc_whole(b))
    ghost_state(b, P, a0, a1, a2, s);  // face ghosts and physical cells as stored
  else
    s = load_cell(b, cidx(b.Pi, b.Pj, a0, a1, a2));
  T x[5], y[5], z[5], u[5];
  const int lead = threadIdx.x & 28;
#pragma unroll
  for (int v = 0; v < 5; v++) {
    x[v] = __shfl_sync(0xffffffffu, s.w[v], lead);
    y[v] = __shfl_sync(0xffffffffu, s.w[v], lead + 1);
    z[v] = __shfl_sync(0xffffffffu, s.w[v], lead + 2);
    u[v] = __shfl_sync(0xffffffffu, s.w[v], lead + 3);
  }
  if (kind < 0 || lane != 0) return;
  const T gamma = (T)P.gamma;
  CellState<T> o;
  if (kind < 2) {
#pragma unroll
    for (int v = 0; v < 5; v++) o.w[v] = x[v] + y[v] - z[v];
  } else {
    const long long dq = cidx(b.Pi, b.Pj, ii, jj, kk);
    const bool asis = j == je && k == 1;
    CellState<T> e;
#pragma unroll
    for (int v = 0; v < 5; v++) {
      const T d = b.w[v * b.N + dq];
      e.w[v] = asis ? u[v] + d - d : x[v] + y[v] - d;  // (ii, j, k)
      const T bq = x[v] + z[v] - d;                     // (i, jj, k)
      const T cq = y[v] + z[v] - d;                     // (i, j, kk)
      o.w[v] = mdiv((e.w[v] + bq + cq) * T(2), T(3), T(1) / T(3)) - d;
    }
    if (asis) {
      e.p = depvars<false>(gamma, e.w);
      store_cell(b, cidx(b.Pi, b.Pj, ii, j, k), e);
    }
  }
  o.p = depvars<false>(gamma, o.w);
  store_cell(b, cidx(b.Pi, b.Pj, i, j, k), o);
}

// part 0: the face ghosts and, with cut, the records' solid states where every
// cloud cell is physical (bc_cutcell then reads none of the ghosts and writes
// only the records); 1: the edge and corner ghosts; 2: the corner cells of
// blocks with a face without a boundary condition
template <typename T, int PART>
__device__ __forceinline__ void body_bcond(const DevBlock<T>& b, const PhysParams& P, unsigned* err, int cut,
                                           long long t) {
  if (PART == 0) {
    const int n1 = bc_n1(b);
    if (t < n1)
      body_bc_face(b, P, (int)t);
    else if (cut && b.cut_beside && t < (long long)n1 + rec_lane_items(b))
      cutcell_lanes(b, P, err, (int)t - n1);
  } else if (PART == 1) {
    const int n2 = bc_n2(b);
    if (t < n2)
      body_bc_edge(b, P, (int)t);
    else if (bc_whole(b) && t < (long long)n2 + bc_n3(b))
      body_bc_corner(b, P, (int)t - n2);
  } else {
    if (!bc_whole(b) && t < bc_n3(b)) body_bc_corner(b, P, (int)t);
  }
}
// Bound by latency at every size that matters: a far-field ghost is a chain
// of some 1,100 dependent instructions.  Three launches for the faces and
// three for the corners, each item of a warp on a branch of its own, took 74 us
// a stage on a 24^3 block; these take 9 us for the faces and, after the last
// stage of an inviscid update only (StageArgs::faces_only), 15 us more.
template <typename T, int PART>
__global__ void k_bcond(DevBlock<T> b, PhysParams P, unsigned* err, int cut) {
  body_bcond<T, PART>(b, P, err, cut, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// --------------------------------------------------------------- residual norm (euler.f90:431-447)
// Deterministic: fixed partial ranges, fixed-order tree per block, one final block.
constexpr int RT_THREADS = 256;
#if MGE_PART == 0
int rtrms_partials(long long ncells) {
  long long per = (long long)RT_THREADS * 8;
  long long n = (ncells + per - 1) / per;
  return (int)(n < 1 ? 1 : (n > 4096 ? 4096 : n));
}
#endif

// An infinite value counts as NaN where the last stage was smoothed: the sweeps turn
// it into NaN except where their short quotient (irs_quick) leaves an infinity, and
// the stop on the residual does not depend on the form of the sweep.  It leaves its
// thread's sum infinite, so only such a sum looks for it (a test of every value took
// 3 us an update at 24^3).
template <typename T>
__device__ void body_rtrms_partial(const DevBlock<T>& b, const PhysParams& P, double* partial, int npart, int part) {
  __shared__ double sh[RT_THREADS];
  const long long tot = (long long)b.nx * b.ny * b.nz;
  const long long per = (tot + npart - 1) / npart;
  const long long lo = (long long)part * per, hi = min(tot, lo + per);
  double acc = 0.0;
  for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    int i, j, k;
    cell_of(t, b.nx, b.ny, 2, i, j, k);
    long long c = cidx(b.Pi, b.Pj, i, j, k);
    double de = smul(P.cfl, (double)(P.vt ? *b.dtim : b.vdtim[c]));
    double rt = 0.0;
    if (b.blank[c] != 0) rt = sdiv((double)b.dw[c], de);
    acc = acc + smul(rt, rt);
  }
  auto infinite = [](double x) { return ((unsigned)__double2hiint(x) & 0x7ff00000u) == 0x7ff00000u; };
  if (P.last_smoothed && infinite(acc)) {
    for (long long t = lo + threadIdx.x; t < hi; t += blockDim.x) {
      int i, j, k;
      cell_of(t, b.nx, b.ny, 2, i, j, k);
      const long long c = cidx(b.Pi, b.Pj, i, j, k);
      if (b.blank[c] != 0 && infinite((double)b.dw[c])) acc = acc * 0.0;
    }
  }
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = RT_THREADS / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] = sh[threadIdx.x] + sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[part] = sh[0];
  __syncthreads();
}

template <typename T>
__global__ void k_rtrms_partial(DevBlock<T> b, PhysParams P, double* partial, int npart) {
  body_rtrms_partial(b, P, partial, npart, blockIdx.x);
}

// The partial sums in a fixed order by one warp: lane l adds the partials
// l, l+32, l+64, ... in turn, then the lanes' sums fold in a fixed halving
// tree.  A NaN norm is the stop of solver.f90:180, recorded in launch order
// like the kernels' other stops (err may be null).  Every lane of warp 0
// calls it.
__device__ __forceinline__ void body_rtrms_final(const double* partial, int npart, double ncell, double* out,
                                                 unsigned* err) {
  const int lane = threadIdx.x & 31;
  double a = 0.0;
  for (int q = lane; q < npart; q += 32) a = a + partial[q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, o);
  if (lane == 0) {
    const double r = sqrt(a / ncell);
    *out = r;
    if (err && r != r) atomicCAS(err, 0u, (unsigned)ERR_NANRES);
  }
}

static __global__ void k_rtrms_final(const double* partial, int npart, double ncell, double* out, unsigned* err) {
  if (blockIdx.x == 0 && threadIdx.x < 32) body_rtrms_final(partial, npart, ncell, out, err);
}

// --------------------------------------------------------------- small whole-array kernels
template <typename T>
__device__ __forceinline__ void body_depvars(const DevBlock<T>& b, double gamma, long long c) {
  if (c >= b.N) return;
  T wv[5];
  for (int v = 0; v < 5; v++) wv[v] = b.w[v * b.N + c];
  b.p[c] = depvars((T)gamma, wv);
}
template <typename T>
__global__ void k_depvars_all(DevBlock<T> b, double gamma) {
  body_depvars(b, gamma, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

template <typename T>
__global__ void k_copy5(const T* __restrict__ src, T* __restrict__ dst, long long n) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < n) dst[c] = src[c];
}

// wn = w on physical cells (euler.f90:80-83, movco.f90:29-35).  The zeros
// euler.f90:84-89 puts into dw and fw need no pass: a stage writes dw whole before
// anything reads it, the first stage writes fw, and no ghost of either is
// ever written after the zeros of their allocation.
template <typename T>
__device__ __forceinline__ void body_copy_wn(const DevBlock<T>& b, long long c) {
  if (c >= b.N) return;
  int i, j, k;
  cell_of(c, b.Pi, b.Pj, 0, i, j, k);
  if (!(i >= 2 && i <= b.il && j >= 2 && j <= b.jl && k >= 2 && k <= b.kl)) return;
  for (int v = 0; v < 5; v++) b.wn[v * b.N + c] = b.w[v * b.N + c];
}
// depvars on every cell and wn = w on the physical ones, from one read of w
template <typename T>
__device__ __forceinline__ void body_depvars_wn(const DevBlock<T>& b, double gamma, long long c) {
  if (c >= b.N) return;
  int i, j, k;
  cell_of(c, b.Pi, b.Pj, 0, i, j, k);
  const bool phys = i >= 2 && i <= b.il && j >= 2 && j <= b.jl && k >= 2 && k <= b.kl;
  T wv[5];
#pragma unroll
  for (int v = 0; v < 5; v++) {
    wv[v] = b.w[v * b.N + c];
    if (phys) b.wn[v * b.N + c] = wv[v];
  }
  b.p[c] = depvars((T)gamma, wv);
}
template <typename T>
__global__ void k_depvars_wn(DevBlock<T> b, double gamma) {
  body_depvars_wn(b, gamma, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
template <typename T>
__global__ void k_copy_wn(DevBlock<T> b) {
  body_copy_wn(b, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

template <typename T>
__global__ void k_init_free(DevBlock<T> b, PhysParams P) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= b.N) return;
  const long long N = b.N;
  double rho0 = P.rho0;
  b.w[c] = (T)rho0;
  b.w[N + c] = (T)(rho0 * P.u0[0]);
  b.w[2 * N + c] = (T)(rho0 * P.u0[1]);
  b.w[3 * N + c] = (T)(rho0 * P.u0[2]);
  b.w[4 * N + c] = (T)P.e0;  // rho0*h0 - p0, init_flow.f90:59
}

// --------------------------------------------------------------- multigrid transfers
__device__ __forceinline__ void trilinear_factor(double x, double y, double z, double* fac) {
  fac[0] = (1.0 - x) * (1.0 - y) * (1.0 - z);
  fac[1] = x * (1.0 - y) * (1.0 - z);
  fac[2] = (1.0 - x) * y * (1.0 - z);
  fac[3] = x * y * (1.0 - z);
  fac[4] = (1.0 - x) * (1.0 - y) * z;
  fac[5] = x * (1.0 - y) * z;
  fac[6] = (1.0 - x) * y * z;
  fac[7] = x * y * z;
}

struct Xfer {
  int r[3], o[3];
  double rinv[3];  // 1/r when r is a power of two (x/r = x*(1/r) exactly), else 0
};

// collc.f90:58-158 for the coarse cells under one child
template <typename TC, typename TF>
__device__ __forceinline__ long long collc_items(const DevBlock<TC>&, const DevBlock<TF>& f, const Xfer& X) {
  return (long long)(f.nx / X.r[0]) * (f.ny / X.r[1]) * (f.nz / X.r[2]);
}
template <typename TC, typename TF>
__device__ __forceinline__ void body_collc(const DevBlock<TC>& c, const DevBlock<TF>& f, const Xfer& X,
                                           uint8_t* marker, long long t) {
  const int n0 = f.nx / X.r[0], n1 = f.ny / X.r[1], n2 = f.nz / X.r[2];
  if (t >= (long long)n0 * n1 * n2) return;
  int ic[3];
  cell_of(t, n0, n1, 2, ic[0], ic[1], ic[2]);
  for (int d = 0; d < 3; d++) ic[d] += X.o[d];
  if (ic[0] < 2 || ic[0] > c.il || ic[1] < 2 || ic[1] > c.jl || ic[2] < 2 || ic[2] > c.kl) return;
  const int lf[3] = {f.il, f.jl, f.kl};
  if constexpr (std::is_same<TC, float>::value && std::is_same<TF, double>::value) {
    // the mixed form's restriction from the FP64 finest level onto an FP32
    // level: the values land in FP32 storage, so the averages are formed in
    // FP32 (the same stencil; the 2:1 weights are exact in FP32)
    int sf[3];
    float xf[3];
    for (int d = 0; d < 3; d++) {
      const float tt = ((float)ic[d] - 1.5f - (float)X.o[d]) * (float)X.r[d];
      int s = (int)floorf(tt + 1.5f);
      s = s < 2 ? 2 : (s > lf[d] - 1 ? lf[d] - 1 : s);
      sf[d] = s;
      xf[d] = tt + 1.5f - (float)s;
    }
    const float wx[2] = {1.0f - xf[0], xf[0]}, wy[2] = {1.0f - xf[1], xf[1]}, wz[2] = {1.0f - xf[2], xf[2]};
    const long long cc = cidx(c.Pi, c.Pj, ic[0], ic[1], ic[2]);
    for (int v = 0; v < 5; v++) {
      float ar = 0.0f, aw = 0.0f;
      for (int dk = 0; dk < 2; dk++)
        for (int dj = 0; dj < 2; dj++)
          for (int di = 0; di < 2; di++) {
            const long long fq = cidx(f.Pi, f.Pj, sf[0] + di, sf[1] + dj, sf[2] + dk);
            const float wt = wx[di] * wy[dj] * wz[dk];
            ar = fmaf((float)f.dw[v * f.N + fq] * f.rvolf, wt, ar);
            aw = fmaf((float)f.w[v * f.N + fq], wt, aw);
          }
      c.wr[v * c.N + cc] = ar * (float)c.vol;
      c.w[v * c.N + cc] = aw;
    }
    marker[cc] = 1;
    return;
  }
  int sh[3];
  double xi[3];
  for (int d = 0; d < 3; d++) {
    double tt = ((double)ic[d] - 1.5 - (double)X.o[d]) * (double)X.r[d];
    int s = (int)floor(tt + 1.5);
    if (s < 2) s = 2;
    if (s > lf[d] - 1) s = lf[d] - 1;
    sh[d] = s;
    xi[d] = tt + 1.5 - (double)s;
  }
  double fac[8];
  trilinear_factor(xi[0], xi[1], xi[2], fac);
  const long long cc = cidx(c.Pi, c.Pj, ic[0], ic[1], ic[2]);
  for (int v = 0; v < 5; v++) {
    double acc = 0.0;
    int nn = 0;
    for (int dk = 0; dk < 2; dk++)
      for (int dj = 0; dj < 2; dj++)
        for (int di = 0; di < 2; di++) {
          long long fq = cidx(f.Pi, f.Pj, sh[0] + di, sh[1] + dj, sh[2] + dk);
          double val = smdiv((double)f.dw[v * f.N + fq], f.vol, f.rvol);
          acc = acc + (dk ? smul(val, fac[nn]) : val * fac[nn]);
          nn++;
        }
    c.wr[v * c.N + cc] = (TC)(acc * c.vol);
    acc = 0.0;
    nn = 0;
    for (int dk = 0; dk < 2; dk++)
      for (int dj = 0; dj < 2; dj++)
        for (int di = 0; di < 2; di++) {
          long long fq = cidx(f.Pi, f.Pj, sh[0] + di, sh[1] + dj, sh[2] + dk);
          acc = acc + (dk ? smul((double)f.w[v * f.N + fq], fac[nn]) : (double)f.w[v * f.N + fq] * fac[nn]);
          nn++;
        }
    c.w[v * c.N + cc] = (TC)acc;
  }
  marker[cc] = 1;
}
template <typename TC, typename TF>
__global__ void k_collc(DevBlock<TC> c, DevBlock<TF> f, Xfer X, uint8_t* marker) {
  body_collc(c, f, X, marker, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

__device__ __forceinline__ bool fine_to_coarse(const Xfer& X, int ncp0, int ncp1, int ncp2, int lc0, int lc1, int lc2,
                                               int i, int j, int k, int* sh, double* fac) {
  int ic[3] = {i, j, k};
  int nc[3] = {ncp0, ncp1, ncp2};
  int lc[3] = {lc0, lc1, lc2};
  double xi[3];
  for (int d = 0; d < 3; d++) {
    const double x = (double)ic[d] - 1.5;
    double u = (double)X.o[d] + (X.rinv[d] > 0.0 ? x * X.rinv[d] : x / (double)X.r[d]);
    if (u < 0.0 || u >= (double)nc[d]) return false;
    int s = (int)floor(u + 1.5);
    if (s < 2) s = 2;
    if (s > lc[d] - 1) s = lc[d] - 1;
    sh[d] = s;
    xi[d] = u + 1.5 - (double)s;
  }
  trilinear_factor(xi[0], xi[1], xi[2], fac);
  return true;
}

// the coarse correction w_c - ws_c of every coarse cell, formed once for the
// 64 fine cells whose interpolation takes it (the same subtraction).  TD: what
// they take it as, FP32 for an FP64 level over an FP32 one: a conversion issues
// at the FP64 rate, and 64 of them for each value took 1.8 of the mixed form's
// 21 ms W-cycle at 192^3.
template <typename TF, typename TC> struct Correction { typedef double type; };
template <> struct Correction<double, float> { typedef float type; };
template <typename TC, typename TD>
__device__ __forceinline__ void body_addw_diff(const DevBlock<TC>& c, TD* dc, long long q) {
  if (q >= c.N) return;
#pragma unroll
  for (int v = 0; v < 5; v++) dc[v * c.N + q] = (TD)((double)c.w[v * c.N + q] - (double)c.ws[v * c.N + q]);
}
template <typename TC, typename TD>
__global__ void k_addw_diff(DevBlock<TC> c, TD* dc) {
  body_addw_diff(c, dc, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// addw.f90:83-188: w_f = store_w + I(w_c - ws_c), or I(w_c) in the FMG step;
// dc holds w_c - ws_c (k_addw_diff) unless fmg
template <typename TF, typename TC>
__device__ __forceinline__ void body_addw(const DevBlock<TF>& f, const DevBlock<TC>& c, const Xfer& X, int fmg,
                                          const typename Correction<TF, TC>::type* dc, int i, int j, int k) {
  if constexpr (std::is_same<TF, double>::value && std::is_same<TC, float>::value) {
    // the mixed form's finest level under an FP32 coarse level: the coarse
    // correction is FP32, so it is interpolated in FP32 (the same stencil
    // and weights, exact in FP32 for power-of-two ratios) and added to the
    // FP64 state in FP64
    if (!fmg) {
      const int ic[3] = {i, j, k}, nc[3] = {c.nx, c.ny, c.nz}, lc[3] = {c.il, c.jl, c.kl};
      int sf[3];
      float xf[3];
      for (int d = 0; d < 3; d++) {
        const float x = (float)ic[d] - 1.5f;
        const float u = (float)X.o[d] + (X.rinv[d] > 0.0 ? x * (float)X.rinv[d] : x / (float)X.r[d]);
        if (u < 0.0f || u >= (float)nc[d]) return;
        int s = (int)floorf(u + 1.5f);
        s = s < 2 ? 2 : (s > lc[d] - 1 ? lc[d] - 1 : s);
        sf[d] = s;
        xf[d] = u + 1.5f - (float)s;
      }
      const long long q = cidx(f.Pi, f.Pj, i, j, k);
      if (f.blank[q] == 0) return;
      const float wx[2] = {1.0f - xf[0], xf[0]}, wy[2] = {1.0f - xf[1], xf[1]}, wz[2] = {1.0f - xf[2], xf[2]};
      for (int v = 0; v < 5; v++) {
        float acc = 0.0f;
        for (int dk = 0; dk < 2; dk++)
          for (int dj = 0; dj < 2; dj++)
            for (int di = 0; di < 2; di++) {
              const long long cq = cidx(c.Pi, c.Pj, sf[0] + di, sf[1] + dj, sf[2] + dk);
              acc = fmaf(dc[v * c.N + cq], wx[di] * wy[dj] * wz[dk], acc);
            }
        f.w[v * f.N + q] = f.w[v * f.N + q] + (double)acc;
      }
      return;
    }
  }
  int sh[3];
  double fac[8];
  if (!fine_to_coarse(X, c.nx, c.ny, c.nz, c.il, c.jl, c.kl, i, j, k, sh, fac)) return;
  const long long q = cidx(f.Pi, f.Pj, i, j, k);
  if (f.blank[q] == 0) return;
  for (int v = 0; v < 5; v++) {
    double acc = 0.0;
    int nn = 0;
    for (int dk = 0; dk < 2; dk++)
      for (int dj = 0; dj < 2; dj++)
        for (int di = 0; di < 2; di++) {
          long long cq = cidx(c.Pi, c.Pj, sh[0] + di, sh[1] + dj, sh[2] + dk);
          double val = fmg ? (double)c.w[v * c.N + cq] : dc[v * c.N + cq];
          // half the products on the integer pipes (smul), half on the FP64 pipe
          acc = acc + (dk ? smul(val, fac[nn]) : val * fac[nn]);
          nn++;
        }
    if (fmg)
      f.w[v * f.N + q] = (TF)acc;
    else
      f.w[v * f.N + q] = (TF)((double)f.w[v * f.N + q] + acc);
  }
}
template <typename TF, typename TC>
__global__ void k_addw(DevBlock<TF> f, DevBlock<TC> c, Xfer X, int fmg, const typename Correction<TF, TC>::type* dc) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)f.nx * f.ny * f.nz) return;
  int i, j, k;
  cell_of(t, f.nx, f.ny, 2, i, j, k);
  body_addw(f, c, X, fmg, dc, i, j, k);
}

// x / 64: the exponent less six where the result is normal (exact), else the product
__device__ __forceinline__ double div64(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const unsigned e = (unsigned)hi & 0x7ff00000u;
  if (e - 0x00700000u < 0x7f800000u) return __hiloint2double(hi - 0x00600000, lo);
  return x * 0.015625;
}
// The 2:1 prolongation of FP64 arithmetic, eight fine cells a thread: the cells
// 2m+1 and 2m+2 along each axis lie between the coarse centres s = o+m+1 and s+1,
// so they share a stencil, and their weights 27, 9, 3 and 1 over 64 make four
// products of each coarse value for all eight instead of one a cell each.  The
// products round and add as a cell by itself forms them.  The fine cells along
// the block's faces, whose stencil may be clamped, take k_addw_shell.  One cell
// a thread spent about 100 FP64 operations on its weights, products and sums;
// this spends 45 (1.0 ms less at 192^3).
template <typename TF, typename TC>
__global__ void __launch_bounds__(128) k_addw_octet(DevBlock<TF> f, DevBlock<TC> c, Xfer X, int fmg, const double* dc) {
  const int n0 = f.nx / 2 - 1, n1 = f.ny / 2 - 1, n2 = f.nz / 2 - 1;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)n0 * n1 * n2) return;
  int mi, mj, mk;
  cell_of(t, n0, n1, 1, mi, mj, mk);
  const long long q0 = cidx(c.Pi, c.Pj, X.o[0] + mi + 1, X.o[1] + mj + 1, X.o[2] + mk + 1);
  const long long f0 = cidx(f.Pi, f.Pj, 2 * mi + 1, 2 * mj + 1, 2 * mk + 1);
  const long long cj = c.Pi, ck = (long long)c.Pi * c.Pj, fj = f.Pi, fk = (long long)f.Pi * f.Pj;
  bool fluid[8];
#pragma unroll
  for (int e = 0; e < 8; e++) fluid[e] = f.blank[f0 + (e & 1) + ((e >> 1) & 1) * fj + (e >> 2) * fk] != 0;
#pragma unroll 1
  for (int v = 0; v < 5; v++) {
    double p[8][4];  // the coarse values times 27, 9, 3, 1 over 64
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const long long q = q0 + (e & 1) + ((e >> 1) & 1) * cj + (e >> 2) * ck;
      const double x = fmg ? (double)c.w[v * c.N + q] : dc[v * c.N + q];
      p[e][0] = x * 0.421875;
      p[e][1] = smul(x, 0.140625);
      p[e][2] = smul(x, 0.046875);
      p[e][3] = div64(x);
    }
#pragma unroll
    for (int e = 0; e < 8; e++) {
      // coarse value n is near fine cell e along the axes where their bits agree:
      // weight 3/4 there, 1/4 where they differ
      double acc = 0.0;
#pragma unroll
      for (int n = 0; n < 8; n++) {
        const int far = ((n ^ e) & 1) + (((n ^ e) >> 1) & 1) + ((n ^ e) >> 2);
        acc = n == 0 ? p[n][far] : acc + p[n][far];
      }
      const long long q = v * f.N + f0 + (e & 1) + ((e >> 1) & 1) * fj + (e >> 2) * fk;
      if (fluid[e]) f.w[q] = fmg ? (TF)acc : (TF)((double)f.w[q] + acc);
    }
  }
}
// the fine cells on the block's six faces, one at a time
template <typename TF>
__host__ __device__ __forceinline__ long long shell_items(const DevBlock<TF>& f) {
  return 2ll * f.nx * f.ny + 2ll * f.nx * (f.nz - 2) + 2ll * (f.ny - 2) * (f.nz - 2);
}
template <typename TF, typename TC>
__global__ void k_addw_shell(DevBlock<TF> f, DevBlock<TC> c, Xfer X, int fmg, const double* dc) {
  long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t0 >= shell_items(f)) return;
  int t = (int)t0, i, j, k;
  if (t < 2 * f.nx * f.ny) {
    const int r = t % (f.nx * f.ny);
    i = 2 + r % f.nx, j = 2 + r / f.nx, k = t < f.nx * f.ny ? 2 : f.kl;
  } else if ((t -= 2 * f.nx * f.ny) < 2 * f.nx * (f.nz - 2)) {
    const int n = f.nx * (f.nz - 2), r = t % n;
    i = 2 + r % f.nx, k = 3 + r / f.nx, j = t < n ? 2 : f.jl;
  } else {
    t -= 2 * f.nx * (f.nz - 2);
    const int n = (f.ny - 2) * (f.nz - 2), r = t % n;
    j = 3 + r % (f.ny - 2), k = 3 + r / (f.ny - 2), i = t < n ? 2 : f.il;
  }
  body_addw(f, c, X, fmg, dc, i, j, k);
}

// bc_overlap.f90:32-90: ghost cell dst[t] of block g takes the trilinear
// interpolation of partner p's state from the 2x2x2 cells at src[t] (its
// physical cells: no cell is both read and written), then depvars
template <typename T>
__global__ void k_overlap(DevBlock<T> g, DevBlock<T> p, const long long* __restrict__ dst,
                          const long long* __restrict__ src, const double* __restrict__ fac, long long n,
                          double gamma) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const long long q = dst[t], s = src[t];
  const long long sj = p.Pi, sk = (long long)p.Pi * p.Pj;
  const double* f = fac + 8 * t;
  T wv[5];
#pragma unroll
  for (int v = 0; v < 5; v++) {
    double acc = 0.0;
    int nn = 0;
    for (int dk = 0; dk < 2; dk++)
      for (int dj = 0; dj < 2; dj++)
        for (int di = 0; di < 2; di++) acc = acc + (double)p.w[v * p.N + s + di + dj * sj + dk * sk] * f[nn++];
    wv[v] = (T)acc;
    g.w[v * g.N + q] = wv[v];
  }
  g.p[q] = depvars((T)gamma, wv);
}

// bc_embed.f90:47-143: fine ghost cells whose centre lies in the parent
template <typename TF, typename TC>
__device__ __forceinline__ void body_embed(const DevBlock<TF>& f, const DevBlock<TC>& c, const Xfer& X, double gamma,
                                           long long t) {
  if (t >= f.N) return;
  int i, j, k;
  cell_of(t, f.Pi, f.Pj, 0, i, j, k);
  if (i >= 2 && i <= f.il && j >= 2 && j <= f.jl && k >= 2 && k <= f.kl) return;
  int sh[3];
  double fac[8];
  if (!fine_to_coarse(X, c.nx, c.ny, c.nz, c.il, c.jl, c.kl, i, j, k, sh, fac)) return;
  const long long q = t;
  TF wv[5];
  for (int v = 0; v < 5; v++) wv[v] = f.w[v * f.N + q];
  if (f.blank[q] != 0) {
    for (int v = 0; v < 5; v++) {
      double acc = 0.0;
      int nn = 0;
      for (int dk = 0; dk < 2; dk++)
        for (int dj = 0; dj < 2; dj++)
          for (int di = 0; di < 2; di++)
            acc = acc + (double)c.w[v * c.N + cidx(c.Pi, c.Pj, sh[0] + di, sh[1] + dj, sh[2] + dk)] * fac[nn++];
      wv[v] = (TF)acc;
      f.w[v * f.N + q] = wv[v];
    }
  }
  f.p[q] = depvars((TF)gamma, wv);
}
template <typename TF, typename TC>
__global__ void k_embed(DevBlock<TF> f, DevBlock<TC> c, Xfer X, double gamma) {
  body_embed(f, c, X, gamma, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// upload_solut.f90:203-237: the cell-centre output variables of the physical
// cells, solut(2:il,2:jl,2:kl,1:nval) in Fortran order (nval 7, or 11 with
// the NS energy and three zero gradients); the expressions in the
// reference's order, in FP64 whatever the block's storage
template <typename T>
__global__ void k_solut(DevBlock<T> b, double gamma, double p0, double rm, double p_tot, int ns, double* out) {
  const long long ncell = (long long)b.nx * b.ny * b.nz;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= ncell) return;
  int i, j, k;
  cell_of(t, b.nx, b.ny, 2, i, j, k);
  const long long N = b.N, c = cidx(b.Pi, b.Pj, i, j, k);
  const double rr = (double)b.w[c];
  const double uu = (double)b.w[N + c] / rr;
  const double vv = (double)b.w[2 * N + c] / rr;
  const double ww = (double)b.w[3 * N + c] / rr;
  const double re = (double)b.w[4 * N + c];
  const double qq = 0.5 * (uu * uu + vv * vv + ww * ww) * rr;
  double pp = (gamma - 1.0) * (re > qq ? re - qq : 0.0);  // dim(re, qq)
  const double mm = sqrt((uu * uu + vv * vv + ww * ww) / gamma / pp * rr);
  const double ptloss = pp * pow(1.0 + 0.2 * mm * mm, 3.5) / p_tot - 1.0;
  pp = (pp / p0 - 1.0) * 2.0 / (gamma * rm * rm);
  out[t] = rr;
  out[ncell + t] = uu;
  out[2 * ncell + t] = vv;
  out[3 * ncell + t] = ww;
  out[4 * ncell + t] = pp;
  out[5 * ncell + t] = mm;
  out[6 * ncell + t] = ptloss;
  if (ns) {
    out[7 * ncell + t] = re / rr;
    out[8 * ncell + t] = 0.0;
    out[9 * ncell + t] = 0.0;
    out[10 * ncell + t] = 0.0;
  }
}

// wall forces from the records (new): 7 sums, fixed order within one block.
// Pressure on each wall face and, when mu > 0 (NS), the wall's viscous
// stress: the momentum the solver's wall flux (rec_wall_terms) gives the
// fluid, with the opposite sign
template <typename T>
__global__ void k_forces(DevBlock<T> b, double ox, double oy, double oz, double hx, double hy, double hz, double cx,
                         double cy, double cz, double mu, double* out) {
  __shared__ double sh[7][256];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};
  const double org[3] = {ox, oy, oz}, h[3] = {hx, hy, hz}, ctr[3] = {cx, cy, cz};
  for (int m = threadIdx.x; m < b.nmir; m += blockDim.x) {
    const int* ri = b.rec_i + 8 * m;
    if (ri[6] == 0) continue;  // a wall face another block of the level counts
    int ax = ri[4] - 1;
    double sgn = ri[3] >= 4 ? 1.0 : -1.0;
    long long c = cidx(b.Pi, b.Pj, ri[0], ri[1], ri[2]);
    double area = b.rec_area[m];
    double pw = 0.5 * ((double)b.p[c] + (double)b.rec_psol[m]);
    double fv[3] = {0, 0, 0};
    if (mu > 0.0) {  // visc_wall of rec_wall_terms, in FP64
      const bool plus = ri[3] >= 4;
      const double S = fabs(b.s[ax]), r0 = (double)b.w[c];
      for (int a = 0; a < 3; a++) {
        const double u = (double)b.w[(1 + a) * b.N + c] / r0;
        const double ug = 2.0 * b.rec_qb[3 * m + a] - u;
        const double gn = plus ? (ug - u) / h[ax] : (u - ug) / h[ax];
        const double tau = (a == ax) ? (4.0 / 3.0) * mu * gn : mu * gn;
        fv[a] = plus ? -(S * tau) : S * tau;
      }
    }
    double f[3];
    for (int d = 0; d < 3; d++) f[d] = (d == ax ? pw * area * sgn : 0.0) + fv[d];
    double xf[3];
    for (int d = 0; d < 3; d++) xf[d] = org[d] + ((double)ri[d] - 1.5) * h[d];
    xf[ax] = xf[ax] + sgn * 0.5 * h[ax];
    double r[3] = {xf[0] - ctr[0], xf[1] - ctr[1], xf[2] - ctr[2]};
    acc[0] += f[0];
    acc[1] += f[1];
    acc[2] += f[2];
    acc[3] += r[1] * f[2] - r[2] * f[1];
    acc[4] += r[2] * f[0] - r[0] * f[2];
    acc[5] += r[0] * f[1] - r[1] * f[0];
  }
  for (int q = 0; q < 6; q++) sh[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s)
      for (int q = 0; q < 6; q++) sh[q][threadIdx.x] += sh[q][threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x < 6) out[threadIdx.x] = sh[threadIdx.x][0];
}

// =============================================================== one-launch-per-phase kernels
template <typename T, bool FAST, bool S>
__global__ void __launch_bounds__(256, S ? 6 : 4) k_prep(DevBlock<T> b, PhysParams P, int dissip_on) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)b.ie * b.je * b.ke) body_prep<T, FAST, S>(b, P, dissip_on, t);
}
// The MUSCL Roe form's prep pass, in two.  First the velocities of every cell,
// ghosts included, into F[0..2] (one reciprocal of the density and mdiv: the
// IEEE quotients); with NS also the velocities and temperature of the viscous
// faces, zero in solid cells (euler.f90:140-154).
template <typename T, bool S>
__global__ void k_prim(DevBlock<T> b, PhysParams P, int dissip_on) {
  long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= b.N) return;
  const long long N = b.N;
  const T r = b.w[c], y = pdiv<S>(T(1), r);
  const bool visc = P.eqn_ns && dissip_on, solid = visc && b.blank[c] == 0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const T u = pmdiv<S>(b.w[(long long)(1 + a) * N + c], r, y);
    b.F[(long long)a * N + c] = u;
    if (visc) b.vt[a * N + c] = solid ? T(0) : u;
  }
  if (visc) b.vt[3 * N + c] = solid ? T(0) : pdiv<S>(b.p[c], pmul<S>(r, (T)P.gas_const));
}
// Then the limited slope of each primitive variable along each direction,
// once per cell, into dlt[dir][var].  A face takes the slope of its lower cell
// for the left state and that of its upper cell for the right state, the same
// van_albada(q(c)-q(c-1), q(c+1)-q(c)) it would form itself.  One direction per
// grid row, at the cells a face along it reads (tangential indices physical).
// The whole-cell pass took 350-530 us at 512x512x2 (the less, the more of the level
// is uniform), the two take 280-420.
template <typename T, bool S, int D>
__device__ __forceinline__ void body_slopes(const DevBlock<T>& b, const PhysParams& P, int t) {
  const int n0 = b.nx + (D == 0 ? 2 : 0), n1 = b.ny + (D == 1 ? 2 : 0), n2 = b.nz + (D == 2 ? 2 : 0);
  if (t >= n0 * n1 * n2) return;
  int i, j, k;
  cell_of(t, n0, n1, 2, i, j, k);
  if (D == 0) i -= 1;
  if (D == 1) j -= 1;
  if (D == 2) k -= 1;
  const long long N = b.N, st = D == 0 ? 1 : (D == 1 ? (long long)b.Pi : (long long)b.Pi * b.Pj);
  const long long c = cidx(b.Pi, b.Pj, i, j, k);
  const T* prim[5] = {b.w, b.F, b.F + N, b.F + 2 * N, b.p};
#pragma unroll
  for (int v = 0; v < 5; v++) {
    const T q0 = prim[v][c], dm = q0 - prim[v][c - st], dp = prim[v][c + st] - q0;
    b.dlt[(long long)(D * 5 + v) * N + c] = van_albada<S>(dm, dp, (T)P.lim_e2[v]);
  }
}
template <typename T, bool S>
__global__ void __launch_bounds__(256) k_slopes(DevBlock<T> b, PhysParams P) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.y == 0) body_slopes<T, S, 0>(b, P, t);
  else if (blockIdx.y == 1) body_slopes<T, S, 1>(b, P, t);
  else body_slopes<T, S, 2>(b, P, t);
}
template <typename T>
__global__ void __launch_bounds__(256, 4)
    k_face(const __grid_constant__ DevBlock<T> b, const __grid_constant__ PhysParams P, int dissip_on, T cd) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)(b.ie - 1) * (b.je - 1) * (b.ke - 1)) body_face<T, FACE_CENTRAL>(b, P, dissip_on, cd, t);
}
template <typename T, bool S>
__global__ void __launch_bounds__(256, S ? 6 : 4) k_face_jst(DevBlock<T> b, PhysParams P, int dissip_on, T cd) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)(b.ie - 1) * (b.je - 1) * (b.ke - 1)) body_face<T, FACE_JST, S>(b, P, dissip_on, cd, t);
}
// the prep and face passes of a small level, one direction per grid row
template <typename T, bool FAST, bool S>
__global__ void __launch_bounds__(256) k_prep_split(DevBlock<T> b, PhysParams P, int dissip_on) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.y == 0) body_prep_dir<T, FAST, S, 0>(b, P, dissip_on, t);
  else if (blockIdx.y == 1) body_prep_dir<T, FAST, S, 1>(b, P, dissip_on, t);
  else body_prep_dir<T, FAST, S, 2>(b, P, dissip_on, t);
}
template <typename T, bool FAST, bool S>
__global__ void __launch_bounds__(256) k_face_split(DevBlock<T> b, PhysParams P, int dissip_on, T cd) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.y == 0) body_face_split<T, FAST, S, 0>(b, P, dissip_on, cd, t);
  else if (blockIdx.y == 1) body_face_split<T, FAST, S, 1>(b, P, dissip_on, cd, t);
  else body_face_split<T, FAST, S, 2>(b, P, dissip_on, cd, t);
}
// The Roe faces (MUSCL states, upwind flux, and the viscous flux with NS), one
// direction per grid row.  Bound by the FP64 pipe and the latency of its chains
// at three blocks an SM.  With the products on the integer pipes (1,300 -> 1,070
// us a dissipative launch at 512x512x2), a direction a thread (1,058), and the states
// and fluxes inlined instead of passed through local memory (980); two blocks
// an SM 1,147, four 1,048.  DISS: a stage without dissipation has its own
// instance, 379 -> 255 us at four blocks an SM.
template <typename T, bool S, bool DISS>
__global__ void __launch_bounds__(256, DISS ? 3 : 4)
    k_face_roe(const __grid_constant__ DevBlock<T> b, const __grid_constant__ PhysParams P, T cd) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (blockIdx.y == 0) body_face_split<T, false, S, 0, FACE_ROE>(b, P, DISS, cd, t);
  else if (blockIdx.y == 1) body_face_split<T, false, S, 1, FACE_ROE>(b, P, DISS, cd, t);
  else body_face_split<T, false, S, 2, FACE_ROE>(b, P, DISS, cd, t);
}
// a stage without dissipation of the central scheme: only the convective
// face fluxes efs(q) = 0.5*(F(q) + F(q-1)), the same expression as face_dir,
// in a kernel small enough to keep the memory system busy
template <typename T>
__device__ __forceinline__ void body_face_conv(const DevBlock<T>& b, long long t) {
  const int ex = b.ie - 1, ey = b.je - 1;
  if (t >= (long long)ex * ey * (b.ke - 1)) return;
  int i, j, k;
  cell_of(t, ex, ey, 2, i, j, k);
  const long long N = b.N, c = cidx(b.Pi, b.Pj, i, j, k);
  const bool on[3] = {j <= b.jl && k <= b.kl, i <= b.il && k <= b.kl, i <= b.il && j <= b.jl};
  const long long sts[3] = {1, (long long)b.Pi, (long long)b.Pi * b.Pj};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (!on[d]) continue;
    const T* F = b.F + (long long)(d * 5) * N;
    T* E = b.efs + (long long)(d * 5) * N;
#pragma unroll
    for (int v = 0; v < 5; v++) E[v * N + c] = mulhalf(F[v * N + c] + F[v * N + c - sts[d]]);
  }
}
template <typename T>
__global__ void __launch_bounds__(256) k_face_conv(DevBlock<T> b) {
  body_face_conv(b, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
template <typename T, bool FAST, bool S>
__global__ void k_combine(DevBlock<T> b, PhysParams P, StageArgs A, unsigned* err) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)b.nx * b.ny * b.nz) body_combine<T, FAST, S>(b, P, A, err, t);
}
template <typename T, typename TC, int D, bool SC, bool QK, int K, bool PAIR>
__global__ void k_irs(DevBlock<T> b, IrsTables tb, TC bb) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < 5 * irs_lines<T, D>(b)) body_irs<T, TC, D, SC, QK, K, PAIR>(b, tb, bb, t);
}
template <typename T, bool S>
__global__ void k_update(DevBlock<T> b, PhysParams P, StageArgs A) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < (long long)b.nx * b.ny * b.nz) body_update<T, S>(b, P, A, t);
}
template <typename T>
__global__ void k_cutcell(DevBlock<T> b, PhysParams P, unsigned* err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < rec_lane_items(b)) cutcell_lanes(b, P, err, t);
}
// =============================================================== one euler update in one launch
// For the small coarse grids of the multigrid hierarchy every phase of
// euler.f90 is latency-bound, so one cooperative kernel runs them all with a
// grid-wide barrier between phases instead of ~70 launches.
struct EulerArgs {
  int mstage;
  int do_timestep;   // timestep.f90 before euler (solver.f90:154,218)
  int lfir, lres, rt;
  int smoo_on;
  StageArgs st[8];
  IrsTables tab[3];
  double* rt_partial;
  int npart;
  double* rt_out;
  unsigned* err;
  unsigned long long* trace;  // optional: globaltimer after every barrier (block 0, thread 0)
};

__device__ __forceinline__ unsigned long long gtimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <typename T, typename TA>
__global__ void __launch_bounds__(256, 1) k_euler_coop(DevBlock<T> b, PhysParams P, EulerArgs E) {
  cg::grid_group g_ = cg::this_grid();
  int ntr = 0;
  struct Sync {
    cg::grid_group& g;
    unsigned long long* tr;
    int& n;
    __device__ void sync() {
      g.sync();
      if (tr && blockIdx.x == 0 && threadIdx.x == 0 && n < 255) tr[1 + n++] = gtimer();
    }
  } g{g_, E.trace, ntr};
  if (E.trace && blockIdx.x == 0 && threadIdx.x == 0) E.trace[0] = gtimer();
  // items go round-robin over the blocks (item q to block q mod G), so that
  // the few cells of a small level still spread over every SM's FP64 pipe
  const long long gt = (long long)threadIdx.x * gridDim.x + blockIdx.x;
  const long long gs = (long long)gridDim.x * blockDim.x;
  const long long ncell = (long long)b.nx * b.ny * b.nz;
  if (E.do_timestep) {
    const int nb = (int)((ncell + blockDim.x - 1) / blockDim.x);
    for (long long base = (long long)blockIdx.x * blockDim.x; base < ncell; base += gs) {
      long long t = base + threadIdx.x;
      unsigned long long mine = ~0ull;
      if (t < ncell) mine = body_timestep<T, TA, false, true>(b, P, E.err, t);
      block_min_dtim(mine, b.dtim, nb);
    }
    g.sync();
  }
  if (E.lfir)
    for (long long q = gt; q < 5 * b.N; q += gs) b.ws[q] = b.w[q];
  if (!E.do_timestep)
    for (long long q = gt; q < b.N; q += gs) body_copy_wn(b, q);
  g.sync();
  const long long nprep = (long long)b.ie * b.je * b.ke;
  const long long nface = (long long)(b.ie - 1) * (b.je - 1) * (b.ke - 1);
  for (int m = 1; m <= E.mstage; m++) {
    const StageArgs& A = E.st[m - 1];
    if (A.fast) {
      for (long long t = gt; t < nprep; t += gs) body_prep<T, true, false>(b, P, A.dissip_on, t);
      g.sync();
      if (A.dissip_on)
        for (long long t = gt; t < 3 * split_row(b, 1); t += gs)
          body_face_rows<T, true, false>(b, P, 1, (T)A.cd, t);
    } else {
      for (long long t = gt; t < nprep; t += gs) body_prep<T, false, false>(b, P, A.dissip_on, t);
      g.sync();
      for (long long t = gt; t < nface; t += gs) body_face<T, FACE_ANY, false>(b, P, A.dissip_on, (T)A.cd, t);
    }
    if (split_scheme(P)) {
      const long long lt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
      for (long long t = lt; t < rec_lane_items(b); t += gs) rec_wall_lanes(b, P, A.dissip_on, (T)A.cd, E.err, (int)t);
    } else {
      for (long long t = gt; t < b.nmir; t += gs) rec_wall_terms(b, P, A.dissip_on, (T)A.cd, E.err, (int)t);
    }
    g.sync();
    if (A.fast)
      for (long long t = gt; t < ncell; t += gs) body_combine<T, true, false>(b, P, A, E.err, t);
    else
      for (long long t = gt; t < ncell; t += gs) body_combine<T, false, false>(b, P, A, E.err, t);
    g.sync();
    if (E.lres) return;
    if (A.irs && P.irs_kind == 1) {
      for (long long t = gt; t < irs_lines<T, 0>(b); t += gs) body_psmoo_line<T, TA, 0>(b, t);
      g.sync();
      for (long long t = gt; t < irs_lines<T, 1>(b); t += gs) body_psmoo_line<T, TA, 1>(b, t);
      g.sync();
      for (long long t = gt; t < irs_lines<T, 2>(b); t += gs) body_psmoo_line<T, TA, 2>(b, t);
      g.sync();
    } else if (A.irs) {
      const TA bb = (TA)(-P.smoo);
      for (long long t = gt; t < 5 * irs_lines<T, 0>(b); t += gs) body_irs<T, TA, 0>(b, E.tab[0], bb, t);
      g.sync();
      for (long long t = gt; t < 5 * irs_lines<T, 1>(b); t += gs) body_irs<T, TA, 1>(b, E.tab[1], bb, t);
      g.sync();
      for (long long t = gt; t < 5 * irs_lines<T, 2>(b); t += gs) body_irs<T, TA, 2>(b, E.tab[2], bb, t);
      g.sync();
    }
    if (A.irs) {
      for (long long t = gt; t < ncell; t += gs) body_update<T, false>(b, P, A, t);
      g.sync();
    }
    // whole warps of consecutive items: the corner cells and records share lanes
    const long long lt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (!b.cut_beside && b.nmir > 0) {
      for (long long t = lt; t < rec_lane_items(b); t += gs) cutcell_lanes(b, P, E.err, (int)t);
      g.sync();
    }
    for (long long t = lt; t < bc_n1(b) + rec_lane_items(b); t += gs) body_bcond<T, 0>(b, P, E.err, 1, t);
    g.sync();
    if (m < E.mstage && A.faces_only) continue;
    for (long long t = lt; t < bc_n2(b) + (bc_whole(b) ? bc_n3(b) : 0); t += gs) body_bcond<T, 1>(b, P, E.err, 0, t);
    g.sync();
    if (!bc_whole(b)) {
      for (long long t = lt; t < bc_n3(b); t += gs) body_bcond<T, 2>(b, P, E.err, 0, t);
      g.sync();
    }
  }
  if (E.rt) {
    for (int part = blockIdx.x; part < E.npart; part += gridDim.x)
      body_rtrms_partial(b, P, E.rt_partial, E.npart, part);
    g.sync();
    if (blockIdx.x == 0 && threadIdx.x < 32) body_rtrms_final(E.rt_partial, E.npart, (double)ncell, E.rt_out, E.err);
  }
  if (E.trace && blockIdx.x == 0 && threadIdx.x == 0) E.trace[255] = (unsigned long long)ntr;
}

// =============================================================== several cases in one launch
// The same phase of a group of cases in one launch: the cases' work items
// laid end to end, each case's range rounded up to whole 256-thread blocks,
// so that a thread block serves one case (the per-block reductions of the
// time step minimum and the residual partial sums stay within a case).
// Each case runs the same bodies in the same order as alone, so its results
// are those of its own launches.
template <typename T>
struct MultiArgs {
  const DevBlock<T>* B;
  const PhysParams* P;
  unsigned* const* err;
  const IrsTables* tab;
  double* const* rt_partial;
  const int* npart;
  double* const* rt_out;
  const long long* off;
  int nc;
};

__device__ __forceinline__ int multi_case(const long long* off, int nc, long long base) {
  __shared__ int sq;
  if (threadIdx.x == 0) {
    int q = 0;
    while (q + 1 < nc && off[q + 1] <= base) q++;
    sq = q;
  }
  __syncthreads();
  return sq;
}

// Blocks of 256 threads an SM is asked to hold for a phase (registers are cut to
// fit), as the phase's own kernel has it
template <typename F> struct MinBlocks { static constexpr int v = 4; };
// A thread block's case is copied to shared memory first: read from the group's
// array in global memory, every field would be loaded again after each store
// that might have changed it.
template <typename T, typename F>
__global__ void __launch_bounds__(256, MinBlocks<F>::v) k_multi(MultiArgs<T> M, F f) {
  __shared__ DevBlock<T> sb;
  __shared__ PhysParams sp;
  static_assert(sizeof(DevBlock<T>) % 4 == 0 && sizeof(PhysParams) % 4 == 0, "copied by words");
  const long long base = (long long)blockIdx.x * 256;
  const int q = multi_case(M.off, M.nc, base);
  for (int w = threadIdx.x; w < (int)(sizeof(DevBlock<T>) / 4); w += 256) ((int*)&sb)[w] = ((const int*)(M.B + q))[w];
  for (int w = threadIdx.x; w < (int)(sizeof(PhysParams) / 4); w += 256) ((int*)&sp)[w] = ((const int*)(M.P + q))[w];
  __syncthreads();
  f(M, q, base - M.off[q] + threadIdx.x, sb, sp);
}

template <typename T, typename TC, bool S> struct FTimestep {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    unsigned long long mine = ~0ull;
    const long long n = (long long)b.nx * b.ny * b.nz;
    if (t < n) mine = body_timestep<T, TC, S, true>(b, P, M.err[q], t);
    block_min_dtim(mine, b.dtim, (int)((n + 255) / 256));  // a call per 256 cells, whichever block makes it
  }
};
template <typename T> struct FCopyWs {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < 5 * b.N) b.ws[t] = b.w[t];
  }
};
template <typename T, bool FAST, bool S> struct FPrep {
  int dissip_on;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < (long long)b.ie * b.je * b.ke) body_prep<T, FAST, S>(b, P, dissip_on, t);
  }
};
template <typename T, bool S> struct FFace {
  int dissip_on;
  T cd;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < (long long)(b.ie - 1) * (b.je - 1) * (b.ke - 1)) body_face<T, FACE_CENTRAL, S>(b, P, dissip_on, cd, t);
  }
};
template <typename T> struct FFaceConv {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const { body_face_conv(b, t); }
};
template <typename T, bool FAST, bool S> struct FPrepRows {
  int dissip_on;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    body_prep_rows<T, FAST, S>(b, P, dissip_on, t);
  }
};
template <typename T, bool FAST, bool S> struct FFaceRows {
  int dissip_on;
  T cd;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    body_face_rows<T, FAST, S>(b, P, dissip_on, cd, t);
  }
};
template <typename T> struct FRec {
  int dissip_on;
  T cd;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (split_scheme(P)) {
      if (t < rec_lane_items(b)) rec_wall_lanes(b, P, dissip_on, cd, M.err[q], (int)t);
    } else if (t < b.nmir) {
      rec_wall_terms(b, P, dissip_on, cd, M.err[q], (int)t);
    }
  }
};
template <typename T, bool FAST, bool S> struct FCombine {
  StageArgs A;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < (long long)b.nx * b.ny * b.nz) body_combine<T, FAST, S>(b, P, A, M.err[q], t);
  }
};
template <typename T, typename TC, int D> struct FIrs {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t >= 5 * irs_lines<T, D>(b)) return;
    if constexpr (std::is_same<TC, double>::value) {
      if (M.tab[3 * q + D].quick) {
        body_irs<T, TC, D, false, true>(b, M.tab[3 * q + D], (TC)(-P.smoo), t);
        return;
      }
    }
    body_irs<T, TC, D>(b, M.tab[3 * q + D], (TC)(-P.smoo), t);
  }
};
// the mixed form's finest level: FP32 sweeps on one FP32 copy of dw (in F)
template <typename TS, typename TO, int D> struct FIrsMixed {
  __device__ void operator()(const MultiArgs<double>& M, int q, long long t, const DevBlock<double>& b,
                             const PhysParams& P) const {
    if (t >= 5 * irs_lines<double, D>(b)) return;
    float* cp = (float*)b.F;
    const TS* src = D == 0 ? (const TS*)b.dw : (const TS*)cp;
    TO* out = D == 2 ? (TO*)b.dw : (TO*)cp;
    body_irs_mixed<TS, TO, D>(b, M.tab[3 * q + D], (float)(-P.smoo), src, cp, out, t);
  }
};
template <typename T, bool S> struct FUpdate {
  StageArgs A;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < (long long)b.nx * b.ny * b.nz) body_update<T, S>(b, P, A, t);
  }
};
template <typename T> struct FCutcell {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    // the blocks whose records do not share the boundary launch
    if (!b.cut_beside && t < rec_lane_items(b)) cutcell_lanes(b, P, M.err[q], (int)t);
  }
};
template <typename T, int PART> struct FBcond {
  int cut;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    body_bcond<T, PART>(b, P, M.err[q], cut, t);
  }
};
template <typename T> struct FDepvars {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const { body_depvars(b, P.gamma, t); }
};
template <typename T> struct FDepvarsWn {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    body_depvars_wn(b, P.gamma, t);
  }
};
template <typename T> struct FCopyWn {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const { body_copy_wn(b, t); }
};
// residual partial sums: thread block (case, part), 256 threads each
template <typename T> struct FRtrmsPartial {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    const int part = (int)(t / 256);
    if (part < M.npart[q]) body_rtrms_partial(b, P, M.rt_partial[q], M.npart[q], part);
  }
};
template <typename T> struct FRtrmsFinal {
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>& b,
                             const PhysParams& P) const {
    if (t < 32) body_rtrms_final(M.rt_partial[q], M.npart[q], (double)b.nx * b.ny * b.nz, M.rt_out[q], M.err[q]);
  }
};

// the transfers between the levels of a group: child f and parent c of each case
template <typename TC, typename TF>
struct MultiPairArgs {
  const DevBlock<TC>* C;
  const DevBlock<TF>* F;
  const Xfer* X;
  uint8_t* const* marker;
  double* const* dc;
  const PhysParams* P;
  const long long* off;
  int nc;
};
template <typename TC, typename TF, typename Fn>
__global__ void __launch_bounds__(256) k_multi2(MultiPairArgs<TC, TF> M, Fn f) {
  const long long base = (long long)blockIdx.x * 256;
  const int q = multi_case(M.off, M.nc, base);
  f(M, q, base - M.off[q] + threadIdx.x);
}
template <typename TC, typename TF> struct FCollc {
  __device__ void operator()(const MultiPairArgs<TC, TF>& M, int q, long long t) const {
    body_collc(M.C[q], M.F[q], M.X[q], M.marker[q], t);
  }
};
template <typename TC, typename TF> struct FAddwDiff {
  __device__ void operator()(const MultiPairArgs<TC, TF>& M, int q, long long t) const {
    body_addw_diff(M.C[q], (typename Correction<TF, TC>::type*)M.dc[q], t);
  }
};
template <typename TC, typename TF> struct FAddw {
  int fmg;
  __device__ void operator()(const MultiPairArgs<TC, TF>& M, int q, long long t) const {
    const DevBlock<TF>& f = M.F[q];
    if (t >= (long long)f.nx * f.ny * f.nz) return;
    int i, j, k;
    cell_of(t, f.nx, f.ny, 2, i, j, k);
    body_addw(f, M.C[q], M.X[q], fmg, (const typename Correction<TF, TC>::type*)M.dc[q], i, j, k);
  }
};
template <typename TC, typename TF> struct FEmbed {
  __device__ void operator()(const MultiPairArgs<TC, TF>& M, int q, long long t) const {
    body_embed(M.F[q], M.C[q], M.X[q], M.P[q].gamma, t);
  }
};

// measured on eight mixed cases of 32^3 to 96^3: the contracted combine 345 us at 4,
// 336 at 5; the prep 270, 257; the dissipation faces 373 at 1 to 5, 337 at 6; the FP32
// faces 60, 44; the i sweep 223, 207 at 1
template <bool S> struct MinBlocks<FCombine<double, true, S>> { static constexpr int v = 5; };
template <bool S> struct MinBlocks<FPrep<double, true, S>> { static constexpr int v = 5; };
template <bool S> struct MinBlocks<FFaceRows<double, true, S>> { static constexpr int v = 6; };
template <bool S> struct MinBlocks<FFace<float, S>> { static constexpr int v = 5; };
template <> struct MinBlocks<FIrsMixed<double, float, 0>> { static constexpr int v = 1; };
template <typename T, typename TC, bool S> struct MinBlocks<FTimestep<T, TC, S>> { static constexpr int v = 6; };
// the plain forms as in their own kernels
template <> struct MinBlocks<FPrep<double, false, true>> { static constexpr int v = 6; };
template <typename T, int D> struct MinBlocks<FIrs<T, T, D>> { static constexpr int v = 3; };

// =============================================================== launchers
constexpr int TPB = 256;

// Threads per block for n work items: 256, halved down to 32 while the grid
// would not give every SM two blocks.  The stage kernels are bound by the FP64
// pipe of the SMs they run on, so on the small coarse levels spreading the
// cells over all SMs is worth more than wide blocks.
inline int tpb_for(long long n) {
  static int nsm = 0;
  if (!nsm) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0) nsm = 152;
  }
  int t = TPB;
  while (t > 32 && n < (long long)t * nsm * 2) t >>= 1;
  return t;
}
#define LAUNCH_N(n) nblk((n), tpb_for(n)), tpb_for(n)

// FP64 blocks of up to this many cells run plain FP64 operations instead of
// the integer-pipe forms (pmul).  Measured, plain against integer: a W-cycle's
// 24^3 update 269 against 281 us, a 64x64x2 one 402 against 421; a 48^3 level's
// cycle 1.18 against 1.09 ms, a 192^3 one 50 against 40.  The line is the central
// scheme's.  An update of the upwind schemes crosses over earlier, first-order Roe
// and MUSCL with NS, ms: 64x64x2 0.345 against 0.403 and 0.511 against 0.574, 24^3 0.320
// against 0.355 and 0.501 against 0.527, 128x64x2 0.457 against 0.465 and 0.714 against
// 0.660, 128x128x2 0.616 against 0.585 and 0.993 against 0.828.
constexpr long long kPlainCells = 32768;
template <typename T> bool on_int_pipes(const DevBlock<T>& b) {
  return (long long)b.nx * b.ny * b.nz > kPlainCells;
}
// f(std::true_type) with the integer-pipe forms, f(std::false_type) without; FP32 has one form
template <typename T, typename F> void with_form(const DevBlock<T>& b, F&& f) {
  if constexpr (std::is_same<T, double>::value) {
    if (!on_int_pipes(b)) return f(std::false_type{});
  }
  f(std::true_type{});
}

// Passes with one thread per cell and direction (body_prep_dir,
// body_face_split).  A level that leaves schedulers without a warp gains from
// the shorter threads; a large one pays for the values read and formed three
// times.  Measured, split against whole, us: FP64 24^3 prep 9.8 against 11.8 and
// face 11 against 18; 48^3 21 against 27 and 22 against 27; 96^3 prep 112 against
// 120 but face 134 against 124; 192^3 face 962 against 897.  The contracted
// dissipation faces share nothing between the directions, and split they keep
// twice the warps resident: 414 against 563 us a launch at 192^3.
inline bool split_prep(bool fast, long long cells) { return cells <= (fast ? 300000 : 1000000); }
inline bool split_face(bool fast, long long cells) { return fast || cells <= 300000; }

template <typename T>
void launch_solut(const DevBlock<T>& b, const PhysParams& P, double rm, double p_tot, int ns, double* out,
                  cudaStream_t s) {
  const long long n = (long long)b.nx * b.ny * b.nz;
  k_solut<T><<<nblk(n, TPB), TPB, 0, s>>>(b, P.gamma, P.p0, rm, p_tot, ns, out);
}


template <typename T>
void launch_timestep(const DevBlock<T>& b, const PhysParams& P, unsigned* err, cudaStream_t s, bool aux32, bool save) {
  long long n = (long long)b.nx * b.ny * b.nz;
  with_form(b, [&](auto S) {
    auto go = [&](auto tc, auto form) {
      using TC = decltype(tc);
      if (save)
        k_timestep<T, TC, form.value, true><<<LAUNCH_N(n), 0, s>>>(b, P, err);
      else
        k_timestep<T, TC, form.value, false><<<LAUNCH_N(n), 0, s>>>(b, P, err);
    };
    if (aux32)
      go(float(), std::true_type{});
    else
      go(T(), S);
  });
}

template <typename T>
void launch_stage_part(int part, const DevBlock<T>& b, const PhysParams& P, const StageArgs& A, unsigned* err,
                       cudaStream_t s) {
  const long long cells = (long long)b.nx * b.ny * b.nz;
  // the largest direction's items of a split pass (e = 2: prep, 1: faces), a row of the grid each
  auto rows = [&](int e) {
    const long long n = std::max({(long long)(b.nx + e) * b.ny * b.nz, (long long)b.nx * (b.ny + e) * b.nz,
                                  (long long)b.nx * b.ny * (b.nz + e)});
    return std::make_pair(dim3(nblk(n, tpb_for(3 * n)), 3), tpb_for(3 * n));
  };
  if (part == 0 && split_scheme(P) && split_prep(A.fast, cells)) {
    const auto g = rows(2);
    with_form(b, [&](auto S) {
      if (A.fast)
        k_prep_split<T, true, S.value><<<g.first, g.second, 0, s>>>(b, P, A.dissip_on);
      else
        k_prep_split<T, false, S.value><<<g.first, g.second, 0, s>>>(b, P, A.dissip_on);
    });
  } else if (part == 1 && split_scheme(P) && split_face(A.fast, cells)) {
    const auto g = rows(1);
    with_form(b, [&](auto S) {
      if (!A.fast)
        k_face_split<T, false, S.value><<<g.first, g.second, 0, s>>>(b, P, A.dissip_on, (T)A.cd);
      else if (A.dissip_on)
        k_face_split<T, true, S.value><<<g.first, g.second, 0, s>>>(b, P, 1, (T)A.cd);
    });
  } else if (part == 0) {
    long long n1 = (long long)b.ie * b.je * b.ke;
    if (P.distype == 2) {
      const auto g = rows(2);
      with_form(b, [&](auto S) {
        k_prim<T, S.value><<<LAUNCH_N(b.N), 0, s>>>(b, P, A.dissip_on);
        k_slopes<T, S.value><<<g.first, g.second, 0, s>>>(b, P);
      });
    } else {
      with_form(b, [&](auto S) {
        if (A.fast)
          k_prep<T, true, S.value><<<LAUNCH_N(n1), 0, s>>>(b, P, A.dissip_on);
        else
          k_prep<T, false, S.value><<<LAUNCH_N(n1), 0, s>>>(b, P, A.dissip_on);
      });
    }
  } else if (part == 1) {
    long long n2 = (long long)(b.ie - 1) * (b.je - 1) * (b.ke - 1);
    if (!A.dissip_on && P.distype == 0)
      k_face_conv<T><<<LAUNCH_N(n2), 0, s>>>(b);
    else if (P.distype == 0 && !P.eqn_ns && !P.matrix)
      with_form(b, [&](auto S) { k_face_jst<T, S.value><<<LAUNCH_N(n2), 0, s>>>(b, P, A.dissip_on, (T)A.cd); });
    else if (P.distype == 0)
      k_face<T><<<LAUNCH_N(n2), 0, s>>>(b, P, A.dissip_on, (T)A.cd);
    else
      with_form(b, [&](auto S) {
        const auto g = rows(1);
        if (A.dissip_on)
          k_face_roe<T, S.value, true><<<g.first, g.second, 0, s>>>(b, P, (T)A.cd);
        else
          k_face_roe<T, S.value, false><<<g.first, g.second, 0, s>>>(b, P, (T)A.cd);
      });
  } else if (part == 2) {
    if (b.nmir > 0 && split_scheme(P))
      k_rec_lanes<T><<<LAUNCH_N(rec_lane_items(b)), 0, s>>>(b, P, A.dissip_on, (T)A.cd, err);
    else if (b.nmir > 0)
      k_rec_wall<T><<<LAUNCH_N(b.nmir), 0, s>>>(b, P, A.dissip_on, (T)A.cd, err);
  } else if (part == 3) {
    long long n3 = (long long)b.nx * b.ny * b.nz;
    with_form(b, [&](auto S) {
      if (A.fast)
        k_combine<T, true, S.value><<<LAUNCH_N(n3), 0, s>>>(b, P, A, err);
      else
        k_combine<T, false, S.value><<<LAUNCH_N(n3), 0, s>>>(b, P, A, err);
    });
  }
}

// One stage.  With a side stream and two events, the record pass runs on the
// side stream beside the prep and face passes (it needs only the state); the
// combine pass waits for both.
template <typename T>
void launch_stage(const DevBlock<T>& b, const PhysParams& P, const StageArgs& A, unsigned* err, cudaStream_t s,
                  cudaStream_t side, cudaEvent_t fork, cudaEvent_t join) {
  const bool beside = b.nmir > 0 && side && fork && join;
  if (beside) {
    cudaEventRecord(fork, s);
    cudaStreamWaitEvent(side, fork, 0);
    launch_stage_part<T>(2, b, P, A, err, side);
    cudaEventRecord(join, side);
  }
  launch_stage_part<T>(0, b, P, A, err, s);
  launch_stage_part<T>(1, b, P, A, err, s);
  if (beside)
    cudaStreamWaitEvent(s, join, 0);
  else
    launch_stage_part<T>(2, b, P, A, err, s);
  launch_stage_part<T>(3, b, P, A, err, s);
}

// the line-sweep variant: 0 = one thread per (line, variable) in global
// memory, 1 = shared-memory tiles of 64 lines; the autotuner picks per block
// and direction
template <typename T, typename TC, int D>
void launch_irs_dir(const DevBlock<T>& b, const IrsTables& tb, TC bb, cudaStream_t s, int variant) {
  const long long lines = D == 0 ? (long long)b.ny * b.nz : (D == 1 ? (long long)b.nx * b.nz : (long long)b.nx * b.ny);
  const int len = (D == 0 ? b.il : (D == 1 ? b.jl : b.kl)) - 1;
  constexpr int LT = 64;
  const size_t sm = irs_smem_bytes<TC, LT>(len | 1);
  if constexpr (D == 0 && std::is_same<T, float>::value && std::is_same<TC, float>::value) {
    const int kk = irs_scan_k(len);
    if (variant == 2 && kk) {  // one warp per (line, variable), in place
      const unsigned g = (unsigned)nblk(32 * 5 * lines, 256);
      float* out = (float*)b.dw;
      if (kk == 2) k_irs_scan_i<2, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      if (kk == 4) k_irs_scan_i<4, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      if (kk == 6) k_irs_scan_i<6, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      if (kk == 8) k_irs_scan_i<8, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      if (kk == 12) k_irs_scan_i<12, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      if (kk == 16) k_irs_scan_i<16, float><<<g, 256, 0, s>>>(b, tb, bb, out);
      return;
    }
  }
  if (variant == 1 && sm <= 200 * 1024) {
    const long long grid = 5 * ((lines + LT - 1) / LT);
    k_irs_smem<T, TC, D, LT><<<(unsigned)grid, LT, sm, s>>>(b, tb, bb);
  } else {
    const auto many = [&](auto QK, auto PAIR) {
      constexpr bool qk = QK.value, pr = PAIR.value;
      if (5 * lines >= 150000)  // about 8 warps per scheduler: the sweep is bound by the FP64 rate
        k_irs<T, TC, D, true, qk, 8, pr><<<LAUNCH_N(5 * lines), 0, s>>>(b, tb, bb);
      else
        k_irs<T, TC, D, false, qk, 8, pr><<<LAUNCH_N(5 * lines), 0, s>>>(b, tb, bb);
    };
    const auto go = [&](auto QK) {
      if (5 * lines <= 8192) {
        // under half the schedulers have a warp: the memory latency a chunk pays shows, and
        // pairs only add the cells around them (24^3 12.7 against 14.6 us)
        k_irs<T, TC, D, false, QK.value, 24, false><<<LAUNCH_N(5 * lines), 0, s>>>(b, tb, bb);
        return;
      }
      if constexpr (D == 0 && std::is_same<T, double>::value && std::is_same<TC, double>::value) {
        if (irs_pairs(b)) return many(QK, std::true_type{});
      }
      many(QK, std::false_type{});
    };
    if constexpr (std::is_same<TC, double>::value) {
      if (tb.quick) return go(std::true_type{});
    }
    go(std::false_type{});
  }
}

template <typename T>
long long irs_lines_h(const DevBlock<T>& b, int D) {
  return D == 0 ? (long long)b.ny * b.nz : (D == 1 ? (long long)b.nx * b.nz : (long long)b.nx * b.ny);
}

template <typename T, typename TC>
void launch_irs_part_t(int part, const DevBlock<T>& b, const PhysParams& P, const IrsTables* tab, cudaStream_t s,
                       const int* variant, const StageArgs* A) {
  StageArgs Au;  // the update's stage (steady without one: lam = 1)
  memset(&Au, 0, sizeof(Au));
  if (A) Au = *A;
  const TC bb = (TC)(-P.smoo);
  const long long ncell = (long long)b.nx * b.ny * b.nz;
  if (P.irs_kind == 1) {  // psmoo + progon3: one thread per line
    if (part == 0) k_psmoo_line<T, TC, 0><<<LAUNCH_N(irs_lines_h(b, 0)), 0, s>>>(b);
    if (part == 1) k_psmoo_line<T, TC, 1><<<LAUNCH_N(irs_lines_h(b, 1)), 0, s>>>(b);
    if (part == 2) {
      k_psmoo_line<T, TC, 2><<<LAUNCH_N(irs_lines_h(b, 2)), 0, s>>>(b);
      with_form(b, [&](auto S) { k_update<T, S.value><<<LAUNCH_N(ncell), 0, s>>>(b, P, Au); });
    }
    return;
  }
  if constexpr (std::is_same<T, double>::value && std::is_same<TC, float>::value) {
    // FP32 sweeps on FP64 storage: one FP32 copy through the three sweeps
    float* cp = (float*)b.F;
    if (part == 0) {
      // the tuned form of the i sweep: global-memory lines or shared-memory tiles
      constexpr int LT = 64;
      const size_t sm = irs_smem_bytes<float, LT>((b.il - 1) | 1);
      const int kk = irs_scan_k(b.il - 1);
      const long long nthr = 32 * 5 * irs_lines_h(b, 0);
      if (variant && variant[0] == 2 && kk) {
        const unsigned g = (unsigned)nblk(nthr, 256);
        if (kk == 2) k_irs_scan_i<2><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
        if (kk == 4) k_irs_scan_i<4><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
        if (kk == 6) k_irs_scan_i<6><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
        if (kk == 8) k_irs_scan_i<8><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
        if (kk == 12) k_irs_scan_i<12><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
        if (kk == 16) k_irs_scan_i<16><<<g, 256, 0, s>>>(b, tab[0], bb, cp);
      } else if (variant && variant[0] == 1 && sm <= 200 * 1024)
        k_irs_smem_fill<LT><<<(unsigned)(5 * ((irs_lines_h(b, 0) + LT - 1) / LT)), LT, sm, s>>>(b, tab[0], bb, cp);
      else
        k_irs_mixed<double, float, 0><<<LAUNCH_N(5 * irs_lines_h(b, 0)), 0, s>>>(b, tab[0], bb, b.dw, cp, cp);
    }
    if (part == 1)
      k_irs_mixed<float, float, 1><<<LAUNCH_N(5 * irs_lines_h(b, 1)), 0, s>>>(b, tab[1], bb, cp, cp, cp);
    if (part == 2) {
      k_irs_mixed<float, double, 2><<<LAUNCH_N(5 * irs_lines_h(b, 2)), 0, s>>>(b, tab[2], bb, cp, cp, b.dw);
      with_form(b, [&](auto S) { k_update<T, S.value><<<LAUNCH_N(ncell), 0, s>>>(b, P, Au); });
    }
    return;
  }
  if (part == 0) launch_irs_dir<T, TC, 0>(b, tab[0], bb, s, variant ? variant[0] : 0);
  if (part == 1) launch_irs_dir<T, TC, 1>(b, tab[1], bb, s, variant ? variant[1] : 0);
  if (part == 2) {
    launch_irs_dir<T, TC, 2>(b, tab[2], bb, s, variant ? variant[2] : 0);
    with_form(b, [&](auto S) { k_update<T, S.value><<<LAUNCH_N(ncell), 0, s>>>(b, P, Au); });
  }
}

template <typename T>
void launch_irs_part(int part, const DevBlock<T>& b, const PhysParams& P, const IrsTables* tab, cudaStream_t s,
                     bool aux32, const int* variant, const StageArgs* A) {
  if (aux32)
    launch_irs_part_t<T, float>(part, b, P, tab, s, variant, A);
  else
    launch_irs_part_t<T, T>(part, b, P, tab, s, variant, A);
}

template <typename T>
void launch_irs(const DevBlock<T>& b, const PhysParams& P, const IrsTables* tab, cudaStream_t s, bool aux32,
                const int* variant, const StageArgs* A) {
  for (int part = 0; part < 3; part++) launch_irs_part<T>(part, b, P, tab, s, aux32, variant, A);
}

template <typename T>
void launch_cutcell(const DevBlock<T>& b, const PhysParams& P, unsigned* err, cudaStream_t s) {
  if (b.nmir > 0) k_cutcell<T><<<LAUNCH_N(rec_lane_items(b)), 0, s>>>(b, P, err);
}

template <typename T>
void launch_bcond(const DevBlock<T>& b, const PhysParams& P, cudaStream_t s, bool faces_only, unsigned* cut_err) {
  k_bcond<T, 0><<<LAUNCH_N(cut_err ? bc_items_t(b, 0) : bc_n1(b)), 0, s>>>(b, P, cut_err, cut_err != nullptr);
  if (faces_only) return;
  k_bcond<T, 1><<<LAUNCH_N(bc_items_t(b, 1)), 0, s>>>(b, P, nullptr, 0);
  const long long n = bc_items_t(b, 2);
  if (n > 0) k_bcond<T, 2><<<LAUNCH_N(n), 0, s>>>(b, P, nullptr, 0);
}

template <typename T>
long long bc_items(const DevBlock<T>& b, int part) {
  return bc_items_t(b, part);
}

template <typename T>
long long split_items(const DevBlock<T>& b, int e) {
  return split_items_t(b, e);
}
#if MGE_PART == 0
void split_passes(const PhysParams& P, bool fast, long long cells, bool* prep, bool* face) {
  *prep = split_scheme(P) && split_prep(fast, cells);
  *face = split_scheme(P) && split_face(fast, cells);
}
#endif

template <typename T>
void launch_rtrms(const DevBlock<T>& b, const PhysParams& P, double* partial, int npartial, double* out,
                  cudaStream_t s, unsigned* err) {
  k_rtrms_partial<T><<<npartial, RT_THREADS, 0, s>>>(b, P, partial, npartial);
  k_rtrms_final<<<1, 32, 0, s>>>(partial, npartial, (double)b.nx * b.ny * b.nz, out, err);
}

#if MGE_PART == 0
template <typename TS, typename TD>
__global__ void k_convert(const TS* __restrict__ a, TD* __restrict__ b, long long n) {
  long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) b[q] = (TD)a[q];
}

void launch_convert(const void* src, bool src32, void* dst, bool dst32, long long n, cudaStream_t s) {
  if (n <= 0) return;
  if (src32 && !dst32) k_convert<float, double><<<nblk(n, TPB), TPB, 0, s>>>((const float*)src, (double*)dst, n);
  else if (!src32 && dst32) k_convert<double, float><<<nblk(n, TPB), TPB, 0, s>>>((const double*)src, (float*)dst, n);
  else if (src32) k_convert<float, float><<<nblk(n, TPB), TPB, 0, s>>>((const float*)src, (float*)dst, n);
  else k_convert<double, double><<<nblk(n, TPB), TPB, 0, s>>>((const double*)src, (double*)dst, n);
}

// movsurf.f90:31 (pnew = psurf + disp) and the wall velocity of
// bc_cutcell.f90:50 (qb = vel/vel_fs), one thread per record component
__global__ void k_movsurf(long long n3, const double* psurf, double* pnew, double* qb, double vel_fs) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n3) return;
  pnew[t] = psurf[t] + pnew[t];
  qb[t] = qb[t] / vel_fs;
}

void launch_movsurf(long long nmir, const double* psurf, double* pnew, double* qb, double vel_fs, cudaStream_t s) {
  if (nmir <= 0) return;
  k_movsurf<<<nblk(3 * nmir, TPB), TPB, 0, s>>>(3 * nmir, psurf, pnew, qb, vel_fs);
}
#endif

// opt-in shared memory of the tiled line sweeps; called once per device at set-up
void init_kernel_attributes_f32();
#define MGE_SMEM_ATTR(T, TC)                                                                                     \
  cudaFuncSetAttribute(k_irs_smem<T, TC, 0, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);     \
  cudaFuncSetAttribute(k_irs_smem<T, TC, 1, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);     \
  cudaFuncSetAttribute(k_irs_smem<T, TC, 2, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
#if MGE_PART == 0
void init_kernel_attributes() {
  MGE_SMEM_ATTR(double, double)
  MGE_SMEM_ATTR(double, float)
  cudaFuncSetAttribute(k_irs_smem_fill<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  init_kernel_attributes_f32();
}
#elif MGE_PART == 1
void init_kernel_attributes_f32() { MGE_SMEM_ATTR(float, float) }
#endif
#undef MGE_SMEM_ATTR

// grid of the cooperative kernel: every block resident at once
template <typename T, typename TA>
int coop_grid(int device) {
  static int cached[64] = {0};
  if (device < 0 || device >= 64) return 0;
  if (cached[device]) return cached[device];
  int nsm = 0, per = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_euler_coop<T, TA>, 256, 0);
  int coop = 0;
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
  cached[device] = (coop && per > 0) ? nsm * per : -1;
  return cached[device];
}

template <typename T>
int launch_euler_coop(const DevBlock<T>& b, const PhysParams& P, const EulerLaunch& L, int device, cudaStream_t s,
                      bool aux32) {
  int grid = aux32 ? coop_grid<T, float>(device) : coop_grid<T, T>(device);
  if (grid <= 0) return -1;
  long long work = (long long)(b.ie) * b.je * b.ke;
  static int nsm = 0;
  if (!nsm && cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) nsm = 1;
  // at least one block per SM: the kernel deals items round-robin over the blocks
  int need = (int)std::min<long long>(std::max<long long>((work + 255) / 256, nsm), (long long)grid);
  if (L.max_ctas > 0 && need > L.max_ctas) need = L.max_ctas;
  if (need < 1) need = 1;
  EulerArgs E;
  memset(&E, 0, sizeof(E));
  E.mstage = L.mstage;
  E.do_timestep = L.do_timestep;
  E.lfir = L.lfir;
  E.lres = L.lres;
  E.rt = L.rt;
  for (int m = 0; m < L.mstage && m < 8; m++) E.st[m] = L.st[m];
  for (int d = 0; d < 3; d++) E.tab[d] = L.tab[d];
  E.rt_partial = L.rt_partial;
  E.npart = L.npart;
  E.rt_out = L.rt_out;
  E.err = L.err;
  E.trace = L.trace;
  DevBlock<T> bb = b;
  PhysParams pp = P;
  void* args[] = {&bb, &pp, &E};
  void* fn = aux32 ? (void*)k_euler_coop<T, float> : (void*)k_euler_coop<T, T>;
  cudaError_t e = cudaLaunchCooperativeKernel(fn, need, 256, args, 0, s);
  return e == cudaSuccess ? 0 : -2;
}

template <typename T>
void launch_depvars_all(const DevBlock<T>& b, const PhysParams& P, cudaStream_t s) {
  k_depvars_all<T><<<LAUNCH_N(b.N), 0, s>>>(b, P.gamma);
}

template <typename T>
void launch_copy_ws(const DevBlock<T>& b, cudaStream_t s) {
  k_copy5<T><<<nblk(5 * b.N, TPB), TPB, 0, s>>>(b.w, b.ws, 5 * b.N);
}

template <typename T>
void launch_depvars_wn(const DevBlock<T>& b, const PhysParams& P, cudaStream_t s) {
  k_depvars_wn<T><<<LAUNCH_N(b.N), 0, s>>>(b, P.gamma);
}

template <typename T>
void launch_copy_wn(const DevBlock<T>& b, cudaStream_t s) {
  k_copy_wn<T><<<nblk(b.N, TPB), TPB, 0, s>>>(b);
}

template <typename T>
void launch_init_free(const DevBlock<T>& b, const PhysParams& P, cudaStream_t s) {
  k_init_free<T><<<nblk(b.N, TPB), TPB, 0, s>>>(b, P);
}

// a transfer's ratio and offset; an exact reciprocal of a power-of-two ratio
inline Xfer make_xfer(const int ratio[3], const int offset[3]) {
  Xfer X;
  for (int d = 0; d < 3; d++) {
    X.r[d] = ratio[d];
    X.o[d] = offset[d];
    X.rinv[d] = (ratio[d] > 0 && (ratio[d] & (ratio[d] - 1)) == 0) ? 1.0 / (double)ratio[d] : 0.0;
  }
  return X;
}

template <typename TC, typename TF>
void launch_collc(const DevBlock<TC>& c, const DevBlock<TF>& f, const int ratio[3], const int offset[3],
                  uint8_t* marker_c, cudaStream_t s) {
  Xfer X = make_xfer(ratio, offset);
  long long n = (long long)(f.nx / ratio[0]) * (f.ny / ratio[1]) * (f.nz / ratio[2]);
  k_collc<TC, TF><<<LAUNCH_N(n), 0, s>>>(c, f, X, marker_c);
}

template <typename TF, typename TC>
void launch_addw(const DevBlock<TF>& f, const DevBlock<TC>& c, const int ratio[3], const int offset[3], int fmg,
                 double* scratch, cudaStream_t s) {
  Xfer X = make_xfer(ratio, offset);
  long long n = (long long)f.nx * f.ny * f.nz;
  // the coarse corrections go to the stage scratch (at least 64 fields of
  // the largest block), free between euler calls
  typedef typename Correction<TF, TC>::type TD;
  TD* dc = (TD*)scratch;
  if (!fmg) k_addw_diff<TC, TD><<<LAUNCH_N(c.N), 0, s>>>(c, dc);
  if constexpr (std::is_same<TD, double>::value) {
    // whole 2:1 coarsening, the fine block inside its parent: eight cells a
    // thread, from the size on at which the saved products outweigh the second
    // launch (a W-cycle with 192^3 finest 37.1 against 38.1 ms, 64^3 3.29 against 3.31; the
    // 48^3 level of a mixed hierarchy 0.46 against 0.45)
    bool octets = n > 200000;
    const int nf[3] = {f.nx, f.ny, f.nz}, nc[3] = {c.nx, c.ny, c.nz};
    for (int d = 0; d < 3; d++)
      octets = octets && X.r[d] == 2 && X.o[d] >= 0 && nf[d] >= 4 && nf[d] % 2 == 0 && X.o[d] + nf[d] / 2 <= nc[d];
    if (octets) {
      const long long no = (long long)(f.nx / 2 - 1) * (f.ny / 2 - 1) * (f.nz / 2 - 1);
      const int to = std::min(tpb_for(no), 128);
      k_addw_octet<TF, TC><<<nblk(no, to), to, 0, s>>>(f, c, X, fmg, dc);
      k_addw_shell<TF, TC><<<LAUNCH_N(shell_items(f)), 0, s>>>(f, c, X, fmg, dc);
      return;
    }
  }
  k_addw<TF, TC><<<LAUNCH_N(n), 0, s>>>(f, c, X, fmg, dc);
}

template <typename TF, typename TC>
void launch_embed(const DevBlock<TF>& f, const DevBlock<TC>& c, const int ratio[3], const int offset[3],
                  const PhysParams& P, cudaStream_t s) {
  Xfer X = make_xfer(ratio, offset);
  k_embed<TF, TC><<<LAUNCH_N(f.N), 0, s>>>(f, c, X, P.gamma);
}

template <typename T>
void launch_overlap(const DevBlock<T>& g, const DevBlock<T>& p, const long long* dst, const long long* src,
                    const double* fac, long long n, const PhysParams& P, cudaStream_t s) {
  if (n > 0) k_overlap<T><<<LAUNCH_N(n), 0, s>>>(g, p, dst, src, fac, n, P.gamma);
}

template <typename T>
void launch_forces(const DevBlock<T>& b, const double* origin, const double* h, const double* center, double mu,
                   double* out7, cudaStream_t s) {
  k_forces<T><<<1, 256, 0, s>>>(b, origin[0], origin[1], origin[2], h[0], h[1], h[2], center[0], center[1], center[2],
                                mu, out7);
}

#if MGE_PART == 2
// --------------------------------------------------------------- a group's lockstep steps
size_t xfer_size() { return sizeof(Xfer); }
void make_xfer_host(const int ratio[3], const int offset[3], void* out) {
  Xfer X = make_xfer(ratio, offset);
  memcpy(out, &X, sizeof(Xfer));
}

template <typename T, typename F>
static void go_multi(const MultiLevel& L, MultiArgs<T>& M, int kind, F f, cudaStream_t s) {
  if (L.tot[kind] <= 0) return;
  M.off = L.off[kind];
  k_multi<T, F><<<(unsigned)(L.tot[kind] / 256), 256, 0, s>>>(M, f);
}

template <typename T>
static MultiArgs<T> multi_args(const MultiLevel& L) {
  return MultiArgs<T>{(const DevBlock<T>*)L.B, L.P, L.err, L.tab, L.rt_partial, L.npart, L.rt_out, nullptr, L.nc};
}

template <typename T>
static void multi_bcond(const MultiLevel& L, MultiArgs<T>& M, cudaStream_t s, bool faces_only = false, int cut = 0) {
  go_multi(L, M, MK_BC0, FBcond<T, 0>{cut}, s);
  if (faces_only) return;
  go_multi(L, M, MK_BC1, FBcond<T, 1>{0}, s);
  go_multi(L, M, MK_BC2, FBcond<T, 2>{0}, s);
}

// timestep (optionally) and euler.f90:1-462 on one block of every case: the
// phases of enqueue_euler's per-phase path (line sweeps in global memory)
template <typename T, bool S>
static void multi_euler_t(const MultiLevel& L, const StageArgs* A, int mstage, bool with_timestep, bool lfir,
                          bool rt, cudaStream_t s) {
  MultiArgs<T> M = multi_args<T>(L);
  if (with_timestep) {
    if (L.aux32)
      go_multi(L, M, MK_PHYS, FTimestep<T, float, true>{}, s);
    else
      go_multi(L, M, MK_PHYS, FTimestep<T, T, S>{}, s);
  }
  if (lfir) go_multi(L, M, MK_N5, FCopyWs<T>{}, s);
  if (!with_timestep) go_multi(L, M, MK_N, FCopyWn<T>{}, s);
  for (int m = 1; m <= mstage; m++) {
    const StageArgs& a = A[m - 1];
    if (L.prep_rows && L.fast)
      go_multi(L, M, MK_PREP3, FPrepRows<T, true, S>{a.dissip_on}, s);
    else if (L.prep_rows)
      go_multi(L, M, MK_PREP3, FPrepRows<T, false, S>{a.dissip_on}, s);
    else if (L.fast)
      go_multi(L, M, MK_PREP, FPrep<T, true, S>{a.dissip_on}, s);
    else
      go_multi(L, M, MK_PREP, FPrep<T, false, S>{a.dissip_on}, s);
    if (L.fast) {
      if (a.dissip_on) go_multi(L, M, MK_FACE3, FFaceRows<T, true, S>{1, (T)a.cd}, s);
    } else if (L.face_rows) {
      go_multi(L, M, MK_FACE3, FFaceRows<T, false, S>{a.dissip_on, (T)a.cd}, s);
    } else if (a.dissip_on) {
      go_multi(L, M, MK_FACE, FFace<T, S>{a.dissip_on, (T)a.cd}, s);
    } else {
      go_multi(L, M, MK_FACE, FFaceConv<T>{}, s);
    }
    go_multi(L, M, MK_REC, FRec<T>{a.dissip_on, (T)a.cd}, s);
    if (L.fast)
      go_multi(L, M, MK_PHYS, FCombine<T, true, S>{a}, s);
    else
      go_multi(L, M, MK_PHYS, FCombine<T, false, S>{a}, s);
    if (a.lres) return;
    if (a.irs) {
      if constexpr (std::is_same<T, double>::value) {
        if (L.aux32) {
          go_multi(L, M, MK_IRS0, FIrsMixed<double, float, 0>{}, s);
          go_multi(L, M, MK_IRS1, FIrsMixed<float, float, 1>{}, s);
          go_multi(L, M, MK_IRS2, FIrsMixed<float, double, 2>{}, s);
        } else {
          go_multi(L, M, MK_IRS0, FIrs<T, T, 0>{}, s);
          go_multi(L, M, MK_IRS1, FIrs<T, T, 1>{}, s);
          go_multi(L, M, MK_IRS2, FIrs<T, T, 2>{}, s);
        }
      } else {
        go_multi(L, M, MK_IRS0, FIrs<T, T, 0>{}, s);
        go_multi(L, M, MK_IRS1, FIrs<T, T, 1>{}, s);
        go_multi(L, M, MK_IRS2, FIrs<T, T, 2>{}, s);
      }
      go_multi(L, M, MK_PHYS, FUpdate<T, S>{a}, s);
    }
    go_multi(L, M, MK_CUT, FCutcell<T>{}, s);
    multi_bcond(L, M, s, a.faces_only && m < mstage, 1);
  }
  if (rt) {
    go_multi(L, M, MK_RTP, FRtrmsPartial<T>{}, s);
    go_multi(L, M, MK_ONE, FRtrmsFinal<T>{}, s);
  }
}

// every case's residual of the cycle and its error word, into two arrays
template <typename T> struct FGather {
  double* res;
  unsigned* errs;
  __device__ void operator()(const MultiArgs<T>& M, int q, long long t, const DevBlock<T>&, const PhysParams&) const {
    if (t == 0) {
      res[q] = *M.rt_out[q];
      errs[q] = *M.err[q];
    }
  }
};

void gather_residuals(const MultiLevel& L, double* res, unsigned* errs, cudaStream_t s) {
  if (L.f32) {
    MultiArgs<float> M = multi_args<float>(L);
    go_multi(L, M, MK_ONE, FGather<float>{res, errs}, s);
  } else {
    MultiArgs<double> M = multi_args<double>(L);
    go_multi(L, M, MK_ONE, FGather<double>{res, errs}, s);
  }
}

// The whole update of every case of a group as ONE persistent cooperative
// launch: the phases of multi_euler_t in the same order, a grid-wide barrier
// between dependent phases, each phase's thread blocks of 256 items dealt
// over the resident blocks (a block serves one case at a time, so the
// per-block reductions stay within a case).  For the small levels, where a
// phase's launch costs more than its work.
struct GroupEuler {
  const long long* off[MK_COUNT];
  long long tot[MK_COUNT];
  int mstage, do_timestep, lfir, rt, fast, aux32, prep_rows, face_rows;
  StageArgs st[8];  // the stages (at most 8)
};

__device__ __forceinline__ int case_of(const long long* off, int nc, long long base) {
  int lo = 0, hi = nc - 1;  // the last q with off[q] <= base
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= base) lo = mid; else hi = mid - 1;
  }
  return lo;
}

template <typename T, typename F>
__device__ __forceinline__ void group_phase(const MultiArgs<T>& M, const GroupEuler& G, int kind, const F& f) {
  const long long tot = G.tot[kind];
  for (long long base = (long long)blockIdx.x * 256; base < tot; base += (long long)gridDim.x * 256) {
    const int q = case_of(G.off[kind], M.nc, base);
    f(M, q, base - G.off[kind][q] + threadIdx.x, M.B[q], M.P[q]);
  }
}

template <typename T, typename TA>
__global__ void __launch_bounds__(256, 1) k_group_euler(MultiArgs<T> M, GroupEuler G) {
  cg::grid_group grid = cg::this_grid();
  if (G.do_timestep) {
    group_phase(M, G, MK_PHYS, FTimestep<T, TA, false>{});
  }
  if (G.lfir) group_phase(M, G, MK_N5, FCopyWs<T>{});
  if (!G.do_timestep) group_phase(M, G, MK_N, FCopyWn<T>{});
  grid.sync();
  for (int m = 1; m <= G.mstage; m++) {
    const StageArgs& a = G.st[m - 1];
    if (G.prep_rows && G.fast)
      group_phase(M, G, MK_PREP3, FPrepRows<T, true, false>{a.dissip_on});
    else if (G.prep_rows)
      group_phase(M, G, MK_PREP3, FPrepRows<T, false, false>{a.dissip_on});
    else
      group_phase(M, G, MK_PREP, FPrep<T, false, false>{a.dissip_on});
    grid.sync();
    if (G.fast) {
      if (a.dissip_on) group_phase(M, G, MK_FACE3, FFaceRows<T, true, false>{1, (T)a.cd});
    } else if (G.face_rows) {
      group_phase(M, G, MK_FACE3, FFaceRows<T, false, false>{a.dissip_on, (T)a.cd});
    } else if (a.dissip_on) {
      group_phase(M, G, MK_FACE, FFace<T, false>{a.dissip_on, (T)a.cd});
    } else {
      group_phase(M, G, MK_FACE, FFaceConv<T>{});
    }
    group_phase(M, G, MK_REC, FRec<T>{a.dissip_on, (T)a.cd});
    grid.sync();
    if (G.fast)
      group_phase(M, G, MK_PHYS, FCombine<T, true, false>{a});
    else
      group_phase(M, G, MK_PHYS, FCombine<T, false, false>{a});
    grid.sync();
    if (a.lres) return;
    if (a.irs) {
      if constexpr (std::is_same<T, double>::value && std::is_same<TA, float>::value) {
        group_phase(M, G, MK_IRS0, FIrsMixed<double, float, 0>{});
        grid.sync();
        group_phase(M, G, MK_IRS1, FIrsMixed<float, float, 1>{});
        grid.sync();
        group_phase(M, G, MK_IRS2, FIrsMixed<float, double, 2>{});
      } else {
        group_phase(M, G, MK_IRS0, FIrs<T, T, 0>{});
        grid.sync();
        group_phase(M, G, MK_IRS1, FIrs<T, T, 1>{});
        grid.sync();
        group_phase(M, G, MK_IRS2, FIrs<T, T, 2>{});
      }
      grid.sync();
      group_phase(M, G, MK_PHYS, FUpdate<T, false>{a});
      grid.sync();
    }
    if (G.tot[MK_CUT] > 0) {
      group_phase(M, G, MK_CUT, FCutcell<T>{});
      grid.sync();
    }
    group_phase(M, G, MK_BC0, FBcond<T, 0>{1});
    grid.sync();
    if (a.faces_only && m < G.mstage) continue;
    group_phase(M, G, MK_BC1, FBcond<T, 1>{0});
    grid.sync();
    if (G.tot[MK_BC2] > 0) {
      group_phase(M, G, MK_BC2, FBcond<T, 2>{0});
      grid.sync();
    }
  }
  if (G.rt) {
    group_phase(M, G, MK_RTP, FRtrmsPartial<T>{});
    grid.sync();
    group_phase(M, G, MK_ONE, FRtrmsFinal<T>{});
  }
}

// resident blocks of the group kernel on the device (0: no cooperative launch)
template <typename T, typename TA>
static int group_grid() {
  static int cached[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 0;
  if (cached[dev]) return cached[dev] > 0 ? cached[dev] : 0;
  int nsm = 0, per = 0, coop = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_group_euler<T, TA>, 256, 0);
  cached[dev] = (coop && per > 0) ? nsm * per : -1;
  return cached[dev] > 0 ? cached[dev] : 0;
}

// the group's update as one cooperative launch; false when it cannot run so
template <typename T>
static bool group_euler_coop(const MultiLevel& L, const StageArgs* A, int mstage, bool with_timestep, bool lfir,
                             bool rt, cudaStream_t s) {
  const bool mixed32 = std::is_same<T, double>::value && L.aux32;
  const int gmax = mixed32 ? group_grid<T, float>() : group_grid<T, T>();
  if (gmax <= 0) return false;
  GroupEuler G;
  memset(&G, 0, sizeof(G));
  long long most = 0;
  for (int k = 0; k < MK_COUNT; k++) {
    G.off[k] = L.off[k];
    G.tot[k] = L.tot[k];
    most = std::max(most, L.tot[k] / 256);
  }
  G.mstage = mstage;
  G.do_timestep = with_timestep;
  G.lfir = lfir;
  G.rt = rt;
  G.fast = L.fast;
  G.aux32 = L.aux32;
  G.prep_rows = L.prep_rows || (L.fast && L.coop);  // a contracted level always has the split scheme
  G.face_rows = L.face_rows;
  for (int m = 0; m < mstage && m < 8; m++) G.st[m] = A[m];
  MultiArgs<T> M = multi_args<T>(L);
  const int grid = (int)std::max<long long>(1, std::min<long long>(most, gmax));
  void* args[] = {&M, &G};
  void* fn = mixed32 ? (void*)k_group_euler<T, float> : (void*)k_group_euler<T, T>;
  if (cudaLaunchCooperativeKernel(fn, grid, 256, args, 0, s) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return true;
}

void multi_euler(const MultiLevel& L, const StageArgs* A, int mstage, bool with_timestep, bool lfir, bool rt,
                 cudaStream_t s) {
  if (L.coop) {
    const bool done = L.f32 ? group_euler_coop<float>(L, A, mstage, with_timestep, lfir, rt, s)
                            : group_euler_coop<double>(L, A, mstage, with_timestep, lfir, rt, s);
    if (done) return;
  }
  if (L.f32)
    multi_euler_t<float, true>(L, A, mstage, with_timestep, lfir, rt, s);
  else if (L.tot[MK_PHYS] > kPlainCells)
    multi_euler_t<double, true>(L, A, mstage, with_timestep, lfir, rt, s);
  else
    multi_euler_t<double, false>(L, A, mstage, with_timestep, lfir, rt, s);
}

template <typename TC, typename TF, typename F>
static void go_pair(const MultiPair& Pp, MultiPairArgs<TC, TF>& M, int kind, F f, cudaStream_t s) {
  if (Pp.tot[kind] <= 0) return;
  M.off = Pp.off[kind];
  k_multi2<TC, TF, F><<<(unsigned)(Pp.tot[kind] / 256), 256, 0, s>>>(M, f);
}

template <typename TC, typename TF>
static MultiPairArgs<TC, TF> pair_args(const MultiPair& Pp) {
  return MultiPairArgs<TC, TF>{(const DevBlock<TC>*)Pp.C, (const DevBlock<TF>*)Pp.F, (const Xfer*)Pp.X, Pp.marker,
                               Pp.dc, Pp.P, nullptr, Pp.nc};
}

// the pair's precisions: (coarse, fine) in {(double, double), (float, double), (float, float)}
template <typename Fn>
static void with_pair_types(const MultiPair& Pp, Fn&& fn) {
  if (!Pp.c32 && !Pp.f32)
    fn((double*)nullptr, (double*)nullptr);
  else if (Pp.c32 && !Pp.f32)
    fn((float*)nullptr, (double*)nullptr);
  else
    fn((float*)nullptr, (float*)nullptr);
}

// movco.f90:21-47 for the group: restriction of each case's child onto its
// block on this level, depvars, wn, bcond (one block per level: no overlap)
void multi_movco_level(const MultiLevel& L, const MultiPair* pair, cudaStream_t s) {
  if (pair)
    with_pair_types(*pair, [&](auto* tc, auto* tf) {
      using TC = std::remove_pointer_t<decltype(tc)>;
      using TF = std::remove_pointer_t<decltype(tf)>;
      MultiPairArgs<TC, TF> M = pair_args<TC, TF>(*pair);
      go_pair(*pair, M, MP_COLLC, FCollc<TC, TF>{}, s);
    });
  auto rest = [&](auto* tp) {
    using T = std::remove_pointer_t<decltype(tp)>;
    MultiArgs<T> M = multi_args<T>(L);
    go_multi(L, M, MK_N, FDepvarsWn<T>{}, s);
    multi_bcond(L, M, s);
  };
  if (L.f32)
    rest((float*)nullptr);
  else
    rest((double*)nullptr);
}

// movfin.f90:20-39 for the group: prolongation from each case's parent,
// depvars, bc_embed, bcond
void multi_movfin_level(const MultiLevel& L, const MultiPair& pair, bool fmg, cudaStream_t s) {
  with_pair_types(pair, [&](auto* tc, auto* tf) {
    using TC = std::remove_pointer_t<decltype(tc)>;
    using TF = std::remove_pointer_t<decltype(tf)>;
    MultiPairArgs<TC, TF> M = pair_args<TC, TF>(pair);
    if (!fmg) go_pair(pair, M, MP_CN, FAddwDiff<TC, TF>{}, s);
    go_pair(pair, M, MP_FPHYS, FAddw<TC, TF>{fmg ? 1 : 0}, s);
    MultiArgs<TF> F = multi_args<TF>(L);
    go_multi(L, F, MK_N, FDepvars<TF>{}, s);
    if (pair.embed) go_pair(pair, M, MP_FN, FEmbed<TC, TF>{}, s);
    multi_bcond(L, F, s);
  });
}

#else

// explicit instantiations
#define MGE_INST(T)                                                                                              \
  template void launch_timestep<T>(const DevBlock<T>&, const PhysParams&, unsigned*, cudaStream_t, bool, bool); \
  template void launch_solut<T>(const DevBlock<T>&, const PhysParams&, double, double, int, double*, cudaStream_t); \
  template void launch_stage<T>(const DevBlock<T>&, const PhysParams&, const StageArgs&, unsigned*, cudaStream_t,     \
                                cudaStream_t, cudaEvent_t, cudaEvent_t);                                               \
  template void launch_stage_part<T>(int, const DevBlock<T>&, const PhysParams&, const StageArgs&, unsigned*,       \
                                     cudaStream_t);                                                             \
  template void launch_irs_part<T>(int, const DevBlock<T>&, const PhysParams&, const IrsTables*, cudaStream_t,    \
                                   bool, const int*, const StageArgs*);                                         \
  template int launch_euler_coop<T>(const DevBlock<T>&, const PhysParams&, const EulerLaunch&, int, cudaStream_t,  \
                                    bool);                                                                      \
  template void launch_irs<T>(const DevBlock<T>&, const PhysParams&, const IrsTables*, cudaStream_t, bool,       \
                              const int*, const StageArgs*);                                                    \
  template void launch_cutcell<T>(const DevBlock<T>&, const PhysParams&, unsigned*, cudaStream_t);              \
  template void launch_bcond<T>(const DevBlock<T>&, const PhysParams&, cudaStream_t, bool, unsigned*);          \
  template long long bc_items<T>(const DevBlock<T>&, int);                                                      \
  template long long split_items<T>(const DevBlock<T>&, int);                                                   \
  template void launch_rtrms<T>(const DevBlock<T>&, const PhysParams&, double*, int, double*, cudaStream_t, \
                                unsigned*);                                                                    \
  template void launch_depvars_all<T>(const DevBlock<T>&, const PhysParams&, cudaStream_t);                     \
  template void launch_copy_ws<T>(const DevBlock<T>&, cudaStream_t);                                            \
  template void launch_copy_wn<T>(const DevBlock<T>&, cudaStream_t);                                            \
  template void launch_depvars_wn<T>(const DevBlock<T>&, const PhysParams&, cudaStream_t);                      \
  template void launch_init_free<T>(const DevBlock<T>&, const PhysParams&, cudaStream_t);                       \
  template void launch_forces<T>(const DevBlock<T>&, const double*, const double*, const double*, double, double*,  \
                                 cudaStream_t);                                                                  \
  template void launch_overlap<T>(const DevBlock<T>&, const DevBlock<T>&, const long long*, const long long*,        \
                                  const double*, long long, const PhysParams&, cudaStream_t);
#if MGE_PART == 0
MGE_INST(double)
#else
MGE_INST(float)
#endif
#undef MGE_INST
#define MGE_XFER(TC, TF)                                                                                         \
  template void launch_collc<TC, TF>(const DevBlock<TC>&, const DevBlock<TF>&, const int*, const int*, uint8_t*,   \
                                     cudaStream_t);                                                             \
  template void launch_addw<TF, TC>(const DevBlock<TF>&, const DevBlock<TC>&, const int*, const int*, int,          \
                                    double*, cudaStream_t);                                                     \
  template void launch_embed<TF, TC>(const DevBlock<TF>&, const DevBlock<TC>&, const int*, const int*,              \
                                     const PhysParams&, cudaStream_t);
#if MGE_PART == 0
MGE_XFER(double, double)
MGE_XFER(float, double)
#else
MGE_XFER(float, float)
#endif
#undef MGE_XFER
#endif  // MGE_PART == 2


}  // namespace mge
