// newton_dev.cuh -- device code shared by the local-solve kernels
// (newton_f32.cu, newton_f64.cu) and the end-of-step kernel (newton.cu): the
// flow rules and the damped Newton iteration in plain order, the block sums, and the
// constants a launch fills.
#pragma once
#include <cmath>
#include <cstring>
#include "mth_common.cuh"
#include "mth_internal.h"
#include "local_solve.cuh"

namespace mth {

// |r|^e for the flow rule; integer exponents by repeated squaring.
template <typename T>
__device__ __forceinline__ T pow_abs(T a, int ei, T ef) {
  if (ei > 0) {
    T r = (T)1, b = a;
    int e = ei;
    while (e) {
      if (e & 1) r *= b;
      b *= b;
      e >>= 1;
    }
    return r;
  }
  return a > (T)0 ? (T)pow(a, ef) : (T)0;
}

// Flow rule in crystal axes at deviatoric stress x (5).  tauf: forward CRSS
// per system; the backward CRSS is forward + tau_off.  Returns edot (5),
// optional Hessian contribution D (15, packed upper triangle) and
// psi = sum gamd0 tau |r|^(n+1)/(n+1) = sum gamd0 |rss| |r|^n/(n+1).
// gam (optional) receives the shear rates.
template <typename TF, bool WANT_D>
__device__ __forceinline__ void flow_rule(const PhaseConst& ph, const TF x[5], const TF* tauf, TF tau_off, TF ed[5],
                                          TF D[15], TF& psi, TF* gam) {
#pragma unroll
  for (int i = 0; i < 5; i++) ed[i] = 0;
  if (WANT_D) {
#pragma unroll
    for (int i = 0; i < 15; i++) D[i] = 0;
  }
  psi = 0;
  const int ns = ph.nsys;
  const TF n = cpick<TF>(ph.nrs, ph.nrsf);
  const TF g0 = cpick<TF>(ph.gamd0, ph.gamd0f);
  const TF inv_np1 = (TF)1 / (n + (TF)1);
  const int nm1 = ph.nrs_int > 0 ? ph.nrs_int - 1 : 0;
  // fully unrolled over the NSYS slots so the per-voxel CRSS stay in registers
#pragma unroll
  for (int s = 0; s < NSYS; s++) {
    if (s < ns) {
      TF m[5];
#pragma unroll
      for (int i = 0; i < 5; i++) m[i] = cpick<TF>(ph.m_xt[s][i], ph.m_xtf[s][i]);
      const TF rss = m[0] * x[0] + m[1] * x[1] + m[2] * x[2] + m[3] * x[3] + m[4] * x[4];
      const TF tau = rss < (TF)0 ? tauf[s] + tau_off : tauf[s];
      const TF itau = (TF)1 / tau;
      const TF r = rss * itau;
      const TF ar = fabs(r);
      const TF pnm1 = pow_abs<TF>(ar, nm1, n - (TF)1);   // |r|^(n-1)
      const TF pn = pnm1 * ar;                             // |r|^n
      const TF g = g0 * (r > (TF)0 ? pn : -pn);
      if (gam) gam[s] = g;
#pragma unroll
      for (int i = 0; i < 5; i++) ed[i] += m[i] * g;
      if (WANT_D) {
        const TF w = g0 * n * pnm1 * itau;
        int q = 0;
#pragma unroll
        for (int i = 0; i < 5; i++)
#pragma unroll
          for (int j = i; j < 5; j++) D[q++] += w * m[i] * m[j];
      }
      psi += g0 * fabs(rss) * pn * inv_np1;
    } else if (gam) {
      gam[s] = 0;
    }
  }
}

// Dislocation-density flow rule of StrainRate_Orowan, forward plus backward
// jumps (src/constitutive.c:507-721), in crystal axes: per system
// gdot = g0 sinh((|rss| - tp)/td) sign(rss) where |rss| > tp, else 0, with
// tp the passing stress, td = tau_0 + cutting stress and g0 the reference
// rate of the step (from the dislocation densities, dd.cu).  It is the
// gradient of the convex potential psi = sum g0 td (cosh(t) - 1),
// t = max(|rss| - tp, 0)/td, written 2 g0 td sinh^2(t/2).
template <typename TF, bool WANT_D>
__device__ __forceinline__ void flow_rule_dd(const PhaseConst& ph, const TF x[5], const TF* tp, const TF* td,
                                             const TF* g0, TF ed[5], TF D[15], TF& psi, TF* gam) {
#pragma unroll
  for (int i = 0; i < 5; i++) ed[i] = 0;
  if (WANT_D) {
#pragma unroll
    for (int i = 0; i < 15; i++) D[i] = 0;
  }
  psi = 0;
  const int ns = ph.nsys;
#pragma unroll
  for (int s = 0; s < NSYS; s++) {
    if (s < ns) {
      TF m[5];
#pragma unroll
      for (int i = 0; i < 5; i++) m[i] = cpick<TF>(ph.m_xt[s][i], ph.m_xtf[s][i]);
      const TF rss = m[0] * x[0] + m[1] * x[1] + m[2] * x[2] + m[3] * x[3] + m[4] * x[4];
      const TF ar = fabs(rss);
      TF g = 0, w = 0;
      if (ar > tp[s]) {
        const TF t = (ar - tp[s]) / td[s];
        const TF sh = sinh(t);
        g = g0[s] * (rss > (TF)0 ? sh : -sh);
        if (WANT_D) w = g0[s] * cosh(t) / td[s];
        const TF h = sinh((TF)0.5 * t);
        psi += (TF)2 * g0[s] * td[s] * h * h;
      }
      if (gam) gam[s] = g;
#pragma unroll
      for (int i = 0; i < 5; i++) ed[i] += m[i] * g;
      if (WANT_D) {
        int q = 0;
#pragma unroll
        for (int i = 0; i < 5; i++)
#pragma unroll
          for (int j = i; j < 5; j++) D[q++] += w * m[i] * m[j];
      }
    } else if (gam) {
      gam[s] = 0;
    }
  }
}

// Slip laws of the local solve.  Power law: forward CRSS per system, the
// backward one offset by tau_off.  Dislocation density: passing stress,
// tau_0 + cutting stress and reference rate per system.
template <typename TF>
struct PlSlip {
  TF tauf[NSYS];
  TF tau_off;
  template <bool WANT_D>
  __device__ __forceinline__ void flow(const PhaseConst& ph, const TF x[5], TF ed[5], TF D[15], TF& psi,
                                       TF* gam) const {
    flow_rule<TF, WANT_D>(ph, x, tauf, tau_off, ed, D, psi, gam);
  }
};
template <typename TF>
struct DdSlip {
  TF tp[NSYS], td[NSYS], g0[NSYS];
  template <bool WANT_D>
  __device__ __forceinline__ void flow(const PhaseConst& ph, const TF x[5], TF ed[5], TF D[15], TF& psi,
                                       TF* gam) const {
    flow_rule_dd<TF, WANT_D>(ph, x, tp, td, g0, ed, D, psi, gam);
  }
};
// slip-law state of voxel v from the fields (LAW 0: power law, 1: dislocation density)
template <int LAW, typename TF, typename TSt>
struct SlipOf;
template <typename TF, typename TSt>
struct SlipOf<0, TF, TSt> {
  using type = PlSlip<TF>;
  __device__ __forceinline__ static void load(const PhaseConst& ph, const Fields<TSt>& f, long long v, type& sl) {
    const long long P = f.nv;
#pragma unroll
    for (int s = 0; s < NSYS; s++) sl.tauf[s] = s < ph.nsys ? (TF)f.crss[s * P + v] : (TF)1;
    sl.tau_off = cpick<TF>(ph.tau_back_minus_fwd, ph.tau_offf);
  }
};
template <typename TF, typename TSt>
struct SlipOf<1, TF, TSt> {
  using type = DdSlip<TF>;
  __device__ __forceinline__ static void load(const PhaseConst& ph, const Fields<TSt>& f, long long v, type& sl) {
    const long long P = f.nv;
#pragma unroll
    for (int s = 0; s < NSYS; s++) {
      const bool a = s < ph.nsys;
      sl.tp[s] = a ? (TF)f.ddc[s * P + v] : (TF)0;
      sl.td[s] = a ? (TF)f.ddc[(NSYS + s) * P + v] : (TF)1;
      sl.g0[s] = a ? (TF)f.ddc[(2 * NSYS + s) * P + v] : (TF)0;
    }
  }
};

__device__ __forceinline__ int pk(int i, int j) {  // packed upper-triangle index of 5x5
  if (i > j) { int t = i; i = j; j = t; }
  return i * 5 - (i * (i - 1)) / 2 + (j - i);
}

// 1/d for a positive normal FP64 pivot, without FP64-pipe work besides
// three DFMA: the FP32 hardware reciprocal (rcp.approx.ftz.f32, within 1 ulp)
// of d's mantissa m in [1, 2), truncated to 24 bits, gives 1/m to within
// 2^-22; its exponent is shifted by d's with integer operations; one
// cubically convergent Newton step x <- x (1 + e + e^2), e = 1 - d x,
// takes the relative error from 2^-22 to below 2^-64, so the result is
// within an ulp or two of 1/d without the special-case handling of a
// correctly rounded divide.
template <bool QUAD = false>
__device__ __forceinline__ double pivot_rcp_nr(double d) {
  const unsigned hi = (unsigned)__double2hiint(d), lo = (unsigned)__double2loint(d);
  const int E = (int)((hi >> 20) & 0x7ffu);   // biased exponent of d (1..2046)
  const float m = __uint_as_float(0x3f800000u | ((hi & 0xfffffu) << 3) | (lo >> 29));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(m));
  const unsigned ru = __float_as_uint(r);     // 1/m in (0.5, 1]
  // 1/d = (1/m) 2^(1023 - (E - 1023)): biased FP64 exponent Er - 127 + 2046 - E
  const int eo = (int)((ru >> 23) & 0xffu) + 1919 - E;
  unsigned xhi = ((unsigned)eo << 20) | ((ru >> 3) & 0xfffffu);
  unsigned xlo = ru << 29;
  if (eo <= 0) xhi = xlo = 0u;                // 1/d below the normal range
  const double x = __hiloint2double((int)xhi, (int)xlo);
  const double e = fma(-d, x, 1.0);
  if constexpr (QUAD) return fma(x, e, x);   // quadratic step: within 2^-43 of 1/d
  return fma(x, fma(e, e, e), x);
}
// QUAD: the quadratic step, for solves whose result is rounded to FP32 (a
// pivot reciprocal off by 2^-43 is a backward error of that size in D,
// far below the FP32 rounding of the assembled Hessian and of the step)
template <typename T, bool NR, bool QUAD = false>
__device__ __forceinline__ T pivot_inv(T d) {
  if constexpr (NR && sizeof(T) == 8) return pivot_rcp_nr<QUAD>(d);
  else return (T)1 / d;
}

// dj > 0 for a pivot; for the FP64 solves of the mixed modes (NR) tested on
// the high word with integer operations instead of an FP64 compare: a
// positive finite double has a high word in [1, 0x7fefffff] (this also
// rejects +inf and the subnormals below 2^-1042, which the reciprocal
// estimate flushes).
template <typename T, bool NR>
__device__ __forceinline__ bool pivot_positive(T d) {
  if constexpr (NR && sizeof(T) == 8) return (unsigned)__double2hiint(d) - 1u < 0x7fefffffu;
  else return d > (T)0;
}

// LDL^T solve of the packed symmetric positive definite 5x5 matrix A:
// x = A^-1 b.  Returns false when a pivot is not positive.  NR: pivot
// reciprocals by pivot_rcp_nr (FP64 solves of the mixed modes).
template <typename T, bool NR = false, bool QUAD = false>
__device__ __forceinline__ bool ldl_solve5(const T* A, const T* b, T* x) {
  // U[i][k] = L[i][k] d[k], the column before its scaling by 1/d[k], kept so
  // the updates need no products L d
  T L[5][5], U[5][5], id[5];
#pragma unroll
  for (int j = 0; j < 5; j++) {
    T dj = A[pk(j, j)];
#pragma unroll
    for (int k = 0; k < 5; k++)
      if (k < j) dj -= U[j][k] * L[j][k];
    if (!pivot_positive<T, NR>(dj)) return false;
    id[j] = pivot_inv<T, NR, QUAD>(dj);
#pragma unroll
    for (int i = 0; i < 5; i++)
      if (i > j) {
        T a = A[pk(i, j)];
#pragma unroll
        for (int k = 0; k < 5; k++)
          if (k < j) a -= U[i][k] * L[j][k];
        U[i][j] = a;
        L[i][j] = a * id[j];
      }
  }
  T y[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    T a = b[i];
#pragma unroll
    for (int k = 0; k < 5; k++)
      if (k < i) a -= L[i][k] * y[k];
    y[i] = a;
  }
#pragma unroll
  for (int i = 4; i >= 0; i--) {
    T a = y[i] * id[i];
#pragma unroll
    for (int k = 0; k < 5; k++)
      if (k > i) a -= L[k][i] * x[k];
    x[i] = a;
  }
  return true;
}

// FP64 LDL^T solve of an FP32 system: the conversions by integer operations
// (f32_to_f64, f64_to_f32), as GB300 executes F2F conversions on its 1/64-rate
// FP64 pipe; the pivot reciprocals with the quadratic step (the result is
// rounded to FP32; 5 DFMA fewer per solve).
__device__ __forceinline__ bool ldl_solve5_wide(const float* H, const float* b, float* x) {
  double Hl[15], bl[5], pl[5];
#pragma unroll
  for (int i = 0; i < 15; i++) Hl[i] = f32_to_f64(H[i]);
#pragma unroll
  for (int i = 0; i < 5; i++) bl[i] = f32_to_f64(b[i]);
  const bool ok = ldl_solve5<double, true, true>(Hl, bl, pl);
#pragma unroll
  for (int i = 0; i < 5; i++) x[i] = f64_to_f32(pl[i]);
  return ok;
}

// Result of one voxel solve.
template <typename TF>
struct VoxelOut {
  TF conv_s, conv_e;   // the voxel's error contributions, in the flow-rule precision
  int iters;
  int failed;
};

// ------------------------------------------------- the local solve, in pieces
// nw_init (set-up), nw_pass_a (one flow-rule evaluation and what it decides;
// when the next Newton direction is needed it returns the system H p = -g),
// nw_pass_b (the move the direction gives) and nw_finish (back to sample
// axes, error contributions): the damped Newton iteration with every
// operation in TF, which the kernels fall back to (solve_full, solve_steep).
template <typename TF>
struct NewtonRegs {
  TF K[15], c[5];
  __device__ __forceinline__ TF k(int i) const { return K[i]; }
  __device__ __forceinline__ TF cc(int i) const { return c[i]; }
  __device__ __forceinline__ void set_k(int i, TF v) { K[i] = v; }
  __device__ __forceinline__ void set_c(int i, TF v) { c[i] = v; }
};
template <typename TF>
struct NewtonState {
  TF x[5];                     // iterate (crystal axes)
  TF h, ref2, dh, hstep2, tol2, ls_thr2;
  TF xt[5];                    // point evaluated next
  TF p[5], pn2, slope, phi0, alpha;
  TF edf[5], psif;             // rates and psi at the last evaluated point
  int it, ls, pass;
  bool done, near_root, trial, failed;
};

template <typename TF, typename Store, typename Load>
__device__ __forceinline__ void nw_init(NewtonState<TF>& s, Store& sh, const NewtonConst& nc,
                                        const TF* __restrict__ et, const Load& load) {
  const TF shh = et[ET_SEL_HH];
  TF lam6[6], eps6[6], ep6[6], Q[25];
  {
    TF R[9];
    load(lam6, eps6, ep6, R, false);
    rot_to_q<TF>(R, Q);
  }
  TF s0s[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    TF a = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) a += cpick<TF>(nc.s0dev[i * 5 + j], nc.s0devf[i * 5 + j]) * lam6[j];
    s0s[i] = a;
  }
#pragma unroll
  for (int i = 0; i < 5; i++) {
    TF a = 0, b = 0, e = 0, d = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) {
      a += Q[i * 5 + j] * lam6[j];
      b += Q[i * 5 + j] * eps6[j];
      e += Q[i * 5 + j] * ep6[j];
      d += Q[i * 5 + j] * s0s[j];
    }
    s.x[i] = a;
    sh.set_c(i, -d + e - b);
  }
  {
    TF St[25], t[25];
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = 0; j < 5; j++) St[i * 5 + j] = et[ET_STOT + pk(i, j)];
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = 0; j < 5; j++) {
        TF a = 0;
#pragma unroll
        for (int k = 0; k < 5; k++) a += Q[i * 5 + k] * St[k * 5 + j];
        t[i * 5 + j] = a;
      }
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = i; j < 5; j++) {
        TF a = 0;
#pragma unroll
        for (int k = 0; k < 5; k++) a += t[i * 5 + k] * Q[j * 5 + k];
        sh.set_k(pk(i, j), a);
      }
  }
  const TF s0hh = cpick<TF>(nc.s0hh, nc.s0hhf);
  s.h = (s0hh * lam6[5] + eps6[5] - ep6[5]) / (s0hh + shh);
  TF ref2 = 0;
#pragma unroll
  for (int i = 0; i < 6; i++) ref2 += lam6[i] * lam6[i];
  s.ref2 = ref2;
  s.dh = s.h - lam6[5];
  const TF tol = cpick<TF>(nc.tol, nc.tolf);
  s.tol2 = tol * tol;
  s.ls_thr2 = (TF)1e-6 * ref2;
  s.hstep2 = s.dh * s.dh;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    s.xt[i] = s.x[i];
    s.p[i] = 0;
  }
  s.pn2 = s.slope = s.phi0 = 0;
  s.alpha = 1;
  s.it = s.ls = s.pass = 0;
  s.done = s.near_root = s.trial = s.failed = false;
}

template <typename TF>
__device__ __forceinline__ void nw_accept(NewtonState<TF>& s) {
#pragma unroll
  for (int i = 0; i < 5; i++) s.x[i] += s.alpha * s.p[i];
  const TF step2 = s.alpha * s.alpha * s.pn2 + s.hstep2;
  s.hstep2 = 0;
  s.near_root = step2 <= s.ls_thr2;
  TF den2 = s.ref2;
  if (!(den2 > (TF)0))
    den2 = s.x[0] * s.x[0] + s.x[1] * s.x[1] + s.x[2] * s.x[2] + s.x[3] * s.x[3] + s.x[4] * s.x[4] + s.h * s.h;
  if (!(den2 > (TF)0) || step2 <= s.tol2 * den2) s.done = true;
  s.it++;
}

// Newton with a backtracking line search on Phi for large steps.  One
// flow-rule evaluation site: every evaluation (with its Hessian) is at the
// point the solve moves to next, so an accepted line-search trial supplies
// the next Newton step and the last accepted iterate supplies the final
// rates, without evaluating any point twice.  At most 41 (itmax + 1)
// passes: each Newton step takes at most 40 trials + 1.
// Returns 0: pass done, no solve; 1: the Newton direction is needed (H, mg
// filled); 2: the solve has ended.
template <typename TF, typename Store, typename Slip>
__device__ __forceinline__ int nw_pass_a(NewtonState<TF>& s, const Store& sh, const NewtonConst& nc,
                                         const PhaseConst& ph, const Slip& slip, const TF* __restrict__ et, TF H[15],
                                         TF mg[5]) {
  if (s.pass >= 41 * (nc.itmax + 1)) return 2;
  s.pass++;
  const TF dt = cpick<TF>(nc.dt, nc.dtf);
  TF Df[15];
  if (nc.flow_off) {
#pragma unroll
    for (int i = 0; i < 5; i++) s.edf[i] = 0;
#pragma unroll
    for (int i = 0; i < 15; i++) Df[i] = 0;
    s.psif = 0;
  } else {
    slip.template flow<true>(ph, s.xt, s.edf, Df, s.psif, nullptr);
  }
  TF Kx[5];
#pragma unroll
  for (int i = 0; i < 5; i++) {
    TF a = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) a += sh.k(pk(i, j)) * s.xt[j];
    Kx[i] = a;
  }
  if (s.trial) {
    TF phi = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) phi += s.xt[i] * ((TF)0.5 * Kx[i] + sh.cc(i));
    phi += dt * s.psif;
    if (!(phi <= s.phi0 + (TF)1e-4 * s.alpha * s.slope)) {
      TF den = (TF)2 * (phi - s.phi0 - s.slope * s.alpha);
      TF an = den > (TF)0 ? -s.slope * s.alpha * s.alpha / den : (TF)0.5 * s.alpha;
      an = fmin(an, (TF)0.5 * s.alpha);
      s.alpha = fmax(an, (TF)0.1 * s.alpha);
      s.ls++;
#pragma unroll
      for (int i = 0; i < 5; i++) s.xt[i] = s.x[i] + s.alpha * s.p[i];
      if (!(s.alpha * s.alpha * s.pn2 <= (TF)1e-28 * (s.ref2 + (TF)1)) && s.ls < 40) return 0;
      nw_accept(s);
      s.trial = false;
      return 0;
    }
    nw_accept(s);
    s.trial = false;
  }
  if (s.done || s.it >= nc.itmax) return 2;
  TF g[5];
#pragma unroll
  for (int i = 0; i < 5; i++) g[i] = Kx[i] + sh.cc(i) + dt * s.edf[i];
  if (sizeof(TF) == 4 && nc.bound_stop) {
    TF den2 = s.ref2;
    if (!(den2 > (TF)0))
      den2 = s.x[0] * s.x[0] + s.x[1] * s.x[1] + s.x[2] * s.x[2] + s.x[3] * s.x[3] + s.x[4] * s.x[4] + s.h * s.h;
    const TF mu = et[ET_STOT_MIN];
    const TF gn2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2] + g[3] * g[3] + g[4] * g[4];
    if (gn2 <= s.tol2 * den2 * mu * mu) {
      s.done = true;
      return 2;
    }
  }
#pragma unroll
  for (int i = 0; i < 15; i++) H[i] = sh.k(i) + dt * Df[i];
#pragma unroll
  for (int i = 0; i < 5; i++) mg[i] = -g[i];
  // Phi at x (= xt here), for a line search along the coming direction
  TF phi0 = 0;
#pragma unroll
  for (int i = 0; i < 5; i++) phi0 += s.x[i] * ((TF)0.5 * Kx[i] + sh.cc(i));
  s.phi0 = phi0 + dt * s.psif;
  return 1;
}

// the move along the solved direction p of -g (mg); false: the solve failed
template <typename TF>
__device__ __forceinline__ bool nw_pass_b(NewtonState<TF>& s, const NewtonConst& nc, const TF p[5], bool ok,
                                          const TF mg[5]) {
  if (!ok) {
    s.failed = true;
    return false;
  }
  s.pn2 = 0;
  s.slope = 0;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    s.p[i] = p[i];
    s.pn2 += p[i] * p[i];
    s.slope -= mg[i] * p[i];
  }
  s.alpha = 1;
  if (s.pn2 > s.ls_thr2 && !nc.flow_off) {
    s.ls = 0;
    s.trial = true;
#pragma unroll
    for (int i = 0; i < 5; i++) s.xt[i] = s.x[i] + s.alpha * s.p[i];
    return true;
  }
  nw_accept(s);
#pragma unroll
  for (int i = 0; i < 5; i++) s.xt[i] = s.x[i];
  return true;
}

template <typename TF, typename Load>
__device__ __forceinline__ VoxelOut<TF> nw_finish(const NewtonState<TF>& s, const NewtonConst& nc,
                                                  const TF* __restrict__ et, const Load& load, TF* sig6, TF* ed6) {
  VoxelOut<TF> o;
  o.iters = s.it;
  o.failed = (s.failed || !s.done) ? 1 : 0;
  const TF dt = cpick<TF>(nc.dt, nc.dtf);
  const TF shh = et[ET_SEL_HH];
  TF lam6[6], eps6[6], ep6[6], Q[25];
  {
    TF R[9];
    load(lam6, eps6, ep6, R, true);
    rot_to_q<TF>(R, Q);
  }
  TF ss[5], es[5];
#pragma unroll
  for (int j = 0; j < 5; j++) {
    TF a = 0, b = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      a += Q[i * 5 + j] * s.x[i];
      b += Q[i * 5 + j] * s.edf[i];
    }
    ss[j] = a;
    es[j] = b;
  }
  TF cs = s.dh * s.dh, ce = 0;
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const TF ds = ss[i] - lam6[i];
    cs += ds * ds;
    TF de = ep6[i] + dt * es[i] - eps6[i];
#pragma unroll
    for (int j = 0; j < 5; j++) de += et[ET_SEL + pk(i, j)] * ss[j];
    ce += de * de;
  }
  {
    const TF de = ep6[5] + shh * s.h - eps6[5];
    ce += de * de;
  }
  o.conv_s = sqrt(cs);
  o.conv_e = sqrt(ce);
#pragma unroll
  for (int j = 0; j < 5; j++) {
    sig6[j] = ss[j];
    ed6[j] = es[j];
  }
  sig6[5] = s.h;
  ed6[5] = 0;
  return o;
}

// Local solve of one crystal voxel by the damped iteration in its plain order:
// the FP64 mode's fallback and the iterations with a tight cap (solve_full), the
// FP32 modes' irregular voxels and iterations in plain order (solve_steep).
// lam6/eps6/ep6: LT sample-frame inputs (lambda = current stress, total strain,
// plastic strain); et: elastic-class row (initial orientation).  Outputs sig6
// (sample frame) and ed6 (plastic strain rate, sample frame).
// TF: flow rule, residual, Hessian assembly, line search and frame transforms;
// TL: precision of the 5x5 solve, at every step or (ROOT_ONLY) for the steps
// within 1e-3 |lambda| of the root, with TF for the large early ones.
// load(lam6, eps6, ep6, R, again) fills the voxel's inputs; it is called
// at the start and again (again = true: loads the compiler may not merge
// with the first) for the back-transform and the error norms, so neither
// the inputs nor the 5x5 frame rotation stay live across the Newton loop.
template <typename TF, typename TL, bool ROOT_ONLY, typename Slip, typename Load>
__device__ VoxelOut<TF> solve_voxel(const NewtonConst& nc, const PhaseConst& ph, const TF* __restrict__ et, const Slip& slip,
                                    const Load& load, TF* sig6, TF* ed6) {
  NewtonState<TF> s;
  NewtonRegs<TF> r;
  nw_init(s, r, nc, et, load);
  for (;;) {
    TF H[15], mg[5];
    const int k = nw_pass_a(s, r, nc, ph, slip, et, H, mg);
    if (k == 2) break;
    if (k == 0) continue;
    TF p[5];
    bool ok;
    if constexpr (sizeof(TL) > sizeof(TF))
      ok = !ROOT_ONLY || s.near_root ? ldl_solve5_wide(H, mg, p) : ldl_solve5<TF>(H, mg, p);
    else
      ok = ldl_solve5<TF>(H, mg, p);
    if (!nw_pass_b(s, nc, p, ok, mg)) break;
  }
  return nw_finish(s, nc, et, load, sig6, ed6);
}

// ------------------------------------------------------------ reductions
// Block sum of W per-thread values for 256-thread blocks, in FP64 in a fixed
// order: the values are staged in shared memory (in their own precision);
// 16 threads per component each sum 16 of them (stride 16), one thread per
// component sums the 16 partials.  The row stride 256 + 16 keeps the
// two components read by one warp on opposite bank halves.
template <typename TV, int W>
__device__ __forceinline__ void block_reduce_smem(const TV (&v)[W], double* out) {
  constexpr int NT = 256, LD = NT + 16;
  static_assert(W <= 16, "at most 16 components");
  __shared__ TV sv[W][LD];
  __shared__ double sp[W][16];
  const int t = threadIdx.x;
#pragma unroll
  for (int i = 0; i < W; i++) sv[i][t] = v[i];
  __syncthreads();
  {
    const int comp = t >> 4, chunk = t & 15;
    if (comp < W) {
      double a = 0.0;
#pragma unroll
      for (int k = 0; k < NT / 16; k++) a += (double)sv[comp][k * 16 + chunk];
      sp[comp][chunk] = a;
    }
  }
  __syncthreads();
  if (t < W) {
    double a = 0.0;
#pragma unroll
    for (int k = 0; k < 16; k++) a += sp[t][k];
    out[(size_t)blockIdx.x * W + t] = a;
  }
}

// Sums over a warp of NC values per lane, in FP64 in a fixed order: rows[c]
// of the warp's 32 columns (row stride LD) hold the values; 32/NC lanes
// per component each add their share, so a warp issues 11 (NC = 10) or 16
// (NC = 16) FP64 additions.  Lane c < NC returns component c's sum.  The
// read order is rotated by the component, so the lanes hit distinct banks.
template <typename TV, int NC, int LD>
__device__ __forceinline__ double warp_sums(const TV* rows, int lane) {
  constexpr int NP = 32 / NC, LEN = (32 + NP - 1) / NP;
  const int comp = lane % NC, part = lane / NC;
  double a = 0.0;
  if (part < NP) {
#pragma unroll
    for (int k = 0; k < LEN; k++) {
      int j = k + comp;
      j -= j >= LEN ? LEN : 0;
      const int i = part * LEN + j;
      if (32 % LEN == 0 || i < 32) a += to_f64(rows[comp * LD + i]);
    }
  }
  double b = a;
#pragma unroll
  for (int p = 1; p < NP; p++) b += __shfl_sync(0xffffffffu, a, (lane + p * NC) & 31);
  return b;
}

// A block's row of partial sums: the NPART values of the Newton kernels.
// !GEN (phase 1 the only crystal phase): the phase-1 stress sums (8..13)
// are the total ones (2..7), added once and written twice.  rows: this
// warp's columns of shared memory, its solve's data no longer needed.
template <typename TV, bool GEN, int LD>
__device__ __forceinline__ void newton_block_sums(const TV (&v)[NPART], const Column<TV, LD>& col,
                                                  double* __restrict__ out) {
  constexpr int NC = GEN ? 16 : 10;
  __shared__ double wsum[LD / 32][NPART];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncwarp();
#pragma unroll
  for (int c = 0; c < NC; c++) col(c) = v[!GEN && c >= 8 ? c + 6 : c];
  __syncwarp();
  const double a = warp_sums<TV, NC, LD>(col.p - lane, lane);
  if (lane < NC) {
    if (GEN || lane < 8) wsum[w][lane] = a;
    else wsum[w][lane + 6] = a;
    if (!GEN && lane >= 2 && lane < 8) wsum[w][lane + 6] = a;
  }
  __syncthreads();
  if (threadIdx.x < NPART) {
    double t = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += wsum[k][threadIdx.x];
    out[(size_t)blockIdx.x * NPART + threadIdx.x] = t;
  }
}

// Loads of a global value that the compiler keeps as separate loads (used to
// re-read a voxel's inputs after the Newton loop instead of holding them).
__device__ __forceinline__ float ld_again(const float* p) {
  float v;
  asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
__device__ __forceinline__ double ld_again(const double* p) {
  double v;
  asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(__cvta_generic_to_global(p)));
  return v;
}
template <typename T>
__device__ __forceinline__ T ld_sel(const T* p, bool again) { return again ? ld_again(p) : *p; }

// ------------------------------------------------------------ launch constants
// the FP32 constants of the local solve; predictor: the FP64 mode's start
inline void fill_local(const NewtonConst& nc, bool predictor, LocalConst& lc) {
  memset(&lc, 0, sizeof(lc));
  for (int k = 0; k < 2; k++) {
    const PhaseConst& ph = nc.ph[k];
    SlipF& s = lc.ph[k];
    s.type = ph.type;
    s.gamd0 = (float)ph.gamd0;
    s.gn = (float)(ph.gamd0 * ph.nrs);
    s.inv_np1 = (float)(1.0 / (ph.nrs + 1.0));
    s.nm1f = (float)(ph.nrs - 1.0);
    const double e = ph.nrs - 1.0, fl = floor(e);
    s.half = e - fl == 0.5;
    s.nm1 = (e == fl || s.half) && fl >= 1.0 && fl < 64.0 ? (int)fl : -1;
    s.tau_off = (float)ph.tau_back_minus_fwd;
    s.chord2 = ph.type == 0 ? (float)pow(0.4 * nc.tol / (ph.nrs * ph.nrs), 2.0 / 3.0) : 0.0f;   // n^2 d^3 / 2 <= tol / 5
    for (int i = 0; i < NSYS; i++) {
      int q = 0;
      for (int a = 0; a < 5; a++) {
        const float hi = (float)ph.m_xt[i][a], lo = (float)(ph.m_xt[i][a] - (double)hi);
        (i & 1 ? s.m[i / 2][a].y : s.m[i / 2][a].x) = hi;
        (i & 1 ? s.ml[i / 2][a].y : s.ml[i / 2][a].x) = lo;
      }
      for (int a = 0; a < 5; a++)
        for (int b = a; b < 5; b++, q++)
          (q & 1 ? s.mm[i][q / 2].y : s.mm[i][q / 2].x) = (float)(ph.m_xt[i][a] * ph.m_xt[i][b]);
    }
  }
  for (int i = 0; i < 25; i++) lc.s0[i] = (float)nc.s0dev[i];
  lc.s0hh = (float)nc.s0hh;
  lc.dt = (float)nc.dt;
  lc.tol = predictor ? 1e-4f : (float)nc.tol;
  lc.tol64 = (float)nc.tol;
  lc.itmax = nc.itmax;
  lc.flow_off = nc.flow_off;
  lc.bound_stop = nc.bound_stop;
}

// The kernels for one crystal phase whose forward and backward CRSS are
// equal and whose n-1 is a whole or half number (GEN = false) read the
// phase's constants at fixed offsets, keep one 1/tau per system and call no
// pow; every other case takes the general ones.
inline bool plain_phase(const NewtonConst& nc, const LocalConst& lc) {
  return nc.ph1_only && nc.ph[0].tau_back_minus_fwd == 0.0 && lc.ph[0].nm1 > 0;
}

}  // namespace mth
