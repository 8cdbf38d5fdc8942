// newton_f64.cu -- the local solve of the FP64 mode and of the array entry
// points (newton.cu describes the problem).
#include <atomic>
#include "newton_dev.cuh"

namespace mth {

constexpr int F64_NT = 64;   // threads of the largest block
using FCol = Column<float, F64_NT>;
using DCol = Column<double, F64_NT>;

// ---- FP64 mode
// GB300 issues FP64 at 1/64 of the FP32 rate, so what bounds a solve is the
// count of its FP64 instructions.  The iteration therefore starts in FP32
// (solve_f32, to a step below 1e-4 |lambda|) and ends on the FP64 residual:
// each of the last steps evaluates rates and residual in FP64 at the FP64
// iterate and takes the step from an FP32 Jacobian, which multiplies the
// error by about 1e-5 (the Jacobian's own error), so one step takes the 1e-6
// of the start to 1e-11 and the second to rounding.  A solve ends when its
// step meets the tolerance (the reference's criterion, src/evolution.c:
// 264-270) and the step after it, estimated by the last two steps' ratio,
// would be below 4e-16 |lambda|; the rates at the accepted iterate are the
// last evaluation's plus the Jacobian times the last step (error of order
// the step squared).  A start that fails, a step above 1e-2 |lambda|, or no
// end within eight steps falls back to the damped FP64 iteration from
// lambda (solve_full), which tight iteration caps use from the start.
// What bounds it is still the FP64 pipe, with about 800 FP64 warp
// instructions a solve instead of about 6700: 128^3, 3.5 ms per launch
// against 24.0 with every pass in FP64, the same fields to 1e-15; the array
// solve of 100 003 points 0.31 against 4.2 ms.

// what the fallback reads and returns
struct FullIo {
  double lam[6], eps[6], ep[6], R[9], slip[3 * NSYS], et[ETAB_W];
  double s6[6], e6[6], conv_s, conv_e;
  int iters, failed;
};
template <int LAW>
__device__ __noinline__ void solve_full(const NewtonConst& nc, const PhaseConst& ph, FullIo& io) {
  auto load = [&](double* l, double* e, double* q, double* r, bool) {
    for (int i = 0; i < 6; i++) { l[i] = io.lam[i]; e[i] = io.eps[i]; q[i] = io.ep[i]; }
    for (int i = 0; i < 9; i++) r[i] = io.R[i];
  };
  VoxelOut<double> o;
  if constexpr (LAW == 0) {
    PlSlip<double> sl;
    for (int s = 0; s < NSYS; s++) sl.tauf[s] = io.slip[s];
    sl.tau_off = ph.tau_back_minus_fwd;
    o = solve_voxel<double, double, false>(nc, ph, io.et, sl, load, io.s6, io.e6);
  } else {
    DdSlip<double> sl;
    for (int s = 0; s < NSYS; s++) {
      sl.tp[s] = io.slip[s];
      sl.td[s] = io.slip[NSYS + s];
      sl.g0[s] = io.slip[2 * NSYS + s];
    }
    o = solve_voxel<double, double, false>(nc, ph, io.et, sl, load, io.s6, io.e6);
  }
  io.conv_s = o.conv_s;
  io.conv_e = o.conv_e;
  io.iters = o.iters;
  io.failed = o.failed;
}

// what rcp_f64 takes: positive, normal, with a normal reciprocal
__device__ __forceinline__ bool rcp_ok(double t) {
  return (unsigned)__double2hiint(t) - 0x00100000u < 0x7fd00000u - 0x00100000u;
}
// 1/t: pivot_rcp_nr, which reads no sign, and a residual correction
__device__ __forceinline__ double rcp_f64(double t) {
  const double x = pivot_rcp_nr<false>(t);
  return fma(x, fma(-t, x, 1.0), x);
}

// rows of doubles in a thread's column, after the FP32 ones
constexpr int LD_Q = 0, LD_TAU = 25;
template <int LAW, bool GEN>
__host__ __device__ constexpr int ld_rows() { return LD_TAU + (LAW == 1 ? 0 : GEN ? 2 * NSYS : NSYS); }
template <int LAW, bool GEN>
constexpr size_t f64_smem() {
  constexpr size_t b = (size_t)F64_NT * (4 * ls_rows<LAW, GEN>() + 8 * ld_rows<LAW, GEN>());
  static_assert(b <= 47 * 1024, "no opt-in to more than 48 KB of shared memory is made");
  return b;
}

// rates (crystal axes) at x in FP64
template <int LAW, bool GEN, typename IO>
__device__ __forceinline__ void rates_f64(const PhaseConst& ph, const SlipF& pf, const IO& io, const DCol& dcol,
                                          const double (&x)[5], double (&ed)[5]) {
#pragma unroll
  for (int i = 0; i < 5; i++) ed[i] = 0.0;
  if constexpr (LAW == 0) {
    double r[NSYS], b[NSYS], p[NSYS];
#pragma unroll
    for (int s = 0; s < NSYS; s++) {
      const double* m = ph.m_xt[s];
      const double rss = m[0] * x[0] + m[1] * x[1] + m[2] * x[2] + m[3] * x[3] + m[4] * x[4];
      double t = dcol(LD_TAU + s);
      if (GEN && __double2hiint(rss) < 0) t = dcol(LD_TAU + NSYS + s);
      r[s] = rss * t;
      b[s] = fabs(r[s]);
    }
    pow_systems<double, GEN>(b, p, pf.nm1, pf.half, ph.nrs - 1.0);
#pragma unroll
    for (int s = 0; s < NSYS; s++) {
      const double g = (ph.gamd0 * p[s]) * r[s];   // |r|^(n-1) r
#pragma unroll
      for (int i = 0; i < 5; i++) ed[i] += ph.m_xt[s][i] * g;
    }
  } else {
#pragma unroll 1
    for (int s = 0; s < NSYS; s++) {
      const double* m = ph.m_xt[s];
      const double rss = m[0] * x[0] + m[1] * x[1] + m[2] * x[2] + m[3] * x[3] + m[4] * x[4];
      const double q = fabs(rss) - io.slip(s);
      if (q > 0.0) {
        const double g = copysign(io.slip(2 * NSYS + s) * sinh(q / io.slip(NSYS + s)), rss);
#pragma unroll
        for (int i = 0; i < 5; i++) ed[i] += m[i] * g;
      }
    }
  }
}

// A number as the unevaluated sum h + l of two FP32 numbers, two at a time
struct F2x2 {
  float2 h, l;
};
// (s, c) += (a + al) (b + bl): the rounding errors of the leading product and of
// the sum are kept in c
__device__ __forceinline__ void acc2(F2x2& s, float2 a, float2 al, float2 b, float2 bl) {
  const float2 m1 = make_float2(-1.0f, -1.0f);
  const float2 p = mul2(a, b), t = add2(s.h, p), z = fma2(s.h, m1, t);
  float2 e = fma2(a, b, mul2(p, m1));   // a b - p
  e = fma2(a, bl, e);
  e = fma2(al, b, e);
  const float2 v = fma2(fma2(z, m1, t), m1, s.h), q = fma2(z, m1, p);
  s.l = add2(s.l, add2(add2(v, q), e));
  s.h = t;
}
__device__ __forceinline__ F2x2 mul2x2(const F2x2& a, const F2x2& b) {
  F2x2 o;
  o.h = mul2(a.h, b.h);
  o.l = fma2(a.h, b.h, mul2(o.h, make_float2(-1.0f, -1.0f)));
  o.l = fma2(a.h, b.l, o.l);
  o.l = fma2(a.l, b.h, o.l);
  return o;
}
// The power law's rates (crystal axes) at an FP32 x to about 1e-13, in pairs of
// FP32 numbers: the first of the last steps only has to reach 1e-11, and FP64
// rates are 204 of the 990 instructions that bound a solve.  Whole and half
// exponents, one CRSS per system.  One pair of systems at a time: 128^3 3.5 ms
// per launch, 3.6 / 3.7 with two / all pairs unrolled (spills), 4.0 with FP64
// rates; 48^3 0.19 and 0.22 ms, 32^3 67 and 74 us.
// The result is the FP64 step's after it: against a solve in FP64 throughout the
// stress is off by 6 to 9e-16 (16^3), 1.0 to 1.7e-15 (32^3), 5.5e-16 (128^3),
// with FP64 rates here 6 to 9e-16, 1.0 to 1.8e-15, 5.3e-16.
__device__ __forceinline__ void rates_2xf32(const SlipF& pf, const DCol& dcol, double gamd0, const float (&x)[5],
                                            double (&ed)[5]) {
  const float2 zero = dup2(0.0f), m1 = make_float2(-1.0f, -1.0f);
  F2x2 a[5];
#pragma unroll
  for (int i = 0; i < 5; i++) a[i] = F2x2{zero, zero};
#pragma unroll 1
  for (int s = 0; s < NSYS / 2; s++) {
    F2x2 r{zero, zero}, b, p, it;
#pragma unroll
    for (int i = 0; i < 5; i++) acc2(r, pf.m[s][i], pf.ml[s][i], dup2(x[i]), zero);
    const double t0 = dcol(LD_TAU + 2 * s), t1 = dcol(LD_TAU + 2 * s + 1);
    it.h = make_float2(f64_to_f32(t0), f64_to_f32(t1));
    it.l = make_float2(f64_to_f32(t0 - f32_to_f64(it.h.x)), f64_to_f32(t1 - f32_to_f64(it.h.y)));
    const float2 n = add2(r.h, r.l);
    r.l = fma2(fma2(r.h, m1, n), m1, r.l);   // l - (n - h)
    r.h = n;
    b = r = mul2x2(r, it);
    int e = pf.nm1;
    while (!(e & 1)) {
      b = mul2x2(b, b);
      e >>= 1;
    }
    p = b;
    while (e >>= 1) {
      b = mul2x2(b, b);
      if (e & 1) p = mul2x2(p, b);
    }
    if (pf.half) {   // times sqrt |r|
      b.h = make_float2(sqrtf(fabsf(r.h.x)), sqrtf(fabsf(r.h.y)));
      auto low = [](float h, float l, float q) {
        return h != 0.0f ? (fmaf(-q, q, fabsf(h)) + copysignf(1.0f, h) * l) / (2.0f * q) : 0.0f;
      };
      b.l = make_float2(low(r.h.x, r.l.x, b.h.x), low(r.h.y, r.l.y, b.h.y));
      p = mul2x2(p, b);
    }
    // |r|^(n-1) r
    p.l = make_float2(p.h.x < 0.0f ? -p.l.x : p.l.x, p.h.y < 0.0f ? -p.l.y : p.l.y);
    p.h = make_float2(fabsf(p.h.x), fabsf(p.h.y));
    r = mul2x2(p, r);
#pragma unroll
    for (int i = 0; i < 5; i++) acc2(a[i], pf.m[s][i], pf.ml[s][i], r.h, r.l);
  }
#pragma unroll
  for (int i = 0; i < 5; i++)
    ed[i] = gamd0 * ((f32_to_f64(a[i].h.x) + f32_to_f64(a[i].h.y)) + (f32_to_f64(a[i].l.x) + f32_to_f64(a[i].l.y)));
}

// One voxel in FP64.  io: load(lam, eps, ep, R), slip(row), stot(v, out)
// (S0 + S_gr), sel(v, out) (S_gr), s_packed(S) (S0 + S_gr in FP32), shh(),
// mu(), full(FullIo&) (class row for the fallback).
struct OutF64 {
  double s6[6], e6[6], conv_s, conv_e;
  int iters, failed;
};
template <int LAW, bool GEN, typename IO>
__device__ __forceinline__ void solve_f64(const NewtonConst& nc, const LocalConst& lc, const PhaseConst& ph,
                                          const SlipF& pf, IO& io, const FCol& col, const DCol& dcol, OutF64& out) {
  double x[5], c[5], ed[5], h, dh;
  float ref2;
  bool ok = nc.itmax >= 50;
  int it = 0;
  if (ok) {
    float xf[5], edf[5];
    {
      double lam[6], u[6];
      {
        double ep[6], R[9], Q[25];
        io.load(lam, u, ep, R);
#pragma unroll
        for (int i = 0; i < 6; i++) u[i] = ep[i] - u[i];
        rot_to_q_dev<double>(R, Q);
#pragma unroll
        for (int i = 0; i < 25; i++) dcol(LD_Q + i) = Q[i];
        float Rf[9], Qf[25], S[15];
#pragma unroll
        for (int i = 0; i < 9; i++) Rf[i] = f64_to_f32(R[i]);
        rot_to_q_dev<float>(Rf, Qf);
        io.s_packed(lc, pf, Qf, S);
        store_k(Qf, S, col);
      }
      h = (nc.s0hh * lam[5] - u[5]) / (nc.s0hh + io.shh());
      dh = h - lam[5];
#pragma unroll
      for (int i = 0; i < 5; i++) {
        double a = u[i];
#pragma unroll
        for (int j = 0; j < 5; j++) a -= nc.s0dev[i * 5 + j] * lam[j];
        x[i] = a;
      }
      ref2 = 0;
#pragma unroll
      for (int i = 0; i < 6; i++) {
        const float l = f64_to_f32(lam[i]);
        ref2 = fmaf(l, l, ref2);
      }
#pragma unroll
      for (int i = 0; i < 5; i++) {
        double a = 0, b = 0;
#pragma unroll
        for (int j = 0; j < 5; j++) {
          const double q = dcol(LD_Q + i * 5 + j);
          a += q * lam[j];
          b += q * x[j];
        }
        xf[i] = f64_to_f32(a);
        c[i] = b;
        col(LS_C + i) = f64_to_f32(b);
      }
    }
    if constexpr (LAW == 0) {
#pragma unroll
      for (int s = 0; s < NSYS; s++) {
        const double t = io.slip(s);
        const bool on = rcp_ok(t);
        ok = ok && (on || s >= ph.nsys);   // a CRSS that is not positive: every pass in FP64
        const double ti = on ? rcp_f64(t) : 0.0;
        dcol(LD_TAU + s) = ti;
        col(LS_LAW + s) = f64_to_f32(ti);
        if (GEN) {
          const double tbk = t + ph.tau_back_minus_fwd;
          const bool onb = on && rcp_ok(tbk);
          ok = ok && (onb || s >= ph.nsys);   // the backward one too
          const double tb = onb ? rcp_f64(tbk) : 0.0;
          dcol(LD_TAU + NSYS + s) = tb;
          col(LS_LAW + NSYS + s) = f64_to_f32(tb);
        }
      }
    } else {
#pragma unroll 4
      for (int s = 0; s < 3 * NSYS; s++) col(LS_LAW + s) = f64_to_f32(io.slip(s));
    }
    const SolveF32 o = solve_f32<LS_FAST, LAW, GEN, true>(lc, pf, col, 0.0f, ref2, f64_to_f32(h), f64_to_f32(dh),
                                                          xf, edf);
    it = o.it;
    ok = ok && !o.failed;
#pragma unroll
    for (int i = 0; i < 5; i++) x[i] = f32_to_f64(xf[i]);
  }
  if (ok) {
    const float tol = lc.tol64;
    const float dt = lc.dt;
    bool done = false;
    float prev = 0;
    for (int k = 0; k < 8 && !done; k++) {
      if (nc.flow_off) {
#pragma unroll
        for (int i = 0; i < 5; i++) ed[i] = 0.0;
      } else if (LAW == 0 && !GEN && k == 0) {
        float xs[5];
#pragma unroll
        for (int i = 0; i < 5; i++) xs[i] = f64_to_f32(x[i]);   // exact: x is the FP32 start
        rates_2xf32(pf, dcol, ph.gamd0, xs, ed);
      } else {
        rates_f64<LAW, GEN, IO>(ph, pf, io, dcol, x, ed);
      }
      float rf[5], xf[5];
      {
        double t[5], u[5];
#pragma unroll
        for (int j = 0; j < 5; j++) {
          double a = 0;
#pragma unroll
          for (int i = 0; i < 5; i++) a += dcol(LD_Q + i * 5 + j) * x[i];
          t[j] = a;
        }
        io.stot(nc, ph, t, u, dcol);
#pragma unroll
        for (int i = 0; i < 5; i++) {
          double a = c[i] + nc.dt * ed[i];
#pragma unroll
          for (int j = 0; j < 5; j++) a += dcol(LD_Q + i * 5 + j) * u[j];
          rf[i] = -f64_to_f32(a);
          xf[i] = f64_to_f32(x[i]);
        }
      }
      float w[NSYS], p[5], edf[5], psi;
      if (lc.flow_off) {
#pragma unroll
        for (int s = 0; s < NSYS; s++) w[s] = 0;
      } else {
        flow_f32<LAW, GEN>(pf, col, xf, edf, psi, w);
      }
      {
        float H[15];
        Ldl5 f;
        hessian_f32<LAW, GEN>(pf, col, w, dt, H);
        ok = ldl5_factor(H, f);
        ldl5_apply(f, rf, p);
      }
      float s2 = 0, den2 = ref2;
#pragma unroll
      for (int i = 0; i < 5; i++) {
        s2 = fmaf(p[i], p[i], s2);
        x[i] += f32_to_f64(p[i]);
      }
      if (!(den2 > 0.0f)) {
        const float hf = f64_to_f32(h);
        den2 = hf * hf;
#pragma unroll
        for (int i = 0; i < 5; i++) den2 = fmaf(xf[i], xf[i], den2);
      }
      it++;
      ok = ok && s2 <= 1e-4f * den2;
      if (!ok || it > nc.itmax) {
        ok = false;
        break;
      }
      const float step = sqrtf(s2), den = sqrtf(den2);
      if (k == 0) prev = step;
      done = step <= tol * den && step * step <= 4e-16f * den * prev;
      prev = step;
      if (done) {
        // rates at the accepted iterate: + sum_s w_s m_s (m_s . p)
        float2 g[NSYS / 2];
        resolved2(pf, p, g);
        const float sc = LAW == 0 ? pf.gn : 1.0f;
#pragma unroll
        for (int s = 0; s < NSYS; s++) at2(g[s / 2], s & 1) *= w[s] * sc;
        rates2(pf, g, edf);
#pragma unroll
        for (int i = 0; i < 5; i++) ed[i] += f32_to_f64(edf[i]);
      }
    }
    ok = ok && done;
  }
  if (!ok) {
    FullIo fi;
    io.load(fi.lam, fi.eps, fi.ep, fi.R);
    io.full(nc, ph, fi);
    solve_full<LAW>(nc, ph, fi);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      out.s6[i] = fi.s6[i];
      out.e6[i] = fi.e6[i];
    }
    out.conv_s = fi.conv_s;
    out.conv_e = fi.conv_e;
    out.iters = fi.iters;
    out.failed = fi.failed;
    return;
  }
#pragma unroll
  for (int j = 0; j < 5; j++) {
    double a = 0, b = 0;
#pragma unroll
    for (int i = 0; i < 5; i++) {
      const double q = dcol(LD_Q + i * 5 + j);
      a += q * x[i];
      b += q * ed[i];
    }
    out.s6[j] = a;
    out.e6[j] = b;
  }
  out.s6[5] = h;
  out.e6[5] = 0.0;
  double lam[6], u[6], cs, ce;
  {
    double ep[6], R[9];
    io.load(lam, u, ep, R);
#pragma unroll
    for (int i = 0; i < 6; i++) u[i] = ep[i] - u[i];
  }
  cs = dh * dh;
  {
    const double de = u[5] + io.shh() * h;
    ce = de * de;
  }
  double se[5], sv[5];
#pragma unroll
  for (int i = 0; i < 5; i++) sv[i] = out.s6[i];
  io.sel(nc, ph, sv, se, dcol);
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const double ds = out.s6[i] - lam[i];
    cs += ds * ds;
    const double de = u[i] + nc.dt * out.e6[i] + se[i];
    ce += de * de;
  }
  out.conv_s = sqrt(cs);
  out.conv_e = sqrt(ce);
  out.iters = it;
  out.failed = 0;
}

// y = A v, A packed symmetric
__device__ __forceinline__ void symv5_packed(const double* __restrict__ A, const double (&v)[5], double (&y)[5]) {
#pragma unroll
  for (int i = 0; i < 5; i++) {
    double a = 0;
#pragma unroll
    for (int j = 0; j < 5; j++) a += A[pk5s(i, j)] * v[j];
    y[i] = a;
  }
}

// a voxel of the volume's fields
template <int LAW>
struct FieldIo {
  const Fields<double>& f;
  long long v;
  const double* et;
  const float* etf;
  __device__ __forceinline__ void load(double (&l)[6], double (&e)[6], double (&q)[6], double (&R)[9]) const {
    const long long P = f.nv;
#pragma unroll
    for (int i = 0; i < 6; i++) {
      l[i] = ld_again(f.sig + i * P + v);
      e[i] = ld_again(f.strain + i * P + v);
      q[i] = ld_again(f.epsp + i * P + v);
    }
#pragma unroll
    for (int i = 0; i < 9; i++) R[i] = ld_again(f.rot + i * P + v);
  }
  __device__ __forceinline__ double slip(int s) const { return (LAW ? f.ddc : f.crss)[s * f.nv + v]; }
  __device__ __forceinline__ double shh() const { return et[ET_SEL_HH]; }
  __device__ __forceinline__ void s_packed(const LocalConst&, const SlipF&, const float (&)[25], float (&S)[15]) const {
#pragma unroll
    for (int i = 0; i < 15; i++) S[i] = etf[ET_STOT + i];
  }
  __device__ __forceinline__ void stot(const NewtonConst&, const PhaseConst&, const double (&t)[5], double (&u)[5],
                                       const DCol&) const {
    symv5_packed(et + ET_STOT, t, u);
  }
  __device__ __forceinline__ void sel(const NewtonConst&, const PhaseConst&, const double (&t)[5], double (&u)[5],
                                      const DCol&) const {
    symv5_packed(et + ET_SEL, t, u);
  }
  __device__ __forceinline__ void full(const NewtonConst&, const PhaseConst& ph, FullIo& o) const {
    for (int s = 0; s < (LAW ? 3 * NSYS : NSYS); s++) o.slip[s] = LAW || s < ph.nsys ? slip(s) : 1.0;
    for (int i = 0; i < ETAB_W; i++) o.et[i] = et[i];
  }
};

template <int LAW, bool GEN>
__global__ void __launch_bounds__(F64_NT, 6) newton_f64_kernel(const __grid_constant__ NewtonConst nc,
                                                              const __grid_constant__ LocalConst lc,
                                                              const __grid_constant__ Fields<double> f,
                                                              double* __restrict__ partials, IterIn it) {
  if (!is_live(it)) return;
  extern __shared__ __align__(16) float ls_sm[];
  const FCol col{ls_sm + threadIdx.x};
  const DCol dcol{reinterpret_cast<double*>(ls_sm + F64_NT * ls_rows<LAW, GEN>()) + threadIdx.x};
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = f.nv;
  double acc[NPART];
#pragma unroll
  for (int i = 0; i < NPART; i++) acc[i] = 0.0;
  if (v < P) {
    const int jph = f.phase[v];
    const PhaseConst& ph = nc.ph[GEN ? jph : 0];
    if (GEN ? ph.type == 0 : jph == 0) {
      const size_t row = (size_t)f.eclass[v] * ETAB_W;
      FieldIo<LAW> io{f, v, f.etab + row, f.etabf + row};
      OutF64 o;
      solve_f64<LAW, GEN>(nc, lc, ph, lc.ph[GEN ? jph : 0], io, col, dcol, o);
#pragma unroll
      for (int i = 0; i < 6; i++) {
        f.sig[i * P + v] = o.s6[i];
        f.edot[i * P + v] = o.e6[i];
        acc[2 + i] = o.s6[i];
        if (GEN && jph == 0) acc[8 + i] = o.s6[i];
      }
      acc[0] = o.conv_s;
      acc[1] = o.conv_e;
      acc[14] = (double)o.iters;
      acc[15] = (double)o.failed;
    } else {
#pragma unroll
      for (int i = 0; i < 6; i++) {
        f.sig[i * P + v] = 0.0;
        f.edot[i * P + v] = 0.0;
      }
    }
  }
  newton_block_sums<double, GEN, F64_NT>(acc, dcol, partials);
}


template <int LAW, bool GEN>
static cudaError_t launch_f64(const NewtonConst& nc, const LocalConst& lc, const Fields<double>& f, double* partials,
                              const IterIn& it, cudaStream_t st) {
  return launch_chain(newton_f64_kernel<LAW, GEN>, dim3(newton_blocks(f.nv, true)), dim3(newton_threads(f.nv, true)),
                      f64_smem<LAW, GEN>(), st, it.pdl, nc, lc, f, partials, it);
}

cudaError_t launch_newton_f64(const NewtonConst& nc_in, const Fields<double>& f, double* partials, const IterIn& it,
                              cudaStream_t st, int law) {
  LocalConst lc;
  fill_local(nc_in, true, lc);
  NewtonConst nc = nc_in;
  fill_float_consts(nc);
  if (law == 1)
    return nc.ph1_only ? launch_f64<1, false>(nc, lc, f, partials, it, st)
                       : launch_f64<1, true>(nc, lc, f, partials, it, st);
  return plain_phase(nc, lc) ? launch_f64<0, false>(nc, lc, f, partials, it, st)
                             : launch_f64<0, true>(nc, lc, f, partials, it, st);
}

// --------------------------------------------------------- batch local solve
// a point of voxel-major FP64 arrays whose elastic axes are its current
// ones: S_gr = Q^T diag(s) Q, formed where it is applied
struct ArrayIo {
  const double *sig, *epsp, *strain, *rot, *crss;
  const PhaseConst& ph;
  long long v;
  __device__ __forceinline__ void load(double (&l)[6], double (&e)[6], double (&q)[6], double (&R)[9]) const {
#pragma unroll
    for (int i = 0; i < 6; i++) {
      l[i] = ld_again(sig + 6 * v + i);
      e[i] = ld_again(strain + 6 * v + i);
      q[i] = ld_again(epsp + 6 * v + i);
    }
#pragma unroll
    for (int i = 0; i < 9; i++) R[i] = ld_again(rot + 9 * v + i);
  }
  __device__ __forceinline__ double slip(int s) const { return s < ph.nsys ? crss[NSYS * v + s] : 0.0; }
  __device__ __forceinline__ double shh() const { return ph.s_xt[5]; }
  __device__ __forceinline__ void s_packed(const LocalConst& lc, const SlipF&, const float (&Q)[25],
                                           float (&S)[15]) const {
    float s[5];
#pragma unroll
    for (int k = 0; k < 5; k++) s[k] = lc.s_xt[k];
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = i; j < 5; j++) {
        float a = lc.s0[i * 5 + j];
#pragma unroll
        for (int k = 0; k < 5; k++) a = fmaf(Q[k * 5 + i] * s[k], Q[k * 5 + j], a);
        S[pk5u(i, j)] = a;
      }
  }
  __device__ __forceinline__ void sel(const NewtonConst&, const PhaseConst&, const double (&t)[5], double (&u)[5],
                                      const DCol& dcol) const {
    double y[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
      double a = 0;
#pragma unroll
      for (int j = 0; j < 5; j++) a += dcol(LD_Q + k * 5 + j) * t[j];
      y[k] = a * ph.s_xt[k];
    }
#pragma unroll
    for (int j = 0; j < 5; j++) {
      double a = 0;
#pragma unroll
      for (int k = 0; k < 5; k++) a += dcol(LD_Q + k * 5 + j) * y[k];
      u[j] = a;
    }
  }
  __device__ __forceinline__ void stot(const NewtonConst& nc, const PhaseConst& p, const double (&t)[5],
                                       double (&u)[5], const DCol& dcol) const {
    sel(nc, p, t, u, dcol);
#pragma unroll
    for (int i = 0; i < 5; i++)
#pragma unroll
      for (int j = 0; j < 5; j++) u[i] += nc.s0dev[i * 5 + j] * t[j];
  }
  __device__ __forceinline__ void full(const NewtonConst& nc, const PhaseConst&, FullIo& o) const {
    double Q[25];
    rot_to_q<double>(o.R, Q);
    for (int s = 0; s < NSYS; s++) o.slip[s] = s < ph.nsys ? slip(s) : 1.0;
    for (int i = 0; i < 5; i++)
      for (int j = i; j < 5; j++) {
        double sg = 0;
        for (int k = 0; k < 5; k++) sg += Q[k * 5 + i] * ph.s_xt[k] * Q[k * 5 + j];
        o.et[ET_SEL + pk(i, j)] = sg;
        o.et[ET_STOT + pk(i, j)] = nc.s0dev[i * 5 + j] + sg;
      }
    o.et[ET_SEL_HH] = ph.s_xt[5];
  }
};

// one thread per point; block_iters receives each block's Newton steps
template <bool GEN>
__global__ void __launch_bounds__(F64_NT, 6) local_solve_kernel(const __grid_constant__ NewtonConst nc,
                                                               const __grid_constant__ LocalConst lc, long long n,
                                                               double* sig, const double* __restrict__ epsp,
                                                               const double* __restrict__ strain,
                                                               const double* __restrict__ rot,
                                                               const double* __restrict__ crss,
                                                               double* __restrict__ edot, double* __restrict__ err,
                                                               double* __restrict__ block_iters) {
  extern __shared__ __align__(16) float ls_sm[];
  __shared__ int steps[F64_NT / 32];
  const FCol col{ls_sm + threadIdx.x};
  const DCol dcol{reinterpret_cast<double*>(ls_sm + F64_NT * ls_rows<0, GEN>()) + threadIdx.x};
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int it = 0;
  if (v < n) {
    ArrayIo io{sig, epsp, strain, rot, crss, nc.ph[0], v};
    OutF64 o;
    solve_f64<0, GEN>(nc, lc, nc.ph[0], lc.ph[0], io, col, dcol, o);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      sig[6 * v + i] = o.s6[i];
      edot[6 * v + i] = o.e6[i];
    }
    err[2 * v] = o.conv_s;
    err[2 * v + 1] = o.conv_e;
    it = o.iters;
  }
  it = __reduce_add_sync(0xffffffffu, it);
  if ((threadIdx.x & 31) == 0) steps[threadIdx.x >> 5] = it;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long t = 0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += steps[k];
    block_iters[blockIdx.x] = (double)t;
  }
}

int local_solve_blocks(long long n) { return newton_blocks(n, true); }

cudaError_t launch_local_solve(const NewtonConst& nc, long long n, double* sig, const double* epsp,
                               const double* strain, const double* rot, const double* crss, double* edot, double* err,
                               double* block_iters, cudaStream_t st) {
  LocalConst lc;
  fill_local(nc, true, lc);
  for (int k = 0; k < 5; k++) lc.s_xt[k] = (float)nc.ph[0].s_xt[k];
  const int nb = newton_blocks(n, true), nt = newton_threads(n, true);
  if (nc.ph[0].tau_back_minus_fwd == 0.0 && lc.ph[0].nm1 > 0) {
    local_solve_kernel<false><<<nb, nt, f64_smem<0, false>(), st>>>(nc, lc, n, sig, epsp, strain, rot, crss, edot, err,
                                                                    block_iters);
  } else {
    local_solve_kernel<true><<<nb, nt, f64_smem<0, true>(), st>>>(nc, lc, n, sig, epsp, strain, rot, crss, edot, err,
                                                                  block_iters);
  }
  return cudaGetLastError();
}

// ------------------------------------------------ allocation-free local solve
// local_solve_kernel for callers that cannot allocate device memory: the
// caller passes device pointers for every input and output, and the only
// scratch (each block's Newton steps and their total) lives in the fixed
// array below, which every GPU that loads the library holds until the
// process exits.  Calls that overlap on the GPU share it and race.
namespace {
constexpr long long NOALLOC_MAX_VOXELS = 1LL << 20;
constexpr int NOALLOC_MAX_BLOCKS = (int)(NOALLOC_MAX_VOXELS / F64_NT);   // smaller blocks only below 2^17 points
static __device__ __align__(256) double g_noalloc_scratch[NOALLOC_MAX_BLOCKS + 1];

__global__ void noalloc_total_kernel(double* scratch, int nblocks) {
  __shared__ double sm[256];
  double a = 0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) a += scratch[b];
  sm[threadIdx.x] = a;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sm[threadIdx.x] += sm[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) scratch[NOALLOC_MAX_BLOCKS] = sm[0];
}

// Device address of g_noalloc_scratch, looked up once per device with that
// device current (the host-side name is only a stand-in, not a device
// address).  Atomic slots: host threads that make their first calls on the
// same device at the same time both look the address up and store the same
// value.
constexpr int NOALLOC_MAX_DEVICES = 64;
std::atomic<double*> g_noalloc_ptr[NOALLOC_MAX_DEVICES];
}  // namespace

long long noalloc_max_voxels() { return NOALLOC_MAX_VOXELS; }

cudaError_t launch_local_solve_noalloc(const NewtonConst& nc, long long n, double* sig, const double* epsp,
                                       const double* strain, const double* rot, const double* crss, double* edot,
                                       double* err, long long* iters_host, cudaStream_t st) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return cudaErrorInvalidDevice;
  double* scratch = g_noalloc_ptr[dev].load(std::memory_order_acquire);
  if (!scratch) {
    e = cudaGetSymbolAddress((void**)&scratch, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_noalloc_ptr[dev].store(scratch, std::memory_order_release);
  }
  const int nb = newton_blocks(n, true);
  // the total slot is the only one read without being written first
  e = cudaMemsetAsync(scratch + NOALLOC_MAX_BLOCKS, 0, sizeof(double), st);
  if (e != cudaSuccess) return e;
  e = launch_local_solve(nc, n, sig, epsp, strain, rot, crss, edot, err, scratch, st);
  if (e != cudaSuccess) return e;
  noalloc_total_kernel<<<1, 256, 0, st>>>(scratch, nb);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  double tot = 0;
  e = cudaMemcpyAsync(&tot, scratch + NOALLOC_MAX_BLOCKS, sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  if (iters_host) *iters_host = (long long)tot;
  return cudaSuccess;
}

}  // namespace mth

