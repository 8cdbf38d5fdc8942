// green_op.cuh -- the Green operator at one wave vector, shared by the
// shared-memory and the TMA x passes.
#pragma once
#include "mth_common.cuh"
#include "mth_internal.h"

namespace mth {

// Frequency of index idx on an axis of n points: idx/n - round(idx/n) of
// src/init.c:778-786 (the Nyquist index maps to -1/2), from integers.
template <typename T> __device__ __forceinline__ T freq(int idx, int n) {
  const int k = (2 * idx >= n) ? idx - n : idx;
  return (T)k / (T)n;
}
template <typename T> struct GreenTab;   // the constants of GreenConst in precision T
template <> struct GreenTab<float> {
  __device__ __forceinline__ static float a(const GreenConst& gc, int p, int q) { return gc.af[p][q]; }
  __device__ __forceinline__ static float s066(const GreenConst& gc, int i) { return gc.s066f[i]; }
  __device__ __forceinline__ static float rn(const GreenConst& gc, int i) { return gc.rnf[i]; }
};
template <> struct GreenTab<double> {
  __device__ __forceinline__ static double a(const GreenConst& gc, int p, int q) { return gc.a[p][q]; }
  __device__ __forceinline__ static double s066(const GreenConst& gc, int i) { return gc.s066[i]; }
  __device__ __forceinline__ static double rn(const GreenConst& gc, int i) { return gc.rn[i]; }
};

// One direction's operator Delta = -Omega(f) (sigma f) (x) f, Omega = (C0 f f)^-1,
// which is of degree 0 in f: the wave vector needs no normalisation.
// Acoustic tensor A_p = sum_q a[p][q] f_j f_l over the six products
// (GreenConst::a holds the symmetrised C0), its cofactors K, 1/det folded
// into the weight: 3 + 6 + 36 + 12 + 3 operations and one division.
template <typename T>
struct GreenDir {
  T f[3], K[6], w;   // K: 00, 11, 22, 12, 02, 01
  __device__ __forceinline__ void set(const GreenConst& gc, const T (&dir)[3], T wgt) {
    T q[6], A[6];
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = dir[i];
    q[0] = f[0] * f[0];
    q[1] = f[1] * f[1];
    q[2] = f[2] * f[2];
    q[3] = f[1] * f[2];
    q[4] = f[0] * f[2];
    q[5] = f[0] * f[1];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      T t = GreenTab<T>::a(gc, p, 0) * q[0];
#pragma unroll
      for (int k = 1; k < 6; k++) t += GreenTab<T>::a(gc, p, k) * q[k];
      A[p] = t;
    }
    K[0] = A[1] * A[2] - A[3] * A[3];
    K[1] = A[0] * A[2] - A[4] * A[4];
    K[2] = A[0] * A[1] - A[5] * A[5];
    K[3] = A[4] * A[5] - A[0] * A[3];
    K[4] = A[5] * A[3] - A[1] * A[4];
    K[5] = A[4] * A[3] - A[2] * A[5];
    w = -wgt / (A[0] * K[0] + A[5] * K[5] + A[4] * K[4]);
  }
  // the same by two neighbouring lanes (part 0 and 1 of one wave vector), each
  // forming half of A and of its cofactors: 24 of the 134 FP64 operations a part
  // takes.  x + Gamma0 pass at 128^3 0.98 ms, 1.10 with both lanes forming all of
  // them; 48^3 81 and 89 us, 32^3 29 and 33 us, 16^3 17.5 and 19.1 us.
  __device__ __forceinline__ void set_pair(const GreenConst& gc, const T (&dir)[3], T wgt, int part) {
    const unsigned mask = 3u << (threadIdx.x & 30);
    auto join = [&](const T (&own)[3], T (&all)[6]) {
#pragma unroll
      for (int j = 0; j < 3; j++) {
        const T o = __shfl_xor_sync(mask, own[j], 1);
        all[j] = part ? o : own[j];
        all[3 + j] = part ? own[j] : o;
      }
    };
    T q[6], A[6], t[3];
#pragma unroll
    for (int i = 0; i < 3; i++) f[i] = dir[i];
    q[0] = f[0] * f[0];
    q[1] = f[1] * f[1];
    q[2] = f[2] * f[2];
    q[3] = f[1] * f[2];
    q[4] = f[0] * f[2];
    q[5] = f[0] * f[1];
#pragma unroll
    for (int j = 0; j < 3; j++) {
      t[j] = GreenTab<T>::a(gc, 3 * part + j, 0) * q[0];
#pragma unroll
      for (int k = 1; k < 6; k++) t[j] += GreenTab<T>::a(gc, 3 * part + j, k) * q[k];
    }
    join(t, A);
    t[0] = (part ? A[4] : A[1]) * (part ? A[5] : A[2]) - (part ? A[0] : A[3]) * A[3];
    t[1] = (part ? A[5] : A[0]) * (part ? A[3] : A[2]) - (part ? A[1] : A[4]) * A[4];
    t[2] = (part ? A[4] : A[0]) * (part ? A[3] : A[1]) - (part ? A[2] : A[5]) * A[5];
    join(t, K);
    w = -wgt / (A[0] * K[0] + A[5] * K[5] + A[4] * K[4]);
  }
  // real or imaginary parts: s LT components of sigma-hat; adds the LT
  // components of sym(Delta) to d and (21, 02, 10) of its antisymmetric part to a
  __device__ __forceinline__ void apply(const T (&s)[6], T (&d)[6], T (&a)[3]) const {
    const T r2 = (T)RSQ2, r3 = (T)RSQ3, r6 = (T)RSQ6;
    const T b = r3 * s[5] - r6 * s[1], e = r2 * s[0];
    const T s00 = b - e, s11 = b + e, s22 = r3 * s[5] + (T)2 * r6 * s[1];
    const T g0 = r2 * f[0], g1 = r2 * f[1], g2 = r2 * f[2];
    const T t0 = (s00 * f[0] + s[4] * g1 + s[3] * g2) * w;
    const T t1 = (s[4] * g0 + s11 * f[1] + s[2] * g2) * w;
    const T t2 = (s[3] * g0 + s[2] * g1 + s22 * f[2]) * w;
    const T v0 = K[0] * t0 + K[5] * t1 + K[4] * t2;
    const T v1 = K[5] * t0 + K[1] * t1 + K[3] * t2;
    const T v2 = K[4] * t0 + K[3] * t1 + K[2] * t2;
    const T d00 = v0 * f[0], d11 = v1 * f[1], d22 = v2 * f[2];
    const T tr = d00 + d11;
    d[0] += r2 * (d11 - d00);
    d[1] += r6 * ((T)2 * d22 - tr);
    d[2] += v1 * g2 + v2 * g1;
    d[3] += v0 * g2 + v2 * g0;
    d[4] += v0 * g1 + v1 * g0;
    d[5] += r3 * (tr + d22);
    const T h = (T)0.5;
    a[0] += h * (v2 * f[1] - v1 * f[2]);
    a[1] += h * (v0 * f[2] - v2 * f[0]);
    a[2] += h * (v1 * f[0] - v0 * f[1]);
  }
};

// The Green operator at one wave vector on NP parts (real and imaginary, or
// one of them: the operator is real, so the FP64 pass gives a vector's two
// parts to two threads).  sig[p]: LT components of sigma-hat's part (in),
// replaced by LT of sym(Delta); anti[p]: antisymmetric part of Delta.  When k
// has Nyquist components the operator is the mean of Gamma at n(k) and n(-k):
// the reference keeps only the real part of its complex inverse transform
// (src/evolution.c:1402), which equals the transform of the Hermitian part of
// Delta-hat.  Frequencies as src/init.c:778-786 (the Nyquist index maps to
// -1/2).  Per launch of the x + Gamma0 pass, before (normalised wave vector,
// 81 coefficients, one thread per vector) and now: FP64 16^3 44 and 17.5 us,
// 32^3 47 and 29 us, 128^3 1.29 and 0.98 ms (FP64 operations bound it);
// FP32 128^3 51 and 43 us.
// PAIR: the two parts are on neighbouring lanes of a warp, part says which one
// this is, and both lanes call.
template <typename T, int NP, bool PAIR = false>
__device__ __forceinline__ void green_point(const GreenConst& gc, int kx, int ky, int kz, int n0, int n1, int n2,
                                            T (&sig)[NP][6], T (&anti)[NP][3], int part = 0) {
  T dsym[NP][6];
#pragma unroll
  for (int p = 0; p < NP; p++) {
#pragma unroll
    for (int i = 0; i < 6; i++) dsym[p][i] = 0;
#pragma unroll
    for (int i = 0; i < 3; i++) anti[p][i] = 0;
  }
  if (kx == 0 && ky == 0 && kz == 0) {
    if (gc.elast_bc == 0) {
      for (int i = 0; i < 6; i++)
        for (int j = 0; j < 6; j++) {
          const T s = GreenTab<T>::s066(gc, i * 6 + j);
#pragma unroll
          for (int p = 0; p < NP; p++) dsym[p][i] -= s * sig[p][j];
        }
    }
  } else {
    const bool q0 = (2 * kx == n0), q1 = (2 * ky == n1), q2 = (2 * kz == n2);
    T f[3] = {(T)(2 * kx >= n0 ? kx - n0 : kx) * GreenTab<T>::rn(gc, 0),
              (T)(2 * ky >= n1 ? ky - n1 : ky) * GreenTab<T>::rn(gc, 1),
              (T)(2 * kz >= n2 ? kz - n2 : kz) * GreenTab<T>::rn(gc, 2)};
    const bool anyq = q0 || q1 || q2;
    const bool anyv = (!q0 && kx != 0) || (!q1 && ky != 0) || (!q2 && kz != 0);
    const int dirs = anyq && anyv ? 2 : 1;
    GreenDir<T> g;
#pragma unroll 1
    for (int m = 0; m < dirs; m++) {
      if (m) {
        f[0] = q0 ? f[0] : -f[0];
        f[1] = q1 ? f[1] : -f[1];
        f[2] = q2 ? f[2] : -f[2];
      }
      if constexpr (PAIR) g.set_pair(gc, f, dirs == 2 ? (T)0.5 : (T)1, part);
      else g.set(gc, f, dirs == 2 ? (T)0.5 : (T)1);
#pragma unroll
      for (int p = 0; p < NP; p++) g.apply(sig[p], dsym[p], anti[p]);
    }
  }
#pragma unroll
  for (int p = 0; p < NP; p++)
#pragma unroll
    for (int i = 0; i < 6; i++) sig[p][i] = dsym[p][i];
}

// The FP32 operator of the iterations in plain order (IterIn::plain): the wave
// vector normalised, A from the 81 coefficients, the full inverse.
// Delta = -Omega(n) (sig n) (x) n for one n; accumulates into dsym (LT, 6
// complex) and danti (3 complex: [2][1], [0][2], [1][0]) with weight wgt.
__device__ __forceinline__ void green_apply_plain(const GreenConst& gc, const float n[3], const float2 s[3][3], float wgt,
                                                  float2 dsym[6], float2 danti[3]) {
  using T = float;
  T A[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = i; k < 3; k++) {
      T a = 0;
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int l = 0; l < 3; l++) a += gc.c0f[((i * 3 + j) * 3 + k) * 3 + l] * n[j] * n[l];
      A[i][k] = a;
      A[k][i] = a;
    }
  T det = A[0][0] * (A[1][1] * A[2][2] - A[1][2] * A[2][1]) - A[0][1] * (A[1][0] * A[2][2] - A[1][2] * A[2][0]) +
          A[0][2] * (A[1][0] * A[2][1] - A[2][0] * A[1][1]);
  T id = (T)1 / det;
  T O[3][3];
  O[0][0] = (A[1][1] * A[2][2] - A[1][2] * A[2][1]) * id;
  O[0][1] = (A[0][2] * A[2][1] - A[0][1] * A[2][2]) * id;
  O[0][2] = (A[0][1] * A[1][2] - A[0][2] * A[1][1]) * id;
  O[1][0] = O[0][1];
  O[1][1] = (A[0][0] * A[2][2] - A[0][2] * A[2][0]) * id;
  O[1][2] = (A[0][2] * A[1][0] - A[0][0] * A[1][2]) * id;
  O[2][0] = O[0][2];
  O[2][1] = O[1][2];
  O[2][2] = (A[0][0] * A[1][1] - A[0][1] * A[1][0]) * id;
  c2<T> t[3], v[3];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    t[k] = mk<T>(s[k][0].x * n[0] + s[k][1].x * n[1] + s[k][2].x * n[2],
                 s[k][0].y * n[0] + s[k][1].y * n[1] + s[k][2].y * n[2]);
  }
#pragma unroll
  for (int i = 0; i < 3; i++)
    v[i] = mk<T>(-(O[i][0] * t[0].x + O[i][1] * t[1].x + O[i][2] * t[2].x) * wgt,
                 -(O[i][0] * t[0].y + O[i][1] * t[1].y + O[i][2] * t[2].y) * wgt);
  // Delta_ij = v_i n_j
  T r2 = (T)RSQ2, r3 = (T)RSQ3, r6 = (T)RSQ6;
  c2<T> d00 = cscale<T>(v[0], n[0]), d11 = cscale<T>(v[1], n[1]), d22 = cscale<T>(v[2], n[2]);
  c2<T> d12 = cscale<T>(v[1], n[2]), d21 = cscale<T>(v[2], n[1]);
  c2<T> d02 = cscale<T>(v[0], n[2]), d20 = cscale<T>(v[2], n[0]);
  c2<T> d01 = cscale<T>(v[0], n[1]), d10 = cscale<T>(v[1], n[0]);
  dsym[0] = cadd<T>(dsym[0], cscale<T>(csub<T>(d11, d00), r2));
  dsym[1] = cadd<T>(dsym[1], cscale<T>(csub<T>(cscale<T>(d22, (T)2), cadd<T>(d00, d11)), r6));
  dsym[2] = cadd<T>(dsym[2], cscale<T>(cadd<T>(d12, d21), r2));
  dsym[3] = cadd<T>(dsym[3], cscale<T>(cadd<T>(d02, d20), r2));
  dsym[4] = cadd<T>(dsym[4], cscale<T>(cadd<T>(d01, d10), r2));
  dsym[5] = cadd<T>(dsym[5], cscale<T>(cadd<T>(cadd<T>(d00, d11), d22), r3));
  danti[0] = cadd<T>(danti[0], cscale<T>(csub<T>(d21, d12), (T)0.5));
  danti[1] = cadd<T>(danti[1], cscale<T>(csub<T>(d02, d20), (T)0.5));
  danti[2] = cadd<T>(danti[2], cscale<T>(csub<T>(d10, d01), (T)0.5));
}

__device__ __forceinline__ void green_point_plain(const GreenConst& gc, int kx, int ky, int kz, int n0, int n1, int n2,
                                                  float (&sg)[2][6], float (&an)[2][3]) {
  using T = float;
  c2<T> sig[6], dsym[6], danti[3];
#pragma unroll
  for (int i = 0; i < 6; i++) sig[i] = mk<T>(sg[0][i], sg[1][i]);
#pragma unroll
  for (int i = 0; i < 6; i++) dsym[i] = mk<T>(0, 0);
#pragma unroll
  for (int i = 0; i < 3; i++) danti[i] = mk<T>(0, 0);
  if (kx == 0 && ky == 0 && kz == 0) {
    if (gc.elast_bc == 0) {
      for (int i = 0; i < 6; i++) {
        T re = 0, im = 0;
        for (int j = 0; j < 6; j++) {
          re -= gc.s066f[i * 6 + j] * sig[j].x;
          im -= gc.s066f[i * 6 + j] * sig[j].y;
        }
        dsym[i] = mk<T>(re, im);
      }
    }
  } else {
    c2<T> s[3][3];
    {
      T re[6], im[6], tr[3][3], ti[3][3];
#pragma unroll
      for (int i = 0; i < 6; i++) { re[i] = sig[i].x; im[i] = sig[i].y; }
      lt_to_cart<T>(re, tr);
      lt_to_cart<T>(im, ti);
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int j = 0; j < 3; j++) s[i][j] = mk<T>(tr[i][j], ti[i][j]);
    }
    T f[3] = {freq<T>(kx, n0), freq<T>(ky, n1), freq<T>(kz, n2)};
    const bool q0 = (2 * kx == n0), q1 = (2 * ky == n1), q2 = (2 * kz == n2);
    T nrm = sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
    T n[3] = {f[0] / nrm, f[1] / nrm, f[2] / nrm};
    const bool anyq = q0 || q1 || q2;
    const bool anyv = (!q0 && kx != 0) || (!q1 && ky != 0) || (!q2 && kz != 0);
    if (anyq && anyv) {
      green_apply_plain(gc, n, s, (T)0.5, dsym, danti);
      T m[3] = {q0 ? n[0] : -n[0], q1 ? n[1] : -n[1], q2 ? n[2] : -n[2]};
      green_apply_plain(gc, m, s, (T)0.5, dsym, danti);
    } else {
      green_apply_plain(gc, n, s, (T)1, dsym, danti);
    }
  }
#pragma unroll
  for (int i = 0; i < 6; i++) {
    sg[0][i] = dsym[i].x;
    sg[1][i] = dsym[i].y;
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    an[0][i] = danti[i].x;
    an[1][i] = danti[i].y;
  }
}

// the operator of the iteration's order (PLAIN: kernels of steps that may be in plain order)
template <typename T, bool PLAIN>
__device__ __forceinline__ void green_point_of(const GreenConst& gc, int kx, int ky, int kz, int n0, int n1, int n2,
                                               T (&sig)[2][6], T (&anti)[2][3], bool plain) {
  if constexpr (PLAIN) {
    if (plain) {
      green_point_plain(gc, kx, ky, kz, n0, n1, n2, sig, anti);
      return;
    }
  }
  green_point<T, 2>(gc, kx, ky, kz, n0, n1, n2, sig, anti);
}

}  // namespace mth
