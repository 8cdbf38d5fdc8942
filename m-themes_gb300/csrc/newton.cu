// newton.cu -- per-voxel kernels: the local stress solve of UpdateStress
// (src/evolution.c:44-310) with the power-law flow rule of StrainRate_eval
// (src/constitutive.c:5-67), the end-of-step updates (plastic strain,
// update_orient src/constitutive.c:196-273, harden src/constitutive.c:275-326)
// and the set-up of InitMicroStruct/InitFields (src/init.c:233-515).
//
// One thread per voxel, structure-of-arrays fields, coalesced loads.
//
// Local problem.  The reference solves, per voxel and in the 6-component
// Lebensohn-Tome basis, R(s) = s - lambda + C066 (S s + e_p + edot_p(s) dt - e)
// = 0 by Newton with a line search on |R|^2 (src/evolution.c:129-253).  Here
// the same root is found from the equivalent system S0 R = 0 (S0 = C066^-1),
// which is the gradient of the strictly convex potential
//   Phi(s) = 1/2 (s-lambda).S0.(s-lambda) + 1/2 s.S.s + (e_p - e).s + dt psi(s),
//   psi(s) = sum_a gamd0 tau_a |r_a|^(n+1) / (n+1),  r_a = m_a.s / tau_a,
// so Newton's direction is always a descent direction and the Hessian
// S0 + S + dt sum_a w_a m_a m_a^T is symmetric positive definite (Cholesky).
// The solve runs in crystal axes: there the cubic compliance S is diagonal and
// the Schmid tensors m_a are the constants of the .sx file, so no per-voxel
// Schmid field is stored (update_schmid, src/kinematics.c:430-463, becomes a
// 5x5 rotation of the stress).  The hydrostatic component decouples exactly
// for cubic crystals (edot_p has no trace, src/constitutive.c:50) and is
// solved in closed form.  Convergence: |step| <= tol |lambda|, as the
// reference's erral (src/evolution.c:264-270).
#include <cstdio>
#include <cmath>
#include "newton_dev.cuh"

namespace mth {

// ------------------------------------------------------------ Newton kernels
// Threads per block: 128 in FP32 and 64 in FP64, less where that would leave
// SMs without a block or with one block more than others (the solves are long
// and independent, so a small grid wants its warps spread: 16^3 voxels are 32
// blocks of 128 threads on 32 of the 152 SMs, or 128 blocks of 32).
int newton_threads(long long nv, bool fp64) {
  constexpr long long SMS = 152;
  if (fp64) return nv >= SMS * 32 * 16 ? 64 : 32;
  return nv >= SMS * 128 * 2 ? 128 : nv >= SMS * 64 * 2 ? 64 : 32;
}
int newton_blocks(long long nv, bool fp64) {
  const int nt = newton_threads(nv, fp64);
  return (int)((nv + nt - 1) / nt);
}

void fill_float_consts(NewtonConst& nc) {
  for (int k = 0; k < 2; k++) {
    PhaseConst& ph = nc.ph[k];
    ph.nrsf = (float)ph.nrs;
    ph.gamd0f = (float)ph.gamd0;
    ph.tau_offf = (float)ph.tau_back_minus_fwd;
    for (int s = 0; s < NSYS; s++) {
      for (int i = 0; i < 5; i++) ph.m_xtf[s][i] = (float)ph.m_xt[s][i];
      for (int i = 0; i < 3; i++) {
        ph.bnf[s][i] = (float)ph.bn[s][i];
        ph.bbf[s][i] = (float)ph.bb[s][i];
      }
      for (int j = 0; j < NSYS; j++) ph.hardf[s][j] = (float)ph.hard[s][j];
    }
    ph.tau0ff = (float)ph.tau0f;
    ph.tau1f = (float)ph.tau1;
    ph.thet0f = (float)ph.thet0;
    ph.thet1f = (float)ph.thet1;
  }
  for (int i = 0; i < 25; i++) nc.s0devf[i] = (float)nc.s0dev[i];
  nc.s0hhf = (float)nc.s0hh;
  nc.dtf = (float)nc.dt;
  nc.tolf = (float)nc.tol;
}

cudaError_t launch_newton(int mixed, const NewtonConst& nc, const void* fields, double* partials, const IterIn& it,
                          cudaStream_t st, int law) {
  if (mixed) return launch_newton_f32(mixed, nc, *static_cast<const Fields<float>*>(fields), partials, it, st, law);
  return launch_newton_f64(nc, *static_cast<const Fields<double>*>(fields), partials, it, st, law);
}

// ------------------------------------------------------- end-of-step kernel
// Eps += Edot dt (src/evolution.c:1500-1504), update_orient + Orientation
// (src/constitutive.c:142-273) and harden (src/constitutive.c:275-326).
// anti_u: uniform part of the lattice spin increment, (2,1),(0,2),(1,0)
// components of 2 Udot_a dt + antisym(sum dDisGradAvg).
template <typename TSt, typename TF, int LAW = 0>
__global__ void __launch_bounds__(256) end_step_kernel(const NewtonConst nc, Fields<TSt> f, double au0, double au1,
                                                       double au2, int do_orient, int do_harden,
                                                       double* __restrict__ partials) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = f.nv;
  TF acc[NPART_END];
#pragma unroll
  for (int i = 0; i < NPART_END; i++) acc[i] = (TF)0;
  if (v < P) {
    const int jph = f.phase[v];
    const PhaseConst& ph = nc.ph[jph];
    const TF dt = cpick<TF>(nc.dt, nc.dtf);
#pragma unroll
    for (int i = 0; i < 6; i++) {
      const TF ed = (TF)f.edot[i * P + v];
      const TF ep = (TF)f.epsp[i * P + v] + ed * dt;
      f.epsp[i * P + v] = (TSt)ep;
      acc[i] = ep;
      acc[6 + i] = ed;
    }
    if (ph.type == 0 && (do_orient || do_harden)) {
      TF R[9], Q[25], s6[6], x[5], gam[NSYS], ed[5], psi;
#pragma unroll
      for (int i = 0; i < 9; i++) R[i] = (TF)f.rot[i * P + v];
#pragma unroll
      for (int i = 0; i < 6; i++) s6[i] = (TF)f.sig[i * P + v];
      typename SlipOf<LAW, TF, TSt>::type slip;
      SlipOf<LAW, TF, TSt>::load(ph, f, v, slip);
      if constexpr (sizeof(TF) == 4) rot_to_q<TF>(R, Q);
      else rot_to_q_dev<TF>(R, Q);
#pragma unroll
      for (int i = 0; i < 5; i++) {
        TF a = 0;
#pragma unroll
        for (int j = 0; j < 5; j++) a += Q[i * 5 + j] * s6[j];
        x[i] = a;
      }
#pragma unroll
      for (int s = 0; s < NSYS; s++) gam[s] = 0;
      if (!nc.flow_off) slip.template flow<false>(ph, x, ed, nullptr, psi, gam);
      if (do_orient) {
        // plastic spin: RotSlip = -1/2 T sum_a gam_a (b_a x n_a)
        TF cx = 0, cy = 0, cz = 0;
#pragma unroll
        for (int s = 0; s < NSYS; s++) {
          if (s >= ph.nsys) break;
          const TF b0 = cpick<TF>(ph.bb[s][0], ph.bbf[s][0]), b1 = cpick<TF>(ph.bb[s][1], ph.bbf[s][1]),
                   b2 = cpick<TF>(ph.bb[s][2], ph.bbf[s][2]);
          const TF n0 = cpick<TF>(ph.bn[s][0], ph.bnf[s][0]), n1 = cpick<TF>(ph.bn[s][1], ph.bnf[s][1]),
                   n2 = cpick<TF>(ph.bn[s][2], ph.bnf[s][2]);
          cx += gam[s] * (b1 * n2 - b2 * n1);
          cy += gam[s] * (b2 * n0 - b0 * n2);
          cz += gam[s] * (b0 * n1 - b1 * n0);
        }
        TF ws[3];
#pragma unroll
        for (int i = 0; i < 3; i++) ws[i] = (TF)-0.5 * (R[i * 3 + 0] * cx + R[i * 3 + 1] * cy + R[i * 3 + 2] * cz);
        // Rot = (Udot_a + RotLoc - RotSlip) dt, as the vector (Rot21, Rot02, Rot10)
        TF w[3];
        w[0] = (TF)au0 + (TF)f.wspin[0 * P + v] - ws[0] * dt;
        w[1] = (TF)au1 + (TF)f.wspin[1 * P + v] - ws[1] * dt;
        w[2] = (TF)au2 + (TF)f.wspin[2 * P + v] - ws[2] * dt;
        // Orientation (src/constitutive.c:142-194)
        TF wn = sqrt(w[0] * w[0] + w[1] * w[1] + w[2] * w[2]);
        TF wt = tan(wn / (TF)2);
        if (fabs(wn) < (TF)1e-6) wn = (TF)1;
#pragma unroll
        for (int i = 0; i < 3; i++) w[i] *= wt / wn;
        TF om[3][3] = {{0, -w[2], w[1]}, {w[2], 0, -w[0]}, {-w[1], w[0], 0}};
        TF rot[3][3];
        wt = wt * wt;
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int j = 0; j < 3; j++) {
            TF o2 = om[i][0] * om[0][j] + om[i][1] * om[1][j] + om[i][2] * om[2][j];
            rot[i][j] = (TF)(i == j) + (TF)2 * (om[i][j] + o2) / ((TF)1 + wt);
          }
        TF Rn[9];
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int j = 0; j < 3; j++) Rn[i * 3 + j] = rot[i][0] * R[0 * 3 + j] + rot[i][1] * R[1 * 3 + j] + rot[i][2] * R[2 * 3 + j];
#pragma unroll
        for (int i = 0; i < 9; i++) f.rot[i * P + v] = (TSt)Rn[i];
      }
      if (do_harden) {
        const TF gamtot = (TF)f.gamacum[v];
        TF deltgam = 0;
#pragma unroll
        for (int s = 0; s < NSYS; s++) deltgam += fabs(gam[s]) * dt;   // gam is 0 past nsys
        if (deltgam > (TF)0) {
          const TF tau0 = cpick<TF>(ph.tau0f, ph.tau0ff), tau1 = cpick<TF>(ph.tau1, ph.tau1f),
                   th0 = cpick<TF>(ph.thet0, ph.thet0f), th1 = cpick<TF>(ph.thet1, ph.thet1f);
          const TF tiny = (TF)1e-4 * tau0;
          TF voce = 0;
          if (fabs(th0) > tiny) {
            voce = th1 * deltgam;
            if (fabs(tau1) > tiny) {
              // the Voce increment of harden (src/constitutive.c:293-316) with
              // exp(-dgam fact) - 1 as expm1 and the second bracket regrouped
              // as (e - 1)(gam fact + 1) + e dgam fact: the same value without
              // the cancellation of nearly equal terms (FP32 in mixed mode)
              const TF fact = fabs(th0 / tau1);
              const TF exp_ini = exp((TF)-1 * gamtot * fact);
              const TF em1 = expm1((TF)-1 * deltgam * fact);
              const TF exp_del = em1 + (TF)1;
              voce += (TF)-1 * (fact * tau1 - th1) / fact * exp_ini * em1 -
                      th1 / fact * exp_ini * (em1 * (gamtot * fact + (TF)1) + exp_del * deltgam * fact);
            }
          }
          // the hardening matrix is hself on the diagonal, hlat off it (fill_phase):
          // 24 operations instead of the 12 x 12 products, which FP32 keeps, as it
          // keeps rot_to_q: its roundings decide later steps of a volume with failed
          // solves (book.cuh); 0.42 ms a step at 128^3 for 0.38
          const TF hl = ph.nsys > 1 ? cpick<TF>(ph.hard[0][1], ph.hardf[0][1]) : (TF)0;
          const TF hs = cpick<TF>(ph.hard[0][0], ph.hardf[0][0]) - hl, vd = voce / deltgam;
#pragma unroll
          for (int s = 0; s < NSYS; s++) {
            if (s >= ph.nsys) break;
            if constexpr (sizeof(TF) == 4) {
              TF dtau = 0;
#pragma unroll
              for (int j = 0; j < NSYS; j++) dtau += cpick<TF>(ph.hard[s][j], ph.hardf[s][j]) * fabs(gam[j]) * dt;
              f.crss[s * P + v] = (TSt)((TF)f.crss[s * P + v] + dtau * voce / deltgam);
            } else {
              f.crss[s * P + v] = (TSt)((TF)f.crss[s * P + v] + (hl * deltgam + hs * (fabs(gam[s]) * dt)) * vd);
            }
          }
          f.gamacum[v] = (TSt)(gamtot + deltgam);
        }
      }
    }
  }
  block_reduce_smem<TF, NPART_END>(acc, partials);
}

cudaError_t launch_end_step(int mixed, const NewtonConst& nc_in, const void* fields, const double au[3], int do_orient,
                            int do_harden, double* partials, int nblocks, cudaStream_t st, int law) {
  NewtonConst nc = nc_in;
  fill_float_consts(nc);
  if (law == 1) {
    if (mixed) {
      const Fields<float>& f = *static_cast<const Fields<float>*>(fields);
      end_step_kernel<float, float, 1><<<nblocks, 256, 0, st>>>(nc, f, au[0], au[1], au[2], do_orient, 0, partials);
    } else {
      const Fields<double>& f = *static_cast<const Fields<double>*>(fields);
      end_step_kernel<double, double, 1><<<nblocks, 256, 0, st>>>(nc, f, au[0], au[1], au[2], do_orient, 0, partials);
    }
    return cudaGetLastError();
  }
  if (mixed) {
    const Fields<float>& f = *static_cast<const Fields<float>*>(fields);
    end_step_kernel<float, float><<<nblocks, 256, 0, st>>>(nc, f, au[0], au[1], au[2], do_orient, do_harden, partials);
  } else {
    const Fields<double>& f = *static_cast<const Fields<double>*>(fields);
    end_step_kernel<double, double><<<nblocks, 256, 0, st>>>(nc, f, au[0], au[1], au[2], do_orient, do_harden, partials);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------ set-up kernel
// Per voxel: crystal->sample matrix from Bunge angles (EulerToTransMatrix,
// src/kinematics.c:187-240, transposed as at src/init.c:276-278), the
// elastic initial stress C_gr : <grad u> (src/init.c:470-480) and the
// initial CRSS (src/init.c:1164-1170).  C066 is summed on the host from the
// elastic classes.
template <typename TSt>
__global__ void __launch_bounds__(256) setup_kernel(const NewtonConst nc, Fields<TSt> f, const double* __restrict__ euler,
                                                    AddVec d6) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = f.nv;
  if (v >= P) return;
  const int jph = f.phase[v];
  const PhaseConst& ph = nc.ph[jph];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    f.strain[i * P + v] = (TSt)0;
    f.epsp[i * P + v] = (TSt)0;
    f.edot[i * P + v] = (TSt)0;
    f.sig[i * P + v] = (TSt)0;
  }
  for (int i = 0; i < 3; i++) f.wspin[i * P + v] = (TSt)0;
  f.gamacum[v] = (TSt)0;
  double R[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  if (ph.type == 0) {
    const double d2r = 3.14159265359 / 180.;
    const double t1 = euler[3 * v] * d2r, p = euler[3 * v + 1] * d2r, t2 = euler[3 * v + 2] * d2r;
    const double ct1 = cos(t1), st1 = sin(t1), cph = cos(p), sph = sin(p), ct2 = cos(t2), st2 = sin(t2);
    double a[3][3];
    a[0][0] = ct1 * ct2 - st1 * st2 * cph;
    a[0][1] = st1 * ct2 + ct1 * st2 * cph;
    a[0][2] = st2 * sph;
    a[1][0] = -1.0 * ct1 * st2 - st1 * ct2 * cph;
    a[1][1] = -1.0 * st1 * st2 + ct1 * ct2 * cph;
    a[1][2] = ct2 * sph;
    a[2][0] = st1 * sph;
    a[2][1] = -1.0 * ct1 * sph;
    a[2][2] = cph;
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) R[i * 3 + j] = a[j][i];
    const double* et = f.etab + (size_t)f.eclass[v] * ETAB_W;
    double s6[6];
#pragma unroll
    for (int i = 0; i < 5; i++) {
      double s = 0;
#pragma unroll
      for (int j = 0; j < 5; j++) s += et[ET_CGR + pk(i, j)] * d6.v[j];
      s6[i] = s;
    }
    s6[5] = et[ET_CGR_HH] * d6.v[5];
#pragma unroll
    for (int i = 0; i < 6; i++) f.sig[i * P + v] = (TSt)s6[i];
    for (int s = 0; s < NSYS; s++) f.crss[s * P + v] = (TSt)(s < ph.nsys ? ph.tau0f : 0.0);
  } else {
    for (int s = 0; s < NSYS; s++) f.crss[s * P + v] = (TSt)0;
  }
#pragma unroll
  for (int i = 0; i < 9; i++) f.rot[i * P + v] = (TSt)R[i];
}

cudaError_t launch_setup(int mixed, const NewtonConst& nc, const void* fields, const double* euler, const double d6[6],
                         int nblocks, cudaStream_t st) {
  AddVec d;
  for (int i = 0; i < 6; i++) d.v[i] = d6[i];
  if (mixed) {
    const Fields<float>& f = *static_cast<const Fields<float>*>(fields);
    setup_kernel<float><<<nblocks, 256, 0, st>>>(nc, f, euler, d);
  } else {
    const Fields<double>& f = *static_cast<const Fields<double>*>(fields);
    setup_kernel<double><<<nblocks, 256, 0, st>>>(nc, f, euler, d);
  }
  return cudaGetLastError();
}

// ------------------------------------------------------------ downloads
// Field planes to voxel-major doubles for the host: a symmetric tensor of 6
// LT planes becomes the 3x3 row-major Cartesian tensor t = sum_i v_i B_i
// (the products and left-to-right sums of the host conversion, with
// rounded, uncontracted operations, so both give the same doubles); other
// fields are interleaved per voxel.
// the symmetric tensor of voxel v's 6 LT planes, row-major into o[9]
template <typename TSt>
__device__ __forceinline__ void sym_to_host(const TSt* __restrict__ src, long long P, long long v, double* o) {
  double a[6];
#pragma unroll
  for (int i = 0; i < 6; i++) a[i] = (double)src[i * P + v];
  const double r2 = RSQ2, r3 = RSQ3, r6 = RSQ6;
  const double t00 = __dadd_rn(__dadd_rn(__dmul_rn(a[0], -r2), __dmul_rn(a[1], -r6)), __dmul_rn(a[5], r3));
  const double t11 = __dadd_rn(__dadd_rn(__dmul_rn(a[0], r2), __dmul_rn(a[1], -r6)), __dmul_rn(a[5], r3));
  const double t22 = __dadd_rn(__dmul_rn(a[1], 2. * r6), __dmul_rn(a[5], r3));
  const double t12 = __dmul_rn(a[2], r2), t02 = __dmul_rn(a[3], r2), t01 = __dmul_rn(a[4], r2);
  o[0] = t00; o[1] = t01; o[2] = t02;
  o[3] = t01; o[4] = t11; o[5] = t12;
  o[6] = t02; o[7] = t12; o[8] = t22;
}

template <typename TSt>
__global__ void to_host_layout_kernel(const TSt* __restrict__ src, long long P, int nc, int sym,
                                      double* __restrict__ dst) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= P) return;
  if (sym) {
    sym_to_host(src, P, v, dst + 9 * v);
  } else {
    for (int i = 0; i < nc; i++) dst[nc * v + i] = (double)src[i * P + v];
  }
}

// DisGrad for the host: the symmetric part from the strain planes plus the
// antisymmetric part W, held as the planes (W21, W02, W10)
template <typename TSt>
__global__ void disgrad_to_host_kernel(const TSt* __restrict__ strain, const TSt* __restrict__ skew, long long P,
                                       double* __restrict__ dst) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= P) return;
  double* o = dst + 9 * v;
  sym_to_host(strain, P, v, o);
  const double w21 = (double)skew[v], w02 = (double)skew[P + v], w10 = (double)skew[2 * P + v];
  o[1] = __dsub_rn(o[1], w10);
  o[3] = __dadd_rn(o[3], w10);
  o[2] = __dadd_rn(o[2], w02);
  o[6] = __dsub_rn(o[6], w02);
  o[5] = __dsub_rn(o[5], w21);
  o[7] = __dadd_rn(o[7], w21);
}

cudaError_t launch_disgrad_to_host(int mixed, const void* strain, const void* skew, long long P, double* dst,
                                   cudaStream_t st) {
  const int nb = (int)((P + 255) / 256);
  if (mixed)
    disgrad_to_host_kernel<float><<<nb, 256, 0, st>>>(static_cast<const float*>(strain),
                                                       static_cast<const float*>(skew), P, dst);
  else
    disgrad_to_host_kernel<double><<<nb, 256, 0, st>>>(static_cast<const double*>(strain),
                                                        static_cast<const double*>(skew), P, dst);
  return cudaGetLastError();
}

// The antisymmetric part of DisGrad grows each step by that of its uniform
// increments (Udot dt at the step's start, the dDisGradAvg corrections
// before each iteration), u, and by that of the Gamma : sigma-hat terms added
// at src/evolution.c:1401, which the Green passes accumulate and the spin
// transform brings to wspin.  skew += u + wspin, all as (W21, W02, W10).
template <typename TSt>
__global__ void disgrad_skew_kernel(const TSt* __restrict__ wspin, TSt* __restrict__ skew, long long P, double u0,
                                    double u1, double u2) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= P) return;
  const double u[3] = {u0, u1, u2};
#pragma unroll
  for (int c = 0; c < 3; c++) skew[c * P + v] = (TSt)((double)skew[c * P + v] + (u[c] + (double)wspin[c * P + v]));
}

cudaError_t launch_disgrad_skew(int mixed, const void* wspin, void* skew, long long P, const double u[3],
                                cudaStream_t st) {
  const int nb = (int)((P + 255) / 256);
  if (mixed)
    disgrad_skew_kernel<float><<<nb, 256, 0, st>>>(static_cast<const float*>(wspin), static_cast<float*>(skew), P,
                                                    u[0], u[1], u[2]);
  else
    disgrad_skew_kernel<double><<<nb, 256, 0, st>>>(static_cast<const double*>(wspin), static_cast<double*>(skew),
                                                     P, u[0], u[1], u[2]);
  return cudaGetLastError();
}

cudaError_t launch_to_host_layout(int mixed, const void* src, long long P, int nc, int sym, double* dst,
                                  cudaStream_t st) {
  const int nb = (int)((P + 255) / 256);
  if (mixed)
    to_host_layout_kernel<float><<<nb, 256, 0, st>>>(static_cast<const float*>(src), P, nc, sym, dst);
  else
    to_host_layout_kernel<double><<<nb, 256, 0, st>>>(static_cast<const double*>(src), P, nc, sym, dst);
  return cudaGetLastError();
}

// --------------------------------------------------- deterministic reduction
// out[w] = sum over blocks (fixed order) of partials[b*width + w].  One
// 1024-thread block per component; each thread keeps four independent
// partial sums so four L2 loads are in flight instead of a chain of
// dependent ones.
constexpr int RED_NT = 1024;   // 32 warps: the second shuffle stage sums one value per warp
__global__ void __launch_bounds__(RED_NT) reduce_partials_kernel(const double* __restrict__ partials, int nblocks,
                                                                 int width, double* __restrict__ out) {
  __shared__ double sm[RED_NT / 32];
  for (int w = blockIdx.x; w < width; w += gridDim.x) {
    double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
    int b = threadIdx.x;
    for (; b + 3 * RED_NT < nblocks; b += 4 * RED_NT) {
      a0 += partials[(size_t)b * width + w];
      a1 += partials[(size_t)(b + RED_NT) * width + w];
      a2 += partials[(size_t)(b + 2 * RED_NT) * width + w];
      a3 += partials[(size_t)(b + 3 * RED_NT) * width + w];
    }
    for (; b < nblocks; b += RED_NT) a0 += partials[(size_t)b * width + w];
    // warp sums by shuffles, then the 32 warp sums by warp 0
    double a = (a0 + a1) + (a2 + a3);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x < 32) {
      a = sm[threadIdx.x];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
      if (threadIdx.x == 0) out[w] = a;
    }
    __syncthreads();
  }
}

cudaError_t launch_reduce_partials(const double* partials, int nblocks, int width, double* out, cudaStream_t st) {
  reduce_partials_kernel<<<width, RED_NT, 0, st>>>(partials, nblocks, width, out);
  return cudaGetLastError();
}

}  // namespace mth
