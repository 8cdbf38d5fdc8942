// newton_f32.cu -- the local solve of the FP32 modes (newton.cu describes the
// problem, local_solve.cuh the iteration).
#include <type_traits>
#include "newton_dev.cuh"

namespace mth {

constexpr int F32_NT = 128;   // threads of the largest block

__device__ __noinline__ bool solve5_f64(const float* H, const float* b, float* x) {
  return ldl_solve5_wide(H, b, x);
}

// A voxel whose solve is not an ordinary one (local_solve.cuh), or with a CRSS
// that softened to zero or below, solved from lambda by the damped iteration in
// its plain order of operations.  In the
// first Green iterations of a volume with a high exponent and a low CRSS (n = 20,
// 12 MPa) dt dgamma/dtau is more than 1e7 times the elastic compliance, so the
// rounding of the FP32 Hessian's entries decides whether its factorisation
// finds a pivot that is not positive; such a solve ends there, keeps its
// iterate and is counted as failed.  Which voxels those are is therefore a
// property of this order of operations, and the volume's later iterations
// start from their stresses.  In the iterations in plain order (book.cuh) every
// voxel takes it, 1.75 ms a launch at 128^3; elsewhere the test for it and the
// call cost the kernel 3 % (0.9 ms of 100 launches).
struct SteepOut {
  float s6[6], e6[6];
  VoxelOut<float> o;
};
template <int SOLVE, int LAW>
__device__ __noinline__ void solve_steep(const NewtonConst& nc, const PhaseConst& ph, const Fields<float>& f,
                                         long long v, SteepOut& out) {
  const long long P = f.nv;
  typename SlipOf<LAW, float, float>::type slip;
  SlipOf<LAW, float, float>::load(ph, f, v, slip);
  auto load = [&](float* lam6, float* eps6, float* ep6, float* R, bool again) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
      lam6[i] = ld_sel(f.sig + i * P + v, again);
      eps6[i] = ld_sel(f.strain + i * P + v, again);
      ep6[i] = ld_sel(f.epsp + i * P + v, again);
    }
#pragma unroll
    for (int i = 0; i < 9; i++) R[i] = ld_sel(f.rot + i * P + v, again);
  };
  const float* et = f.etabf + (size_t)f.eclass[v] * ETAB_W;
  using TL = std::conditional_t<SOLVE == LS_FAST, float, double>;
  out.o = solve_voxel<float, TL, SOLVE == LS_NEAR_ROOT>(nc, ph, et, slip, load, out.s6, out.e6);
}

// FP32 modes: one voxel per thread, everything of the solve in FP32 but the
// systems the refinement leaves to FP64 (local_solve.cuh).  Each thread's
// K, c and slip-law constants live in its column of shared memory.
//
// What bounds it: issue slots (0.70 of the cycles issue; the FP32 pipe is
// half busy, DRAM a tenth).  128^3, 100 Green iterations, ms (events around
// each launch): 35.1; 103.5 for the earlier kernels, whose blocks stepped their
// solves in lock step to share the FP64 solves; the FP32-solve mode at 64^3 4.6
// and 10.7, the dislocation-density law at 96^3 17.8 and 31.5.
template <int SOLVE, int LAW, bool GEN, int MINB>
__global__ void __launch_bounds__(F32_NT, MINB) newton_f32_kernel(const __grid_constant__ LocalConst lc,
                                                                 const __grid_constant__ NewtonConst nc,
                                                                 const __grid_constant__ Fields<float> f,
                                                                 double* __restrict__ partials, IterIn it) {
  if (!is_live(it)) return;
  extern __shared__ __align__(16) float ls_sm[];
  const Column<float, F32_NT> col{ls_sm + threadIdx.x};
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = f.nv;
  float acc[NPART];
#pragma unroll
  for (int i = 0; i < NPART; i++) acc[i] = 0.0f;
  if (v < P) {
    const int jph = f.phase[v];
    const SlipF& ph = lc.ph[GEN ? jph : 0];
    if (GEN ? ph.type == 0 : jph == 0) {
      const float* et = f.etabf + (size_t)f.eclass[v] * ETAB_W;
      float x[5], ed[5], h, dh, ref2;
      {
        float lam[6], u[6], R[9], Q[25];
#pragma unroll
        for (int i = 0; i < 6; i++) {
          lam[i] = f.sig[i * P + v];
          u[i] = f.epsp[i * P + v] - f.strain[i * P + v];
        }
#pragma unroll
        for (int i = 0; i < 9; i++) R[i] = f.rot[i * P + v];
        // c = Q (eps_p - eps - S0 lambda)
        h = (lc.s0hh * lam[5] - u[5]) / (lc.s0hh + et[ET_SEL_HH]);
        dh = h - lam[5];
        ref2 = lam[5] * lam[5];
#pragma unroll
        for (int i = 0; i < 5; i++) {
          float a = lc.s0[i * 5] * lam[0];
#pragma unroll
          for (int j = 1; j < 5; j++) a = fmaf(lc.s0[i * 5 + j], lam[j], a);
          u[i] -= a;
          ref2 = fmaf(lam[i], lam[i], ref2);
        }
        rot_to_q_dev<float>(R, Q);
#pragma unroll
        for (int i = 0; i < 5; i++) {
          float a = Q[i * 5] * lam[0], b = Q[i * 5] * u[0];
#pragma unroll
          for (int j = 1; j < 5; j++) {
            a = fmaf(Q[i * 5 + j], lam[j], a);
            b = fmaf(Q[i * 5 + j], u[j], b);
          }
          x[i] = a;
          col(LS_C + i) = b;
        }
        float S[15];
#pragma unroll
        for (int i = 0; i < 15; i++) S[i] = et[ET_STOT + i];
        store_k(Q, S, col);
      }
      if constexpr (LAW == 0) {
        const int ns = nc.ph[GEN ? jph : 0].nsys;
#pragma unroll
        for (int s = 0; s < NSYS; s++) {
          const float t = f.crss[s * P + v];
          // 0 in the slots past nsys; a CRSS of an active system that softened to zero
          // or below gives no direction (steep)
          const float none = s < ns ? __int_as_float(0x7fffffff) : 0.0f;
          col(LS_LAW + s) = t > 0.0f ? rcp_f32(t) : none;
          if (GEN) {
            const float tb = t + ph.tau_off;
            col(LS_LAW + NSYS + s) = t > 0.0f && tb > 0.0f ? rcp_f32(tb) : none;
          }
        }
      } else {
#pragma unroll
        for (int s = 0; s < 3 * NSYS; s++) col(LS_LAW + s) = f.ddc[s * P + v];
      }
      SolveF32 o{0, false, true};
      if (LAW == 1 || !is_plain(it))
        o = solve_f32<SOLVE, LAW, GEN, false>(lc, ph, col, et[ET_STOT_MIN], ref2, h, dh, x, ed);
      if (o.steep) {
        SteepOut r;
        solve_steep<SOLVE, LAW>(nc, nc.ph[GEN ? jph : 0], f, v, r);
#pragma unroll
        for (int i = 0; i < 6; i++) {
          f.sig[i * P + v] = r.s6[i];
          f.edot[i * P + v] = r.e6[i];
          acc[2 + i] = r.s6[i];
        }
        acc[0] = r.o.conv_s;
        acc[1] = r.o.conv_e;
        acc[14] = (float)r.o.iters;
        acc[15] = (float)r.o.failed;
      } else {
        // back to sample axes; the inputs are read again rather than held
        // through the solve
        float lam[6], u[6], R[9], ss[5], es[5];
#pragma unroll
        for (int i = 0; i < 9; i++) R[i] = ld_again(f.rot + i * P + v);
        {
          float2 xe[5], se[5];
#pragma unroll
          for (int i = 0; i < 5; i++) xe[i] = make_float2(x[i], ed[i]);
          if constexpr (LAW == 0) {
            dev_to_sample2(R, xe, se);
          } else {
            // Q^T x: two roundings fewer than T X T^T.  The sinh law's stress is off by
            // 2.34e-7 from 64 bits with it and by 2.50e-7 without (96^3, three seeds; 17.9
            // and 17.8 ms for 100 launches); the power law's by the same 2.1e-7 either way.
            float Q[25];
            rot_to_q_dev<float>(R, Q);
#pragma unroll
            for (int j = 0; j < 5; j++) {
              se[j] = mul2(dup2(Q[j]), xe[0]);
#pragma unroll
              for (int i = 1; i < 5; i++) se[j] = fma2(dup2(Q[i * 5 + j]), xe[i], se[j]);
            }
          }
#pragma unroll
          for (int i = 0; i < 5; i++) {
            ss[i] = se[i].x;
            es[i] = se[i].y;
          }
        }
#pragma unroll
        for (int i = 0; i < 6; i++) {
          lam[i] = ld_again(f.sig + i * P + v);
          u[i] = ld_again(f.epsp + i * P + v) - ld_again(f.strain + i * P + v);
        }
        float cs = dh * dh, ce;
        {
          const float de = fmaf(et[ET_SEL_HH], h, u[5]);
          ce = de * de;
        }
#pragma unroll
        for (int i = 0; i < 5; i++) {
          const float ds = ss[i] - lam[i];
          cs = fmaf(ds, ds, cs);
          float de = fmaf(lc.dt, es[i], u[i]);
#pragma unroll
          for (int j = 0; j < 5; j++) de = fmaf(et[ET_SEL + pk5s(i, j)], ss[j], de);
          ce = fmaf(de, de, ce);
        }
#pragma unroll
        for (int i = 0; i < 5; i++) {
          f.sig[i * P + v] = ss[i];
          f.edot[i * P + v] = es[i];
          acc[2 + i] = ss[i];
        }
        f.sig[5 * P + v] = h;
        f.edot[5 * P + v] = 0.0f;
        acc[7] = h;
        acc[0] = sqrtf(cs);
        acc[1] = sqrtf(ce);
        acc[14] = (float)o.it;   // small integers: exact
      }
      if (GEN && jph == 0) {
#pragma unroll
        for (int i = 0; i < 6; i++) acc[8 + i] = acc[2 + i];
      }
    } else {
#pragma unroll
      for (int i = 0; i < 6; i++) {
        f.sig[i * P + v] = 0.0f;
        f.edot[i * P + v] = 0.0f;
      }
    }
  }
  newton_block_sums<float, GEN, F32_NT>(acc, col, partials);
}

// Blocks of 128 threads per SM the kernels are compiled for.  100 launches of
// an earlier state, ms: 128^3 33.3 with 4 (128 registers), 35.9 with 3, 36.1 with 5, 39.9 with 6;
// dislocation-density law at 96^3 17.2 with 4, 19.0 with 3, 23.4 with 5.
#ifndef MTH_F32_MINB
#define MTH_F32_MINB 4
#endif
#ifndef MTH_DD_MINB
#define MTH_DD_MINB 4
#endif

template <int SOLVE, int LAW, bool GEN, int MINB>
static cudaError_t launch_f32(const LocalConst& lc, const NewtonConst& nc, const Fields<float>& f, double* partials,
                              const IterIn& it, cudaStream_t st) {
  const int nt = newton_threads(f.nv, false);
  static_assert(sizeof(float) * F32_NT * ls_rows<LAW, GEN>() <= 47 * 1024, "no opt-in above 48 KB is made");
  return launch_chain(newton_f32_kernel<SOLVE, LAW, GEN, MINB>, dim3(newton_blocks(f.nv, false)), dim3(nt),
                      sizeof(float) * F32_NT * ls_rows<LAW, GEN>(), st, it.pdl, lc, nc, f, partials, it);
}
template <int SOLVE, int LAW, int MINB>
static cudaError_t launch_f32_gen(bool plain, const LocalConst& lc, const NewtonConst& nc, const Fields<float>& f,
                                  double* partials, const IterIn& it, cudaStream_t st) {
  return plain ? launch_f32<SOLVE, LAW, false, MINB>(lc, nc, f, partials, it, st)
               : launch_f32<SOLVE, LAW, true, MINB>(lc, nc, f, partials, it, st);
}
cudaError_t launch_newton_f32(int mixed, const NewtonConst& nc_in, const Fields<float>& f, double* partials,
                              const IterIn& it, cudaStream_t st, int law) {
  LocalConst lc;
  fill_local(nc_in, false, lc);
  NewtonConst nc = nc_in;
  fill_float_consts(nc);
  const bool plain = plain_phase(nc, lc);
  // dislocation-density law: refined solves at every step in all mixed modes
  if (law == 1) return launch_f32_gen<LS_REFINED, 1, MTH_DD_MINB>(nc.ph1_only != 0, lc, nc, f, partials, it, st);
  if (mixed == 2) return launch_f32_gen<LS_FAST, 0, MTH_F32_MINB>(plain, lc, nc, f, partials, it, st);
  if (mixed == 3) return launch_f32_gen<LS_NEAR_ROOT, 0, MTH_F32_MINB>(plain, lc, nc, f, partials, it, st);
  return launch_f32_gen<LS_REFINED, 0, MTH_F32_MINB>(plain, lc, nc, f, partials, it, st);
}

}  // namespace mth
