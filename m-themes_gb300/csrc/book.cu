// book.cu -- the end of a Green iteration on the device: the Newton kernels'
// rows of partial sums reduced to the iteration's sums, and the bookkeeping
// of book.cuh on them, so that mth_step can queue Green iterations without a
// host round trip.  One kernel: up to 128 blocks each sum their share of the
// rows in a fixed order, the last one to finish sums the shares (the same
// order whichever block that is) and its first warp does the bookkeeping.
// GB300 issues FP64 at one warp instruction per sub-partition every few
// dozen cycles whatever the active lanes, so the lanes compute independent
// entries (the 9 of a tensor, the 6 of a vector) side by side, each with
// exactly the operations, in the order, of book.cuh's loops less the
// products with the basis tensors' zeros.  The state is worked on in shared
// memory and written back once.  Compiled without FMA contraction like the
// host code; tests require the two to give the same doubles.
// It is a chain of latencies: 17 us per iteration at 64^3 with the launch,
// against 25 us for a reduction and a one-warp kernel of its own (events
// around the launches, which add about 4 us each).
#include "book.cuh"
#include "mth_internal.h"

namespace mth {

namespace {

constexpr int RB_NT = 512;     // threads
constexpr int RB_ROWS = 128;   // rows a block sums before another block is added
constexpr int RB_MAX = 128;    // blocks

// Sums of the 16 components over n rows: thread t adds component t % 16 of
// every 32nd row, then the 32 row lanes are combined in a fixed order.
// Lanes 0..15 of warp 0 return component lane's sum.
__device__ __forceinline__ double sum_rows(const double* __restrict__ rows, int n, double (*sm)[16]) {
  const int t = threadIdx.x, comp = t & 15;
  double a0 = 0, a1 = 0, a2 = 0, a3 = 0;
  int r = t >> 4;
  for (; r + 96 < n; r += 128) {   // four rows in flight
    a0 += __ldcg(&rows[(size_t)r * 16 + comp]);
    a1 += __ldcg(&rows[(size_t)(r + 32) * 16 + comp]);
    a2 += __ldcg(&rows[(size_t)(r + 64) * 16 + comp]);
    a3 += __ldcg(&rows[(size_t)(r + 96) * 16 + comp]);
  }
  for (; r < n; r += 32) a0 += __ldcg(&rows[(size_t)r * 16 + comp]);
  double a = (a0 + a1) + (a2 + a3);
  a += __shfl_xor_sync(0xffffffffu, a, 16);
  if ((t & 31) < 16) sm[t >> 5][comp] = a;
  __syncthreads();
  double b = 0;
  if (t < 32) {
    const int h = (t >> 4) * 8;
#pragma unroll
    for (int k = 0; k < 8; k++) b += sm[h + k][comp];
    b += __shfl_xor_sync(0xffffffffu, b, 16);
  }
  return b;
}

// entry e = 3 m + n of the tensor of LT components v (the first nv of them)
__device__ __forceinline__ double v2t_entry(const double* v, int e, int nv) {
  const int m = e / 3, n = e % 3;
  if (m != n) return v[5 - (m + n)] * RSQ2;
  double s = v[0] * book_basis(0, m, m);
  s += v[1] * book_basis(1, m, m);
  if (nv > 5) s += v[5] * RSQ3;
  return s;
}
// LT component i of tensor t
__device__ __forceinline__ double t2v_entry(const double* t, int i) {
  if (i < 2 || i == 5) {
    double s = t[0] * book_basis(i, 0, 0);
    s += t[4] * book_basis(i, 1, 1);
    s += t[8] * book_basis(i, 2, 2);
    return s;
  }
  const int m = i == 2 ? 1 : 0, n = i == 4 ? 1 : 2;
  double s = t[m * 3 + n] * RSQ2;
  s += t[n * 3 + m] * RSQ2;
  return s;
}

struct BookTmp {
  double s6[6], s16[6], sg[9], sg1[9], v6[6], v61[6], dv[9], dv1[9], u[9];
  int more;
};

// book_finish on the sums red (one warp, b and red in shared memory); false
// when a sum is not finite
__device__ __forceinline__ bool book_end(IterBook& b, const double* red, BookTmp& w) {
  const int lane = threadIdx.x & 31;
  const bool ok = lane >= NPART || isfinite(red[lane]);
  if (!__all_sync(0xffffffffu, ok)) {
    if (lane == 0) b.nan = 1;
    return false;
  }
  if (lane < 6) w.s6[lane] = red[2 + lane] * b.wgt;
  else if (lane < 12) w.s16[lane - 6] = red[8 + lane - 6] * (b.wgt / b.wgt_ph1);
  else if (lane == 12) b.it_nit += (long long)red[14];
  else if (lane == 13) b.it_nbad += (long long)red[15];
  else if (lane == 14) b.err_s = red[0] * b.wgt;
  else if (lane == 15) b.err_e = red[1] * b.wgt;
  else if (lane == 16 && b.plain == 1 && b.it_iter == 1 && !(red[15] > 0.0)) b.plain = 0;
  __syncwarp();
  if (lane < 18) {   // v2t: sig_avg (lanes 0-8), sig_avg1 (lanes 9-17)
    const int e = lane % 9;
    const double s = v2t_entry(lane < 9 ? w.s6 : w.s16, e, 6);
    if (lane < 9) {
      b.sig_avg[e / 3][e % 3] = s;
      w.sg[e] = s;
    } else {
      b.sig_avg1[e / 3][e % 3] = s;
      w.sg1[e] = s;
    }
  }
  __syncwarp();
  if (lane < 6) {   // the mixed-boundary correction, component a = lane
    const int IJV[2][6] = {{0, 1, 2, 1, 0, 0}, {0, 1, 2, 2, 2, 1}};
    const int ii = lane < 3 ? lane : lane == 3 ? 1 : 0, jj = lane < 3 ? lane : lane == 5 ? 1 : 2;
    double d = 0.0;
    if (b.vbc[lane] == 0)
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const int kk = IJV[0][q], ll = IJV[1][q];
        d += b.s0_4[((ii * 3 + jj) * 3 + kk) * 3 + ll] * b.sbc[q] * (b.scauchy[kk][ll] - w.sg[kk * 3 + ll]);
      }
    b.ddg[ii][jj] = d;
  } else if (lane < 18) {   // t2v: of sig_avg (lanes 6-11), of sig_avg1 (lanes 12-17)
    const int i = (lane - 6) % 6;
    if (lane < 12) w.v6[i] = t2v_entry(w.sg, i);
    else w.v61[i] = t2v_entry(w.sg1, i);
  }
  __syncwarp();
  if (lane < 9) b.ddg_acum[lane / 3][lane % 3] += b.ddg[lane / 3][lane % 3];
  if (lane < 18) {   // v2t of the deviatoric parts (5 components)
    const int e = lane % 9;
    if (lane < 9) w.dv[e] = v2t_entry(w.v6, e, 5);
    else w.dv1[e] = v2t_entry(w.v61, e, 5);
  }
  __syncwarp();
  double sq = 0;   // squares of the von Mises sums, entry lane % 9
  if (lane < 18) {
    const int e = lane % 9;
    double d = lane < 9 ? w.dv[e] : w.dv1[e];
    if (lane < 9 && e % 4 == 0) d = d - (w.dv[4] + w.dv[8] + w.sg1[0]) / 3.0;   // the word past SigDevAvg (book_smacro)
    sq = d * d;
  }
  __syncwarp();
  if (lane < 9) w.dv[lane] = sq;
  else if (lane < 18) w.dv1[lane - 9] = sq;
  __syncwarp();
  if (lane < 2) {
    const double* t = lane == 0 ? w.dv : w.dv1;
    double s = 0;
#pragma unroll
    for (int e = 0; e < 9; e++) s += t[e];
    s = sqrt(3. / 2. * s);
    if (lane == 0) b.s_vm = s;
    else b.s_vm1 = s;
  }
  __syncwarp();
  if (lane == 0) b.err_s /= b.s_vm;
  else if (lane == 1) {
    if (fabs(b.e_vm) < 1E-5) b.err_e = 0.0;
    else b.err_e /= b.e_vm;
  }
  __syncwarp();
  return true;
}

// book_more and book_add: the next iteration's increment into add, or live
// dropped (one warp)
__device__ __forceinline__ void book_next(IterBook& b, double* __restrict__ add, int* __restrict__ live, BookTmp& w) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    w.more = book_more(b) ? 1 : 0;
    if (w.more) b.it_iter++;
    else *live = 0;
  }
  __syncwarp();
  if (!w.more) return;
  if (lane < 9) {
    const int i = lane / 3, j = lane % 3;
    w.u[lane] = b.ddg[i][j] + (b.it_iter == 1 ? b.udot[i][j] * b.dt : 0.0);
    b.ddg_applied[i][j] += b.ddg[i][j];
  }
  __syncwarp();
  if (lane < 6) add[lane] = t2v_entry(w.u, lane);
}

// all threads of the block copy the state, in 8-byte words
__device__ __forceinline__ void copy_book(IterBook* to, const IterBook* from) {
  static_assert(sizeof(IterBook) % 8 == 0, "copied in 8-byte words");
  const unsigned long long* a = reinterpret_cast<const unsigned long long*>(from);
  unsigned long long* c = reinterpret_cast<unsigned long long*>(to);
  for (int i = threadIdx.x; i < (int)(sizeof(IterBook) / 8); i += blockDim.x) c[i] = a[i];
}

// the step's start: live set, the first iteration's increment
__global__ void __launch_bounds__(32) book_start_kernel(IterBook* __restrict__ b, double* __restrict__ add,
                                                        int* __restrict__ live) {
  __shared__ IterBook sb;
  __shared__ BookTmp w;
  copy_book(&sb, b);
  if (threadIdx.x == 0) *live = 1;
  __syncwarp();
  book_next(sb, add, live, w);
  __syncwarp();
  copy_book(b, &sb);
}

// The end of an iteration: rows -> red, then (b not null) the bookkeeping.
// live drops to 0 when the step's iterations are done (Err met or IterMax)
// or a sum is not finite, and the iteration kernels queued after that return
// at once.  share: RB_MAX rows of 16 and the ticket (0 before and after).
__global__ void __launch_bounds__(RB_NT) iter_end_kernel(const double* __restrict__ rows, int nrows, int per,
                                                         double* __restrict__ share, unsigned* __restrict__ ticket,
                                                         double* __restrict__ red, IterBook* __restrict__ b,
                                                         double* __restrict__ add, int* __restrict__ live, IterIn it) {
  if (!is_live(it)) return;
  __shared__ IterBook sb;
  __shared__ BookTmp w;
  __shared__ double sm[RB_NT / 32][16], sr[16];
  __shared__ bool last;
  if (b) copy_book(&sb, b);   // every block: the copy's latency passes under the sums
  const int r0 = blockIdx.x * per;
  double a = sum_rows(rows + (size_t)r0 * 16, min(per, nrows - r0), sm);
  if (gridDim.x > 1) {
    if (threadIdx.x < 16) {
      __stcg(&share[blockIdx.x * 16 + threadIdx.x], a);
      __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    a = sum_rows(share, (int)gridDim.x, sm);
    if (threadIdx.x == 0) *ticket = 0;
  }
  if (threadIdx.x < 16) {
    sr[threadIdx.x] = a;
    red[threadIdx.x] = a;
  }
  if (!b) return;
  __syncthreads();
  if (threadIdx.x < 32) {
    if (book_end(sb, sr, w)) book_next(sb, add, live, w);
    else if (threadIdx.x == 0) *live = 0;
  }
  __syncthreads();
  copy_book(b, &sb);
}

}  // namespace

size_t iter_end_scratch() { return sizeof(double) * 16 * RB_MAX + sizeof(unsigned) * 4; }

cudaError_t launch_book_start(IterBook* b, double* add, int* live, cudaStream_t st) {
  book_start_kernel<<<1, 32, 0, st>>>(b, add, live);
  return cudaGetLastError();
}

cudaError_t launch_iter_end(const double* rows, int nrows, void* scratch, double* red, IterBook* b, double* add,
                            int* live, const IterIn& it, cudaStream_t st) {
  int per = RB_ROWS;
  if ((nrows + per - 1) / per > RB_MAX) per = (nrows + RB_MAX - 1) / RB_MAX;
  double* share = static_cast<double*>(scratch);
  unsigned* ticket = reinterpret_cast<unsigned*>(share + 16 * RB_MAX);
  return launch_chain(iter_end_kernel, dim3((nrows + per - 1) / per), dim3(RB_NT), 0, st, it.pdl, rows, nrows, per,
                      share, ticket, red, b, add, live, it);
}

}  // namespace mth
