// drx.cu -- dynamic recrystallisation on the GPU: grain-boundary nucleation
// with a counter-based generator (NucleationCheckDRX, src/integrated.c:161-494)
// and the sparse order-parameter Allen-Cahn relaxation (PF_XRX / Update_grid /
// Update_gID, src/pf_xrx.c:6-66,895-1311,1469-1698), the reference's
// sequential sweep computed in parallel passes (section "phase field").
// This translation unit is compiled without FMA contraction so that FP64
// results are the separately rounded operations of the reference, bit for
// bit.
#include <climits>
#include <cstdint>
#include "mth_common.cuh"
#include "mth_internal.h"

namespace mth {

#define PF_EPS 5.0e-3
#define PF_KEEP 1.0e-4

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ULL;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
  return x ^ (x >> 31);
}
// uniform in (0, 1] from a (seed, counter) pair
__device__ __forceinline__ double uniform01(uint64_t seed, uint64_t counter) {
  uint64_t h = mix64(seed * 0xD1342543DE82EF95ULL + mix64(counter));
  return (double)((h >> 11) + 1) * (1.0 / 9007199254740992.0);
}

struct Dims {
  int n0, n1, n2;
  __device__ __forceinline__ long long idx(int x, int y, int z) const {
    x = (x % n0 + n0) % n0;
    y = (y % n1 + n1) % n1;
    z = (z % n2 + n2) % n2;
    return ((long long)x * n1 + y) * n2 + z;
  }
};

// The periodic 3x3x3 neighbourhood of voxel (x, y, z) without divisions:
// the wrapped coordinates of the three planes, rows and columns once, a
// neighbour's index by multiply-adds.
struct Nbhd {
  long long px[3];   // plane offsets of x-1, x, x+1 (times n1 n2)
  int py[3], pz[3];  // row offsets of y-1, y, y+1 (times n2); columns z-1, z, z+1
  __device__ __forceinline__ Nbhd(const Dims& d, int x, int y, int z) {
    const int xm = x == 0 ? d.n0 - 1 : x - 1, xp = x == d.n0 - 1 ? 0 : x + 1;
    const int ym = y == 0 ? d.n1 - 1 : y - 1, yp = y == d.n1 - 1 ? 0 : y + 1;
    const long long pl = (long long)d.n1 * d.n2;
    px[0] = xm * pl; px[1] = x * pl; px[2] = xp * pl;
    py[0] = ym * d.n2; py[1] = y * d.n2; py[2] = yp * d.n2;
    pz[0] = z == 0 ? d.n2 - 1 : z - 1; pz[1] = z; pz[2] = z == d.n2 - 1 ? 0 : z + 1;
  }
  // neighbour at offset (a, b, c), each in -1..1
  __device__ __forceinline__ long long at(int a, int b, int c) const { return px[a + 1] + py[b + 1] + pz[c + 1]; }
};

// -------------------------------------------------------------- nucleation
// Candidate: grain-boundary voxel as the reference marks it
// (src/evolution.c:816-829 from Gradient_ExchangeGrainID,
// src/constitutive.c:724-873: the +x, -x, +y, -y or +z neighbour in another
// grain -- its "-z" check compares with the -y neighbour), crystal phase,
// rho > rho_nuc, u(seed, counter) < prob.  Candidates are appended in
// arbitrary order; the host sorts them.
__global__ void nucleation_candidates_kernel(Dims d, const int* __restrict__ grain, const uint8_t* __restrict__ crystal,
                                             const double* __restrict__ rho, double rho_nuc, double prob,
                                             uint64_t seed, uint64_t counter0, long long* __restrict__ out,
                                             unsigned long long* __restrict__ count, long long cap) {
  const long long nv = (long long)d.n0 * d.n1 * d.n2;
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  if (!crystal[v]) return;
  const int x = (int)(v / ((long long)d.n1 * d.n2)), y = (int)((v / d.n2) % d.n1), z = (int)(v % d.n2);
  const int g = grain[v];
  const bool gb = (grain[d.idx(x + 1, y, z)] != g) | (grain[d.idx(x - 1, y, z)] != g) |
                  (grain[d.idx(x, y + 1, z)] != g) | (grain[d.idx(x, y - 1, z)] != g) |
                  (grain[d.idx(x, y, z + 1)] != g);
  if (!gb || !(rho[v] > rho_nuc)) return;
  const double u = uniform01(seed, counter0 + (uint64_t)v);
  if (u < prob) {
    unsigned long long k = atomicAdd(count, 1ULL);
    if ((long long)k < cap) out[k] = v;
  }
}

// Disc painting (src/integrated.c:397-402): winner[v] = max nucleus index
// whose squared distance to v is <= radius2 (the reference's nucleus_radius,
// compared with |d|^2), without periodic images; later nuclei win, as the
// sequential overwrite.
__global__ void paint_mark_kernel(Dims d, const long long* __restrict__ sites, int nn, int r, int radius2,
                                  int* __restrict__ winner) {
  const int side = 2 * r + 1;
  const int per = side * side * side;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)nn * per) return;
  const int k = (int)(t / per);
  const int o = (int)(t % per);
  const int dx = o / (side * side) - r, dy = (o / side) % side - r, dz = o % side - r;
  if (dx * dx + dy * dy + dz * dz > radius2) return;
  const long long v = sites[k];
  const int x = (int)(v / ((long long)d.n1 * d.n2)) + dx, y = (int)((v / d.n2) % d.n1) + dy, z = (int)(v % d.n2) + dz;
  if (x < 0 || x >= d.n0 || y < 0 || y >= d.n1 || z < 0 || z >= d.n2) return;
  atomicMax(&winner[((long long)x * d.n1 + y) * d.n2 + z], k);
}

__global__ void paint_apply_kernel(long long nv, int first_id, int* __restrict__ winner, int* __restrict__ grain) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  const int w = winner[v];
  if (w >= 0) {
    grain[v] = first_id + w;
    winner[v] = -1;
  }
}

// ------------------------------------------------------------ phase field
// PF_XRX / Update_grid / Update_gID (src/pf_xrx.c:6-66,895-1311,1469-1698)
// as the reference's sequential sweep computes it, in parallel passes.
//
// The reference sweeps x, y, z over the voxels and, while it does, changes
// the grid it reads: looking up an id a voxel does not hold takes over that
// voxel's last entry when the entry is below EPSILON (relabelling it) or
// appends (id, 0) (PFdata::operator[], src/PFgrid.h:70-90); it writes a
// global rho_avg table that later voxels read for ids they do not hold; and
// it resets the stored energy of a voxel a recrystallised id crosses
// (src/pf_xrx.c:1217-1219), which later voxels' window averages see.  Every
// one of these effects reaches a voxel only from voxels earlier in the sweep,
// and reads return the same value whatever the relabelling (a missing id
// reads the weak last entry's value, or 0), so each voxel's outcome is a
// function of the previous substep and of decisions of earlier voxels.  The
// passes compute those decisions to their fixed point (iterating until no
// voxel's decision changes, which happens after at most the length of the
// longest chain of dependent voxels, in practice two to four iterations):
//   tile    N(v): ids with eta > EPSILON over the 3x3x3 block, scan order, and
//           the stencil sums of those ids;
//   upd     whether the voxel holds more than one entry when the sweep
//           reaches it: it does if it held several, or if it held one strong
//           entry and one of its nine preceding stencil neighbours that
//           updates has an id it lacks in N (that neighbour's Laplacian
//           lookup appends it) -- fixed point;
//   tail    the id its last entry carries by then: the last such lookup, from
//           the latest preceding updating neighbour;
//   window  per held entry, the mean stored energy over the 7x7x7 window of
//           voxels whose initial grain id matches, with the resets of
//           earlier voxels in this substep;
//   rows    per row of voxels, the last value each id wrote to the table;
//   update  the new lists, with rho_avg of ids not held read from the latest
//           earlier writer (same row, then earlier rows, then the table) and
//           the energy resets this substep causes -- window/rows/update are
//           iterated to the fixed point of the resets;
//   table   each id's last writer's value into the table; finish: resets
//           applied, grain id = first maximum.
// Summation orders and the Laplacian's term order are the reference's, and
// this file is compiled without FMA contraction, so FP64 results equal the
// reference's sweep bit for bit (the oracle restates that sweep literally).

struct PfView {
  Dims d;
  long long nv;
  int rows;
};

// PFdata lookup by value: the entry's eta, else the weak last entry's, else 0
template <typename T>
__device__ __forceinline__ T pf_read_local(const int* id, const T* ph, int n, int j) {
  for (int k = 0; k < n; k++)
    if (id[k] == j) return ph[k];
  if (n > 0 && ph[n - 1] < (T)PF_EPS) return ph[n - 1];
  return (T)0;
}
__device__ __forceinline__ unsigned pf_hash(int id) { return ((unsigned)id * 2654435761u) >> 16; }

// PFdata lookup for assignment into a list under construction
template <typename T>
__device__ __forceinline__ void pf_write_local(int* id, T* ph, int& n, int j, T val, unsigned* bad) {
  for (int k = 0; k < n; k++)
    if (id[k] == j) { ph[k] = val; return; }
  if (n > 0 && ph[n - 1] < (T)PF_EPS) { id[n - 1] = j; ph[n - 1] = val; return; }
  if (n == PF_K) { *bad |= PF_BAD_LIST; return; }
  id[n] = j;
  ph[n] = val;
  n++;
}
// the list a voxel holds when the sweep reaches it: its stored list with the
// last entry relabelled or (tail, 0) appended
template <typename T>
__device__ __forceinline__ int pf_held(const PfView& g, const int* __restrict__ ids, const T* __restrict__ phi,
                                       const uint8_t* __restrict__ cnt, const int* __restrict__ tail,
                                       const uint8_t* __restrict__ tmode, long long v, int* hid, T* hph) {
  int n = cnt[v];
  for (int k = 0; k < n; k++) {
    hid[k] = ids[(long long)k * g.nv + v];
    hph[k] = phi[(long long)k * g.nv + v];
  }
  const int m = tmode[v];
  if (m == 1) hid[n - 1] = tail[v];
  else if (m == 2) { hid[n] = tail[v]; hph[n] = (T)0; n++; }
  return n;
}
// the nine stencil neighbours that precede v in the sweep, latest first
__constant__ int8_t c_pred[9][3] = {{0, 0, -1}, {0, -1, 1}, {0, -1, 0}, {0, -1, -1}, {-1, 1, 0},
                                    {-1, 0, 1}, {-1, 0, 0}, {-1, 0, -1}, {-1, -1, 0}};

template <typename T>
__global__ void pf_init_kernel(PfView g, const int* __restrict__ grain, const T* __restrict__ rho, int* __restrict__ ids,
                               T* __restrict__ phi, uint8_t* __restrict__ cnt, T* __restrict__ energy,
                               int* __restrict__ gid) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.nv) return;
  ids[v] = grain[v];
  phi[v] = (T)1;
  cnt[v] = 1;
  energy[v] = rho[v];
  gid[v] = grain[v];
}

// PFdata look-up by value at voxel w: the entry's eta, else the weak last
// entry's, else 0
template <typename T>
__device__ T pf_read_g(const int* __restrict__ ids, const T* __restrict__ phi, const uint8_t* __restrict__ cnt,
                       long long nv, long long w, int j) {
  const int n = cnt[w];
  T e = (T)0;
  for (int k = 0; k < n; k++) {
    e = phi[(long long)k * nv + w];
    if (ids[(long long)k * nv + w] == j) return e;
  }
  return n > 0 && e < (T)PF_EPS ? e : (T)0;
}

// The stencil in the order laplacian() adds it: it receives left_up.. as its
// right_up.. parameters (src/pf_xrx.c:6-9 against the call at :1193-1198):
// right left front back up down, then the twelve edges.
__constant__ int8_t c_sten[18][3] = {{1, 0, 0},  {-1, 0, 0},  {0, 1, 0},  {0, -1, 0}, {0, 0, 1},  {0, 0, -1},
                                     {0, -1, 1}, {0, -1, -1}, {0, 1, 1},  {0, 1, -1}, {-1, 0, -1}, {-1, 0, 1},
                                     {-1, -1, 0}, {-1, 1, 0}, {1, 0, 1},  {1, 1, 0},  {1, 0, -1}, {1, -1, 0}};
// the stencil's sum without the centre: 0.5 (faces) + 0.125 (edges), from the lists
template <typename T>
__device__ T pf_sten_lists(const int* __restrict__ ids, const T* __restrict__ phi, const uint8_t* __restrict__ cnt,
                           long long nv, const Nbhd& nb, int j) {
  T s1 = (T)0, s2 = (T)0;
#pragma unroll 1
  for (int o = 0; o < 18; o++) {
    const T e = pf_read_g<T>(ids, phi, cnt, nv, nb.at(c_sten[o][0], c_sten[o][1], c_sten[o][2]), j);
    if (o < 6) s1 = o == 0 ? e : s1 + e;
    else s2 = o == 6 ? e : s2 + e;
  }
  return (T)0.5 * s1 + (T)0.125 * s2;
}

// N(v) and the stencil sums of its ids, one 4x8x16 tile of voxels per block.
// The ids of the tile and its one-voxel halo (about a dozen at a thousand
// grains in 128^3) get numbers; a position's strong ids are a 64-bit mask of
// them, so the scan for N(v) tests a word per position and looks into a list
// only where a new id appears, and the etas are laid out densely in shared
// memory (missing ids hold what a look-up of them returns), PF_TB ids at a
// time, so that a stencil term is one load.  (One walk over a neighbour's list
// per term: 441 million warp instructions a launch at 128^3 for the update, 281
// million for N(v).)  The sums do not depend on the averages, so the iterates
// of a substep share them.  sten: PF_NS planes; ids past them, and tiles of
// more than 64 ids, go through the lists.
constexpr int PF_TX = 4, PF_TY = 8, PF_TZ = 16, PF_TV = PF_TX * PF_TY * PF_TZ;
constexpr int PF_HY = PF_TY + 2, PF_HZ = PF_TZ + 2, PF_HN = (PF_TX + 2) * PF_HY * PF_HZ;
constexpr int PF_TH = 128;   // hash slots
constexpr int PF_TB = 8;     // ids laid out at a time (ten substeps at 128^3: 24.5 ms, with 12 25.0, with 16 26.5)
constexpr int PF_NS = 8;
template <typename T>
__global__ void __launch_bounds__(256) pf_tile_kernel(PfView g, const int* __restrict__ ids, const T* __restrict__ phi,
                                                      const uint8_t* __restrict__ cnt, int* __restrict__ nid,
                                                      uint8_t* __restrict__ ncnt, T* __restrict__ sten, int tiles_y,
                                                      int tiles_z, unsigned* __restrict__ word) {
  extern __shared__ __align__(16) unsigned char pf_dyn[];
  T* dense = reinterpret_cast<T*>(pf_dyn);   // [PF_TB][PF_HN]
  __shared__ unsigned long long s_mask[PF_HN];
  __shared__ unsigned s_num[PF_HN];          // numbers of a position's first four entries
  __shared__ uint8_t s_cnt[PF_HN];
  __shared__ int s_id[PF_TH], s_of[64];      // hash table, id of a number
  __shared__ unsigned s_w[PF_HN];            // voxel of a halo position
  __shared__ uint8_t s_no[PF_TH];            // number of a slot
  __shared__ int s_n, s_over;
  const int t = threadIdx.x;
  const int tz = blockIdx.x % tiles_z, ty = (blockIdx.x / tiles_z) % tiles_y, tx = blockIdx.x / (tiles_z * tiles_y);
  const int x0 = tx * PF_TX, y0 = ty * PF_TY, z0 = tz * PF_TZ;
  const long long nv = g.nv;
  auto voxel_of = [&](int i) { return (long long)s_w[i]; };
  auto find = [&](int id) {
    int slot = (int)(pf_hash(id) & (PF_TH - 1));
    // every id of the tile was inserted, so this ends before the table does
    for (int tries = 0; tries < PF_TH && s_id[slot] != id; tries++) slot = (slot + 1) & (PF_TH - 1);
    return (int)s_no[slot];
  };
  if (t < PF_TH) s_id[t] = INT_MIN;
  if (t == 0) s_n = s_over = 0;
  __syncthreads();
  for (int i = t; i < PF_HN; i += blockDim.x) {
    const long long w =
        g.d.idx(x0 - 1 + i / (PF_HY * PF_HZ), y0 - 1 + (i / PF_HZ) % PF_HY, z0 - 1 + i % PF_HZ);
    s_w[i] = (unsigned)w;
    const int c = cnt[w];
    s_cnt[i] = (uint8_t)c;
    for (int k = 0; k < c; k++) {
      const int id = ids[(long long)k * nv + w];
      int slot = (int)(pf_hash(id) & (PF_TH - 1)), tries = 0;
      for (; tries < PF_TH; tries++, slot = (slot + 1) & (PF_TH - 1)) {
        const int prev = s_id[slot] == id ? id : atomicCAS(&s_id[slot], INT_MIN, id);
        if (prev == INT_MIN || prev == id) break;
      }
      if (tries == PF_TH || id == INT_MIN) s_over = 1;
    }
  }
  __syncthreads();
  if (t < PF_TH && s_id[t] != INT_MIN) {
    const int no = atomicAdd(&s_n, 1);   // any numbering will do
    if (no < 64) {
      s_no[t] = (uint8_t)no;
      s_of[no] = s_id[t];
    }
  }
  __syncthreads();
  const int n_ids = s_n;
  unsigned bad = 0;
  if (s_over || n_ids > 64) {
    for (int i = t; i < PF_TV; i += blockDim.x) {
      const int x = x0 + i / (PF_TY * PF_TZ), y = y0 + (i / PF_TZ) % PF_TY, z = z0 + i % PF_TZ;
      if (x >= g.d.n0 || y >= g.d.n1 || z >= g.d.n2) continue;
      const long long v = ((long long)x * g.d.n1 + y) * g.d.n2 + z;
      const Nbhd nb(g.d, x, y, z);
      int L[PF_NM];
      int n = 0;
      for (int dx = -1; dx <= 1; dx++)
        for (int dy = -1; dy <= 1; dy++)
          for (int dz = -1; dz <= 1; dz++) {
            const long long w = nb.at(dx, dy, dz);
            const int c = cnt[w];
            for (int k = 0; k < c; k++) {
              if (!(phi[(long long)k * nv + w] > (T)PF_EPS)) continue;
              const int j = ids[(long long)k * nv + w];
              bool seen = false;
              for (int a = 0; a < n; a++) seen |= (L[a] == j);
              if (seen) continue;
              if (n == PF_NM) { bad |= PF_BAD_NEIGH; continue; }
              L[n++] = j;
            }
          }
      ncnt[v] = (uint8_t)n;
      for (int a = 0; a < n; a++) {
        nid[(long long)a * nv + v] = L[a];
        if (a < PF_NS) sten[(long long)a * nv + v] = pf_sten_lists<T>(ids, phi, cnt, nv, nb, L[a]);
      }
    }
    if (bad) atomicOr(&word[1], bad);
    return;
  }
  for (int i = t; i < PF_HN; i += blockDim.x) {
    const long long w = voxel_of(i);
    const int c = s_cnt[i];
    unsigned long long m = 0;
    unsigned num = 0;
    for (int k = 0; k < c; k++) {
      const int no = find(ids[(long long)k * nv + w]);
      if (phi[(long long)k * nv + w] > (T)PF_EPS) m |= 1ull << no;
      if (k < 4) num |= (unsigned)no << (8 * k);
    }
    s_mask[i] = m;
    s_num[i] = num;
  }
  __syncthreads();
  // N(v): new ids in scan order, then list order
  unsigned long long mine[2];   // numbers of the first PF_NS ids of this thread's two voxels
  int mine_n[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = t + 256 * h;
    const int lx = i / (PF_TY * PF_TZ), ly = (i / PF_TZ) % PF_TY, lz = i % PF_TZ;
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    mine[h] = 0;
    mine_n[h] = 0;
    if (x >= g.d.n0 || y >= g.d.n1 || z >= g.d.n2) continue;
    const long long v = ((long long)x * g.d.n1 + y) * g.d.n2 + z;
    unsigned long long seen = 0;
    int n = 0;
#pragma unroll 1
    for (int o = 0; o < 9; o++) {
      const int q0 = ((lx + o / 3) * PF_HY + ly + o % 3) * PF_HZ + lz;
#pragma unroll
      for (int dz = 0; dz < 3; dz++) {
        const unsigned long long m = s_mask[q0 + dz] & ~seen;
        if (!m) continue;
        const int c = s_cnt[q0 + dz];
        const unsigned num = s_num[q0 + dz];
        for (int k = 0; k < c; k++) {
          const int no = k < 4 ? (int)(num >> (8 * k) & 255u) : find(ids[(long long)k * nv + voxel_of(q0 + dz)]);
          if (!(m >> no & 1ull)) continue;
          seen |= 1ull << no;
          if (n == PF_NM) { bad |= PF_BAD_NEIGH; continue; }
          nid[(long long)n * nv + v] = s_of[no];
          if (n < PF_NS) mine[h] |= (unsigned long long)no << (8 * n);
          n++;
        }
      }
    }
    ncnt[v] = (uint8_t)n;
    mine_n[h] = min(n, PF_NS);
  }
  if (bad) atomicOr(&word[1], bad);
  for (int b0 = 0; b0 < n_ids; b0 += PF_TB) {
    const int nb = min(PF_TB, n_ids - b0);
    __syncthreads();
    for (int i = t; i < PF_HN; i += blockDim.x) {
      const long long w = voxel_of(i);
      const int c = s_cnt[i];
      const unsigned num = s_num[i];
      T miss = (T)0;
      if (c > 0) {
        const T e = phi[(long long)(c - 1) * nv + w];
        if (e < (T)PF_EPS) miss = e;
      }
      for (int q = 0; q < nb; q++) dense[q * PF_HN + i] = miss;
      for (int k = 0; k < c; k++) {
        const int no = (k < 4 ? (int)(num >> (8 * k) & 255u) : find(ids[(long long)k * nv + w])) - b0;
        if (no >= 0 && no < nb) dense[no * PF_HN + i] = phi[(long long)k * nv + w];
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = t + 256 * h;
      const int lx = i / (PF_TY * PF_TZ), ly = (i / PF_TZ) % PF_TY, lz = i % PF_TZ;
      const long long v = ((long long)(x0 + lx) * g.d.n1 + (y0 + ly)) * g.d.n2 + (z0 + lz);
      const int at = ((lx + 1) * PF_HY + ly + 1) * PF_HZ + lz + 1;
      for (int a = 0; a < mine_n[h]; a++) {
        const int no = (int)(mine[h] >> (8 * a) & 255u) - b0;
        if (no < 0 || no >= nb) continue;
        const T* e = dense + no * PF_HN + at;
        constexpr int DX = PF_HY * PF_HZ, DY = PF_HZ;
        const T s1 = e[DX] + e[-DX] + e[DY] + e[-DY] + e[1] + e[-1];
        const T s2 = e[-DY + 1] + e[-DY - 1] + e[DY + 1] + e[DY - 1] + e[-DX - 1] + e[-DX + 1] + e[-DX - DY] +
                     e[-DX + DY] + e[DX + 1] + e[DX + DY] + e[DX - 1] + e[DX - DY];
        sten[(long long)a * nv + v] = (T)0.5 * s1 + (T)0.125 * s2;
      }
    }
  }
}

// What a voxel's update flag depends on: PF_GEN when it updates whatever its
// neighbours do (it holds several entries), else bit o when the o-th preceding
// neighbour (c_pred), if it updates, appends an id here: the voxel holds one
// strong entry and the neighbour's N has an id besides it.
constexpr unsigned PF_GEN = 1u << 15;
template <typename T>
__global__ void __launch_bounds__(256) pf_pred_kernel(PfView g, const int* __restrict__ ids, const T* __restrict__ phi,
                                                      const uint8_t* __restrict__ cnt, const int* __restrict__ nid,
                                                      const uint8_t* __restrict__ ncnt,
                                                      unsigned short* __restrict__ pred) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.nv) return;
  const int c = cnt[v];
  unsigned m = c > 1 ? PF_GEN : 0u;
  if (c == 1 && phi[v] >= (T)PF_EPS) {
    const int X = ids[v];
    const int x = (int)(v / ((long long)g.d.n1 * g.d.n2)), y = (int)((v / g.d.n2) % g.d.n1), z = (int)(v % g.d.n2);
#pragma unroll
    for (int o = 0; o < 9; o++) {
      const int qx = x + c_pred[o][0], qy = y + c_pred[o][1], qz = z + c_pred[o][2];
      if (qx < 0 || qy < 0 || qy >= g.d.n1 || qz < 0 || qz >= g.d.n2) continue;
      const long long q = ((long long)qx * g.d.n1 + qy) * g.d.n2 + qz;
      const int nq = ncnt[q];
      if (nq >= 2 || (nq == 1 && nid[q] != X)) m |= 1u << o;
    }
  }
  pred[v] = (unsigned short)m;
}

// One pass of the update flags' fixed point, in place.  The flags only turn
// on as the passes proceed (a flag is an OR over earlier voxels' flags), so
// reading some neighbours' flags of this pass and some of the last one still
// ends at the same fixed point, and a pass that changes nothing is at it.
// Within a warp (consecutive z of one row) the chain through the (0,0,-1)
// neighbour is resolved in the pass itself: u(z) = G(z) | (P(z) & u(z-1)),
// G the voxel's own and its other eight neighbours' part, P whether the
// z-1 neighbour's flag would carry over, solved for the warp's 32 lanes by
// a prefix over ballot masks.  Passes are queued in groups without a look
// from the host: pass i counts its changes in chg[i] and returns at once when
// pass i - 1 counted none (a group of 8 at 128^3: 3 us for an idle pass against
// 20 us for a host round trip).
__global__ void __launch_bounds__(256) pf_upd_kernel(PfView g, const unsigned short* __restrict__ pred,
                                                     uint8_t* __restrict__ upd, unsigned* __restrict__ chg, int pass) {
  if (pass > 0 && chg[pass - 1] == 0) return;
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = v < g.nv;
  const int lane = threadIdx.x & 31;
  uint8_t old = 0;
  unsigned m = 0;
  if (in) {
    old = upd[v];
    m = old ? PF_GEN : pred[v];
  }
  bool gen = (m & PF_GEN) != 0;
  const bool prop = (m & 1u) != 0;   // (0,0,-1): the previous voxel of the row
  // a set bit's neighbour lies inside the volume, so its index needs no check
#pragma unroll
  for (int o = 1; o < 9; o++)
    if (!gen && (m >> o & 1u))
      gen = upd[v + ((long long)c_pred[o][0] * g.d.n1 + c_pred[o][1]) * g.d.n2 + c_pred[o][2]] != 0;
  const bool zin = lane == 0 && prop && upd[v - 1] != 0;
  // u = G | (P & u(z-1)) over the warp; lane 0 takes u(z-1) from the buffer
  const unsigned am = __activemask();
  unsigned gm = __ballot_sync(am, gen || zin), pm = __ballot_sync(am, prop);
#pragma unroll
  for (int s = 1; s < 32; s <<= 1) {
    gm |= pm & (gm << s);
    pm &= pm << s;
  }
  if (in) {
    const uint8_t u = (uint8_t)((gm >> lane) & 1u);
    if (u != old) {
      upd[v] = u;
    }
  }
  // one store per warp, and none once the flag is seen set (a store per voxel
  // made the pass in which most flags turn on 0.25 ms)
  const bool changed = in && (uint8_t)((gm >> lane) & 1u) != old;
  if (__ballot_sync(am, changed) && lane == __ffs((int)am) - 1 && *(volatile unsigned*)&chg[pass] == 0) chg[pass] = 1;
}

template <typename T>
__global__ void __launch_bounds__(256) pf_tail_kernel(PfView g, const int* __restrict__ ids, const T* __restrict__ phi,
                                                      const uint8_t* __restrict__ cnt, const int* __restrict__ nid,
                                                      const uint8_t* __restrict__ ncnt, const uint8_t* __restrict__ upd,
                                                      int* __restrict__ tail, uint8_t* __restrict__ tmode,
                                                      unsigned* __restrict__ word) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.nv) return;
  const int c = cnt[v];
  const bool weak = c > 0 && phi[(long long)(c - 1) * g.nv + v] < (T)PF_EPS;
  const int ns = weak ? c - 1 : c;
  int sid[PF_K];
  for (int k = 0; k < ns; k++) sid[k] = ids[(long long)k * g.nv + v];
  const int x = (int)(v / ((long long)g.d.n1 * g.d.n2)), y = (int)((v / g.d.n2) % g.d.n1), z = (int)(v % g.d.n2);
  int t = -1;
  for (int o = 0; o < 9 && t < 0; o++) {
    const int qx = x + c_pred[o][0], qy = y + c_pred[o][1], qz = z + c_pred[o][2];
    if (qx < 0 || qy < 0 || qy >= g.d.n1 || qz < 0 || qz >= g.d.n2) continue;
    const long long q = ((long long)qx * g.d.n1 + qy) * g.d.n2 + qz;
    if (!upd[q]) continue;
    for (int a = ncnt[q] - 1; a >= 0; a--) {
      const int j = nid[(long long)a * g.nv + q];
      bool strong = false;
      for (int k = 0; k < ns; k++) strong |= (sid[k] == j);
      if (!strong) { t = j; break; }
    }
  }
  uint8_t m = 0;
  if (t >= 0) {
    if (weak) m = 1;
    else if (c < PF_K) m = 2;
    else atomicOr(&word[1], (unsigned)PF_BAD_LIST);
  }
  tail[v] = t;
  tmode[v] = m;
}

// Window averages, one 8x8x8 tile of voxels per block: the tile and its
// 3-voxel halo (periodic) of initial grain ids and energies are staged in
// shared memory once, and every voxel of the tile that updates sums its 7x7x7
// window from there, in window order, up to four held entries in one walk
// over the window (one walk each took 1.34 ms at 128^3).  The window
// positions before the centre in that order are exactly the voxels earlier in
// the sweep (the first 171), so a reset applies there when the position lies
// inside the volume (a periodic image is a halo copy, refreshed only after
// the sweep).
//
// The first iterate of a substep (ow_prev null) has no resets.  A later one
// differs only where resets changed: a tile none of whose positions changed
// its reset returns at once; else the averages that come out different are
// stored, their voxels marked in vdirty and their ids in idirty, and the
// value is passed on to the row's summary when this voxel is the row's last
// writer of the id.
constexpr int PF_WT = 8;
constexpr int PF_WH = PF_WT + 6;
constexpr int PF_WN = PF_WH * PF_WH * PF_WH;

// slot of id j >= 1 in row r's table of mask + 1 slots, -1 when absent
__device__ __forceinline__ int pf_row_find(const int* __restrict__ rw_id, int mask, int r, int j) {
  const int* t = rw_id + (long long)r * PF_RH;
  int slot = (int)(pf_hash(j) & (unsigned)mask);
  for (int tries = 0; tries <= mask; tries++, slot = (slot + 1) & mask) {
    const int id = t[slot];
    if (id == j) return slot;
    if (id == 0) return -1;
  }
  return -1;
}
// id of held entry k of voxel v (c stored entries)
__device__ __forceinline__ int pf_held_id(const int* __restrict__ ids, const int* __restrict__ tail, long long nv,
                                          long long v, int k, int c, int mode) {
  return (k == c || (mode == 1 && k == c - 1)) ? tail[v] : ids[(long long)k * nv + v];
}

template <typename T, int W, bool RESET>
__device__ __forceinline__ void pf_window_sums(const int* __restrict__ s_gid, const T* __restrict__ s_e,
                                               const uint8_t* __restrict__ s_reset, int base0, const int (&id)[W],
                                               T (&A)[W], int (&C)[W]) {
#pragma unroll
  for (int u = 0; u < W; u++) {
    A[u] = (T)0;
    C[u] = 0;
  }
  for (int i = 0; i < 7; i++)
    for (int j = 0; j < 7; j++) {
      const int base = base0 + (i * PF_WH + j) * PF_WH;
      const int q0 = (i * 7 + j) * 7;
#pragma unroll
      for (int m = 0; m < 7; m++) {
        const int w = base + m, g = s_gid[w];
        T e = s_e[w];
        if (RESET && q0 + m < 171 && s_reset[w]) e = (T)100;
        if constexpr (sizeof(T) == 8) {
          // at most one of the ids matches: one FP64 addition, to the selected sum
          T a = (T)0;
#pragma unroll
          for (int u = 0; u < W; u++) a = g == id[u] ? A[u] : a;
          a = a + e;
#pragma unroll
          for (int u = 0; u < W; u++) {
            A[u] = g == id[u] ? a : A[u];
            C[u] += g == id[u];
          }
        } else {
#pragma unroll
          for (int u = 0; u < W; u++)
            if (g == id[u]) {
              A[u] = A[u] + e;
              C[u]++;
            }
        }
      }
    }
}

template <typename T>
__global__ void __launch_bounds__(256) pf_window_kernel(PfView g, const int* __restrict__ ids,
                                                        const uint8_t* __restrict__ cnt, const int* __restrict__ tail,
                                                        const uint8_t* __restrict__ tmode, const int* __restrict__ gid0,
                                                        const T* __restrict__ energy, const uint8_t* __restrict__ ow,
                                                        const uint8_t* __restrict__ ow_prev, T* __restrict__ wavg,
                                                        const int* __restrict__ rw_id, T* __restrict__ rw_val,
                                                        const int* __restrict__ rw_zl,
                                                        const uint8_t* __restrict__ rw_mask,
                                                        uint8_t* __restrict__ vdirty, uint8_t* __restrict__ idirty,
                                                        int table_len, int tiles_y, int tiles_z) {
  __shared__ int s_gid[PF_WN];
  __shared__ T s_e[PF_WN];
  __shared__ uint8_t s_reset[PF_WN];
  const int tz = blockIdx.x % tiles_z, ty = (blockIdx.x / tiles_z) % tiles_y, tx = blockIdx.x / (tiles_z * tiles_y);
  const int x0 = tx * PF_WT, y0 = ty * PF_WT, z0 = tz * PF_WT;
  const bool again = ow_prev != nullptr;
  if (again) {
    bool diff = false;
    for (int i = threadIdx.x; i < PF_WN; i += blockDim.x) {
      const int gx = x0 - 3 + i / (PF_WH * PF_WH), gy = y0 - 3 + (i / PF_WH) % PF_WH, gz = z0 - 3 + i % PF_WH;
      uint8_t r = 0;
      if (gx >= 0 && gx < g.d.n0 && gy >= 0 && gy < g.d.n1 && gz >= 0 && gz < g.d.n2) {
        const long long p = ((long long)gx * g.d.n1 + gy) * g.d.n2 + gz;
        r = ow[p];
        diff |= r != ow_prev[p];
      }
      s_reset[i] = r;
    }
    if (!__syncthreads_or(diff)) return;
  }
  for (int i = threadIdx.x; i < PF_WN; i += blockDim.x) {
    const long long p = g.d.idx(x0 - 3 + i / (PF_WH * PF_WH), y0 - 3 + (i / PF_WH) % PF_WH, z0 - 3 + i % PF_WH);
    s_gid[i] = gid0[p];
    s_e[i] = energy[p];
  }
  __syncthreads();
  // the voxels that update, those with up to two entries from the front of
  // the list and those with more from its end, so that a warp's voxels take
  // the same walk (by voxel, half of the lanes idled)
  __shared__ unsigned short s_list[PF_WT * PF_WT * PF_WT];
  __shared__ int s_n2, s_n4;
  if (threadIdx.x == 0) s_n2 = s_n4 = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < PF_WT * PF_WT * PF_WT; i += blockDim.x) {
    const int x = x0 + i / (PF_WT * PF_WT), y = y0 + (i / PF_WT) % PF_WT, z = z0 + i % PF_WT;
    if (x >= g.d.n0 || y >= g.d.n1 || z >= g.d.n2) continue;
    const long long v = ((long long)x * g.d.n1 + y) * g.d.n2 + z;
    const int n = cnt[v] + (tmode[v] == 2 ? 1 : 0);
    if (n <= 1) continue;
    if (n == 2) s_list[atomicAdd(&s_n2, 1)] = (unsigned short)i;
    else s_list[PF_WT * PF_WT * PF_WT - 1 - atomicAdd(&s_n4, 1)] = (unsigned short)i;
  }
  __syncthreads();
  const int n2 = s_n2, n4 = s_n4;
  // whole warps of each kind
  const int w2 = (n2 + 31) & ~31, all = w2 + n4;
  for (int e = threadIdx.x; e < all; e += blockDim.x) {
    const bool four = e >= w2;
    if (!four && e >= n2) continue;
    const int i = four ? s_list[PF_WT * PF_WT * PF_WT - 1 - (e - w2)] : s_list[e];
    const int lx = i / (PF_WT * PF_WT), ly = (i / PF_WT) % PF_WT, lz = i % PF_WT;
    const int x = x0 + lx, y = y0 + ly, z = z0 + lz;
    const long long v = ((long long)x * g.d.n1 + y) * g.d.n2 + z;
    const int c = cnt[v], mode = tmode[v];
    const int n = c + (mode == 2 ? 1 : 0);
    const int base0 = (lx * PF_WH + ly) * PF_WH + lz;
    for (int k0 = 0; k0 < n; k0 += 4) {
      int id[4], C[4];
      T A[4];
#pragma unroll
      for (int u = 0; u < 4; u++) id[u] = k0 + u < n ? pf_held_id(ids, tail, g.nv, v, k0 + u, c, mode) : INT_MIN;
      if (again) {
        pf_window_sums<T, 4, true>(s_gid, s_e, s_reset, base0, id, A, C);
      } else if (four) {
        pf_window_sums<T, 4, false>(s_gid, s_e, s_reset, base0, id, A, C);
      } else {
        int id2[2] = {id[0], id[1]}, C2[2];
        T A2[2];
        pf_window_sums<T, 2, false>(s_gid, s_e, s_reset, base0, id2, A2, C2);
        A[0] = A2[0]; A[1] = A2[1]; A[2] = A[3] = (T)0;
        C[0] = C2[0]; C[1] = C2[1]; C[2] = C[3] = 0;
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (k0 + u >= n) continue;
        const T a = C[u] > 0 ? A[u] / (T)C[u] : (T)0;
        T* out = &wavg[(long long)(k0 + u) * g.nv + v];
        if (!again) {
          *out = a;
        } else if (a != *out) {
          *out = a;
          vdirty[v] = 1;
          if (id[u] >= 1 && id[u] <= table_len) idirty[id[u] - 1] = 1;
          const int r = x * g.d.n1 + y;
          const int slot = id[u] >= 1 ? pf_row_find(rw_id, rw_mask[r], r, id[u]) : -1;
          if (slot >= 0 && rw_zl[(long long)r * PF_RH + slot] == z) rw_val[(long long)r * PF_RH + slot] = a;
        }
      }
    }
  }
}

// Row summaries, one block per row of voxels (x, y): every id the row's
// updating voxels hold, with the first and last z holding it and the value
// the last one writes, as a hash table (open addressing, 64 slots, 256 where
// those fill up), so that a look-up by id takes one or two probes.  The row's
// bit is set in each id's bitmap of writing rows and the bitmap of that
// bitmap's words: the latest row before a given one that writes an id is a
// count of leading zeros away (a prefix of last writers over all blocks of
// rows, carried forward per substep, took 0.45 ms and the walk to it half of
// the update's time).
template <typename T>
__global__ void __launch_bounds__(128) pf_rows_kernel(PfView g, const int* __restrict__ ids,
                                                      const uint8_t* __restrict__ cnt, const int* __restrict__ tail,
                                                      const uint8_t* __restrict__ tmode, const T* __restrict__ wavg,
                                                      int* __restrict__ rw_id, T* __restrict__ rw_val,
                                                      int* __restrict__ rw_zf, int* __restrict__ rw_zl,
                                                      uint8_t* __restrict__ rw_mask, unsigned* __restrict__ bm,
                                                      unsigned* __restrict__ bl, int bm_w, int bl_w, int table_len,
                                                      unsigned* __restrict__ word) {
  __shared__ int h_id[PF_RH], h_zf[PF_RH], h_zl[PF_RH];
  __shared__ int h_n, h_full;
  const int r = blockIdx.x;
  unsigned bad = 0;
  int mask = 63;
  for (;;) {
    for (int i = threadIdx.x; i <= mask; i += blockDim.x) {
      h_id[i] = 0;   // grain ids are >= 1 in a table-writing list; 0 marks a free slot
      h_zf[i] = INT_MAX;
      h_zl[i] = -1;
    }
    if (threadIdx.x == 0) h_n = h_full = 0;
    __syncthreads();
    for (int z = threadIdx.x; z < g.d.n2; z += blockDim.x) {
      const long long v = (long long)r * g.d.n2 + z;
      const int c = cnt[v], mode = tmode[v];
      const int n = c + (mode == 2 ? 1 : 0);
      if (n <= 1) continue;
      for (int k = 0; k < n; k++) {
        const int id = pf_held_id(ids, tail, g.nv, v, k, c, mode);
        if (id < 1) { bad |= PF_BAD_TABLE; continue; }
        int slot = (int)(pf_hash(id) & (unsigned)mask), tries = 0;
        for (; tries <= mask; tries++, slot = (slot + 1) & mask) {
          const int prev = atomicCAS(&h_id[slot], 0, id);
          if (prev == 0) { atomicAdd(&h_n, 1); break; }
          if (prev == id) break;
        }
        if (tries > mask) { h_full = 1; continue; }
        atomicMin(&h_zf[slot], z);
        atomicMax(&h_zl[slot], z);
      }
    }
    __syncthreads();
    if (mask == 63 && (h_full || h_n > 48)) {
      mask = PF_RH - 1;
      __syncthreads();
      continue;
    }
    break;
  }
  if (h_full || h_n > PF_RW) bad |= PF_BAD_ROW;
  if (threadIdx.x == 0) rw_mask[r] = (uint8_t)mask;
  for (int i = threadIdx.x; i <= mask; i += blockDim.x) {
    const int id = h_id[i];
    rw_id[(long long)r * PF_RH + i] = id;
    if (id == 0) continue;
    rw_zf[(long long)r * PF_RH + i] = h_zf[i];
    rw_zl[(long long)r * PF_RH + i] = h_zl[i];
    if (table_len == 0) continue;
    if (id > table_len) { bad |= PF_BAD_TABLE; continue; }
    atomicOr(&bm[(long long)(id - 1) * bm_w + (r >> 5)], 1u << (r & 31));
    atomicOr(&bl[(long long)(id - 1) * bl_w + (r >> 10)], 1u << ((r >> 5) & 31));
  }
  for (int z = threadIdx.x; z < g.d.n2; z += blockDim.x) {
    const long long v = (long long)r * g.d.n2 + z;
    const int c = cnt[v], mode = tmode[v];
    const int n = c + (mode == 2 ? 1 : 0);
    if (n <= 1) continue;
    for (int k = 0; k < n; k++) {
      const int id = pf_held_id(ids, tail, g.nv, v, k, c, mode);
      if (id < 1) continue;
      int slot = (int)(pf_hash(id) & (unsigned)mask);
      for (int tries = 0; tries <= mask && h_id[slot] != id; tries++) slot = (slot + 1) & mask;
      if (h_id[slot] == id && h_zl[slot] == z) rw_val[(long long)r * PF_RH + slot] = wavg[(long long)k * g.nv + v];
    }
  }
  if (bad) atomicOr(&word[1], bad);
}

// the latest row before row r (all rows: r = rows) that writes id j, -1 if none
__device__ __forceinline__ int pf_row_before(const unsigned* __restrict__ bm, const unsigned* __restrict__ bl, int bm_w,
                                             int bl_w, int j, int r) {
  const unsigned* b = bm + (long long)(j - 1) * bm_w;
  int w = r >> 5;
  if (r & 31) {
    const unsigned m = b[w] & ((1u << (r & 31)) - 1u);
    if (m) return (w << 5) + 31 - __clz(m);
  }
  const unsigned* t = bl + (long long)(j - 1) * bl_w;
  int q = w >> 5;
  unsigned m = (w & 31) ? t[q] & ((1u << (w & 31)) - 1u) : 0u;
  while (!m) {
    if (--q < 0) return -1;
    m = t[q];
  }
  w = (q << 5) + 31 - __clz(m);
  return (w << 5) + 31 - __clz(b[w]);
}

// what the look-ups of the rho_avg table read
template <typename T>
struct PfRows {
  const int* id;
  const T* val;
  const int* zf;
  const int* zl;
  const uint8_t* mask;
  const unsigned* bm;
  const unsigned* bl;
  int bm_w, bl_w;
  const T* table;
  int table_len;
};

// A row's ids and, per id, the bitmap of the z that hold it, in shared memory
struct PfRowBits {
  const int* id;          // mask + 1 slots
  const unsigned* bits;   // words per slot: (n2 + 31) / 32; null: not built
  int mask, words;
};

// rho_avg of id j as the sweep leaves it just before voxel v: the latest
// earlier writer in v's row, else in the earlier rows, else the table as the
// previous substep left it
template <typename T>
__device__ T pf_stale(const PfView& g, long long v, int r, int z, int j, const int* __restrict__ ids,
                      const uint8_t* __restrict__ cnt, const int* __restrict__ tail, const uint8_t* __restrict__ tmode,
                      const T* __restrict__ wavg, const PfRows<T>& rw, const PfRowBits& rb, unsigned* bad) {
  auto held_at = [&](long long w, T* out) {
    const int c = cnt[w], m = tmode[w];
    const int n = c + (m == 2 ? 1 : 0);
    if (n <= 1) return false;
    for (int k = 0; k < n; k++)
      if (pf_held_id(ids, tail, g.nv, w, k, c, m) == j) {
        *out = wavg[(long long)k * g.nv + w];
        return true;
      }
    return false;
  };
  if (j >= 1) {
    T a;
    if (rb.bits) {
      int slot = (int)(pf_hash(j) & (unsigned)rb.mask), tries = 0;
      for (; tries <= rb.mask && rb.id[slot] != j; tries++, slot = (slot + 1) & rb.mask)
        if (rb.id[slot] == 0) tries = rb.mask + 1;
      if (tries <= rb.mask) {
        const unsigned* b = rb.bits + slot * rb.words;
        int w = z >> 5;
        unsigned m = b[w] & ((1u << (z & 31)) - 1u);
        while (!m && --w >= 0) m = b[w];
        if (m && held_at(v - z + (w << 5) + 31 - __clz(m), &a)) return a;
      }
    } else {
      const int slot = pf_row_find(rw.id, rw.mask[r], r, j);
      if (slot >= 0) {
        const long long at = (long long)r * PF_RH + slot;
        if (rw.zl[at] < z) return rw.val[at];
        const int zf = rw.zf[at];
        for (long long w = v - 1; w >= v - z + zf; w--)   // the latest writer before v lies in [zf, z)
          if (held_at(w, &a)) return a;
      }
    }
  }
  if (j < 1 || j > rw.table_len) { *bad |= PF_BAD_TABLE; return (T)0; }
  const int q = pf_row_before(rw.bm, rw.bl, rw.bm_w, rw.bl_w, j, r);
  if (q >= 0) {
    const int slot = pf_row_find(rw.id, rw.mask[q], q, j);
    if (slot >= 0) return rw.val[(long long)q * PF_RH + slot];
  }
  return rw.table[j - 1];
}

// New lists, one row of voxels (or, where rows are shorter than a block,
// several) per block.  The row's own earlier writers come from bitmaps in
// shared memory (the walk back along the row was half of the kernel's time).
// Later iterates of a substep (again) redo a voxel only when one of its
// averages or a table value it reads changed.  128^3, ms per launch: 3.4 before
// the tables, tiles and bitmaps, now 0.41 for a first iterate and 0.1 to 0.3
// for a later one.
template <typename T>
__global__ void __launch_bounds__(128) pf_update_kernel(PfView g, const int* __restrict__ ids, const T* __restrict__ phi,
                                                        const uint8_t* __restrict__ cnt, const int* __restrict__ nid,
                                                        const uint8_t* __restrict__ ncnt, const T* __restrict__ sten,
                                                        const int* __restrict__ tail,
                                                        const uint8_t* __restrict__ tmode, const T* __restrict__ wavg,
                                                        PfRows<T> rw, int init_gid, T mcoef, T kappa, T mwell, T edisl,
                                                        const uint8_t* __restrict__ ow_in, uint8_t* __restrict__ ow_out,
                                                        int again, const uint8_t* __restrict__ vdirty,
                                                        const uint8_t* __restrict__ idirty, int* __restrict__ ids2,
                                                        T* __restrict__ phi2, uint8_t* __restrict__ cnt2,
                                                        int per, int words, unsigned* __restrict__ word) {
  extern __shared__ int s_rows[];   // per row: PF_RH ids, PF_RH x words bits
  const long long nv = g.nv;
  const int lr = per > 1 ? threadIdx.x / g.d.n2 : 0;
  const int r = blockIdx.x * per + lr;
  const bool in = lr < per && r < g.rows;
  PfRowBits rb{nullptr, nullptr, 0, words};
  if (words) {
    const int row_ints = PF_RH * (1 + words);
    for (int q = 0; q < per && blockIdx.x * per + q < g.rows; q++) {
      const int rq = blockIdx.x * per + q, mask = rw.mask[rq];
      int* t = s_rows + q * row_ints;
      for (int i = threadIdx.x; i <= mask; i += blockDim.x) t[i] = rw.id[(long long)rq * PF_RH + i];
      for (int i = threadIdx.x; i < (mask + 1) * words; i += blockDim.x) t[PF_RH + i] = 0;
    }
    __syncthreads();
    if (in) {
      int* t = s_rows + lr * row_ints;
      rb.id = t;
      rb.bits = reinterpret_cast<unsigned*>(t + PF_RH);
      rb.mask = rw.mask[r];
      for (int z = per > 1 ? threadIdx.x - lr * g.d.n2 : threadIdx.x; z < g.d.n2; z += per > 1 ? g.d.n2 : blockDim.x) {
        const long long w = (long long)r * g.d.n2 + z;
        const int c = cnt[w], mode = tmode[w];
        const int n = c + (mode == 2 ? 1 : 0);
        if (n <= 1) continue;
        for (int k = 0; k < n; k++) {
          const int id = pf_held_id(ids, tail, nv, w, k, c, mode);
          if (id < 1) continue;
          int slot = (int)(pf_hash(id) & (unsigned)rb.mask);
          for (int tries = 0; tries <= rb.mask && t[slot] != id; tries++) slot = (slot + 1) & rb.mask;
          if (t[slot] == id) atomicOr(reinterpret_cast<unsigned*>(t + PF_RH) + slot * words + (z >> 5), 1u << (z & 31));
        }
      }
    }
    __syncthreads();
  }
  if (!in) return;
  for (int z = per > 1 ? threadIdx.x - lr * g.d.n2 : threadIdx.x; z < g.d.n2; z += per > 1 ? g.d.n2 : blockDim.x) {
  const long long v = (long long)r * g.d.n2 + z;
  const int nn = ncnt[v];
  if (again) {
    const int c = cnt[v], mode = tmode[v];
    const int n = c + (mode == 2 ? 1 : 0);
    bool redo = false;
    if (n > 1) {
      redo = vdirty[v] != 0;
      for (int a = 0; a < nn && !redo; a++) {
        const int j = nid[(long long)a * nv + v];
        if (j < 1 || j > rw.table_len || !idirty[j - 1]) continue;
        bool held = false;
        for (int k = 0; k < n; k++) held |= pf_held_id(ids, tail, nv, v, k, c, mode) == j;
        redo = !held;
      }
    }
    if (!redo) {
      ow_out[v] = ow_in[v];
      continue;
    }
  }
  int hid[PF_K + 1];
  T hph[PF_K + 1];
  const int n = pf_held<T>(g, ids, phi, cnt, tail, tmode, v, hid, hph);
  int oid[PF_K];
  T oph[PF_K];
  int on = 0;
  unsigned bad = 0;
  bool reset = false;
  if (n > 1) {
    T sum_rex = 0, sum1 = 0, hdef = 0;
    for (int k = 0; k < n; k++) {
      const T a = wavg[(long long)k * nv + v];
      if (a > (T)0) {
        const T e = hph[k];
        sum_rex = sum_rex + e * e;
        sum1 = sum1 + e * e * e * ((T)10.0 - (T)15.0 * e + (T)6.0 * e * e);
        hdef = hdef + (e * e * e * ((T)10.0 - (T)15.0 * e + (T)6.0 * e * e)) * a;
      }
    }
    for (int a = 0; a < nn; a++) {
      const int j = nid[(long long)a * nv + v];
      const T c = pf_read_local<T>(hid, hph, n, j);
      const T h = c * c * c * ((T)10.0 - (T)15.0 * c + (T)6.0 * c * c);
      const T dh = c * c * ((T)30.0 - (T)60.0 * c + (T)30.0 * c * c);
      const T st = a < PF_NS ? sten[(long long)a * nv + v]
                             : pf_sten_lists<T>(ids, phi, cnt, nv, Nbhd(g.d, r / g.d.n1, r % g.d.n1, z), j);
      const T lap = st - (T)4.5 * c;
      T ra;
      int k = 0;
      while (k < n && hid[k] != j) k++;
      if (k < n) ra = wavg[(long long)k * nv + v];
      else ra = pf_stale<T>(g, v, r, z, j, ids, cnt, tail, tmode, wavg, rw, rb, &bad);
      if (ra > (T)0) {
        const T val = c - mcoef * (mwell * (c * c * c - c + (T)3.0 * c * (sum_rex - c * c)) - kappa * lap +
                                   edisl * dh * ((sum1 - h) * ra - (hdef - h * ra)) / (sum1 * sum1));
        if (j > init_gid && c < (T)0.5 && val > (T)0.5) reset = true;
        if (val > (T)PF_KEEP) pf_write_local<T>(oid, oph, on, j, val, &bad);
      }
    }
  } else if (n == 1) {
    for (int a = 0; a < nn; a++) {
      const int j = nid[(long long)a * nv + v];
      pf_write_local<T>(oid, oph, on, j, pf_read_local<T>(hid, hph, n, j), &bad);
    }
  }
  cnt2[v] = (uint8_t)on;
  for (int k = 0; k < on; k++) {
    ids2[(long long)k * nv + v] = oid[k];
    phi2[(long long)k * nv + v] = oph[k];
  }
  ow_out[v] = (uint8_t)reset;
  if ((uint8_t)reset != ow_in[v]) word[0] = 1;   // any number of writers of the same value
  if (bad) atomicOr(&word[1], bad);
  }
}

// After the sweep, each id's last writer's value into the table.
template <typename T>
__global__ void pf_table_final_kernel(PfView g, PfRows<T> rw, T* __restrict__ table) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= rw.table_len) return;
  const int q = pf_row_before(rw.bm, rw.bl, rw.bm_w, rw.bl_w, j + 1, g.rows);
  if (q < 0) return;
  const int slot = pf_row_find(rw.id, rw.mask[q], q, j + 1);
  if (slot >= 0) table[j] = rw.val[(long long)q * PF_RH + slot];
}

// resets applied to the energy; grain id = first maximum, 0 when no eta > 0
// (Update_gID, src/pf_xrx.c:11-66)
template <typename T>
__global__ void pf_finish_kernel(PfView g, const int* __restrict__ ids, const T* __restrict__ phi,
                                 const uint8_t* __restrict__ cnt, const uint8_t* __restrict__ ow, T* __restrict__ energy,
                                 int* __restrict__ gid) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= g.nv) return;
  if (ow[v]) energy[v] = (T)100;
  T best = (T)0;
  int id = 0;
  const int c = cnt[v];
  for (int k = 0; k < c; k++) {
    const T e = phi[(long long)k * g.nv + v];
    if (best < e) { best = e; id = ids[(long long)k * g.nv + v]; }
  }
  gid[v] = id;
}

// ------------------------------------------------------------- launchers
static inline int nb(long long n, int t) { return (int)((n + t - 1) / t); }

cudaError_t launch_nucleation_candidates(const int dims[3], const int* grain, const uint8_t* crystal, const double* rho,
                                         double rho_nuc, double prob, uint64_t seed, uint64_t counter0,
                                         long long* out, unsigned long long* count, long long cap, cudaStream_t st) {
  Dims d{dims[0], dims[1], dims[2]};
  const long long nv = (long long)dims[0] * dims[1] * dims[2];
  nucleation_candidates_kernel<<<nb(nv, 256), 256, 0, st>>>(d, grain, crystal, rho, rho_nuc, prob, seed, counter0,
                                                            out, count, cap);
  return cudaGetLastError();
}

cudaError_t launch_paint_nuclei(const int dims[3], const long long* sites, int nn, int radius2, int first_id,
                                int* winner, int* grain, cudaStream_t st) {
  Dims d{dims[0], dims[1], dims[2]};
  const long long nv = (long long)dims[0] * dims[1] * dims[2];
  int r = 0;
  while ((r + 1) * (r + 1) <= radius2) r++;
  const int side = 2 * r + 1;
  const long long work = (long long)nn * side * side * side;
  if (work > 0 && radius2 >= 0) paint_mark_kernel<<<nb(work, 256), 256, 0, st>>>(d, sites, nn, r, radius2, winner);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  paint_apply_kernel<<<nb(nv, 256), 256, 0, st>>>(nv, first_id, winner, grain);
  return cudaGetLastError();
}

template <typename T>
cudaError_t pf_alloc(PfBuffers<T>& b, const int dims[3], int table_len) {
  memset(&b, 0, sizeof(b));
  const long long nv = (long long)dims[0] * dims[1] * dims[2];
  b.rows = dims[0] * dims[1];
  b.bm_w = b.rows / 32 + 1;   // a word past the last row, for the look-up from the end
  b.bl_w = (b.bm_w + 31) / 32 + 1;
  cudaError_t e = cudaSuccess;
  auto get = [&](void** p, size_t bytes) {
    if (e == cudaSuccess) e = cudaMalloc(p, bytes);
  };
  for (int i = 0; i < 2; i++) {
    get((void**)&b.ids[i], sizeof(int) * PF_K * nv);
    get((void**)&b.phi[i], sizeof(T) * PF_K * nv);
    get((void**)&b.cnt[i], (size_t)nv);
    get((void**)&b.ow[i], (size_t)nv);
  }
  get((void**)&b.upd, (size_t)nv);
  get((void**)&b.pred, sizeof(unsigned short) * nv);
  get((void**)&b.gid, sizeof(int) * nv);
  get((void**)&b.energy, sizeof(T) * nv);
  get((void**)&b.nid, sizeof(int) * PF_NM * nv);
  get((void**)&b.ncnt, (size_t)nv);
  get((void**)&b.sten, sizeof(T) * PF_NS * nv);
  get((void**)&b.tail, sizeof(int) * nv);
  get((void**)&b.tmode, (size_t)nv);
  get((void**)&b.wavg, sizeof(T) * (PF_K + 1) * nv);
  get((void**)&b.rw_id, sizeof(int) * PF_RH * (size_t)b.rows);
  get((void**)&b.rw_val, sizeof(T) * PF_RH * (size_t)b.rows);
  get((void**)&b.rw_zf, sizeof(int) * PF_RH * (size_t)b.rows);
  get((void**)&b.rw_zl, sizeof(int) * PF_RH * (size_t)b.rows);
  get((void**)&b.rw_mask, (size_t)b.rows);
  get((void**)&b.vdirty, (size_t)nv);
  get((void**)&b.word, sizeof(unsigned) * (2 + PF_UPD_GROUP));
  if (e == cudaSuccess) e = pf_table_reserve(b, table_len, nullptr);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  return e;
}

template <typename T>
void pf_free(PfBuffers<T>& b) {
  for (int i = 0; i < 2; i++) {
    cudaFree(b.ids[i]); cudaFree(b.phi[i]); cudaFree(b.cnt[i]); cudaFree(b.ow[i]);
  }
  cudaFree(b.upd); cudaFree(b.pred); cudaFree(b.gid); cudaFree(b.energy); cudaFree(b.nid); cudaFree(b.ncnt); cudaFree(b.sten); cudaFree(b.tail); cudaFree(b.tmode);
  cudaFree(b.wavg); cudaFree(b.rw_id); cudaFree(b.rw_val); cudaFree(b.rw_zf); cudaFree(b.rw_zl); cudaFree(b.rw_mask); cudaFree(b.vdirty);
  cudaFree(b.bm); cudaFree(b.bl); cudaFree(b.idirty);
  cudaFree(b.table); cudaFree(b.word);
  memset(&b, 0, sizeof(b));
}

template <typename T>
cudaError_t pf_table_reserve(PfBuffers<T>& b, int len, cudaStream_t st) {
  if (len <= b.table_cap) {
    b.table_len = b.table_cap;
    return cudaSuccess;
  }
  const int cap = len + 1024;
  T* t = nullptr;
  unsigned *bm = nullptr, *bl = nullptr;
  uint8_t* dirty = nullptr;
  cudaError_t e = cudaMalloc(&t, sizeof(T) * cap);
  if (e == cudaSuccess) e = cudaMalloc(&bm, sizeof(unsigned) * (size_t)b.bm_w * cap);
  if (e == cudaSuccess) e = cudaMalloc(&bl, sizeof(unsigned) * (size_t)b.bl_w * cap);
  if (e == cudaSuccess) e = cudaMalloc(&dirty, (size_t)cap);
  if (e == cudaSuccess) e = cudaMemsetAsync(t, 0, sizeof(T) * cap, st);
  if (e == cudaSuccess && b.table_cap > 0)
    e = cudaMemcpyAsync(t, b.table, sizeof(T) * b.table_cap, cudaMemcpyDeviceToDevice, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaFree(t);
    cudaFree(bm);
    cudaFree(bl);
    cudaFree(dirty);
    return e;
  }
  cudaFree(b.table);
  cudaFree(b.bm);
  cudaFree(b.bl);
  cudaFree(b.idirty);
  b.table = t;
  b.bm = bm;
  b.bl = bl;
  b.idirty = dirty;
  b.table_cap = b.table_len = cap;
  return cudaSuccess;
}

// fixed-point driver: the host reads the change counter after each iterate
static cudaError_t pf_read_counter(unsigned* word_d, unsigned* out, cudaStream_t st) {
  cudaError_t e = cudaMemcpyAsync(out, word_d, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e;
}

template <typename T>
cudaError_t launch_pf_relax(const int dims[3], const int* grain, const T* rho, int substeps, int init_gid,
                            const PfCoef& co, PfBuffers<T>& b, cudaStream_t st, int* launches, unsigned* bad) {
  PfView g{Dims{dims[0], dims[1], dims[2]}, (long long)dims[0] * dims[1] * dims[2], dims[0] * dims[1]};
  const long long nv = g.nv;
  int nl = 0;
  *bad = 0;
#define PF_CK(call)                        \
  do {                                     \
    cudaError_t e__ = (call);              \
    if (e__ != cudaSuccess) {              \
      *launches = nl;                      \
      return e__;                          \
    }                                      \
  } while (0)
#define PF_K_LAUNCH(...)          \
  do {                            \
    __VA_ARGS__;                  \
    nl++;                         \
    PF_CK(cudaGetLastError());    \
  } while (0)
  PF_CK(cudaMemsetAsync(b.word, 0, sizeof(unsigned) * 2, st));
  PF_K_LAUNCH(pf_init_kernel<T><<<nb(nv, 256), 256, 0, st>>>(g, grain, rho, b.ids[0], b.phi[0], b.cnt[0], b.energy, b.gid));
  int cur = 0;
  unsigned changed = 0;
  const int wtx = (dims[0] + PF_WT - 1) / PF_WT, wty = (dims[1] + PF_WT - 1) / PF_WT, wtz = (dims[2] + PF_WT - 1) / PF_WT;
  const int wtiles = wtx * wty * wtz;
  const int ntx = (dims[0] + PF_TX - 1) / PF_TX, nty = (dims[1] + PF_TY - 1) / PF_TY,
            ntz = (dims[2] + PF_TZ - 1) / PF_TZ;
  const int ntiles = ntx * nty * ntz;
  const size_t tsm = sizeof(T) * PF_TB * PF_HN;
  PF_CK(cudaFuncSetAttribute(pf_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tsm));
  // the update's rows per 128-thread block, and the words of a row's bitmaps:
  // none (the walk along the row) where they would pass 47 KB: z lines over 1472,
  // and lines of 5 voxels or fewer, of which a block takes 25 or more
  const int uper = dims[2] >= 128 ? 1 : 128 / dims[2];
  int uwords = (dims[2] + 31) / 32;
  size_t usm = sizeof(int) * (size_t)uper * PF_RH * (1 + uwords);
  if (usm > 47 * 1024) {
    uwords = 0;
    usm = 0;
  }
  for (int s = 0; s < substeps; s++) {
    const int* ids = b.ids[cur];
    const T* phi = b.phi[cur];
    const uint8_t* cnt = b.cnt[cur];
    PF_K_LAUNCH(pf_tile_kernel<T><<<ntiles, 256, tsm, st>>>(g, ids, phi, cnt, b.nid, b.ncnt, b.sten, nty, ntz,
                                                            b.word));
    // update flags to their fixed point (in place), in groups of passes
    PF_K_LAUNCH(pf_pred_kernel<T><<<nb(nv, 256), 256, 0, st>>>(g, ids, phi, cnt, b.nid, b.ncnt, b.pred));
    PF_CK(cudaMemsetAsync(b.upd, 0, (size_t)nv, st));
    for (long long it = 0; it <= nv; it += PF_UPD_GROUP) {
      unsigned* chg = b.word + 2;
      PF_CK(cudaMemsetAsync(chg, 0, sizeof(unsigned) * PF_UPD_GROUP, st));
      for (int k = 0; k < PF_UPD_GROUP; k++)
        PF_K_LAUNCH(pf_upd_kernel<<<nb(nv, 256), 256, 0, st>>>(g, b.pred, b.upd, chg, k));
      PF_CK(pf_read_counter(chg + PF_UPD_GROUP - 1, &changed, st));
      if (changed == 0) break;
    }
    PF_K_LAUNCH(pf_tail_kernel<T><<<nb(nv, 256), 256, 0, st>>>(g, ids, phi, cnt, b.nid, b.ncnt, b.upd, b.tail,
                                                                b.tmode, b.word));
    // values, with the stored-energy resets to their fixed point; the row
    // summaries' ids and bitmaps are those of the first iterate
    PF_CK(cudaMemsetAsync(b.ow[0], 0, (size_t)nv, st));
    const PfRows<T> rw{b.rw_id, b.rw_val, b.rw_zf, b.rw_zl, b.rw_mask, b.bm, b.bl, b.bm_w, b.bl_w, b.table,
                       b.table_len};
    int o = 0;
    for (long long it = 0; it <= nv; it++) {
      PF_CK(cudaMemsetAsync(b.word, 0, sizeof(unsigned), st));
      if (it > 0) {
        PF_CK(cudaMemsetAsync(b.vdirty, 0, (size_t)nv, st));
        PF_CK(cudaMemsetAsync(b.idirty, 0, (size_t)b.table_cap, st));
      }
      PF_K_LAUNCH(pf_window_kernel<T><<<wtiles, 256, 0, st>>>(g, ids, cnt, b.tail, b.tmode, grain, b.energy, b.ow[o],
                                                               it > 0 ? b.ow[1 - o] : nullptr, b.wavg, b.rw_id,
                                                               b.rw_val, b.rw_zl, b.rw_mask, b.vdirty, b.idirty,
                                                               b.table_len, wty, wtz));
      if (it == 0) {
        PF_CK(cudaMemsetAsync(b.bm, 0, sizeof(unsigned) * (size_t)b.bm_w * b.table_cap, st));
        PF_CK(cudaMemsetAsync(b.bl, 0, sizeof(unsigned) * (size_t)b.bl_w * b.table_cap, st));
        PF_K_LAUNCH(pf_rows_kernel<T><<<g.rows, 128, 0, st>>>(g, ids, cnt, b.tail, b.tmode, b.wavg, b.rw_id, b.rw_val,
                                                              b.rw_zf, b.rw_zl, b.rw_mask, b.bm, b.bl, b.bm_w, b.bl_w,
                                                              b.table_len, b.word));
      }
      PF_K_LAUNCH(pf_update_kernel<T><<<nb(g.rows, uper), 128, usm, st>>>(
          g, ids, phi, cnt, b.nid, b.ncnt, b.sten, b.tail, b.tmode, b.wavg, rw, init_gid, (T)co.mcoef, (T)co.kappa,
          (T)co.mwell, (T)co.edisl, b.ow[o], b.ow[1 - o], it > 0 ? 1 : 0, b.vdirty, b.idirty, b.ids[1 - cur],
          b.phi[1 - cur], b.cnt[1 - cur], uper, uwords, b.word));
      o = 1 - o;
      PF_CK(pf_read_counter(b.word, &changed, st));
      if (changed == 0) break;
    }
    if (b.table_len > 0)
      PF_K_LAUNCH(pf_table_final_kernel<T><<<nb(b.table_len, 256), 256, 0, st>>>(g, rw, b.table));
    cur = 1 - cur;
    PF_K_LAUNCH(pf_finish_kernel<T><<<nb(nv, 256), 256, 0, st>>>(g, b.ids[cur], b.phi[cur], b.cnt[cur], b.ow[o],
                                                                  b.energy, b.gid));
  }
  b.cur = cur;
  unsigned w[2] = {0, 0};
  PF_CK(cudaMemcpyAsync(w, b.word, sizeof(w), cudaMemcpyDeviceToHost, st));
  PF_CK(cudaStreamSynchronize(st));
  *bad = w[1];
  *launches = nl;
#undef PF_K_LAUNCH
#undef PF_CK
  return cudaSuccess;
}

template cudaError_t pf_alloc<float>(PfBuffers<float>&, const int*, int);
template cudaError_t pf_alloc<double>(PfBuffers<double>&, const int*, int);
template void pf_free<float>(PfBuffers<float>&);
template void pf_free<double>(PfBuffers<double>&);
template cudaError_t pf_table_reserve<float>(PfBuffers<float>&, int, cudaStream_t);
template cudaError_t pf_table_reserve<double>(PfBuffers<double>&, int, cudaStream_t);
template cudaError_t launch_pf_relax<float>(const int*, const int*, const float*, int, int, const PfCoef&,
                                            PfBuffers<float>&, cudaStream_t, int*, unsigned*);
template cudaError_t launch_pf_relax<double>(const int*, const int*, const double*, int, int, const PfCoef&,
                                             PfBuffers<double>&, cudaStream_t, int*, unsigned*);

}  // namespace mth

namespace mth {

// ------------------------------------------- microstructure update kernels
// rho = rho0 + rho_k * accumulated slip (crystal voxels; 0 in gas, which has
// no slip systems, as rho_tot in src/evolution.c:976-994)
template <typename TSt>
__global__ void drx_rho_kernel(Fields<TSt> f, double rho0, double rho_k, double* __restrict__ rho_d,
                               TSt* __restrict__ rho_t) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= f.nv) return;
  const double r = f.phase[v] == 0 ? rho0 + rho_k * (double)f.gamacum[v] : 0.0;
  rho_d[v] = r;
  rho_t[v] = (TSt)r;
}

// Per recrystallised grain k: its voxels after the relaxation (cnt[k]) and
// those of them that joined it in this step (cnt[n_drx + k]), for the
// "< 1 % grew" rule of src/integrated.c:1537-1582.
template <typename TSt>
__global__ void drx_count_kernel(Fields<TSt> f, const int* __restrict__ grain, const int* __restrict__ grain_prev,
                                 const int* __restrict__ gid_new, int first_drx_id, int n_drx,
                                 int* __restrict__ cnt) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= f.nv) return;
  const int gn = gid_new[v] != 0 ? gid_new[v] : grain[v];
  const int k = gn - first_drx_id;
  if (k < 0 || k >= n_drx) return;
  atomicAdd(&cnt[k], 1);
  if (gn != grain_prev[v] && f.phase[v] == 0) atomicAdd(&cnt[n_drx + k], 1);
}

// Voxels whose relaxed grain id differs from the id before this step's
// nucleation and belongs to a recrystallised grain become part of it: the
// treatment of growth==1 voxels after PF_XRX (src/evolution.c:1120-1200):
// stress zeroed, dislocation content reset (accumulated slip and CRSS back
// to the initial state), orientation and stiffness of the new grain.  Other
// id changes only relabel the voxel (src/integrated.c:1613-1615).
template <typename TSt>
__global__ void drx_update_kernel(Fields<TSt> f, int* __restrict__ grain, const int* __restrict__ grain_prev,
                                  const int* __restrict__ gid_new, int first_drx_id, int n_drx,
                                  const double* __restrict__ drx_rot, const int* __restrict__ drx_class, double tau0f,
                                  int nsys, const int* __restrict__ cnt) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = f.nv;
  if (v >= P) return;
  // a voxel the phase field left without a positive eta (grain id 0, where
  // the reference stops on GetStatistics' assert, src/pf_xrx.c:1383-1386)
  // keeps the grain it had
  const int gn = gid_new[v] != 0 ? gid_new[v] : grain[v];
  grain[v] = gn;
  if (gn == grain_prev[v] || f.phase[v] != 0) return;
  const int k = gn - first_drx_id;
  if (k < 0 || k >= n_drx) return;
  // a grain whose joining voxels are under 1 % of it (integer percent 0,
  // src/integrated.c:1562-1577) resets none of them: they take its id only
  if ((long long)cnt[n_drx + k] * 100 / cnt[k] == 0) return;
  for (int i = 0; i < 6; i++) f.sig[i * P + v] = (TSt)0;
  f.gamacum[v] = (TSt)0;
  for (int s = 0; s < NSYS; s++) f.crss[s * P + v] = (TSt)(s < nsys ? tau0f : 0.0);
  for (int i = 0; i < 9; i++) f.rot[i * P + v] = (TSt)drx_rot[9 * k + i];
  const_cast<int*>(f.eclass)[v] = drx_class[k];
}

__global__ void class_histogram_kernel(long long nv, const uint8_t* __restrict__ crystal, const int* __restrict__ eclass,
                                       unsigned long long* __restrict__ hist) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv || !crystal[v]) return;
  atomicAdd(&hist[eclass[v]], 1ULL);
}

cudaError_t launch_drx_rho(int mixed, const void* fields, double rho0, double rho_k, double* rho_d, void* rho_t,
                           cudaStream_t st) {
  if (mixed) {
    const Fields<float>& f = *static_cast<const Fields<float>*>(fields);
    drx_rho_kernel<float><<<nb(f.nv, 256), 256, 0, st>>>(f, rho0, rho_k, rho_d, static_cast<float*>(rho_t));
  } else {
    const Fields<double>& f = *static_cast<const Fields<double>*>(fields);
    drx_rho_kernel<double><<<nb(f.nv, 256), 256, 0, st>>>(f, rho0, rho_k, rho_d, static_cast<double*>(rho_t));
  }
  return cudaGetLastError();
}

cudaError_t launch_drx_update(int mixed, const void* fields, int* grain, const int* grain_prev, const int* gid_new,
                              int first_drx_id, int n_drx, const double* drx_rot, const int* drx_class, double tau0f,
                              int nsys, int* cnt, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int) * 2 * (size_t)n_drx, st);
  if (e != cudaSuccess) return e;
  if (mixed) {
    const Fields<float>& f = *static_cast<const Fields<float>*>(fields);
    drx_count_kernel<float><<<nb(f.nv, 256), 256, 0, st>>>(f, grain, grain_prev, gid_new, first_drx_id, n_drx, cnt);
    drx_update_kernel<float><<<nb(f.nv, 256), 256, 0, st>>>(f, grain, grain_prev, gid_new, first_drx_id, n_drx, drx_rot,
                                                            drx_class, tau0f, nsys, cnt);
  } else {
    const Fields<double>& f = *static_cast<const Fields<double>*>(fields);
    drx_count_kernel<double><<<nb(f.nv, 256), 256, 0, st>>>(f, grain, grain_prev, gid_new, first_drx_id, n_drx, cnt);
    drx_update_kernel<double><<<nb(f.nv, 256), 256, 0, st>>>(f, grain, grain_prev, gid_new, first_drx_id, n_drx,
                                                             drx_rot, drx_class, tau0f, nsys, cnt);
  }
  return cudaGetLastError();
}

cudaError_t launch_class_histogram(long long nv, const uint8_t* crystal, const int* eclass, unsigned long long* hist,
                                   cudaStream_t st) {
  class_histogram_kernel<<<nb(nv, 256), 256, 0, st>>>(nv, crystal, eclass, hist);
  return cudaGetLastError();
}

// ------------------------------------------ PF <-> mechanical grid transfer
// InterpolateGrid / InterpolateGID (src/integrated.c:496-760) and the
// coarse-graining of gID_new (src/integrated.c:821-860): node coordinates
// x = i/(N-1) on [0,1], source cell floor(x/dx), dx = 1/(Ns-1), upper corner
// clamped to the last node (the reference aborts when rounding puts a node
// past the last source node; here the last cell is used).  Same operations
// in the same order as the oracle (this file is compiled without FMA
// contraction), so FP64 results are bit-identical.
__device__ __forceinline__ void axis_pos(int i, int nd, int ns, int& i0, int& i1, double& s) {
  if (nd < 2 || ns < 2) { i0 = 0; i1 = 0; s = 0.0; return; }
  const double dxd = 1.0 / (nd - 1), dxs = 1.0 / (ns - 1);
  const double x = 0.0 + (double)i * dxd;
  int ix = (int)floor(x / dxs);
  if (ix > ns - 1) ix = ns - 1;
  if (ix < 0) ix = 0;
  s = x / dxs - (double)ix;
  i0 = ix;
  i1 = ix + 1 < ns ? ix + 1 : ns - 1;
}

// integer field: value at the nearest of the eight corners, first minimum in
// the order 000,100,110,010,001,101,111,011 (TrilinearInterpolationINT)
__global__ void resample_nearest_kernel(Dims ds, const int* __restrict__ src, Dims dd, int* __restrict__ dst) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nv = (long long)dd.n0 * dd.n1 * dd.n2;
  if (v >= nv) return;
  const int k = (int)(v % dd.n2), j = (int)((v / dd.n2) % dd.n1), i = (int)(v / ((long long)dd.n1 * dd.n2));
  int x0, x1, y0, y1, z0, z1;
  double sx, sy, sz;
  axis_pos(i, dd.n0, ds.n0, x0, x1, sx);
  axis_pos(j, dd.n1, ds.n1, y0, y1, sy);
  axis_pos(k, dd.n2, ds.n2, z0, z1, sz);
  double dist[8];
  dist[0] = sx * sx + sy * sy + sz * sz;
  dist[1] = (1 - sx) * (1 - sx) + sy * sy + sz * sz;
  dist[2] = (1 - sx) * (1 - sx) + (1 - sy) * (1 - sy) + sz * sz;
  dist[3] = sx * sx + (1 - sy) * (1 - sy) + sz * sz;
  dist[4] = sx * sx + sy * sy + (1 - sz) * (1 - sz);
  dist[5] = (1 - sx) * (1 - sx) + sy * sy + (1 - sz) * (1 - sz);
  dist[6] = (1 - sx) * (1 - sx) + (1 - sy) * (1 - sy) + (1 - sz) * (1 - sz);
  dist[7] = sx * sx + (1 - sy) * (1 - sy) + (1 - sz) * (1 - sz);
  const int cx[8] = {x0, x1, x1, x0, x0, x1, x1, x0};
  const int cy[8] = {y0, y0, y1, y1, y0, y0, y1, y1};
  const int cz[8] = {z0, z0, z0, z0, z1, z1, z1, z1};
  int m = 0;
#pragma unroll
  for (int c = 1; c < 8; c++)
    if (dist[m] > dist[c]) m = c;
  dst[v] = src[((long long)cx[m] * ds.n1 + cy[m]) * ds.n2 + cz[m]];
}

// double field: trilinear interpolation, terms in the reference's order
// (TrilinearInterpolation); stored as TO
template <typename TO>
__global__ void resample_trilinear_kernel(Dims ds, const double* __restrict__ src, Dims dd, TO* __restrict__ dst) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long nv = (long long)dd.n0 * dd.n1 * dd.n2;
  if (v >= nv) return;
  const int k = (int)(v % dd.n2), j = (int)((v / dd.n2) % dd.n1), i = (int)(v / ((long long)dd.n1 * dd.n2));
  int x0, x1, y0, y1, z0, z1;
  double sx, sy, sz;
  axis_pos(i, dd.n0, ds.n0, x0, x1, sx);
  axis_pos(j, dd.n1, ds.n1, y0, y1, sy);
  axis_pos(k, dd.n2, ds.n2, z0, z1, sz);
  auto V = [&](int a, int b, int c) { return src[((long long)a * ds.n1 + b) * ds.n2 + c]; };
  const double r = V(x0, y0, z0) * (1.0 - sx) * (1.0 - sy) * (1.0 - sz) + V(x1, y0, z0) * sx * (1.0 - sy) * (1.0 - sz) +
                   V(x0, y1, z0) * sy * (1.0 - sx) * (1.0 - sz) + V(x0, y0, z1) * sz * (1.0 - sy) * (1.0 - sx) +
                   V(x1, y0, z1) * sx * (1.0 - sy) * sz + V(x0, y1, z1) * sy * (1.0 - sx) * sz +
                   V(x1, y1, z0) * sx * (1.0 - sz) * sy + V(x1, y1, z1) * sx * sy * sz;
  dst[v] = (TO)r;
}

cudaError_t launch_resample_nearest(const int ns[3], const int* src, const int nd[3], int* dst, cudaStream_t st) {
  const long long nv = (long long)nd[0] * nd[1] * nd[2];
  resample_nearest_kernel<<<nb(nv, 256), 256, 0, st>>>(Dims{ns[0], ns[1], ns[2]}, src, Dims{nd[0], nd[1], nd[2]}, dst);
  return cudaGetLastError();
}

cudaError_t launch_resample_trilinear(const int ns[3], const double* src, const int nd[3], void* dst, int to_float,
                                      cudaStream_t st) {
  const long long nv = (long long)nd[0] * nd[1] * nd[2];
  if (to_float)
    resample_trilinear_kernel<float><<<nb(nv, 256), 256, 0, st>>>(Dims{ns[0], ns[1], ns[2]}, src,
                                                                  Dims{nd[0], nd[1], nd[2]}, static_cast<float*>(dst));
  else
    resample_trilinear_kernel<double><<<nb(nv, 256), 256, 0, st>>>(Dims{ns[0], ns[1], ns[2]}, src,
                                                                   Dims{nd[0], nd[1], nd[2]}, static_cast<double*>(dst));
  return cudaGetLastError();
}

// rotation matrices (9 components, component-major fields) of the parent
// voxels of the nn nuclei, as double, nucleus-major: out[k*9 + i]
template <typename TSt>
__global__ void gather_rot_kernel(const TSt* __restrict__ rot, long long nv, const long long* __restrict__ sites, int nn,
                                  double* __restrict__ out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 9LL * nn) return;
  const long long k = t / 9;
  const int i = (int)(t - 9 * k);
  out[t] = (double)rot[(size_t)i * nv + sites[k]];
}

cudaError_t launch_gather_rot(int mixed, const void* rot, long long nv, const long long* sites, int nn, double* out,
                              cudaStream_t st) {
  if (nn <= 0) return cudaSuccess;
  if (mixed)
    gather_rot_kernel<float><<<nb(9LL * nn, 256), 256, 0, st>>>(static_cast<const float*>(rot), nv, sites, nn, out);
  else
    gather_rot_kernel<double><<<nb(9LL * nn, 256), 256, 0, st>>>(static_cast<const double*>(rot), nv, sites, nn, out);
  return cudaGetLastError();
}

}  // namespace mth
