// Wall-force pressure of slit systems (ForceField::CalcPressureForceLJELSlit,
// pressure.cc:404-488) on the device: the per-item arithmetic of
// slit_pressure.h in four launches.
//
//  k_slit_pairs  (site, bead) pairs -- LJ and real-space Ewald z forces -- a
//                thread per bead against a chunk of sites staged in shared
//                memory, so a bead's molecule, kind and type mix are found once
//                and not per pair; then the wall force of every system bead;
//                each block writes six partial sums
//  k_slit_sk     the five group structure factors over (k unit tile) x (bead
//                group) blocks from per-axis phase tables, two vectors (+-nz)
//                per four multiply-adds
//  k_slit_recip  the bead groups' parts added in order, and the reciprocal z
//                forces of every k; each block writes three partial sums
//  k_slit_sum    one block adds the partials in a fixed order: the result is
//                run-to-run identical
//
// Bound: the FP64 pipe (about 75 operations per pair within r_c, 5 per unit
// and charged bead), spread over every SM. A thread per k over all beads with
// a sincos each kept 6 of 152 SMs busy for 6.6 ms on a 1,391-vector,
// 3,200-bead brush; the tables need one sincos per bead and axis. The whole
// evaluation takes 0.18 ms there (7.1 ms before).
#include <algorithm>

#include "device_common.cuh"
#include "engine.h"
#include "kspace64.cuh"
#include "slit_pressure.h"

namespace plum {

namespace {

constexpr int kSlitThreads = 256;

template <int NQ>
__device__ __forceinline__ void block_sums(double* v, double* out) {
  __shared__ double red[NQ][kSlitThreads / 32];
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < NQ; q++) {
    double x = v[q];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (l == 0) red[q][w] = x;
  }
  __syncthreads();
  if (threadIdx.x < NQ) {
    double t = 0.0;
    for (int i = 0; i < kSlitThreads / 32; i++) t += red[threadIdx.x][i];
    out[threadIdx.x] = t;
  }
}

// The real-space force factor from the FP64 g(u) table (directly below it).
struct SlitTab {
  const double* tab;
  double alpha, scale;  // scale = alpha^{3/2}
  __device__ __forceinline__ double operator()(double d2) const {
    const long long bits = __double_as_longlong(alpha * d2);
    return bits >= kH64LoBits ? scale * h64_tab(tab, bits) : SlitErfc{alpha}(d2);
  }
};

// A warp takes 32 sites of one wall (a lane each) against the beads of its
// block's tile, one at a time: the bead's kind is the same for every lane, and
// as the sites of a wall share their z, so is the test that drops images
// beyond r_c along z (half the pairs of a slit wider than r_c). With a bead
// per lane the lanes' z differ and a warp ran nearly every image: 207 us
// against 89 us on 128 sites x 3,200 beads (with the force's one table load in
// place of an exponential, an erfc and two divisions).
// Block (x, y): beads bead0 + x per .. of 32-site group y. The second wall's
// sites meet system beads only (pressure.cc:419-455).
__global__ void __launch_bounds__(kSlitThreads)
    k_slit_pairs(const SlitPressParams S, const DevBuffers B, SlitGrid G, int wall_b0,
                 const double* __restrict__ gtab, double* part) {
  __shared__ double s_b[kSlitThreads][4];
  __shared__ int s_kid[kSlitThreads], s_t[kSlitThreads];
  __shared__ SlitMix s_mix[kSlitMaxTypes][kSlitMaxTypes];
  for (int i = threadIdx.x; i < S.n_type * S.n_type; i += kSlitThreads)
    s_mix[i / S.n_type][i % S.n_type] = slit_mix(S, i / S.n_type, i % S.n_type);
  double acc[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int c0 = G.bead0 + blockIdx.x * G.per, cn = min(G.per, S.n_bead - c0);
  if ((int)threadIdx.x < cn) {
    const int b = c0 + threadIdx.x;
    const double4_32a p = B.pos[b];
    s_b[threadIdx.x][0] = p.x, s_b[threadIdx.x][1] = p.y;
    s_b[threadIdx.x][2] = p.z, s_b[threadIdx.x][3] = p.w;
    s_t[threadIdx.x] = B.type[b];
    const int j = slit_mol_of(B.mol_start, S.n_mol, b);
    const int kid = j >= S.phantom ? (B.mol_start[j + 1] - B.mol_start[j] > 1 ? 1 : 0) : 2;
    s_kid[threadIdx.x] = kid;
    if (blockIdx.y == 0 && S.use_ext && b >= wall_b0)
      slit_add(acc, 0, kid, 0.5 * slit_wall_force(S, p.z, B.type[b]));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, half = S.phantom / 2;
  const bool second = (int)blockIdx.y >= G.groups1;
  const int w = (second ? half + 32 * ((int)blockIdx.y - G.groups1) : 32 * (int)blockIdx.y) + lane;
  if (w < G.sites && (second || w < half)) {
    const double4_32a p = B.pos[B.mol_start[w]];
    const double pw[4] = {p.x, p.y, p.z, p.w};
    const int tw = B.type[B.mol_start[w]];
    const SlitTab term{gtab, S.alpha, S.alpha * sqrt(S.alpha)};
    for (int i = threadIdx.x >> 5; i < cn; i += kSlitThreads / 32) {
      const int kid = s_kid[i];
      if (second && kid == 2) continue;
      double v[2] = {0.0, 0.0};
      slit_site_force(S, pw, s_b[i], s_mix[s_t[i]][tw], term, v);
      const double C = kid == 2 ? -1.0 : (second ? 0.5 : -0.5);
      slit_add(acc, 0, kid, C * v[0]);
      slit_add(acc, 3, kid, C * v[1]);
    }
  }
  block_sums<6>(acc, part + 6 * ((size_t)blockIdx.y * gridDim.x + blockIdx.x));
}

// The group sums (KUnit's A, B) of kSlitPer units per thread over one part of
// the beads, written as S(k) parts [bead part][5][n_k], and which groups the
// part has (mask[bead part]; the other groups' slots are neither written nor
// read). A bead's group is the same for every thread and beads of a kind are
// consecutive, so one pair of sums runs until the group changes and is then
// added to the group's slots: five predicated sums per unit kept the FP64 pipe
// on four idle ones (21 operations per unit and bead instead of 5, 131 us
// against 52 us). A block takes 768 units, so that a usual brush's k-set
// is one tile and each bead's phase tables are built once; the tables' tasks
// run axis by axis, so that a warp's lanes share the length of their recursion.
constexpr int kSlitPer = 2;
constexpr int kSlitSkThreads = 384;

__global__ void __launch_bounds__(kSlitSkThreads, 1)
    k_slit_sk(const SlitPressParams S, const DevParams P, const DevBuffers B, int groups,
              double2* part, int* mask) {
  extern __shared__ __align__(32) unsigned char smem[];
  double2* tabs = reinterpret_cast<double2*>(smem);
  __shared__ int s_g[32];
  const int per_g = (S.n_bead + groups - 1) / groups;
  const int b0 = blockIdx.y * per_g, b1 = min(S.n_bead, b0 + per_g);
  KUnit un[kSlitPer];
  bool mine[kSlitPer], col[kSlitPer];
  double2 A[kSlitPer], Bs[kSlitPer];
#pragma unroll
  for (int q = 0; q < kSlitPer; q++) {
    const int u = (blockIdx.x * kSlitSkThreads + threadIdx.x) * kSlitPer + q;
    mine[q] = u < P.n_ku;
    un[q] = mine[q] ? B.ku[u] : KUnit{0, 0, 0, 0, -1, -1};
    col[q] = q == 0 || un[q].nx != un[q - 1].nx || un[q].ny != un[q - 1].ny;
    A[q] = Bs[q] = make_double2(0.0, 0.0);
  }
  int run = 0, seen = 0;  // the current beads' groups, the groups written so far
  double2* const out = part + (size_t)blockIdx.y * 5 * P.n_k;
  auto flush = [&]() {
    if (run == 0) return;
#pragma unroll
    for (int q = 0; q < kSlitPer; q++) {
      const double2 v[2] = {unit_plus(A[q], Bs[q]), unit_minus(A[q], Bs[q])};
      const int at[2] = {un[q].kp, un[q].km};
      for (int r = 0; r < 5; r++)
        if (run >> r & 1)
          for (int h = 0; h < 2; h++)
            if (at[h] >= 0) {
              double2* o = out + (size_t)r * P.n_k + at[h];
              const double2 old = seen >> r & 1 ? *o : make_double2(0.0, 0.0);
              *o = make_double2(old.x + v[h].x, old.y + v[h].y);
            }
      A[q] = Bs[q] = make_double2(0.0, 0.0);
    }
    seen |= run;
  };
  for (int c0 = b0; c0 < b1; c0 += P.kchunk_sk) {
    const int cnt = min(P.kchunk_sk, b1 - c0);
    __syncthreads();  // the previous chunk is consumed
    if (threadIdx.x < cnt)
      s_g[threadIdx.x] =
          B.pos[c0 + threadIdx.x].w != 0.0 ? slit_bead_groups(S, B.mol_start, c0 + threadIdx.x) : 0;
    for (int t = threadIdx.x; t < 3 * 32; t += kSlitSkThreads)
      if ((t & 31) < cnt)
        build_axis_table(P, B.pos[c0 + (t & 31)], t >> 5, tabs + (t & 31) * P.kper);
    __syncthreads();
    for (int i = 0; i < cnt; i++) {
      const int g = s_g[i];
      if (!g) continue;
      if (g != run) {
        flush();
        run = g;
      }
      const double2* tab = tabs + i * P.kper;
      double2 xy = make_double2(0.0, 0.0);
#pragma unroll
      for (int q = 0; q < kSlitPer; q++) {
        if (!mine[q]) continue;
        if (col[q]) xy = unit_xy(P, tab, un[q].nx, un[q].ny);
        unit_add(xy, tab[P.koff[2] + un[q].nz], A[q], Bs[q]);
      }
    }
  }
  flush();
  if (blockIdx.x == 0 && threadIdx.x == 0) mask[blockIdx.y] = seen;
}

constexpr int kSlitK = 8;  // k vectors per block, 32 threads each

__global__ void __launch_bounds__(kSlitThreads)
    k_slit_recip(const SlitPressParams S, const DevParams P, const DevBuffers B, int groups,
                 const double2* sk_part, const int* mask, double* part) {
  __shared__ double2 s_sum[kSlitThreads / kSlitK][5][kSlitK];
  const int l = threadIdx.x % kSlitK, sl = threadIdx.x / kSlitK;
  const int k = blockIdx.x * kSlitK + l;
  const bool on = k < P.n_k;
  double2 s[5];
#pragma unroll
  for (int r = 0; r < 5; r++) s[r] = make_double2(0.0, 0.0);
  if (on)
    for (int g = sl; g < groups; g += kSlitThreads / kSlitK) {
      const int m = mask[g];
#pragma unroll
      for (int r = 0; r < 5; r++)
        if (m >> r & 1) {
          const double2 v = sk_part[((size_t)g * 5 + r) * P.n_k + k];
          s[r].x += v.x;
          s[r].y += v.y;
        }
    }
#pragma unroll
  for (int r = 0; r < 5; r++) s_sum[sl][r][l] = s[r];
  __syncthreads();
  // the 32 slices of each (group, vector), added in order by a thread each
  if (threadIdx.x < 5 * kSlitK) {
    const int r = threadIdx.x / kSlitK, v = threadIdx.x % kSlitK;
    double2 t = s_sum[0][r][v];
    for (int q = 1; q < kSlitThreads / kSlitK; q++) {
      t.x += s_sum[q][r][v].x;
      t.y += s_sum[q][r][v].y;
    }
    s_sum[0][r][v] = t;
  }
  __syncthreads();
  double o[3] = {0.0, 0.0, 0.0};
  if (on && sl == 0) {
    double re[5], im[5];
    for (int r = 0; r < 5; r++) {
      re[r] = s_sum[0][r][l].x;
      im[r] = s_sum[0][r][l].y;
    }
    slit_k_terms(B.kn[k].z * P.kunit[2], B.kw[k], re, im, o);
  }
  const double pre = slit_recip_prefactor(S);
  for (int q = 0; q < 3; q++) o[q] *= pre;
  block_sums<3>(o, part + 3 * (size_t)blockIdx.x);
}

// out6 = {LJ ion, LJ polymer, LJ wall-wall, Ewald ion, Ewald polymer, Ewald
// wall-wall}: the increments of p_tensor[6..11] before the reference's
// wall-wall guard.
__global__ void __launch_bounds__(kSlitThreads)
    k_slit_sum(const double* part, int n1, const double* part3, int n2, double* out6) {
  double v[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int i = threadIdx.x; i < n1; i += kSlitThreads)
    for (int q = 0; q < 6; q++) v[q] += part[6 * (size_t)i + q];
  for (int i = threadIdx.x; i < n2; i += kSlitThreads)
    for (int q = 0; q < 3; q++) v[3 + q] += part3[3 * (size_t)i + q];
  block_sums<6>(v, out6);
}

}  // namespace

// Pair kernel: bead tiles x 32-site groups of each wall, about two blocks per
// SM (a tile is a multiple of the block's eight warps). k kernel: unit tiles x
// bead groups, one block per SM; fewer groups where that would leave a group
// under 8 beads (its tables then cost more than its sums).
SlitGrid slit_grid(const SlitPressParams& S, const DevParams& P, long long n_pair, int bead0) {
  SlitGrid G;
  G.bead0 = bead0;
  G.sites = n_pair > 0 ? S.phantom : 0;
  G.groups1 = (G.sites / 2 + 31) / 32;
  G.groups = std::max(1, G.groups1 + (G.sites - G.sites / 2 + 31) / 32);
  const int nb = std::max(1, S.n_bead - bead0);
  const long long per = ((long long)nb * G.groups + pair_grid() - 1) / pair_grid();
  G.per = (int)std::min<long long>(kSlitThreads, (per + 7) / 8 * 8);
  G.tiles = (nb + G.per - 1) / G.per;
  G.n1 = G.tiles * G.groups;
  G.ktiles = G.kgroups = G.n2 = 0;
  if (S.use_ewald && S.phantom > 0 && P.n_k > 0) {
    const int units = kSlitSkThreads * kSlitPer;
    G.ktiles = (P.n_ku + units - 1) / units;
    G.kgroups = std::max(1, std::min((S.n_bead + 7) / 8, pair_grid() / 2 / G.ktiles));
    G.n2 = (P.n_k + kSlitK - 1) / kSlitK;
  }
  G.sk_off = 6LL * G.n1;  // even: the S(k) parts are double2
  G.part3_off = G.sk_off + 10LL * G.kgroups * P.n_k;
  G.mask_off = G.part3_off + 3LL * G.n2;
  G.out_off = G.mask_off + G.kgroups;  // room for kgroups ints
  G.total = G.out_off + 6;
  return G;
}

void launch_slit_pressure(const SlitPressParams& S, const DevParams& P, const DevBuffers& B,
                          const SlitGrid& G, int wall_b0, const double* gtab, double* scratch,
                          cudaStream_t s) {
  k_slit_pairs<<<dim3(G.tiles, G.groups), kSlitThreads, 0, s>>>(S, B, G, wall_b0, gtab, scratch);
  if (G.n2 > 0) {
    static OncePerDevice once;
    allow_smem(once, k_slit_sk, kKTableBytes);
    double2* sk = reinterpret_cast<double2*>(scratch + G.sk_off);
    int* mask = reinterpret_cast<int*>(scratch + G.mask_off);
    k_slit_sk<<<dim3(G.ktiles, G.kgroups), kSlitSkThreads,
                (size_t)P.kchunk_sk * P.kper * sizeof(double2), s>>>(S, P, B, G.kgroups, sk, mask);
    k_slit_recip<<<G.n2, kSlitThreads, 0, s>>>(S, P, B, G.kgroups, sk, mask,
                                               scratch + G.part3_off);
  }
  k_slit_sum<<<1, kSlitThreads, 0, s>>>(scratch, G.n1, scratch + G.part3_off, G.n2,
                                        scratch + G.out_off);
}

}  // namespace plum
