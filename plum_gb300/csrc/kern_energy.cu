// FP64 energy kernels of the plain form.
//
//  k_delta64   energy difference of the pending move (one fused launch):
//                pairs        every (moved, other) pair: LJ
//                             (potential_truncated_lj.cc:49-85) and Ewald real
//                             space (potential_ewald_coul.cc:134-164) at trial
//                             minus current positions; moved x moved pairs once
//                             (potential_pair.cc:156-175, potential_ewald.cc:436-476)
//                k blocks     dS(k) and the |S|^2 change of a run of k units over
//                             all moved beads, which equals the reference's
//                             pairwise PairEnergyRepl sum
//                             (potential_ewald_coul.cc:198-225) on the same k-set
//              Every block writes its own partial sums; the serial step adds them
//              in a fixed order, so results are run-to-run identical.
//  k_total64*  all i<j pairs from scratch (tile pairs)
//  k_sk64      S(k) from scratch (k unit tile x bead group partials)
//  k_misc64    bonds, walls, self energy, self images, sum q z
//
// Phases e^{i k.r} come from per-axis tables e^{i n theta_a}, n = 0..kmax,
// built by complex recursion from one exponential per bead and axis, with theta_a
// = 2 kPi w_a / L_a on coordinates wrapped into the primary cell (periodic
// axes). This replaces the reference's cos(k.r) per pair and k.
#include <algorithm>
#include <cmath>
#include <cstdio>

#include "engine.h"
#include "device_common.cuh"
#include "fix_device.cuh"
#include "kspace64.cuh"

namespace plum {

// sum over periodic images with 0 < |d + n L| <= r_c of erfc(sqrt(a) r)/r.
// An image whose single component already exceeds r_c cannot be inside the
// cut-off, so those shifts are skipped per axis.
__device__ __forceinline__ double real_images64(const DevParams& P, double dx,
                                                double dy, double dz) {
  double e = 0.0;
  const double rc = P.real_cut;
  const double rc2 = rc * rc;
  if (P.single_image) {
    // r_c <= L/2 on every axis: any other image has a component >= L/2 >= r_c
    // (ties at exactly L/2 are a set of measure zero)
    const double r2 = dx * dx + dy * dy + dz * dz;
    if (r2 > 0.0 && r2 <= rc2) e = real_term64(P, r2);
    return e;
  }
  for (int a = -P.real_cell[0]; a <= P.real_cell[0]; a++) {
    double x = dx + a * P.ebox[0];
    if (fabs(x) > rc) continue;
    for (int b = -P.real_cell[1]; b <= P.real_cell[1]; b++) {
      double y = dy + b * P.ebox[1];
      if (fabs(y) > rc) continue;
      for (int c = -P.real_cell[2]; c <= P.real_cell[2]; c++) {
        double z = dz + c * P.ebox[2];
        if (fabs(z) > rc) continue;
        const double r2 = x * x + y * y + z * z;
        if (r2 > 0.0 && r2 <= rc2) e += real_term64(P, r2);
      }
    }
  }
  return e;
}

// LJ and real-space Ewald of bead a (type ta) with bead b (type tb).
__device__ __forceinline__ void pair64(const DevParams& P, double4_32a a, int ta,
                                       double4_32a b, int tb, double& lj, double& re) {
  double dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
  if (P.same_wrap) {
    // the pair box wraps every periodic axis as the Ewald box does: one
    // minimum-image vector for both terms
    const double x = wrap_d(dx, P.box[0], P.inv_box[0]);
    const double y = wrap_d(dy, P.box[1], P.inv_box[1]);
    const double z = P.npbc > 2 ? wrap_d(dz, P.box[2], P.inv_box[2]) : dz;
    const double r2 = x * x + y * y + z * z;
    if (P.use_pair && r2 < P.lj_max2) lj += lj64(P, ta * P.n_type + tb, r2);
    if (P.use_ewald) {
      const double qq = a.w * b.w;
      if (qq != 0.0) re += P.lB * qq * real_images64(P, x, y, z);
    }
    return;
  }
  if (P.use_pair) {
    double x = wrap_d(dx, P.box[0], P.inv_box[0]);
    double y = wrap_d(dy, P.box[1], P.inv_box[1]);
    double z = P.npbc > 2 ? wrap_d(dz, P.box[2], P.inv_box[2]) : dz;
    lj += lj64(P, ta * P.n_type + tb, x * x + y * y + z * z);
  }
  if (P.use_ewald) {
    double qq = a.w * b.w;
    if (qq != 0.0) {
      double x = wrap_d(dx, P.ebox[0], P.inv_ebox[0]);
      double y = wrap_d(dy, P.ebox[1], P.inv_ebox[1]);
      double z = P.npbc > 2 ? wrap_d(dz, P.ebox[2], P.inv_ebox[2]) : dz;
      re += P.lB * qq * real_images64(P, x, y, z);
    }
  }
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < NT / 32; i++) t += sh[i];
  return t;  // valid in thread 0
}

// ---------------------------------------------------------------- delta
// One launch per move, one block per SM. Four of its warps (k role) own a run of
// k units, so dS(k), the commit of the last accepted change and the |S|^2 change
// need no other block; their work is FP64. The other twelve (pair role) deal out
// the m x N (moved, other) pairs; in the integer form (fix_pair.h) a thread takes
// one other bead against a run of moved beads, its sums staying integers over
// beads of one charge, so the two roles load different pipes. Each block leaves
// three sums to the serial step, which adds the blocks in order: a ticket and a
// last block doing so cost 3 us per move, and three blocks per SM a second wave.
// Pairs with both beads moved are taken once (j > i), at trial positions for both.
//
// A move with its serial step (kern_moves.cu): 21 us for 1,000 beads and 1,687
// k-vectors, 22 us with image cells, 44 us for 20,000 beads and 7,812 k-vectors
// (50, 94 and 130 us with FP64 pairs, k tiles x bead groups and a move generated
// in the serial step).
constexpr int kDeltaThreads = 512;
constexpr int kKThreads = 128;  // k role
constexpr int kFixStage = 256;  // moved beads staged at a time
constexpr int kFixRun = 4;      // most moved beads per thread and other bead
constexpr int kUnits = 32;      // k units of a block at a time

// Moved beads per phase-table chunk of the k role: 32 where their z tables and xy
// parts fit the table budget.
__host__ __device__ inline int k_beads(const DevParams& P) {
  const int fit = kKTableBytes / (2 * (P.kmax[2] + 1 + kUnits) * (int)sizeof(double2));
  return fit < 1 ? 1 : (fit > 32 ? 32 : fit);
}

// (an integer comparison: one of doubles takes the FP64 pipe)
__device__ __forceinline__ bool same_bits(double a, double b) {
  return __double_as_longlong(a) == __double_as_longlong(b);
}

struct FixStage {
  ulonglong2 a, b, c;  // trial (x, y, z), current (x, y, z)
  double q;            // charge x lB sqrt(alpha) x table unit
  int k, pad;          // row of the LJ table
};

// The integer pair sweep of pair thread t of nt in every block. The table is
// read in place for a few pairs per thread; from 4 on, copying it to shared
// memory first (51 KB a block, about 1 us) pays: a gather then takes 10 cycles
// and not 32.
constexpr int kFixStagePairs = 4;

template <int kMode>
__device__ __forceinline__ void fix_sweep(const DevParams& P, const DevBuffers& B, FixStage* st,
                                          unsigned char* tabs, int t0, int nt, int b_lo, int m,
                                          double& acc_lj, double& acc_re) {
  FixTab T = P.fx;
  const double qs = fix_scale(P), hs = 1.0 / T.unit;
  const int N = P.n_bead;
  const int G = (int)gridDim.x * nt, p0 = (int)blockIdx.x * nt + t0;
  const long long pairs = (long long)m * N;
  if (pairs >= (long long)kFixStagePairs * G) fix_stage(T, tabs, t0, nt);
  const auto tab = [&](uint64_t s) { return fix_h(T.c01, T.c23, T.c45, T.base, s); };
  // a run of moved beads per job, shorter while there are fewer jobs than threads
  const int run_len = pairs >= 2LL * kFixRun * G ? kFixRun : (pairs >= 4LL * G ? 2 : 1);
  double lj1 = 0.0, lj0 = 0.0;
  for (int g0 = 0; g0 < m; g0 += kFixStage) {
    const int gn = min(kFixStage, m - g0);
    if (g0) role_sync(2, nt);  // the previous group is consumed
    for (int t = t0; t < gn; t += nt) {
      const int i = b_lo + g0 + t;
      const ulonglong4_32a a = B.ftrial64[g0 + t], c = B.fpos64[i];
      st[t].a = make_ulonglong2(a.x, a.y);
      st[t].b = make_ulonglong2(a.z, c.x);
      st[t].c = make_ulonglong2(c.y, c.z);
      st[t].q = __longlong_as_double((long long)c.w) * qs;
      st[t].k = B.type[i] * P.n_type;
    }
    role_sync(2, nt);
    const int runs = (gn + run_len - 1) / run_len;
    // job run * N + j, dealt with stride G; (run, j) advanced without a division
    const int gq = G / N, gr = G % N;
    for (int run = p0 / N, j = p0 % N; run < runs; run += gq, j += gr) {
      if (j >= N) {
        j -= N;
        if (++run >= runs) break;
      }
      const ulonglong4_32a o0 = B.fpos64[j];
      const int tj = B.type[j];
      const double qj = __longlong_as_double((long long)o0.w);
      // a moved other bead: its trial position, and only moved beads before it
      const int l = j - b_lo - g0;
      const bool jm = j >= b_lo && j < b_lo + m;
      const ulonglong4_32a o1 = jm ? B.ftrial64[j - b_lo] : o0;
      const int u0 = run * run_len, u1 = min(gn, u0 + run_len);
      double acc = 0.0, q = st[u0].q;
      int64_t sum = 0;
      for (int u = u0; u < u1; u++) {
        const ulonglong2 a = st[u].a, b = st[u].b, c = st[u].c;
        if (jm && u >= l) break;
        if (!same_bits(st[u].q, q)) {
          acc = fma(q, (double)sum, acc);
          q = st[u].q;
          sum = 0;
        }
        uint64_t s1, s0;
        sum += fix_term<kMode>(T, tab, o1.x - a.x, o1.y - a.y, o1.z - b.x, s1);
        sum -= fix_term<kMode>(T, tab, o0.x - b.y, o0.y - c.x, o0.z - c.y, s0);
        if (min(s1, s0) < T.s_near) {
          const int k = st[u].k + tj;
          double h = 0.0;
          const int i = b_lo + g0 + u;
          if (s1 < T.s_near)
            h = fix_near(P, B.trial[i], jm ? B.trial[j] : B.pos[j], s1 < T.s_lo, k, lj1);
          if (s0 < T.s_near) h -= fix_near(P, B.pos[i], B.pos[j], s0 < T.s_lo, k, lj0);
          acc = fma(q * hs, h, acc);
        }
      }
      acc = fma(q, (double)sum, acc);
      acc_re = fma(acc, qj, acc_re);
    }
  }
  acc_lj += lj1 - lj0;
}

// dS(k), the S(k) commit and the |S|^2 change of units [u0, u1) by the k role's
// threads. A thread takes one of up to 32 units and every slices-th moved bead (a
// block of a small k-set has few units: their beads then spread over the lanes), at both
// its places one after the other: a sum over the trial places alone is large where the
// change is small, and its rounding stays.
// smem, kb = k_beads: [kb][2][zn] e^{i n theta_z}, then [kb][2][kUnits] xy parts.
template <int kMode>
__device__ __forceinline__ double k_role(const DevParams& P, const DevBuffers& B,
                                         unsigned char* smem, int u0, int u1, int b_lo, int b_hi,
                                         int sk_pend, int sk_buf, int cur_buf) {
  const int zn = P.kmax[2] + 1, kb = k_beads(P);
  double2* s_z = reinterpret_cast<double2*>(smem);
  double2* s_xy = s_z + (size_t)kb * 2 * zn;
  __shared__ short2 s_col[kUnits];
  __shared__ double s_sum[4][kKThreads];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double e = 0.0;
  for (int c0 = u0; c0 < u1; c0 += kUnits) {
    const int un = min(kUnits, u1 - c0);
    // the units' (nx, ny) columns, numbered in order (the same in every warp)
    const KUnit lu = lane < un ? B.ku[c0 + lane] : KUnit{0, 0, 0, 0, -1, -1};
    const int px = __shfl_up_sync(0xffffffffu, lu.nx, 1), py = __shfl_up_sync(0xffffffffu, lu.ny, 1);
    const bool head = lane < un && (lane == 0 || px != lu.nx || py != lu.ny);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int ncol = __popc(heads);
    int zmax = lane < un ? lu.nz : 0;
    for (int o = 16; o > 0; o >>= 1) zmax = max(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    const int slices = kKThreads / un;
    const int u = (int)threadIdx.x % un, sl = (int)threadIdx.x / un;
    const int col = __popc(heads & (0xffffffffu >> (31 - u))) - 1;
    const int nz = __shfl_sync(0xffffffffu, (int)lu.nz, u);
    if (warp == 0 && head)
      s_col[__popc(heads & (0xffffffffu >> (31 - lane))) - 1] = make_short2(lu.nx, lu.ny);
    double2 A = make_double2(0.0, 0.0), Bs = A;
    for (int g0 = b_lo; g0 < b_hi; g0 += kb) {
      const int nt = 2 * min(kb, b_hi - g0);
      role_sync(1, kKThreads);  // the tables (and s_sum) are free, s_col is written
      // nt z recursions, then nt x ncol xy phases, one per thread
      for (int t = threadIdx.x; t < nt * (1 + ncol); t += kKThreads) {
        const int c = t / nt - 1, it = t - (c + 1) * nt;
        const int bead = g0 + (it >> 1);
        uint64_t tx, ty, tz;
        double q;
        if (kMode) {  // in integers from the mirrors
          const ulonglong4_32a p = (it & 1) ? B.fpos64[bead] : B.ftrial64[bead - b_lo];
          tx = turn_fix(P, p.x);
          ty = turn_fix(P, p.y);
          tz = turn_fix(P, p.z);
          q = __longlong_as_double((long long)p.w);
        } else {
          const double4_32a p = (it & 1) ? B.pos[bead] : B.trial[bead];
          tx = c < 0 ? 0 : turn64(P, p.x, 0);
          ty = c < 0 ? 0 : turn64(P, p.y, 1);
          tz = c < 0 ? turn64(P, p.z, 2) : 0;
          q = charge_of(p);
        }
        if (c < 0) {
          const double2 e1 = turn_exp(tz);
          double2 v = make_double2(1.0, 0.0);
          double2* z = s_z + (size_t)it * zn;
          z[0] = v;
          for (int n = 1; n <= zmax; n++) {
            v = cmul(v, e1);
            z[n] = v;
          }
        } else {
          const short2 kc = s_col[c];
          const double2 v = turn_exp(tx * (uint64_t)(int64_t)kc.x + ty * (uint64_t)(int64_t)kc.y);
          if (it & 1) q = -q;  // trial minus current
          s_xy[it * kUnits + c] = make_double2(q * v.x, q * v.y);
        }
      }
      role_sync(1, kKThreads);
      if (sl < slices)
        for (int it = 2 * sl; it < nt; it += 2 * slices)
          for (int h = 0; h < 2; h++)
            unit_add(s_xy[(it + h) * kUnits + col], s_z[(size_t)(it + h) * zn + nz], A, Bs);
    }
    s_sum[0][threadIdx.x] = A.x;
    s_sum[1][threadIdx.x] = A.y;
    s_sum[2][threadIdx.x] = Bs.x;
    s_sum[3][threadIdx.x] = Bs.y;
    role_sync(1, kKThreads);
    // the slices of each (unit, sum), added in order by a thread each
    if ((int)threadIdx.x < 4 * un) {
      const int q = (int)threadIdx.x / un, v = (int)threadIdx.x % un;
      double t = 0.0;
      for (int w = 0; w < slices; w++) t += s_sum[q][w * un + v];
      s_sum[q][v] = t;  // slice 0's place: read by this thread only
    }
    role_sync(1, kKThreads);
    if (warp < 2 && lane < un) {  // warp 0: +nz, warp 1: -nz
      const int k = warp == 0 ? lu.kp : lu.km;
      if (k >= 0) {
        const double2 SA = make_double2(s_sum[0][lane], s_sum[1][lane]);
        const double2 SB = make_double2(s_sum[2][lane], s_sum[3][lane]);
        const double2 ds = warp == 0 ? unit_plus(SA, SB) : unit_minus(SA, SB);
        double2 s = B.sk[k];
        if (sk_pend) {
          const double2 p = B.dsk[(size_t)sk_buf * P.n_k + k];
          s = make_double2(s.x + p.x, s.y + p.y);
          B.sk[k] = s;
        }
        B.dsk[(size_t)cur_buf * P.n_k + k] = ds;
        e += B.kw[k] * (2.0 * (s.x * ds.x + s.y * ds.y) + (ds.x * ds.x + ds.y * ds.y));
      }
    }
  }
  return e;
}

template <int kMode>
__global__ void __launch_bounds__(kDeltaThreads, 1)
    k_delta64(const DevParams P, const DevBuffers B, int tab_bytes) {
  extern __shared__ __align__(32) unsigned char smem[];
  __shared__ double s_part[kDeltaThreads / 32][2];
  const DevState* st = B.state;
  const int b_lo = st->b_lo, b_hi = st->b_hi;
  const int m = st->pending ? b_hi - b_lo : 0;
  const int kthreads = P.use_ewald && P.n_ku > 0 ? kKThreads : 0;
  const int warp = threadIdx.x >> 5;
  double a = 0.0, b = 0.0;  // k role: k energy; pair role: LJ and real space
  if ((int)threadIdx.x < kthreads) {
    const int u0 = (int)((long long)P.n_ku * blockIdx.x / gridDim.x);
    const int u1 = (int)((long long)P.n_ku * (blockIdx.x + 1) / gridDim.x);
    if (m > 0)
      a = k_role<kMode>(P, B, smem + tab_bytes, u0, u1, b_lo, b_hi, st->sk_pending, st->sk_buf,
                 st->cur_buf);
  } else {
    const int t0 = (int)threadIdx.x - kthreads, nt = kDeltaThreads - kthreads;
    const int N = P.n_bead;
    if (kMode) {
      if (m > 0)
        fix_sweep<kMode>(P, B, reinterpret_cast<FixStage*>(smem),
                         smem + kFixStage * sizeof(FixStage), t0, nt, b_lo, m, a, b);
    } else if (P.use_pair || P.use_ewald) {
      // pair p = ii * N + j, dealt with stride G; (ii, j) advanced without a
      // division per pair
      const long long total = (long long)m * N;
      const long long G = (long long)gridDim.x * nt;
      const long long p0 = (long long)blockIdx.x * nt + t0;
      const int gq = (int)(G / N), gr = (int)(G % N);
      int ii = (int)(p0 / N), j = (int)(p0 % N);
      for (long long p = p0; p < total; p += G, ii += gq, j += gr) {
        if (j >= N) {
          j -= N;
          ii++;
        }
        const int i = b_lo + ii;
        const bool jm = j >= b_lo && j < b_hi;
        if (jm && j <= i) continue;
        const double4_32a ti = B.trial[i], ci = B.pos[i];
        const int tyi = B.type[i], tyj = B.type[j];
        const double4_32a cj = B.pos[j];
        const double4_32a tj = jm ? B.trial[j] : cj;
        double l1 = 0, r1 = 0, l0 = 0, r0 = 0;
        pair64(P, ti, tyi, tj, tyj, l1, r1);
        pair64(P, ci, tyi, cj, tyj, l0, r0);
        if (!hs_bonded(P, B.mol_start, i, j)) a += l1 - l0;
        b += r1 - r0;
      }
    }
  }
  // (LJ is zero in most warps)
  __syncwarp();
  if (__any_sync(0xffffffffu, a != 0.0)) a = warp_sum(a);
  if ((int)threadIdx.x >= kthreads) b = warp_sum(b);
  if ((threadIdx.x & 31) == 0) {
    s_part[warp][0] = a;
    s_part[warp][1] = b;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    // sums 0 LJ, 1 real space over the pair warps, 2 over the k warps
    const int kw = kthreads / 32, w0 = threadIdx.x == 2 ? 0 : kw;
    const int w1 = threadIdx.x == 2 ? kw : kDeltaThreads / 32;
    double t = 0.0;
    for (int w = w0; w < w1; w++) t += s_part[w][threadIdx.x == 1];
    B.partial[4 * blockIdx.x + threadIdx.x] = t;
  }
}

int pair_grid() { return 2 * device_sms(); }

// One block per SM (a block takes nearly all of an SM's registers), but for the
// SMs that the next move's candidates run on meanwhile: with a block on every SM
// those waited for the energy change, or it for them.
int delta_blocks() { return std::max(1, pair_grid() / 2 - kCands); }

template <int kMode>
static void launch_delta64(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  constexpr size_t stage = kFixStage * sizeof(FixStage) + kFixMaxBins * 40;
  static OncePerDevice once;
  allow_smem(once, k_delta64<kMode>, stage + kKTableBytes);
  // the staged moved beads and the table, then the k role's phase tables
  const size_t tab = kMode ? kFixStage * sizeof(FixStage) + (size_t)P.fx.n_bin * 40 : 0;
  const size_t k = P.use_ewald && P.n_ku > 0
                       ? (size_t)k_beads(P) * 2 * (P.kmax[2] + 1 + kUnits) * sizeof(double2) : 0;
  k_delta64<kMode><<<delta_blocks(), kDeltaThreads, tab + k, s>>>(P, B, (int)tab);
}

void launch_delta_pairs64(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  if (P.fx.mode == 1)
    launch_delta64<1>(P, B, s);
  else if (P.fx.mode == 2)
    launch_delta64<2>(P, B, s);
  else
    launch_delta64<0>(P, B, s);
}

// ---------------------------------------------------------------- totals
constexpr int kTotTile = 128;

__device__ __forceinline__ void tri_unrank(long long t, int n, int& a, int& b) {
  // t-th (a <= b) pair of an n x n upper triangle, row-major.
  int r = (int)((2.0 * n + 1 - sqrt((2.0 * n + 1) * (2.0 * n + 1) - 8.0 * t)) / 2);
  if (r < 0) r = 0;
  auto start = [n](long long rr) { return rr * n - rr * (rr - 1) / 2; };
  while (r > 0 && start(r) > t) r--;
  while (r + 1 < n && start(r + 1) <= t) r++;
  a = r;
  b = r + (int)(t - start(r));
}

__global__ void __launch_bounds__(kTotTile)
    k_total64(const DevParams P, const DevBuffers B, double* out) {
  __shared__ double4_32a sp[kTotTile];
  __shared__ int st[kTotTile];
  __shared__ double red[kTotTile / 32];
  const int nt = (P.n_bead + kTotTile - 1) / kTotTile;
  int ta, tb;
  tri_unrank(blockIdx.x, nt, ta, tb);
  const int j0 = tb * kTotTile;
  const int jn = min(kTotTile, P.n_bead - j0);
  if (threadIdx.x < jn) {
    sp[threadIdx.x] = B.pos[j0 + threadIdx.x];
    st[threadIdx.x] = B.type[j0 + threadIdx.x];
  }
  __syncthreads();
  double lj = 0.0, re = 0.0;
  const int i = ta * kTotTile + threadIdx.x;
  if (i < P.n_bead) {
    const double4_32a pi = B.pos[i];
    const int ti = B.type[i];
    for (int jj = 0; jj < jn; jj++) {
      if (ta == tb && jj <= (int)threadIdx.x) continue;
      double l = 0.0;
      pair64(P, pi, ti, sp[jj], st[jj], l, re);
      if (!hs_bonded(P, B.mol_start, i, j0 + jj)) lj += l;
    }
  }
  double a = block_sum<kTotTile>(lj, red);
  double b = block_sum<kTotTile>(re, red);
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = a;
    out[2 * blockIdx.x + 1] = b;
  }
}

// The same sum in the integer form (fix_pair.h): 256 x 256 tiles of the i < j
// triangle, a thread per i against the staged j's (their sums stay integers
// over up to 16 beads of one charge). The table is staged too, as the lanes'
// gathers from it run at a bank's pace there and a line's pace from L1; a small
// system's tiles are cut into `parts` of the j's instead, so that they fill the
// SMs, and read it in place. 20,000 beads: 1.1 ms (6.2 ms in FP64).
constexpr int kFixTile = 256;
constexpr int kFixFlush = 16;
struct FixOther {
  ulonglong2 a;  // x, y
  unsigned long long z;
  double q;
};

template <int kMode, bool kStaged>
__global__ void __launch_bounds__(kFixTile)
    k_total64_fix(const DevParams P, const DevBuffers B, double* out, int parts) {
  extern __shared__ __align__(32) unsigned char smem[];
  __shared__ FixOther so[kFixTile];
  __shared__ int st[kFixTile];
  __shared__ double red[kFixTile / 32];
  const int nt = (P.n_bead + kFixTile - 1) / kFixTile;
  int ta, tb;
  tri_unrank(blockIdx.x / parts, nt, ta, tb);
  const int per = kFixTile / parts;
  const int j0 = tb * kFixTile + (int)(blockIdx.x % parts) * per;
  const int jn = min(per, P.n_bead - j0);
  FixTab T = P.fx;
  if (kStaged) fix_stage(T, smem, threadIdx.x, kFixTile);
  if ((int)threadIdx.x < jn) {
    const ulonglong4_32a p = fix64x4(P, B.pos[j0 + threadIdx.x]);
    so[threadIdx.x].a = make_ulonglong2(p.x, p.y);
    so[threadIdx.x].z = p.z;
    so[threadIdx.x].q = __longlong_as_double((long long)p.w);
    st[threadIdx.x] = B.type[j0 + threadIdx.x];
  }
  __syncthreads();
  const auto tab = [&](uint64_t s) { return fix_h(T.c01, T.c23, T.c45, T.base, s); };
  double lj = 0.0, re = 0.0;
  const int i = ta * kFixTile + threadIdx.x;
  if (i < P.n_bead && jn > 0) {
    const ulonglong4_32a pi = fix64x4(P, B.pos[i]);
    const double hs = 1.0 / T.unit;
    const int kt = B.type[i] * P.n_type;
    double q = so[0].q;
    int64_t sum = 0;
    int held = 0;
    for (int jj = 0; jj < jn; jj++) {
      const ulonglong2 a = so[jj].a;
      const unsigned long long z = so[jj].z;
      if (!same_bits(so[jj].q, q) || held == kFixFlush) {
        re = fma(q, (double)sum, re);
        q = so[jj].q;
        sum = 0;
        held = 0;
      }
      held++;
      if (j0 + jj <= i) continue;
      uint64_t s;
      sum += fix_term<kMode>(T, tab, a.x - pi.x, a.y - pi.y, z - pi.z, s);
      if (s < T.s_near)
        re = fma(q * hs, fix_near(P, B.pos[i], B.pos[j0 + jj], s < T.s_lo, kt + st[jj], lj), re);
    }
    re = fma(q, (double)sum, re);
    re *= __longlong_as_double((long long)pi.w) * fix_scale(P);
  }
  const double a = block_sum<kFixTile>(lj, red);
  const double b = block_sum<kFixTile>(re, red);
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = a;
    out[2 * blockIdx.x + 1] = b;
  }
}

// The plain form's 64-bit mirror of every bead's position.
__global__ void k_fix64_all(const DevParams P, const DevBuffers B) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n_bead; i += gridDim.x * blockDim.x)
    B.fpos64[i] = fix64x4(P, B.pos[i]);
}

void launch_fix64_all(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  if (B.fpos64 && P.n_bead > 0) k_fix64_all<<<(P.n_bead + 255) / 256, 256, 0, s>>>(P, B);
}

// Parts of a 256 x 256 tile: enough for two blocks per SM, at most 16.
static int fix_parts(const DevParams& P) {
  const long long nt = (P.n_bead + kFixTile - 1) / kFixTile, tiles = nt * (nt + 1) / 2;
  int parts = 1;
  while (parts < 16 && tiles * parts < pair_grid()) parts *= 2;
  return parts;
}

int total_partials_count(const DevParams& P) {
  const int tile = P.fx.mode ? kFixTile : kTotTile;
  const long long nt = (P.n_bead + tile - 1) / tile;
  return (int)(nt * (nt + 1) / 2) * (P.fx.mode ? fix_parts(P) : 1);
}

template <int kMode>
static void launch_total_fix(const DevParams& P, const DevBuffers& B, double* out, int n_part,
                             cudaStream_t s) {
  const int parts = fix_parts(P);
  const size_t smem = (size_t)P.fx.n_bin * (2 * sizeof(FixPair64) + sizeof(FixPair32));
  if (parts == 1) {
    static OncePerDevice once;
    allow_smem(once, k_total64_fix<kMode, true>, kFixMaxBins * 40);
    k_total64_fix<kMode, true><<<n_part, kFixTile, smem, s>>>(P, B, out, parts);
  } else {
    k_total64_fix<kMode, false><<<n_part, kFixTile, 0, s>>>(P, B, out, parts);
  }
}

void launch_total64(const DevParams& P, const DevBuffers& B, double* out, int n_part,
                    cudaStream_t s) {
  if (P.fx.mode == 1)
    launch_total_fix<1>(P, B, out, n_part, s);
  else if (P.fx.mode == 2)
    launch_total_fix<2>(P, B, out, n_part, s);
  else
    k_total64<<<n_part, kTotTile, 0, s>>>(P, B, out);
}

// S(k) from scratch: block (unit tile, bead group) writes a partial, a second
// pass adds the groups in order. A thread takes kSkPer consecutive units (+-nz
// pairs, see KUnit), which mostly share their column's xy product: five FP64
// operations per unit and bead, 2.5 per vector (6.5 with a complex product per
// vector). The grid is one wave of two blocks per SM.
constexpr int kSkPer = 4;
constexpr int kSkTile = kSkPer * kPairThreads;
constexpr int kSkGroupsMax = 512;

int sk_full_groups(const DevParams& P) {
  const int tiles = std::max(1, (P.n_ku + kSkTile - 1) / kSkTile);
  return std::max(1, std::min(kSkGroupsMax, pair_grid() / tiles));
}

__global__ void __launch_bounds__(kPairThreads, 2)
    k_sk64(const DevParams P, const DevBuffers B, double2* part, int groups) {
  extern __shared__ __align__(32) unsigned char smem[];
  double2* tabs = reinterpret_cast<double2*>(smem);
  const int per = P.kper;
  const int chunk = P.kchunk_sk;
  const int g = blockIdx.y;
  const int per_g = (P.n_bead + groups - 1) / groups;
  const int b0 = g * per_g, b1 = min(P.n_bead, b0 + per_g);
  KUnit un[kSkPer];
  bool mine[kSkPer], col[kSkPer];
  double2 A[kSkPer], Bs[kSkPer];
#pragma unroll
  for (int q = 0; q < kSkPer; q++) {
    const int u = blockIdx.x * kSkTile + threadIdx.x * kSkPer + q;
    mine[q] = u < P.n_ku;
    un[q] = mine[q] ? B.ku[u] : KUnit{0, 0, 0, 0, -1, -1};
    // a new (nx, ny) column: recompute the xy product
    col[q] = q == 0 || un[q].nx != un[q - 1].nx || un[q].ny != un[q - 1].ny;
    A[q] = Bs[q] = make_double2(0.0, 0.0);
  }
  for (int c0 = b0; c0 < b1; c0 += chunk) {
    const int cnt = min(chunk, b1 - c0);
    __syncthreads();
    // axis by axis, so that a warp's lanes share the length of their recursion
    for (int t = threadIdx.x; t < 3 * 32; t += kPairThreads)
      if ((t & 31) < cnt) build_axis_table(P, B.pos[c0 + (t & 31)], t >> 5, tabs + (t & 31) * per);
    __syncthreads();
    if (mine[0])
      for (int b = 0; b < cnt; b++) {
        const double2* tb = tabs + b * per;
        double2 xy = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < kSkPer; q++)
          if (mine[q]) {
            if (col[q]) xy = unit_xy(P, tb, un[q].nx, un[q].ny);
            unit_add(xy, tb[P.koff[2] + un[q].nz], A[q], Bs[q]);
          }
      }
  }
#pragma unroll
  for (int q = 0; q < kSkPer; q++)
    if (mine[q]) {
      if (un[q].kp >= 0) part[(size_t)g * P.n_k + un[q].kp] = unit_plus(A[q], Bs[q]);
      if (un[q].km >= 0) part[(size_t)g * P.n_k + un[q].km] = unit_minus(A[q], Bs[q]);
    }
}

// Eight threads per k-vector add every eighth group, then their sums in order.
__global__ void __launch_bounds__(256) k_sk_sum(int n_k, int groups, const double2* part,
                                                double2* sk) {
  __shared__ double2 sh[8][32];
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5, k = blockIdx.x * 32 + l;
  double2 s = make_double2(0.0, 0.0);
  if (k < n_k)
    for (int g = w; g < groups; g += 8) {
      const double2 p = part[(size_t)g * n_k + k];
      s.x += p.x;
      s.y += p.y;
    }
  sh[w][l] = s;
  __syncthreads();
  if (w == 0 && k < n_k) {
    for (int q = 1; q < 8; q++) {
      s.x += sh[q][l].x;
      s.y += sh[q][l].y;
    }
    sk[k] = s;
  }
}

void launch_sk_full64(const DevParams& P, const DevBuffers& B, double2* part, cudaStream_t s) {
  if (!P.use_ewald || P.n_k == 0) return;
  static OncePerDevice once;
  allow_smem(once, k_sk64, kKTableBytes + 4096);
  size_t smem = (size_t)P.kchunk_sk * P.kper * sizeof(double2);
  // a group of fewer than 8 beads would spend more on its tables than its sums
  const int groups = std::max(1, std::min(sk_full_groups(P), (P.n_bead + 7) / 8));
  dim3 grid((P.n_ku + kSkTile - 1) / kSkTile, groups);
  k_sk64<<<grid, kPairThreads, smem, s>>>(P, B, part, groups);
  k_sk_sum<<<(P.n_k + 31) / 32, 256, 0, s>>>(P.n_k, groups, part, B.sk);
}

// Misc totals: block b writes its {bond, ext, self, self_images, mz} to out +
// 5 b (k_assemble_total adds the blocks in order) and bond_mol[]. A warp per
// molecule sums its bonds (potential_spring.cc:22-48); the beads are dealt over
// the grid. (One block with a thread per molecule took 470 us on 20,000 beads.)
__global__ void __launch_bounds__(256) k_misc64(const DevParams P, const DevBuffers B,
                                                double* out) {
  __shared__ double red[8];
  __shared__ double s_img;
  double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  if (threadIdx.x == 0) s_img = P.use_ewald ? real_images64(P, 0.0, 0.0, 0.0) : 0.0;
  __syncthreads();
  const double img = s_img;
  const int lane = threadIdx.x & 31;
  for (int m = blockIdx.x * 8 + (threadIdx.x >> 5); m < P.n_mol; m += gridDim.x * 8) {
    double e = 0.0;
    if (P.use_bond) {
      const int b0 = B.mol_start[m], b1 = B.mol_start[m + 1];
      for (int i = b0 + lane; i < b1 - 1; i += 32) {
        const double4_32a p = B.pos[i], q = B.pos[i + 1];
        const double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        const double r = sqrt(dx * dx + dy * dy + dz * dz);
        e += 0.5 * P.k_bond * (r - P.r0) * (r - P.r0);
      }
      for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    }
    if (lane == 0) {
      B.bond_mol[m] = e;
      v[0] += e;
    }
  }
  for (int i = blockIdx.x * 256 + threadIdx.x; i < P.n_bead; i += gridDim.x * 256) {
    const double4_32a p = B.pos[i];
    if (P.use_ext) v[1] += wall64(P, p.z, B.type[i]);
    if (P.use_ewald) {
      v[2] += P.self_coef * p.w * p.w;
      v[3] += 0.5 * P.lB * p.w * p.w * img;
      v[4] += p.w * p.z;
    }
  }
  for (int q = 0; q < 5; q++) {
    const double t = block_sum<256>(v[q], red);
    if (threadIdx.x == 0) out[5 * blockIdx.x + q] = t;
  }
}

void launch_misc_total64(const DevParams& P, const DevBuffers& B, double* out, cudaStream_t s) {
  k_misc64<<<kMiscBlocks, 256, 0, s>>>(P, B, out);
}

// Rg^2, axis components and end-to-end^2 (simulation.cc:406-500); one block
// per chain writes its terms, thread 0 of a final pass adds them in order.
__global__ void k_obs_chain(const DevParams P, const DevBuffers B, double* per_mol) {
  __shared__ double red[8];
  const int m = blockIdx.x;
  const int b0 = B.mol_start[m], n = B.mol_start[m + 1] - b0;
  double g = 0, gx = 0, gy = 0, gz = 0;
  if (n > 1) {
    long long np = (long long)n * (n - 1) / 2;
    for (long long p = threadIdx.x; p < np; p += blockDim.x) {
      int j = (int)((2.0 * n - 1 - sqrt((2.0 * n - 1) * (2.0 * n - 1) - 8.0 * p)) / 2);
      auto st = [n](long long jj) { return jj * (2 * n - jj - 1) / 2; };
      while (j > 0 && st(j) > p) j--;
      while (st(j + 1) <= p) j++;
      int k = j + 1 + (int)(p - st(j));
      double4_32a a = B.pos[b0 + j], b = B.pos[b0 + k];
      double x = fabs(a.x - b.x), y = fabs(a.y - b.y), z = fabs(a.z - b.z);
      double r = sqrt(x * x + y * y + z * z);
      g += r * r;
      gx += x * x, gy += y * y, gz += z * z;
    }
  }
  double v[4] = {g, gx, gy, gz};
  for (int q = 0; q < 4; q++) {
    double t = block_sum<256>(v[q], red);
    if (threadIdx.x == 0) per_mol[5 * m + q] = n > 1 ? t / ((double)n * n) : 0.0;
  }
  if (threadIdx.x == 0) {
    double e = 0.0;
    if (n > 1) {
      double4_32a a = B.pos[b0], b = B.pos[b0 + n - 1];
      double x = a.x - b.x, y = a.y - b.y, z = a.z - b.z;
      double r = sqrt(x * x + y * y + z * z);
      e = r * r;
    }
    per_mol[5 * m + 4] = e;
  }
}

__global__ void k_obs_sum(int n_mol, int n_chains, const double* per_mol, double* out5) {
  if (threadIdx.x != 0) return;
  double s[5] = {0, 0, 0, 0, 0};
  for (int m = 0; m < n_mol; m++)
    for (int q = 0; q < 5; q++) s[q] += per_mol[5 * m + q];
  for (int q = 0; q < 5; q++) out5[q] = n_chains > 0 ? s[q] / n_chains : s[q];
}

void launch_observables64(const DevParams& P, const DevBuffers& B, double* per_mol,
                          double* out5, cudaStream_t s) {
  k_obs_chain<<<P.n_mol, 256, 0, s>>>(P, B, per_mol);
  k_obs_sum<<<1, 32, 0, s>>>(P.n_mol, P.n_chain_total, per_mol, out5);
}

// rho(z) counts of one configuration (Simulation::CalcRhoZ,
// simulation.cc:1029-1045): molecules from `phantom` on, category 0 for
// chains, 1 for ions with q >= 0, 2 for q < 0; z wrapped into [0, Lz) by
// floor; bin floor(z / res) kept when inside [0, n_bins). Integer counts
// (order-independent); the host scales them by 1 / (Lx Ly res).
__global__ void k_rhoz(const DevParams P, const DevBuffers B, double res, int n_bins,
                       unsigned* cnt) {
  for (int m = P.phantom + blockIdx.x; m < P.n_mol; m += gridDim.x) {
    const int b0 = B.mol_start[m], n = B.mol_start[m + 1] - b0;
    const int id = n > 1 ? 0 : (B.pos[b0].w >= 0.0 ? 1 : 2);
    for (int j = b0 + threadIdx.x; j < b0 + n; j += blockDim.x) {
      double z = B.pos[j].z;
      z -= P.box[2] * floor(z / P.box[2]);
      const int bz = (int)floor(z / res);
      if (bz >= 0 && bz < n_bins) atomicAdd(&cnt[3 * bz + id], 1u);
    }
  }
}

void launch_rhoz(const DevParams& P, const DevBuffers& B, double res, int n_bins, unsigned* cnt,
                 cudaStream_t s) {
  cudaMemsetAsync(cnt, 0, sizeof(unsigned) * 3 * (size_t)n_bins, s);
  const int m = P.n_mol - P.phantom;
  if (m > 0) k_rhoz<<<std::min(m, 4 * 152), 128, 0, s>>>(P, B, res, n_bins, cnt);
}

}  // namespace plum
