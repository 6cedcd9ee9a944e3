// Configurational-bias trial-site energies (ForceField::BeadsEnergy,
// cbmc.cc:5-151) for all trial sites of one growth step at once.
//
//   k_cbmc_so     S_o(k): the committed S(k) (plus any pending accepted
//                 change), minus the molecules being deleted, plus the grown
//                 chain and its counterions
//   k_cbmc_sys    grid (bead groups) x (trials): LJ and real-space Ewald of
//                 each trial bead (and its trial counterion) with every
//                 system bead outside the deleted molecules; per-block sums
//   k_cbmc_fin    one block per trial: the block sums in order, the grown
//                 chain terms (no LJ with the preceding grown bead,
//                 cbmc.cc:57-58), bead-counterion cross terms, self terms,
//                 k-space |S_o + q1 e1 + q2 e2|^2 - |S_o|^2, walls, dipole
//                 change; 1e8 when the pair sum reaches 1e8 (cbmc.cc:146-148)
// The arithmetic is the plain form's (FP64) with the same pair functions as
// the move kernels.
#include <cstdio>
#include <mutex>

#include "device_common.cuh"
#include "engine.h"
#include "fix_device.cuh"
#include "kspace64.cuh"

namespace plum {

// pair helpers shared with kern_energy.cu (same formulas, inlined here)
__device__ __forceinline__ double cb_wrap(double d, double L, double invL) {
  return d - L * rint(d * invL);
}

__device__ __forceinline__ double cb_lj(const DevParams& P, int ta, int tb, double4_32a a,
                                        double4_32a b) {
  double x = cb_wrap(b.x - a.x, P.box[0], P.inv_box[0]);
  double y = cb_wrap(b.y - a.y, P.box[1], P.inv_box[1]);
  double z = P.npbc > 2 ? cb_wrap(b.z - a.z, P.box[2], P.inv_box[2]) : b.z - a.z;
  double r2 = x * x + y * y + z * z;
  int k = ta * P.n_type + tb;
  if (P.pair_kind == 1) return sqrt(r2) <= P.hs_sum[k] ? kVeryLarge : 0.0;  // hard spheres
  if (r2 <= 0.0) return kVeryLarge;
  if (r2 < P.lj_rc2[k]) {
    double s2 = P.lj_sig2[k] / r2;
    double s6 = s2 * s2 * s2;
    return P.lj_eps4[k] * (s6 * s6 - s6) - P.lj_eref[k];
  }
  return 0.0;
}

__device__ __forceinline__ double cb_real(const DevParams& P, double4_32a a, double4_32a b) {
  double qq = a.w * b.w;
  if (qq == 0.0) return 0.0;
  double dx = cb_wrap(b.x - a.x, P.ebox[0], P.inv_ebox[0]);
  double dy = cb_wrap(b.y - a.y, P.ebox[1], P.inv_ebox[1]);
  double dz = P.npbc > 2 ? cb_wrap(b.z - a.z, P.ebox[2], P.inv_ebox[2]) : b.z - a.z;
  double e = 0.0;
  const double rc = P.real_cut;
  for (int i = -P.real_cell[0]; i <= P.real_cell[0]; i++) {
    double x = dx + i * P.ebox[0];
    if (fabs(x) > rc) continue;
    for (int j = -P.real_cell[1]; j <= P.real_cell[1]; j++) {
      double y = dy + j * P.ebox[1];
      if (fabs(y) > rc) continue;
      for (int k = -P.real_cell[2]; k <= P.real_cell[2]; k++) {
        double z = dz + k * P.ebox[2];
        if (fabs(z) > rc) continue;
        const double r2 = x * x + y * y + z * z;
        if (r2 > 0.0 && r2 <= rc * rc) e += real_term64(P, r2);
      }
    }
  }
  return P.lB * qq * e;
}

__device__ __forceinline__ double2 cb_phase(const DevParams& P, short4 kn, double4_32a p) {
  double w[3] = {p.x, p.y, p.z};
  for (int a = 0; a < P.npbc; a++) w[a] -= P.ebox[a] * floor(w[a] * P.inv_ebox[a]);
  double ph = kn.x * P.kunit[0] * w[0] + kn.y * P.kunit[1] * w[1] + kn.z * P.kunit[2] * w[2];
  double s, c;
  sincos(ph, &s, &c);
  return make_double2(p.w * c, p.w * s);
}

__global__ void k_cbmc_so(const DevParams P, const DevBuffers B, CbmcJob J) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.n_k) return;
  const DevState* st = B.state;
  const short4 kn = B.kn[k];
  double2 s = B.sk[k];
  if (st->sk_pending) {
    double2 d = B.dsk[(size_t)st->sk_buf * P.n_k + k];
    s.x += d.x;
    s.y += d.y;
  }
  for (int j = J.ex_lo; j < J.ex_hi; j++) {
    double2 e = cb_phase(P, kn, B.pos[j]);
    s.x -= e.x;
    s.y -= e.y;
  }
  for (int i = 0; i < J.cl; i++) {
    double2 e = cb_phase(P, kn, J.chain[i]);
    s.x += e.x;
    s.y += e.y;
    if (J.charged) {
      e = cb_phase(P, kn, J.chain_ci[i]);
      s.x += e.x;
      s.y += e.y;
    }
  }
  J.s_o[k] = s;
}

template <int NT>
__device__ __forceinline__ double cb_bsum(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  for (int i = 0; i < NT / 32; i++) t += sh[i];
  __syncthreads();
  return t;
}

constexpr int kCbThreads = 256;

__global__ void __launch_bounds__(kCbThreads)
    k_cbmc_sys(const DevParams P, const DevBuffers B, CbmcJob J) {
  __shared__ double red[kCbThreads / 32];
  const int t = blockIdx.y;
  const double4_32a b1 = J.b1[t];
  const double4_32a b2 = J.charged ? J.b2[t] : b1;
  double lj = 0.0, re = 0.0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < P.n_bead; j += gridDim.x * blockDim.x) {
    if (j >= J.ex_lo && j < J.ex_hi) continue;
    const double4_32a pj = B.pos[j];
    const int tj = B.type[j];
    if (P.use_pair) {
      lj += cb_lj(P, J.type, tj, b1, pj);
      if (J.charged) lj += cb_lj(P, J.type, tj, b2, pj);
    }
    if (P.use_ewald) {
      re += cb_real(P, b1, pj);
      if (J.charged) re += cb_real(P, b2, pj);
    }
  }
  lj = cb_bsum<kCbThreads>(lj, red);
  re = cb_bsum<kCbThreads>(re, red);
  if (threadIdx.x == 0) {
    J.part[2 * (t * gridDim.x + blockIdx.x)] = lj;
    J.part[2 * (t * gridDim.x + blockIdx.x) + 1] = re;
  }
}

__global__ void __launch_bounds__(kCbThreads)
    k_cbmc_fin(const DevParams P, const DevBuffers B, CbmcJob J, int n_groups) {
  __shared__ double red[kCbThreads / 32];
  const int t = blockIdx.x;
  const double4_32a b1 = J.b1[t];
  const double4_32a b2 = J.charged ? J.b2[t] : b1;
  const int ty = J.type;
  double lj = 0.0, re = 0.0, ek = 0.0, mz = 0.0;
  for (int g = threadIdx.x; g < n_groups; g += blockDim.x) {
    lj += J.part[2 * (t * n_groups + g)];
    re += J.part[2 * (t * n_groups + g) + 1];
  }
  for (int i = threadIdx.x; i < J.cl; i += blockDim.x) {
    const double4_32a ci = J.chain[i];
    const double4_32a cc = J.charged ? J.chain_ci[i] : ci;
    if (P.use_pair) {
      if (i < J.cl - 1) lj += cb_lj(P, ty, ty, b1, ci);
      if (J.charged) {
        lj += cb_lj(P, ty, ty, b1, cc);
        lj += cb_lj(P, ty, ty, b2, ci);
        lj += cb_lj(P, ty, ty, b2, cc);
      }
    }
    if (P.use_ewald) {
      re += cb_real(P, b1, ci);
      if (J.charged) re += cb_real(P, b1, cc) + cb_real(P, b2, ci) + cb_real(P, b2, cc);
    }
    mz += ci.w * ci.z + (J.charged ? cc.w * cc.z : 0.0);
  }
  if (P.use_ewald)
    for (int k = threadIdx.x; k < P.n_k; k += blockDim.x) {
      const double2 so = J.s_o[k];
      const short4 kn = B.kn[k];
      double2 e = cb_phase(P, kn, b1);
      if (J.charged) {
        double2 e2 = cb_phase(P, kn, b2);
        e.x += e2.x;
        e.y += e2.y;
      }
      const double nx = so.x + e.x, ny = so.y + e.y;
      ek += B.kw[k] * ((nx * nx + ny * ny) - (so.x * so.x + so.y * so.y));
    }
  // dipole base: the system minus the deleted molecules, plus the grown chain
  if (P.dipole)
    for (int j = J.ex_lo + threadIdx.x; j < J.ex_hi; j += blockDim.x) {
      const double4_32a p = B.pos[j];
      mz -= p.w * p.z;
    }
  lj = cb_bsum<kCbThreads>(lj, red);
  re = cb_bsum<kCbThreads>(re, red);
  ek = cb_bsum<kCbThreads>(ek, red);
  mz = cb_bsum<kCbThreads>(mz, red);
  if (threadIdx.x == 0) {
    double pair_e = lj;
    if (P.use_pair && J.charged) pair_e += cb_lj(P, ty, ty, b1, b2);
    double ew = 0.0;
    if (P.use_ewald && pair_e < kVeryLarge) {
      ew = re + P.kpref * ek;
      ew += P.self_coef * b1.w * b1.w + 0.5 * cb_real(P, b1, b1);
      if (J.charged)
        ew += P.self_coef * b2.w * b2.w + cb_real(P, b1, b2) + 0.5 * cb_real(P, b2, b2);
      if (P.dipole) {
        const double mzo = B.state->mz + mz;
        const double mzn = mzo + b1.w * b1.z + (J.charged ? b2.w * b2.z : 0.0);
        ew += P.dip_coef * (mzn * mzn - mzo * mzo);
      }
    }
    if (P.use_ext) {
      pair_e += wall64(P, b1.z, ty);
      if (J.charged) pair_e += wall64(P, b2.z, ty);
    }
    J.u[t] = pair_e >= kVeryLarge ? kVeryLarge : pair_e + ew;
  }
}

// The same energies where the integer pair form applies (and the context keeps
// the 64-bit position mirror), in a sweep and a sum per trial.
//   pair role  a warp's lanes take 32 trials, so a system bead (and, as the
//              list's tail, a grown bead) is one broadcast load and no sum
//              crosses lanes; opposite charges of a trial and its counterion
//              leave one integer per bead
//   k role     (charged species) a block's own k units: S_o(k) from the
//              committed S(k), the deleted and the grown beads, then every
//              trial's kw (2 S_o.e + |e|^2)
// k_cbmc64_sum adds the blocks' sums of a trial in order and its own terms, a block
// per trial (the last block of the sweep doing it for all took longer than the
// launch). No split depends on the number of trials, so neither does a result. One
// growth step of 32 charged trials on 6,400 beads, r_c = 0.7 L: 31 us on the device
// and 54 us a call (430 and 477 us in three FP64 launches: 27 image cells per pair, a
// sincos per trial and k).
constexpr int kCb64Threads = 512, kCb64K = 128;

int cbmc_blocks() { return pair_grid() / 2; }

template <int kMode>
__global__ void __launch_bounds__(kCb64Threads, 1)
    k_cbmc64(const DevParams P, const DevBuffers B, CbmcJob J) {
  extern __shared__ __align__(32) unsigned char smem[];
  __shared__ double s_red[3][kCb64Threads];
  __shared__ double s_w[2][kCb64K / 32][4];
  __shared__ ulonglong4_32a s_site[2][32];
  const int kth = J.charged && P.use_ewald && P.n_ku > 0 ? kCb64K : 0;
  const int tid = threadIdx.x, T = J.n_trials, N = P.n_bead;
  const int grown = J.cl * (J.charged ? 2 : 1);
  const auto grown_bead = [&](int i) { return i < J.cl ? J.chain[i] : J.chain_ci[i - J.cl]; };
  double* const slots = J.slots + (size_t)blockIdx.x * T * 3;
  if (tid < kth) {
    for (int c0 = 0; c0 < T; c0 += kCb64K) {
      const int tl = min(kCb64K, T - c0);
      uint64_t x[2] = {0, 0}, y[2] = {0, 0}, z[2] = {0, 0};
      double q[2] = {0.0, 0.0};
      if (tid < tl)
        for (int b = 0; b < 2; b++) {
          const ulonglong4_32a v = fix64x4(P, b ? J.b2[c0 + tid] : J.b1[c0 + tid]);
          x[b] = turn_fix(P, v.x);
          y[b] = turn_fix(P, v.y);
          z[b] = turn_fix(P, v.z);
          q[b] = __longlong_as_double((long long)v.w);
        }
      const int u0 = (int)((long long)P.n_ku * blockIdx.x / gridDim.x);
      const int u1 = (int)((long long)P.n_ku * (blockIdx.x + 1) / gridDim.x);
      const int gone = J.ex_hi - J.ex_lo;
      const int pend = B.state->sk_pending, buf = B.state->sk_buf;
      double acc = 0.0;
      for (int u = u0; u < u1; u++) {
        const KUnit ku = B.ku[u];
        const uint64_t nx = (uint64_t)ku.nx, ny = (uint64_t)(int64_t)ku.ny, nz = (uint64_t)ku.nz;
        double o[4] = {0.0, 0.0, 0.0, 0.0};
        for (int i = tid; i < gone + grown; i += kCb64K) {
          const ulonglong4_32a v =
              i < gone ? B.fpos64[J.ex_lo + i] : fix64x4(P, grown_bead(i - gone));
          const double w0 = __longlong_as_double((long long)v.w), w = i < gone ? -w0 : w0;
          const uint64_t xy = nx * turn_fix(P, v.x) + ny * turn_fix(P, v.y);
          const uint64_t zz = nz * turn_fix(P, v.z);
          const double2 ep = turn_exp(xy + zz), em = turn_exp(xy - zz);
          o[0] = fma(w, ep.x, o[0]);
          o[1] = fma(w, ep.y, o[1]);
          o[2] = fma(w, em.x, o[2]);
          o[3] = fma(w, em.y, o[3]);
        }
        for (int c = 0; c < 4; c++) {
          o[c] = warp_sum(o[c]);
          if ((tid & 31) == 0) s_w[u & 1][tid >> 5][c] = o[c];
        }
        role_sync(1, kCb64K);  // (the other buffer is read before the next one)
        if (tid < tl) {
          double2 e[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
          for (int b = 0; b < 2; b++) {
            const uint64_t xy = nx * x[b] + ny * y[b], zz = nz * z[b];
            const double2 ep = turn_exp(xy + zz), em = turn_exp(xy - zz);
            e[0].x = fma(q[b], ep.x, e[0].x);
            e[0].y = fma(q[b], ep.y, e[0].y);
            e[1].x = fma(q[b], em.x, e[1].x);
            e[1].y = fma(q[b], em.y, e[1].y);
          }
          for (int h = 0; h < 2; h++) {
            const int k = h ? ku.km : ku.kp;
            if (k < 0) continue;
            double2 so = B.sk[k];
            if (pend) {
              const double2 d = B.dsk[(size_t)buf * P.n_k + k];
              so.x += d.x;
              so.y += d.y;
            }
            for (int w = 0; w < kCb64K / 32; w++) {
              so.x += s_w[u & 1][w][2 * h];
              so.y += s_w[u & 1][w][2 * h + 1];
            }
            acc += B.kw[k] * (2.0 * (so.x * e[h].x + so.y * e[h].y) +
                              (e[h].x * e[h].x + e[h].y * e[h].y));
          }
        }
      }
      if (tid < tl) slots[3 * (c0 + tid) + 2] = acc;
      role_sync(1, kCb64K);  // s_w is read
    }
  } else {
    const int id = tid - kth, nt = kCb64Threads - kth;
    const int lane = id & 31, sl = id >> 5, slices = nt >> 5;
    FixTab Tb = P.fx;
    if (J.charged) fix_stage(Tb, smem, id, nt);
    const auto tab = [&](uint64_t s) { return fix_h(Tb.c01, Tb.c23, Tb.c45, Tb.base, s); };
    const double unit = fix_scale(P), hs = 1.0 / Tb.unit;
    const int nb = J.charged ? 2 : 1;
    role_sync(2, nt);
    for (int c0 = 0; c0 < T; c0 += 32) {
      // (the lanes past the last trial repeat it)
      const int t = min(c0 + lane, T - 1);
      const double4_32a p1 = J.b1[t];
      const double4_32a p2 = J.charged ? J.b2[t] : p1;
      if (sl < nb) s_site[sl][lane] = fix64x4(P, sl ? p2 : p1);
      role_sync(2, nt);
      const ulonglong4_32a f1 = s_site[0][lane], f2 = nb > 1 ? s_site[1][lane] : f1;
      double lj = 0.0, re = 0.0;
      for (int j = (int)blockIdx.x * slices + sl; j < N + grown; j += (int)gridDim.x * slices) {
        if (j >= J.ex_lo && j < J.ex_hi) continue;
        const bool own = j >= N;
        const ulonglong4_32a o = own ? fix64x4(P, grown_bead(j - N)) : B.fpos64[j];
        const int k = J.type * P.n_type + (own ? J.type : B.type[j]);
        int64_t v = 0;  // the trial's table sum minus its counterion's
        double h = 0.0, none = 0.0;
        for (int b = 0; b < nb; b++) {
          const uint64_t dx = o.x - (b ? f2.x : f1.x), dy = o.y - (b ? f2.y : f1.y),
                         dz = o.z - (b ? f2.z : f1.z);
          uint64_t s0;
          if (J.charged) {
            const int64_t w = fix_term<kMode>(Tb, tab, dx, dy, dz, s0);
            v += b ? -w : w;
          } else {
            s0 = fix_near_r2<kMode>(dx, dy, dz);
          }
          if (s0 < Tb.s_near) {
            // no LJ with the preceding grown bead (cbmc.cc:57-58)
            const bool bonded = own && b == 0 && j - N == J.cl - 1;
            const double w = fix_near(P, b ? p2 : p1, own ? grown_bead(j - N) : B.pos[j],
                                      J.charged && s0 < Tb.s_lo, k, bonded ? none : lj);
            h += b ? -w : w;
          }
        }
        if (J.charged)
          re = fma(p1.w * __longlong_as_double((long long)o.w) * unit, (double)v + h * hs, re);
      }
      s_red[0][id] = lj;
      s_red[1][id] = re;
      role_sync(2, nt);
      if (sl < 2 && c0 + lane < T) {  // the slices of each sum, in order
        double x = 0.0;
        for (int w = 0; w < slices; w++) x += s_red[sl][w * 32 + lane];
        slots[3 * t + sl] = x;
        if (!kth && sl == 0) slots[3 * t + 2] = 0.0;
      }
      role_sync(2, nt);
    }
  }
}

constexpr int kCb64Sum = 128;

template <int kMode>
__global__ void __launch_bounds__(kCb64Sum)
    k_cbmc64_sum(const DevParams P, const DevBuffers B, CbmcJob J, int blocks) {
  __shared__ double s_w[kCb64Sum / 32][3];
  const int t = blockIdx.x, tid = threadIdx.x;
  double v[3] = {0.0, 0.0, 0.0};
  for (int b = tid; b < blocks; b += kCb64Sum)
    for (int c = 0; c < 3; c++) v[c] += J.slots[((size_t)b * J.n_trials + t) * 3 + c];
  for (int c = 0; c < 3; c++) {
    v[c] = warp_sum(v[c]);
    if ((tid & 31) == 0) s_w[tid >> 5][c] = v[c];
  }
  __syncthreads();
  if (tid) return;
  for (int c = 0; c < 3; c++) {
    v[c] = 0.0;
    for (int w = 0; w < kCb64Sum / 32; w++) v[c] += s_w[w][c];
  }
  const double4_32a b1 = J.b1[t], b2 = J.charged ? J.b2[t] : b1;
  double pair_e = v[0], ew = 0.0;
  if (J.charged) {
    const ulonglong4_32a f1 = fix64x4(P, b1), f2 = fix64x4(P, b2);
    uint64_t s0;
    const auto tab = [&](uint64_t s) {
      return fix_h(P.fx.c01, P.fx.c23, P.fx.c45, P.fx.base, s);
    };
    double re = (double)fix_term<kMode>(P.fx, tab, f2.x - f1.x, f2.y - f1.y, f2.z - f1.z, s0) *
                P.fx.unit;
    if (s0 < P.fx.s_near)
      re += fix_near(P, b1, b2, s0 < P.fx.s_lo, J.type * P.n_type + J.type, pair_e);
    if (P.use_ewald && pair_e < kVeryLarge) {
      ew = v[1] + P.kpref * v[2] + P.lB * P.sqrt_alpha * b1.w * b2.w * re;
      ew += P.self_coef * (b1.w * b1.w + b2.w * b2.w);
      if (P.real_cut >= P.ebox[0])  // a bead's own images
        ew += 0.5 * (cb_real(P, b1, b1) + cb_real(P, b2, b2));
    }
  } else if (P.use_ewald && P.n_k > 0 && pair_e < kVeryLarge) {
    // a neutral species' is zero, or NaN where it or a grown bead is not finite
    ew = J.lost ? __longlong_as_double(0x7FF8000000000000ll) : charge_of(b1);
  }
  if (P.use_ext) {
    pair_e += wall64(P, b1.z, J.type);
    if (J.charged) pair_e += wall64(P, b2.z, J.type);
  }
  J.u[t] = pair_e >= kVeryLarge ? kVeryLarge : pair_e + ew;
}

template <int kMode>
static void launch_one64(const DevParams& P, const DevBuffers& B, const CbmcJob& J,
                         cudaStream_t s) {
  static OncePerDevice once;
  allow_smem(once, k_cbmc64<kMode>, kFixMaxBins * 40);
  k_cbmc64<kMode><<<cbmc_blocks(), kCb64Threads, J.charged ? (size_t)P.fx.n_bin * 40 : 0, s>>>(
      P, B, J);
  k_cbmc64_sum<kMode><<<J.n_trials, kCb64Sum, 0, s>>>(P, B, J, cbmc_blocks());
}

void launch_cbmc64(const DevParams& P, const DevBuffers& B, const CbmcJob& J, cudaStream_t s) {
  if (P.fx.mode == 1)
    launch_one64<1>(P, B, J, s);
  else
    launch_one64<2>(P, B, J, s);
}

int cbmc_groups(const DevParams& P) {
  int g = (P.n_bead + kCbThreads * 4 - 1) / (kCbThreads * 4);
  return g < 1 ? 1 : (g > kCbmcGroups ? kCbmcGroups : g);
}

void launch_cbmc(const DevParams& P, const DevBuffers& B, const CbmcJob& J, cudaStream_t s) {
  if (P.use_ewald && P.n_k > 0) k_cbmc_so<<<(P.n_k + 255) / 256, 256, 0, s>>>(P, B, J);
  const int g = cbmc_groups(P);
  k_cbmc_sys<<<dim3(g, J.n_trials), kCbThreads, 0, s>>>(P, B, J);
  k_cbmc_fin<<<J.n_trials, kCbThreads, 0, s>>>(P, B, J, g);
}


// ------------------------------------------------------------- no-alloc
// Working memory of plum_cbmc_trials_noalloc, for callers that must not
// allocate device memory (hosts whose device memory belongs to their own
// allocator, or drivers that cannot take the device-wide synchronisation of
// cudaMalloc/cudaFree). One fixed array on every GPU
// that loads the library, held until the process exits:
//   trial beads + counterions  2 * kMaxTrials double4          16 KiB
//   grown chain + counterions  2 * kMaxChain  double4          64 KiB
//   S_o(k)                     kMaxK          double2         512 KiB
//   per-block sums             2 * kMaxTrials * kMaxGroups    256 KiB
//   results                    kMaxTrials     double            2 KiB
// Nothing in it has to start at zero: each call writes every element it
// reads (k_na_pack the beads and chain, k_cbmc_so all n_k entries of S_o,
// k_cbmc_sys one sum pair per (trial, block), k_cbmc_fin one result per
// trial) before reading it. All calls on a device share the array, so calls
// that overlap on the GPU race.
namespace na {
constexpr int kMaxTrials = 256, kMaxChain = 1024, kMaxK = 32768, kMaxGroups = kCbmcGroups;
constexpr size_t kBeadsOff = 0;
constexpr size_t kChainOff = kBeadsOff + sizeof(double4_32a) * 2 * kMaxTrials;
constexpr size_t kSoOff = kChainOff + sizeof(double4_32a) * 2 * kMaxChain;
constexpr size_t kPartOff = kSoOff + sizeof(double2) * kMaxK;
constexpr size_t kUOff = kPartOff + sizeof(double) * 2 * kMaxTrials * kMaxGroups;
constexpr size_t kBytes = kUOff + sizeof(double) * kMaxTrials;
}  // namespace na

static __device__ __align__(256) unsigned char g_cbmc_noalloc_scratch[na::kBytes];

// Device address of the scratch array per device, resolved on the first call
// made with that device current (a host-side name of a __device__ array is
// not a device address).
static std::mutex g_na_mu;
static unsigned char* g_na_ptr[64];

// Packs caller device arrays (xyz triples) into the scratch's double4 rows.
__global__ void k_na_pack(const double* b1, const double* b2, int T, const double* chain,
                          const double* chain_ci, int cl, double q1, double q2, int charged,
                          double4_32a* beads, double4_32a* cbuf) {
  for (int i = threadIdx.x; i < T; i += blockDim.x) {
    beads[i] = make_double4_32a(b1[3 * i], b1[3 * i + 1], b1[3 * i + 2], q1);
    beads[T + i] = charged ? make_double4_32a(b2[3 * i], b2[3 * i + 1], b2[3 * i + 2], q2)
                           : beads[i];
  }
  for (int i = threadIdx.x; i < cl; i += blockDim.x) {
    cbuf[i] = make_double4_32a(chain[3 * i], chain[3 * i + 1], chain[3 * i + 2], q1);
    cbuf[cl + i] = charged ? make_double4_32a(chain_ci[3 * i], chain_ci[3 * i + 1],
                                              chain_ci[3 * i + 2], q2)
                           : cbuf[i];
  }
}

int cbmc_trials_noalloc(const DevParams& P, const DevBuffers& B, cudaStream_t s, int device,
                        int n_trials, const double* d_b1, const double* d_b2, int chain_len,
                        const double* d_chain, const double* d_chain_ci, int type, int charged,
                        double q1, double q2, int ex_lo, int ex_hi, double* d_u, char* err,
                        int err_cap) {
  auto say = [&](const char* m) {
    if (err && err_cap > 0) snprintf(err, (size_t)err_cap, "%s", m);
  };
  if (n_trials < 1 || n_trials > na::kMaxTrials) {
    say("plum_cbmc_trials_noalloc: n_trials must be 1..256");
    return 1;
  }
  if (chain_len < 0 || chain_len > na::kMaxChain) {
    say("plum_cbmc_trials_noalloc: chain_len must be 0..1024");
    return 1;
  }
  if (P.n_k > na::kMaxK) {
    say("plum_cbmc_trials_noalloc: more than 32768 half-space k-vectors");
    return 1;
  }
  if (device < 0 || device >= 64) {
    say("plum_cbmc_trials_noalloc: device index out of range");
    return 1;
  }
  unsigned char* base = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (!g_na_ptr[device]) {
      void* p = nullptr;
      cudaError_t e = cudaGetSymbolAddress(&p, g_cbmc_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        say("plum_cbmc_trials_noalloc: cudaGetSymbolAddress failed");
        return 2;
      }
      g_na_ptr[device] = static_cast<unsigned char*>(p);
    }
    base = g_na_ptr[device];
  }
  double4_32a* beads = reinterpret_cast<double4_32a*>(base + na::kBeadsOff);
  double4_32a* cbuf = reinterpret_cast<double4_32a*>(base + na::kChainOff);
  k_na_pack<<<1, 256, 0, s>>>(d_b1, d_b2, n_trials, d_chain, d_chain_ci, chain_len, q1, q2,
                              charged, beads, cbuf);
  CbmcJob J;
  J.n_trials = n_trials;
  J.charged = charged;
  J.cl = chain_len;
  J.type = type;
  J.ex_lo = ex_lo;
  J.ex_hi = ex_hi;
  J.b1 = beads;
  J.b2 = beads + n_trials;
  J.chain = cbuf;
  J.chain_ci = cbuf + chain_len;
  J.s_o = reinterpret_cast<double2*>(base + na::kSoOff);
  J.part = reinterpret_cast<double*>(base + na::kPartOff);
  J.u = reinterpret_cast<double*>(base + na::kUOff);
  launch_cbmc(P, B, J, s);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(d_u, J.u, sizeof(double) * n_trials, cudaMemcpyDeviceToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    say(cudaGetErrorString(e));
    return 2;
  }
  return 0;
}

}  // namespace plum
