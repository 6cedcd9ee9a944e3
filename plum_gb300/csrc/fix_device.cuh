// Device side of the integer pair form (fix_pair.h), and small helpers of the
// FP64 kernels that use it.
#pragma once

#include "device_common.cuh"
#include "engine.h"

namespace plum {

// LJ of one pair at squared distance r2 (the reference's r <= 0 overlap gives
// the 1e8 sentinel).
__device__ __forceinline__ double lj64(const DevParams& P, int k, double r2) {
  if (P.pair_kind == 1) return sqrt(r2) <= P.hs_sum[k] ? kVeryLarge : 0.0;  // hard spheres
  if (r2 <= 0.0) return kVeryLarge;
  if (r2 < P.lj_rc2[k]) {
    double s2 = P.lj_sig2[k] / r2;
    double s6 = s2 * s2 * s2;
    return P.lj_eps4[k] * (s6 * s6 - s6) - P.lj_eref[k];
  }
  return 0.0;
}

__device__ __forceinline__ double wrap_d(double d, double L, double invL) {
  return d - L * rint(d * invL);
}

// A pair near enough for LJ or below the table, in FP64 from the beads'
// positions (whose difference is exact for near pairs; the box's fractions carry
// the rounding of x / L, which r^-12 would magnify). Adds LJ to lj; returns h
// where the table has none.
__device__ __forceinline__ double fix_near(const DevParams& P, double4_32a a, double4_32a b,
                                           bool below, int k, double& lj) {
  const double x = wrap_d(b.x - a.x, P.box[0], P.inv_box[0]);
  const double y = wrap_d(b.y - a.y, P.box[1], P.inv_box[1]);
  const double z = wrap_d(b.z - a.z, P.box[2], P.inv_box[2]);
  const double r2 = x * x + y * y + z * z;
  if (P.use_pair && r2 < P.lj_max2) lj += lj64(P, k, r2);
  return below && r2 > 0.0 ? real_term64(P, r2) / P.sqrt_alpha : 0.0;
}

// lB sqrt(alpha) per table unit.
__device__ __forceinline__ double fix_scale(const DevParams& P) {
  return P.lB * P.sqrt_alpha * P.fx.unit;
}

// The table copied to shared memory (n_bin * 40 bytes at s, threads t of nt; the
// caller's barrier follows), where a warp's gather goes at a bank's pace and not
// a line's.
__device__ __forceinline__ void fix_stage(FixTab& T, unsigned char* s, int t, int nt) {
  FixPair64* s01 = reinterpret_cast<FixPair64*>(s);
  FixPair64* s23 = s01 + T.n_bin;
  FixPair32* s45 = reinterpret_cast<FixPair32*>(s23 + T.n_bin);
#pragma unroll 4
  for (int i = t; i < T.n_bin; i += nt) {
    s01[i] = T.c01[i];
    s23[i] = T.c23[i];
    s45[i] = T.c45[i];
  }
  T.c01 = s01, T.c23 = s23, T.c45 = s45;
}

// Barrier of one role's threads.
__device__ __forceinline__ void role_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

}  // namespace plum
