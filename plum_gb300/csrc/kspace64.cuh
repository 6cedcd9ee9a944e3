// Reciprocal-space helpers of the FP64 kernels.
#pragma once

#include "device_common.cuh"
#include "engine.h"

namespace plum {

// A coordinate as a 64-bit fraction of a turn: frac(w / L) 2^64, times kPi / pi
// (the reference's phases are 2 kPi n w / L with its 12-digit kPi), so that n
// times it, mod 2^64, is the phase of n exactly. w / L is carried in two doubles:
// rounded to one it left e^{i theta} off by 2.5e-16, n times that in its n-th power, and
// S(k) of 20,000 beads further off (2.3e-15) than a sincos of the FP64 angle (1.9e-15).
__device__ __forceinline__ uint64_t turn64(const DevParams& P, double w, int axis) {
  double f = w * P.inv_ebox[axis];
  const double lo = fma(w, P.inv_ebox_lo[axis], fma(w, P.inv_ebox[axis], -f));
  double g = f - floor(f);
  if (axis < P.npbc) f = g;  // wrapped into the primary cell
  if (g >= 1.0) g = 0.0;     // a tiny negative w / L rounds up to 1
  return __double2ull_rn(g * 0x1p64) +
         (uint64_t)__double2ll_rn(fma(f, P.turn_eps, lo * 0x1p64));
}

// The same of a coordinate's box fraction X (fix64; a cubic periodic box): X kPi /
// pi, in integers.
__device__ __forceinline__ uint64_t turn_fix(const DevParams& P, uint64_t X) {
  return X + __umulhi((uint32_t)(X >> 32), P.turn_eps32);
}

// e^{2 pi i phi / 2^64}: the nearest quarter turn taken off in integers, then the
// Taylor series of sine and cosine on |theta| <= pi / 4 (through theta^15 and
// theta^16: the next terms are under 5e-17). About 20 FP64 operations, with no
// range reduction (sincos of a general argument: five times that).
__device__ __forceinline__ double2 turn_exp(uint64_t phi) {
  const int q = (int)((phi + (1ull << 61)) >> 62);
  const double t = (double)(int64_t)(phi - ((uint64_t)q << 62)) *
                   (6.283185307179586476925286766559 * 0x1p-64);
  const double x = t * t;
  double s = -1.0 / 1307674368000.0;
  s = fma(s, x, 1.0 / 6227020800.0);
  s = fma(s, x, -1.0 / 39916800.0);
  s = fma(s, x, 1.0 / 362880.0);
  s = fma(s, x, -1.0 / 5040.0);
  s = fma(s, x, 1.0 / 120.0);
  s = fma(s, x, -1.0 / 6.0);
  s = fma(s * x, t, t);
  double c = 1.0 / 20922789888000.0;
  c = fma(c, x, -1.0 / 87178291200.0);
  c = fma(c, x, 1.0 / 479001600.0);
  c = fma(c, x, -1.0 / 3628800.0);
  c = fma(c, x, 1.0 / 40320.0);
  c = fma(c, x, -1.0 / 720.0);
  c = fma(c, x, 1.0 / 24.0);
  c = fma(c, x, -0.5);
  c = fma(c, x, 1.0);
  const double a = q & 1 ? s : c, b = q & 1 ? c : s;  // |cos|, |sin| of the turn
  return make_double2(q == 1 || q == 2 ? -a : a, q & 2 ? -b : b);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// e^{i n theta} tables for one bead: tab[koff[axis] + n], n = 0..kmax[axis];
// q folded into the x table.
__device__ __forceinline__ void build_axis_table(const DevParams& P, double4_32a p,
                                                 int axis, double2* tab) {
  const double2 e1 = turn_exp(turn64(P, axis == 0 ? p.x : (axis == 1 ? p.y : p.z), axis));
  double2 e = axis == 0 ? make_double2(charge_of(p), 0.0) : make_double2(1.0, 0.0);
  double2* t = tab + P.koff[axis];
  t[0] = e;
  for (int n = 1; n <= P.kmax[axis]; n++) {
    e = cmul(e, e1);
    t[n] = e;
  }
}

// The xy part c = q e^{i(kx x + ky y)} of a unit's column from a bead's tables
// (q is folded into the x table).
__device__ __forceinline__ double2 unit_xy(const DevParams& P, const double2* tab, int nx, int ny) {
  const double2 ex = tab[P.koff[0] + nx];
  double2 ey = tab[P.koff[1] + (ny >= 0 ? ny : -ny)];
  if (ny < 0) ey.y = -ey.y;
  return cmul(ex, ey);
}

// Adds one bead to a unit's sums (xy from unit_xy, ez its e^{i nz theta_z}).
__device__ __forceinline__ void unit_add(double2 xy, double2 ez, double2& A, double2& B) {
  A.x = fma(xy.x, ez.x, A.x);
  A.y = fma(xy.y, ez.x, A.y);
  B.x = fma(xy.x, ez.y, B.x);
  B.y = fma(xy.y, ez.y, B.y);
}
// The unit's two structure factors, at +nz and -nz.
__device__ __forceinline__ double2 unit_plus(double2 A, double2 B) {
  return make_double2(A.x - B.y, A.y + B.x);
}
__device__ __forceinline__ double2 unit_minus(double2 A, double2 B) {
  return make_double2(A.x + B.y, A.y - B.x);
}

}  // namespace plum
