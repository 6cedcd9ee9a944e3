// Reciprocal-space helpers of the FP64 kernels.
#pragma once

#include "engine.h"

namespace plum {

// e^{i n theta} tables for one bead: tab[koff[axis] + n], n = 0..kmax[axis];
// q folded into the x table.
__device__ __forceinline__ void build_axis_table(const DevParams& P, double4_32a p,
                                                 int axis, double2* tab) {
  double w = axis == 0 ? p.x : (axis == 1 ? p.y : p.z);
  if (axis < P.npbc) w -= P.ebox[axis] * floor(w * P.inv_ebox[axis]);
  double s, c;
  sincos(P.kunit[axis] * w, &s, &c);
  double2 e = axis == 0 ? make_double2(p.w, 0.0) : make_double2(1.0, 0.0);
  double2* t = tab + P.koff[axis];
  t[0] = e;
  for (int n = 1; n <= P.kmax[axis]; n++) {
    double re = e.x * c - e.y * s;
    double im = e.x * s + e.y * c;
    e = make_double2(re, im);
    t[n] = e;
  }
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
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
