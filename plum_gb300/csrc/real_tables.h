// Tables of the real-space Ewald term, made on the host in long double.
#pragma once

#include <memory>
#include <vector>

#include "fix_pair.h"

namespace plum {

// The FP64 table of h(u): kH64Per bins per octave of u for octaves
// 2^kH64ELo .. 2^(kH64EHi - 1), a degree-8 polynomial in y = f - 1/2 per bin
// (kH64Stride doubles per bin, the last zero, for 16-byte loads): Chebyshev
// interpolation of erfcl at 9 nodes in long double, converted to powers of y.
// About 2e-16 relative below u = 8; above it h < 3e-5 and the absolute error
// stays below 1e-17. u below the table takes erfc / r directly.
constexpr int kH64ELo = -12, kH64EHi = 5, kH64Per = 32, kH64Stride = 10;
constexpr int kH64Bins = (kH64EHi - kH64ELo) * kH64Per;
const std::vector<double>& h64_table();  // kH64Bins * kH64Stride entries
// The same bins of g(u) = (h(u) + 2 e^{-u} / sqrt(kPi)) / u, the real-space
// force: (erfc(sqrt(alpha) r) / r + 2 sqrt(alpha / kPi) e^{-alpha r^2}) / r^2 =
// alpha^{3/2} g(alpha r^2) (kPi the reference's constant).
const std::vector<double>& g64_table();
// The integer pair form's table for a system (null where the form does not
// apply); t holds its constants, without the device pointers.
struct FixTable {
  std::vector<FixPair64> c01, c23;
  std::vector<FixPair32> c45;
  FixTab t;
};
// What the table depends on: a cubic box, r_c <= L; lj_max2 the largest squared
// LJ reach (0 without LJ).
struct FixSystem {
  double alpha, box, real_cut, lj_max2;
};
std::shared_ptr<const FixTable> fix_table(const FixSystem& P);
// The integer pair form's table: at most ten octaves of 128 bins.
constexpr int kFixMaxBins = 10 << kFixBinsLog;

}  // namespace plum
