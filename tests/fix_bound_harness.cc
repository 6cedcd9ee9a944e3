// The table sums of the integer pair form (plum_gb300/csrc/fix_pair.h, real_tables.h)
// against long double and a bound on their error, term by term:
//
//   fix_bound_harness <alpha> <box> <real_cut> <pairs> <first seed> <seeds>
//
// h(u) = erfc(sqrt u) / sqrt u = (1 / sqrt pi) int_1^inf e^{-u t} t^{-1/2} dt, so its
// n-th derivative is (-1)^n G(n + 1/2, u) / (sqrt pi u^{n + 1/2}), G the upper
// incomplete gamma function: decreasing in u. With U the table unit, for one image:
//   interpolation  (w / 2)^6 / (2^5 6!) |h^(6)(lo)| on a bin [lo, lo + w], its six
//                  nodes being Chebyshev's
//   coefficients   1 U each (rounded to whole units; a rounding below zero to zero)
//   Horner         a step with a fraction cut to 32 bits: value 2^-32 + 1 U; with all
//                  64: 3 U (the partial products' floors and the one left out)
//   argument       |h'| times 6 units of S: the squares are cut by under 1.25 per axis,
//                  halved components by 0.5
//   long double    64 ulp of h, and 16 ulp of u, in the table's making and here
//
// Prints: mode, bins, unit, largest error, largest error over its bound, and the
// largest error and relative error of a single image between 0.85 and 0.95 r_c.
// Exits 1 on an index outside the table.
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../plum_gb300/csrc/real_tables.h"

using namespace plum;
typedef long double ld;

static const ld kSqrtPi = std::sqrt(3.141592653589793238462643383279503L);

static ld h_of(ld u) { return std::erfc(std::sqrt(u)) / std::sqrt(u); }

// |h^(n)(u)|: G(a + 1, u) = a G(a, u) + u^a e^{-u} from G(1/2, u) = sqrt(pi) erfc(sqrt u)
static ld h_derivative(int n, ld u) {
  ld g = kSqrtPi * std::erfc(std::sqrt(u)), a = 0.5L;
  for (int i = 0; i < n; i++, a += 1) g = a * g + std::pow(u, a) * std::exp(-u);
  return g / (kSqrtPi * std::pow(u, a));
}

int main(int argc, char** argv) {
  if (argc < 7) return 2;
  const double alpha = atof(argv[1]), box = atof(argv[2]), rc = atof(argv[3]);
  const int n = atoi(argv[4]), seed0 = atoi(argv[5]), seeds = atoi(argv[6]);
  const auto F = fix_table(FixSystem{alpha, box, rc, 6.25});
  if (!F) {
    std::printf("0 0 0 0 0 0 0\n");
    return 0;
  }
  const FixTab& T = F->t;
  const int shift = T.mode - 1;
  const ld kappa = (ld)alpha * box * box * std::ldexp((ld)1, 2 * shift - 64), U = T.unit;
  bool bad = false;
  const auto bin = [&](uint64_t s) {
    const int lz = fix_clz((uint32_t)(s >> 32));
    return (int)((s << lz) >> 56) - (lz << kFixBinsLog) + T.base;
  };
  const auto tab = [&](uint64_t s) {
    const int i = bin(s);
    if (i < 0 || i >= T.n_bin) {
      bad = true;
      return (uint64_t)0;
    }
    return fix_h(F->c01.data(), F->c23.data(), F->c45.data(), T.base, s);
  };
  const auto bound = [&](ld s) {
    const uint64_t at = (uint64_t)s;
    const int i = bin(at);
    if (i < 0 || i >= T.n_bin) return (ld)0;
    const int top = 63 - __builtin_clzll(at);
    const ld w = std::ldexp(1.0L, top - kFixBinsLog);
    const ld lo = std::floor((ld)at / w) * w;
    const ld c[6] = {(ld)F->c01[i].a, (ld)F->c01[i].b, (ld)F->c23[i].a,
                     (ld)F->c23[i].b, (ld)F->c45[i].a, (ld)F->c45[i].b};
    ld e = 1, v = c[5];  // the error so far, in units, and the value it is of
    for (int q = 4; q >= 0; q--) {
      e += 1 + (q >= 2 ? v * 0x1p-32L + 1 : 3);
      v += c[q];
    }
    const ld x = kappa * w / 2;
    const ld interp = std::pow(x, 6) / (32.0L * 720.0L) * h_derivative(6, kappa * lo);
    const ld arg = kappa * h_derivative(1, kappa * (s - 6)) * (6 + 16 * LDBL_EPSILON * s);
    return interp + e * U + arg + 64 * LDBL_EPSILON * h_of(kappa * lo);
  };
  tab(T.s_lo), tab(T.s_cut);
  ld worst = 0, ratio = 0, far = 0, far_rel = 0;
  for (int seed = seed0; seed < seed0 + seeds; seed++) {
    std::mt19937_64 g(seed);
    for (int k = 0; k < n; k++) {
      uint64_t d[3];  // all scales of separation, and the corners: 0 and half a box
      for (int a = 0; a < 3; a++) {
        const int s = (int)(g() % 12);
        d[a] = (uint64_t)((int64_t)g() >> s);
        if (k % 17 == a) d[a] = 0;
        if (k % 23 == a) d[a] = 1ull << 63;
      }
      uint64_t s0;
      const int64_t v = T.mode == 1 ? fix_term<1>(T, tab, d[0], d[1], d[2], s0)
                                    : fix_term<2>(T, tab, d[0], d[1], d[2], s0);
      ld want = 0, most = 0;
      bool edge = false;
      int images = 0;
      ld at = 0;
      for (int x = -shift; x <= shift; x++)
        for (int y = -shift; y <= shift; y++)
          for (int z = -shift; z <= shift; z++) {
            const ld dx = (ld)(int64_t)d[0] + x * 0x1p64L, dy = (ld)(int64_t)d[1] + y * 0x1p64L,
                     dz = (ld)(int64_t)d[2] + z * 0x1p64L;
            const ld s = (dx * dx + dy * dy + dz * dz) * 0x1p-64L / (shift ? 4 : 1);
            if (std::fabs(s - (ld)T.s_cut) < 64 || std::fabs(s - (ld)T.s_lo) < 64) edge = true;
            if (s > (ld)T.s_cut || s < (ld)T.s_lo) continue;
            want += h_of(kappa * s);
            most += bound(s);
            images++;
            at = std::sqrt(s / (ld)T.s_cut);
          }
      if (edge) continue;  // on the cut-off, or two images of an axis equally far
      const ld err = std::fabs((ld)v * U - want);
      if (most == 0 ? err != 0 : err > most * ratio) ratio = most == 0 ? 1e9L : err / most;
      if (err > worst) worst = err;
      if (images == 1 && at > 0.85L && at < 0.95L) {
        if (err > far) far = err;
        if (err / want > far_rel) far_rel = err / want;
      }
    }
  }
  std::printf("%d %d %.3Lg %.3Lg %.3Lg %.3Lg %.3Lg\n", T.mode, T.n_bin, U, worst, ratio, far,
              far_rel);
  return bad ? 1 : 0;
}
