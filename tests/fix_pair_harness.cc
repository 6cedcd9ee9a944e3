// The integer pair form (plum_gb300/csrc/fix_pair.h, real_tables.h), compiled
// here for the host, against long-double arithmetic.
//
//   fix_pair_harness <alpha> <box> <real_cut> <n> <seed>
//
// Prints: mode, bins, unit, the largest error of the table sum over n random
// pairs (in units of 1e-16) and that error over its bound, the bound being
//   8 table units (rounding and truncation of the Horner steps)
//   + 2^-55 h (the degree-5 interpolant)
//   + |dh/dS| x 6 units of S (the truncated squares).
// Exits 1 on an index outside the table.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../plum_gb300/csrc/real_tables.h"

using namespace plum;
typedef long double ld;

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const double alpha = atof(argv[1]), box = atof(argv[2]), rc = atof(argv[3]);
  const int n = atoi(argv[4]);
  const auto F = fix_table(FixSystem{alpha, box, rc, 6.25});
  if (!F) {
    std::printf("0 0 0 0 0\n");
    return 0;
  }
  const FixTab& T = F->t;
  const int shift = T.mode - 1;
  const ld kappa = (ld)alpha * box * box * std::ldexp((ld)1, 2 * shift - 64);
  const auto h = [&](ld s) {
    const ld r = std::sqrt(kappa * s);
    return std::erfc(r) / r;
  };
  bool bad = false;
  const auto tab = [&](uint64_t s) {
    const int lz = fix_clz((uint32_t)(s >> 32));
    const int i = (int)((s << lz) >> 56) - (lz << kFixBinsLog) + T.base;
    if (i < 0 || i >= T.n_bin) {
      bad = true;
      return (uint64_t)0;
    }
    return fix_h(F->c01.data(), F->c23.data(), F->c45.data(), T.base, s);
  };
  tab(T.s_lo), tab(T.s_cut);
  std::mt19937_64 g(atoi(argv[5]));
  ld worst = 0, ratio = 0;
  for (int k = 0; k < n; k++) {
    // all scales of separation, and the corners: 0 and half a box
    uint64_t d[3];
    for (int a = 0; a < 3; a++) {
      const int s = (int)(g() % 12);
      d[a] = (uint64_t)((int64_t)g() >> s);
      if (k % 17 == a) d[a] = 0;
      if (k % 23 == a) d[a] = 1ull << 63;
    }
    uint64_t s0;
    const int64_t v = T.mode == 1 ? fix_term<1>(T, tab, d[0], d[1], d[2], s0)
                                  : fix_term<2>(T, tab, d[0], d[1], d[2], s0);
    ld want = 0, bound = 0;
    bool edge = false;
    const int m = shift;  // images -1..1 per axis when r_c may pass L / 2
    for (int x = -m; x <= m; x++)
      for (int y = -m; y <= m; y++)
        for (int z = -m; z <= m; z++) {
          const ld dx = (ld)(int64_t)d[0] + x * 0x1p64L, dy = (ld)(int64_t)d[1] + y * 0x1p64L,
                   dz = (ld)(int64_t)d[2] + z * 0x1p64L;
          const ld s = (dx * dx + dy * dy + dz * dz) * 0x1p-64L / (shift ? 4 : 1);
          if (std::fabs(s - (ld)T.s_cut) < 64 || std::fabs(s - (ld)T.s_lo) < 64) edge = true;
          if (s > (ld)T.s_cut || s < (ld)T.s_lo) continue;
          want += h(s);
          bound += 8 * (ld)T.unit + 0x1p-55L * h(s) + 6 * std::fabs(h(s + 1024) - h(s)) / 1024;
        }
    // ties: on the cut-off, and the two images of an axis at exactly half a box
    // or of a zero component a box length away
    if (edge) continue;
    const ld err = std::fabs((ld)v * (ld)T.unit - want);
    if (bound == 0 ? err != 0 : err > bound * ratio) ratio = bound == 0 ? 1e9L : err / bound;
    if (err > worst) worst = err;
  }
  std::printf("%d %d %.3Lg %.3Lg %.3Lg\n", T.mode, T.n_bin, (ld)T.unit, worst * 1e16L, ratio);
  return bad ? 1 : 0;
}
