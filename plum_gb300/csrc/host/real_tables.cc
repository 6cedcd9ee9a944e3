#include "../real_tables.h"

#include <algorithm>
#include <cmath>
#include <mutex>

namespace plum {

// An FP64 table over u: per bin the degree-8 Chebyshev interpolant of f at the
// 9 Chebyshev nodes of y in [-1/2, 1/2] (u = lo + (y + 1/2) w), in long double,
// then rewritten in powers of y.
template <class F>
static std::vector<double> build_table64(F f_of) {
  constexpr int n = 9;
  const long double pi = 3.141592653589793238462643383279503L;
  long double T[n][n] = {};  // T_j(t) coefficients in powers of t
  T[0][0] = 1.0L;
  T[1][1] = 1.0L;
  for (int j = 2; j < n; j++)
    for (int q = 0; q < n; q++)
      T[j][q] = (q ? 2.0L * T[j - 1][q - 1] : 0.0L) - T[j - 2][q];
  long double tk[n], cs[n][n];  // nodes t = 2 y in [-1, 1], cos(j arccos t)
  for (int k = 0; k < n; k++) {
    tk[k] = std::cos(pi * (k + 0.5L) / n);
    for (int j = 0; j < n; j++) cs[j][k] = std::cos(pi * j * (k + 0.5L) / n);
  }
  std::vector<double> out((size_t)kH64Bins * kH64Stride, 0.0);
  int b = 0;
  for (int e = kH64ELo; e < kH64EHi; e++)
    for (int j = 0; j < kH64Per; j++, b++) {
      const long double lo = std::ldexp(1.0L + (long double)j / kH64Per, e);
      const long double w = std::ldexp(1.0L / kH64Per, e);
      long double f[n];
      for (int k = 0; k < n; k++) f[k] = f_of(lo + (0.5L * tk[k] + 0.5L) * w);
      long double mono[n] = {};  // powers of y
      for (int jj = 0; jj < n; jj++) {
        long double a = 0.0L;
        for (int k = 0; k < n; k++) a += f[k] * cs[jj][k];
        a *= (jj ? 2.0L : 1.0L) / n;
        for (int q = 0; q < n; q++) mono[q] += a * T[jj][q] * std::ldexp(1.0L, q);
      }
      for (int q = 0; q < n; q++) out[(size_t)b * kH64Stride + q] = (double)mono[q];
    }
  return out;
}

// The tables hold constants, so a process makes each once (5,000 long-double
// erfcs; on aarch64, where long double is done in software, tens of
// milliseconds that every context used to spend).
const std::vector<double>& h64_table() {
  static const std::vector<double> t = build_table64([](long double u) {
    const long double r = std::sqrt(u);
    return std::erfc(r) / r;
  });
  return t;
}

const std::vector<double>& g64_table() {
  static const std::vector<double> t = build_table64([](long double u) {
    const long double r = std::sqrt(u);
    return (std::erfc(r) / r + 2.0L / std::sqrt(3.14159265359L) * std::exp(-u)) / u;
  });
  return t;
}

// The integer pair form's table. It starts
// 512 times below r_c^2 (r_c / 23): nearer pairs, under 1e-4 of those inside r_c,
// take the FP64 path that LJ takes anyway. L <= 32 r_c keeps the granularity of
// S below the rounding of the coordinates there.
static bool build_fix_table(const FixSystem& P, FixTable* F) {
  constexpr int n = 6, per = 1 << kFixBinsLog;
  FixTab& T = F->t;
  T = FixTab{};
  const int shift = P.real_cut <= 0.5 * P.box ? 0 : 1;
  const long double L = P.box, rc = P.real_cut, pi = 3.141592653589793238462643383279503L;
  const long double units = std::ldexp(1.0L, 64 - 2 * shift) / (L * L);  // S per r^2
  const long double kappa = P.alpha / units, cut = rc * rc * units;
  T.s_cut = (uint64_t)cut;
  const int k1 = 63 - __builtin_clzll(T.s_cut), k0 = (int)std::floor(std::log2(cut / 512));
  if (k0 < 33) return false;
  const auto h = [](long double u) {
    const long double r = std::sqrt(u);
    return std::erfc(r) / r;
  };
  // sums of sixteen values below 2^58 stay in 64 bits, and 2^-scale is still
  // below the interpolant's own error
  int e;
  std::frexp(h(kappa * std::ldexp(1.0L, k0)), &e);
  const int scale = 58 - e;
  T.mode = 1 + shift;
  T.n_bin = (k1 - k0 + 1) * per;
  if (T.n_bin > kFixMaxBins) return false;
  T.base = per * (63 - k0) - 128;
  T.s_lo = (uint64_t)1 << k0;
  const long double near = P.lj_max2 > 0 ? P.lj_max2 * units + 8 : 0.0L;
  T.s_near = std::max(T.s_lo, near < 1.8e19L ? (uint64_t)near : ~(uint64_t)0);
  T.unit = std::ldexp(1.0, -scale);
  long double x[n];
  for (int k = 0; k < n; k++) x[k] = 0.5L * std::cos(pi * (k + 0.5L) / n) + 0.5L;
  const auto whole = [&](long double v, uint64_t most, uint64_t* out) {
    const long double w = std::ldexp(v, scale) + 0.5L;
    if (!(w >= 0.0L && w < (long double)most)) return false;
    *out = (uint64_t)w;
    return true;
  };
  for (int o = k0; o <= k1; o++)
    for (int j = 0; j < per; j++) {
      const long double lo = std::ldexp(1.0L + (long double)j / per, o);
      const long double w = std::ldexp(1.0L / per, o);
      // Newton's divided differences at the Chebyshev nodes, then powers of t
      long double a[n], mono[n] = {};
      for (int k = 0; k < n; k++) a[k] = h(kappa * (lo + (1.0L - x[k]) * w));
      for (int q = 1; q < n; q++)
        for (int k = n - 1; k >= q; k--) a[k] = (a[k] - a[k - 1]) / (x[k] - x[k - q]);
      for (int k = n - 1; k >= 0; k--) {
        for (int q = n - 1; q > 0; q--) mono[q] = mono[q - 1] - x[k] * mono[q];
        mono[0] = -x[k] * mono[0] + a[k];
      }
      uint64_t c[n];
      for (int q = 0; q < n; q++) {
        // (far out the coefficients fall below the unit, and may be a rounding
        // below zero)
        if (mono[q] < 0.0L && std::ldexp(mono[q], scale) > -1.0L) mono[q] = 0.0L;
        if (!whole(mono[q], (uint64_t)1 << (q < 4 ? 62 : 31), &c[q])) return false;
      }
      F->c01.push_back(FixPair64{c[0], c[1]});
      F->c23.push_back(FixPair64{c[2], c[3]});
      F->c45.push_back(FixPair32{(uint32_t)c[4], (uint32_t)c[5]});
    }
  return true;
}

// Contexts of one system (replicas) share the table: the last few are kept.
std::shared_ptr<const FixTable> fix_table(const FixSystem& P) {
  if (!(P.real_cut > 0.0 && P.real_cut <= P.box && P.box <= 32.0 * P.real_cut && P.alpha > 0.0))
    return nullptr;
  struct Entry {
    double key[4];
    std::shared_ptr<const FixTable> t;
  };
  static std::mutex mu;
  static std::vector<Entry> kept;
  const Entry want{{P.alpha, P.box, P.real_cut, P.lj_max2}, nullptr};
  std::lock_guard<std::mutex> lock(mu);
  for (const Entry& k : kept)
    if (std::equal(k.key, k.key + 4, want.key)) return k.t;
  auto t = std::make_shared<FixTable>();
  Entry made = want;
  if (build_fix_table(P, t.get())) made.t = t;
  if (kept.size() >= 8) kept.erase(kept.begin());
  kept.push_back(made);
  return made.t;
}

}  // namespace plum
