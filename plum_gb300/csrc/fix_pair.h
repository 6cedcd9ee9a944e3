// The FP64 forms' real-space Ewald term in 64-bit integer arithmetic.
//
// GB300 issues an FP64 instruction every 16 cycles per SM, an integer one twice
// a cycle, so a pair evaluated in FP64 (a minimum image, r^2 and a degree-8
// polynomial: about 18 operations) costs 280 cycles per warp, and the same pair
// in integers about 45.
//
// Accuracy. Positions are fractions of the box (64 bits, of which 58 are kept within
// 16 boxes of the origin), r^2 a 64-bit integer, and h (below) has one absolute unit,
// 2.8e-17 for the bulk workloads, where an FP64 value is rounded relative to itself:
// the near pairs, which set a sum's error, are the better for it and the far ones the
// worse. A pair's h is off by at most 9e-16 with one image (L = 40, r_c = 20; L = 80,
// r_c = 40) and 7e-15 with image cells (L = 40, r_c = 28; L = 50, r_c = 34), nearest
// the table's lower end, where h itself is 7 to 8; around 0.9 r_c by 1e-16 to
// 2e-16, which is 5e-13, 2e-12 and (image cells) 7e-11 of h there, against 1e-15 of h
// from the FP64 polynomial. The Horner steps truncate, so most of that has a sign
// (low); charges of both signs cancel it. Whole results, against 64-bit sums and with
// FP64 pairs in brackets: a 20,000-bead frame (energies and S(k)) is off by 2.7e-15
// (2.7e-15), the energies of a 1,000-bead run by 1e-16 to 6e-16 (3e-16 to 8e-16),
// growth steps by 3e-17 (3e-17).
//
// Units. X = frac(x / L) 2^64 (fix64), d = X_b - X_a as a signed 64-bit number
// is the minimum-image difference. With shift = 0 (r_c <= L / 2) S = |d|^2 /
// 2^64 of the three components; with shift = 1 (r_c <= L) the components are
// halved first, so that the image a box length to the other side is the same
// number with its top bit flipped and still fits 64 bits. S is good to about 4
// units: at r = 1 and L = 80 an error of 7e-16 in r, below the rounding of x / L
// itself (9e-15), and the ratio of the two stays under 1 while L < 1000 r.
//
// Table. h(u) = erfc(sqrt u) / sqrt u, u = alpha r^2 = kappa S, in bins of
// 1/128 octave of S from s_lo (a power of two) on; a bin holds the degree-5
// Chebyshev interpolant in t = 1 - f, f the fraction of S inside its bin. h is
// completely monotone, so in t every coefficient is positive and the whole
// Horner scheme is unsigned: c0..c3 in 64 bits, c4 and c5 in 32, all scaled by
// 2^scale with h(s_lo) 2^scale < 2^58.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define PLUM_FIX_HD __host__ __device__ __forceinline__
#else
#define PLUM_FIX_HD inline
#endif

namespace plum {

constexpr int kFixBinsLog = 7;  // bins per octave of S

struct alignas(16) FixPair64 {
  uint64_t a, b;
};
struct alignas(8) FixPair32 {
  uint32_t a, b;
};

struct FixTab {
  int mode;   // 0: none; 1: one image (shift 0); 2: image cells (shift 1)
  int n_bin;
  int base;   // bin of S = (top byte of the normalised S) - 128 clz(S) + base
  int pad;
  uint64_t s_lo, s_cut;  // the table's first S; r_c^2
  uint64_t s_near;       // below it a pair takes the FP64 path (LJ reach, s_lo)
  double unit;           // 2^-scale
  const FixPair64* c01;  // [n_bin]
  const FixPair64* c23;
  const FixPair32* c45;
};

PLUM_FIX_HD uint32_t fix_mulhi(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

PLUM_FIX_HD int fix_clz(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return __clz((int)x);
#else
  return x ? __builtin_clz(x) : 32;
#endif
}

PLUM_FIX_HD int fix_ctz(uint32_t x) {  // x != 0
#if defined(__CUDA_ARCH__)
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}

// d = h 2^32 + l with a signed l: |d|^2 / 2^64 = h^2 + h l / 2^31 + l^2 / 2^64,
// the last under 1/4. Adds h^2 to hh and h l to hl.
PLUM_FIX_HD void fix_square(uint64_t d, uint64_t& hh, uint64_t& hl) {
  const int32_t h = (int32_t)((d + 0x80000000ull) >> 32), l = (int32_t)d;
  hh += (uint64_t)((int64_t)h * h);
  hl += (uint64_t)((int64_t)h * l);
}

PLUM_FIX_HD uint64_t fix_sum(uint64_t hh, uint64_t hl) {
  return hh + (uint64_t)((int64_t)hl >> 31);
}

PLUM_FIX_HD uint64_t fix_r2(uint64_t dx, uint64_t dy, uint64_t dz) {
  uint64_t hh = 0, hl = 0;
  fix_square(dx, hh, hl);
  fix_square(dy, hh, hl);
  fix_square(dz, hh, hl);
  return fix_sum(hh, hl);
}

// (v t) / 2^64 of a 64-bit v and the fraction t = (p, r), low partial product
// left out (under 1).
PLUM_FIX_HD uint64_t fix_mul(uint64_t v, uint32_t p, uint32_t r, uint64_t add) {
  const uint32_t a = (uint32_t)(v >> 32), b = (uint32_t)v;
  return (uint64_t)a * p + add + fix_mulhi(b, p) + fix_mulhi(a, r);
}

// h 2^scale at s_lo <= S <= s_cut. c01, c23, c45: the table (shared or global).
PLUM_FIX_HD uint64_t fix_h(const FixPair64* c01, const FixPair64* c23, const FixPair32* c45,
                           int base, uint64_t S) {
  const int lz = fix_clz((uint32_t)(S >> 32));
  const uint64_t m = S << lz;
  const int i = (int)(m >> 56) - (lz << kFixBinsLog) + base;
  const uint64_t t = ~(m << 8);
  const uint32_t p = (uint32_t)(t >> 32), r = (uint32_t)t;
  const FixPair64 k01 = c01[i], k23 = c23[i];
  const FixPair32 k45 = c45[i];
  const uint32_t v4 = k45.a + fix_mulhi(k45.b, p);
  const uint64_t v3 = k23.b + fix_mulhi(v4, p);
  const uint64_t v2 = k23.a + (uint64_t)(uint32_t)(v3 >> 32) * p + fix_mulhi((uint32_t)v3, p);
  const uint64_t v1 = fix_mul(v2, p, r, k01.b);
  return fix_mul(v1, p, r, k01.a);
}

// S of the nearest image alone.
template <int kMode>
PLUM_FIX_HD uint64_t fix_near_r2(uint64_t dx, uint64_t dy, uint64_t dz) {
  if (kMode == 1) return fix_r2(dx, dy, dz);
  return fix_r2((uint64_t)((int64_t)dx >> 1), (uint64_t)((int64_t)dy >> 1),
                (uint64_t)((int64_t)dz >> 1));
}

// The table sum (in table units) of one pair at difference d, image
// cells included; S of the nearest image in s0.
template <int kMode, class Tab>
PLUM_FIX_HD int64_t fix_term(const FixTab& T, const Tab& tab, uint64_t dx,
                                            uint64_t dy, uint64_t dz, uint64_t& s0) {
  const uint64_t span = T.s_cut - T.s_lo;
  if (kMode == 1) {
    s0 = fix_r2(dx, dy, dz);
    return s0 - T.s_lo <= span ? (int64_t)tab(s0) : 0;
  }
  const uint64_t flip = 1ull << 63;  // the image a box length to the other side
  dx = (uint64_t)((int64_t)dx >> 1);
  dy = (uint64_t)((int64_t)dy >> 1);
  dz = (uint64_t)((int64_t)dz >> 1);
  uint64_t hx = 0, mx = 0, hy = 0, my = 0, hz = 0, mz = 0;
  fix_square(dx, hx, mx);
  fix_square(dy, hy, my);
  fix_square(dz, hz, mz);
  const uint64_t ax = fix_sum(hx, mx), ay = fix_sum(hy, my), az = fix_sum(hz, mz);
  s0 = ax + ay + az;
  int64_t v = s0 - T.s_lo <= span ? (int64_t)tab(s0) : 0;
  hx = mx = hy = my = hz = mz = 0;
  fix_square(dx ^ flip, hx, mx);
  fix_square(dy ^ flip, hy, my);
  fix_square(dz ^ flip, hz, mz);
  const uint64_t bx = fix_sum(hx, mx), by = fix_sum(hy, my), bz = fix_sum(hz, mz);
  // images of one, two and three axes, those inside r_c one after the other
  unsigned in = 0;
#if defined(__CUDACC__)
#pragma unroll
#endif
  for (int c = 1; c < 8; c++) {
    const uint64_t s = (c & 1 ? bx : ax) + (c & 2 ? by : ay) + (c & 4 ? bz : az);
    if (s <= T.s_cut) in |= 1u << c;
  }
  while (in) {
    const int c = fix_ctz(in);
    in &= in - 1;
    v += (int64_t)tab((c & 1 ? bx : ax) + (c & 2 ? by : ay) + (c & 4 ? bz : az));
  }
  return v;
}

}  // namespace plum
