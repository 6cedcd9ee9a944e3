// Precision form: the pending move's energy difference with FP32 pair and
// k-space arithmetic (FP64 kept for S(k), the running totals and the
// periodic full recompute, see kern_energy.cu / capi.cu).
//
// Coordinates are mirrored as 32-bit fixed-point fractions of the Ewald box
// (fpos: X = round(w / L * 2^32), w wrapped into the primary cell on periodic
// axes). Then
//   * a minimum-image difference is one integer subtraction: int32 wraparound
//     is the periodic wrap, and the difference converts to FP32 with a
//     relative error of 2^-24 of |d| (close pairs stay accurate);
//   * the phase of k = 2 pi n / L is n * X mod 2^32 exactly (integer
//     multiply-add), so e^{i k.r} = sincospi(phase * 2^-31) has no FP32
//     range-reduction error.
// In the slab geometry z is not wrapped (|dz| < H < L_z,Ewald / 2), so the same
// subtraction gives the raw dz the reference uses (GetDistVector, npbc = 2). Where no
// dipole correction pads that box, z covers two of it (DevParams::z_turns).
//
// Per-thread and per-block sums are FP32; blocks are added in FP64 by the
// serial kernel.
#include <algorithm>
#include <cmath>

#include "engine.h"
#include "device_common.cuh"
#include "fix_device.cuh"
#include "fp32_pair.cuh"

namespace plum {

// Two sums of a block's values at once, one barrier pair; valid in thread 0. sh:
// 2 NT / 32 floats.
template <int NT>
__device__ __forceinline__ float2 block_sum32x2(float a, float b, float* sh) {
  static_assert(NT / 32 <= 16, "the warps' sums of both values in one warp");
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) {
    sh[w] = a;
    sh[NT / 32 + w] = b;
  }
  __syncthreads();
  float t = 0.0f;
  if (w == 0) {
    t = l < 2 * (NT / 32) ? sh[l] : 0.0f;
    for (int o = NT / 64; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    a = t;
    b = __shfl_sync(0xffffffffu, t, NT / 32);
  }
  return make_float2(a, b);
}

// ---------------------------------------------------------------- pair evaluation
// Constants of the table-driven real-space term. Lengths are real ones, or fixed-point
// units (cs: real r^2 per unit of r^2).
struct TabPair {
  float2 sx, sy, sz, ua;     // scales; table variable per r^2
  float rc2, ljlim, cs, ius; // cut-off; largest LJ cut-off^2; u per table variable
  unsigned last;             // the cut-off's bin: lanes beyond it share one address
  float bx, by, bz;          // DevParams::f_img
  int two;                   // DevParams::two_axes
};

// kCubic (equal fixed-point scales on the three axes): r^2 stays in fixed-point units
// and the box scale is folded into the constants.
template <bool kCubic, bool kCut>
__device__ __forceinline__ TabPair tab_pair(const DevParams& P, float cut_scale) {
  TabPair K;
  const float s0 = P.f_scale[0], s1 = P.f_scale[1], s2 = P.f_scale[2];
  K.sx = make_float2(s0, s0);
  K.sy = make_float2(s1, s1);
  K.sz = make_float2(s2, s2);
  K.cs = kCubic ? s0 * s0 : 1.0f;
  const float ics = 1.0f / K.cs;
  K.rc2 = P.f_real_cut * P.f_real_cut * ics;
  const float ua = P.f_sqrt_alpha * P.f_sqrt_alpha * K.cs * (kCut ? cut_scale : 1.0f);
  K.ua = make_float2(ua, ua);
  K.ius = kCut ? 1.0f / cut_scale : 1.0f;
  const int cut = __float_as_int(kCut ? (float)kH32Cut : K.rc2 * ua);
  K.last = max(0, min(kH32Bins - 1, (cut >> 18) - ((127 + kH32ELo) << 5)));
  K.ljlim = P.f_lj_max2 * ics;
  K.bx = P.f_img[0];
  K.by = P.f_img[1];
  K.bz = P.f_img[2];
  K.two = P.two_axes;
  return K;
}

// h at the trial r^2 (r.x) less h at the current one (r.y). kCut: the table is zero
// from the cut-off on; else a select at r_c. kNear: r may lie below the table.
template <bool kCut, bool kNear>
__device__ __forceinline__ float tab_diff(const TabPair& K, const float4* s_h, float2 r) {
  const float2 u = __fmul2_rn(r, K.ua);
  const int b1 = __float_as_int(u.x), b0 = __float_as_int(u.y);
  float h1 = h32_tab(s_h, b1, K.last), h0 = h32_tab(s_h, b0, K.last);
  if (kNear && min(b1, b0) < kH32LoBits) {
    if (b1 < kH32LoBits) h1 = h32_small(u.x * K.ius);
    if (b0 < kH32LoBits) h0 = h32_small(u.y * K.ius);
  }
  if (!kCut) {
    h1 = r.x <= K.rc2 ? h1 : 0.0f;
    h0 = r.y <= K.rc2 ? h0 : 0.0f;
  }
  return h1 - h0;
}

__device__ __forceinline__ float2 sq2(float2 a) { return __fmul2_rn(a, a); }
__device__ __forceinline__ float2 add3(float2 a, float2 b, float2 c) {
  return __fadd2_rn(__fadd2_rn(a, b), c);
}
// the image a box length to the other side: |d| -> L - |d|
__device__ __forceinline__ float2 flip2(float b, float2 d) {
  return make_float2(b - fabsf(d.x), b - fabsf(d.y));
}

// The real-space change (in units of lB sqrt(alpha) q q') of staged bead (t trial, c
// current) with other bead (ot, oc), and the LJ change. kImg (r_c below every box
// length): an axis has at most one more image in range, the one on the other side, and
// two axes at once have one only where r_c reaches past half a face's diagonal. (Leaving
// out the lookups of neutral staged beads, a branch per bead, gained nothing on brushes
// with 13 to 77 % of their beads charged and cost 5 % on a fully charged system.)
template <bool kCubic, bool kCut, bool kImg>
__device__ __forceinline__ float tab_eval(const DevParams& P, const TabPair& K, const float4* s_h,
                                          const int4 t, const int4 c, const int4 ot, const int4 oc,
                                          int k, float& acc_lj) {
  float2 dx = make_float2((float)(int)((unsigned)ot.x - (unsigned)t.x),
                          (float)(int)((unsigned)oc.x - (unsigned)c.x));
  float2 dy = make_float2((float)(int)((unsigned)ot.y - (unsigned)t.y),
                          (float)(int)((unsigned)oc.y - (unsigned)c.y));
  float2 dz = make_float2((float)(int)((unsigned)ot.z - (unsigned)t.z),
                          (float)(int)((unsigned)oc.z - (unsigned)c.z));
  if (!kCubic) {
    dx = __fmul2_rn(dx, K.sx);
    dy = __fmul2_rn(dy, K.sy);
    dz = __fmul2_rn(dz, K.sz);
  }
  if (!kImg) {
    const float2 r = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
    if (fminf(r.x, r.y) < K.ljlim)
      acc_lj += lj32(P, k, r.x * K.cs) - lj32(P, k, r.y * K.cs);
    return tab_diff<kCut, true>(K, s_h, r);
  }
  const float2 xx = sq2(dx), yy = sq2(dy), zz = sq2(dz);
  const float2 r = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, zz));  // (LJ's: two roundings less)
  if (fminf(r.x, r.y) < K.ljlim) acc_lj += lj32(P, k, r.x) - lj32(P, k, r.y);
  float h = tab_diff<kCut, true>(K, s_h, r);
  const float2 fx = sq2(flip2(K.bx, dx)), fy = sq2(flip2(K.by, dy)), fz = sq2(flip2(K.bz, dz));
  if (K.bx < kNoImage) h += tab_diff<kCut, false>(K, s_h, add3(fx, yy, zz));
  if (K.by < kNoImage) h += tab_diff<kCut, false>(K, s_h, add3(xx, fy, zz));
  if (K.bz < kNoImage) h += tab_diff<kCut, false>(K, s_h, add3(xx, yy, fz));
  if (K.two) {
    const float2 xy = add3(fx, fy, zz), xz = add3(fx, yy, fz), yz = add3(xx, fy, fz);
    if (fminf(fminf(fminf(xy.x, xy.y), fminf(xz.x, xz.y)), fminf(yz.x, yz.y)) <= K.rc2) {
      h += tab_diff<kCut, false>(K, s_h, xy) + tab_diff<kCut, false>(K, s_h, xz);
      h += tab_diff<kCut, false>(K, s_h, yz) + tab_diff<kCut, false>(K, s_h, add3(fx, fy, fz));
    }
  }
  return h;
}

// ---------------------------------------------------------------- one system
// As the FP64 form's k_delta64: one block per SM but for the SMs that the next
// move's candidates run on, k warps that own a run of k units and pair warps that
// deal out the (moved, other) pairs; each block leaves three sums to the serial
// step. What bounds it for a short move is latency, so a thread takes one other bead
// against a run of staged moved beads and the h(u) table is copied to shared memory
// (10 KB); for a long one the FP32 pipe (some 25 instructions per evaluation).
// With 20,000 beads and 7,812 k-vectors: 13.4 us, and 21.5 us a move (32.6 and 34.3 us
// with every pair's four loads, k tiles x bead groups and a ticket for the last block).
// Hard spheres and a cut-off beyond the table or the box take the general pair loop
// below.
constexpr int kD32Threads = 768;
constexpr int kD32K = 256;      // k role
constexpr int kD32Stage = 256;  // moved beads staged at a time
constexpr int kD32Run = 4;      // most moved beads per thread and other bead
constexpr int kD32Units = 32;   // k units of a block at a time

struct Stage32 {
  int4 t, c;  // trial (w: charge as float bits), current (w: row of the LJ table)
};

__host__ __device__ inline int k_beads32(const DevParams& P) {
  const int fit = kKTableBytes / (2 * (P.kmax[2] + 1 + kD32Units) * (int)sizeof(float2));
  return fit < 1 ? 1 : (fit > 64 ? 64 : fit);
}

__device__ __forceinline__ float2 turn32(unsigned phi) {
  float s, c;
  sincospif((float)(int)phi * 4.6566128730773926e-10f, &s, &c);  // * 2^-31
  return make_float2(c, s);
}

// The pairs of pair thread t0 of nt: LJ + Ewald, the h(u) table.
template <bool kImg>
__device__ __forceinline__ void sweep32(const DevParams& P, const DevBuffers& B, Stage32* st,
                                        float4* s_h, int t0, int nt, int b_lo, int m,
                                        float& acc_lj, float& acc_re) {
  const int N = P.n_bead, n_type = P.n_type;
  const int G = (int)gridDim.x * nt, p0 = (int)blockIdx.x * nt + t0;
  const long long pairs = (long long)m * N;
  const int run_len = pairs >= 2LL * kD32Run * G ? kD32Run : (pairs >= 4LL * G ? 2 : 1);
  const TabPair K = tab_pair<false, false>(P, 0.0f);
  const float pref = P.f_lB * P.f_sqrt_alpha;
  for (int i = t0; i < kH32Bins; i += nt) s_h[i] = P.htab[i];
  for (int g0 = 0; g0 < m; g0 += kD32Stage) {
    const int gn = min(kD32Stage, m - g0);
    if (g0) role_sync(2, nt);  // the previous group is consumed
    for (int t = t0; t < gn; t += nt) {
      const int i = b_lo + g0 + t;
      int4 a = B.ftrial[g0 + t], c = B.fpos[i];
      a.w = __float_as_int(B.fq[i]);
      c.w *= n_type;
      st[t] = Stage32{a, c};
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
      // a moved other bead: its trial position, and only moved beads before it
      const int4 o0 = B.fpos[j];
      const float qj = B.fq[j] * pref;
      const int l = j - b_lo - g0;
      const bool jm = j >= b_lo && j < b_lo + m;
      const int4 o1 = jm ? B.ftrial[j - b_lo] : o0;
      const int u0 = run * run_len, u1 = min(gn, jm ? min(l, u0 + run_len) : u0 + run_len);
      float acc = 0.0f;
      for (int u = u0; u < u1; u++) {
        const int4 t = st[u].t, c = st[u].c;
        acc = fmaf(__int_as_float(t.w),
                   tab_eval<false, false, kImg>(P, K, s_h, t, c, o1, o0, c.w + o0.w, acc_lj),
                   acc);
      }
      acc_re = fmaf(qj, acc, acc_re);
    }
  }
}

// dS(k), the S(k) commit and the |S|^2 change of units [u0, u1). smem, kb =
// k_beads32: [kb][2][zn] e^{i nz theta_z}, then [kb][2][kD32Units] xy parts, every
// entry from its exact integer phase.
__device__ __forceinline__ float k_role32(const DevParams& P, const DevBuffers& B,
                                          unsigned char* smem, int u0, int u1, int b_lo, int b_hi,
                                          int sk_pend, int sk_buf, int cur_buf) {
  const int zn = P.kmax[2] + 1, kb = k_beads32(P);
  float2* s_z = reinterpret_cast<float2*>(smem);
  float2* s_xy = s_z + (size_t)kb * 2 * zn;
  __shared__ short2 s_col[kD32Units];
  __shared__ float s_sum[4][kD32K];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float e = 0.0f;
  for (int c0 = u0; c0 < u1; c0 += kD32Units) {
    const int un = min(kD32Units, u1 - c0);
    // the units' (nx, ny) columns, numbered in order (the same in every warp)
    const KUnit lu = lane < un ? B.ku[c0 + lane] : KUnit{0, 0, 0, 0, -1, -1};
    const int px = __shfl_up_sync(0xffffffffu, lu.nx, 1), py = __shfl_up_sync(0xffffffffu, lu.ny, 1);
    const bool head = lane < un && (lane == 0 || px != lu.nx || py != lu.ny);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int ncol = __popc(heads);
    int zmax = lane < un ? lu.nz : 0;
    for (int o = 16; o > 0; o >>= 1) zmax = max(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    const int slices = kD32K / un;
    const int u = (int)threadIdx.x % un, sl = (int)threadIdx.x / un;
    const int col = __popc(heads & (0xffffffffu >> (31 - u))) - 1;
    const int nz = __shfl_sync(0xffffffffu, (int)lu.nz, u);
    if (warp == 0 && head)
      s_col[__popc(heads & (0xffffffffu >> (31 - lane))) - 1] = make_short2(lu.nx, lu.ny);
    float2 A = make_float2(0.0f, 0.0f), Bs = A;
    for (int g0 = b_lo; g0 < b_hi; g0 += kb) {
      const int nt = 2 * min(kb, b_hi - g0);
      role_sync(1, kD32K);  // the tables (and s_sum) are free, s_col is written
      // one entry per thread: nt x (zmax + 1) z phases, then nt x ncol xy phases
      for (int t = threadIdx.x; t < nt * (zmax + 1 + ncol); t += kD32K) {
        const int c = t / nt, it = t - c * nt;
        const int bead = g0 + (it >> 1);
        const int4 f = (it & 1) ? B.fpos[bead] : B.ftrial[bead - b_lo];
        if (c <= zmax) {
          s_z[(size_t)it * zn + c] = turn32((unsigned)f.z * (P.z_turns * (unsigned)c));
        } else {
          const short2 kc = s_col[c - zmax - 1];
          const float2 v = turn32((unsigned)f.x * (unsigned)(int)kc.x +
                                  (unsigned)f.y * (unsigned)(int)kc.y);
          const float q = (it & 1) ? -B.fq[bead] : B.fq[bead];  // trial minus current
          s_xy[it * kD32Units + c - zmax - 1] = make_float2(q * v.x, q * v.y);
        }
      }
      role_sync(1, kD32K);
      if (sl < slices)
        for (int b = 2 * sl; b < nt; b += 2 * slices)
#pragma unroll
          for (int it = b; it < b + 2; it++) {  // both places of a bead (see k_item32)
            const float2 xy = s_xy[it * kD32Units + col], ez = s_z[(size_t)it * zn + nz];
            A.x = fmaf(xy.x, ez.x, A.x);
            A.y = fmaf(xy.y, ez.x, A.y);
            Bs.x = fmaf(xy.x, ez.y, Bs.x);
            Bs.y = fmaf(xy.y, ez.y, Bs.y);
          }
    }
    s_sum[0][threadIdx.x] = A.x;
    s_sum[1][threadIdx.x] = A.y;
    s_sum[2][threadIdx.x] = Bs.x;
    s_sum[3][threadIdx.x] = Bs.y;
    role_sync(1, kD32K);
    // the slices of each (unit, sum), added in order by a thread each
    if ((int)threadIdx.x < 4 * un) {
      const int q = (int)threadIdx.x / un, v = (int)threadIdx.x % un;
      float t = 0.0f;
      for (int w = 0; w < slices; w++) t += s_sum[q][w * un + v];
      s_sum[q][v] = t;  // slice 0's place: read by this thread only
    }
    role_sync(1, kD32K);
    if (warp < 2 && lane < un) {  // warp 0: +nz, warp 1: -nz
      const int k = warp == 0 ? lu.kp : lu.km;
      if (k >= 0) {
        const float2 SA = make_float2(s_sum[0][lane], s_sum[1][lane]);
        const float2 SB = make_float2(s_sum[2][lane], s_sum[3][lane]);
        const float2 ds = warp == 0 ? make_float2(SA.x - SB.y, SA.y + SB.x)
                                    : make_float2(SA.x + SB.y, SA.y - SB.x);
        double2 s = B.sk[k];
        if (sk_pend) {
          const double2 p = B.dsk[(size_t)sk_buf * P.n_k + k];
          s = make_double2(s.x + p.x, s.y + p.y);
          B.sk[k] = s;
        }
        B.dsk[(size_t)cur_buf * P.n_k + k] = make_double2((double)ds.x, (double)ds.y);
        const float sx = (float)s.x, sy = (float)s.y;
        e += (float)B.kw[k] * (2.0f * (sx * ds.x + sy * ds.y) + (ds.x * ds.x + ds.y * ds.y));
      }
    }
  }
  return e;
}

// kMode: 0 the general pair loop, 1 one image, 2 image cells (DevParams::images)
template <int kMode>
__global__ void __launch_bounds__(kD32Threads, 1)
    k_delta32(const DevParams P, const DevBuffers B, int tab_bytes) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float s_part[kD32Threads / 32][2];
  const DevState* st = B.state;
  const int b_lo = st->b_lo, b_hi = st->b_hi;
  const int m = st->pending ? b_hi - b_lo : 0;
  const int kthreads = P.use_ewald && P.n_ku > 0 ? kD32K : 0;
  const int warp = threadIdx.x >> 5;
  float a = 0.0f, b = 0.0f;  // k role: k energy; pair role: LJ and real space
  if ((int)threadIdx.x < kthreads) {
    const int u0 = (int)((long long)P.n_ku * blockIdx.x / gridDim.x);
    const int u1 = (int)((long long)P.n_ku * (blockIdx.x + 1) / gridDim.x);
    if (m > 0)
      a = k_role32(P, B, smem + tab_bytes, u0, u1, b_lo, b_hi, st->sk_pending, st->sk_buf,
                   st->cur_buf);
  } else {
    const int t0 = (int)threadIdx.x - kthreads, nt = kD32Threads - kthreads;
    const int N = P.n_bead;
    if (kMode) {
      if (m > 0)
        sweep32<kMode == 2>(P, B, reinterpret_cast<Stage32*>(smem),
                            reinterpret_cast<float4*>(smem + kD32Stage * sizeof(Stage32)), t0, nt,
                            b_lo, m, a, b);
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
        const int4 ti = B.ftrial[ii], ci = B.fpos[i];
        const float qi = B.fq[i], qj = B.fq[j];
        const int4 cj = B.fpos[j];
        const int4 tj = jm ? B.ftrial[j - b_lo] : cj;
        float l1 = 0, r1 = 0, l0 = 0, r0 = 0;
        pair32(P, ti, qi, tj, qj, l1, r1);
        pair32(P, ci, qi, cj, qj, l0, r0);
        if (!hs_bonded(P, B.mol_start, i, j)) a += l1 - l0;
        b += r1 - r0;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_part[warp][0] = a;
    s_part[warp][1] = b;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    // sums 0 LJ, 1 real space over the pair warps, 2 over the k warps
    const int kw = kthreads / 32, w0 = threadIdx.x == 2 ? 0 : kw;
    const int w1 = threadIdx.x == 2 ? kw : kD32Threads / 32;
    float t = 0.0f;
    for (int w = w0; w < w1; w++) t += s_part[w][threadIdx.x == 1];
    B.partial[4 * blockIdx.x + threadIdx.x] = (double)t;
  }
}

int pair_grid32() { return 4 * device_sms(); }

template <int kMode>
static void launch_delta32(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  const size_t tab = kMode ? kD32Stage * sizeof(Stage32) + kH32Bins * sizeof(float4) : 0;
  static OncePerDevice once;
  allow_smem(once, k_delta32<kMode>, kKTableBytes + 4096 + tab);
  const size_t k = P.use_ewald && P.n_ku > 0
                       ? (size_t)k_beads32(P) * 2 * (P.kmax[2] + 1 + kD32Units) * sizeof(float2)
                       : 0;
  k_delta32<kMode><<<delta_blocks(), kD32Threads, tab + k, s>>>(P, B, (int)tab);
}

void launch_delta_pairs32(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  const int mode = P.htab && P.pair_kind == 0 && P.use_ewald ? P.images : 0;
  if (mode == 1)
    launch_delta32<1>(P, B, s);
  else if (mode == 2)
    launch_delta32<2>(P, B, s);
  else
    launch_delta32<0>(P, B, s);
}

// Loop constants of a replica's pair sweep, in registers.
struct PairConst {
  float sx, sy, sz, rc, sa, lB, ljmax2;
  int nt, use_pair, use_ewald;
};

__device__ __forceinline__ PairConst pair_const(const DevParams& P) {
  PairConst K;
  K.sx = P.f_scale[0];
  K.sy = P.f_scale[1];
  K.sz = P.f_scale[2];
  K.rc = P.f_real_cut;
  K.sa = P.f_sqrt_alpha;
  K.lB = P.f_lB;
  K.nt = P.n_type;
  K.use_pair = P.use_pair;
  K.use_ewald = P.use_ewald;
  K.ljmax2 = P.f_lj_max2;
  return K;
}

// pair32 with the LJ table read only inside the largest LJ cut-off and, for
// kSingle (r_c <= L/2 on every axis), the minimum image inlined.
template <bool kSingle>
__device__ __forceinline__ void pair32k(const DevParams& P, const PairConst& K, int4 a, float qa,
                                        int4 b, float qb, float& lj, float& re) {
  const float dx = fdiff(a.x, b.x, K.sx);
  const float dy = fdiff(a.y, b.y, K.sy);
  const float dz = fdiff(a.z, b.z, K.sz);
  const float r2 = dx * dx + dy * dy + dz * dz;
  if (K.use_pair && r2 < K.ljmax2) lj += lj32(P, a.w * K.nt + b.w, r2);
  if (K.use_ewald) {
    const float qq = qa * qb;
    if (qq != 0.0f) {
      float e = 0.0f;
      if (kSingle) {
        if (r2 <= K.rc * K.rc) e = real_term32(P, r2);
      } else {
        e = real_images32(P, dx, dy, dz);
      }
      re += K.lB * qq * e;
    }
  }
}

// One thread per other bead j in [c0, c1) (moved beads skipped), against the
// gn staged moved beads at their trial (s_mt[u]) and current
// (s_mt[kPairGroup + u]) positions.
template <bool kSingle>
__device__ __forceinline__ float2 pair_sweep(const DevParams& P, const DevBuffers& B,
                                          const int4* s_mt, const float* s_mq, int gn, int g_lo,
                                          int c0, int c1, int b_lo, int b_hi) {
  const PairConst K = pair_const(P);
  const bool hs = P.pair_kind == 1;
  float acc_lj = 0.0f, acc_re = 0.0f;
  for (int j = c0 + threadIdx.x; j < c1; j += kPairThreads) {
    if (j >= b_lo && j < b_hi) continue;  // moved pairs: the last item
    const int4 cj = B.fpos[j];
    const float qj = B.fq[j];
#pragma unroll 2
    for (int u = 0; u < gn; u++) {
      float l1 = 0, r1 = 0, l0 = 0, r0 = 0;
      pair32k<kSingle>(P, K, s_mt[u], s_mq[u], cj, qj, l1, r1);
      pair32k<kSingle>(P, K, s_mt[kPairGroup + u], s_mq[u], cj, qj, l0, r0);
      if (!(hs && hs_bonded(P, B.mol_start, g_lo + u, j))) acc_lj += l1 - l0;
      acc_re += r1 - r0;
    }
  }
  return make_float2(acc_lj, acc_re);
}

// ------------------------------------------------ table-driven real space
// pair_sweep for LJ + Ewald from the h(u) table: per (moved u, other j) the trial and
// current distances share the other bead's load, one LJ pre-test and the packed
// (two-lane FP32) arithmetic of r^2 and u, so a warp runs no divergent erfc. A thread
// takes one other bead; in an item of fewer others than threads, several threads share
// the staged beads of each. The trial entry's w holds the staged bead's charge (float
// bits) and the current entry's w its type; the other bead's charge multiplies its sum
// once, after the staged beads. kCut: the table is the batch's cut table (variable
// u' = cut_scale u, zero from the cut-off on), so the cut-off costs nothing.
template <bool kCubic, bool kCut, bool kImg>
__device__ __forceinline__ float2 pair_sweep_tab(const DevParams& P, const DevBuffers& B,
                                                 const int4* s_mt, const float4* s_h, int gn,
                                                 int chunk, int c0, int c1, int b_lo, int b_hi,
                                                 float cut_scale) {
  float acc_lj = 0.0f, acc_re = 0.0f;
  const TabPair K = tab_pair<kCubic, kCut>(P, cut_scale);
  const float pref = P.f_lB * P.f_sqrt_alpha;
  const int nt = P.n_type;
  const int per = min(chunk, kPairThreads), split = kPairThreads / per;
  const int sub = (int)threadIdx.x / per;
  const int u0 = gn * sub / split, u1 = sub < split ? gn * (sub + 1) / split : u0;
  for (int j = c0 + (int)threadIdx.x - sub * per; j < c1; j += per) {
    if (j >= b_lo && j < b_hi) continue;  // moved pairs: the last item
    const int4 o = B.fpos[j];
    const float q = B.fq[j] * pref;
    float a = 0.0f;
#pragma unroll(kImg ? 2 : 4)
    for (int u = u0; u < u1; u++) {
      const int4 t = s_mt[u], c = s_mt[kPairGroup + u];
      a = fmaf(__int_as_float(t.w),
               tab_eval<kCubic, kCut, kImg>(P, K, s_h, t, c, o, o, c.w * nt + o.w, acc_lj),
               a);
    }
    acc_re = fmaf(q, a, acc_re);
  }
  return make_float2(acc_lj, acc_re);
}

// The pairs among the m moved beads, each once, from the table: rows a and m - 1 - a
// together hold m - 1 pairs, dealt out by columns.
template <bool kCut, bool kImg>
__device__ __forceinline__ float2 moved_pairs_tab(const DevParams& P, const DevBuffers& B,
                                               const float4* s_h, int b_lo, int m,
                                               float cut_scale) {
  float acc_lj = 0.0f, acc_re = 0.0f;
  const TabPair K = tab_pair<false, kCut>(P, cut_scale);
  const float pref = P.f_lB * P.f_sqrt_alpha;
  const int n = ((m + 1) / 2) * (m - 1);
  for (int p = threadIdx.x; p < n; p += kPairThreads) {
    int a = p / (m - 1), b = p - a * (m - 1);
    if (b < m - 1 - a) {
      b += a + 1;
    } else {
      if (2 * a == m - 1) continue;  // the middle row stands alone
      a = m - 1 - a;
      b++;
    }
    const int4 c = B.fpos[b_lo + a], oc = B.fpos[b_lo + b];
    const float h = tab_eval<false, kCut, kImg>(P, K, s_h, B.ftrial[a], c, B.ftrial[b], oc,
                                                c.w * P.n_type + oc.w, acc_lj);
    acc_re = fmaf(B.fq[b_lo + a] * B.fq[b_lo + b] * pref, h, acc_re);
  }
  return make_float2(acc_lj, acc_re);
}

// The table (kH32Bins float4): per bin the cubic in w = f / 32 (f the
// bin-local fraction) through h(u' / scale) at the four Chebyshev nodes of the
// bin, h in double precision from std::erfc; the 4 x 4 Vandermonde system in
// f solved by Gaussian elimination with partial pivoting, the coefficients
// then scaled by powers of 32 (exactly) to the kernel's w. With cut > 0 every
// bin at or above u' = cut is zero.
void build_h32_table(float4* out, double scale, double cut) {
  const double kPi = 3.14159265358979323846;
  int i = 0;
  for (int e = kH32ELo; e < kH32EHi; e++)
    for (int j = 0; j < kH32Per; j++, i++) {
      const double lo = std::ldexp(1.0 + (double)j / kH32Per, e);
      const double w = std::ldexp(1.0 / kH32Per, e);
      if (cut > 0.0 && lo >= cut) {
        out[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        continue;
      }
      double A[4][5];
      for (int k = 0; k < 4; k++) {
        const double f = 0.5 + 0.5 * std::cos(kPi * (k + 0.5) / 4.0);  // in (0, 1)
        const double u = (lo + f * w) / scale;
        const double r = std::sqrt(u);
        double p = 1.0;
        for (int q = 0; q < 4; q++, p *= f) A[k][q] = p;
        A[k][4] = std::erfc(r) / r;
      }
      for (int col = 0; col < 4; col++) {
        int piv = col;
        for (int rr = col + 1; rr < 4; rr++)
          if (std::fabs(A[rr][col]) > std::fabs(A[piv][col])) piv = rr;
        for (int q = 0; q < 5; q++) std::swap(A[col][q], A[piv][q]);
        for (int rr = 0; rr < 4; rr++) {
          if (rr == col) continue;
          const double g = A[rr][col] / A[col][col];
          for (int q = col; q < 5; q++) A[rr][q] -= g * A[col][q];
        }
      }
      double c[4];
      for (int q = 0; q < 4; q++) c[q] = std::ldexp(A[q][4] / A[q][q], 5 * q);  // f^q = 32^q w^q
      out[i] = make_float4((float)c[0], (float)c[1], (float)c[2], (float)c[3]);
    }
}

// ------------------------------------------------------------ replicas
constexpr int kKUnitsMost = kPairThreads;  // most k units of a k item

// dS(k), the S(k) commit and the |S|^2 change of units [u0, u0 + un), at most
// kKUnitsMost. A thread takes one unit and every slices-th moved bead, at its trial and
// its current place (the two nearly cancel: dealt out to different threads, as every
// other entry, they left partial sums of the trial places alone, whose rounding put the
// energy change off by 3.6 times as much in a bulk and 7 times in a slab). smem:
// e^{i nz theta_z} of as many moved beads (trial and current) as fit, then their xy
// parts per (nx, ny) column, every entry one thread's, from its exact integer phase.
// (A vector's phase as a product of three table entries, the tables built by six
// threads a bead: four times the instructions per vector.)
__device__ __forceinline__ float k_item32(const DevParams& P, const DevBuffers& B,
                                          unsigned char* smem, int smem_bytes, int u0, int un,
                                          int b_lo, int b_hi, int sk_pend, int sk_buf,
                                          int cur_buf) {
  __shared__ short2 s_col[kKUnitsMost];
  __shared__ float s_sum[4][kPairThreads];
  __shared__ int s_zmax;
  const int slices = kPairThreads / un;
  const int u = (int)threadIdx.x % un, sl = (int)threadIdx.x / un;
  const KUnit ku = B.ku[u0 + u];
  const int col0 = B.ku[u0].col;
  const int ncol = ((B.ku[u0 + un - 1].col - col0) & 0xFFFF) + 1, col = (ku.col - col0) & 0xFFFF;
  if (threadIdx.x == 0) s_zmax = 0;
  __syncthreads();
  const int zw = __reduce_max_sync(0xffffffffu, (int)ku.nz);
  if ((threadIdx.x & 31) == 0 && zw > 0) atomicMax(&s_zmax, zw);
  if (sl == 0) s_col[col] = make_short2(ku.nx, ku.ny);
  float2 A = make_float2(0.0f, 0.0f), Bs = A;
  __syncthreads();
  const int nz = s_zmax + 1, ne = nz + ncol;
  const int kb = min(64, smem_bytes / (2 * ne * (int)sizeof(float2)));
  float2* s_z = reinterpret_cast<float2*>(smem);
  float2* s_xy = s_z + (size_t)kb * 2 * nz;
  for (int g0 = b_lo; g0 < b_hi; g0 += kb) {
    const int nt = 2 * min(kb, b_hi - g0);
    if (g0 > b_lo) __syncthreads();  // the tables are free
    for (int t = threadIdx.x; t < nt * ne; t += kPairThreads) {
      const int c = t / nt, it = t - c * nt;
      const int bead = g0 + (it >> 1);
      const int4 f = (it & 1) ? B.fpos[bead] : B.ftrial[bead - b_lo];
      if (c < nz) {
        s_z[it * nz + c] = turn32((unsigned)f.z * (P.z_turns * (unsigned)c));
      } else {
        const short2 kc = s_col[c - nz];
        const float2 v = turn32((unsigned)f.x * (unsigned)(int)kc.x +
                                (unsigned)f.y * (unsigned)(int)kc.y);
        const float w = (it & 1) ? -B.fq[bead] : B.fq[bead];  // trial minus current
        s_xy[it * ncol + c - nz] = make_float2(w * v.x, w * v.y);
      }
    }
    __syncthreads();
    if (sl < slices) {
#pragma unroll 2
      for (int b = 2 * sl; b < nt; b += 2 * slices)
#pragma unroll
        for (int it = b; it < b + 2; it++) {
          const float2 xy = s_xy[it * ncol + col], ez = s_z[it * nz + ku.nz];
          A.x = fmaf(xy.x, ez.x, A.x);
          A.y = fmaf(xy.y, ez.x, A.y);
          Bs.x = fmaf(xy.x, ez.y, Bs.x);
          Bs.y = fmaf(xy.y, ez.y, Bs.y);
        }
    }
  }
  s_sum[0][threadIdx.x] = A.x;
  s_sum[1][threadIdx.x] = A.y;
  s_sum[2][threadIdx.x] = Bs.x;
  s_sum[3][threadIdx.x] = Bs.y;
  __syncthreads();
  // slices 0 and 1: +nz and -nz (one thread for both where there is one slice)
  float e = 0.0f;
  if (sl > 1 || sl >= slices) return e;
  A = Bs = make_float2(0.0f, 0.0f);
  for (int w = 0; w < slices; w++) {  // the slices of each (unit, sum), added in order
    A.x += s_sum[0][w * un + u];
    A.y += s_sum[1][w * un + u];
    Bs.x += s_sum[2][w * un + u];
    Bs.y += s_sum[3][w * un + u];
  }
  for (int h = sl; h < 2; h += slices > 1 ? 2 : 1) {
    const int k = h ? ku.km : ku.kp;
    if (k < 0) continue;
    const float2 ds = h ? make_float2(A.x + Bs.y, A.y - Bs.x) : make_float2(A.x - Bs.y, A.y + Bs.x);
    double2 s = B.sk[k];
    if (sk_pend) {
      const double2 p = B.dsk[(size_t)sk_buf * P.n_k + k];
      s = make_double2(s.x + p.x, s.y + p.y);
      B.sk[k] = s;
    }
    B.dsk[(size_t)cur_buf * P.n_k + k] = make_double2((double)ds.x, (double)ds.y);
    const float sx = (float)s.x, sy = (float)s.y;
    e += (float)B.kw[k] * (2.0f * (sx * ds.x + sy * ds.y) + (ds.x * ds.x + ds.y * ds.y));
  }
  return e;
}

// Batched replicas: every replica's pending move contributes pair items
// (up to kPairGroup moved beads, staged in shared memory at their trial and
// current positions, x a chunk of other beads), one item for the pairs among the
// moved beads, and k items (k_tile / 2 units over all moved beads). Every block
// derives the same item list from the replicas' states; its first item is its own
// number, the next ones come from a queue, drawn while the one before is worked on.
// Each item writes its own slot: pair items {lj, real}, k items {k-space energy
// change}. The serial step of each replica adds its slots in item order, so the
// result does not depend on which block took which item.
// The item sizes, the grid and the register budget (kMinBlocks resident
// blocks per SM) are run-time choices (BatchTune, picked by
// plum_batch_autotune); defaults: 4096 pairs per item, 64 units per k item,
// 4 blocks per SM, 2 resident.
template <int kMinBlocks>
__global__ void __launch_bounds__(kPairThreads, kMinBlocks)
    k_batch_delta32(const DevParams* __restrict__ rp, const DevBuffers* __restrict__ rb,
                    int n_rep, int* __restrict__ item_off, double* __restrict__ slots,
                    BatchTune tune, int* __restrict__ queue, const float4* __restrict__ htab,
                    float cut_scale, int smem_bytes) {
  const int kItemPairs = tune.item_pairs, kUnitsPer = min(tune.k_tile / 2, kKUnitsMost);
  extern __shared__ __align__(16) unsigned char smem_all[];
  // the staging / k-table area, the h(u) table where there is one, the item counts
  unsigned char* smem = smem_all;
  float4* s_h = reinterpret_cast<float4*>(smem_all + smem_bytes);
  int* s_pref = reinterpret_cast<int*>(s_h + (htab ? kH32Bins : 0));  // [n_rep + 1]
  int* s_np = s_pref + n_rep + 1;                                     // [n_rep]
  int* s_lo = s_np + n_rep;                                           // [n_rep]
  int* s_m = s_lo + n_rep;                                            // [n_rep]
  if (htab)
    for (int i = threadIdx.x; i < kH32Bins; i += blockDim.x) s_h[i] = htab[i];
  __shared__ float red[2 * (kPairThreads / 32)];
  __shared__ int s_item;
  // 1. item counts per replica and their prefix (same in every block)
  for (int r = threadIdx.x; r < n_rep; r += blockDim.x) {
    const DevState* st = rb[r].state;
    // a move rejected by the surrogate's stage one has no exact change
    const int m = (st->pending && !st->da_skip) ? st->b_hi - st->b_lo : 0;
    const DevParams& pr = rp[r];
    const int np = (pr.use_pair || pr.use_ewald) ? pair_item_count(m, pr.n_bead, kItemPairs) : 0;
    const int nk = (pr.use_ewald && m > 0) ? (pr.n_ku + kUnitsPer - 1) / kUnitsPer : 0;
    s_np[r] = np;
    s_lo[r] = st->b_lo;
    s_m[r] = m;
    s_pref[r + 1] = np + nk;
  }
  __syncthreads();
  if (threadIdx.x < 32) {  // a run of replicas per lane, then across the lanes
    const int per = (n_rep + 31) / 32, r0 = min(n_rep, (int)threadIdx.x * per);
    const int r1 = min(n_rep, r0 + per);
    int sum = 0;
    for (int r = r0; r < r1; r++) sum += s_pref[r + 1];
    int off = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, off, o);
      if ((int)threadIdx.x >= o) off += v;
    }
    off -= sum;
    for (int r = r0; r < r1; r++) {
      off += s_pref[r + 1];
      s_pref[r + 1] = off;
    }
    if (threadIdx.x == 0) s_pref[0] = 0;
  }
  __syncthreads();
  if (blockIdx.x == 0)
    for (int r = threadIdx.x; r < n_rep; r += blockDim.x) {
      item_off[4 * r] = s_pref[r];
      item_off[4 * r + 1] = s_np[r];
      item_off[4 * r + 2] = s_pref[r] + s_np[r];
      item_off[4 * r + 3] = s_pref[r + 1] - s_pref[r] - s_np[r];
    }
  // 2. items are taken one at a time: blocks that drew cheap items take more.
  // Every item writes only its own slot, so the results do not depend on which
  // block took it. The last block to run out resets the queue for the next launch.
  const int T = s_pref[n_rep];
  int item = blockIdx.x;
  while (item < T) {
    int next = 0;
    if (threadIdx.x == 0) next = (int)gridDim.x + atomicAdd(&queue[0], 1);
    // replica of this item (s_pref is ascending)
    int lo = 0, hi = n_rep - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (s_pref[mid] <= item) lo = mid; else hi = mid - 1;
    }
    const int r = lo;
    const DevParams& P = rp[r];
    const DevBuffers& B = rb[r];
    const int b_lo = s_lo[r], m = s_m[r], b_hi = b_lo + m, N = P.n_bead;
    const int local = item - s_pref[r];
    if (local < s_np[r]) {
      float2 acc = make_float2(0.0f, 0.0f);  // LJ, real space
      const int chunk = pair_chunk(m, kItemPairs);
      const int n_chunk = (N + chunk - 1) / chunk;
      const int n_grid = ((m + kPairGroup - 1) / kPairGroup) * n_chunk;
      const int tab = htab && P.pair_kind == 0 && P.use_ewald ? P.images : 0;
      if (local < n_grid) {
        const int g0 = (local / n_chunk) * kPairGroup, gn = min(kPairGroup, m - g0);
        const int c0 = (local % n_chunk) * chunk, c1 = min(N, c0 + chunk);
        int4* s_mt = reinterpret_cast<int4*>(smem);  // trial, then current
        float* s_mq = reinterpret_cast<float*>(s_mt + 2 * kPairGroup);
        // (the barriers at the end of the item loop: every thread is done
        // with the previous item's staging area)
        for (int u = threadIdx.x; u < gn; u += kPairThreads) {
          const float q = B.fq[b_lo + g0 + u];
          int4 t = B.ftrial[g0 + u];
          if (tab) t.w = __float_as_int(q);  // the type stays in c.w
          s_mt[u] = t;
          s_mt[kPairGroup + u] = B.fpos[b_lo + g0 + u];
          s_mq[u] = q;
        }
        __syncthreads();
        const bool cubic = tab == 1 && P.npbc == 3 && P.f_scale[0] == P.f_scale[1] &&
                           P.f_scale[1] == P.f_scale[2];
        const float cs = cut_scale;
        if (!tab) {
          acc = P.single_image
                    ? pair_sweep<true>(P, B, s_mt, s_mq, gn, b_lo + g0, c0, c1, b_lo, b_hi)
                    : pair_sweep<false>(P, B, s_mt, s_mq, gn, b_lo + g0, c0, c1, b_lo, b_hi);
        } else if (cs > 0.0f) {
          if (cubic)
            acc = pair_sweep_tab<true, true, false>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                    cs);
          else if (tab == 1)
            acc = pair_sweep_tab<false, true, false>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                     cs);
          else
            acc = pair_sweep_tab<false, true, true>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                    cs);
        } else if (cubic) {
          acc = pair_sweep_tab<true, false, false>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                   cs);
        } else if (tab == 1) {
          acc = pair_sweep_tab<false, false, false>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                    cs);
        } else {
          acc = pair_sweep_tab<false, false, true>(P, B, s_mt, s_h, gn, chunk, c0, c1, b_lo, b_hi,
                                                   cs);
        }
      } else if (tab) {
        acc = cut_scale > 0.0f ? moved_pairs_tab<true, true>(P, B, s_h, b_lo, m, cut_scale)
                               : moved_pairs_tab<false, true>(P, B, s_h, b_lo, m, cut_scale);
      } else {
        // pairs among the moved beads, each once (both trial / both current)
        const int lane = threadIdx.x & 31;
        for (int a = threadIdx.x >> 5; a < m; a += kPairThreads / 32)
          for (int bb = a + 1 + lane; bb < m; bb += 32) {
          float l1 = 0, r1 = 0, l0 = 0, r0 = 0;
          pair32(P, B.ftrial[a], B.fq[b_lo + a], B.ftrial[bb], B.fq[b_lo + bb], l1, r1);
          pair32(P, B.fpos[b_lo + a], B.fq[b_lo + a], B.fpos[b_lo + bb], B.fq[b_lo + bb], l0,
                 r0);
          // the moved beads are one molecule's: neighbours are bonded
          if (!(P.pair_kind == 1 && bb == a + 1)) acc.x += l1 - l0;
          acc.y += r1 - r0;
        }
      }
      const float2 ab = block_sum32x2<kPairThreads>(acc.x, acc.y, red);
      if (threadIdx.x == 0) {
        slots[2 * item] = (double)ab.x;
        slots[2 * item + 1] = (double)ab.y;
      }
    } else {
      const int u0 = (local - s_np[r]) * kUnitsPer;
      const DevState* st = B.state;
      const float e = k_item32(P, B, smem, smem_bytes, u0, min(kUnitsPer, P.n_ku - u0), b_lo, b_hi,
                         st->sk_pending, st->sk_buf, st->cur_buf);
      const float2 ek = block_sum32x2<kPairThreads>(e, 0.0f, red);
      if (threadIdx.x == 0) {
        slots[2 * item] = (double)ek.x;
        slots[2 * item + 1] = 0.0;
      }
    }
    __syncthreads();  // this item is done with the staging area and s_item
    if (threadIdx.x == 0) s_item = next;
    __syncthreads();
    item = s_item;
  }
  // every block takes its last (empty) item before it counts itself out, so
  // the last one out knows that no block will read the queue again
  if (threadIdx.x == 0 && atomicAdd(&queue[1], 1) == (int)gridDim.x - 1) {
    queue[0] = 0;
    queue[1] = 0;
  }
}

constexpr int kKAreaBytes = 16 * 1024;

int batch_delta_smem(const DevParams& P) {
  const int k = P.use_ewald ? 2 * (P.kmax[2] + 1 + kKUnitsMost) * (int)sizeof(float2) : 0;
  return std::max(kKAreaBytes, k);  // (the staged beads of a pair item take 2.2 KB)
}

void launch_batch_delta32(const DevParams* rp, const DevBuffers* rb, int n_rep, int* item_off,
                          double* slots, size_t smem, BatchTune tune, int* queue,
                          const float4* htab, float cut_scale, cudaStream_t s) {
  static OncePerDevice once[3];
  constexpr size_t most = kKAreaBytes + 2 * (kMaxKmax + 1 + kKUnitsMost) * sizeof(float2) +
                          kH32Bins * sizeof(float4) + (4 * kMaxReplicas + 1) * sizeof(int);
  allow_smem(once[0], k_batch_delta32<2>, most);
  allow_smem(once[1], k_batch_delta32<3>, most);
  allow_smem(once[2], k_batch_delta32<4>, most);
  const int grid = tune.grid > 0 ? tune.grid : pair_grid32();
  if (!tune.htab) htab = nullptr;
  if (!htab) cut_scale = 0.0f;
  const int area = (int)smem;
  if (htab) smem += kH32Bins * sizeof(float4);
  smem += (4 * (size_t)n_rep + 1) * sizeof(int);
  if (tune.min_blocks == 4)
    k_batch_delta32<4><<<grid, kPairThreads, smem, s>>>(rp, rb, n_rep, item_off, slots, tune,
                                                        queue, htab, cut_scale, area);
  else if (tune.min_blocks == 3)
    k_batch_delta32<3><<<grid, kPairThreads, smem, s>>>(rp, rb, n_rep, item_off, slots, tune,
                                                        queue, htab, cut_scale, area);
  else
    k_batch_delta32<2><<<grid, kPairThreads, smem, s>>>(rp, rb, n_rep, item_off, slots, tune,
                                                        queue, htab, cut_scale, area);
}

__global__ void k_fix_all(const DevParams P, const DevBuffers B) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < P.n_bead; i += gridDim.x * blockDim.x) {
    double4_32a p = B.pos[i];
    B.fpos[i] = fix_point(P, p, B.type[i]);
    B.fq[i] = (float)p.w;
  }
}

void launch_fix_all(const DevParams& P, const DevBuffers& B, cudaStream_t s) {
  k_fix_all<<<(P.n_bead + 255) / 256, 256, 0, s>>>(P, B);
}

}  // namespace plum
