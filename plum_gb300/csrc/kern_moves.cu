// Serial part of a Monte Carlo step. Two kernels:
//
// k_serial64 / k_batch_serial, one block per system, on the step's critical path:
//   finish  takes the pending move's pair and k sums (the delta kernel's) and its
//           wall, bond and q dz sums (the generator's) and composes dE exactly as
//           ForceField::EnergyDifference does (force_field.cc:407-434): pair,
//           early return at >= 1e8, external, early return, Ewald (real +
//           reciprocal + the dipole term from the *current* z, which is what
//           the reference evaluates at potential_ewald.cc:527-531), bond.
//   decide  one draw u; accept if dE < 1e8 and u < exp(-beta dE); no draw at
//           dE >= 1e8 (simulation.cc:324-332)
//   commit  trial -> current, running totals (force_field.cc:436-451,
//           simulation.cc:336-351); S(k) += dS(k) is left to the next delta kernel
//   adopt   the next move: the candidate that came true
//
// k_gen / k_batch_gen, one block per candidate, beside the energy change:
//   the next step's draws in the reference's order: one draw for the GC check
//   (simulation.cc:221), chain and ion picks, move type (simulation.cc:247-276),
//   then the move itself (molecule.cc:103-312), its walls
//   (potential_external.cc:100-117), bonds (potential_spring.cc:63-80) and q dz.
//
// Generating a move is a chain of dependent draws, scans and FP64 arithmetic on
// one block; as part of the serial step it stood on the critical path of every
// move (1,000 beads: 40 us per move with it there, 30 us beside the energy
// change; 21 us with the shorter chains below and the energy change on one block
// per SM. 32 replicas of 20,000 beads: the serial step 36 us, 24 us, 13 us).
//
// Build note: this file is compiled with -fmad=false. The draw-consuming
// tests (randSphere's r1^2 + r2^2 > 1, the move-type and pick thresholds)
// must round exactly like the reference or the draw sequence would diverge.
#include "engine.h"
#include "mlp.h"
#include "device_common.cuh"
#include "unit_draw.h"

namespace plum {


struct Draws {
  const uint32_t* g;
  const uint32_t* win;
  long long pos, len, wbase;
  int wlen;
  int overrun;
  __device__ uint32_t next() {
    if (pos >= len) {
      overrun = 1;
      return 0u;
    }
    long long o = pos - wbase;
    uint32_t v = (o >= 0 && o < wlen) ? win[o] : g[pos];
    pos++;
    return v;
  }
  __device__ double u() { return unit_draw(next()); }
  __device__ uint32_t at(long long o) const {
    long long w = o - wbase;
    return (w >= 0 && w < wlen) ? win[w] : g[o];
  }
};

// randSphere (misc.cc:95-109) rejects the pair (u1, u2) while
// r1^2 + r2^2 > 1 with r = 1 - 2 u / M, M = 2^32 - 1. In exact arithmetic
// that is (M - 2 u1)^2 + (M - 2 u2)^2 > M^2, decided here in 64-bit integers.
// The reference decides it in FP64, whose rounding can only matter within a
// few ulps of the unit circle; there (|difference| < 2^26 of M^2 ~ 1.8e19)
// the reference's own FP64 expression decides.
__device__ __forceinline__ bool sphere_reject(uint32_t u1, uint32_t u2) {
  const long long M = 4294967295LL;
  long long a = M - 2LL * (long long)u1, b = M - 2LL * (long long)u2;
  unsigned long long a2 = (unsigned long long)(a < 0 ? -a : a);
  unsigned long long b2 = (unsigned long long)(b < 0 ? -b : b);
  a2 *= a2;
  b2 *= b2;
  const unsigned long long M2 = 18446744065119617025ull;  // (2^32 - 1)^2
  const unsigned long long rhs = M2 - b2;
  const unsigned long long diff = a2 > rhs ? a2 - rhs : rhs - a2;
  if (diff > (1ull << 26)) return a2 > rhs;
  double r1 = 1.0 - 2.0 * unit_draw(u1);
  double r2 = 1.0 - 2.0 * unit_draw(u2);
  return r1 * r1 + r2 * r2 > 1.0;
}

// Consumes randSphere's draws; returns the stream index of the accepted pair.
__device__ __forceinline__ long long sphere_scan(Draws& d) {
  for (int guard = 0; guard < (1 << 20); guard++) {
    long long o = d.pos;
    uint32_t u1 = d.next(), u2 = d.next();
    if (d.overrun) return -1;
    if (!sphere_reject(u1, u2)) return o;
  }
  d.overrun = 1;
  return -1;
}

// Same, using accept bits precomputed by the block for every window
// position p: bit p set when the pair (p, p+1) is accepted. A pair starting at
// `pos` is followed by the pair at pos+2, so thread 0 looks for the next set
// bit of pos's parity; past the window it falls back to sphere_scan.
__device__ __forceinline__ long long sphere_scan_bits(Draws& d, const unsigned* accbits) {
  const long long rel0 = d.pos - d.wbase;
  if (rel0 < 0) return sphere_scan(d);
  long long rel = rel0;
  while (rel + 1 < d.wlen) {
    const int w = (int)(rel >> 5), b = (int)(rel & 31);
    const unsigned par = (rel & 1) ? 0xAAAAAAAAu : 0x55555555u;
    const unsigned msk = accbits[w] & par & (0xFFFFFFFFu << b);
    if (msk) {
      const long long p = ((long long)w << 5) + (__ffs(msk) - 1);
      d.pos = d.wbase + p + 2;
      return d.wbase + p;
    }
    rel = ((long long)(w + 1) << 5) + (rel0 & 1);
  }
  // every pair of this parity inside the window was rejected: continue from
  // the first pair not covered by the bits
  if (rel0 + 1 < d.wlen) d.pos = d.wbase + rel0 + 2 * ((d.wlen - rel0) / 2);
  return sphere_scan(d);
}

// The unit vector randSphere returns for an accepted pair.
__device__ __forceinline__ void sphere_vec(uint32_t u1, uint32_t u2, double* v) {
  double r1 = 1.0 - 2.0 * unit_draw(u1);
  double r2 = 1.0 - 2.0 * unit_draw(u2);
  double rs = r1 * r1 + r2 * r2;
  double ranh = 2.0 * sqrt(1.0 - rs);
  v[0] = r1 * ranh;
  v[1] = r2 * ranh;
  v[2] = (1.0 - 2.0 * rs);
}

__device__ __forceinline__ void rand_sphere(Draws& d, double* v, const unsigned* accbits) {
  long long o = sphere_scan_bits(d, accbits);
  if (o < 0) {
    v[0] = v[1] = 0.0;
    v[2] = 1.0;
    return;
  }
  sphere_vec(d.at(o), d.at(o + 1), v);
}

// Three block sums of values that only the first n threads hold (the others zero):
// value q ends in thread q, q < 3. Lanes are added pairwise, then the warps in
// order, by one thread per value: on this chip's FP64 pipe (16 cycles an
// instruction, 64 until its result) eight warps adding all three for every thread
// took 5,000 cycles. sh: 3 NT / 32 doubles.
template <int NT>
__device__ __forceinline__ double bsum3(double a, double b, double c, int n, double* sh) {
  constexpr int W = NT / 32;
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  double v[3] = {a, b, c};
  if (32 * w < n) {
    const int left = n - 32 * w;  // lanes with a value, when under a warp
#pragma unroll
    for (int q = 0; q < 3; q++) {
      const bool any = __any_sync(0xffffffffu, __double_as_longlong(v[q]) << 1 != 0);
      if (any)
        for (int o = 16; o > 0; o >>= 1)
          if (o < left) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    }
  }
  __syncthreads();
  if (l == 0)
#pragma unroll
    for (int q = 0; q < 3; q++) sh[q * W + w] = v[q];
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 3)
    for (int i = 0; i < W && 32 * i < n; i++) t += sh[threadIdx.x * W + i];
  return t;
}

struct GenPlan {
  int type;      // move type, -1 none
  int mol, b0, b1, b_lo, b_hi;
  double vec[3];  // COM shift / reptation end step
  double R[9];    // crankshaft rotation
  int first;      // crankshaft first bead (molecule-relative)
  int dir;        // reptation direction
  int end;        // reptation end bead (molecule-relative)
  double s;       // pivot displacement size
  int pivot;      // pivot bead (molecule-relative); -1: generated sequentially
  int scan;       // pivot: the block locates the beads' draws (pivot_draws)
  int scan_rel;   // window offset of the first bead's draws
  int scan_ok;    // every bead's draws lay inside the window
  int scan_end;   // window offset after the last bead's draws
};

constexpr int kPivotMax = 512;  // chains up to this length pivot in parallel
constexpr int kJumpLevels = 9;  // 2^9 >= kPivotMax - 1 beads per pivot

// First window position q >= x of x's parity whose pair (q, q+1) randSphere
// accepts, kDrawWindow if there is none: the bit scan sphere_scan_bits makes
// from window offset x, without consuming anything.
__device__ __forceinline__ int next_accept(const unsigned* accbits, int wlen, int x) {
  if (x + 1 >= wlen) return kDrawWindow;
  const unsigned par = (x & 1) ? 0xAAAAAAAAu : 0x55555555u;
  int w = x >> 5;
  unsigned m = accbits[w] & par & (0xFFFFFFFFu << (x & 31));
  while (!m) {
    if (++w >= (wlen + 31) / 32) return kDrawWindow;
    m = accbits[w] & par;
  }
  return (w << 5) + (__ffs(m) - 1);
}

// Molecule::Pivot's draws for every bead at once. Bead k of the scan order
// (forward from the pivot, then backward) takes randSphere's accepted pair at
// p_k and, with the bond potential on, one bond-length draw at p_k + 2, so
// p_{k+1} = next_accept(p_k + step) with step 2 or 3: thread 0's sequential
// scan is the chain p_0 = next_accept(rel0), p_k = F^k(p_0). The block tabulates
// F^(2^l) for every window offset (pointer doubling) and each thread composes
// the jumps of its bead's rank. Offsets, and therefore results, are those of
// the sequential scan; plan.scan_ok is cleared when any bead's draws run past
// the window, and thread 0 then makes the sequential scan instead.
__device__ __forceinline__ void pivot_draws(const DevParams& P, int wlen, GenPlan& plan,
                                            int* s_off, int* s_boff,
                                            short (*jump)[kDrawWindow + 1],
                                            const unsigned* accbits) {
  const int step = P.vary_bond ? 3 : 2;
  const int len = plan.b1 - plan.b0, pv = plan.pivot;
  const int n = len - 1, nf = len - 1 - pv;
  int nl = 0;
  while ((1 << nl) < n) nl++;  // ranks 0 .. n-1 need nl bits
  // offsets past lim count as outside the window: a bead takes 3.5 words on
  // average, so n beads stay below it (else the sequential scan)
  const int lim = min(kDrawWindow, plan.scan_rel + 6 * n + 64);
  const auto inside = [&](int p) { return p < lim ? p : kDrawWindow; };
  for (int x = plan.scan_rel + (int)threadIdx.x; x < lim; x += blockDim.x)
    jump[0][x] = (short)inside(next_accept(accbits, wlen, x + step));
  if ((int)threadIdx.x < nl) jump[threadIdx.x][kDrawWindow] = kDrawWindow;
  for (int l = 1; l < nl; l++) {
    __syncthreads();
    for (int x = plan.scan_rel + (int)threadIdx.x; x < lim; x += blockDim.x)
      jump[l][x] = jump[l - 1][jump[l - 1][x]];
  }
  if (threadIdx.x == 0) {
    plan.scan_ok = 1;
    plan.scan_end = plan.scan_rel;
  }
  __syncthreads();
  const int p0 = inside(next_accept(accbits, wlen, plan.scan_rel));
  for (int k = threadIdx.x; k < n; k += blockDim.x) {
    int p = p0;
    for (int l = 0; l < nl; l++)
      if ((k >> l) & 1) p = jump[l][p];
    const int i = k < nf ? pv + 1 + k : pv - 1 - (k - nf);
    if (p >= kDrawWindow || p + step > wlen) {
      plan.scan_ok = 0;  // every writer stores the same value
    } else {
      s_off[i] = p;
      s_boff[i] = p + 2;
    }
    if (k == n - 1) plan.scan_end = p + step;
  }
  __syncthreads();
}

// The positions a candidate starts from: the current ones, with the pending
// move's trial beads [lo, hi) in their place where it is taken as accepted.
struct PosView {
  const double4_32a* pos;
  const double4_32a* trial;
  int lo, hi;
  __device__ __forceinline__ double4_32a at(int i) const {
    return i >= lo && i < hi ? trial[i] : pos[i];
  }
};

// Thread 0, after the move's own draws: delayed acceptance's stage-one draw,
// the stream check and the stream position.
__device__ __forceinline__ void gen_tail(const DevState* st, const DevBuffers& B, Draws& d,
                                         GenPlan& plan, MoveCand& C) {
  // Delayed acceptance: a chain move (pivot, crankshaft, reptation) takes
  // its stage-one draw right after its own draws.
  C.u1 = 0.0;
  if (plan.type >= 2 && st->da_on && B.desc_acc && B.desc_fine) C.u1 = d.u();
  C.overrun = d.overrun;
  if (d.overrun) plan.type = -1;
  C.pos = d.pos;
}

// Thread 0's sequential pivot scan for chains up to kPivotMax beads: records
// each bead's draw offsets for the block.
__device__ __forceinline__ void pivot_draws_seq(const DevParams& P, Draws& d, long long wbase,
                                                int len, int pivot, int* s_off, int* s_boff,
                                                const unsigned* accbits) {
  for (int dirn = 0; dirn < 2; dirn++) {
    int i = dirn == 0 ? pivot + 1 : pivot - 1;
    for (; dirn == 0 ? i < len : i >= 0; i += dirn == 0 ? 1 : -1) {
      long long o = sphere_scan_bits(d, accbits);
      s_off[i] = (int)(o - wbase);
      if (P.vary_bond) {
        s_boff[i] = (int)(d.pos - wbase);
        (void)d.next();
      }
      if (d.overrun) break;
    }
  }
}

// Where a candidate's trial positions go ([max_len], from its b_lo on).
struct TrialOut {
  double4_32a* t;
  int4* f;
  ulonglong4_32a* u;
};

// The trial position of bead i, and its fixed-point mirror for the precision
// form's pair sweep.
__device__ __forceinline__ void put_trial(const DevParams& P, const DevBuffers& B, TrialOut O,
                                          int b_lo, int i, double4_32a t) {
  O.t[i - b_lo] = t;
  if (P.form) O.f[i - b_lo] = fix_point(P, t, B.type[i]);
  if (B.fpos64) O.u[i - b_lo] = fix64x4(P, t);
}

// Walls and sum q dz of the moved beads [b_lo, b_hi), and the bonds of their
// molecule [m0, m1) at the trial positions, into C.
template <class Trial>
__device__ __forceinline__ void move_sums(const DevParams& P, const DevBuffers& B, bool on, int m0,
                                          int m1, int b_lo, int b_hi, const PosView& V,
                                          const Trial& T, MoveCand& C, double* red) {
  if (threadIdx.x == 0) C.ext_bad = C.lost = 0;
  __syncthreads();
  double ext = 0.0, dmz = 0.0, bt = 0.0;
  if (on) {
    for (int i = b_lo + threadIdx.x; i < b_hi; i += blockDim.x) {
      double4_32a t = T(i), p = V.at(i);
      if (P.use_ext) {
        int ty = B.type[i];
        double en = wall64(P, t.z, ty);
        if (en >= kVeryLarge) C.ext_bad = 1;  // every writer stores the same value
        ext += en - wall64(P, p.z, ty);
      }
      if (!finite3(t)) C.lost = 1;
      dmz += t.w * (t.z - p.z);
    }
    if (P.use_bond && m1 - m0 > 1)
      for (int i = m0 + threadIdx.x; i < m1 - 1; i += blockDim.x) {
        double4_32a p = T(i), q = T(i + 1);
        double dx = p.x - q.x, dy = p.y - q.y, dz = p.z - q.z;
        double r = sqrt(dx * dx + dy * dy + dz * dz);
        bt += 0.5 * P.k_bond * (r - P.r0) * (r - P.r0);
      }
  }
  const double v = bsum3<kSerialThreads>(ext, dmz, bt, on ? max(b_hi - b_lo, m1 - m0) : 0, red);
  if (threadIdx.x == 0) C.ext = v;
  if (threadIdx.x == 1) C.dmz = v;
  if (threadIdx.x == 2) C.bond = v;
  __syncwarp();
}

// Worked out beside the picks by the other warps, from the draws' fixed places: a
// move's own draws start at the fifth word. *_end: window offset after the draws
// (0: they ran past the window, and warp 0 makes them one by one).
struct GenPre {
  double crank_s, crank_c;  // of the angle drawn by the seventh word
  double pivot_s;           // from the sixth
  double ion[3], com[3], rep[3];
  int ion_end, rep_end;
};

// The vector of the first pair randSphere accepts from window offset k on, a lane
// per pair: offset after the pair, or 0 where none of 32 lies in the window.
__device__ __forceinline__ int pre_sphere(const uint32_t* win, int wlen, int k, double* v) {
  const int p = k + 2 * (int)(threadIdx.x & 31);
  const unsigned ok =
      __ballot_sync(0xffffffffu, p + 1 < wlen && !sphere_reject(win[p], win[p + 1]));
  if (!ok) return 0;
  const int o = k + 2 * (__ffs(ok) - 1);
  sphere_vec(win[o], win[o + 1], v);
  return o + 2;
}

// floor(n x / M) of a draw x, M = 2^32 - 1, 0 <= n < 2^20: the reference's FP64
// product is exact and its quotient, at least 1 / M away from the next integer
// unless it is one, cannot round up to it; so the integer quotient, and no
// division (n x = a 2^32 + b = a M + (a + b)).
__device__ __forceinline__ int draw_floor(int n, uint32_t x) {
  const unsigned long long v = (unsigned long long)n * x;
  const unsigned long long a = v >> 32, r = a + (v & 0xFFFFFFFFull);
  return (int)(a + (r >= 0xFFFFFFFFull ? 1 : 0));
}

// floor(fl(fl(x / M) n)): the picks' product. Both roundings together move it by
// less than n 2^-52, under 1 / M for n < 2^20, so unless n x / M is a whole number
// the floor is the integer quotient's.
__device__ __forceinline__ int draw_pick(int n, uint32_t x) {
  const unsigned long long v = (unsigned long long)n * x;
  const unsigned long long a = v >> 32, r = a + (v & 0xFFFFFFFFull);
  if (n < 0 || n >= (1 << 20) || r == 0 || r == 0xFFFFFFFFull || r == 0x1FFFFFFFEull)
    return (int)floor(unit_draw(x) * n);
  return (int)(a + (r >= 0xFFFFFFFFull ? 1 : 0));
}

// What warp 0 finds before the acceptance bits are there.
struct GenPicks {
  int mt, mol, b0, b1;  // mol -1: nothing is moved
  double bond_old;      // the molecule's bond energy
  bool any;             // molecules to pick from: the picks' draws are taken
};

__device__ __forceinline__ GenPicks gen_picks(const DevParams& P, const DevBuffers& B, Draws& d) {
  GenPicks g{0, -1, 0, 0, 0.0, P.n_mol - P.phantom > 0};
  (void)d.next();  // simulation.cc:221 (the GC draw)
  if (!g.any) return g;
  const int n_ch = P.n_chain_total, n_io = P.n_ion_total;
  int wc = draw_pick(n_ch, d.next());
  int wi = draw_pick(n_io, d.next());
  if (wc == n_ch) wc--;
  if (wi == n_io) wi--;
  const int4 none = make_int4(-1, 0, 0, 0);
  const int4 chain = (wc >= 0 && wc < n_ch) ? B.chain_ids[wc] : none;
  const int4 ion = (wi >= 0 && wi < n_io) ? B.ion_ids[wi] : none;
  // the reference's running sum of the probabilities (move_cum) against the draw,
  // as bits: non-negative doubles order as integers
  const long long u = __double_as_longlong(unit_draw(d.next()));
  while (g.mt < 4 && P.move_cum[g.mt] < u) g.mt++;
  int4 m = none;
  if (g.mt == 0 && n_io > 0)
    m = ion;
  else if (g.mt > 0 && n_ch > 0)
    m = chain;
  g.mol = m.x;
  g.b0 = m.y;
  g.b1 = m.z;
  return g;
}

// Component `lane` (0, 1, else 2) of v.
__device__ __forceinline__ double pick3(const double* v, int lane) {
  return lane == 0 ? v[0] : (lane == 1 ? v[1] : v[2]);
}
// That component of the ion's displacement and of the reptation's end bond along
// randSphere's v.
__device__ __forceinline__ double ion_part(const DevParams& P, const double* v, int lane) {
  double vl = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  if (vl > 0) vl = 3 * P.move_size / vl;
  return vl * pick3(v, lane);
}
__device__ __forceinline__ double rep_part(double bl, const double* v, int lane) {
  const double vl = sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
  return bl * pick3(v, lane) / vl;
}

// Generates candidate C from stream position d.pos and positions V. Warp 0
// consumes the draws, every lane the same way but for the three components of a
// vector, which take a lane each (one division's latency instead of three); the
// block applies the geometry.
__device__ __forceinline__ void gen_move(const DevParams& P, const DevBuffers& B,
                                      const DevState* st, const PosView& V, TrialOut O,
                                      MoveCand& C, Draws& d, long long wbase, GenPlan& plan,
                                      int* s_off, int* s_boff, double (*s_w)[kPivotMax],
                                      short (*jump)[kDrawWindow + 1],
                                      const unsigned* accbits, double* red, const GenPicks& gp,
                                      const GenPre& pre) {
  // ----------------------------------------------------- generate next move
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const auto part = [&](const double* v) { return pick3(v, lane); };
    plan.type = -1;
    plan.scan = 0;
    if (gp.any) {
      const int mt = gp.mt, molid = gp.mol;
      if (molid >= 0) {
        const int b0 = gp.b0, b1 = gp.b1;
        const int len = b1 - b0;
        plan.mol = molid;
        plan.b0 = b0;
        plan.b1 = b1;
        plan.b_lo = b0;
        plan.b_hi = b1;
        plan.type = mt;
        if (mt == 0) {
          // Molecule::BeadTranslate (molecule.cc:103-133)
          double x;
          if (pre.ion_end) {
            x = part(pre.ion);
            d.pos = wbase + pre.ion_end;
          } else {
            double v[3];
            rand_sphere(d, v, accbits);
            x = ion_part(P, v, lane);
          }
          if (lane < 3) plan.vec[lane] = x;
          plan.b_hi = b0 + 1;
        } else if (mt == 1) {
          // Molecule::COMTranslate (molecule.cc:135-151). Here, and in the
          // pivot's displacement, the reference multiplies the word before
          // dividing, so these keep the division (unit_draw is the quotient of
          // the word alone).
          for (int a = 0; a < 6; a++) (void)d.next();
          if (lane < 3) plan.vec[lane] = pre.com[lane];
        } else if (mt == 2) {
          // Molecule::Pivot (molecule.cc:153-237). Bead i's new position is
          // the previous one plus bl_i * unit(old_i - old_prev + s v_i): the
          // reference's running translation of the chain tail cancels out of
          // the bond direction. Thread 0 only locates each bead's draws; the
          // geometry and the running sum are done by the block below.
          int pivot = draw_floor(len, d.next());
          if (pivot == len) pivot--;
          (void)d.next();
          const double s = pre.pivot_s;
          plan.s = s;
          plan.pivot = pivot;
          if (len <= kPivotMax) {
            // the block locates every bead's draws (pivot_draws)
            plan.scan = 1;
            plan.scan_rel = (int)(d.pos - wbase);
          } else {
            plan.pivot = -1;
            const double eq = P.bond_len;
            O.t[pivot] = V.at(b0 + pivot);
            for (int dirn = 0; dirn < 2; dirn++) {
              double T[3] = {0.0, 0.0, 0.0};
              double4_32a pv = V.at(b0 + pivot);
              double prev[3] = {pv.x, pv.y, pv.z};
              int i = dirn == 0 ? pivot + 1 : pivot - 1;
              for (; dirn == 0 ? i < len : i >= 0; i += dirn == 0 ? 1 : -1) {
                double v[3];
                rand_sphere(d, v, accbits);
                double4_32a o = V.at(b0 + i);
                double p[3] = {o.x + T[0], o.y + T[1], o.z + T[2]};
                double dx = (p[0] + s * v[0]) - prev[0];
                double dy = (p[1] + s * v[1]) - prev[1];
                double dz = (p[2] + s * v[2]) - prev[2];
                double bl = eq;
                if (P.vary_bond) bl += (eq / 5.0) * (unit_draw(d.next()) - 0.5);
                double norm = bl / sqrt(dx * dx + dy * dy + dz * dz);
                double c[3] = {norm * dx + prev[0], norm * dy + prev[1], norm * dz + prev[2]};
                for (int a = 0; a < 3; a++) {
                  T[a] += c[a] - p[a];
                  prev[a] = c[a];
                }
                O.t[i] = make_double4_32a(c[0], c[1], c[2], o.w);
                if (d.overrun) break;
              }
            }
          }
        } else if (mt == 3) {
          // Molecule::Crankshaft (molecule.cc:239-265); Rodrigues rotation in
          // the per-entry grouping of Eigen's AngleAxis::toRotationMatrix.
          int first = draw_floor(len - 2, d.next());
          int last = draw_floor(len - first, d.next()) + first;
          (void)d.next();  // the angle
          if (last > len - 1) last = len - 1;  // the reference reads past the chain here
          double4_32a pf = V.at(b0 + first), pl = V.at(b0 + last);
          double ax[3] = {pl.x - pf.x, pl.y - pf.y, pl.z - pf.z};
          double z2 = ax[0] * ax[0] + ax[1] * ax[1] + ax[2] * ax[2];
          if (z2 > 0) {
            double n = sqrt(z2);
            const double al = part(ax) / n;
            for (int a = 0; a < 3; a++) ax[a] = __shfl_sync(0xffffffffu, al, a);
          }
          const double sn = pre.crank_s, cs = pre.crank_c;
          double sa[3] = {sn * ax[0], sn * ax[1], sn * ax[2]};
          double ca[3] = {(1.0 - cs) * ax[0], (1.0 - cs) * ax[1], (1.0 - cs) * ax[2]};
          double t = ca[0] * ax[1];
          plan.R[1] = t - sa[2];
          plan.R[3] = t + sa[2];
          t = ca[0] * ax[2];
          plan.R[2] = t + sa[1];
          plan.R[6] = t - sa[1];
          t = ca[1] * ax[2];
          plan.R[5] = t - sa[0];
          plan.R[7] = t + sa[0];
          for (int a = 0; a < 3; a++) plan.R[4 * a] = ca[a] * ax[a] + cs;
          plan.first = first;
          plan.b_lo = b0 + first + 1;
          plan.b_hi = b0 + (last > first + 1 ? last : first + 1);
        } else {
          // Molecule::RandomReptation (molecule.cc:267-312)
          double bl = P.bond_len;
          if (P.vary_bond) bl += (P.bond_len / 5.0) * (unit_draw(d.next()) - 0.5);
          int dir = 1, end = len - 1;
          if (d.next() % 2u == 0u) {
            dir = -1;
            end = 0;
          }
          double x;
          if (pre.rep_end) {
            x = part(pre.rep);
            d.pos = wbase + pre.rep_end;
          } else {
            double v[3];
            rand_sphere(d, v, accbits);
            x = rep_part(bl, v, lane);
          }
          if (lane < 3) plan.vec[lane] = x;
          plan.dir = dir;
          plan.end = end;
        }
      }
    }
    if (!plan.scan) gen_tail(st, B, d, plan, C);
  }
  __syncthreads();
  if (plan.scan) {
    pivot_draws(P, d.wlen, plan, s_off, s_boff, jump, accbits);
    if (threadIdx.x == 0) {
      if (plan.scan_ok) {
        d.pos = wbase + plan.scan_end;
      } else {
        d.pos = wbase + plan.scan_rel;
        pivot_draws_seq(P, d, wbase, plan.b1 - plan.b0, plan.pivot, s_off, s_boff, accbits);
      }
      gen_tail(st, B, d, plan, C);
    }
    __syncthreads();
  }
  // Apply the plan in parallel (the sequential pivot of a long chain already
  // wrote its trial positions).
  const GenPlan g = plan;
  if (g.type == 0 || g.type == 1) {
    for (int i = g.b_lo + threadIdx.x; i < g.b_hi; i += blockDim.x) {
      double4_32a o = V.at(i);
      put_trial(P, B, O, g.b_lo, i,
                make_double4_32a(o.x + g.vec[0], o.y + g.vec[1], o.z + g.vec[2], o.w));
    }
  } else if (g.type == 3) {
    const double4_32a pf = V.at(g.b0 + g.first);
    for (int i = g.b_lo + threadIdx.x; i < g.b_hi; i += blockDim.x) {
      double4_32a o = V.at(i);
      double v[3] = {o.x - pf.x, o.y - pf.y, o.z - pf.z};
      double r[3];
      for (int a = 0; a < 3; a++)
        r[a] = ((g.R[3 * a] * v[0] + g.R[3 * a + 1] * v[1]) + g.R[3 * a + 2] * v[2]);
      put_trial(P, B, O, g.b_lo, i, make_double4_32a(r[0] + pf.x, r[1] + pf.y, r[2] + pf.z, o.w));
    }
  } else if (g.type == 2 && g.pivot >= 0) {
    const int len = g.b1 - g.b0, pv = g.pivot;
    const double eq = P.bond_len;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      if (i == pv) continue;
      const int j = i > pv ? i - 1 : i + 1;
      double v[3];
      sphere_vec(d.at(wbase + s_off[i]), d.at(wbase + s_off[i] + 1), v);
      double bl = eq;
      if (P.vary_bond) bl += (eq / 5.0) * (unit_draw(d.at(wbase + s_boff[i])) - 0.5);
      const double4_32a oi = V.at(g.b0 + i), oj = V.at(g.b0 + j);
      double dx = (oi.x - oj.x) + g.s * v[0];
      double dy = (oi.y - oj.y) + g.s * v[1];
      double dz = (oi.z - oj.z) + g.s * v[2];
      double norm = bl / sqrt(dx * dx + dy * dy + dz * dz);
      // scan slot: forward beads first (pivot+1 ..), then backward (pivot-1 ..)
      const int k = i > pv ? i - pv - 1 : (len - 1 - pv) + (pv - 1 - i);
      s_w[0][k] = norm * dx;
      s_w[1][k] = norm * dy;
      s_w[2][k] = norm * dz;
    }
    // Inclusive running sums within the two segments (Hillis-Steele).
    const int nf = len - 1 - pv, n = len - 1;
    for (int off = 1; off < n; off <<= 1) {
      __syncthreads();
      double add[3][2];
      for (int r = 0; r < 2; r++) {
        int k = threadIdx.x + r * blockDim.x;
        bool ok = k < n && (k < nf ? k - off >= 0 : k - off >= nf);
        for (int a = 0; a < 3; a++) add[a][r] = ok ? s_w[a][k - off] : 0.0;
      }
      __syncthreads();
      for (int r = 0; r < 2; r++) {
        int k = threadIdx.x + r * blockDim.x;
        if (k < n)
          for (int a = 0; a < 3; a++) s_w[a][k] += add[a][r];
      }
    }
    __syncthreads();
    const double4_32a pp = V.at(g.b0 + pv);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
      const int i = k < nf ? pv + 1 + k : pv - 1 - (k - nf);
      const double q = V.at(g.b0 + i).w;
      put_trial(P, B, O, g.b_lo, g.b0 + i,
                make_double4_32a(pp.x + s_w[0][k], pp.y + s_w[1][k], pp.z + s_w[2][k], q));
    }
    // the pivot bead stays where it is
    if (threadIdx.x == 0) put_trial(P, B, O, g.b_lo, g.b0 + pv, pp);
  } else if (g.type == 4) {
    const int len = g.b1 - g.b0;
    for (int i = threadIdx.x; i < len; i += blockDim.x) {
      double4_32a nw;
      if (i == g.end) {
        double4_32a o = V.at(g.b0 + i);
        nw = make_double4_32a(o.x + g.vec[0], o.y + g.vec[1], o.z + g.vec[2], o.w);
      } else {
        double4_32a o = V.at(g.b0 + i + g.dir);
        nw = make_double4_32a(o.x, o.y, o.z, V.at(g.b0 + i).w);
      }
      put_trial(P, B, O, g.b_lo, g.b0 + i, nw);
    }
  }
  __syncthreads();
  if (g.type == 2 && g.pivot < 0)
    // fixed-point trial coordinates of the sequential pivot
    for (int i = g.b_lo + threadIdx.x; i < g.b_hi; i += blockDim.x)
      put_trial(P, B, O, g.b_lo, i, O.t[i - g.b_lo]);
  move_sums(P, B, g.type >= 0, g.b0, g.b1, g.b_lo, g.b_hi, V,
            [&](int i) { return i >= g.b_lo && i < g.b_hi ? O.t[i - g.b_lo] : V.at(i); }, C, red);
  if (threadIdx.x == 0) {
    C.type = g.type;
    if (g.type >= 0) {
      C.mol = g.mol;
      C.b_lo = g.b_lo;
      C.b_hi = g.b_hi;
      C.bonded = g.b1 - g.b0 > 1;
      C.bond_old = gp.bond_old;
    }
  }
}

// Shared memory of one candidate's generation.
struct GenSmem {
  uint32_t win[kDrawWindow];
  unsigned accbits[kDrawWindow / 32];  // randSphere acceptance per position
  double red[3 * (kSerialThreads / 32)];
  GenPlan plan;
  int s_off[kPivotMax], s_boff[kPivotMax];  // draw offsets per bead
  union {
    short jump[kJumpLevels][kDrawWindow + 1];  // pivot draws: 2^l beads on
    double s_w[3][kPivotMax];                  // pivot bond steps (used after)
  };
  MoveCand C;
  GenPre pre;
};

// Candidate c of the step after the pending move.
__device__ __forceinline__ void gen_body(const DevParams& P, const DevBuffers& B, int c,
                                         GenSmem& sm) {
  const DevState* st = B.state;
  const int pending = st->pending;
  if (st->error || (!pending && c != kCandSkip)) return;
  const long long base = st->stream_pos + (c == kCandSkip ? 0 : 1), len = st->stream_len;
  const long long avail = len - base;
  // the words a move of the longest molecule takes (see pivot_draws), within the
  // window; moves that take more make their draws one by one
  const int most = min(kDrawWindow, (6 * P.max_len + 80 + 63) & ~31);
  const int wlen = (int)(avail < most ? (avail > 0 ? avail : 0) : most);
  for (int i = threadIdx.x; i < wlen; i += blockDim.x) sm.win[i] = B.stream[base + i];
  __syncthreads();
  Draws d{B.stream, sm.win, base, len, base, wlen, 0};
  GenPicks gp{0, -1, 0, 0, 0.0, false};
  const int warp = threadIdx.x >> 5;
  if (warp == 0) {
    gp = gen_picks(P, B, d);
    if (gp.mol >= 0 && P.use_bond)
      gp.bond_old =
          c == kCandAccept && gp.mol == st->mol ? B.plan->now.bond : B.bond_mol[gp.mol];
  }
  if (warp == 1 && base + 6 < len) {
    const double pi_libm = 3.14159265358979323846;
    const double ang = P.move_size * (unit_draw(d.at(base + 6)) * 2 * pi_libm - pi_libm);
    sincos(ang, &sm.pre.crank_s, &sm.pre.crank_c);
  }
  const int lane = threadIdx.x & 31;
  if (warp == 2 && base + 5 < len)
    sm.pre.pivot_s = P.move_size * (double)d.at(base + 5) / kMtMax;
  if (warp == 3) {
    double v[3] = {0.0, 0.0, 1.0};
    const int end = pre_sphere(sm.win, wlen, 4, v);
    const double x = ion_part(P, v, lane);
    if (lane < 3) sm.pre.ion[lane] = x;
    if (lane == 0) sm.pre.ion_end = end;
  }
  if (warp == 4) {
    const int k = P.vary_bond ? 5 : 4;  // the direction's word
    double v[3] = {0.0, 0.0, 1.0}, bl = P.bond_len;
    if (P.vary_bond && wlen > 4) bl += (P.bond_len / 5.0) * (unit_draw(sm.win[4]) - 0.5);
    const int end = pre_sphere(sm.win, wlen, k + 1, v);
    const double x = rep_part(bl, v, lane);
    if (lane < 3) sm.pre.rep[lane] = x;
    if (lane == 0) sm.pre.rep_end = end;
  }
  if (warp == 5 && lane < 3 && base + 9 < len) {
    const double x = 0.5 * P.move_size * (double)d.at(base + 4 + lane) / kMtMax;
    sm.pre.com[lane] = d.at(base + 7 + lane) % 2u == 0u ? -x : x;
  }
  // every window position's randSphere test, one position per thread; a
  // warp's ballot makes the word of its 32 positions
  for (int p0 = threadIdx.x & ~31; p0 < most; p0 += blockDim.x) {
    const int p = p0 + (threadIdx.x & 31);
    const bool ok = p + 1 < wlen && !sphere_reject(sm.win[p], sm.win[p + 1]);
    const unsigned bits = __ballot_sync(0xFFFFFFFFu, ok);
    if ((threadIdx.x & 31) == 0) sm.accbits[p0 >> 5] = bits;
  }
  __syncthreads();
  const bool took = c == kCandAccept;
  const PosView V{B.pos, B.trial, took ? st->b_lo : 0, took ? st->b_hi : 0};
  const size_t at = (size_t)c * P.max_len;
  const TrialOut O{B.ctrial + at, B.cftrial + at, B.ctrial64 + at};
  gen_move(P, B, st, V, O, sm.C, d, base, sm.plan, sm.s_off, sm.s_boff, sm.s_w, sm.jump, sm.accbits,
           sm.red, gp, sm.pre);
  if (threadIdx.x == 0) B.plan->cand[c] = sm.C;
}

// Shared memory of one serial step.
struct SerialSmem {
  double red[3 + 3 * (kSerialThreads / 32)];  // block sums, then bsum3's
  int s_accept, s_cand;
  StepPlan plan;
  // The state lives in shared memory for the step: thread 0's chain of
  // decisions then never waits on global memory for it.
  DevState S;
};

// Batched replicas: the pending move's sums are per-item slots of the batch
// delta kernel, added here in item order.
struct SlotSums {
  const double* slots;  // [items][2]
  int pair_off, n_pair, k_off, n_k;
};

// The FP64 energy change's block sums {LJ, real space, k, unused} by one warp,
// lane l taking blocks l, l + 32, ...; a lane's loads are all in flight at once
// (a loop of load and add took 2.4 us for 149 blocks).
__device__ __forceinline__ void block_sums(const double* part, int blocks, double* sum) {
  const int lane = threadIdx.x & 31;
  const double4_32a* p = reinterpret_cast<const double4_32a*>(part);
  double a = 0.0, b = 0.0, c = 0.0;
  for (int i0 = 0; i0 < blocks; i0 += 256) {
    double4_32a v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const int i = i0 + lane + 32 * u;
      v[u] = i < blocks ? p[i] : make_double4_32a(0.0, 0.0, 0.0, 0.0);
    }
#pragma unroll
    for (int h = 4; h > 0; h >>= 1)
      for (int u = 0; u < h; u++) {
        v[u].x += v[u + h].x;
        v[u].y += v[u + h].y;
        v[u].z += v[u + h].z;
      }
    a += v[0].x;
    b += v[0].y;
    c += v[0].z;
  }
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
  }
  if (lane == 0) {
    sum[0] = a;
    sum[1] = b;
    sum[2] = c;
  }
}

__device__ __forceinline__ void serial_body(const DevParams& P, const DevBuffers& B, int mode,
                                            SerialSmem& sm, const SlotSums* slots,
                                            int part_blocks) {
  double* const red = sm.red;
  int& s_accept = sm.s_accept;
  DevState& S = sm.S;
  // (beside the state's load; with no pending move nobody reads them)
  if (part_blocks && (mode & kModeFinish) && (threadIdx.x >> 5) == 7)
    block_sums(B.partial, part_blocks, red);
  {
    const int nw = (int)(sizeof(DevState) / sizeof(int));
    const int* src = reinterpret_cast<const int*>(B.state);
    int* dst = reinterpret_cast<int*>(&S);
    for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = src[i];
    const int np = (int)(sizeof(StepPlan) / sizeof(int));
    src = reinterpret_cast<const int*>(B.plan);
    dst = reinterpret_cast<int*>(&sm.plan);
    for (int i = threadIdx.x; i < np; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  if (S.error) return;
  if (slots && (mode & kModeFinish) && S.pending) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int i = threadIdx.x; i < slots->n_pair; i += blockDim.x) {
      a += slots->slots[2 * (slots->pair_off + i)];
      b += slots->slots[2 * (slots->pair_off + i) + 1];
    }
    for (int i = threadIdx.x; i < slots->n_k; i += blockDim.x)
      c += slots->slots[2 * (slots->k_off + i)];
    const double v = bsum3<kSerialThreads>(a, b, c, max(slots->n_pair, slots->n_k), red + 3);
    if (threadIdx.x == 0) S.red_lj = v;
    if (threadIdx.x == 1) S.red_re = v;
    if (threadIdx.x == 2) S.red_k = v;
    __syncthreads();
  }

  if (part_blocks && (mode & kModeFinish) && threadIdx.x == 0) {
    S.red_lj = red[0];
    S.red_re = red[1];
    S.red_k = red[2];
  }

  // the acceptance test's draw, loaded while dE is composed
  uint32_t word = 0;
  const int have = (mode & kModeDecide) && S.stream_pos < S.stream_len ? 1 : 0;
  if (have && threadIdx.x == 0) word = B.stream[S.stream_pos];
  Draws d{B.stream, &word, S.stream_pos, S.stream_len, S.stream_pos, have, 0};

  const int pending = S.pending;
  const int b_lo = S.b_lo, b_hi = S.b_hi, mol = S.mol;

  if ((mode & kModeFinish) && pending && S.da_skip) {
    // Stage one rejected the move: no exact change was computed. The S(k) change
    // of the last accepted move, if still pending, stays so until the next energy
    // change applies it (7,812 vectors added by this one block took 10 us).
    if (threadIdx.x == 0) S.de = 0.0;
    __syncthreads();
  } else if ((mode & kModeFinish) && pending) {
    // a move set by the host has no candidate's sums
    MoveCand& now = sm.plan.now;
    if (S.move_type < 0) {
      const int m0 = B.mol_start[mol], m1 = B.mol_start[mol + 1];
      move_sums(P, B, true, m0, m1, b_lo, b_hi, PosView{B.pos, B.trial, 0, 0},
                [&](int i) { return B.trial[i]; }, now, red + 3);
      if (threadIdx.x == 0) {
        now.bonded = m1 - m0 > 1;
        now.bond_old = B.bond_mol[mol];
      }
    }
    if (threadIdx.x == 0) {
      const double ext = now.ext, dmz = now.dmz, bt = now.bond;
      const int ext_bad = now.ext_bad;
      // the delta kernel applied any pending S(k) commit if it ran k units
      if (P.use_ewald && b_hi > b_lo) S.sk_pending = 0;
      const double de_lj = S.red_lj, de_re = S.red_re, de_k = b_hi > b_lo ? S.red_k : 0.0;
      double de = 0.0, dp = 0.0, dx = 0.0, dw = 0.0, db = 0.0;
      double dip_t = S.dipl_cur;
      bool done = false;
      if (P.use_pair) {
        dp = de_lj;
        de += dp;
        done = de >= kVeryLarge;
      }
      if (!done && P.use_ext) {
        dx = ext_bad ? kVeryLarge : ext;
        de += dx;
        done = de >= kVeryLarge;
      }
      if (!done && P.use_ewald) {
        dw = de_re + P.kpref * de_k;
        // (fixed-point pairs and phases have no NaN)
        if (now.lost) dw = __longlong_as_double(0x7FF8000000000000ll);
        if (P.dipole) {
          dip_t = P.dip_coef * S.mz * S.mz;
          dw += dip_t - S.dipl_cur;
        }
        de += dw;
      }
      if (!done && P.use_bond && now.bonded) {
        db = bt - now.bond_old;
        de += db;
      }
      if (!isfinite(de)) S.n_nonfinite++;  // flagged, rejected as the reference does
      S.de = de;
      S.de_pair = dp;
      S.de_ext = dx;
      S.de_ewald = dw;
      S.de_bond = db;
      S.bond_trial = bt;
      S.dipl_trial = dip_t;
      S.dmz = dmz;
    }
    __syncthreads();
    // training log: (descriptor, exact dE) of a surrogate move
    if (S.da_active && B.log_desc && S.log_n < S.log_cap) {
      const long long row = S.log_n;  // rows of mlp::kIn values
      for (int k = threadIdx.x; k < mlp::kIn; k += blockDim.x)
        B.log_desc[row * mlp::kIn + k] = (float)B.desc_acc[k] * mlp::kDescUnit;
      if (threadIdx.x == 0) {
        B.log_de[row] = S.de;
        S.log_n++;
      }
      __syncthreads();
    }
  }

  // Metropolis (simulation.cc:324-332) or the host's decision.
  if ((mode & (kModeDecide | kModeCommit)) && pending) {
    if (threadIdx.x == 0) {
      int acc = 0;
      const long long at = d.pos;
      if (mode & kModeDecide) {
        if (S.da_active && S.da_on) {
          // Delayed acceptance, stage two: with the stage-one probability
          // min(1, exp(-beta s)) and s antisymmetric under reversing the
          // move, min(1, exp(-beta (dE - s))) gives the same ratio
          // exp(-beta dE) of forward to reverse acceptance as Metropolis.
          if (!S.da_skip && !(S.de >= kVeryLarge))
            acc = metropolis(d.u(), P.beta * (S.de - S.da_s));
          S.da_n_moves++;
          S.da_n_pass += S.da_skip ? 0 : 1;
          S.da_n_accept += acc;
        } else if (!(S.de >= kVeryLarge)) {
          acc = metropolis(d.u(), P.beta * S.de);  // a NaN dE still draws
        }
        if (d.overrun) S.error = PLUM_ERR_STREAM_DEV;
      } else {
        acc = mode & kModeAccept ? 1 : 0;
      }
      s_accept = acc;
      sm.s_cand = acc ? kCandAccept : (d.pos != at ? kCandReject : kCandSkip);
    }
    __syncthreads();
    const int acc = s_accept;
    if (acc) {
      for (int i = b_lo + threadIdx.x; i < b_hi; i += blockDim.x) {
        const int4 old_f = P.form ? B.fpos[i] : make_int4(0, 0, 0, 0);
        B.pos[i] = B.trial[i];
        if (B.fpos64) B.fpos64[i] = B.ftrial64[i - b_lo];
        if (P.form) B.fpos[i] = B.ftrial[i - b_lo];
        // (lists that were never built, or have overflowed, hold nothing to follow:
        // their keys may be anything)
        if (P.cell_cap && B.cell_key && S.cell_ok) {
          // the bead's entry follows it: rewritten in place while it stays in
          // its cell (or already is in the extra list), else marked dead and
          // the bead appended to the extra list
          const int4 f = B.ftrial[i - b_lo];
          const int4 ent = make_int4(f.x, f.y, f.z, (i << 3) | f.w);
          const int key = B.cell_key[i];
          if (key >= 0 && cell_index(P, old_f) == cell_index(P, f)) {
            B.cell_ent[key] = ent;
          } else if (key <= -2) {
            B.cell_extra[-2 - key] = ent;
          } else {
            if (key >= 0) B.cell_ent[key] = make_int4(0, 0, 0, -1);
            const int nc = P.cell_nc[0] * P.cell_nc[1] * P.cell_nc[2];
            const int e = atomicAdd(&B.cell_n[nc], 1);
            if (e < P.cell_cap) {
              B.cell_extra[e] = ent;
              B.cell_key[i] = -2 - e;
            } else {
              B.cell_key[i] = -1;
              S.cell_ok = 0;  // every writer stores the same value
            }
          }
        }
      }
    } else {
      for (int i = b_lo + threadIdx.x; i < b_hi; i += blockDim.x) B.trial[i] = B.pos[i];
    }
    if (threadIdx.x == 0) {
      if (acc) {
        S.e_pair += S.de_pair;
        S.e_ext += S.de_ext;
        S.e_ewald += S.de_ewald;
        S.e_bond += S.de_bond;
        S.mz += S.dmz;
        if (P.dipole) S.dipl_cur = S.dipl_trial;
        if (P.use_bond && B.mol_start[mol + 1] - B.mol_start[mol] > 1)
          B.bond_mol[mol] = S.bond_trial;
        if (P.use_ewald && b_hi > b_lo) {
          // the next delta kernel adds dsk[cur_buf] into S(k)
          S.sk_pending = 1;
          S.sk_buf = S.cur_buf;
          S.cur_buf ^= 1;
        }
        S.n_accept++;
      }
      S.last_accept = acc;
      S.pending = 0;
    }
  }
  // Per-step log (also for steps where nothing was attempted).
  if ((mode & kModeDecide) && S.step_open && threadIdx.x == 0) {
    int sidx = S.step;
    if (B.log_type) B.log_type[sidx] = pending ? S.move_type : -1;
    if (B.log_accept) B.log_accept[sidx] = pending ? S.last_accept : 0;
    if (B.log_etot) B.log_etot[sidx] = S.e_pair + S.e_ewald + S.e_bond + S.e_ext;
    if (B.log_step_de) B.log_step_de[sidx] = pending ? S.de : __longlong_as_double(0x7ff8000000000000LL);
    S.step = sidx + 1;
    S.step_open = 0;
  }
  __syncthreads();

  if ((mode & kModeGen) && !S.error) {
    const int c = pending ? sm.s_cand : kCandSkip;
    const MoveCand& C = sm.plan.cand[c];
    const double4_32a* t = B.ctrial + (size_t)c * P.max_len;
    const int4* f = B.cftrial + (size_t)c * P.max_len;
    if (C.type >= 0)
      for (int i = threadIdx.x; i < C.b_hi - C.b_lo; i += blockDim.x) {
        B.trial[C.b_lo + i] = t[i];
        if (P.form) B.ftrial[i] = f[i];
        if (B.fpos64) B.ftrial64[i] = B.ctrial64[(size_t)c * P.max_len + i];
      }
    // surrogate move: its descriptor is accumulated from zero by the next launch
    const bool surr = C.type >= 2 && B.desc_acc && B.desc_fine && (S.da_on || B.log_desc);
    if (surr)
      for (int k = threadIdx.x; k < mlp::kFineAll; k += blockDim.x) B.desc_fine[k] = 0u;
    if (threadIdx.x == 0) {
      S.step_open = 1;
      S.stream_pos = C.pos;
      if (C.overrun) S.error = PLUM_ERR_STREAM_DEV;
      S.da_active = surr ? 1 : 0;
      S.da_skip = 0;
      if (surr && S.da_on) S.da_u1 = C.u1;
      if (C.type >= 0) {
        S.pending = 1;
        S.mol = C.mol;
        S.b_lo = C.b_lo;
        S.b_hi = C.b_hi;
        S.move_type = C.type;
        B.plan->now = C;
      } else {
        S.pending = 0;
      }
    }
  }

  if (mode == kModeFinish && B.host_out && threadIdx.x == 0) {
    B.host_out[0] = S.de;
    B.host_out[1] = S.de_pair;
    B.host_out[2] = S.de_ewald;
    B.host_out[3] = S.de_bond;
    B.host_out[4] = S.de_ext;
    B.host_out[5] = (double)S.error;
  }
  // write the state back
  if (threadIdx.x == 0 && S.stream_pos < d.pos) S.stream_pos = d.pos;
  __syncthreads();
  {
    const int nw = (int)(sizeof(DevState) / sizeof(int));
    int* dst = reinterpret_cast<int*>(B.state);
    const int* src = reinterpret_cast<const int*>(&S);
    for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = src[i];
  }
}

__global__ void __launch_bounds__(kSerialThreads)
    k_serial64(const DevParams P, const DevBuffers B, int mode, int part_blocks) {
  __shared__ SerialSmem sm;
  serial_body(P, B, mode, sm, nullptr, part_blocks);
}

// A replica's parameters and buffers into shared memory.
__device__ __forceinline__ void stage_system(const DevParams* rp, const DevBuffers* rb,
                                             DevParams& P, DevBuffers& B) {
  const int* src = reinterpret_cast<const int*>(rp);
  int* dst = reinterpret_cast<int*>(&P);
  for (int i = threadIdx.x; i < (int)(sizeof(DevParams) / sizeof(int)); i += blockDim.x)
    dst[i] = src[i];
  const long long* bs = reinterpret_cast<const long long*>(rb);
  long long* bd = reinterpret_cast<long long*>(&B);
  for (int i = threadIdx.x; i < (int)(sizeof(DevBuffers) / sizeof(long long)); i += blockDim.x)
    bd[i] = bs[i];
  __syncthreads();
}

// One block per replica: the replica's parameters and buffers are staged in
// shared memory, then the same serial step runs on them.
__global__ void __launch_bounds__(kSerialThreads)
    k_batch_serial(const DevParams* __restrict__ rp, const DevBuffers* __restrict__ rb,
                   const int* __restrict__ item_off, const double* __restrict__ slots, int mode) {
  __shared__ SerialSmem sm;
  __shared__ DevParams P;
  __shared__ DevBuffers B;
  const int r = blockIdx.x;
  stage_system(rp + r, rb + r, P, B);
  SlotSums ss{slots, item_off[4 * r], item_off[4 * r + 1], item_off[4 * r + 2],
              item_off[4 * r + 3]};
  serial_body(P, B, mode, sm, &ss, 0);
}

__global__ void __launch_bounds__(kSerialThreads)
    k_gen(const DevParams P, const DevBuffers B, int c0) {
  __shared__ GenSmem sm;
  gen_body(P, B, c0 + (int)blockIdx.x, sm);
}

__global__ void __launch_bounds__(kSerialThreads)
    k_batch_gen(const DevParams* __restrict__ rp, const DevBuffers* __restrict__ rb, int c0) {
  __shared__ GenSmem sm;
  __shared__ DevParams P;
  __shared__ DevBuffers B;
  stage_system(rp + blockIdx.x, rb + blockIdx.x, P, B);
  gen_body(P, B, c0 + (int)blockIdx.y, sm);
}

void launch_gen64(const DevParams& P, const DevBuffers& B, bool first, cudaStream_t s) {
  k_gen<<<first ? 1 : kCands, kSerialThreads, 0, s>>>(P, B, first ? kCandSkip : 0);
}

void launch_batch_gen(const DevParams* rp, const DevBuffers* rb, int n_rep, bool first,
                      cudaStream_t s) {
  k_batch_gen<<<dim3(n_rep, first ? 1 : kCands), kSerialThreads, 0, s>>>(rp, rb,
                                                                        first ? kCandSkip : 0);
}

void launch_batch_serial(const DevParams* rp, const DevBuffers* rb, const int* item_off,
                         const double* slots, int n_rep, int mode, cudaStream_t s) {
  k_batch_serial<<<n_rep, kSerialThreads, 0, s>>>(rp, rb, item_off, slots, mode);
}

void launch_serial64(const DevParams& P, const DevBuffers& B, int mode, cudaStream_t s) {
  k_serial64<<<1, kSerialThreads, 0, s>>>(P, B, mode, delta_blocks());
}

// span: the trial positions of [b_lo, b_hi) in pinned host memory, read from there
// (no copy of their own ahead of the kernel).
__global__ void k_set_move(const DevParams P, const DevBuffers B, int mol, int b_lo, int b_hi,
                           const double4_32a* __restrict__ span) {
  if (threadIdx.x == 0) {
    DevState* st = B.state;
    st->pending = 1;
    st->mol = mol;
    st->b_lo = b_lo;
    st->b_hi = b_hi;
    st->move_type = -1;
  }
  for (int i = threadIdx.x; i < b_hi - b_lo; i += blockDim.x) {
    const double4_32a p = span[i];
    B.trial[b_lo + i] = p;
    if (B.fpos64) B.ftrial64[i] = fix64x4(P, p);
    if (P.form) B.ftrial[i] = fix_point(P, p, B.type[b_lo + i]);
  }
}

void launch_set_move(const DevParams& P, const DevBuffers& B, int mol, int b_lo, int b_hi,
                     const double4_32a* span, cudaStream_t s) {
  k_set_move<<<1, 128, 0, s>>>(P, B, mol, b_lo, b_hi, span);
}

// ------------------------------------------------------------ mt19937 fill
// One block; state[624] holds the output index as in std::mt19937.
__device__ __forceinline__ uint32_t mt_twist(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t y = (a & 0x80000000u) | (b & 0x7fffffffu);
  uint32_t v = c ^ (y >> 1);
  if (y & 1u) v ^= 0x9908b0dfu;
  return v;
}

// Word x[g] of the sequence needs x[g - 624], x[g - 623] and x[g - 227], so 227 words
// are made at a time, one per thread with one barrier, in a ring of the last 1,024;
// the generator's state is the block of 624 words that holds the last one taken.
// (Block by block, in three phases with eight barriers, it took 1.3 ns a word and, with
// 4 M words at a time, 5.5 ms of a new state's first call.)
constexpr int kMtThreads = 256, kMtLag = 227, kMtRing = 1024;

// (without out, n words are skipped)
__device__ __forceinline__ void mt_fill_body(uint32_t* state, uint32_t* out, long long n) {
  __shared__ uint32_t x[kMtRing];
  if (n <= 0) return;
  const long long idx = state[624];
  const int t = threadIdx.x;
  auto emit = [&](long long g, uint32_t y) {  // word g, tempered, if it is asked for
    if (!out || g < idx || g >= idx + n) return;
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    out[g - idx] = y;
  };
  for (int i = t; i < 624; i += blockDim.x) {
    x[i] = state[i];
    emit(i, x[i]);
  }
  const long long block = (idx + n - 1) / 624, end = 624 * (block + 1);
  __syncthreads();
  for (long long g0 = 624; g0 < end; g0 += kMtLag) {
    const long long g = g0 + t;
    if (t < kMtLag && g < end) {
      const uint32_t v = mt_twist(x[(g - 624) & (kMtRing - 1)],
                                  x[(g - 623) & (kMtRing - 1)],
                                  x[(g - kMtLag) & (kMtRing - 1)]);
      x[g & (kMtRing - 1)] = v;
      emit(g, v);
    }
    __syncthreads();
  }
  for (int i = t; i < 624; i += blockDim.x) state[i] = x[(624 * block + i) & (kMtRing - 1)];
  if (t == 0) state[624] = (uint32_t)(idx + n - 624 * block);
}

__global__ void __launch_bounds__(kMtThreads) k_mt_fill(uint32_t* state, uint32_t* out,
                                                        long long n) {
  mt_fill_body(state, out, n);
}

__global__ void __launch_bounds__(kMtThreads)
    k_mt_fill_batch(uint32_t* const* states, uint32_t* const* outs, const long long* pos,
                    const long long* len, const long long* cap, const int* need,
                    DevState* const* sts) {
  const int r = blockIdx.x;
  if (!need[r]) return;
  uint32_t* out = outs[r];
  const long long p = pos[r], l = len[r];
  const long long tail = l > p ? l - p : 0;
  // move the unread words to the front (forward copy; source is ahead)
  for (long long i0 = 0; i0 < tail; i0 += blockDim.x) {
    long long i = i0 + threadIdx.x;
    uint32_t v = i < tail ? out[p + i] : 0u;
    __syncthreads();
    if (i < tail) out[i] = v;
    __syncthreads();
  }
  mt_fill_body(states[r], out + tail, cap[r] - tail);
  if (threadIdx.x == 0) {
    sts[r]->stream_pos = 0;
    sts[r]->stream_len = cap[r];
  }
}

// Compact copy of every replica's stream cursor, counters and error flag:
// out[r] = {stream_pos, stream_len, error, n_accept, n_nonfinite, 0}.
__global__ void k_gather_states(DevState* const* sts, int n_rep, long long* out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rep; r += gridDim.x * blockDim.x) {
    const DevState* st = sts[r];
    out[6 * r] = st->stream_pos;
    out[6 * r + 1] = st->stream_len;
    out[6 * r + 2] = st->error;
    out[6 * r + 3] = st->n_accept;
    out[6 * r + 4] = st->n_nonfinite;
    out[6 * r + 5] = st->cell_ok;
  }
}

void launch_gather_states(DevState* const* sts, int n_rep, long long* out, cudaStream_t s) {
  k_gather_states<<<(n_rep + 255) / 256, 256, 0, s>>>(sts, n_rep, out);
}

// Running totals {pair, ewald, bond, ext} of every replica into out[4 r + q].
__global__ void k_gather_energies(DevState* const* sts, int n_rep, double* out) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rep; r += gridDim.x * blockDim.x) {
    const DevState* st = sts[r];
    out[4 * r] = st->e_pair;
    out[4 * r + 1] = st->e_ewald;
    out[4 * r + 2] = st->e_bond;
    out[4 * r + 3] = st->e_ext;
  }
}

void launch_gather_energies(DevState* const* sts, int n_rep, double* out, cudaStream_t s) {
  k_gather_energies<<<(n_rep + 255) / 256, 256, 0, s>>>(sts, n_rep, out);
}

void launch_mt_fill_batch(uint32_t* const* states, uint32_t* const* outs, const long long* pos,
                          const long long* len, const long long* cap, const int* need,
                          DevState* const* sts, int n_rep, cudaStream_t s) {
  k_mt_fill_batch<<<n_rep, kMtThreads, 0, s>>>(states, outs, pos, len, cap, need, sts);
}

void launch_mt_fill(uint32_t* state, uint32_t* out, long long n, cudaStream_t s) {
  if (n > 0) k_mt_fill<<<1, kMtThreads, 0, s>>>(state, out, n);
}

}  // namespace plum
