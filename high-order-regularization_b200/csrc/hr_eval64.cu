// hr_eval64.cu — the FP64 boundary sums: one persistent CTA per SM.
//
// A batch's work items (a block of 128 targets and a run of its interaction
// segments, hr_device.h) are cut into units of one warp: half a block, two
// targets per lane, FP64 accumulators in registers. Every warp takes units
// from a common counter (the first by position, the rest in the items' order
// of decreasing cost) until none is left; a unit's partial sums go to its own
// slot and reduce_kernel adds the slots in order, so results do not depend on
// which warp took a unit.
//   * near segment -> direct sum over a range of a node's sources
//                     (Call_Ds_*, 2S/KITC.cpp:807-1062; in direct mode the one
//                     node holds all sources: eval_Stokes_*_{on,off}Surf of
//                     2S/stokeslets.cpp and 2S/stresslets.cpp, E2G/stokes.cpp)
//   * far segment  -> the node's (P+1)^3 proxy points (Call_Treecode_*,
//                     2S/KITC.cpp:671-777)
//
// What bounds them, measured with probes on this GPU:
//   * The FP64 pipe takes a warp instruction every 2 cycles per SM quarter,
//     but an FMA with three different vector-register operands takes 3 (67 %
//     of the peak); two operands, a repeated one or an immediate take 2. The
//     mix of the pair and proxy loops comes to ~2.4.
//   * A shared-memory load of 16 bytes per lane takes 2 cycles per SM when all
//     lanes read the same address, 4 when they read eight addresses per
//     128-byte phase without bank conflict, 10 from random pieces of a table.
// Measured for the two launches of a batch (two-surface problem, h = 1/64, P =
// 6, N0 = 2000), against one-thread-per-target CTAs with a table each and
// CUDA's rsqrt, erf and exp: stresslet 4.91 -> 3.60 ms (on-surface 2.98 -> 2.31,
// FP64 pipe 57 -> 67 %, data pipe 70 -> 54 %), Stokeslet 4.91 -> 3.58 ms;
// extend-to-grid sums at N = 96 / 192 2.36 / 29.0 -> 1.80 / 22.9 ms (box faces
// 81 % of the FP64 pipe). What they do for that:
//   * Smoothing factors come from piecewise polynomials in s = r^2/delta^2
//     (pieces of width 1/4, hr_eval64_tables.inc), not from erf. Each lane
//     reads its own piece, a gather, so the table is kept eight times, copy c
//     in 16-byte bank group c, and lane l reads copy l mod 8. That takes 131 -
//     165 KB of shared memory: hence one CTA per SM with one table for all its
//     warps, and the persistent form, which stages it once per SM.
//   * Factors that are derivatives of one another (G2 = -2 G1',
//     F = -2 E0', T = -(2/3) F') come from one polynomial, by value and
//     derivative; off-surface factors add a polynomial with the target's
//     coefficients times e^-s, which is a table value e^{-i/4} times a
//     constant-coefficient polynomial in the piece's offset.
//   * A piece's polynomial is in the offset from its centre in pieces, which
//     one multiply-add forms from r^2. Offsets in r^2 with the powers of delta
//     in the coefficients cost the same (two-surface sums; extend-to-grid sums
//     at N = 192 / 384 22.8 / 335 ms against 22.9 / 340) and lose the high-order
//     coefficients to underflow from delta = 1e12 on (delta^-23).
//   * 1/r^3 and 1/r^5 come from the hardware's approximate reciprocal square
//     root y (rsqrt.approx.ftz.f64: a 20-bit result, so y^2 is exact) and the
//     binomial series (1 - e)^{-k/2} in e = 1 - r^2 y^2 (|e| < 2^-18) to second
//     order: no branch, so that consecutive pairs overlap.
//   * Branches (smoothed or plain) are taken by a whole warp, by vote, for all
//     pairs of a step, whose chains overlap; a pair takes what it needs.
//   * Two targets per lane share each source and proxy read. The off-surface
//     stresslet's direct pairs take one at a time (19 more doubles per target).
//   * Sources are packed in tree order, 10 or 12 doubles each, with the area
//     weight already multiplied in, and arrive in the warp's tile by
//     asynchronous copies, double-buffered.
// Warps per CTA and pairs per step (Shape) are the fastest of 8 - 24 warps and
// 1 - 4 sources per step: fewer warps with more registers beat more warps,
// which saturate nothing more (stresslet on-surface 12 warps 2.32 ms, 16 warps
// 2.53, 8 warps 2.43). Measured and not kept: row lengths of the proxy loop
// compiled in (-2 % off the surface, +-0 on it), votes per target set (+2 %).
#include <type_traits>

#include "hr_device.h"
#include "hr_pairs.cuh"

namespace hr {

namespace {

#define HR_SMOOTH_STORAGE __device__ const
#include "hr_eval64_tables.inc"

constexpr int kRep = 8;                             // table copies, one per 16-byte bank group
constexpr double kRoundMagic = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer in the low word
constexpr int kMaxP1 = 16;
constexpr unsigned kFull = 0xffffffffu;

// Classes of work, one kernel each.
enum Cls : int { C_SL_ON = 0, C_SL_OFF, C_DL_ON, C_DL_OFF, C_FACE, C_BAND };

// Smoothing table, warps per CTA, sources per tile, doubles per packed source,
// sources per step of the pair loops, and whether those take both of a lane's
// targets at once.
template <int CLS>
struct Shape;
template <>
struct Shape<C_SL_ON> {
  static constexpr int pieces = HR_T64_G1_PIECES, coef = HR_T64_G1_COEF, warps = 12, tile = 32, rec = 10, unroll = 2;
  static constexpr bool exp = false, pair = true;
};
template <>
struct Shape<C_SL_OFF> {
  static constexpr int pieces = HR_T64_E0_PIECES, coef = HR_T64_E0_COEF, warps = 8, tile = 32, rec = 10, unroll = 2;
  static constexpr bool exp = true, pair = true;
};
template <>
struct Shape<C_DL_ON> {
  static constexpr int pieces = HR_T64_G3_PIECES, coef = HR_T64_G3_COEF, warps = 12, tile = 32, rec = 10, unroll = 2;
  static constexpr bool exp = false, pair = true;
};
template <>
struct Shape<C_DL_OFF> {
  static constexpr int pieces = HR_T64_F0_PIECES, coef = HR_T64_F0_COEF, warps = 8, tile = 32, rec = 10, unroll = 4;
  static constexpr bool exp = true, pair = false;
};
template <>
struct Shape<C_FACE> {
  static constexpr int pieces = 0, coef = 2, warps = 12, tile = 32, rec = 12, unroll = 2;
  static constexpr bool exp = false, pair = true;
};
template <>
struct Shape<C_BAND> {
  static constexpr int pieces = HR_T64_E0_PIECES, coef = HR_T64_E0_COEF, warps = 8, tile = 32, rec = 12, unroll = 1;
  static constexpr bool exp = true, pair = true;
};

template <int CLS>
struct Lay : Shape<CLS> {
  enum : int {
    pairs = (Shape<CLS>::coef + 1) / 2,  // double2s per piece
    tab_d2 = Shape<CLS>::pieces * pairs * kRep,
    exp_d = Shape<CLS>::exp ? 258 : 0,
    tile_d = Shape<CLS>::rec * Shape<CLS>::tile,
    // doubles per warp: two source tiles (or two runs of proxy rows) and the node's Chebyshev points
    warp_d = 2 * tile_d + 3 * kMaxP1,
    smem = 8 * (2 * tab_d2 + exp_d + Shape<CLS>::warps * warp_d)  // bytes
  };
};

// Constants of a task's regularization length.
struct Len {
  double inv_d2;
  double inv_w;    // 4 / delta^2: pieces per unit of r^2
  double df, dt;   // -2 and -2/3 d(pieces)/d(r^2): from a derivative by the piece's offset to G2, F and T
  int hi_tab;      // high word of the largest tabulated r^2
  int hi_zero;     // high word of the reference's r < 1e-14 limit, squared
};

template <int CLS>
__device__ __forceinline__ Len make_len(double d) {
  Len g;
  const double inv = 1.0 / d;
  g.inv_d2 = inv * inv;
  // correctly rounded but for the last step: its relative error is that of every s
  const double d2 = d * d, q = 4.0 / d2;
  g.inv_w = fma(fma(-q, fma(d, d, -d2), fma(-q, d2, 4.0)), 0.25 * q, q);
  g.df = -2.0 * g.inv_w;
  g.dt = -2.0 / 3.0 * g.inv_w;
  // on the surface the factors equal the singular kernel's to 2^-54 from s = 51
  // on (hr_pairs.cuh); off it the reference's switch at r = 8 delta
  const bool on = CLS == C_SL_ON || CLS == C_DL_ON;
  g.hi_tab = __double2hiint((on ? kPlainOnSurf64 : 64.0) * d * d);
  g.hi_zero = __double2hiint(1e-28);
  return g;
}

// Approximate 1/sqrt(x) with 20 significant bits (result's low word zero).
__device__ __forceinline__ double rsqrt20(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// r^2 with its exponent limited to 2^1020, so that the series below gives ~0
// and not NaN where r^2 overflows.
__device__ __forceinline__ double cap(double r2) {
  return __hiloint2double(min(__double2hiint(r2), 0x7fb00000), __double2loint(r2));
}

// The piece of r^2 and the offset from its centre (in pieces: |t| <= 1/2).
template <int CLS>
__device__ __forceinline__ const double2* piece(const double2* tab, const Len& g, double r2, double& t, int& i) {
  const double f = fma(r2, g.inv_w, kRoundMagic);
  t = fma(r2, g.inv_w, kRoundMagic - f);
  i = (int)min((unsigned)__double2loint(f), (unsigned)(Shape<CLS>::pieces - 1));
  return tab + (size_t)i * (Lay<CLS>::pairs * kRep);
}

template <int CLS>
__device__ __forceinline__ void load_piece(const double2* p, double (&c)[2 * Lay<CLS>::pairs]) {
#pragma unroll
  for (int k = 0; k < Lay<CLS>::pairs; k++) {
    const double2 v = p[k * kRep];
    c[2 * k] = v.x;
    c[2 * k + 1] = v.y;
  }
}

// Value of the piece's polynomial.
template <int CLS>
__device__ __forceinline__ double poly(const double (&c)[2 * Lay<CLS>::pairs], double t) {
  double v = c[Shape<CLS>::coef - 1];
#pragma unroll
  for (int k = Shape<CLS>::coef - 2; k >= 0; k--) v = fma(v, t, c[k]);
  return v;
}

// Value and derivative.
template <int CLS>
__device__ __forceinline__ void poly2(const double (&c)[2 * Lay<CLS>::pairs], double t, double& v, double& dv) {
  v = fma(c[Shape<CLS>::coef - 1], t, c[Shape<CLS>::coef - 2]);
  dv = c[Shape<CLS>::coef - 1];
#pragma unroll
  for (int k = Shape<CLS>::coef - 3; k >= 0; k--) {
    dv = fma(dv, t, v);
    v = fma(v, t, c[k]);
  }
}

// e^{-s} at s = (i + t) / 4.
__device__ __forceinline__ double exp_piece(const double* ex, int i, double t) {
  constexpr double c[] = {HR_T64_EXP_COEFS};
  constexpr double q[] = {1.0, 0x1p-2, 0x1p-4, 0x1p-6, 0x1p-8, 0x1p-10, 0x1p-12, 0x1p-14, 0x1p-16, 0x1p-18};
  double v = c[9] * q[9];
#pragma unroll
  for (int k = 8; k >= 0; k--) v = fma(v, t, c[k] * q[k]);
  return v * ex[i];
}

// A lane's target as every class needs it: the position, and what the proxy
// sums and the on-surface pairs subtract (stresslet: the density at the
// target; Stokeslet: f0.n0; extend-to-grid: nothing).
template <bool DL>
struct Tgt {
  double px, py, pz;
  double g0[DL ? 3 : 1];
};

template <int KIND>
__device__ __forceinline__ void load_target(const EvalTask& T, int t, Tgt<KIND == K_DL_ON || KIND == K_DL_OFF>& S) {
  S.px = T.txyz[3 * t];
  S.py = T.txyz[3 * t + 1];
  S.pz = T.txyz[3 * t + 2];
  if constexpr (KIND == K_DL_ON || KIND == K_DL_OFF) {
    const double* g0 = KIND == K_DL_ON ? T.tq : T.tg0;
    for (int k = 0; k < 3; k++) S.g0[k] = g0[3 * t + k];
  } else if constexpr (KIND == K_SL_ON || KIND == K_SL_OFF) {
    // f0.n0: the target's own (2S/KITC.cpp:1461), or at its nearest point (:1568)
    const double *f = KIND == K_SL_ON ? T.tq : T.tf0, *n = KIND == K_SL_ON ? T.tnrm : T.tn0;
    S.g0[0] = f[3 * t] * n[3 * t] + f[3 * t + 1] * n[3 * t + 1] + f[3 * t + 2] * n[3 * t + 2];
  } else {
    S.g0[0] = 0.0;
  }
}

// Polynomials in r^2 of the e^-s terms of the off-surface factors:
//   s1 = (E0 + P e^-s) / delta,     P = c1 - 2 (c2 + c3) s + 4 c3 s^2
//   s2 = (F + Q e^-s) / delta^3,    Q = 2 (c1 + 2 (c2 + c3)) - 4 (c2 + 5 c3) s + 8 c3 s^2
//   s3 = (T + R e^-s) / delta^5,    R = 4/3 [(c1 + 4 c2 + 12 c3) - 2 (c2 + 9 c3) s + 4 c3 s^2]
// The table's e^-s carries 1/delta^m of the family's first factor, the
// polynomials the rest.
struct NearDL {  // an off-surface stresslet target's data for its direct pairs, loaded per segment
  int near;
  // The target is x0 + b n0 with |n0| = 1, up to 1e-13 delta (true for any
  // target without subtraction): beyond 8 delta, where s2 = r^2 s3, its pairs
  // are plain stresslets of g - g0.
  bool foot;
  double b, x0[3], n0[3], g0[3], Q[3], R[3];  // g0: zero without subtraction
  template <int KIND>
  __device__ __forceinline__ void load(const EvalTask& T, int t, const Len& g) {
    near = T.tnear[t];
    b = T.tb[t];
    double off = 0.0, nn = -1.0;
    for (int k = 0; k < 3; k++) {
      x0[k] = T.tx0[3 * t + k];
      n0[k] = T.tn0[3 * t + k];
      g0[k] = near ? T.tg0[3 * t + k] : 0.0;
      off = fmax(off, fabs(fma(-b, n0[k], T.txyz[3 * t + k] - x0[k])));
      nn = fma(n0[k], n0[k], nn);
    }
    foot = !near || (off <= 1e-13 * T.DEL && fabs(nn) <= 1e-13);
    Coef c;
    c.c1 = c.c2 = c.c3 = 0.0;
    if (near) c = reg_coeff(b / T.DEL);
    const double i2 = g.inv_d2, i4 = i2 * i2;
    Q[0] = 2.0 * (c.c1 + 2.0 * (c.c2 + c.c3));
    Q[1] = -4.0 * (c.c2 + 5.0 * c.c3) * i2;
    Q[2] = 8.0 * c.c3 * i4;
    R[0] = 4.0 / 3.0 * (c.c1 + 4.0 * c.c2 + 12.0 * c.c3) * i2;
    R[1] = -8.0 / 3.0 * (c.c2 + 9.0 * c.c3) * i4;
    R[2] = 16.0 / 3.0 * c.c3 * (i4 * i2);
  }
};
struct NearSL {  // the same for the Stokeslet and the extend-to-grid band
  int near;
  double f0n0, P[3], Q[3], v[3];  // f0n0: 0 for a far target (no subtraction, 2S/KITC.cpp:856-882); v = n0 x f0
  template <int KIND>
  __device__ __forceinline__ void load(const EvalTask& T, int t, const Len& g) {
    near = KIND == K_SL_OFF ? T.tnear[t] : 1;
    double f[3], n[3];
    for (int k = 0; k < 3; k++) {
      f[k] = T.tf0[3 * t + k];
      n[k] = T.tn0[3 * t + k];
    }
    f0n0 = near ? f[0] * n[0] + f[1] * n[1] + f[2] * n[2] : 0.0;
    v[0] = n[1] * f[2] - n[2] * f[1];
    v[1] = n[2] * f[0] - n[0] * f[2];
    v[2] = n[0] * f[1] - n[1] * f[0];
    Coef c;
    c.c1 = c.c2 = c.c3 = 0.0;
    if (near) c = reg_coeff(T.tb[t] / T.DEL);
    const double i2 = g.inv_d2, i4 = i2 * i2;
    P[0] = c.c1;
    P[1] = -2.0 * (c.c2 + c.c3) * i2;
    P[2] = 4.0 * c.c3 * i4;
    Q[0] = 2.0 * (c.c1 + 2.0 * (c.c2 + c.c3)) * i2;
    Q[1] = -4.0 * (c.c2 + 5.0 * c.c3) * i4;
    Q[2] = 8.0 * c.c3 * (i4 * i2);
  }
};
struct NearNone {
  template <int KIND>
  __device__ __forceinline__ void load(const EvalTask&, int, const Len&) {}
};

// Work counters of a lane (counting launches only).
struct Count {
  unsigned long long reg = 0, plain = 0, far = 0, prox = 0;
};

struct Src {
  double x, y, z, a, nx, ny, nz, qx, qy, qz;
};
__device__ __forceinline__ Src load_src(const double2* s) {
  const double2 v0 = s[0], v1 = s[1], v2 = s[2], v3 = s[3], v4 = s[4];
  return {v0.x, v0.y, v1.x, v1.y, v2.x, v2.y, v3.x, v3.y, v4.x, v4.y};
}

template <bool COUNT>
__device__ __forceinline__ void count_pair(double r2, const EvalTask& T, bool near, Count& c) {
  if (!COUNT) return;
  const double d64 = 64.0 * T.DEL * T.DEL;
  if (!near) c.far++;
  else if (r2 <= d64 && r2 >= 1e-28) c.reg++;
  else c.plain++;
}

// U consecutive sources and the lane's NT targets of an on-surface stresslet
// sum (Call_Ds_DL_onSurf, 2S/KITC.cpp:921-957). The tile holds area x normal.
template <int NT, int U, bool COUNT>
__device__ __forceinline__ void pairs_dl_on(const double2* s, const Tgt<true> (&S)[NT], const Len& g,
                                            const double2* tab, const bool (&act)[NT], const EvalTask& T, Count& cnt,
                                            double (&a)[NT][4]) {
  double dx[U][NT], dy[U][NT], dz[U][NT], r2[U][NT], w[U][NT], h[U][NT];
  bool tb[U][NT], any_t = false, any_p = false;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const Src q = load_src(s + 5 * u);
#pragma unroll
    for (int k = 0; k < NT; k++) {
      dx[u][k] = S[k].px - q.x;
      dy[u][k] = S[k].py - q.y;
      dz[u][k] = S[k].pz - q.z;
      r2[u][k] = fma(dx[u][k], dx[u][k], fma(dy[u][k], dy[u][k], dz[u][k] * dz[u][k]));
      const double gdd = fma(q.qx - S[k].g0[0], dx[u][k], fma(q.qy - S[k].g0[1], dy[u][k], (q.qz - S[k].g0[2]) * dz[u][k]));
      const double ndd = fma(q.nx, dx[u][k], fma(q.ny, dy[u][k], q.nz * dz[u][k]));
      w[u][k] = ndd * gdd;
      tb[u][k] = __double2hiint(r2[u][k]) <= g.hi_tab;
      any_t |= act[k] && tb[u][k];
      any_p |= act[k] && !tb[u][k];
      if (act[k]) count_pair<COUNT>(r2[u][k], T, true, cnt);
      h[u][k] = 0.0;
    }
  }
  if (__any_sync(kFull, any_t)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++) {
        double t, c[2 * Lay<C_DL_ON>::pairs];
        int i;
        load_piece<C_DL_ON>(piece<C_DL_ON>(tab, g, r2[u][k], t, i), c);
        h[u][k] = poly<C_DL_ON>(c, t);
      }
  }
  if (__any_sync(kFull, any_p)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++) {
        const double x = cap(r2[u][k]), y = rsqrt20(x), y2 = y * y;
        const double e = fma(-x, y2, 1.0);
        const double p = fma(fma(4.375, e, 2.5), e, 1.0) * (y2 * y2 * y);  // r^-5
        h[u][k] = tb[u][k] ? h[u][k] : p;
      }
  }
#pragma unroll
  for (int u = 0; u < U; u++)
#pragma unroll
    for (int k = 0; k < NT; k++) {
      const double v = w[u][k] * h[u][k];
      a[k][0] = fma(dx[u][k], v, a[k][0]);
      a[k][1] = fma(dy[u][k], v, a[k][1]);
      a[k][2] = fma(dz[u][k], v, a[k][2]);
    }
}

// U consecutive sources of an off-surface stresslet sum (Call_Ds_DL,
// 2S/KITC.cpp:962-1062): the subtraction form for near targets, the plain
// stresslet for the others. With m1 = d c1a - n0 c1b and m2 = -sig m1 + d c2a +
// xh c2b the reference's m1 s2 + m2 s3 is d (c1a al + c2a s3) + xh c2b s3 -
// n0 c1b al, al = s2 - sig s3; the n0 terms add up in a scalar (a[3]). The
// tile holds area x normal. A step without a near pair inside 8 delta (by a
// count over all sources four of five of the near warps' pairs of sources at h
// = 1/32, 92 % at h = 1/64) takes the subtraction form's pairs as plain
// stresslets too, where every target of the warp allows it (plain): with x =
// x0 + b n0, d = b n0 - xh and r^2 = sig + b^2 the two are the same, and the
// plain one takes 30 FP64 operations instead of 75. Operator application at h
// = 1/64 3.90 -> 3.73 ms, at h = 1/32 0.811 -> 0.749 ms (steps of 2 / 3 / 4
// sources 3.75 / 3.74 / 3.73; 4 for the plain pairs and 2 for the others
// 3.77). Measured and not kept: whole tiles beyond 8 delta of the box around
// the unit's near targets first, both targets of a lane at once, 3.84 ms.
template <int U, bool COUNT>
__device__ __forceinline__ void pairs_dl_off(const double2* s, const Tgt<true>& P, const NearDL& S, const Len& g,
                                             const double2* tab, const double* ex, bool act, bool any_near, bool any_far, bool plain,
                                             const EvalTask& T, Count& cnt, double (&a)[4]) {
  double dx[U], dy[U], dz[U], r2[U], s2[U], s3[U];
  bool tb[U], any_t = false, any_p = false;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const double2 v0 = s[5 * u], v1 = s[5 * u + 1];
    dx[u] = P.px - v0.x;
    dy[u] = P.py - v0.y;
    dz[u] = P.pz - v1.x;
    r2[u] = fma(dx[u], dx[u], fma(dy[u], dy[u], dz[u] * dz[u]));
    if (act) count_pair<COUNT>(r2[u], T, S.near, cnt);
    tb[u] = S.near && __double2hiint(r2[u]) <= g.hi_tab;
    any_t |= tb[u];
    any_p |= !tb[u];
    s2[u] = s3[u] = 0.0;
  }
  const bool tables = __any_sync(kFull, act && any_t);
  if (!tables && plain) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const Src q = load_src(s + 5 * u);
      const double xr = cap(r2[u]), y = rsqrt20(xr), y2 = y * y;
      const double e = fma(-xr, y2, 1.0);
      const double p5 = fma(fma(4.375, e, 2.5), e, 1.0) * (y2 * y2 * y);
      const double gdd = fma(q.qx - S.g0[0], dx[u], fma(q.qy - S.g0[1], dy[u], (q.qz - S.g0[2]) * dz[u]));
      const double ndd = fma(q.nx, dx[u], fma(q.ny, dy[u], q.nz * dz[u]));
      const double k = gdd * ndd * p5;
      a[0] = fma(dx[u], k, a[0]);
      a[1] = fma(dy[u], k, a[1]);
      a[2] = fma(dz[u], k, a[2]);
    }
    return;
  }
  if (tables) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      double t, c[2 * Lay<C_DL_OFF>::pairs], f, df;
      int i;
      load_piece<C_DL_OFF>(piece<C_DL_OFF>(tab, g, r2[u], t, i), c);
      poly2<C_DL_OFF>(c, t, f, df);
      const double x = exp_piece(ex, i, t);
      s2[u] = fma(fma(fma(S.Q[2], r2[u], S.Q[1]), r2[u], S.Q[0]), x, f);
      s3[u] = fma(fma(fma(S.R[2], r2[u], S.R[1]), r2[u], S.R[0]), x, g.dt * df);
      if (__double2hiint(r2[u]) < g.hi_zero) {  // the reference's values for r < 1e-14
        s2[u] = 256.0 / 15.0 / d_rootpi() / (T.DEL * T.DEL * T.DEL);
        s3[u] = 0.0;
      }
    }
  }
  if (__any_sync(kFull, act && any_p)) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const double xr = cap(r2[u]), y = rsqrt20(xr), y2 = y * y, y3 = y2 * y;
      const double e = fma(-xr, y2, 1.0);
      const double p3 = fma(fma(1.875, e, 1.5), e, 1.0) * y3;         // r^-3
      const double p5 = fma(fma(4.375, e, 2.5), e, 1.0) * (y3 * y2);  // r^-5
      s2[u] = tb[u] ? s2[u] : p3;
      s3[u] = tb[u] ? s3[u] : p5;
    }
  }
  if (any_near) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const Src q = load_src(s + 5 * u);
      const double xh = q.x - S.x0[0], yh = q.y - S.x0[1], zh = q.z - S.x0[2];
      const double gx = q.qx - S.g0[0], gy = q.qy - S.g0[1], gz = q.qz - S.g0[2];
      const double xhn0 = fma(xh, S.n0[0], fma(yh, S.n0[1], zh * S.n0[2]));
      const double sig = fma(-2.0 * S.b, xhn0, fma(xh, xh, fma(yh, yh, zh * zh)));
      const double gn0 = fma(gx, S.n0[0], fma(gy, S.n0[1], gz * S.n0[2]));
      const double gxh = fma(gx, xh, fma(gy, yh, gz * zh));
      const double n0n = fma(q.nx, S.n0[0], fma(q.ny, S.n0[1], q.nz * S.n0[2]));
      const double xhn = fma(q.nx, xh, fma(q.ny, yh, q.nz * zh));
      const double c1b = fma(gxh, n0n, gn0 * xhn);
      const double al = fma(-sig, s3[u], s2[u]);
      const double A = fma(gn0 * n0n, al, gxh * xhn * s3[u]);
      const double B = S.b * c1b * s3[u];
      if (S.near) {
        a[0] = fma(dx[u], A, fma(xh, B, a[0]));
        a[1] = fma(dy[u], A, fma(yh, B, a[1]));
        a[2] = fma(dz[u], A, fma(zh, B, a[2]));
        a[3] = fma(c1b, al, a[3]);
      }
    }
  }
  if (any_far) {
#pragma unroll
    for (int u = 0; u < U; u++) {
      const Src q = load_src(s + 5 * u);
      const double gdd = fma(q.qx, dx[u], fma(q.qy, dy[u], q.qz * dz[u]));
      const double ndd = fma(q.nx, dx[u], fma(q.ny, dy[u], q.nz * dz[u]));
      const double k = gdd * ndd * s3[u];
      if (!S.near) {
        a[0] = fma(dx[u], k, a[0]);
        a[1] = fma(dy[u], k, a[1]);
        a[2] = fma(dz[u], k, a[2]);
      }
    }
  }
}

// 1/r and 1/r^3.
__device__ __forceinline__ void inv13(double r2, double& i1, double& i3) {
  const double x = cap(r2), y = rsqrt20(x), y2 = y * y;
  const double e = fma(-x, y2, 1.0);
  i1 = fma(fma(0.375, e, 0.5) * e, y, y);
  i3 = i1 * i1 * i1;
}

// The smoothed factors s1, s2 of one pair of an off-surface target.
template <int CLS>
__device__ __forceinline__ void factors_off(double r2, const NearSL& N, const Len& g, double del, const double2* tab,
                                            const double* ex, double& s1, double& s2) {
  double t, c[2 * Lay<CLS>::pairs], v, dv;
  int i;
  load_piece<CLS>(piece<CLS>(tab, g, r2, t, i), c);
  poly2<CLS>(c, t, v, dv);
  const double x = exp_piece(ex, i, t);
  s1 = fma(fma(fma(N.P[2], r2, N.P[1]), r2, N.P[0]), x, v);
  s2 = fma(fma(fma(N.Q[2], r2, N.Q[1]), r2, N.Q[0]), x, g.df * dv);
  if (__double2hiint(r2) < g.hi_zero) {  // the reference's values for r < 1e-14
    s1 = 32.0 / 5.0 / d_rootpi() / del;
    s2 = 256.0 / 15.0 / d_rootpi() / (del * del * del);
  }
}

// U consecutive sources and the lane's NT targets of a Stokeslet sum, on the
// surface (Call_Ds_SL_onSurf, 2S/KITC.cpp:807-846) or off it (Call_Ds_SL,
// 2S/KITC.cpp:847-914; a far target's plain kernel is the same form with
// f0.n0 = 0). The tile holds area x normal and area x density.
template <int CLS, int NT, int U, bool COUNT, class NEAR>
__device__ __forceinline__ void pairs_sl(const double2* s, const Tgt<false> (&S)[NT], const NEAR (&N)[NT], const Len& g,
                                         const double2* tab, const double* ex, const bool (&act)[NT],
                                         const EvalTask& T, Count& cnt, double (&a)[NT][4]) {
  constexpr bool ON = CLS == C_SL_ON;
  double dx[U][NT], dy[U][NT], dz[U][NT], r2[U][NT], s1[U][NT], s2[U][NT];
  bool tb[U][NT], any_t = false, any_p = false;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const double2 v0 = s[5 * u], v1 = s[5 * u + 1];
#pragma unroll
    for (int k = 0; k < NT; k++) {
      dx[u][k] = S[k].px - v0.x;
      dy[u][k] = S[k].py - v0.y;
      dz[u][k] = S[k].pz - v1.x;
      r2[u][k] = fma(dx[u][k], dx[u][k], fma(dy[u][k], dy[u][k], dz[u][k] * dz[u][k]));
      bool near = true;
      if constexpr (!ON) near = N[k].near;
      tb[u][k] = near && __double2hiint(r2[u][k]) <= g.hi_tab;
      any_t |= act[k] && tb[u][k];
      any_p |= act[k] && !tb[u][k];
      if (act[k]) count_pair<COUNT>(r2[u][k], T, near, cnt);
      s1[u][k] = s2[u][k] = 0.0;
    }
  }
  if (__any_sync(kFull, any_t)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++) {
        if constexpr (ON) {
          double t, c[2 * Lay<CLS>::pairs], dv;
          int i;
          load_piece<CLS>(piece<CLS>(tab, g, r2[u][k], t, i), c);
          poly2<CLS>(c, t, s1[u][k], dv);
          s2[u][k] = g.df * dv;
        } else {
          factors_off<CLS>(r2[u][k], N[k], g, T.DEL, tab, ex, s1[u][k], s2[u][k]);
        }
      }
  }
  if (__any_sync(kFull, any_p)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++) {
        double i1, i3;
        inv13(r2[u][k], i1, i3);
        s1[u][k] = tb[u][k] ? s1[u][k] : i1;
        s2[u][k] = tb[u][k] ? s2[u][k] : i3;
      }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    const Src q = load_src(s + 5 * u);
#pragma unroll
    for (int k = 0; k < NT; k++) {
      double fn;
      if constexpr (ON) fn = S[k].g0[0];
      else fn = N[k].f0n0;
      const double fx = fma(-fn, q.nx, q.qx), fy = fma(-fn, q.ny, q.qy), fz = fma(-fn, q.nz, q.qz);
      const double w = fma(fx, dx[u][k], fma(fy, dy[u][k], fz * dz[u][k])) * s2[u][k];
      a[k][0] = fma(fx, s1[u][k], fma(dx[u][k], w, a[k][0]));
      a[k][1] = fma(fy, s1[u][k], fma(dy[u][k], w, a[k][1]));
      a[k][2] = fma(fz, s1[u][k], fma(dz[u][k], w, a[k][2]));
    }
  }
}

// The box-face sums (E2G/stokes.cpp:13-45, 102-126): the plain Stokeslet, the
// plain pressure A f.d / r^3, or both (the pressure's term is the Stokeslet's
// factor of d). Records: (x, y) (z, area) (qx, qy) (qz, n.n) (nx, ny) (nz, 0).
template <int KIND, int NT, int U>
__device__ __forceinline__ void pairs_face(const double2* s, const Tgt<false> (&S)[NT], double (&a)[NT][4]) {
#pragma unroll
  for (int u = 0; u < U; u++) {
    const double2 v0 = s[6 * u], v1 = s[6 * u + 1], v2 = s[6 * u + 2];
    const double qz = s[6 * u + 3].x;
#pragma unroll
    for (int k = 0; k < NT; k++) {
      const double dx = S[k].px - v0.x, dy = S[k].py - v0.y, dz = S[k].pz - v1.x;
      const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
      double i1, i3;
      inv13(r2, i1, i3);
      const double w = fma(v2.x, dx, fma(v2.y, dy, qz * dz)) * (i3 * v1.y);
      if constexpr (KIND != K_E2G_P_AWAY) {
        const double h = v1.y * i1;
        a[k][0] = fma(v2.x, h, fma(dx, w, a[k][0]));
        a[k][1] = fma(v2.y, h, fma(dy, w, a[k][1]));
        a[k][2] = fma(qz, h, fma(dz, w, a[k][2]));
      }
      if constexpr (KIND == K_E2G_P_AWAY) a[k][0] += w;
      if constexpr (KIND == K_E2G_UP_AWAY) a[k][3] += w;
    }
  }
}

// The band sums: stokes_SL_7ord (E2G/stokes.cpp:53-97), stokes_pressure_7ord
// (E2G/stokes.cpp:134-203), or both at once. The pressure's
//   -(f.n - f0.n0) n.d - (n x f - n0 x f0).(n x d)
// is f0.n0 (n.d) - (n.n) (f.d) + (n0 x f0).(n x d), by Lagrange's identity, and the
// Stokeslet's (f - f0.n0 n).d is f.d - f0.n0 n.d, so both take f.d and n.d once.
template <int KIND, int NT, int U>
__device__ __forceinline__ void pairs_band(const double2* s, const Tgt<false> (&S)[NT], const NearSL (&N)[NT],
                                           const Len& g, const double2* tab, const double* ex, const bool (&act)[NT],
                                           double del, double (&a)[NT][4]) {
  double dx[U][NT], dy[U][NT], dz[U][NT], r2[U][NT], s1[U][NT], s2[U][NT];
  bool tb[U][NT], any_t = false, any_p = false;
#pragma unroll
  for (int u = 0; u < U; u++) {
    const double2 v0 = s[6 * u], v1 = s[6 * u + 1];
#pragma unroll
    for (int k = 0; k < NT; k++) {
      dx[u][k] = S[k].px - v0.x;
      dy[u][k] = S[k].py - v0.y;
      dz[u][k] = S[k].pz - v1.x;
      r2[u][k] = fma(dx[u][k], dx[u][k], fma(dy[u][k], dy[u][k], dz[u][k] * dz[u][k]));
      tb[u][k] = __double2hiint(r2[u][k]) <= g.hi_tab;
      any_t |= act[k] && tb[u][k];
      any_p |= act[k] && !tb[u][k];
      s1[u][k] = s2[u][k] = 0.0;
    }
  }
  if (__any_sync(kFull, any_t)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++)
        factors_off<C_BAND>(r2[u][k], N[k], g, del, tab, ex, s1[u][k], s2[u][k]);
  }
  if (__any_sync(kFull, any_p)) {
#pragma unroll
    for (int u = 0; u < U; u++)
#pragma unroll
      for (int k = 0; k < NT; k++) {
        double i1, i3;
        inv13(r2[u][k], i1, i3);
        s1[u][k] = tb[u][k] ? s1[u][k] : i1;
        s2[u][k] = tb[u][k] ? s2[u][k] : i3;
      }
  }
#pragma unroll
  for (int u = 0; u < U; u++) {
    const double2 v1 = s[6 * u + 1], v2 = s[6 * u + 2], v3 = s[6 * u + 3], v4 = s[6 * u + 4], v5 = s[6 * u + 5];
    const double qx = v2.x, qy = v2.y, qz = v3.x, nn = v3.y, nx = v4.x, ny = v4.y, nz = v5.x;
#pragma unroll
    for (int k = 0; k < NT; k++) {
      const double x = dx[u][k], y = dy[u][k], z = dz[u][k], fn = N[k].f0n0;
      const double fd = fma(qx, x, fma(qy, y, qz * z)), nd = fma(nx, x, fma(ny, y, nz * z));
      const double h2 = s2[u][k] * v1.y;
      if constexpr (KIND != K_E2G_P7) {
        const double h1 = s1[u][k] * v1.y, w = fma(-fn, nd, fd) * h2;
        a[k][0] = fma(fma(-fn, nx, qx), h1, fma(x, w, a[k][0]));
        a[k][1] = fma(fma(-fn, ny, qy), h1, fma(y, w, a[k][1]));
        a[k][2] = fma(fma(-fn, nz, qz), h1, fma(z, w, a[k][2]));
      }
      if constexpr (KIND != K_E2G_SL7) {
        const double cx = fma(ny, z, -(nz * y)), cy = fma(nz, x, -(nx * z)), cz = fma(nx, y, -(ny * x));
        const double vc = fma(N[k].v[0], cx, fma(N[k].v[1], cy, N[k].v[2] * cz));
        const double p = fma(fn, nd, fma(-nn, fd, vc));
        constexpr int c = KIND == K_E2G_P7 ? 0 : 3;
        a[k][c] = fma(p, h2, a[k][c]);
      }
    }
  }
}

// Proxy interactions of a run of Chebyshev rows (row r = i (P+1) + j holds
// proxies (i, j, 0..P)) from the warp's shared copy of the node's proxy-major
// moments. Stresslet per proxy: (M00, M11) (M22, M01 + M10) (M02 + M20,
// M12 + M21) (n0, n1) (n2, 0), the kernel d (d.M.d - (g0.d)(n.d)) / r^5 with
// d.M.d in powers of the row's variable d2 (Call_Treecode_DL,
// 2S/KITC.cpp:753-771, regrouped); Stokeslet: f, n (Call_Treecode_SL,
// 2S/KITC.cpp:700-714). The x and y components of a row are multiplied by
// its d0, d1 once, at its end.
template <bool DL, int NT>
__device__ __forceinline__ void proxy_rows(const double2* __restrict__ s2, int row0, int nrows, int P1,
                                           const double* __restrict__ cheb, const Tgt<DL> (&S)[NT],
                                           double (&a)[NT][4]) {
  constexpr int W = DL ? 5 : 3;  // double2 per proxy
  int pi = row0 / P1, pj = row0 - pi * P1;
  for (int r = 0; r < nrows; r++) {
    const double cx = cheb[pi], cy = cheb[P1 + pj];
    if (++pj == P1) {
      pj = 0;
      pi++;
    }
    const double2* row = s2 + r * P1 * W;
    double d0[NT], d1[NT], d00[NT], d11[NT], d01[NT], r01[NT], g0r[NT], t0[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) {
      d0[k] = S[k].px - cx;
      d1[k] = S[k].py - cy;
      d00[k] = d0[k] * d0[k];
      d11[k] = d1[k] * d1[k];
      r01[k] = d00[k] + d11[k];
      if constexpr (DL) {
        d01[k] = d0[k] * d1[k];
        g0r[k] = fma(S[k].g0[0], d0[k], S[k].g0[1] * d1[k]);
      }
      t0[k] = 0.0;
    }
#pragma unroll 2
    for (int pk = 0; pk < P1; pk++) {
      const double cz = cheb[2 * P1 + pk];
      const double2* m = row + pk * W;
      if constexpr (DL) {
        const double2 s01 = m[0], s23 = m[1], s45 = m[2], n01 = m[3];
        const double n2 = m[4].x;
#pragma unroll
        for (int k = 0; k < NT; k++) {
          const double d2 = S[k].pz - cz;
          const double r2 = fma(d2, d2, r01[k]);
          const double y = rsqrt20(r2), y2 = y * y, y4 = y2 * y2;
          const double e = fma(-r2, y2, 1.0);
          const double A = fma(s01.x, d00[k], fma(s01.y, d11[k], s23.y * d01[k]));
          const double B = fma(s45.x, d0[k], s45.y * d1[k]);
          const double mnd = fma(n2, d2, fma(n01.x, d0[k], n01.y * d1[k]));
          const double g0d = fma(S[k].g0[2], d2, g0r[k]);
          const double num = fma(-g0d, mnd, fma(fma(s23.x, d2, B), d2, A));
          const double v = (num * (y4 * y)) * fma(fma(4.375, e, 2.5), e, 1.0);
          t0[k] += v;
          a[k][2] = fma(d2, v, a[k][2]);
        }
      } else {
        const double2 m01 = m[0], m23 = m[1], m45 = m[2];
#pragma unroll
        for (int k = 0; k < NT; k++) {
          const double d2 = S[k].pz - cz;
          const double r2 = cap(fma(d2, d2, r01[k]));
          const double y = rsqrt20(r2), y2 = y * y;
          const double e = fma(-r2, y2, 1.0);
          const double rinv = fma(fma(0.375, e, 0.5) * e, y, y);
          const double q0 = fma(-S[k].g0[0], m23.y, m01.x);
          const double q1 = fma(-S[k].g0[0], m45.x, m01.y);
          const double q2 = fma(-S[k].g0[0], m45.y, m23.x);
          const double v = fma(q0, d0[k], fma(q1, d1[k], q2 * d2)) * (rinv * rinv * rinv);
          a[k][0] = fma(q0, rinv, a[k][0]);
          a[k][1] = fma(q1, rinv, a[k][1]);
          a[k][2] = fma(q2, rinv, fma(v, d2, a[k][2]));
          t0[k] += v;
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NT; k++) {
      a[k][0] = fma(d0[k], t0[k], a[k][0]);
      a[k][1] = fma(d1[k], t0[k], a[k][1]);
    }
  }
}

// Asynchronous copy of `bytes` (a multiple of 16, both addresses 16-byte
// aligned) from global to shared memory by the 32 lanes of a warp.
__device__ __forceinline__ void warp_copy_async(void* dst, const void* src, int bytes, int lane) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  const char* s = static_cast<const char*>(src);
  for (int o = lane * 16; o < bytes; o += 32 * 16)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d + o), "l"(s + o) : "memory");
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void copy_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// A near segment (sources s0 .. s0 + n - 1) for the lane's NT targets t, tile by tile.
template <int CLS, int KIND, int NT, bool COUNT>
__device__ __forceinline__ void near_segment(const EvalTask& T, int s0, int n,
                                             const Tgt<KIND == K_DL_ON || KIND == K_DL_OFF> (&S)[NT],
                                             const int (&t)[NT], const bool (&act)[NT], const Len& g,
                                             const double2* tab, const double* ex, double* wsm, Count& cnt,
                                             double (&p)[NT][4]) {
  constexpr int kTile = Shape<CLS>::tile, kTileD = Lay<CLS>::tile_d, kRec = Shape<CLS>::rec, U = Shape<CLS>::unroll;
  const int lane = threadIdx.x & 31;
  const double* src = T.pk + kRec * (size_t)s0;
  const int ntile = (n + kTile - 1) / kTile;
  warp_copy_async(wsm, src, min(kTile, n) * 8 * kRec, lane);
  using NEAR = std::conditional_t<CLS == C_DL_OFF, NearDL, std::conditional_t<CLS == C_SL_OFF || CLS == C_BAND, NearSL, NearNone>>;
  NEAR N[NT];
  for (int k = 0; k < NT; k++) N[k].template load<KIND>(T, t[k], g);
  bool any_near = true, any_far = false, plain = false;
  if constexpr (KIND == K_DL_OFF) {
    plain = !__any_sync(kFull, act[0] && !N[0].foot);
    any_near = __any_sync(kFull, act[0] && N[0].near);
    any_far = __any_sync(kFull, act[0] && !N[0].near);
  }
  for (int i = 0; i < ntile; i++) {
    const int c = min(kTile, n - i * kTile);
    if (i + 1 < ntile) {
      warp_copy_async(wsm + ((i + 1) & 1) * kTileD, src + (size_t)(i + 1) * kTileD,
                      min(kTile, n - (i + 1) * kTile) * 8 * kRec, lane);
      copy_async_wait<1>();
    } else {
      copy_async_wait<0>();
    }
    __syncwarp();
    const double2* s = reinterpret_cast<const double2*>(wsm + (i & 1) * kTileD);
    auto step = [&](auto uc, int j) {
      constexpr int V = decltype(uc)::value;
      const double2* q = s + (kRec / 2) * j;
      if constexpr (KIND == K_DL_ON) pairs_dl_on<NT, V, COUNT>(q, S, g, tab, act, T, cnt, p);
      else if constexpr (KIND == K_DL_OFF)
        pairs_dl_off<V, COUNT>(q, S[0], N[0], g, tab, ex, act[0], any_near, any_far, plain, T, cnt, p[0]);
      else if constexpr (KIND == K_SL_ON || KIND == K_SL_OFF) pairs_sl<CLS, NT, V, COUNT>(q, S, N, g, tab, ex, act, T, cnt, p);
      else if constexpr (CLS == C_FACE) pairs_face<KIND, NT, V>(q, S, p);
      else pairs_band<KIND, NT, V>(q, S, N, g, tab, ex, act, T.DEL, p);
    };
    int j = 0;
    for (; j + U <= c; j += U) step(std::integral_constant<int, U>(), j);
    for (; j < c; j++) step(std::integral_constant<int, 1>(), j);
    __syncwarp();
  }
  if constexpr (KIND == K_DL_OFF) {  // the n0 terms; a far target's n0 is never used and may hold anything
    if (N[0].near)
      for (int c = 0; c < 3; c++) p[0][c] = fma(-N[0].n0[c], p[0][3], p[0][c]);
    p[0][3] = 0.0;
  }
}

// A far node for the lane's NT targets: its moments stream through the two
// halves of the warp's tile in runs of whole Chebyshev rows.
template <int CLS, bool DL, int NT>
__device__ __forceinline__ void far_node(const EvalTask& T, int nd, const Tgt<DL> (&S)[NT], double* wsm, double* cheb,
                                         double (&p)[NT][4]) {
  constexpr int kHalf = 8 * Lay<CLS>::tile_d;  // bytes
  const int lane = threadIdx.x & 31;
  const int P1 = T.P1, rowb = P1 * (DL ? 80 : 48), nr = kHalf / rowb, nrow_all = P1 * P1;
  const char* src = reinterpret_cast<const char*>(T.mom + (size_t)nd * T.Pf * T.C);
  char* buf = reinterpret_cast<char*>(wsm);
  for (int i = lane; i < 3 * P1; i += 32) cheb[i] = T.tcheb[(size_t)nd * 3 * P1 + i];
  const int nch = (nrow_all + nr - 1) / nr;
  warp_copy_async(buf, src, min(nr, nrow_all) * rowb, lane);
  for (int ch = 0; ch < nch; ch++) {
    const int row0 = ch * nr, rows = min(nr, nrow_all - row0);
    if (ch + 1 < nch) {
      const int r1 = row0 + nr;
      warp_copy_async(buf + ((ch + 1) & 1) * kHalf, src + (size_t)r1 * rowb, min(nr, nrow_all - r1) * rowb, lane);
      copy_async_wait<1>();
    } else {
      copy_async_wait<0>();
    }
    __syncwarp();
    proxy_rows<DL, NT>(reinterpret_cast<const double2*>(buf + (ch & 1) * kHalf), row0, rows, P1, cheb, S, p);
    __syncwarp();
  }
}

// One unit: half h (64 targets, two per lane: lane and lane + 32) of an item's
// target block, all its segments.
template <int CLS, int KIND, bool COUNT>
__device__ __forceinline__ void run_unit(const EvalTask& T, const BlockRef& it, int h, const Seg* __restrict__ segs,
                                         const double2* tab, const double* ex, double* wsm, double* cheb) {
  constexpr bool kTree = KIND == K_SL_ON || KIND == K_SL_OFF || KIND == K_DL_ON || KIND == K_DL_OFF;
  constexpr bool DL = KIND == K_DL_ON || KIND == K_DL_OFF;
  constexpr bool kPair = Shape<CLS>::pair;  // near segments take both targets at once
  const int lane = threadIdx.x & 31;
  const int k0 = it.blk * kTB + h * 64 + lane;
  const bool valid[2] = {k0 < T.nt, k0 + 32 < T.nt};
  if (!__any_sync(kFull, valid[0])) return;  // the block's tail: no slot of these targets is read
  const Len g = make_len<CLS>(T.DEL);
  Tgt<DL> S[2];
  int t[2];
  double a[2][4];
  for (int k = 0; k < 2; k++) {
    t[k] = T.tord[valid[k] ? k0 + 32 * k : it.blk * kTB];
    load_target<KIND>(T, t[k], S[k]);
    for (int c = 0; c < 4; c++) a[k][c] = 0.0;
  }
  Count cnt;
  for (int base = it.seg0; base < it.seg1; base += 32) {
    // 32 segments at a time, one per lane; those without a target of this half drop out
    const int q = base + lane;
    Seg sg{0, 0, 0};
    int node = 0, type = 0;
    uint32_t w0 = 0, w1 = 0;
    if (q < it.seg1) {
      sg = segs[q];
      const Entry* E = T.entries + sg.entry;
      node = E->node;
      type = E->type;
      w0 = E->mask[2 * h];
      w1 = E->mask[2 * h + 1];
    }
    unsigned live = __ballot_sync(kFull, (w0 | w1) != 0u);
    while (live) {
      const int l = __ffs(live) - 1;
      live &= live - 1;
      const uint32_t m0 = __shfl_sync(kFull, w0, l), m1 = __shfl_sync(kFull, w1, l);
      const int ty = __shfl_sync(kFull, type, l), nd = __shfl_sync(kFull, node, l);
      const int s0 = __shfl_sync(kFull, sg.s0, l), n = __shfl_sync(kFull, sg.s1, l) - s0;
      const bool act[2] = {valid[0] && ((m0 >> lane) & 1u), valid[1] && ((m1 >> lane) & 1u)};
      if (m0 != 0u && m1 != 0u && (ty == 0 || kPair)) {
        double p[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
        if (ty == 1) {
          if constexpr (kPair) near_segment<CLS, KIND, 2, COUNT>(T, s0, n, S, t, act, g, tab, ex, wsm, cnt, p);
        } else if constexpr (kTree) {
          far_node<CLS, DL, 2>(T, nd, S, wsm, cheb, p);
        }
        for (int k = 0; k < 2; k++)
          if (act[k])
            for (int c = 0; c < 4; c++) a[k][c] += p[k][c];
      } else {
#pragma unroll 1
        for (int k = 0; k < 2; k++) {  // one target per lane at a time
          if ((k == 0 ? m0 : m1) == 0u) continue;
          const Tgt<DL> S1[1] = {k == 0 ? S[0] : S[1]};
          const int t1[1] = {k == 0 ? t[0] : t[1]};
          const bool act1[1] = {k == 0 ? act[0] : act[1]};
          double p[1][4] = {{0.0, 0.0, 0.0, 0.0}};
          if (ty == 1) near_segment<CLS, KIND, 1, COUNT>(T, s0, n, S1, t1, act1, g, tab, ex, wsm, cnt, p);
          else if constexpr (kTree) far_node<CLS, DL, 1>(T, nd, S1, wsm, cheb, p);
          if (act1[0])
            for (int c = 0; c < 4; c++) {
              a[0][c] += k == 0 ? p[0][c] : 0.0;
              a[1][c] += k == 1 ? p[0][c] : 0.0;
            }
        }
      }
      if (COUNT && ty == 0) cnt.prox += (unsigned long long)T.Pf * (act[0] + act[1]);
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    double2* o = reinterpret_cast<double2*>(T.partial + ((size_t)it.slot * kTB + h * 64 + 32 * k + lane) * kPartComps);
    o[0] = make_double2(a[k][0], a[k][1]);
    o[1] = make_double2(a[k][2], a[k][3]);
  }
  if (COUNT && T.counters) {
    unsigned long long v[4] = {cnt.reg, cnt.plain, cnt.far, cnt.prox};
    for (int c = 0; c < 4; c++) {
      for (int off = 16; off > 0; off >>= 1) v[c] += __shfl_down_sync(kFull, v[c], off);
      if (lane == 0 && v[c]) atomicAdd(&T.counters[c], v[c]);
    }
  }
}

template <int CLS, bool COUNT>
__global__ void __launch_bounds__(Shape<CLS>::warps * 32, 1)
    eval64_kernel(const EvalTask* __restrict__ tasks, const BlockRef* __restrict__ items,
                  const Seg* __restrict__ segs, unsigned nunits, unsigned* __restrict__ next) {
  extern __shared__ __align__(16) double sm[];
  double2* tab = reinterpret_cast<double2*>(sm);
  double* ex = sm + 2 * Lay<CLS>::tab_d2;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* wsm = ex + Lay<CLS>::exp_d + warp * Lay<CLS>::warp_d;
  // the smoothing table, eight copies, its coefficients scaled to offsets in
  // pieces (exactly, by powers of four) and to the power of 1/delta of the factor
  // (all tasks of a batch share one delta)
  if constexpr (Shape<CLS>::pieces > 0) {
    const double inv = 1.0 / tasks[items[0].task].DEL, i2 = inv * inv;
    const double lead = CLS == C_DL_ON ? i2 * i2 * inv : (CLS == C_DL_OFF ? i2 * inv : inv);
    const double* src = CLS == C_DL_ON ? kT64G3 : (CLS == C_DL_OFF ? kT64F0 : (CLS == C_SL_ON ? kT64G1 : kT64E0));
    constexpr int kP = Lay<CLS>::pairs;
    double scale[2 * kP];
    scale[0] = lead;
#pragma unroll
    for (int k = 1; k < 2 * kP; k++) scale[k] = scale[k - 1] * 0.25;
    for (int i = threadIdx.x; i < Shape<CLS>::pieces; i += blockDim.x) {
#pragma unroll
      for (int k = 0; k < kP; k++) {
        const double2 v = make_double2(src[i * 2 * kP + 2 * k] * scale[2 * k], src[i * 2 * kP + 2 * k + 1] * scale[2 * k + 1]);
#pragma unroll
        for (int c = 0; c < kRep; c++) tab[((size_t)i * kP + k) * kRep + ((c + i) & (kRep - 1))] = v;
      }
    }
    if (Shape<CLS>::exp)
      for (int i = threadIdx.x; i < 257; i += blockDim.x) ex[i] = kT64Exp[i] * lead;
  }
  __syncthreads();
  tab += lane & (kRep - 1);
  for (unsigned u = warp * gridDim.x + blockIdx.x; u < nunits;) {
    unsigned nx = 0;
    if (lane == 0) nx = atomicAdd(next, 1u);  // returns while the unit runs
    const BlockRef it = items[u >> 1];
    const EvalTask& T = tasks[it.task];
    double* cheb = wsm + 2 * Lay<CLS>::tile_d;
    auto unit = [&](auto kc) { run_unit<CLS, decltype(kc)::value, COUNT>(T, it, u & 1, segs, tab, ex, wsm, cheb); };
    if constexpr (CLS == C_SL_ON) unit(std::integral_constant<int, K_SL_ON>());
    if constexpr (CLS == C_SL_OFF) unit(std::integral_constant<int, K_SL_OFF>());
    if constexpr (CLS == C_DL_ON) unit(std::integral_constant<int, K_DL_ON>());
    if constexpr (CLS == C_DL_OFF) unit(std::integral_constant<int, K_DL_OFF>());
    if constexpr (CLS == C_FACE) {
      if (T.kind == K_E2G_UP_AWAY) unit(std::integral_constant<int, K_E2G_UP_AWAY>());
      else if (T.kind == K_E2G_SL_AWAY) unit(std::integral_constant<int, K_E2G_SL_AWAY>());
      else unit(std::integral_constant<int, K_E2G_P_AWAY>());
    }
    if constexpr (CLS == C_BAND) {
      if (T.kind == K_E2G_UP7) unit(std::integral_constant<int, K_E2G_UP7>());
      else if (T.kind == K_E2G_SL7) unit(std::integral_constant<int, K_E2G_SL7>());
      else unit(std::integral_constant<int, K_E2G_P7>());
    }
    u = __shfl_sync(kFull, nx, 0) + gridDim.x * Shape<CLS>::warps;
  }
}

template <int CLS, bool COUNT>
void launch_one(const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems, unsigned* next,
                int num_sms, cudaStream_t st) {
  static_assert(Lay<CLS>::smem <= 227 * 1024, "the table and the tiles fit one CTA");
  // set on every launch: the attribute belongs to the current device's context
  cudaFuncSetAttribute(eval64_kernel<CLS, COUNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay<CLS>::smem);
  const unsigned nunits = 2u * (unsigned)nitems;
  const unsigned grid = nunits < (unsigned)num_sms ? nunits : (unsigned)num_sms;
  eval64_kernel<CLS, COUNT><<<grid, Shape<CLS>::warps * 32, Lay<CLS>::smem, st>>>(d_tasks, d_items, d_segs, nunits, next);
}

}  // namespace

void launch_eval64(int family, const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems,
                   int n_on, unsigned* next, int num_sms, cudaStream_t st, cudaStream_t side, bool count) {
  const int n_off = nitems - n_on;
  auto both = [&](auto on, auto off) {
    if (n_on > 0) on(d_items, n_on, next, st);
    if (n_off > 0) off(d_items + n_on, n_off, next + 1, side);
  };
#define HR_LAUNCH(CLS, COUNT)                                                       \
  [&](const BlockRef* items, int n, unsigned* nx, cudaStream_t s) {                 \
    launch_one<CLS, COUNT>(d_tasks, items, d_segs, n, nx, num_sms, s);              \
  }
  if (family == F_SL) {
    if (count) both(HR_LAUNCH(C_SL_ON, true), HR_LAUNCH(C_SL_OFF, true));
    else both(HR_LAUNCH(C_SL_ON, false), HR_LAUNCH(C_SL_OFF, false));
  } else if (family == F_DL) {
    if (count) both(HR_LAUNCH(C_DL_ON, true), HR_LAUNCH(C_DL_OFF, true));
    else both(HR_LAUNCH(C_DL_ON, false), HR_LAUNCH(C_DL_OFF, false));
  } else {  // the extend-to-grid tasks carry no counters
    both(HR_LAUNCH(C_FACE, false), HR_LAUNCH(C_BAND, false));
  }
#undef HR_LAUNCH
}

}  // namespace hr
