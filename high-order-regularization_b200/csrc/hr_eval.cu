// hr_eval.cu — the reduced-precision boundary sums (HR_MIXED, HR_FP32) and the
// reduction of every batch; the FP64 sums are in hr_eval64.cu.
//
// Two-surface sums: one persistent CTA of 12 warps per SM; every warp takes
// units (half a block of 128 spatially sorted targets, two targets per lane,
// FP64 accumulators in registers) from a common counter, walks the unit's
// interaction segments in order and writes the unit's own partial sums, so
// results do not depend on scheduling. Extend-to-grid sums: a CTA per item.
//   * near segment -> direct sum over the node's member sources, staged in
//                     shared memory in tiles (Call_Ds_*, 2S/KITC.cpp:807-1062;
//                     in direct mode the single node holds all sources, i.e.
//                     eval_Stokes_*_{on,off}Surf of 2S/stokeslets.cpp and
//                     2S/stresslets.cpp, and the sums of E2G/stokes.cpp);
//   * far segment  -> the node's (P+1)^3 proxy points with their moments staged
//                     in shared memory (Call_Treecode_*, 2S/KITC.cpp:671-777).
//
// What bounds the two-surface kernels: the issue slots and the FP32 pipe. The
// packed operations (two sources or two proxies of a target per instruction)
// have the pipe's FP32 rate at half the issue slots: a probe gives 0.47 packed
// FMAs per cycle and SM quarter against 1.0 scalar ones (0.38 with three
// different operands). With them, rsqrt without denormal scaling and units
// taken by the warp, the stresslet batch's kernels (two-surface problem, h =
// 1/64, P = 6, N0 = 2000) execute 0.73e9 + 0.69e9 instructions instead of
// 1.21e9 + 0.90e9; on-surface 1.92 -> 1.17 ms, off-surface 1.71 -> 1.15 ms,
// the operator application 3.53 -> 2.47 ms against one scalar pair at a time
// in CTAs per item. Twelve warps: 168 registers, two targets' sums without
// spills; 8 / 10 / 13 / 14 warps 3.41 (8, before the finer items) / 2.57 /
// 2.55 / 2.62 ms.
//
// Precision. MIXED: FP32 pairs from FP32 coordinates relative to the target
// block's first target, summed per 16 terms in FP32 and added to the FP64
// per-target accumulators:
//   * on-surface kinds: every pair, the smoothing factors from FP32
//     piecewise polynomials in s = r^2/delta^2 (no erf / exp, and no
//     cancellation at any r);
//   * off-surface kinds: pairs with r > 3 delta (the plain kernels of far
//     targets, the regularized kernels with erff / expf, the subtraction
//     forms) in FP32; pairs with r <= 3 delta, where the erf / exp brackets
//     with the target's coefficients cancel, in FP64;
//   * all proxy interactions in FP32.
// FP32 (all pairs): as MIXED with every off-surface pair in FP32 too.
#include "hr_device.h"
#include "hr_pairs.cuh"

namespace hr {

namespace {

#define HR_SMOOTH_STORAGE __device__ const
#include "hr_smoothing_tables.inc"

// The singular kernel takes over at s = kPlainOnSurf32; the tables are staged
// up to there, in kRep32 copies (a lane reads copy lane & 7).
constexpr int kPieces32 = (int)(kPlainOnSurf32 * HR_SMOOTH32_PIECES / 64.0f) + 1, kRep32 = 8;

// FP32 piece: (centre, c0, c1, c2) (c3, c4, c5, 0); index floor(s * pieces / 64)
// for 0 <= s <= kPlainOnSurf32, formed on the FMA / ALU pipes: adding 1.5 * 2^23
// to s * pieces / 64 - 1/2 leaves round-to-nearest of it, i.e. the floor (a tie
// picks the lower piece, whose polynomial covers its right end), in the low
// mantissa bits.
__device__ __forceinline__ float smooth_eval_f(const float4* __restrict__ tab, float s) {
  const float f = fmaf(s, HR_SMOOTH32_PIECES / 64.0f, -0.5f) + 12582912.0f;
  const int i = __float_as_int(f) - 0x4B400000;
  const float4 a = tab[2 * i * kRep32], b = tab[(2 * i + 1) * kRep32];
  const float t = s - a.x;
  return fmaf(fmaf(fmaf(fmaf(fmaf(b.z, t, b.y), t, b.x), t, a.w), t, a.z), t, a.y);
}

constexpr int kWarps = kTB / 32;     // warps per CTA, each with its own tiles
constexpr int kNT = 64;              // sources per (per-warp) shared-memory tile
constexpr int kWarpSm = 10 * kNT;    // doubles per warp: a source tile, 10 values per source
constexpr int kSmem = kWarps * kWarpSm;
constexpr int kMaxP1 = 16;

struct Tgt {
  double px, py, pz;
  double b;
  int near;
  double f0n0;
  double x0[3], n0[3], g0[3];
  double n0xf0[3];
  Coef c;
};

struct Tgt32 {
  float px, py, pz;  // relative to the FP32 origin of the target block
  float f0n0;        // 0 for targets without subtraction
  float g0[3];
  float n0xf0[3];
  float b;
  float x0[3];       // relative to the FP32 origin of the target block
  float n0[3];
  CoefF c;
};

template <int KIND>
__device__ __forceinline__ void load_target(const EvalTask& T, int t, bool valid, const double* cb, Tgt& S,
                                            Tgt32& F) {
  S.px = S.py = S.pz = 0.0;
  S.b = 0.0;
  S.f0n0 = 0.0;
  for (int k = 0; k < 3; k++) S.x0[k] = S.n0[k] = S.g0[k] = S.n0xf0[k] = 0.0;
  S.c.c1 = S.c.c2 = S.c.c3 = 0.0;
  // regularized-kernel kinds: on-surface sums and the extend-to-grid band sums
  S.near = (KIND == K_SL_ON || KIND == K_DL_ON || KIND == K_E2G_UP7) ? 1 : 0;
  if (valid) {
    S.px = T.txyz[3 * t];
    S.py = T.txyz[3 * t + 1];
    S.pz = T.txyz[3 * t + 2];
    if (KIND == K_SL_ON) {
      // f0_dot_n0 = Surfc[i].f . Surfc[i].Nrml  (2S/KITC.cpp:1461, 2S/stokeslets.cpp:167)
      S.f0n0 = T.tq[3 * t] * T.tnrm[3 * t] + T.tq[3 * t + 1] * T.tnrm[3 * t + 1] +
               T.tq[3 * t + 2] * T.tnrm[3 * t + 2];
    } else if (KIND == K_SL_OFF) {
      S.b = T.tb[t];
      S.near = T.tnear[t];
      // f0_dot_n0 = nrst_f . nrst_Nrml  (2S/KITC.cpp:1568)
      S.f0n0 = T.tf0[3 * t] * T.tn0[3 * t] + T.tf0[3 * t + 1] * T.tn0[3 * t + 1] +
               T.tf0[3 * t + 2] * T.tn0[3 * t + 2];
      if (S.near) S.c = reg_coeff(S.b / T.DEL);
    } else if (KIND == K_DL_ON) {
      for (int k = 0; k < 3; k++) S.g0[k] = T.tq[3 * t + k];
    } else if (KIND == K_DL_OFF) {
      S.b = T.tb[t];
      S.near = T.tnear[t];
      for (int k = 0; k < 3; k++) {
        S.x0[k] = T.tx0[3 * t + k];
        S.n0[k] = T.tn0[3 * t + k];
        S.g0[k] = T.tg0[3 * t + k];
      }
      if (S.near) S.c = reg_coeff(S.b / T.DEL);
    } else if (KIND == K_E2G_UP7) {
      S.b = T.tb[t];
      double f0[3], n0[3];
      for (int k = 0; k < 3; k++) {
        f0[k] = T.tf0[3 * t + k];
        n0[k] = T.tn0[3 * t + k];
      }
      // E2G/stokes.cpp:144-145
      S.f0n0 = f0[0] * n0[0] + f0[1] * n0[1] + f0[2] * n0[2];
      S.n0xf0[0] = n0[1] * f0[2] - n0[2] * f0[1];
      S.n0xf0[1] = n0[2] * f0[0] - n0[0] * f0[2];
      S.n0xf0[2] = n0[0] * f0[1] - n0[1] * f0[0];
      S.c = reg_coeff(S.b / T.DEL);
    }
  }
  F.px = (float)(S.px - cb[0]);
  F.py = (float)(S.py - cb[1]);
  F.pz = (float)(S.pz - cb[2]);
  // the direct sum of a far Stokeslet target has no subtraction (2S/KITC.cpp:856-882),
  // nor has the plain stresslet of a far target (2S/KITC.cpp:970-995)
  F.f0n0 = (KIND == K_SL_OFF && !S.near) ? 0.0f : (float)S.f0n0;
  const bool no_g0 = KIND == K_DL_OFF && !S.near;
  for (int k = 0; k < 3; k++) {
    F.g0[k] = no_g0 ? 0.0f : (float)S.g0[k];
    F.n0xf0[k] = (float)S.n0xf0[k];
    F.x0[k] = (float)(S.x0[k] - cb[k]);
    F.n0[k] = (float)S.n0[k];
  }
  F.b = (float)S.b;
  F.c.c1 = (float)S.c.c1;
  F.c.c2 = (float)S.c.c2;
  F.c.c3 = (float)S.c.c3;
}

// ---------------------------------------------------------------- FP64 pairs

// One FP64 pair of a target that uses the regularized forms, for r <= 3 delta.
template <int KIND>
__device__ __forceinline__ void pair64(const double* __restrict__ sm, int j, const Tgt& S, const Reg& g, double& a0,
                                       double& a1, double& a2) {
  // source j of the warp's tile: (x, y) (z, area) (nx, ny) (nz, qx) (qy, qz)
  const double2* s2 = reinterpret_cast<const double2*>(sm) + 5 * j;
  const double2 v0 = s2[0], v1 = s2[1], v2 = s2[2], v3 = s2[3], v4 = s2[4];
  const double Xj = v0.x, Yj = v0.y, Zj = v1.x, Aj = v1.y;
  const double NXj = v2.x, NYj = v2.y, NZj = v3.x, QXj = v3.y, QYj = v4.x, QZj = v4.y;
  const double dx = S.px - Xj, dy = S.py - Yj, dz = S.pz - Zj;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double rinv = rsqrt(r2);
  if (KIND == K_SL_OFF) {
    // Call_Ds_SL regularized branch (2S/KITC.cpp:847)
    const double area = Aj;
    const double fx = QXj - S.f0n0 * NXj;
    const double fy = QYj - S.f0n0 * NYj;
    const double fz = QZj - S.f0n0 * NZj;
    const double fdd = fx * dx + fy * dy + fz * dz;
    double H1, H2;
    sl_7ord(r2, rinv, g, S.c, H1, H2);
    H1 *= area;
    H2 *= area * fdd;
    a0 += fx * H1 + dx * H2;
    a1 += fy * H1 + dy * H2;
    a2 += fz * H1 + dz * H2;
  } else {  // K_DL_OFF
    // Call_Ds_DL regularized branch (2S/KITC.cpp:996-1059), stokes_DL_7ord
    const double b = S.b;
    const double xh0 = Xj - S.x0[0];
    const double xh1 = Yj - S.x0[1];
    const double xh2 = Zj - S.x0[2];
    const double gx = QXj - S.g0[0];
    const double gy = QYj - S.g0[1];
    const double gz = QZj - S.g0[2];
    const double sig_sq = (xh0 * xh0 + xh1 * xh1 + xh2 * xh2) -
                          2.0 * b * (xh0 * S.n0[0] + xh1 * S.n0[1] + xh2 * S.n0[2]);
    const double g_dot_n0 = gx * S.n0[0] + gy * S.n0[1] + gz * S.n0[2];
    const double g_dot_xh = gx * xh0 + gy * xh1 + gz * xh2;
    const double n0_dot_n = S.n0[0] * NXj + S.n0[1] * NYj + S.n0[2] * NZj;
    const double xh_dot_n = xh0 * NXj + xh1 * NYj + xh2 * NZj;
    const double c_m1a = g_dot_n0 * n0_dot_n;
    const double c_m1b = g_dot_xh * n0_dot_n + g_dot_n0 * xh_dot_n;
    const double c_m2a = g_dot_xh * xh_dot_n;
    const double c_m2b = b * c_m1b;
    double H2, H3;
    dl_7ord(r2, rinv, g, S.c, H2, H3);
    const double area = Aj;
    H2 *= area;
    H3 *= area;
    double m1 = dx * c_m1a - S.n0[0] * c_m1b;
    double m2 = -sig_sq * m1 + dx * c_m2a + xh0 * c_m2b;
    a0 += m1 * H2 + m2 * H3;
    m1 = dy * c_m1a - S.n0[1] * c_m1b;
    m2 = -sig_sq * m1 + dy * c_m2a + xh1 * c_m2b;
    a1 += m1 * H2 + m2 * H3;
    m1 = dz * c_m1a - S.n0[2] * c_m1b;
    m2 = -sig_sq * m1 + dz * c_m2a + xh2 * c_m2b;
    a2 += m1 * H2 + m2 * H3;
  }
}

// The band sums of one target in one pass (K_E2G_UP7): stokes_SL_7ord and
// stokes_pressure_7ord (E2G/stokes.cpp:53-97, 134-203) share the offset, the
// distance and the regularized factors' erf and exp (sl_lapl_7ord); each
// keeps its own expressions; a3 collects the pressure.
__device__ __forceinline__ void pair64_band(const double* __restrict__ sm, int j, const Tgt& S, const Reg& g,
                                            double& a0, double& a1, double& a2, double& a3) {
  const double2* s2v = reinterpret_cast<const double2*>(sm) + 5 * j;
  const double2 v0 = s2v[0], v1 = s2v[1], v2 = s2v[2], v3 = s2v[3], v4 = s2v[4];
  const double Xj = v0.x, Yj = v0.y, Zj = v1.x, Aj = v1.y;
  const double NXj = v2.x, NYj = v2.y, NZj = v3.x, QXj = v3.y, QYj = v4.x, QZj = v4.y;
  const double dx = S.px - Xj, dy = S.py - Yj, dz = S.pz - Zj;
  const double r2 = dx * dx + dy * dy + dz * dz;
  const double rinv = rsqrt(r2);
  double H1, H2, H2p;
  sl_lapl_7ord(r2, rinv, g, S.c, H1, H2, H2p);
  {
    const double area = Aj;
    const double fx = QXj - S.f0n0 * NXj;
    const double fy = QYj - S.f0n0 * NYj;
    const double fz = QZj - S.f0n0 * NZj;
    const double fdd = fx * dx + fy * dy + fz * dz;
    H1 *= area;
    H2 *= area * fdd;
    a0 += fx * H1 + dx * H2;
    a1 += fy * H1 + dy * H2;
    a2 += fz * H1 + dz * H2;
  }
  {
    const double n0 = NXj, n1 = NYj, n2 = NZj;
    const double f0 = QXj, f1 = QYj, f2 = QZj;
    const double f_dot_n = f0 * n0 + f1 * n1 + f2 * n2;
    const double ncf0 = (n1 * f2 - n2 * f1) - S.n0xf0[0];
    const double ncf1 = (n2 * f0 - n0 * f2) - S.n0xf0[1];
    const double ncf2 = (n0 * f1 - n1 * f0) - S.n0xf0[2];
    const double n_dot_dx = n0 * dx + n1 * dy + n2 * dz;
    const double ncd0 = n1 * dz - n2 * dy;
    const double ncd1 = n2 * dx - n0 * dz;
    const double ncd2 = n0 * dy - n1 * dx;
    const double normal = -(f_dot_n - S.f0n0) * n_dot_dx;
    const double tangential = -(ncf0 * ncd0 + ncf1 * ncd1 + ncf2 * ncd2);
    a3 += (normal + tangential) * H2p * Aj;
  }
}

// ------------------------------------------------------- FP32 extend-to-grid pairs
// The box-face sums (E2G/stokes.cpp:13-45, 102-126) in FP32 in one pass, sharing
// the offset, the distance and f.dx.
__device__ __forceinline__ void pair32_face(const float4* __restrict__ s4, int j, const Tgt32& F, float& p0,
                                            float& p1, float& p2, float& p3) {
  const float4 P = s4[j];  // x, y, z, area
  const float4 Q = s4[2 * kNT + j];
  const float dx = F.px - P.x, dy = F.py - P.y, dz = F.pz - P.z;
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float rinv = rsqrtf(r2);
  const float rinv2 = rinv * rinv;
  const float fdd = Q.x * dx + Q.y * dy + Q.z * dz;
  const float H1 = P.w * rinv;
  const float H2 = fdd * H1 * rinv2;
  p0 += Q.x * H1 + dx * H2;
  p1 += Q.y * H1 + dy * H2;
  p2 += Q.z * H1 + dz * H2;
  p3 += fdd * (rinv2 * rinv) * P.w;
}

// The band sums in FP32 in one pass, for pairs with r > 3 delta.
__device__ __forceinline__ void pair32r_band(const float4* __restrict__ s4, int j, const Tgt32& F, const RegF& gf,
                                             float& p0, float& p1, float& p2, float& p3) {
  const float4 P = s4[j];  // x, y, z, area
  const float4 N = s4[kNT + j];
  const float4 Q = s4[2 * kNT + j];
  const float dx = F.px - P.x, dy = F.py - P.y, dz = F.pz - P.z;
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float rinv = rsqrtf(r2);
  float H1, H2, H2p;
  sl_lapl_7ord_f(r2, rinv, gf, F.c, H1, H2, H2p);
  {
    const float fx = Q.x - F.f0n0 * N.x;
    const float fy = Q.y - F.f0n0 * N.y;
    const float fz = Q.z - F.f0n0 * N.z;
    const float fdd = fx * dx + fy * dy + fz * dz;
    H1 *= P.w;
    H2 *= P.w * fdd;
    p0 += fx * H1 + dx * H2;
    p1 += fy * H1 + dy * H2;
    p2 += fz * H1 + dz * H2;
  }
  {
    const float n0 = N.x, n1 = N.y, n2 = N.z;
    const float f0 = Q.x, f1 = Q.y, f2 = Q.z;
    const float f_dot_n = f0 * n0 + f1 * n1 + f2 * n2;
    const float ncf0 = (n1 * f2 - n2 * f1) - F.n0xf0[0];
    const float ncf1 = (n2 * f0 - n0 * f2) - F.n0xf0[1];
    const float ncf2 = (n0 * f1 - n1 * f0) - F.n0xf0[2];
    const float n_dot_dx = n0 * dx + n1 * dy + n2 * dz;
    const float ncd0 = n1 * dz - n2 * dy;
    const float ncd1 = n2 * dx - n0 * dz;
    const float ncd2 = n0 * dy - n1 * dx;
    const float normal = -(f_dot_n - F.f0n0) * n_dot_dx;
    const float tangential = -(ncf0 * ncd0 + ncf1 * ncd1 + ncf2 * ncd2);
    p3 += (normal + tangential) * H2p * P.w;
  }
}

// ------------------------------------------------ FP32 pairs, r > 3 delta
// The full kernel of a target that uses the regularized forms (the smoothed
// branch for r <= 8 delta, the singular one beyond, with the target's
// subtraction), in FP32 for pairs with r > 3 delta.
template <int KIND>
__device__ __forceinline__ void pair32r(const float4* __restrict__ s4, int j, const Tgt32& F, const RegF& gf,
                                        float& p0, float& p1, float& p2) {
  const float4 P = s4[j];  // x, y, z, area
  const float4 N = s4[kNT + j];
  const float4 Q = s4[2 * kNT + j];
  const float dx = F.px - P.x, dy = F.py - P.y, dz = F.pz - P.z;
  const float r2 = dx * dx + dy * dy + dz * dz;
  const float rinv = rsqrtf(r2);
  if (KIND == K_SL_OFF) {
    const float fx = Q.x - F.f0n0 * N.x;
    const float fy = Q.y - F.f0n0 * N.y;
    const float fz = Q.z - F.f0n0 * N.z;
    const float fdd = fx * dx + fy * dy + fz * dz;
    float H1, H2;
    sl_7ord_f(r2, rinv, gf, F.c, H1, H2);
    H1 *= P.w;
    H2 *= P.w * fdd;
    p0 += fx * H1 + dx * H2;
    p1 += fy * H1 + dy * H2;
    p2 += fz * H1 + dz * H2;
  } else {  // K_DL_OFF
    // the subtraction form of a near target (2S/KITC.cpp:996-1059)
    const float b = F.b;
    const float xh0 = P.x - F.x0[0], xh1 = P.y - F.x0[1], xh2 = P.z - F.x0[2];
    const float gx = Q.x - F.g0[0], gy = Q.y - F.g0[1], gz = Q.z - F.g0[2];
    const float sig_sq = (xh0 * xh0 + xh1 * xh1 + xh2 * xh2) - 2.0f * b * (xh0 * F.n0[0] + xh1 * F.n0[1] + xh2 * F.n0[2]);
    const float g_dot_n0 = gx * F.n0[0] + gy * F.n0[1] + gz * F.n0[2];
    const float g_dot_xh = gx * xh0 + gy * xh1 + gz * xh2;
    const float n0_dot_n = F.n0[0] * N.x + F.n0[1] * N.y + F.n0[2] * N.z;
    const float xh_dot_n = xh0 * N.x + xh1 * N.y + xh2 * N.z;
    const float c_m1a = g_dot_n0 * n0_dot_n;
    const float c_m1b = g_dot_xh * n0_dot_n + g_dot_n0 * xh_dot_n;
    const float c_m2a = g_dot_xh * xh_dot_n;
    const float c_m2b = b * c_m1b;
    float H2, H3;
    dl_7ord_f(r2, rinv, gf, F.c, H2, H3);
    H2 *= P.w;
    H3 *= P.w;
    float m1 = dx * c_m1a - F.n0[0] * c_m1b;
    float m2 = -sig_sq * m1 + dx * c_m2a + xh0 * c_m2b;
    p0 += m1 * H2 + m2 * H3;
    m1 = dy * c_m1a - F.n0[1] * c_m1b;
    m2 = -sig_sq * m1 + dy * c_m2a + xh1 * c_m2b;
    p1 += m1 * H2 + m2 * H3;
    m1 = dz * c_m1a - F.n0[2] * c_m1b;
    m2 = -sig_sq * m1 + dz * c_m2a + xh2 * c_m2b;
    p2 += m1 * H2 + m2 * H3;
  }
}

// ------------------------------------------------------------ proxy tiles

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

// ------------------------------------------- two-surface sums: packed FP32
// Two FP32 values in a 64-bit register: the packed operations round each half
// as the scalar ones do. One instruction serves two sources (or two proxies)
// of a target; the sums over sources stay scalar, in source order.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
  f2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float lo(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) {
  f2 v;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
  return v;
}
__device__ __forceinline__ f2 vmul(f2 a, f2 b) {
  f2 v;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ f2 vsub(f2 a, f2 b) {
  f2 v;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
  return v;
}
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float vmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float vsub(float a, float b) { return __fsub_rn(a, b); }
// rsqrtf without the scaling of denormal arguments (r below 1.1e-19)
__device__ __forceinline__ float vrsqrt(float x) {
  float v;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(v) : "f"(x));
  return v;
}
__device__ __forceinline__ f2 vrsqrt(f2 x) { return pack2(vrsqrt(lo(x)), vrsqrt(hi(x))); }
template <class V>
__device__ __forceinline__ V dup(float x);
template <>
__device__ __forceinline__ float dup<float>(float x) {
  return x;
}
template <>
__device__ __forceinline__ f2 dup<f2>(float x) {
  return pack2(x, x);
}
// p + a b and p + a, the halves in order
__device__ __forceinline__ float sum_mul(float p, float a, float b) { return __fmaf_rn(a, b, p); }
__device__ __forceinline__ float sum_mul(float p, f2 a, f2 b) {
  return __fmaf_rn(hi(a), hi(b), __fmaf_rn(lo(a), lo(b), p));
}
__device__ __forceinline__ float sum(float p, float a) { return __fadd_rn(p, a); }
__device__ __forceinline__ float sum(float p, f2 a) { return __fadd_rn(__fadd_rn(p, lo(a)), hi(a)); }

// The FP32 data of a lane's target (offsets from the block's origin): of the
// Stokeslet -f0.n0, of the stresslet -g0, zero without subtraction.
struct Tgt2 {
  float px, py, pz;
  float m0, m1, m2;
};

template <bool DL>
struct Rec {
  static constexpr int vals = DL ? 9 : 6;          // FP32 moments per proxy
  static constexpr int pair_b = DL ? 80 : 48;      // bytes of two proxies, interleaved value by value
};

// One proxy (V = float) or two (V = f2) of a Chebyshev row for one target.
// Stresslet moments: S = (M00, M11, M22, M01 + M10, M02 + M20, M12 + M21), Mn;
// Stokeslet: f, n. The stresslet kernel uses
//   sum_l (sum_k (M[3l+k] - g0_l Mn_k) d_k) d_l = d.M.d - (g0.d)(Mn.d),
// the reference's proxy sum (Call_Treecode_DL, 2S/KITC.cpp:753-771)
// regrouped, with d.M.d from the symmetric part and the products of d0, d1
// taken once per row; Call_Treecode_SL (2S/KITC.cpp:700-714) as written. The
// rounding of each operation, and so each result bit, is that of the scalar
// loops this replaces, whose on-surface form (ON) sums Mn.d in another order.
template <bool DL, bool ON, class V>
struct RowT {
  V d0, d1, r01, d00, d11, d01, s;  // s: DL the (d0, d1) part of -g0.d, SL -f0.n0
  V pz, mz;
  __device__ __forceinline__ RowT(const Tgt2& F, float cx, float cy) {
    const float e0 = F.px - cx, e1 = F.py - cy;
    const float e11 = __fmul_rn(e1, e1);
    d0 = dup<V>(e0);
    d1 = dup<V>(e1);
    pz = dup<V>(F.pz);
    if (DL) {
      const float e00 = __fmul_rn(e0, e0);
      d00 = dup<V>(e00);
      r01 = dup<V>(__fadd_rn(e00, e11));
      d11 = dup<V>(e11);
      d01 = dup<V>(__fmul_rn(e0, e1));
      s = dup<V>(__fmaf_rn(F.m0, e0, __fmul_rn(F.m1, e1)));
      mz = dup<V>(F.m2);
    } else {
      r01 = dup<V>(__fmaf_rn(e0, e0, e11));
      s = dup<V>(F.m0);
    }
  }
  __device__ __forceinline__ void add(const V (&m)[Rec<DL>::vals], V cz, float (&p)[3]) const {
    const V d2 = vsub(pz, cz);
    const V rinv = vrsqrt(vfma(d2, d2, r01));
    if constexpr (DL) {
      V dmd = vfma(m[0], d00, vmul(m[1], d11));
      dmd = vfma(m[2], vmul(d2, d2), dmd);
      dmd = vfma(m[3], d01, dmd);
      dmd = vfma(m[4], vmul(d0, d2), dmd);
      dmd = vfma(m[5], vmul(d1, d2), dmd);
      const V mnd = vfma(m[8], d2, ON ? vfma(m[7], d1, vmul(m[6], d0)) : vfma(m[6], d0, vmul(m[7], d1)));
      const V g0d = vfma(mz, d2, s);  // negated
      const V ri2 = vmul(rinv, rinv);
      const V kernel = vmul(vfma(g0d, mnd, dmd), vmul(vmul(ri2, ri2), rinv));
      p[0] = sum_mul(p[0], d0, kernel);
      p[1] = sum_mul(p[1], d1, kernel);
      p[2] = sum_mul(p[2], d2, kernel);
    } else {
      const V m0 = vfma(s, m[3], m[0]), m1 = vfma(s, m[4], m[1]), m2 = vfma(s, m[5], m[2]);
      const V temp = vmul(vfma(m2, d2, vfma(m0, d0, vmul(m1, d1))), vmul(vmul(rinv, rinv), rinv));
      p[0] = sum(p[0], vfma(m0, rinv, vmul(temp, d0)));
      p[1] = sum(p[1], vfma(m1, rinv, vmul(temp, d1)));
      p[2] = sum(p[2], vfma(m2, rinv, vmul(temp, d2)));
    }
  }
};

// Proxy interactions of a run of Chebyshev rows (row r = i (P+1) + j holds
// proxies (i, j, 0..P)) from the warp's shared copy of the node's moments,
// two proxies at a time, an odd last one alone. Every lane reads the same
// proxies (a shared-memory broadcast). FP32 per row, FP64 across the rows;
// act: whose sums count. P1C > 0 compiles the row length.
template <bool DL, bool ON, int NT, int P1C>
__device__ __forceinline__ void proxy_rows(const char* buf, int row0, int nrows, int P1rt, const float* cheb,
                                           const Tgt2 (&F)[NT], const bool (&act)[NT], double (&a)[NT][3]) {
  constexpr int kV = Rec<DL>::vals;
  const int P1 = P1C > 0 ? P1C : P1rt;
  const int rowb = ((P1 + 1) / 2) * Rec<DL>::pair_b;
  int pi = row0 / P1, pj = row0 - pi * P1;
  for (int r = 0; r < nrows; r++) {
    const float cx = cheb[pi], cy = cheb[kMaxP1 + pj];
    if (++pj == P1) pj = 0, pi++;
    float p[NT][3];
    const char* row = buf + r * rowb;
    auto pairs = [&](auto one) {
      using V = decltype(one);
      constexpr bool kPair = sizeof(V) == 8;
      if constexpr (kPair)
        for (int k = 0; k < NT; k++) p[k][0] = p[k][1] = p[k][2] = 0.f;
      const RowT<DL, ON, V> R0(F[0], cx, cy), R1(F[NT - 1], cx, cy);
#pragma unroll
      for (int q = kPair ? 0 : P1 / 2; q < (kPair ? P1 / 2 : P1 / 2 + 1); q++) {
        const ulonglong2* v = reinterpret_cast<const ulonglong2*>(row + q * Rec<DL>::pair_b);
        f2 w[kV + 1];
#pragma unroll
        for (int i = 0; i < kV / 2; i++) {
          const ulonglong2 u = v[i];
          w[2 * i] = u.x;
          w[2 * i + 1] = u.y;
        }
        if (kV & 1) w[kV - 1] = reinterpret_cast<const f2*>(v)[kV - 1];
        V m[kV], cz;
#pragma unroll
        for (int i = 0; i < kV; i++)
          if constexpr (kPair) m[i] = w[i];
          else m[i] = lo(w[i]);
        if constexpr (kPair) cz = reinterpret_cast<const f2*>(cheb + 2 * kMaxP1)[q];
        else cz = cheb[2 * kMaxP1 + 2 * q];
        R0.add(m, cz, p[0]);
        if (NT == 2) R1.add(m, cz, p[NT - 1]);
      }
    };
    pairs(f2());
    if (P1 & 1) pairs(float());
#pragma unroll
    for (int k = 0; k < NT; k++)
      if (act[k])
        for (int c = 0; c < 3; c++) a[k][c] += (double)p[k][c];
  }
}

constexpr int kTile = 64;             // sources of a tile
constexpr int kPairF = 20;            // floats of two sources, interleaved value by value
constexpr int kBufB = 5120;           // a warp's buffer: two runs of proxy rows, or a tile
constexpr int kChebB = 3 * kMaxP1 * 4;
// An off-surface warp's buffer also holds the FP64 tile of the targets that
// use the regularized forms; their FP32 tile and the pair tile follow.
constexpr int kNearB = 3 * kTile * 16, kTileB = kTile / 2 * kPairF * 4;

// A far node for the lane's NT targets: its moments stream through the two
// halves of the warp's buffer in runs of whole Chebyshev rows; the copy of the
// next run overlaps the interactions of this one.
template <bool DL, bool ON, int NT>
__device__ __forceinline__ void far_node(const EvalTask& T, int nd, const Tgt2 (&F)[NT], const bool (&act)[NT],
                                         const double (&cb)[3], char* buf, float* cheb, double (&a)[NT][3]) {
  constexpr int kHalf = kBufB / 2;
  const int lane = threadIdx.x & 31;
  const int P1 = T.P1, rowb = ((P1 + 1) / 2) * Rec<DL>::pair_b, nr = kHalf / rowb, nrow_all = P1 * P1;
  const char* src = reinterpret_cast<const char*>(T.momf) + (size_t)nd * nrow_all * rowb;
  __syncwarp();
  for (int i = lane; i < 3 * P1; i += 32) {
    const int c = i / P1;
    cheb[c * kMaxP1 + i - c * P1] = (float)(T.tcheb[(size_t)nd * 3 * P1 + i] - cb[c]);
  }
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
    const char* b = buf + (ch & 1) * kHalf;
    switch (P1) {  // degrees 3 to 10 compiled: P = 7 10 % faster than with a counted loop, P = 6 5 %
      case 4: proxy_rows<DL, ON, NT, 4>(b, row0, rows, P1, cheb, F, act, a); break;
      case 5: proxy_rows<DL, ON, NT, 5>(b, row0, rows, P1, cheb, F, act, a); break;
      case 6: proxy_rows<DL, ON, NT, 6>(b, row0, rows, P1, cheb, F, act, a); break;
      case 7: proxy_rows<DL, ON, NT, 7>(b, row0, rows, P1, cheb, F, act, a); break;
      case 8: proxy_rows<DL, ON, NT, 8>(b, row0, rows, P1, cheb, F, act, a); break;
      case 9: proxy_rows<DL, ON, NT, 9>(b, row0, rows, P1, cheb, F, act, a); break;
      case 10: proxy_rows<DL, ON, NT, 10>(b, row0, rows, P1, cheb, F, act, a); break;
      case 11: proxy_rows<DL, ON, NT, 11>(b, row0, rows, P1, cheb, F, act, a); break;
      default: proxy_rows<DL, ON, NT, 0>(b, row0, rows, P1, cheb, F, act, a);
    }
    __syncwarp();
  }
}

// A tile's sources, two interleaved; an odd last one is followed by a copy of
// its position without area, normal or density. On-surface: (x, y, z), area x
// normal, density (SL: area x density); off-surface (x, y, z), area, normal,
// density.
template <int KIND>
__device__ __forceinline__ void stage_pairs(const EvalTask& T, int s0, int cnt, const double (&cb)[3], float* tile) {
  constexpr bool kOn = KIND == K_SL_ON || KIND == K_DL_ON;
  for (int i = threadIdx.x & 31; i < ((cnt + 1) & ~1); i += 32) {
    const int s = s0 + min(i, cnt - 1);
    float v[10];
    v[0] = (float)(T.sx[s] - cb[0]);
    v[1] = (float)(T.sy[s] - cb[1]);
    v[2] = (float)(T.sz[s] - cb[2]);
    for (int c = 3; c < 10; c++) v[c] = 0.f;
    if (i < cnt) {
      if (kOn) {
        const double as = T.sa[s];
        v[3] = (float)(as * T.snx[s]);
        v[4] = (float)(as * T.sny[s]);
        v[5] = (float)(as * T.snz[s]);
        v[6] = KIND == K_SL_ON ? (float)(as * T.qx[s]) : T.fqx[s];
        v[7] = KIND == K_SL_ON ? (float)(as * T.qy[s]) : T.fqy[s];
        v[8] = KIND == K_SL_ON ? (float)(as * T.qz[s]) : T.fqz[s];
      } else {
        v[3] = T.fnx[s];
        v[4] = T.fny[s];
        v[5] = T.fnz[s];
        v[6] = T.fqx[s];
        v[7] = T.fqy[s];
        v[8] = T.fqz[s];
        v[9] = T.fa[s];
      }
    }
    float* w = tile + (i >> 1) * kPairF + (i & 1);
#pragma unroll
    for (int c = 0; c < (kOn ? 9 : 10); c++) w[2 * c] = v[c];
  }
}

// Two sources for the lane's NT targets.
// On-surface (Call_Ds_SL_onSurf / Call_Ds_DL_onSurf, 2S/KITC.cpp:807-846,
// 921-957): the smoothing factor from the table up to s = kPlainOnSurf32, the
// singular kernel beyond; the warp looks tables up only where one of its pairs
// needs them (lim: -1 for a target whose sums do not count).
// Off-surface, targets beyond 8 delta: the singular kernel.
template <int KIND, int NT>
__device__ __forceinline__ void pairs_step(const float* q, const Tgt2 (&F)[NT], const float (&lim)[NT], f2 inv_d2,
                                           const float4* tab, float (&p)[NT][3]) {
  constexpr bool kOn = KIND == K_SL_ON || KIND == K_DL_ON, kSL = KIND == K_SL_ON || KIND == K_SL_OFF;
  f2 w[10];
  const ulonglong2* v = reinterpret_cast<const ulonglong2*>(q);
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const ulonglong2 u = v[i];
    w[2 * i] = u.x;
    w[2 * i + 1] = u.y;
  }
  f2 dx[NT], dy[NT], dz[NT], r2[NT], sq[NT];
  bool in = false;
#pragma unroll
  for (int k = 0; k < NT; k++) {
    dx[k] = vsub(dup<f2>(F[k].px), w[0]);
    dy[k] = vsub(dup<f2>(F[k].py), w[1]);
    dz[k] = vsub(dup<f2>(F[k].pz), w[2]);
    r2[k] = vfma(dz[k], dz[k], vfma(dx[k], dx[k], vmul(dy[k], dy[k])));
    if (kOn) {
      sq[k] = vmul(r2[k], inv_d2);
      in = in || lo(sq[k]) <= lim[k] || hi(sq[k]) <= lim[k];
    }
  }
  if constexpr (kOn) in = __any_sync(0xffffffffu, in);
#pragma unroll
  for (int k = 0; k < NT; k++) {
    f2 H1, H2;
    const f2 ri = vrsqrt(r2[k]), ri2 = vmul(ri, ri);
    if (kSL) {
      H1 = ri;
      H2 = vmul(ri2, ri);
    } else {
      H2 = vmul(vmul(ri2, ri2), ri);
    }
    if constexpr (kOn) {
      if (in) {
        const float s0 = lo(sq[k]), s1 = hi(sq[k]);
        const float t0 = fminf(s0, kPlainOnSurf32), t1 = fminf(s1, kPlainOnSurf32);
        if (kSL) {
          const float u0 = smooth_eval_f(tab, t0), u1 = smooth_eval_f(tab, t1);
          H1 = pack2(s0 <= kPlainOnSurf32 ? u0 : lo(H1), s1 <= kPlainOnSurf32 ? u1 : hi(H1));
          tab += 2 * kPieces32 * kRep32;
        }
        const float u0 = smooth_eval_f(tab, t0), u1 = smooth_eval_f(tab, t1);
        H2 = pack2(s0 <= kPlainOnSurf32 ? u0 : lo(H2), s1 <= kPlainOnSurf32 ? u1 : hi(H2));
        if (kSL) tab -= 2 * kPieces32 * kRep32;
      }
    }
    if constexpr (kSL) {
      const f2 nf = dup<f2>(F[k].m0);
      const f2 fx = vfma(nf, w[3], w[6]), fy = vfma(nf, w[4], w[7]), fz = vfma(nf, w[5], w[8]);
      const f2 fdd = vfma(fz, dz[k], vfma(fx, dx[k], vmul(fy, dy[k])));
      f2 h2;
      if (kOn) {
        h2 = vmul(H2, fdd);
      } else {
        H1 = vmul(w[9], ri);
        h2 = vmul(vmul(fdd, H1), ri2);
      }
      p[k][0] = sum(p[k][0], vfma(fx, H1, vmul(dx[k], h2)));
      p[k][1] = sum(p[k][1], vfma(fy, H1, vmul(dy[k], h2)));
      p[k][2] = sum(p[k][2], vfma(fz, H1, vmul(dz[k], h2)));
    } else {
      // a far target has no subtraction
      const f2 gx = kOn ? vsub(w[6], dup<f2>(-F[k].m0)) : w[6], gy = kOn ? vsub(w[7], dup<f2>(-F[k].m1)) : w[7],
               gz = kOn ? vsub(w[8], dup<f2>(-F[k].m2)) : w[8];
      const f2 gdd = vfma(gz, dz[k], vfma(gx, dx[k], vmul(gy, dy[k])));
      const f2 ndd = vfma(w[5], dz[k], vfma(w[3], dx[k], vmul(w[4], dy[k])));
      f2 kernel = vmul(vmul(ndd, gdd), H2);
      if (!kOn) kernel = vmul(kernel, w[9]);
      p[k][0] = sum_mul(p[k][0], dx[k], kernel);
      p[k][1] = sum_mul(p[k][1], dy[k], kernel);
      p[k][2] = sum_mul(p[k][2], dz[k], kernel);
    }
  }
}

// A tile of cnt sources for NT targets, FP32 sums of 16 sources added in FP64.
template <int KIND, int NT>
__device__ __forceinline__ void tile_pairs(const float* tile, int cnt, const Tgt2 (&F)[NT], const bool (&act)[NT],
                                           f2 inv_d2, const float4* tab, double (&a)[NT][3]) {
  constexpr bool kDL = KIND == K_DL_ON || KIND == K_DL_OFF;
  float lim[NT];
  for (int k = 0; k < NT; k++) lim[k] = act[k] ? kPlainOnSurf32 : -1.0f;
  const int np = (cnt + 1) >> 1;
  for (int j0 = 0; j0 < np; j0 += 8) {
    float p[NT][3];
    for (int k = 0; k < NT; k++) p[k][0] = p[k][1] = p[k][2] = 0.f;
    const int j1 = min(np, j0 + 8);
#pragma unroll(kDL ? 2 : 1)
    for (int j = j0; j < j1; j++) pairs_step<KIND, NT>(tile + j * kPairF, F, lim, inv_d2, tab, p);
#pragma unroll
    for (int k = 0; k < NT; k++)
      if (act[k])
        for (int c = 0; c < 3; c++) a[k][c] += (double)p[k][c];
  }
}

// The pairs of one target per lane that uses the regularized forms: FP64 for
// r <= 3 delta (all-FP32 mode: only the r < 1e-14 limits), FP32 beyond.
template <int KIND>
__device__ __noinline__ double3 tile_near(const EvalTask& T, int t, bool act, int cnt, double3 org,
                                          const double* wsm, const float4* ws4, double3 a) {
  if (!act) return a;
  const double cb[3] = {org.x, org.y, org.z};
  Tgt S;
  Tgt32 F;
  load_target<KIND>(T, t, true, cb, S, F);
  const Reg g = make_reg(T.DEL);
  RegF gf;
  gf.inv_d = (float)g.inv_d;
  gf.d64 = (float)g.d64;
  const float cut2f = T.mixed == 2 ? 1e-28f : (float)(9.0 * T.DEL * T.DEL);
  double a0 = a.x, a1 = a.y, a2 = a.z;
  for (int j0 = 0; j0 < cnt; j0 += 16) {
    float p0 = 0.f, p1 = 0.f, p2 = 0.f;
    const int j1 = min(cnt, j0 + 16);
    for (int j = j0; j < j1; j++) {
      const float4 Pj = ws4[j];
      const float dx = F.px - Pj.x, dy = F.py - Pj.y, dz = F.pz - Pj.z;
      if (dx * dx + dy * dy + dz * dz > cut2f) pair32r<KIND>(ws4, j, F, gf, p0, p1, p2);
      else pair64<KIND>(wsm, j, S, g, a0, a1, a2);
    }
    a0 += (double)p0;
    a1 += (double)p1;
    a2 += (double)p2;
  }
  return make_double3(a0, a1, a2);
}

// The FP64 and FP32 tiles of tile_near.
__device__ __forceinline__ void stage_near(const EvalTask& T, int s0, int cnt, const double (&cb)[3], double* wsm,
                                           float4* ws4) {
  for (int i = threadIdx.x & 31; i < cnt; i += 32) {
    const int s = s0 + i;
    const double x = T.sx[s], y = T.sy[s], z = T.sz[s];
    double2* w2 = reinterpret_cast<double2*>(wsm) + 5 * i;
    w2[0] = make_double2(x, y);
    w2[1] = make_double2(z, T.sa[s]);
    w2[2] = make_double2(T.snx[s], T.sny[s]);
    w2[3] = make_double2(T.snz[s], T.qx[s]);
    w2[4] = make_double2(T.qy[s], T.qz[s]);
    ws4[i] = make_float4((float)(x - cb[0]), (float)(y - cb[1]), (float)(z - cb[2]), T.fa[s]);
    ws4[kNT + i] = make_float4(T.fnx[s], T.fny[s], T.fnz[s], 0.f);
    ws4[2 * kNT + i] = make_float4(T.fqx[s], T.fqy[s], T.fqz[s], 0.f);
  }
}

// A near segment [s0, s0 + n) for NT targets; near: which of them use the
// regularized forms (off-surface kinds).
template <int KIND, int NT>
__device__ __forceinline__ void near_segment(const EvalTask& T, int s0, int n, const Tgt2 (&F)[NT],
                                             const int (&t)[NT], const bool (&act)[NT], const bool (&near)[NT],
                                             const double (&cb)[3], f2 inv_d2, const float4* tab, char* buf,
                                             double (&a)[NT][3]) {
  constexpr bool kOn = KIND == K_SL_ON || KIND == K_DL_ON;
  bool far[NT], any_far = kOn, any_near = false;
  for (int k = 0; k < NT; k++) {
    far[k] = act[k] && (kOn || !near[k]);
    if (!kOn) {
      any_far = any_far || __any_sync(0xffffffffu, far[k]);
      any_near = any_near || __any_sync(0xffffffffu, act[k] && near[k]);
    }
  }
  float* tile = reinterpret_cast<float*>(buf + (kOn ? 0 : kBufB + kNearB));
  double* wsm = reinterpret_cast<double*>(buf);
  float4* ws4 = reinterpret_cast<float4*>(buf + kBufB);
  for (int b = 0; b < n; b += kTile) {
    const int cnt = min(kTile, n - b);
    __syncwarp();
    if (any_far) stage_pairs<KIND>(T, s0 + b, cnt, cb, tile);
    if constexpr (!kOn)
      if (any_near) stage_near(T, s0 + b, cnt, cb, wsm, ws4);
    __syncwarp();
    if (any_far) tile_pairs<KIND, NT>(tile, cnt, F, far, inv_d2, tab, a);
    if constexpr (!kOn) {
#pragma unroll
      for (int k = 0; k < NT; k++)
        if (__any_sync(0xffffffffu, act[k] && near[k])) {
          const double3 v = tile_near<KIND>(T, t[k], act[k] && near[k], cnt, make_double3(cb[0], cb[1], cb[2]), wsm, ws4,
                                            make_double3(a[k][0], a[k][1], a[k][2]));
          a[k][0] = v.x;
          a[k][1] = v.y;
          a[k][2] = v.z;
        }
    }
  }
  __syncwarp();
}

// One unit: half h (64 targets, two per lane: lane and lane + 32) of an item's
// target block, all its segments in order.
template <int KIND>
__device__ __forceinline__ void run_unit(const EvalTask& T, const BlockRef& it, int h, const Seg* __restrict__ segs,
                                         const float4* tab, char* buf, float* cheb) {
  constexpr bool kOn = KIND == K_SL_ON || KIND == K_DL_ON, DL = KIND == K_DL_ON || KIND == K_DL_OFF;
  const int lane = threadIdx.x & 31;
  const int k0 = it.blk * kTB + h * 64 + lane;
  const bool valid[2] = {k0 < T.nt, k0 + 32 < T.nt};
  if (!__any_sync(0xffffffffu, valid[0])) return;  // the block's tail: no slot of these targets is read
  // origin of the FP32 coordinates: the block's first target (the sources a
  // block meets lie within a few leaf sizes of it, so FP32 offsets stay small)
  double cb[3];
  {
    const int t0 = T.tord[it.blk * kTB];
    cb[0] = T.txyz[3 * t0];
    cb[1] = T.txyz[3 * t0 + 1];
    cb[2] = T.txyz[3 * t0 + 2];
  }
  Tgt2 F[2];
  int t[2];
  bool near[2];
  double a[2][3];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    t[k] = valid[k] ? T.tord[k0 + 32 * k] : 0;
    Tgt S;
    Tgt32 f;
    load_target<KIND>(T, t[k], valid[k], cb, S, f);
    near[k] = !kOn && S.near != 0;
    F[k] = {f.px, f.py, f.pz, DL ? -f.g0[0] : -f.f0n0, DL ? -f.g0[1] : 0.f, DL ? -f.g0[2] : 0.f};
    for (int c = 0; c < 3; c++) a[k][c] = 0.0;
  }
  const f2 inv_d2 = dup<f2>((float)make_reg(T.DEL).inv_d2);
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
    unsigned live = __ballot_sync(0xffffffffu, (w0 | w1) != 0u);
    while (live) {
      const int l = __ffs(live) - 1;
      live &= live - 1;
      const uint32_t m0 = __shfl_sync(0xffffffffu, w0, l), m1 = __shfl_sync(0xffffffffu, w1, l);
      const int ty = __shfl_sync(0xffffffffu, type, l), nd = __shfl_sync(0xffffffffu, node, l);
      const int s0 = __shfl_sync(0xffffffffu, sg.s0, l), n = __shfl_sync(0xffffffffu, sg.s1, l) - s0;
      const bool act[2] = {valid[0] && ((m0 >> lane) & 1u), valid[1] && ((m1 >> lane) & 1u)};
      if (m0 != 0u && m1 != 0u) {
        if (ty == 1) {
          near_segment<KIND, 2>(T, s0, n, F, t, act, near, cb, inv_d2, tab, buf, a);
        } else if (kOn) {  // a node's rows are summed by themselves
          double p[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
          far_node<DL, kOn, 2>(T, nd, F, act, cb, buf, cheb, p);
          for (int k = 0; k < 2; k++)
            if (act[k])
              for (int c = 0; c < 3; c++) a[k][c] += p[k][c];
        } else {
          far_node<DL, kOn, 2>(T, nd, F, act, cb, buf, cheb, a);
        }
      } else {  // one target per lane
        const int k = m0 != 0u ? 0 : 1;
        const Tgt2 F1[1] = {k == 0 ? F[0] : F[1]};
        const int t1[1] = {k == 0 ? t[0] : t[1]};
        const bool act1[1] = {k == 0 ? act[0] : act[1]}, near1[1] = {k == 0 ? near[0] : near[1]};
        double a1[1][3], p1[1][3] = {{0.0, 0.0, 0.0}};
        for (int c = 0; c < 3; c++) a1[0][c] = k == 0 ? a[0][c] : a[1][c];
        if (ty == 1) {
          near_segment<KIND, 1>(T, s0, n, F1, t1, act1, near1, cb, inv_d2, tab, buf, a1);
        } else if (kOn) {
          far_node<DL, kOn, 1>(T, nd, F1, act1, cb, buf, cheb, p1);
          if (act1[0])
            for (int c = 0; c < 3; c++) a1[0][c] += p1[0][c];
        } else {
          far_node<DL, kOn, 1>(T, nd, F1, act1, cb, buf, cheb, a1);
        }
        for (int c = 0; c < 3; c++) {
          a[0][c] = k == 0 ? a1[0][c] : a[0][c];
          a[1][c] = k == 1 ? a1[0][c] : a[1][c];
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    double2* o = reinterpret_cast<double2*>(T.partial + ((size_t)it.slot * kTB + h * 64 + 32 * k + lane) * kPartComps);
    o[0] = make_double2(a[k][0], a[k][1]);
    o[1] = make_double2(a[k][2], 0.0);
  }
}

template <int KIND>
struct Shape32 {
  static constexpr bool on = KIND == K_SL_ON || KIND == K_DL_ON;
  static constexpr int warps = 12;
  static constexpr int warp_b = kBufB + (on ? 0 : kNearB + kTileB) + kChebB;
  static constexpr int tab_b = !on ? 0 : (KIND == K_SL_ON ? 2 : 1) * 2 * kPieces32 * kRep32 * 16;
  static constexpr int smem = tab_b + warps * warp_b;
};

// A launch's items, one persistent CTA per SM: every warp takes units from a
// common counter (the first by position, the rest in the items' order of
// decreasing cost); a unit's sums go to its own slot.
template <int KIND>
__global__ void __launch_bounds__(Shape32<KIND>::warps * 32, 1)
    units_kernel(const EvalTask* __restrict__ tasks, const BlockRef* __restrict__ items,
                 const Seg* __restrict__ segs, unsigned nunits, unsigned* __restrict__ next) {
  using SH = Shape32<KIND>;
  extern __shared__ __align__(16) char smc[];
  float4* tab = reinterpret_cast<float4*>(smc);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  char* buf = smc + SH::tab_b + warp * SH::warp_b;
  float* cheb = reinterpret_cast<float*>(buf + SH::warp_b - kChebB);
  if constexpr (SH::on) {
    // the tables with the powers of 1/delta in the coefficients, eight copies
    // (all tasks of a batch share one delta)
    const Reg gs = make_reg(tasks[items[0].task].DEL);
    float* t32 = reinterpret_cast<float*>(tab);
    for (int i = threadIdx.x; i < kPieces32 * 8; i += blockDim.x) {
      const bool centre = (i & 7) == 0;
      for (int c = 0; c < kRep32; c++) {
        float* o = t32 + ((i >> 2) * kRep32 + c) * 4 + (i & 3);
        if (KIND == K_SL_ON) {
          o[0] = kSmooth32G1[i] * (centre ? 1.0f : (float)gs.inv_d);
          o[2 * kPieces32 * kRep32 * 4] = kSmooth32G2[i] * (centre ? 1.0f : (float)gs.inv_d3);
        } else {
          o[0] = kSmooth32G3[i] * (centre ? 1.0f : (float)gs.inv_d5);
        }
      }
    }
    __syncthreads();
    tab += lane & (kRep32 - 1);
  }
  for (unsigned u = warp * gridDim.x + blockIdx.x; u < nunits;) {
    unsigned nx = 0;
    if (lane == 0) nx = atomicAdd(next, 1u);  // returns while the unit runs
    const BlockRef it = items[u >> 1];
    run_unit<KIND>(tasks[it.task], it, u & 1, segs, tab, buf, cheb);
    u = __shfl_sync(0xffffffffu, nx, 0) + gridDim.x * SH::warps;
  }
}

template <int KIND>
void launch_units(const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems, unsigned* next,
                  int num_sms, cudaStream_t st) {
  if (nitems <= 0) return;
  static_assert(Shape32<KIND>::smem <= 227 * 1024, "the table and the buffers fit one CTA");
  // set on every launch: the attribute belongs to the current device's context
  cudaFuncSetAttribute(units_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape32<KIND>::smem);
  const unsigned nunits = 2u * (unsigned)nitems;
  const unsigned grid = nunits < (unsigned)num_sms ? nunits : (unsigned)num_sms;
  units_kernel<KIND><<<grid, Shape32<KIND>::warps * 32, Shape32<KIND>::smem, st>>>(d_tasks, d_items, d_segs, nunits, next);
}

// ------------------------------------------------- extend-to-grid sums

// One item of an extend-to-grid task.
template <int KIND>
__device__ __forceinline__ void run_item(const EvalTask& T, const BlockRef& it, const Seg* __restrict__ segs,
                                         double* sm, float4* s4) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blk = it.blk;
  const int k = blk * kTB + tid;
  const bool valid = k < T.nt;
  const int t = valid ? T.tord[k] : 0;
  // origin of the FP32 coordinates: the block's first target (the sources a
  // block meets lie within a few leaf sizes of it, so FP32 offsets stay small)
  double cb[3];
  {
    const int t0 = T.tord[blk * kTB];
    cb[0] = T.txyz[3 * t0];
    cb[1] = T.txyz[3 * t0 + 1];
    cb[2] = T.txyz[3 * t0 + 2];
  }
  Tgt S;
  Tgt32 F;
  load_target<KIND>(T, t, valid, cb, S, F);
  const Reg g = make_reg(T.DEL);
  RegF gf;
  gf.inv_d = (float)g.inv_d;
  gf.d64 = (float)g.d64;
  // FP64 below, FP32 above: (3 delta)^2 in the mixed mode; in the all-FP32 mode
  // only the r < 1e-14 limits of the reference stay in FP64
  const float cut2f = T.mixed == 2 ? 1e-28f : (float)(9.0 * T.DEL * T.DEL);
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;  // a3: the pressure of the extend-to-grid sums
  constexpr bool kFace = KIND == K_E2G_UP_AWAY;
  constexpr bool kSrcNrm = !kFace;
  // Each warp walks the item's segments on its own: its own source tiles in
  // shared memory, __syncwarp only, and an entry whose mask is zero for this
  // warp is skipped outright.
  double* wsm = sm + warp * kWarpSm;
  float4* ws4 = s4 + warp * 3 * kNT;
  for (int q = it.seg0; q < it.seg1; q++) {
    const Seg sg = segs[q];
    const Entry E = T.entries[sg.entry];
    const uint32_t wm = E.mask[warp];
    if (wm == 0u) continue;
    const bool act = valid && ((wm >> lane) & 1u);
    if (E.type == 1) {
      const int m0 = sg.s0, m1 = sg.s1 - 1;
      for (int s0 = m0; s0 <= m1; s0 += kNT) {
        const int cnt = min(kNT, m1 - s0 + 1);
        __syncwarp();
        for (int i = lane; i < cnt; i += 32) {
          const int s = s0 + i;
          const double x = T.sx[s], y = T.sy[s], z = T.sz[s];
          double2* w2 = reinterpret_cast<double2*>(wsm) + 5 * i;
          w2[0] = make_double2(x, y);
          w2[1] = make_double2(z, T.sa[s]);
          w2[2] = kSrcNrm ? make_double2(T.snx[s], T.sny[s]) : make_double2(0.0, 0.0);
          w2[3] = make_double2(kSrcNrm ? T.snz[s] : 0.0, T.qx[s]);
          w2[4] = make_double2(T.qy[s], T.qz[s]);
          ws4[i] = make_float4((float)(x - cb[0]), (float)(y - cb[1]), (float)(z - cb[2]), T.fa[s]);
          if (kSrcNrm) ws4[kNT + i] = make_float4(T.fnx[s], T.fny[s], T.fnz[s], 0.f);
          ws4[2 * kNT + i] = make_float4(T.fqx[s], T.fqy[s], T.fqz[s], 0.f);
        }
        __syncwarp();
        if (!act) continue;
        if constexpr (kFace) {
          for (int j0 = 0; j0 < cnt; j0 += 16) {
            float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
            const int j1 = min(cnt, j0 + 16);
            if (j1 - j0 == 16) {
#pragma unroll 4
              for (int j = j0; j < j0 + 16; j++) pair32_face(ws4, j, F, p0, p1, p2, p3);
            } else {
              for (int j = j0; j < j1; j++) pair32_face(ws4, j, F, p0, p1, p2, p3);
            }
            a0 += (double)p0;
            a1 += (double)p1;
            a2 += (double)p2;
            a3 += (double)p3;
          }
        } else {
          for (int j0 = 0; j0 < cnt; j0 += 16) {
            float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f;
            const int j1 = min(cnt, j0 + 16);
#pragma unroll 2
            for (int j = j0; j < j1; j++) {
              const float4 Pj = ws4[j];
              const float dx = F.px - Pj.x, dy = F.py - Pj.y, dz = F.pz - Pj.z;
              if (dx * dx + dy * dy + dz * dz > cut2f) pair32r_band(ws4, j, F, gf, p0, p1, p2, p3);
              else pair64_band(wsm, j, S, g, a0, a1, a2, a3);
            }
            a0 += (double)p0;
            a1 += (double)p1;
            a2 += (double)p2;
            a3 += (double)p3;
          }
        }
      }
    }
  }
  // partial sums of this item
  double* o = T.partial + ((size_t)it.slot * kTB + tid) * kPartComps;
  o[0] = a0;
  o[1] = a1;
  o[2] = a2;
  o[3] = a3;
}

// The extend-to-grid items, a CTA each. FACE: the box-face sums, whose code
// path needs fewer registers (no nearest-point data, no per-target
// coefficients), six CTAs per SM; the band's four.
template <bool FACE>
__global__ void __launch_bounds__(kTB, FACE ? 6 : 4)
    eval_kernel_e2g(const EvalTask* __restrict__ tasks, const BlockRef* __restrict__ items,
                    const Seg* __restrict__ segs) {
  __shared__ __align__(16) double sm[kSmem];
  // per-warp FP32 source tiles: (x, y, z, area), (n, 0), (q, 0) per source
  __shared__ float4 sf[kWarps * 3 * kNT];
  __shared__ EvalTask sT;
  const BlockRef it = items[blockIdx.x];
  if (threadIdx.x == 0) sT = tasks[it.task];
  __syncthreads();
  run_item<FACE ? K_E2G_UP_AWAY : K_E2G_UP7>(sT, it, segs, sm, sf);
}

// Sums a target block's item partials (kSplit consecutive runs of slots, each in
// slot order, then the runs in order) and applies the reference drivers'
// per-target epilogue (scale and jump terms). A block has tens of slots and
// there are few blocks, so what bounds this is the loads' latency: kSplit
// threads per target with eight slots in flight each (solve at h = 1/32 with 1 /
// 2 / 4 / 8: 11.91 / 11.85 / 11.82 / 11.83 ms).
constexpr int kSplit = 4;
__global__ void __launch_bounds__(kSplit* kTB) reduce_kernel(const EvalTask* __restrict__ tasks,
                                                            const int2* __restrict__ task_blocks,
                                                            unsigned* __restrict__ next) {
  __shared__ double2 part[(kSplit - 1) * 2 * kTB];
  if (blockIdx.x == 0 && threadIdx.x < 2) next[threadIdx.x] = 0u;
  const int2 tb = task_blocks[blockIdx.x];  // (task, block)
  const EvalTask& T = tasks[tb.x];
  const int blk = tb.y, tid = threadIdx.x & (kTB - 1), run = threadIdx.x / kTB;
  const int k = blk * kTB + tid;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  if (k < T.nt) {
    const int b0 = T.item_start[blk], n = T.item_start[blk + 1] - b0;
    const int s0 = b0 + n * run / kSplit, s1 = b0 + n * (run + 1) / kSplit;
#pragma unroll 8
    for (int s = s0; s < s1; s++) {
      const double2* p = reinterpret_cast<const double2*>(T.partial + ((size_t)s * kTB + tid) * kPartComps);
      const double2 u = p[0], v = p[1];
      a0 += u.x;
      a1 += u.y;
      a2 += v.x;
      a3 += v.y;
    }
  }
  if (run > 0) {
    part[(2 * run - 2) * kTB + tid] = make_double2(a0, a1);
    part[(2 * run - 1) * kTB + tid] = make_double2(a2, a3);
  }
  __syncthreads();
  if (run > 0 || k >= T.nt) return;
#pragma unroll
  for (int r = 0; r < kSplit - 1; r++) {
    const double2 u = part[2 * r * kTB + tid], v = part[(2 * r + 1) * kTB + tid];
    a0 += u.x;
    a1 += u.y;
    a2 += v.x;
    a3 += v.y;
  }
  const int t = T.tord[k];
  const double sc = T.scale;
  double* o = T.out;
  const int kind = T.kind;
  if (kind == K_SL_ON || kind == K_SL_OFF || kind == K_E2G_SL_AWAY || kind == K_E2G_SL7) {
    o[3 * t] = a0 * sc;
    o[3 * t + 1] = a1 * sc;
    o[3 * t + 2] = a2 * sc;
  } else if (kind == K_E2G_UP_AWAY) {
    o[3 * t] = a0 * sc;
    o[3 * t + 1] = a1 * sc;
    o[3 * t + 2] = a2 * sc;
    T.out2[t] = a3 * T.scale2;
  } else if (kind == K_E2G_UP7) {
    o[3 * t] = a0 * sc;
    o[3 * t + 1] = a1 * sc;
    o[3 * t + 2] = a2 * sc;
    // p *= -denom_FourPI (scale2); inside: p -= f0.n0 (E2G/stokes.cpp:196-200)
    double p = a3 * T.scale2;
    if (T.tb[t] < -1.e-12) {
      const double* f0 = T.tf0 + 3 * t;
      const double* n0 = T.tn0 + 3 * t;
      p -= f0[0] * n0[0] + f0[1] * n0[1] + f0[2] * n0[2];
    }
    T.out2[t] = p;
  } else if (kind == K_DL_ON) {
    // DL[3i+k] = u[k] * EightPI6 + 0.5 * g0[k]   (2S/KITC.cpp:1693, 2S/stresslets.cpp:271-278)
    const double* g0 = T.tq + 3 * t;
    o[3 * t] = a0 * sc + 0.5 * g0[0];
    o[3 * t + 1] = a1 * sc + 0.5 * g0[1];
    o[3 * t + 2] = a2 * sc + 0.5 * g0[2];
  } else if (kind == K_DL_OFF) {
    const double b = T.tb[t];
    const double* g0 = T.tg0 + 3 * t;
    double xi = 0.0;
    if (T.jump_mode == 0) {
      // tree: xi = 1/2 on the surface, 1 inside (2S/KITC.cpp:1805-1815)
      if (fabs(b) < 1.0e-12) xi = 0.5;
      else if (b < 0.0) xi = 1.0;
    } else {
      // direct: + g0 inside or on the surface, near targets only (2S/stresslets.cpp:174-178)
      if (T.tnear[t] && ((b < 0.0) || (fabs(b) < 1.0e-14))) xi = 1.0;
    }
    o[3 * t] = a0 * sc + xi * g0[0];
    o[3 * t + 1] = a1 * sc + xi * g0[1];
    o[3 * t + 2] = a2 * sc + xi * g0[2];
  } else if (kind == K_E2G_P_AWAY) {
    o[t] = a0 * sc;
  } else {
    // p *= -denom_FourPI; inside: p -= f0.n0 (E2G/stokes.cpp:196-200)
    double p = a0 * sc;
    if (T.tb[t] < -1.e-12) {
      const double* f0 = T.tf0 + 3 * t;
      const double* n0 = T.tn0 + 3 * t;
      p -= f0[0] * n0[0] + f0[1] * n0[1] + f0[2] * n0[2];
    }
    o[t] = p;
  }
}

}  // namespace

void launch_eval(int family, const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems, int n_on,
                 unsigned* next, int num_sms, cudaStream_t st, cudaStream_t side) {
  const int n_off = nitems - n_on;
  const BlockRef* off = d_items + n_on;
  // the off-surface items first: their units' times differ most (near targets),
  // and the other launch fills their tail (operator at h = 1/32 0.735 -> 0.665 ms,
  // h = 1/24 0.42 -> 0.39)
  if (family == F_SL) {
    launch_units<K_SL_OFF>(d_tasks, off, d_segs, n_off, next + 1, num_sms, st);
    launch_units<K_SL_ON>(d_tasks, d_items, d_segs, n_on, next, num_sms, side);
  } else if (family == F_DL) {
    launch_units<K_DL_OFF>(d_tasks, off, d_segs, n_off, next + 1, num_sms, st);
    launch_units<K_DL_ON>(d_tasks, d_items, d_segs, n_on, next, num_sms, side);
  } else {
    if (n_on > 0) eval_kernel_e2g<true><<<n_on, kTB, 0, st>>>(d_tasks, d_items, d_segs);
    if (n_off > 0) eval_kernel_e2g<false><<<n_off, kTB, 0, side>>>(d_tasks, off, d_segs);
  }
}

void launch_reduce(const EvalTask* d_tasks, int ntask_blocks, const int2* d_task_blocks, unsigned* next,
                   cudaStream_t st) {
  if (ntask_blocks > 0) reduce_kernel<<<ntask_blocks, kSplit * kTB, 0, st>>>(d_tasks, d_task_blocks, next);
}

}  // namespace hr
