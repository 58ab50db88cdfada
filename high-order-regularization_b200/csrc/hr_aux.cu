// hr_aux.cu — upward pass, density interpolation, permutations, combines and
// the deterministic vector kernels used by GMRES.
#include <algorithm>

#include "hr_device.h"
#include "hr_pairs.cuh"

namespace hr {

namespace {

// Upward pass: the barycentric Lagrange proxy moments of Panel_Moments_SL /
// Panel_Moments_DL (2S/KITC.cpp:351-668) of one (node, source range) item,
//   M[c][ijk] = sum_s L_i(x_s) L_j(y_s) L_k(z_s) A_s q_c(s),
//   L_i(x) = (w_i / (x - t_i)) / sum_m (w_m / (x - t_m)),  w_j = (-1)^j d_j,
// with the removable singularity |x - t_j| < 1e-7 handled as in the reference.
// SL channels: f (3), n (3). DL channels: the combinations that the far field
// reads (moments_reduce_kernel): the six of the symmetric part of g (x) n, n (3).
//
// It is a contraction, D[(j,k), (c,i)] = sum_s (L_j L_k)(s) (L_i A q_c)(s), and
// runs on the FP64 matrix instruction (mma m8n8k4): the same 16 multiply-adds
// per cycle and SM quarter as the FP64 pipe's peak, but with one operand
// fetch per 8 of them, where the scalar form (one thread per proxy, 5 operands
// from shared memory per source and channel) was bound by shared-memory reads.
// A warp owns 4 x 4 tiles of 8 x 8 (8 fragment loads per 16 MMAs, no test per
// tile: rows and columns are padded with zero fragments to whole groups); a
// CTA, up to 8 warps, shares the operands of 32 sources at a time, written
// fragment by fragment (32 consecutive doubles, no bank conflicts). More tiles
// than 8 warps hold (P > 7) go to further CTAs of the item, so that several
// CTAs per SM overlap one another's operand and MMA phases.
// Both surfaces at h = 1/64, P = 6: 220 -> 78 us (stresslet; two launches of 110 us
// before), the operator application 4.07 -> 3.93 ms; P = 10: the work around the
// boundary sums 0.96 -> 0.41 ms. 8 x 2 tiles per warp and one CTA of 14 warps per
// item measured the same (77 / 306 us): the operand phase between the MMAs bounds
// it now.
constexpr int kMomSrc = 32, kMomRT = 4, kMomCT = 4, kMomWarps = 8;

struct MomShape {
  int P1, nrt, nct;  // row and column tiles, in whole groups
  int jobs;          // warp jobs: row groups x column groups
  int warps;         // per CTA
  int ctas;          // per item
  int smem;          // bytes
};

MomShape mom_shape(int C, int P1) {
  MomShape m;
  m.P1 = P1;
  m.nrt = ((P1 * P1 + 7) / 8 + kMomRT - 1) / kMomRT * kMomRT;
  m.nct = ((C * P1 + 7) / 8 + kMomCT - 1) / kMomCT * kMomCT;
  m.jobs = (m.nrt / kMomRT) * (m.nct / kMomCT);
  m.ctas = (m.jobs + kMomWarps - 1) / kMomWarps;
  m.warps = (m.jobs + m.ctas - 1) / m.ctas;
  m.smem = (int)sizeof(double) * (kMomSrc * 8 * (m.nrt + m.nct) + 3 * P1 * (kMomSrc + 1) + C * kMomSrc + 3 * P1);
  return m;
}

__device__ __forceinline__ void mma_f64(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

template <int C>
__global__ void __launch_bounds__(kMomWarps * 32) moments_kernel(MomTree t0, MomTree t1, MomShape sh) {
  constexpr bool DL = C == 9;
  extern __shared__ __align__(16) double msm[];
  const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
  const int P1 = sh.P1, M2 = P1 * P1, Pf = M2 * P1;
  double* sA = msm;                                   // [source quad][row tile][32]
  double* sB = sA + kMomSrc * 8 * sh.nrt;             // [source quad][column tile][32]
  double* sL = sB + kMomSrc * 8 * sh.nct;             // [axis][P1][kMomSrc + 1]
  double* sQ = sL + 3 * P1 * (kMomSrc + 1);           // [C][kMomSrc]
  double* sT = sQ + C * kMomSrc;                      // Chebyshev points
  const bool first = (int)blockIdx.x < t0.nitems;
  const MomTree& t = first ? t0 : t1;
  const MomItem it = t.items[first ? blockIdx.x : blockIdx.x - t0.nitems];
  for (int i = tid; i < 3 * P1; i += nthr) sT[i] = t.tcheb[(size_t)it.node * 3 * P1 + i];
  const int nrg = sh.nrt / kMomRT;
  const int job = blockIdx.y * sh.warps + warp;
  const bool has_job = job < sh.jobs;
  const int rt0 = (job % nrg) * kMomRT, ct0 = (job / nrg) * kMomCT;
  double acc[kMomRT][kMomCT][2];
#pragma unroll
  for (int r = 0; r < kMomRT; r++)
#pragma unroll
    for (int c = 0; c < kMomCT; c++) acc[r][c][0] = acc[r][c][1] = 0.0;
  __syncthreads();
  for (int s0 = it.s0; s0 < it.s1; s0 += kMomSrc) {
    const int cnt = min(kMomSrc, it.s1 - s0);
    // the Lagrange values of one (axis, source) per thread, normalized by
    // their own axis sum; then the channels of a source per thread. Beyond the
    // last source both are zero.
    for (int e = tid; e < 4 * kMomSrc; e += nthr) {
      const int ax = e / kMomSrc, src = e - ax * kMomSrc, s = s0 + src;
      if (ax < 3) {
        double* L = sL + (ax * P1) * (kMomSrc + 1) + src;
        if (src < cnt) {
          const double pc = ax == 0 ? t.x[s] : (ax == 1 ? t.y[s] : t.z[s]);
          int flag = -1;
          double S = 0.0;
          for (int jj = 0; jj < P1; jj++) {
            // barycentric weights w_j = (-1)^j d_j, d_0 = d_P = 1/2 (2S/KITC.cpp:365-375)
            const double w = ((jj % 2 == 0) ? 1.0 : -1.0) * ((jj == 0 || jj == P1 - 1) ? 0.5 : 1.0);
            const double d = pc - sT[ax * P1 + jj];
            double v = 0.0;
            if (fabs(d) < 1.e-07) {
              flag = jj;
            } else {
              v = w / d;
              S += v;
            }
            L[jj * (kMomSrc + 1)] = v;
          }
          const double inv = 1.0 / S;
          for (int jj = 0; jj < P1; jj++)
            L[jj * (kMomSrc + 1)] = (flag > -1) ? (jj == flag ? 1.0 : 0.0) : L[jj * (kMomSrc + 1)] * inv;
        } else {
          for (int jj = 0; jj < P1; jj++) L[jj * (kMomSrc + 1)] = 0.0;
        }
      } else {
        double v[C];
#pragma unroll
        for (int c = 0; c < C; c++) v[c] = 0.0;
        if (src < cnt) {
          const double A = t.a[s], n0 = A * t.nx[s], n1 = A * t.ny[s], n2 = A * t.nz[s];
          const double q0 = t.qx[s], q1 = t.qy[s], q2 = t.qz[s];
          if (DL) {
            v[0] = q0 * n0;
            v[1] = q1 * n1;
            v[2] = q2 * n2;
            v[3] = q0 * n1 + q1 * n0;
            v[4] = q0 * n2 + q2 * n0;
            v[5] = q1 * n2 + q2 * n1;
          } else {
            v[0] = A * q0;
            v[1] = A * q1;
            v[2] = A * q2;
          }
          v[C - 3] = n0;
          v[C - 2] = n1;
          v[C - 1] = n2;
        }
#pragma unroll
        for (int c = 0; c < C; c++) sQ[c * kMomSrc + src] = v[c];
      }
    }
    __syncthreads();
    // operand fragments (a row or column tile at a time per warp): lane l of a
    // fragment is row (column) l / 4, source l mod 4 of its quad
    for (int f = warp; f < sh.nrt + sh.nct; f += nthr / 32) {
      const bool rows = f < sh.nrt;
      const int tile = rows ? f : f - sh.nrt, n = rows ? sh.nrt : sh.nct, at = tile * 8 + (lane >> 2);
      const double *u = nullptr, *v = nullptr;  // the two factors, per source
      if (rows && at < M2) {
        const int j = at / P1, k = at - j * P1;
        u = sL + (P1 + j) * (kMomSrc + 1);
        v = sL + (2 * P1 + k) * (kMomSrc + 1);
      } else if (!rows && at < C * P1) {
        const int c = at / P1, i = at - c * P1;
        u = sL + i * (kMomSrc + 1);
        v = sQ + c * kMomSrc;
      }
      double* o = (rows ? sA : sB) + tile * 32 + lane;
#pragma unroll
      for (int q = 0; q < kMomSrc / 4; q++) {
        const int src = 4 * q + (lane & 3);
        o[q * n * 32] = u ? u[src] * v[src] : 0.0;
      }
    }
    __syncthreads();
    if (has_job) {
      const int nq = (cnt + 3) / 4;
      const double *pa = sA + rt0 * 32 + lane, *pb = sB + ct0 * 32 + lane;
#pragma unroll 2
      for (int q = 0; q < nq; q++) {
        double fa[kMomRT], fb[kMomCT];
#pragma unroll
        for (int r = 0; r < kMomRT; r++) fa[r] = pa[(q * sh.nrt + r) * 32];
#pragma unroll
        for (int c = 0; c < kMomCT; c++) fb[c] = pb[(q * sh.nct + c) * 32];
#pragma unroll
        for (int r = 0; r < kMomRT; r++)
#pragma unroll
          for (int c = 0; c < kMomCT; c++) mma_f64(acc[r][c], fa[r], fb[c]);
      }
    }
    __syncthreads();
  }
  if (!has_job) return;
  // accumulator of a lane: row l / 4, columns 2 (l mod 4) and the next
#pragma unroll
  for (int r = 0; r < kMomRT; r++) {
    const int row = (rt0 + r) * 8 + (lane >> 2);
#pragma unroll
    for (int c = 0; c < kMomCT; c++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int col = (ct0 + c) * 8 + 2 * (lane & 3) + h;
        if (row < M2 && col < C * P1) {
          const int ch = col / P1, i = col - ch * P1;
          t.partial[((size_t)it.out * C + ch) * Pf + (size_t)i * M2 + row] = acc[r][c][h];
        }
      }
  }
}

// Sums the partial moments of each node in item order (deterministic) and
// stores them proxy-major. The stresslet's channels (g (x) n) enter the far
// field only through
//   d.M.d = M00 d0^2 + M11 d1^2 + M22 d2^2 + (M01 + M10) d0 d1
//         + (M02 + M20) d0 d2 + (M12 + M21) d1 d2   and   Mn.d,
// so they are stored as those 6 symmetric combinations and Mn: FP64 10
// doubles per proxy (the last one zero), FP32 as momf_stride says.
// The FP64 upward pass gives the combinations (C = 9), the tensor-core one the
// 12 products g-major, then n (C = 12). The Stokeslet's 6 channels (f, n) are
// stored as they are: FP64 6 doubles, FP32 likewise in pairs.
__global__ void moments_reduce_kernel(int C, int P1, int Pf, MomTree t0, MomTree t1) {
  // one thread per (node, proxy, stored value): a value is one channel, or of
  // 12 channels the sum of two, each summed over the node's items in item order
  const bool first = (int)blockIdx.x < t0.nn;
  const MomTree& t = first ? t0 : t1;
  const int node = first ? blockIdx.x : blockIdx.x - t0.nn, o = blockIdx.z;
  const int kk = blockIdx.y * blockDim.x + threadIdx.x;
  if (kk >= Pf) return;
  const bool dl = C != 6;
  int c0 = o < C ? o : -1, c1 = -1;
  if (C == 12) {
    const int first_c[10] = {0, 4, 8, 1, 2, 5, 9, 10, 11, -1};
    const int second_c[10] = {-1, -1, -1, 3, 6, 7, -1, -1, -1, -1};
    c0 = first_c[o];
    c1 = second_c[o];
  }
  const int a = t.item_start[node], b = t.item_start[node + 1];
  double s0 = 0.0, s1 = 0.0;
  if (c0 >= 0) {
#pragma unroll 8
    for (int q = a; q < b; q++) s0 += t.partial[((size_t)q * C + c0) * Pf + kk];
  }
  if (c1 >= 0) {
#pragma unroll 8
    for (int q = a; q < b; q++) s1 += t.partial[((size_t)q * C + c1) * Pf + kk];
  }
  const double v = c1 >= 0 ? s0 + s1 : s0;
  const size_t k = (size_t)node * Pf + kk;
  const int row = kk / P1, pk = kk - row * P1, pair = row * ((P1 + 1) / 2) + pk / 2, half = pk & 1;
  if (dl) {
    t.mom[k * 10 + o] = v;  // o = 9: the zero pad
    if (o < 9) t.momf[node * momf_stride(P1, 20) + (size_t)pair * 20 + 2 * o + half] = (float)v;
  } else {
    t.mom[k * 6 + o] = v;
    t.momf[node * momf_stride(P1, 12) + (size_t)pair * 12 + 2 * o + half] = (float)v;
  }
}

__global__ void permute_kernel(PermTree t0, PermTree t1, int pack) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool first = p < t0.n;
  const PermTree& t = first ? t0 : t1;
  if (!first) p -= t0.n;
  if (p >= t.n) return;
  const int o = t.perm[p];
  const double a = t.q3[3 * o], b = t.q3[3 * o + 1], c = t.q3[3 * o + 2];
  t.qx[p] = a;
  t.qy[p] = b;
  t.qz[p] = c;
  if (t.fqx) {
    t.fqx[p] = (float)a;
    t.fqy[p] = (float)b;
    t.fqz[p] = (float)c;
  }
  if (!t.pk) return;
  const double w = t.a[p], u = t.nx[p], v = t.ny[p], z = t.nz[p];
  double2* r = reinterpret_cast<double2*>(t.pk);
  if (pack == PACK_E2G) {
    r += 6 * (size_t)p;
    r[0] = make_double2(t.x[p], t.y[p]);
    r[1] = make_double2(t.z[p], w);
    r[2] = make_double2(a, b);
    r[3] = make_double2(c, u * u + v * v + z * z);
    r[4] = make_double2(u, v);
    r[5] = make_double2(z, 0.0);
  } else {
    const double wq = pack == PACK_SL ? w : 1.0;
    r += 5 * (size_t)p;
    r[0] = make_double2(t.x[p], t.y[p]);
    r[1] = make_double2(t.z[p], w);
    r[2] = make_double2(w * u, w * v);
    r[3] = make_double2(w * z, wq * a);
    r[4] = make_double2(wq * b, wq * c);
  }
}

// sixPoint_coeff (2S/main.cpp:750-757)
__device__ __forceinline__ void six_coeff(double p, double c[6]) {
  c[0] = -p * (p * p - 1.0) * (p - 2.0) * (p - 3.0) / 120.0;
  c[1] = p * (p - 1.0) * (p * p - 4.0) * (p - 3.0) / 24.0;
  c[2] = -(p * p - 1.0) * (p * p - 4.0) * (p - 3.0) / 12.0;
  c[3] = p * (p + 1.0) * (p * p - 4.0) * (p - 3.0) / 12.0;
  c[4] = -p * (p * p - 1.0) * (p + 2.0) * (p - 3.0) / 24.0;
  c[5] = p * (p * p - 1.0) * (p * p - 4.0) / 120.0;
}

// sixPointInterpolate over the precomputed stencil (2S/main.cpp:759-778,
// 1019-1039), one thread per entry and component.
__global__ void interp_kernel(InterpSet s0, InterpSet s1) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  const bool first = e < 3 * s0.ne;
  const InterpSet& S = first ? s0 : s1;
  if (!first) e -= 3 * s0.ne;
  if (e >= 3 * S.ne) return;
  const int comp = e % 3;
  e /= 3;
  double a[6], b[6];
  six_coeff(S.pq[2 * e], a);
  six_coeff(S.pq[2 * e + 1], b);
  const int* st = S.idx + 36 * (size_t)e;
  double ft[6];
#pragma unroll
  for (int jj = 0; jj < 6; jj++) {
    double s = 0.0;
#pragma unroll
    for (int ii = 0; ii < 6; ii++) s += a[ii] * S.g[3 * st[6 * ii + jj] + comp];
    ft[jj] = s;
  }
  double v = 0.0;
#pragma unroll
  for (int jj = 0; jj < 6; jj++) v += b[jj] * ft[jj];
  S.g0[3 * S.tgt[e] + comp] = v;
}

// u_out = u_in - on*factor; u_out -= comp*factor   (2S/main.cpp:612-676), both
// target sets (set 1 subtracts comp first: its a is comp, its b is on)
__global__ void matvec_combine_kernel(CombineSet s0, CombineSet s1, double factor, const double* __restrict__ x,
                                      double* __restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s0.n + s1.n) return;
  const CombineSet& S = i < s0.n ? s0 : s1;
  const int k = i < s0.n ? i : i - s0.n;
  double v = x[i] - S.a[k] * factor;
  v -= S.b[k] * factor;
  y[i] = v;
}

// SL = a; SL += b; rhs = -SL * factor   (2S/main.cpp:202-207, 478-536)
__global__ void rhs_combine_kernel(CombineSet s0, CombineSet s1, double factor, double* __restrict__ b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= s0.n + s1.n) return;
  const CombineSet& S = i < s0.n ? s0 : s1;
  const int k = i < s0.n ? i : i - s0.n;
  double s = S.a[k];
  s += S.b[k];
  b[i] = -s * factor;
}

constexpr int kDotThreads = 256;
constexpr int kMaxCols = 64;

// One Gram-Schmidt pass: (kSub) w -= sum_c coef[c] V[c] first, then out[c] = U[c] .
// w for ncols columns (U = V, or the norm's U = w). A thread updates and reads
// the same elements of w. The blocks' partial sums are added by the last block
// to finish: one warp per column, lane l the blocks l, l + 32, ... in order,
// then a fixed shuffle tree (deterministic). One launch instead of three of
// ~3 us each around microseconds of work.
template <bool kSub>
__global__ void __launch_bounds__(kDotThreads) dots_kernel(int n, int nsub, const double* V, long ldv,
                                                           const double* __restrict__ coef, double* w, int ncols,
                                                           const double* U, double* __restrict__ partial,
                                                           unsigned* __restrict__ done, double* __restrict__ out) {
  __shared__ double red[kDotThreads / 32][kMaxCols];
  __shared__ double sc[kMaxCols];
  __shared__ bool last;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if constexpr (kSub) {
    if (tid < nsub) sc[tid] = coef[tid];
    __syncthreads();
    for (int i = blockIdx.x * kDotThreads + tid; i < n; i += gridDim.x * kDotThreads) {
      double v = w[i];
      for (int c = 0; c < nsub; c++) v += -1.0 * sc[c] * V[(size_t)c * ldv + i];
      w[i] = v;
    }
  }
  for (int c0 = 0; c0 < ncols; c0 += 8) {
    double acc[8];
#pragma unroll
    for (int q = 0; q < 8; q++) acc[q] = 0.0;
    for (int i = blockIdx.x * kDotThreads + tid; i < n; i += gridDim.x * kDotThreads) {
      const double wi = w[i];
#pragma unroll
      for (int q = 0; q < 8; q++)
        if (c0 + q < ncols) acc[q] += U[(size_t)(c0 + q) * ldv + i] * wi;
    }
#pragma unroll
    for (int q = 0; q < 8; q++) {
      double v = acc[q];
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0 && c0 + q < ncols) red[warp][c0 + q] = v;
    }
  }
  __syncthreads();
  if (tid < ncols) {
    double s = 0.0;
    for (int wq = 0; wq < kDotThreads / 32; wq++) s += red[wq][tid];
    partial[(size_t)blockIdx.x * kMaxCols + tid] = s;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int c = warp; c < ncols; c += kDotThreads / 32) {
    double s = 0.0;
    for (unsigned b = lane; b < gridDim.x; b += 32) s += __ldcg(&partial[(size_t)b * kMaxCols + c]);
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if (lane == 0) out[c] = s;
  }
  if (tid == 0) *done = 0u;
}

// w += sign * sum_c coef[c] V[c]
__global__ void axpy_multi_kernel(int n, int ncols, const double* __restrict__ V, long ldv,
                                  const double* __restrict__ coef, double sign,
                                  double* __restrict__ w) {
  __shared__ double sc[kMaxCols];
  if (threadIdx.x < ncols) sc[threadIdx.x] = coef[threadIdx.x];
  __syncthreads();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double v = w[i];
    for (int c = 0; c < ncols; c++) v += sign * sc[c] * V[(size_t)c * ldv + i];
    w[i] = v;
  }
}

// w *= s, and a copy of the result
__global__ void scale_kernel(int n, double s, double* __restrict__ w, double* __restrict__ copy) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double v = w[i] * s;
    w[i] = v;
    copy[i] = v;
  }
}
__global__ void sub_kernel(int n, const double* __restrict__ a, const double* __restrict__ b,
                           double* __restrict__ o) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    o[i] = a[i] - b[i];
}
__global__ void copy_kernel(int n, const double* __restrict__ a, double* __restrict__ o) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) o[i] = a[i];
}

// FP64 FMA throughput loop: 8 independent chains per thread.
__global__ void fma_peak_kernel(double* out, int iters) {
  double a[8];
  for (int q = 0; q < 8; q++) a[q] = 1.0 + 1e-9 * (threadIdx.x + q);
  const double m = 0.999999999, c = 1e-12;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int q = 0; q < 8; q++) a[q] = fma(a[q], m, c);
  }
  double s = 0;
  for (int q = 0; q < 8; q++) s += a[q];
  if (s == 12345.678) out[0] = s;  // keeps the loop alive
}

// FP32 counterpart: 16 independent FMA chains per thread.
__global__ void fma_peak32_kernel(float* out, int iters) {
  float a[16];
  for (int q = 0; q < 16; q++) a[q] = 1.0f + 1e-6f * (threadIdx.x + q);
  const float m = 0.9999999f, c = 1e-7f;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int q = 0; q < 16; q++) a[q] = fmaf(a[q], m, c);
  }
  float s = 0;
  for (int q = 0; q < 16; q++) s += a[q];
  if (s == 12345.678f) out[0] = s;  // keeps the loop alive
}

inline int nblk(long n, int t) { return (int)std::min<long>((n + t - 1) / t, 148L * 16); }

}  // namespace

void launch_moments(int C, int P1, const MomTree& t0, const MomTree& t1, cudaStream_t st) {
  const int nitems = t0.nitems + t1.nitems;
  if (nitems <= 0) return;
  const MomShape m = mom_shape(C, P1);
  auto* fn = C == 9 ? moments_kernel<9> : moments_kernel<6>;
  allow_shared(fn);
  fn<<<dim3(nitems, m.ctas), m.warps * 32, m.smem, st>>>(t0, t1, m);
}

void launch_moments_reduce(int C, int P1, const MomTree& t0, const MomTree& t1, cudaStream_t st) {
  if (t0.nn + t1.nn <= 0) return;
  const int Pf = P1 * P1 * P1;
  dim3 grid(t0.nn + t1.nn, (Pf + 127) / 128, C == 6 ? 6 : 10);
  moments_reduce_kernel<<<grid, 128, 0, st>>>(C, P1, Pf, t0, t1);
}

void launch_permute(const PermTree& t0, const PermTree& t1, int pack, cudaStream_t st) {
  const int n = t0.n + t1.n;
  if (n <= 0) return;
  permute_kernel<<<(n + 255) / 256, 256, 0, st>>>(t0, t1, pack);
}

void launch_interp(const InterpSet& s0, const InterpSet& s1, cudaStream_t st) {
  const int n = 3 * (s0.ne + s1.ne);
  if (n <= 0) return;
  interp_kernel<<<(n + 127) / 128, 128, 0, st>>>(s0, s1);
}

void launch_matvec_combine(const CombineSet& s0, const CombineSet& s1, double factor, const double* x, double* y,
                           cudaStream_t st) {
  matvec_combine_kernel<<<(s0.n + s1.n + 255) / 256, 256, 0, st>>>(s0, s1, factor, x, y);
}

void launch_rhs_combine(const CombineSet& s0, const CombineSet& s1, double factor, double* b, cudaStream_t st) {
  rhs_combine_kernel<<<(s0.n + s1.n + 255) / 256, 256, 0, st>>>(s0, s1, factor, b);
}

void launch_dots(int n, int ncols, const double* U, long ldv, const double* w, const DotWork& d, double* out,
                 cudaStream_t st) {
  dots_kernel<false><<<kRedBlocks, kDotThreads, 0, st>>>(n, 0, nullptr, ldv, nullptr, const_cast<double*>(w), ncols, U,
                                                         d.partial, d.done, out);
}

void launch_sub_dots(int n, int nsub, const double* V, long ldv, const double* coef, double* w, int ncols,
                     const double* U, const DotWork& d, double* out, cudaStream_t st) {
  dots_kernel<true><<<kRedBlocks, kDotThreads, 0, st>>>(n, nsub, V, ldv, coef, w, ncols, U, d.partial, d.done, out);
}

void launch_axpy_multi(int n, int ncols, const double* V, long ldv, const double* coef,
                       double sign, double* w, cudaStream_t st) {
  axpy_multi_kernel<<<nblk(n, 256), 256, 0, st>>>(n, ncols, V, ldv, coef, sign, w);
}

void launch_scale_copy(int n, double s, double* w, double* copy, cudaStream_t st) {
  scale_kernel<<<nblk(n, 256), 256, 0, st>>>(n, s, w, copy);
}
void launch_sub(int n, const double* a, const double* b, double* out, cudaStream_t st) {
  sub_kernel<<<nblk(n, 256), 256, 0, st>>>(n, a, b, out);
}
void launch_copy(int n, const double* a, double* out, cudaStream_t st) {
  copy_kernel<<<nblk(n, 256), 256, 0, st>>>(n, a, out);
}

void launch_fma_peak(double* out, int iters, int blocks, cudaStream_t st) {
  fma_peak_kernel<<<blocks, 256, 0, st>>>(out, iters);
}

void launch_fma_peak32(float* out, int iters, int blocks, cudaStream_t st) {
  fma_peak32_kernel<<<blocks, 256, 0, st>>>(out, iters);
}

}  // namespace hr
