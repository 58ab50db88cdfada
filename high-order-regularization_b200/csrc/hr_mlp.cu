// hr_mlp.cu — the learned GMRES warm start: a pointwise MLP
// 12 -> 64 -> 64 -> 64 -> 3 with SiLU hidden activations and FP32 weights,
// trained on the GPU by these kernels (forward, backward, Adam) and applied by
// an inference kernel that writes an FP64 initial guess.
//
// Parameter layout (flat, 9347 floats): W1[12][64] b1[64] W2[64][64] b2[64]
// W3[64][64] b3[64] W4[64][3] b4[3]; W[i][j] is the weight from input i to
// output j. Inputs are normalized in the kernels: x' = (x - mean) / std; the
// output is scaled by out_scale.
//
// Kernels:
//   train_kernel     forward, loss, backward and the partial parameter gradient
//                    of a tile of 128 samples per CTA, everything between the
//                    samples' inputs and the gradient in shared memory and
//                    registers (below).
//   grad_adam_kernel sums the tiles' partial gradients in tile order
//                    (deterministic) and takes the Adam step with bias
//                    correction (Kingma & Ba 2015).
//   infer_kernel     guess = base + out_scale * MLP(x), FP64 out; one thread per
//                    sample, weights in shared memory.
// The network is FP32 SIMT arithmetic: about 55 kflop per training sample, so
// a whole training run is a small fraction of the solves that produce its data.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "hr_runtime.h"

namespace {

constexpr int kIn = 12, kH = 64, kOut = 3;
constexpr int oW1 = 0, ob1 = oW1 + kIn * kH, oW2 = ob1 + kH, ob2 = oW2 + kH * kH, oW3 = ob2 + kH,
              ob3 = oW3 + kH * kH, oW4 = ob3 + kH, ob4 = oW4 + kH * kOut, kNP = ob4 + kOut;
static_assert(kNP == 9347, "parameter count");
constexpr int kThreads = 128;
constexpr int kPpad = (kNP + 3) & ~3;

__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  // splitmix64 finalizer (Steele, Lea, Flood 2014)
  x += 0x9e3779b97f4a7c15ULL;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
  return x ^ (x >> 31);
}

struct Norm {
  float mean[kIn], inv_std[kIn];
  float out_scale;
};

// Batch sample s: s itself (in-order batches) or a hash of (seed, step, s).
__device__ __forceinline__ long sample_index(long s, long n, unsigned long long seed, long step, int random) {
  if (!random) return s;
  const unsigned long long h = mix64(seed ^ mix64(((unsigned long long)step << 32) ^ (unsigned long long)s));
  return (long)(h % (unsigned long long)n);
}

// z[j] = bias[j] + sum_i col[i] * W[i][j], col = this thread's activation column.
__device__ __forceinline__ void dense64(const float* __restrict__ P, int oW, int ob, const float* col,
                                        float z[kH]) {
#pragma unroll
  for (int j = 0; j < kH; j++) z[j] = P[ob + j];
#pragma unroll 2
  for (int i = 0; i < kH; i++) {
    const float ai = col[i * kThreads];
    const float4* w = reinterpret_cast<const float4*>(P + oW + i * kH);
#pragma unroll
    for (int j4 = 0; j4 < kH / 4; j4++) {
      const float4 v = w[j4];
      z[4 * j4] += ai * v.x;
      z[4 * j4 + 1] += ai * v.y;
      z[4 * j4 + 2] += ai * v.z;
      z[4 * j4 + 3] += ai * v.w;
    }
  }
}

// Forward of one sample; col: this thread's activation column.
__device__ __forceinline__ void forward(const float* __restrict__ P, const float* __restrict__ xin,
                                        const Norm& nm, float* col, float z[kH], float y[kOut]) {
  float x[kIn];
#pragma unroll
  for (int i = 0; i < kIn; i++) x[i] = (xin[i] - nm.mean[i]) * nm.inv_std[i];
#pragma unroll
  for (int j = 0; j < kH; j++) z[j] = P[ob1 + j];
#pragma unroll
  for (int i = 0; i < kIn; i++) {
    const float4* w = reinterpret_cast<const float4*>(P + oW1 + i * kH);
#pragma unroll
    for (int j4 = 0; j4 < kH / 4; j4++) {
      const float4 v = w[j4];
      z[4 * j4] += x[i] * v.x;
      z[4 * j4 + 1] += x[i] * v.y;
      z[4 * j4 + 2] += x[i] * v.z;
      z[4 * j4 + 3] += x[i] * v.w;
    }
  }
  for (int layer = 0; layer < 3; layer++) {
#pragma unroll
    for (int j = 0; j < kH; j++) col[j * kThreads] = silu(z[j]);
    if (layer < 2) dense64(P, layer == 0 ? oW2 : oW3, layer == 0 ? ob2 : ob3, col, z);
  }
#pragma unroll
  for (int j = 0; j < kOut; j++) y[j] = P[ob4 + j];
#pragma unroll 4
  for (int i = 0; i < kH; i++) {
    const float ai = col[i * kThreads];
#pragma unroll
    for (int j = 0; j < kOut; j++) y[j] += ai * P[oW4 + i * kOut + j];
  }
}

// All loads of a thread in flight at once (one memory latency, not 37).
template <int kThr>
__device__ __forceinline__ void load_params(float* P, const float* __restrict__ params) {
  constexpr int kV = kNP / 4, kN = (kV + kThr - 1) / kThr;
  const float4* src = reinterpret_cast<const float4*>(params);
  float4 v[kN];
#pragma unroll
  for (int i = 0; i < kN; i++) {
    const int e = threadIdx.x + i * kThr;
    if (e < kV) v[i] = src[e];
  }
#pragma unroll
  for (int i = 0; i < kN; i++) {
    const int e = threadIdx.x + i * kThr;
    if (e < kV) reinterpret_cast<float4*>(P)[e] = v[i];
  }
  if (threadIdx.x < kNP - 4 * kV) P[4 * kV + threadIdx.x] = params[4 * kV + threadIdx.x];
}

// Training pass over a tile of kS samples: forward, squared-error loss (mean
// over batch and components of (y - t / out_scale)^2), backward deltas, and the
// tile's partial gradient dW = A^T Delta.
//
// FP32 multiply-adds on the SIMT cores: 27 k per sample, 12 us for 16384
// samples at their peak rate. One thread per sample with its activations in
// shared-memory columns, pre-activations and deltas through global memory and a
// gradient kernel with two shared reads per multiply-add took 150 us. Here
// every layer is a small matrix product with register tiles, 8 features x 4
// samples per thread (3 shared reads of 16 bytes per 32 multiply-adds: the
// shared-memory pipe and the multiply-adds take about equally long), with the
// activations a_l and the derivatives s'(z_l) in shared memory; the deltas
// overwrite the derivatives, so a tile's state fits one CTA (213 KB). Lanes run
// along the samples, so that stores and gathers meet different banks and the
// weights are broadcast. A batch of 16384 is 128 tiles: one CTA on each of 128
// SMs. Measured: a step of that batch 148 -> 45 us (batch 300: 111 -> 44, 60000:
// 474 -> 160); issue slots 52 % busy, shared-memory pipe 52 %, the rest the
// latencies between barriers with two warps per SM quarter. Four warps with 8 x 8
// tiles and every layer's code unrolled took 64 us: the code is fetched once
// per CTA, so the layers loop over one copy of it.
constexpr int kS = 128, kSP = kS + 4;  // samples per tile; row stride (rows 4 banks apart)
constexpr int kTrainThreads = 256;
constexpr int kActR = kH * kSP;        // floats of one [feature][sample] array

// acc[f][q] += sum_k w(k, f) a[k][sample q]: features 8 tx + f, samples 4 ty + q.
// a: K rows of kSP; w: row k, 64 columns.
__device__ __forceinline__ void tile_mul(const float* a, const float* w, int K, int tx, int ty, float (&acc)[8][4]) {
#pragma unroll 4
  for (int k = 0; k < K; k++) {
    const float4 av4 = *reinterpret_cast<const float4*>(a + k * kSP + 4 * ty);
    const float4 w0 = *reinterpret_cast<const float4*>(w + k * kH + 8 * tx);
    const float4 w1 = *reinterpret_cast<const float4*>(w + k * kH + 8 * tx + 4);
    const float av[4] = {av4.x, av4.y, av4.z, av4.w};
    const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
#pragma unroll
    for (int f = 0; f < 8; f++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[f][q] += av[q] * wv[f];
  }
}

// The same with the weights' transpose: acc[f][q] += sum_j W[8 tx + f][j] d[j][sample q].
__device__ __forceinline__ void tile_mul_t(const float* d, const float* w, int tx, int ty, float (&acc)[8][4]) {
#pragma unroll 1
  for (int j = 0; j < kH; j += 4) {
    float4 wr[8];
#pragma unroll
    for (int f = 0; f < 8; f++) wr[f] = *reinterpret_cast<const float4*>(w + (8 * tx + f) * kH + j);
#pragma unroll
    for (int jj = 0; jj < 4; jj++) {
      const float4 dv4 = *reinterpret_cast<const float4*>(d + (j + jj) * kSP + 4 * ty);
      const float dv[4] = {dv4.x, dv4.y, dv4.z, dv4.w};
#pragma unroll
      for (int f = 0; f < 8; f++) {
        const float wv = jj == 0 ? wr[f].x : (jj == 1 ? wr[f].y : (jj == 2 ? wr[f].z : wr[f].w));
#pragma unroll
        for (int q = 0; q < 4; q++) acc[f][q] += wv * dv[q];
      }
    }
  }
}

__device__ __forceinline__ void store_row(float* row, int ty, const float (&v)[4]) {
  *reinterpret_cast<float4*>(row + 4 * ty) = make_float4(v[0], v[1], v[2], v[3]);
}

// Partial gradient of one layer over the tile: dW[i][j] = sum_s a[i][s] d[j][s]
// for kI rows i and the 64 columns j, and db[j] = sum_s d[j][s]. Each half of
// the CTA sums half of the samples (a thread: rows gx + 8 r, columns gy + 16 c);
// the second half's sums go to the first through `a`, which nothing reads again.
template <int kI>
__device__ __forceinline__ void tile_grad(float* a, const float* d, float* __restrict__ dw, float* __restrict__ db) {
  constexpr int kR = (kI + 7) / 8;
  const int half = threadIdx.x >> 7, t = threadIdx.x & 127, lane = t & 31, warp = t >> 5;
  const int gy = (lane & 7) + 8 * (warp & 1), gx = (lane >> 3) + 4 * (warp >> 1);
  float acc[kR][4], accb[4];
#pragma unroll
  for (int c = 0; c < 4; c++) {
    accb[c] = 0.f;
#pragma unroll
    for (int r = 0; r < kR; r++) acc[r][c] = 0.f;
  }
#pragma unroll 1
  for (int s = half * (kS / 2); s < (half + 1) * (kS / 2); s += 4) {
    float4 av[kR], dv[4];
#pragma unroll
    for (int r = 0; r < kR; r++) {
      const int i = gx + 8 * r;
      av[r] = *reinterpret_cast<const float4*>(a + (i < kI ? i : 0) * kSP + s);
    }
#pragma unroll
    for (int c = 0; c < 4; c++) dv[c] = *reinterpret_cast<const float4*>(d + (gy + 16 * c) * kSP + s);
#pragma unroll
    for (int c = 0; c < 4; c++) {
#pragma unroll
      for (int r = 0; r < kR; r++) {
        acc[r][c] += av[r].x * dv[c].x;
        acc[r][c] += av[r].y * dv[c].y;
        acc[r][c] += av[r].z * dv[c].z;
        acc[r][c] += av[r].w * dv[c].w;
      }
      accb[c] += (dv[c].x + dv[c].y) + (dv[c].z + dv[c].w);
    }
  }
  __syncthreads();  // everyone has read a
  if (half == 1) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
#pragma unroll
      for (int r = 0; r < kR; r++) a[(c * kR + r) * 128 + t] = acc[r][c];
      if (gx == 0) a[(4 * kR + c) * 128 + gy] = accb[c];
    }
  }
  __syncthreads();
  if (half == 0) {
#pragma unroll
    for (int c = 0; c < 4; c++) {
#pragma unroll
      for (int r = 0; r < kR; r++) {
        const int i = gx + 8 * r;
        if (i < kI) dw[i * kH + gy + 16 * c] = acc[r][c] + a[(c * kR + r) * 128 + t];
      }
      if (gx == 0) db[gy + 16 * c] = accb[c] + a[(4 * kR + c) * 128 + gy];
    }
  }
}
static_assert((4 * 8 + 4) * 128 <= kActR && (4 * 2 + 4) * 128 <= kIn * kSP, "a half's sums fit in place of the inputs");

__global__ void __launch_bounds__(kTrainThreads) train_kernel(
    const float* __restrict__ params, Norm nm, const float* __restrict__ X, const float* __restrict__ T, long n,
    int batch, unsigned long long seed, long step, int random, float* partial, double* __restrict__ loss_part) {
  extern __shared__ __align__(16) float sm[];
  float* P = sm;                    // weights (padded)
  float* x = P + kPpad;             // normalized inputs, kIn rows
  float* act = x + kIn * kSP;       // activations a1, a2, a3 (later d3)
  float* der = act + 3 * kActR;     // derivatives s'(z1), s'(z2), later the deltas d1, d2
  float* d4 = der + 2 * kActR;      // output deltas, kOut rows
  __shared__ double red[kTrainThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ty = (lane & 7) + 8 * (warp & 3), tx = (lane >> 3) + 4 * (warp >> 2);
  const int s = blockIdx.x * kS + tid;  // this thread's sample in the per-sample parts (tid < kS)
  const bool valid = tid < kS && s < batch;
  // past the batch's end a tile repeats its first sample with output deltas of
  // zero: what a sample without input (the biases alone) gives may overflow where
  // no sample of the batch does, and 0 x inf would reach the gradient
  const long g = tid < kS ? sample_index(valid ? s : blockIdx.x * kS, n, seed, step, random) : 0;
  load_params<kTrainThreads>(P, params);
  if (tid < kS) {
#pragma unroll
    for (int i = 0; i < kIn; i++) x[i * kSP + tid] = (X[g * kIn + i] - nm.mean[i]) * nm.inv_std[i];
  }
  __syncthreads();
  float z[8][4];
  // one copy of the layers' code: it is fetched once per CTA, by one CTA per SM
#pragma unroll 1
  for (int l = 0; l < 3; l++) {
    const int ob = l == 0 ? ob1 : (l == 1 ? ob2 : ob3), oW = l == 0 ? oW1 : (l == 1 ? oW2 : oW3);
#pragma unroll
    for (int f = 0; f < 8; f++)
#pragma unroll
      for (int q = 0; q < 4; q++) z[f][q] = P[ob + 8 * tx + f];
    tile_mul(l == 0 ? x : act + (l - 1) * kActR, P + oW, l == 0 ? kIn : kH, tx, ty, z);
    // a = silu(z), z <- silu'(z), one sigmoid each; the last layer's derivatives
    // stay in registers
#pragma unroll
    for (int f = 0; f < 8; f++) {
      float av[4];
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const float sg = sigm(z[f][q]);
        av[q] = z[f][q] * sg;
        z[f][q] = sg * (1.0f + z[f][q] * (1.0f - sg));
      }
      store_row(act + l * kActR + (8 * tx + f) * kSP, ty, av);
      if (l < 2) store_row(der + l * kActR + (8 * tx + f) * kSP, ty, z[f]);
    }
    __syncthreads();
  }
  float* a3 = act + 2 * kActR;
  // output, loss and its delta: one sample per thread
  double l2 = 0.0;
  if (tid < kS) {
    float y[kOut];
#pragma unroll
    for (int j = 0; j < kOut; j++) y[j] = P[ob4 + j];
#pragma unroll 8
    for (int i = 0; i < kH; i++) {
      const float ai = a3[i * kSP + tid];
#pragma unroll
      for (int j = 0; j < kOut; j++) y[j] += ai * P[oW4 + i * kOut + j];
    }
    const float inv = 2.0f / (float)((long)batch * kOut);
#pragma unroll
    for (int j = 0; j < kOut; j++) {
      const float e = valid ? y[j] - T[g * kOut + j] / nm.out_scale : 0.f;
      l2 += (double)e * (double)e;
      d4[j * kSP + tid] = e * inv;
    }
  }
  __syncthreads();
  float* out = partial + (size_t)blockIdx.x * kNP;
  // output layer's gradient: thread i < 64 row i of dW4, threads 64..66 the biases
  if (tid < kH + kOut) {
    float acc[kOut] = {0.f, 0.f, 0.f};
#pragma unroll 2
    for (int q = 0; q < kS; q += 4) {
      const float4 av = tid < kH ? *reinterpret_cast<const float4*>(a3 + tid * kSP + q) : make_float4(1.f, 1.f, 1.f, 1.f);
#pragma unroll
      for (int j = 0; j < kOut; j++) {
        const float4 dv = *reinterpret_cast<const float4*>(d4 + j * kSP + q);
        acc[j] += av.x * dv.x;
        acc[j] += av.y * dv.y;
        acc[j] += av.z * dv.z;
        acc[j] += av.w * dv.w;
      }
    }
    if (tid < kH) {
#pragma unroll
      for (int j = 0; j < kOut; j++) out[oW4 + tid * kOut + j] = acc[j];
    } else {
      const int j = tid - kH;
      out[ob4 + j] = j == 0 ? acc[0] : (j == 1 ? acc[1] : acc[2]);
    }
  }
  __syncthreads();
  // d3 = (W4 d4) s'(z3), in place of a3
#pragma unroll
  for (int f = 0; f < 8; f++) {
    float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < kOut; j++) {
      const float w = P[oW4 + (8 * tx + f) * kOut + j];
      const float4 e = *reinterpret_cast<const float4*>(d4 + j * kSP + 4 * ty);
      v[0] += w * e.x;
      v[1] += w * e.y;
      v[2] += w * e.z;
      v[3] += w * e.w;
    }
#pragma unroll
    for (int q = 0; q < 4; q++) v[q] *= z[f][q];
    store_row(a3 + (8 * tx + f) * kSP, ty, v);
  }
  __syncthreads();
  // layers 3 and 2: the gradient from a_{l-1} and d_l, then d_{l-1} = (W d_l)
  // s'(z_{l-1}) in place of the derivatives
#pragma unroll 1
  for (int l = 2; l > 0; l--) {
    const float* d = l == 2 ? a3 : der + kActR;
    const int oW = l == 2 ? oW3 : oW2, ob = l == 2 ? ob3 : ob2;
    tile_grad<kH>(act + (l - 1) * kActR, d, out + oW, out + ob);
#pragma unroll
    for (int f = 0; f < 8; f++)
#pragma unroll
      for (int q = 0; q < 4; q++) z[f][q] = 0.f;
    tile_mul_t(d, P + oW, tx, ty, z);
#pragma unroll
    for (int f = 0; f < 8; f++) {
      float* row = der + (l - 1) * kActR + (8 * tx + f) * kSP;
      const float4 sg = *reinterpret_cast<const float4*>(row + 4 * ty);
      const float v[4] = {z[f][0] * sg.x, z[f][1] * sg.y, z[f][2] * sg.z, z[f][3] * sg.w};
      store_row(row, ty, v);
    }
    __syncthreads();
  }
  tile_grad<kIn>(x, der, out + oW1, out + ob1);
  for (int off = 16; off > 0; off >>= 1) l2 += __shfl_down_sync(0xffffffffu, l2, off);
  if (lane == 0) red[warp] = l2;
  __syncthreads();
  if (tid == 0) {
    double t = 0;
    for (int w = 0; w < kTrainThreads / 32; w++) t += red[w];
    loss_part[blockIdx.x] = t;
  }
}

struct Adam {
  float lr, b1, b2, eps, c1, c2;
};

// The gradient, summed over the tiles, and (lr > 0) the Adam step. A CTA of four
// warps takes 32 parameters; each warp sums a quarter of the tiles, eight at a
// time by pairs and the eights in FP64, then the quarters are added in order
// (deterministic). Loads and chains of additions bound it: one FP32 chain per
// quarter made a step of batch 16384 47.2 us instead of 45.1 (60000: 166 and
// 160), one FP64 chain 49.2 us.
__global__ void __launch_bounds__(128) grad_adam_kernel(const float* __restrict__ partial, int ntiles,
                                                        float* __restrict__ grad, float* __restrict__ params,
                                                        float* __restrict__ m, float* __restrict__ v, Adam o) {
  __shared__ double part[4][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane;
  const int per = (ntiles + 3) / 4, c0 = warp * per, c1 = min(ntiles, c0 + per);
  double sum = 0.0;
  if (p < kNP) {
    int c = c0;
    for (; c + 8 <= c1; c += 8) {
      float t[8];
#pragma unroll
      for (int i = 0; i < 8; i++) t[i] = partial[(size_t)(c + i) * kNP + p];
      sum += (double)(((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7])));
    }
    for (; c < c1; c++) sum += (double)partial[(size_t)c * kNP + p];
  }
  part[warp][lane] = sum;
  __syncthreads();
  if (warp != 0 || p >= kNP) return;
  const float g = (float)(((part[0][lane] + part[1][lane]) + part[2][lane]) + part[3][lane]);
  grad[p] = g;
  if (!(o.lr > 0.f)) return;
  const float mm = o.b1 * m[p] + (1.0f - o.b1) * g;
  const float vv = o.b2 * v[p] + (1.0f - o.b2) * g * g;
  m[p] = mm;
  v[p] = vv;
  params[p] -= o.lr * (mm / o.c1) / (sqrtf(vv / o.c2) + o.eps);
}

// Output frames of inference: samples start[f] .. start[f+1]-1 are rotated
// by R[f]^T (v_body = R v_world); n = 0 leaves the output as it is.
constexpr int kMaxFrames = 8;
struct Frames {
  int n;
  long start[kMaxFrames + 1];
  double R[kMaxFrames][9];
};

__global__ void __launch_bounds__(kThreads) infer_kernel(const float* __restrict__ params, Norm nm,
                                                         const float* __restrict__ X, long n,
                                                         const double* __restrict__ base,
                                                         double* __restrict__ out, float* __restrict__ raw,
                                                         Frames fr) {
  extern __shared__ __align__(16) float sm[];
  float* P = sm;
  float* cols = sm + kPpad;
  load_params<kThreads>(P, params);
  __syncthreads();
  const long s = (long)blockIdx.x * kThreads + threadIdx.x;
  if (s >= n) return;
  float z[kH], y[kOut];
  forward(P, X + s * kIn, nm, cols + threadIdx.x, z, y);
  double v[kOut] = {y[0], y[1], y[2]};
  for (int f = 0; f < fr.n; f++) {
    if (s >= fr.start[f] && s < fr.start[f + 1]) {
      const double* R = fr.R[f];
      v[0] = R[0] * y[0] + R[3] * y[1] + R[6] * y[2];
      v[1] = R[1] * y[0] + R[4] * y[1] + R[7] * y[2];
      v[2] = R[2] * y[0] + R[5] * y[1] + R[8] * y[2];
    }
  }
#pragma unroll
  for (int j = 0; j < kOut; j++) {
    if (raw) raw[s * kOut + j] = y[j];
    if (out) out[s * kOut + j] = (base ? base[s * kOut + j] : 0.0) + (double)nm.out_scale * v[j];
  }
}

__global__ void sum_kernel(const double* __restrict__ part, int n, double* out) {
  double s = 0.0;
  for (int i = 0; i < n; i++) s += part[i];
  *out = s;
}

constexpr size_t kFwdSmem = sizeof(float) * ((size_t)kPpad + (size_t)kH * kThreads);
constexpr size_t kTrainSmem = sizeof(float) * ((size_t)kPpad + (kIn + kOut) * kSP + 5 * (size_t)kActR);
static_assert(kTrainSmem + 64 <= 227 * 1024, "a tile's state fits one CTA");

}  // namespace

struct hr_mlp {
  hr_ctx* owner = nullptr;
  Norm nm;
  hr::DBuf<float> params, grad, m, v, partial;
  hr::DBuf<double> loss_part, loss;
  int cap = 0;
  long step = 0;
  void ensure(int batch) {
    hr::grow(cap, batch, [&] {
      const size_t tiles = ((size_t)batch + kS - 1) / kS;
      loss_part.alloc(tiles);
      partial.alloc(tiles * kNP);
    });
  }
};

namespace {

template <class F>
int mlp_guard(hr_mlp* M, F&& f) {
  try {
    f();
    return HR_OK;
  } catch (const hr::Error& e) {
    if (M && M->owner) M->owner->c.err = e.what();
    return e.code;
  } catch (const std::exception& e) {
    if (M && M->owner) M->owner->c.err = e.what();
    return HR_ERR_CUDA;
  }
}

void set_smem_attrs() {
  static bool done = false;
  if (done) return;
  HR_CHECK_CUDA(cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem));
  HR_CHECK_CUDA(cudaFuncSetAttribute(infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem));
  done = true;
}

// FNV-1a 64-bit over a byte string.
unsigned long long fnv1a(const unsigned char* p, size_t n) {
  unsigned long long h = 1469598103934665603ULL;
  for (size_t i = 0; i < n; i++) {
    h ^= p[i];
    h *= 1099511628211ULL;
  }
  return h;
}

}  // namespace

extern "C" int hr_mlp_nparams(void) { return kNP; }

extern "C" int hr_mlp_create(hr_ctx* ctx, unsigned long long seed, hr_mlp** out) {
  if (!ctx || !out) return HR_ERR_ARG;
  *out = nullptr;
  std::unique_ptr<hr_mlp> M(new hr_mlp);
  M->owner = ctx;
  int rc = mlp_guard(M.get(), [&] {
    cudaStream_t st = ctx->c.stream;
    set_smem_attrs();
    // Glorot-uniform weights, zero biases; uniforms from splitmix64 of (seed, index)
    std::vector<float> p(kNP, 0.0f);
    auto fill = [&](int off, int fan_in, int fan_out) {
      const double lim = sqrt(6.0 / (double)(fan_in + fan_out));
      for (int k = 0; k < fan_in * fan_out; k++) {
        unsigned long long h = seed + 0x9e3779b97f4a7c15ULL * (unsigned long long)(off + k + 1);
        h = (h ^ (h >> 30)) * 0xbf58476d1ce4e5b9ULL;
        h = (h ^ (h >> 27)) * 0x94d049bb133111ebULL;
        h ^= h >> 31;
        const double u = (double)(h >> 11) / 9007199254740992.0;
        p[off + k] = (float)((2.0 * u - 1.0) * lim);
      }
    };
    fill(oW1, kIn, kH);
    fill(oW2, kH, kH);
    fill(oW3, kH, kH);
    fill(oW4, kH, kOut);
    M->params.upload(p, st);
    M->grad.alloc(kNP);
    M->m.alloc(kNP);
    M->v.alloc(kNP);
    M->m.zero(st);
    M->v.zero(st);
    M->loss.alloc(1);
    for (int i = 0; i < kIn; i++) {
      M->nm.mean[i] = 0.f;
      M->nm.inv_std[i] = 1.f;
    }
    M->nm.out_scale = 1.f;
    HR_CHECK_CUDA(cudaStreamSynchronize(st));
  });
  if (rc != HR_OK) return rc;
  *out = M.release();
  return HR_OK;
}

// Frees the network's device buffers (cudaFree waits for work using them);
// it does not touch the owning context, which may already be gone.
extern "C" void hr_mlp_destroy(hr_mlp* M) { delete M; }

extern "C" int hr_mlp_set_normalization(hr_mlp* M, const float* mean, const float* stdv, float out_scale) {
  if (!M || !mean || !stdv || !(out_scale > 0)) return HR_ERR_ARG;
  for (int i = 0; i < kIn; i++)
    if (!(stdv[i] > 0)) return HR_ERR_ARG;
  for (int i = 0; i < kIn; i++) {
    M->nm.mean[i] = mean[i];
    M->nm.inv_std[i] = 1.0f / stdv[i];
  }
  M->nm.out_scale = out_scale;
  return HR_OK;
}

extern "C" int hr_mlp_get_params(hr_mlp* M, float* host) {
  if (!M || !host) return HR_ERR_ARG;
  return mlp_guard(M, [&] {
    cudaStream_t st = M->owner->c.stream;
    HR_CHECK_CUDA(cudaMemcpyAsync(host, M->params.p, sizeof(float) * kNP, cudaMemcpyDeviceToHost, st));
    HR_CHECK_CUDA(cudaStreamSynchronize(st));
  });
}

extern "C" int hr_mlp_set_params(hr_mlp* M, const float* host) {
  if (!M || !host) return HR_ERR_ARG;
  return mlp_guard(M, [&] {
    cudaStream_t st = M->owner->c.stream;
    HR_CHECK_CUDA(cudaMemcpyAsync(M->params.p, host, sizeof(float) * kNP, cudaMemcpyHostToDevice, st));
    M->m.zero(st);
    M->v.zero(st);
    M->step = 0;
    HR_CHECK_CUDA(cudaStreamSynchronize(st));
  });
}

extern "C" int hr_mlp_train_step(hr_mlp* M, const float* X_dev, const float* T_dev, long n, int batch,
                                 int random, unsigned long long seed, float lr, double* loss) {
  if (!M || !X_dev || !T_dev || n < 1 || batch < 1 || (!random && batch > n) || !(lr >= 0)) return HR_ERR_ARG;
  return mlp_guard(M, [&] {
    hr::Ctx& C = M->owner->c;
    cudaStream_t st = C.stream;
    set_smem_attrs();
    M->ensure(batch);
    const int nb = (batch + kS - 1) / kS;
    const long step = M->step + 1;
    train_kernel<<<nb, kTrainThreads, kTrainSmem, st>>>(M->params.p, M->nm, X_dev, T_dev, n, batch, seed, step, random,
                                                   M->partial.p, M->loss_part.p);
    const float b1 = 0.9f, b2 = 0.999f;
    const Adam o = {lr, b1, b2, 1e-8f, 1.0f - powf(b1, (float)step), 1.0f - powf(b2, (float)step)};
    grad_adam_kernel<<<(kNP + 31) / 32, 128, 0, st>>>(M->partial.p, nb, M->grad.p, M->params.p, M->m.p, M->v.p, o);
    C.launches += 2;
    if (lr > 0) M->step = step;
    HR_CHECK_CUDA(cudaGetLastError());
    if (loss) {
      sum_kernel<<<1, 1, 0, st>>>(M->loss_part.p, nb, M->loss.p);
      C.launches++;
      double l = 0;
      HR_CHECK_CUDA(cudaMemcpyAsync(&l, M->loss.p, sizeof(double), cudaMemcpyDeviceToHost, st));
      HR_CHECK_CUDA(cudaStreamSynchronize(st));
      *loss = l / (double)((long)batch * kOut);
    }
  });
}

extern "C" int hr_mlp_gradient(hr_mlp* M, const float* X_dev, const float* T_dev, int batch, float* grad_host,
                               double* loss) {
  if (!M || !grad_host) return HR_ERR_ARG;
  int rc = hr_mlp_train_step(M, X_dev, T_dev, batch, batch, 0, 0, 0.0f, loss);
  if (rc != HR_OK) return rc;
  return mlp_guard(M, [&] {
    cudaStream_t st = M->owner->c.stream;
    HR_CHECK_CUDA(cudaMemcpyAsync(grad_host, M->grad.p, sizeof(float) * kNP, cudaMemcpyDeviceToHost, st));
    HR_CHECK_CUDA(cudaStreamSynchronize(st));
  });
}

static int infer(hr_mlp* M, const float* X_dev, long n, const double* base_dev, double* out_dev, float* raw_dev,
                 const Frames& fr) {
  if (!M || n < 0 || (n > 0 && !X_dev)) return HR_ERR_ARG;
  if (n == 0) return HR_OK;
  return mlp_guard(M, [&] {
    hr::Ctx& C = M->owner->c;
    set_smem_attrs();
    infer_kernel<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, kFwdSmem, C.stream>>>(
        M->params.p, M->nm, X_dev, n, base_dev, out_dev, raw_dev, fr);
    C.launches++;
    HR_CHECK_CUDA(cudaGetLastError());
  });
}

extern "C" int hr_mlp_infer(hr_mlp* M, const float* X_dev, long n, const double* base_dev, double* out_dev,
                            float* raw_dev) {
  Frames fr;
  memset(&fr, 0, sizeof(fr));
  return infer(M, X_dev, n, base_dev, out_dev, raw_dev, fr);
}

extern "C" int hr_mlp_infer_frames(hr_mlp* M, const float* X_dev, long n, const double* base_dev, double* out_dev,
                                   int nframes, const long* frame_start, const double* rot) {
  if (nframes < 0 || nframes > kMaxFrames || (nframes > 0 && (!frame_start || !rot))) return HR_ERR_ARG;
  Frames fr;
  memset(&fr, 0, sizeof(fr));
  fr.n = nframes;
  for (int f = 0; f <= nframes; f++) fr.start[f] = frame_start[f];
  for (int f = 0; f < nframes; f++) {
    if (fr.start[f + 1] < fr.start[f]) return HR_ERR_ARG;
    for (int k = 0; k < 9; k++) fr.R[f][k] = rot[9 * f + k];
  }
  return infer(M, X_dev, n, base_dev, out_dev, nullptr, fr);
}

// Weights file: "HRMLP001", layer widths (5 x int32), 12 input means, 12 input
// stds, out_scale, the 9347 parameters (FP32), FNV-1a 64 of everything before.
extern "C" int hr_mlp_save(hr_mlp* M, const char* path) {
  if (!M || !path) return HR_ERR_ARG;
  std::vector<float> p(kNP);
  int rc = hr_mlp_get_params(M, p.data());
  if (rc != HR_OK) return rc;
  std::vector<unsigned char> buf;
  auto put = [&](const void* d, size_t n) {
    const unsigned char* c = (const unsigned char*)d;
    buf.insert(buf.end(), c, c + n);
  };
  put("HRMLP001", 8);
  const int shape[5] = {kIn, kH, kH, kH, kOut};
  put(shape, sizeof(shape));
  float stdv[kIn];
  for (int i = 0; i < kIn; i++) stdv[i] = 1.0f / M->nm.inv_std[i];
  put(M->nm.mean, sizeof(float) * kIn);
  put(stdv, sizeof(float) * kIn);
  put(&M->nm.out_scale, 4);
  put(p.data(), sizeof(float) * kNP);
  const unsigned long long h = fnv1a(buf.data(), buf.size());
  put(&h, 8);
  FILE* f = fopen(path, "wb");
  if (!f) {
    M->owner->c.err = std::string("cannot open ") + path;
    return HR_ERR_ARG;
  }
  const size_t w = fwrite(buf.data(), 1, buf.size(), f);
  fclose(f);
  return w == buf.size() ? HR_OK : HR_ERR_ARG;
}

extern "C" int hr_mlp_load(hr_mlp* M, const char* path) {
  if (!M || !path) return HR_ERR_ARG;
  FILE* f = fopen(path, "rb");
  if (!f) {
    M->owner->c.err = std::string("cannot open ") + path;
    return HR_ERR_ARG;
  }
  std::vector<unsigned char> buf;
  unsigned char tmp[4096];
  size_t r;
  while ((r = fread(tmp, 1, sizeof(tmp), f)) > 0) buf.insert(buf.end(), tmp, tmp + r);
  fclose(f);
  const size_t need = 8 + 5 * 4 + 4 * (2 * kIn + 1) + 4 * (size_t)kNP + 8;
  const int shape[5] = {kIn, kH, kH, kH, kOut};
  unsigned long long h = 0;
  if (buf.size() == need) memcpy(&h, buf.data() + need - 8, 8);
  if (buf.size() != need || memcmp(buf.data(), "HRMLP001", 8) != 0 || memcmp(buf.data() + 8, shape, 20) != 0 ||
      h != fnv1a(buf.data(), need - 8)) {
    M->owner->c.err = std::string("not a 12-64-64-64-3 warm-start weights file (header, shape or checksum): ") + path;
    return HR_ERR_ARG;
  }
  float mean[kIn], stdv[kIn], sc;
  memcpy(mean, buf.data() + 28, 4 * kIn);
  memcpy(stdv, buf.data() + 28 + 4 * kIn, 4 * kIn);
  memcpy(&sc, buf.data() + 28 + 8 * kIn, 4);
  const int rc = hr_mlp_set_normalization(M, mean, stdv, sc);
  if (rc != HR_OK) return rc;
  std::vector<float> p(kNP);
  memcpy(p.data(), buf.data() + 32 + 8 * kIn, 4 * (size_t)kNP);
  return hr_mlp_set_params(M, p.data());
}
