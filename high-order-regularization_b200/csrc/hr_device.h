// hr_device.h — device task descriptors and kernel launchers (internal).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "hr_engine.h"

namespace hr {

// doubles per target in a work item's partial sums (3 velocity + 1 pressure)
constexpr int kPartComps = 4;

// One boundary sum: a source surface (tree order SoA) evaluated at a target
// set (reference order). All pointers are device pointers.
struct EvalTask {
  int kind;       // Kind
  int jump_mode;  // DL kinds: 0 = treecode convention, 1 = direct-sum convention
  int P1, Pf;     // treecode degree + 1 and (P+1)^3
  int C;          // FP64 moment values stored per proxy (6 SL, 10 DL)
  int nt;         // number of targets
  int mixed;      // 0 FP64; 1: pairs beyond 3 delta and proxies in FP32 (FP64 accumulation); 2: all pairs FP32
  int pad;
  double DEL;     // regularization length delta
  double scale;   // final factor of the sum (1/8pi, -6/8pi, ...)
  const double *sx, *sy, *sz, *snx, *sny, *snz, *sa;  // sources, tree order
  const double *qx, *qy, *qz;                         // density, tree order
  const double* pk;                                   // packed sources, tree order (Pack), for the FP64 sums
  const float *fnx, *fny, *fnz, *fa, *fqx, *fqy, *fqz;  // FP32 copies (reduced-precision sums)
  const double* tcheb;                                // 3*P1 per node
  const double* mom;                                  // Pf*C per node, proxy-major
  const float* momf;                                  // FP32 copy per node: momf_stride floats
  const int* tord;                                    // target order -> target index
  const double* txyz;                                 // 3nt targets
  const double* tb;                                   // nt signed distances
  const uint8_t* tnear;                               // nt regularized-branch flag
  const double* tf0;                                  // 3nt nearest force (SL off, E2G)
  const double *tx0, *tn0, *tg0;                      // 3nt nearest point, normal, density
  const double *tq, *tnrm;                            // 3nt own density and normal (on-surface)
  double* out;                                        // 3nt (or nt for pressure)
  double* out2;                                       // nt pressure of K_E2G_UP_AWAY (scaled by scale2)
  double scale2;
  const Entry* entries;                               // interaction entries
  unsigned long long* counters;  // [0] regularized pairs [1] near-target plain [2] far-target [3] proxy
  const int* item_start;  // per target block: its work items' partial slots [start, end)
  double* partial;        // kTB x kPartComps doubles per work item
};

// A piece of one entry: a near entry's source sub-range [s0, s1), or a whole
// far entry (proxy points).
struct Seg {
  int entry;
  int s0, s1;
};

// A work item: a run of consecutive segments of one target block. Each
// item writes its partial sums into its own slot; the reduce kernel adds the
// slots of a block in order, so results do not depend on scheduling.
struct BlockRef {
  int task;
  int blk;
  int seg0, seg1;
  int slot;
};

enum Family : int { F_SL = 0, F_DL = 1, F_E2G = 2 };

// A source's packed record; the area weight a is multiplied into what a
// family's pairs only use times it.
enum Pack : int {
  PACK_SL = 0,   // 10 doubles: x, y, z, a, a normal, a density
  PACK_DL = 1,   // 10 doubles: x, y, z, a, a normal, density
  PACK_E2G = 2,  // 12 doubles: x, y, z, a, density, normal.normal, normal, 0
};

// The reduced-precision sums of a batch: every work item of a combined list,
// the first n_on items (lean: on-surface tasks, or the extend-to-grid box-face
// sums) in one launch on st, the rest in another on side. next: two zeroed work
// counters (one per launch); launch_reduce zeroes them again.
void launch_eval(int family, const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems, int n_on,
                 unsigned* next, int num_sms, cudaStream_t st, cudaStream_t side);

// The FP64 sums of a batch likewise (hr_eval64.cu). With count, the per-branch
// pair counts are added to the tasks' counters.
void launch_eval64(int family, const EvalTask* d_tasks, const BlockRef* d_items, const Seg* d_segs, int nitems,
                   int n_on, unsigned* next, int num_sms, cudaStream_t st, cudaStream_t side, bool count);
// The batch's reduction (the items' partial sums per target, in slot order) and
// epilogue; zeroes the two counters at next.
void launch_reduce(const EvalTask* d_tasks, int ntask_blocks, const int2* d_task_blocks, unsigned* next,
                   cudaStream_t st);

// Upward pass: proxy moments of every non-root node of a tree.
struct MomItem {
  int node;
  int s0;  // first source (tree order)
  int s1;  // one past last source
  int out; // partial slot
};
// Poisson extension (solve_Poisson, E2G/main.cpp:969-1044) with a reusable
// work area (FFT plan, tables, grid buffers) for one grid size N.
struct PoissonWork;
PoissonWork* poisson_work_create(struct Ctx& C, int N);
void poisson_work_destroy(PoissonWork* w);
void solve_poisson_dev(struct Ctx& C, int N, double L, const uint8_t* band2_dev, const uint8_t* out_dev,
                       const double* p_dev, double* u_dev, int variable, PoissonWork* work = nullptr);

// Tensor-core (tcgen05, 3xTF32) upward pass for the reduced-precision operator:
// the same items; partial moments of 12 (stresslet) or 6 channels per item; a timed-out wait sets *err.
bool moments_tc_supported(int P1);
size_t moments_tc_smem(int dl, int P1, int* npad, int* cols);
void launch_moments_tc(int dl, const MomItem* d_items, int nitems, int P1, const double* tcheb, const double* x,
                       const double* y, const double* z, const double* nx, const double* ny, const double* nz,
                       const double* a, const double* qx, const double* qy, const double* qz, double* partial,
                       int* err, cudaStream_t st);
// The FP32 moments of a node: per Chebyshev row (P+1)/2 pairs of proxies (an
// odd last one fills half a pair), interleaved value by value: 20 floats per
// pair of the stresslet's 9 values, 12 of the Stokeslet's 6.
inline __host__ __device__ size_t momf_stride(int P1, int pair_floats) {
  return (size_t)P1 * P1 * ((P1 + 1) / 2) * pair_floats;
}
// One tree's part of an upward pass.
struct MomTree {
  const MomItem* items;
  int nitems, nn;  // items, nodes
  const int* item_start;
  const double *tcheb, *x, *y, *z, *nx, *ny, *nz, *a, *qx, *qy, *qz;
  double *partial, *mom;
  float* momf;
};
// FP64 upward pass of one or two trees (the second may be empty) of the same
// degree: C = 9 stresslet, 6 Stokeslet channels; then the reduction per node (C
// = 12: the layout of launch_moments_tc).
void launch_moments(int C, int P1, const MomTree& t0, const MomTree& t1, cudaStream_t st);
void launch_moments_reduce(int C, int P1, const MomTree& t0, const MomTree& t1, cudaStream_t st);

// Gathers the interleaved reference-order densities of one or two trees into
// tree-order SoA, FP32 copies (fqx, if not null) and packed records as `pack`
// says (pk, if not null).
struct PermTree {
  int n;
  const int* perm;
  const double *q3, *x, *y, *z, *nx, *ny, *nz, *a;
  double *qx, *qy, *qz;
  float *fqx, *fqy, *fqz;
  double* pk;
};
void launch_permute(const PermTree& t0, const PermTree& t1, int pack, cudaStream_t st);

// Six-point density interpolation at nearest points, one or two target sets.
struct InterpSet {
  int ne;  // entries
  const int *tgt, *idx;
  const double *pq, *g;
  double* g0;
};
void launch_interp(const InterpSet& s0, const InterpSet& s1, cudaStream_t st);

// Two-surface combine steps; a is taken before b.
struct CombineSet {
  int n;
  const double *a, *b;
};
void launch_matvec_combine(const CombineSet& s0, const CombineSet& s1, double factor, const double* x, double* y,
                           cudaStream_t st);
void launch_rhs_combine(const CombineSet& s0, const CombineSet& s1, double factor, double* b, cudaStream_t st);

// Lets a kernel (without static shared memory) be launched with any dynamic shared
// memory that a CTA can have. The limit belongs to the kernel on its device, not
// to a launch: one set to what a launch needs would refuse a larger launch by
// another thread, or by a plan made earlier.
constexpr int kCtaShared = 227 * 1024;
template <class F>
inline cudaError_t allow_shared(F* kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCtaShared);
}

// Vector kernels for GMRES (deterministic reductions).
constexpr int kRedBlocks = 296;
struct DotWork {
  double* partial;  // kRedBlocks x 64
  unsigned* done;   // zero between launches
};
// out[c] = U[c] . w (columns of stride ldv)
void launch_dots(int n, int ncols, const double* U, long ldv, const double* w, const DotWork& d, double* out,
                 cudaStream_t st);
// w -= sum_c coef[c] V[c], then out[c] = U[c] . w
void launch_sub_dots(int n, int nsub, const double* V, long ldv, const double* coef, double* w, int ncols,
                     const double* U, const DotWork& d, double* out, cudaStream_t st);
void launch_axpy_multi(int n, int ncols, const double* V, long ldv, const double* coef,
                       double sign, double* w, cudaStream_t st);
// w *= s; copy = w
void launch_scale_copy(int n, double s, double* w, double* copy, cudaStream_t st);
void launch_sub(int n, const double* a, const double* b, double* out, cudaStream_t st);
void launch_copy(int n, const double* a, double* out, cudaStream_t st);

// FP64 FMA peak loop.
void launch_fma_peak(double* out, int iters, int blocks, cudaStream_t st);
void launch_fma_peak32(float* out, int iters, int blocks, cudaStream_t st);

}  // namespace hr
