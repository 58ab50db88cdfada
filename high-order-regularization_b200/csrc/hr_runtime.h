// hr_runtime.h — context, device buffers and the device-resident objects the
// C ABI is built from (internal).
#pragma once
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/highreg_b200.h"
#include "hr_device.h"
#include "hr_engine.h"

namespace hr {

struct Error : std::runtime_error {
  int code;
  Error(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

// The error is taken from the runtime when it is thrown, so that a later call
// does not report it again for a launch of its own.
#define HR_CHECK_CUDA(call)                                                                  \
  do {                                                                                       \
    cudaError_t e_ = (call);                                                                 \
    if (e_ != cudaSuccess) {                                                                 \
      cudaGetLastError();                                                                    \
      throw ::hr::Error(HR_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));    \
    }                                                                                        \
  } while (0)

#define HR_REQUIRE(cond, msg)                                   \
  do {                                                          \
    if (!(cond)) throw ::hr::Error(HR_ERR_ARG, std::string(msg)); \
  } while (0)

// The library's device buffers come from one stream-ordered memory pool per
// device that keeps freed blocks mapped (up to a few GiB), so building and
// destroying plans does not map and unmap pages for every buffer. dev_alloc
// returns memory that every stream may use at once; dev_free first waits for
// the pointer's device to go idle, as cudaFree does, and never throws.
void* dev_alloc(size_t bytes);
void dev_free(void* p) noexcept;

// The workspace of a context's stateless calls (single sums, interpolation,
// transforms): device memory handed out front to back and page-locked staging
// that collects a call's small uploads, both kept between calls. A call of such
// an entry point made ~55 allocations, as many uploads and as many frees, each
// with a synchronization: most of the 0.7 ms of a small sum. What does not fit
// comes from dev_alloc as before and grows the workspace, up to its limits, when
// the call is over. One call at a time (a context belongs to one thread). An
// allocation for which the device has no room gets the memory of the workspaces
// that are between calls.
struct Workspace {
  static constexpr size_t kDevMax = size_t(256) << 20, kPinMax = size_t(32) << 20;
  static constexpr size_t kSmall = size_t(4) << 20;  // uploads up to this size are collected
  int device = 0;
  bool busy = false;  // in a WorkspaceScope: otherwise dev_alloc may take the device memory back
  char* dev = nullptr;
  char* pin = nullptr;
  size_t dev_cap = 0, pin_cap = 0;    // capacities
  size_t low = 0, high = 0;           // uploads from the front, scratch from the back
  size_t flushed = 0;                 // uploads already copied
  size_t want_dev = 0, want_pin = 0;  // this call's total needs that fit the limits
  // `bytes` of device memory, null if they do not fit; up: among the uploads
  void* take(size_t bytes, bool up);
  // copies the uploads collected since the last flush
  void flush(cudaStream_t st);
  void free_all();
};
// The calling thread's active workspace (null outside a WorkspaceScope).
Workspace*& active_workspace();

template <class T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  bool borrowed = false;  // from the active workspace, not freed here
  DBuf() = default;
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), borrowed(o.borrowed) {
    o.p = nullptr;
    o.n = 0;
  }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      borrowed = o.borrowed;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
  ~DBuf() { release(); }
  void release() {
    if (p && !borrowed) dev_free(p);
    p = nullptr;
    n = 0;
  }
  void alloc(size_t count) { get(count, false); }
  void upload(const T* h, size_t count, cudaStream_t st) {
    const size_t bytes = count * sizeof(T);
    Workspace* w = active_workspace();
    const bool small = w && h && count && bytes <= Workspace::kSmall;
    get(count, small);
    if (!h || !count) return;
    if (small && borrowed) {  // collected: copied by flush
      std::memcpy(w->pin + (reinterpret_cast<char*>(p) - w->dev), h, bytes);
      return;
    }
    HR_CHECK_CUDA(cudaMemcpyAsync(p, h, bytes, cudaMemcpyHostToDevice, st));
  }
  void upload(const std::vector<T>& v, cudaStream_t st) { upload(v.data(), v.size(), st); }
  void zero(cudaStream_t st) {
    if (p) HR_CHECK_CUDA(cudaMemsetAsync(p, 0, n * sizeof(T), st));
  }

 private:
  void get(size_t count, bool up) {
    release();
    if (count == 0) count = 1;
    Workspace* w = active_workspace();
    p = w ? static_cast<T*>(w->take(count * sizeof(T), up)) : nullptr;
    borrowed = p != nullptr;
    if (!p) p = static_cast<T*>(dev_alloc(count * sizeof(T)));
    n = count;
  }
};

// Grows buffers that are kept between calls: alloc allocates them anew for `want`,
// `have` is what they hold now. It is zero while alloc runs, which lets go of
// the old memory first: after a failed allocation the next call, of any size,
// allocates again.
template <class N, class F>
void grow(N& have, N want, F&& alloc) {
  if (want <= have) return;
  have = 0;
  alloc();
  have = want;
}

struct Ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  // a second stream forked from and joined back to `stream` around the two
  // launches of a boundary-sum batch, so that each fills the other's tail
  cudaStream_t side = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  std::string err;
  long long launches = 0;
  int num_sms = 148;
  // while set, FP64 boundary-sum launches record their per-branch pair counts
  // (the tasks' work counters); other launches skip the tests
  bool count_work = false;
  DBuf<unsigned long long> counters;  // [0] reg pairs [1] plain pairs [2] proxies
  DBuf<int> tc_err;                   // set by a tensor-core kernel whose bounded wait ran out
  // two pinned host buffers of kPinChunk bytes for staged reads (d2h_staged),
  // allocated on first use, and the events that mark each one filled
  void* pin = nullptr;
  cudaEvent_t pin_ev[2] = {nullptr, nullptr};
  Workspace ws;
  // throws if a tensor-core kernel of this context reported a timed-out wait
  void check_tc();
};

// Makes a context's workspace the calling thread's active one for the duration
// of a synchronous call; on the way out (also by an exception) it waits for the
// context's streams, so that the memory is idle, and grows the workspace to the
// call's needs.
struct WorkspaceScope {
  Ctx& C;
  explicit WorkspaceScope(Ctx& c);
  ~WorkspaceScope();
  WorkspaceScope(const WorkspaceScope&) = delete;
  WorkspaceScope& operator=(const WorkspaceScope&) = delete;
};

// Bytes of one pinned staging buffer of d2h_staged.
constexpr size_t kPinChunk = size_t(16) << 20;

// Reads `bytes` from device memory into (pageable) host memory through the
// context's two pinned buffers: the copy of chunk k + 1 runs while host threads
// move chunk k into place. Returns when all of it has arrived. Small reads and
// those into page-locked memory go straight to `dst`.
void d2h_staged(Ctx& C, void* dst, const void* src, size_t bytes);
// The same the other way: returns when a pageable `src` has been read (the last
// chunk may still be on its way on the context's stream); a page-locked one is
// read until the stream has passed the copy.
void h2d_staged(Ctx& C, void* dst, const void* src, size_t bytes);

// A surface on the device: sources in tree order, its tree, density buffers
// and the upward-pass work items.
struct DevTree {
  Tree host;
  int n = 0, nn = 0, P1 = 0, Pf = 0;
  DBuf<double> x, y, z, nx, ny, nz, a;
  DBuf<int> perm;
  DBuf<double> tcheb;
  DBuf<double> qx, qy, qz;
  DBuf<double> pk;  // packed records (Pack), up to 12 doubles per source
  DBuf<float> fnx, fny, fnz, fa, fqx, fqy, fqz;  // FP32 copies
  DBuf<double> mom;  // nn * Pf * C, proxy-major (C = 10 DL symmetric form, 6 SL)
  DBuf<float> momf;  // FP32 copy, momf_stride floats per node
  DBuf<MomItem> items;
  DBuf<int> item_start;
  DBuf<double> partial;
  int nitems = 0;
  long long moment_terms = 0;  // sum over non-root nodes of Pf * members
  // fp32: with the FP32 copies that the reduced-precision sums read
  void build(const hr_surface& S, int P, int N0, double theta, bool direct, cudaStream_t st, bool fp32 = true);
  // density (reference order, interleaved, device) -> tree-order SoA (+ moments)
  // and packed records as `pack` (PACK_DL: stresslet moments, otherwise Stokeslet);
  // tc: the upward pass on the tensor cores (reduced-precision operator)
  void set_density(Ctx& C, const double* q3_dev, int pack, bool moments, bool tc = false);
  MomTree mom_tree() const;
};

// set_density of two trees of one degree (t1 may be null), their upward passes in one launch.
void set_densities(Ctx& C, DevTree* t0, DevTree* t1, const double* q0, const double* q1, int pack, bool moments,
                   bool tc);

// Target data on the device, reference order.
struct DevTargets {
  int n = 0;
  DBuf<double> xyz, b, x0, n0, f0, g0;
  DBuf<uint8_t> near;
  DBuf<double> nrm;  // own normals for on-surface targets
};

struct DevLists {
  Lists host;
  DBuf<int> tord;
  DBuf<Entry> entries;
  void build(const Tree& T, int nt, const double* txyz, const uint8_t* near, cudaStream_t st,
             const std::vector<int>* morton = nullptr);
};

struct DevStencils {
  int ne = 0;
  DBuf<int> tgt, idx;
  DBuf<double> pq;
  void build(const Stencils& S, cudaStream_t st);
};

// The order of a batch's items: the lean ones first, each part by decreasing cost,
// equal costs as they stand. Costs are multiples of 1/2 (from 2^30 on compared to
// 31 bits).
std::vector<int> item_order(const std::vector<double>& cost, const std::vector<uint8_t>& lean);

// A batch of boundary sums evaluated together (one or two kernel launches and
// one reduction).
struct Batch {
  int family = F_SL;
  std::vector<EvalTask> tasks;
  std::vector<const Lists*> lists;
  std::vector<const Tree*> trees;  // source tree of each task (member ranges of near entries)
  DBuf<EvalTask> d_tasks;
  DBuf<BlockRef> d_items;
  DBuf<Seg> d_segs;
  DBuf<int> d_item_start;
  DBuf<int2> d_task_blocks;
  DBuf<double> d_partial;
  DBuf<unsigned> d_next;  // work counters of the launches, zero between launches
  int nitems = 0, ntask_blocks = 0;
  int n_on = 0;  // leading lean items (on-surface / box-face tasks, launched on their own)
  bool ready = false;  // finalize has run
  // builds the segments and cost-balanced work items of all tasks
  void finalize(cudaStream_t st, int num_sms = 148);
  void launch(Ctx& C);
};

EvalTask make_task(int kind, double DEL, double scale, const DevTree& T, const DevLists& L,
                   const DevTargets& tg, double* out);

}  // namespace hr

// The C ABI's opaque context.
struct hr_ctx {
  hr::Ctx c;
};
