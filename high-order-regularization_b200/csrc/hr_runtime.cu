// hr_runtime.cu — device trees, target lists, stencils and evaluation batches.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <numeric>

#include "hr_runtime.h"

namespace hr {

namespace {

// Freed blocks the pool keeps mapped before it returns memory to the CUDA driver.
constexpr uint64_t kPoolKeepBytes = 8ull << 30;
constexpr int kMaxDevices = 64;

struct DevPool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t st = nullptr;  // the pool's own stream: allocations and frees only
};

std::mutex g_pool_mu;
DevPool g_pools[kMaxDevices];

DevPool& pool_of(int dev) {
  HR_REQUIRE(dev >= 0 && dev < kMaxDevices, "device index out of range");
  std::lock_guard<std::mutex> lk(g_pool_mu);
  DevPool& P = g_pools[dev];
  if (!P.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    HR_CHECK_CUDA(cudaMemPoolCreate(&P.pool, &props));
    uint64_t keep = kPoolKeepBytes;
    HR_CHECK_CUDA(cudaMemPoolSetAttribute(P.pool, cudaMemPoolAttrReleaseThreshold, &keep));
    HR_CHECK_CUDA(cudaStreamCreateWithFlags(&P.st, cudaStreamNonBlocking));
  }
  return P;
}

// The workspaces that hold device memory, so that an allocation for which the
// device has no room can have that of contexts which are in no stateless call.
std::mutex g_ws_mu;  // also guards Workspace::busy
std::vector<Workspace*>& g_ws = *new std::vector<Workspace*>;  // never destroyed: a context may outlive static objects

bool release_idle_workspaces(int dev) {
  std::lock_guard<std::mutex> lk(g_ws_mu);
  bool any = false;
  for (Workspace* w : g_ws) {
    if (w->busy || !w->dev || w->device != dev) continue;
    dev_free(w->dev);
    w->dev = nullptr;
    w->dev_cap = 0;
    any = true;
  }
  return any;
}

}  // namespace

void* dev_alloc(size_t bytes) {
  int dev = 0;
  HR_CHECK_CUDA(cudaGetDevice(&dev));
  DevPool& P = pool_of(dev);
  void* p = nullptr;
  cudaError_t e = cudaMallocFromPoolAsync(&p, bytes, P.pool, P.st);
  if (e == cudaErrorMemoryAllocation && release_idle_workspaces(dev)) {
    cudaGetLastError();
    e = cudaMallocFromPoolAsync(&p, bytes, P.pool, P.st);
  }
  HR_CHECK_CUDA(e);
  // complete before any other stream sees the pointer
  HR_CHECK_CUDA(cudaStreamSynchronize(P.st));
  return p;
}

void dev_free(void* p) noexcept {
  if (!p) return;
  try {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess || a.type != cudaMemoryTypeDevice) return;
    int cur = 0;
    cudaGetDevice(&cur);
    if (a.device != cur) cudaSetDevice(a.device);
    cudaDeviceSynchronize();
    DevPool& P = pool_of(a.device);
    cudaFreeAsync(p, P.st);
    if (a.device != cur) cudaSetDevice(cur);
  } catch (...) {
  }
}

Workspace*& active_workspace() {
  static thread_local Workspace* w = nullptr;
  return w;
}

void* Workspace::take(size_t bytes, bool up) {
  bytes = (bytes + 255) & ~size_t(255);
  // a buffer that would not fit a workspace at its limits is no reason to grow it
  if (want_dev + bytes <= kDevMax && (!up || want_pin + bytes <= kPinMax)) {
    want_dev += bytes;
    if (up) want_pin += bytes;
  }
  if (low + bytes > dev_cap - high || (up && low + bytes > pin_cap)) return nullptr;
  if (up) {
    low += bytes;
    return dev + low - bytes;
  }
  high += bytes;
  return dev + dev_cap - high;
}

void Workspace::flush(cudaStream_t st) {
  if (low > flushed) HR_CHECK_CUDA(cudaMemcpyAsync(dev + flushed, pin + flushed, low - flushed, cudaMemcpyHostToDevice, st));
  flushed = low;
}

void Workspace::free_all() {
  std::lock_guard<std::mutex> lk(g_ws_mu);
  g_ws.erase(std::remove(g_ws.begin(), g_ws.end(), this), g_ws.end());
  if (dev) dev_free(dev);
  if (pin) cudaFreeHost(pin);
  dev = pin = nullptr;
  dev_cap = pin_cap = 0;
}

WorkspaceScope::WorkspaceScope(Ctx& c) : C(c) {
  Workspace& w = C.ws;
  {
    std::lock_guard<std::mutex> lk(g_ws_mu);
    w.device = C.device;
    w.busy = true;
    if (std::find(g_ws.begin(), g_ws.end(), &w) == g_ws.end()) g_ws.push_back(&w);
  }
  w.low = w.high = w.flushed = w.want_dev = w.want_pin = 0;
  active_workspace() = &w;
}

WorkspaceScope::~WorkspaceScope() {
  Workspace& w = C.ws;
  active_workspace() = nullptr;
  cudaStreamSynchronize(C.side);
  cudaStreamSynchronize(C.stream);
  // the buffers of this call are idle; the next call finds room for its like
  // (powers of two, so that slowly growing calls do not allocate each time)
  auto grown = [](size_t want, size_t limit) {
    size_t c = size_t(1) << 20;
    while (c < want) c *= 2;
    return std::min(c, limit);
  };
  try {
    if (w.want_dev > w.dev_cap) {
      if (w.dev) dev_free(w.dev);
      w.dev = nullptr;
      w.dev_cap = 0;
      const size_t c = grown(w.want_dev, Workspace::kDevMax);
      w.dev = static_cast<char*>(dev_alloc(c));
      w.dev_cap = c;
    }
    if (w.want_pin > w.pin_cap) {
      if (w.pin) cudaFreeHost(w.pin);
      w.pin = nullptr;
      w.pin_cap = 0;
      const size_t c = grown(w.want_pin, Workspace::kPinMax);
      void* p = nullptr;
      if (cudaMallocHost(&p, c) == cudaSuccess) {
        w.pin = static_cast<char*>(p);
        w.pin_cap = c;
      } else {
        cudaGetLastError();
      }
    }
  } catch (...) {  // no memory to keep: the next call allocates as it goes
  }
  std::lock_guard<std::mutex> lk(g_ws_mu);
  w.busy = false;
}

namespace {

// The two pinned buffers; chunks of an eighth of the copy, 512 KB to kPinChunk.
// 0 where the host gives no page-locked memory: the copy is then a plain one.
size_t staging(Ctx& C, size_t bytes) {
  for (auto& e : C.pin_ev)
    if (!e) HR_CHECK_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  if (!C.pin && cudaMallocHost(&C.pin, 2 * kPinChunk) != cudaSuccess) {
    cudaGetLastError();
    C.pin = nullptr;
    return 0;
  }
  const size_t c = (bytes / 8 + 4095) & ~size_t(4095);
  return std::min(kPinChunk, std::max(size_t(512) << 10, c));
}

void copy_parallel(char* out, const char* in, size_t n) {
  constexpr size_t kPart = size_t(128) << 10;  // bytes per host thread's piece
  const long nparts = (long)((n + kPart - 1) / kPart);
#pragma omp parallel for schedule(static)
  for (long q = 0; q < nparts; q++) {
    const size_t o = (size_t)q * kPart;
    std::memcpy(out + o, in + o, std::min(kPart, n - o));
  }
}

constexpr size_t kStageMin = size_t(1) << 20;  // smaller copies gain nothing from staging

// Whether the copy engines reach the caller's array themselves (page-locked or
// managed memory): a copy by way of the pinned buffers is slower there (21.9 MB
// of grids 719 us instead of 397, a Poisson transform of 95^3 points 560 and 373).
bool page_locked(const void* p, size_t bytes) {
  for (const void* q : {p, static_cast<const void*>(static_cast<const char*>(p) + bytes - 1)}) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, q) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (a.type == cudaMemoryTypeUnregistered) return false;
  }
  return true;
}

}  // namespace

void d2h_staged(Ctx& C, void* dst, const void* src, size_t bytes) {
  cudaStream_t st = C.stream;
  const size_t chunk = bytes < kStageMin || page_locked(dst, bytes) ? 0 : staging(C, bytes);
  if (!chunk) {
    HR_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
    HR_CHECK_CUDA(cudaStreamSynchronize(st));
    return;
  }
  char* buf[2] = {static_cast<char*>(C.pin), static_cast<char*>(C.pin) + kPinChunk};
  const char* s = static_cast<const char*>(src);
  char* d = static_cast<char*>(dst);
  const size_t nch = (bytes + chunk - 1) / chunk;
  auto len = [&](size_t k) { return std::min(chunk, bytes - k * chunk); };
  auto enqueue = [&](size_t k) {
    HR_CHECK_CUDA(cudaMemcpyAsync(buf[k & 1], s + k * chunk, len(k), cudaMemcpyDeviceToHost, st));
    HR_CHECK_CUDA(cudaEventRecord(C.pin_ev[k & 1], st));
  };
  enqueue(0);
  if (nch > 1) enqueue(1);
  for (size_t k = 0; k < nch; k++) {
    HR_CHECK_CUDA(cudaEventSynchronize(C.pin_ev[k & 1]));
    copy_parallel(d + k * chunk, buf[k & 1], len(k));
    if (k + 2 < nch) enqueue(k + 2);
  }
}

void h2d_staged(Ctx& C, void* dst, const void* src, size_t bytes) {
  cudaStream_t st = C.stream;
  const size_t chunk = bytes < kStageMin || page_locked(src, bytes) ? 0 : staging(C, bytes);
  if (!chunk) {
    HR_CHECK_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
    return;
  }
  char* buf[2] = {static_cast<char*>(C.pin), static_cast<char*>(C.pin) + kPinChunk};
  const char* s = static_cast<const char*>(src);
  char* d = static_cast<char*>(dst);
  const size_t nch = (bytes + chunk - 1) / chunk;
  // the buffers may hold the last chunks of an earlier upload
  for (auto& e : C.pin_ev) HR_CHECK_CUDA(cudaEventSynchronize(e));
  for (size_t k = 0; k < nch; k++) {
    const size_t n = std::min(chunk, bytes - k * chunk);
    HR_CHECK_CUDA(cudaEventSynchronize(C.pin_ev[k & 1]));
    copy_parallel(buf[k & 1], s + k * chunk, n);
    HR_CHECK_CUDA(cudaMemcpyAsync(d + k * chunk, buf[k & 1], n, cudaMemcpyHostToDevice, st));
    HR_CHECK_CUDA(cudaEventRecord(C.pin_ev[k & 1], st));
  }
}

void DevTree::build(const hr_surface& S, int P, int N0, double theta, bool direct,
                    cudaStream_t st, bool fp32) {
  HR_REQUIRE(S.n >= 0 && (S.n == 0 || (S.xyz && S.nrml && S.area)), "surface arrays missing");
  HR_REQUIRE(P >= 1 && P + 1 <= 16, "treecode degree P must be in [1, 15]");
  HR_REQUIRE(N0 >= 1, "leaf size N0 must be >= 1");
  host = build_tree(S.n, S.xyz, S.center, P, N0, theta, direct);
  n = S.n;
  nn = host.nnodes();
  P1 = P + 1;
  Pf = P1 * P1 * P1;
  std::vector<double> hx(n), hy(n), hz(n), hnx(n), hny(n), hnz(n), ha(n);
  for (int p = 0; p < n; p++) {
    int o = host.perm[p];
    hx[p] = S.xyz[3 * o];
    hy[p] = S.xyz[3 * o + 1];
    hz[p] = S.xyz[3 * o + 2];
    hnx[p] = S.nrml[3 * o];
    hny[p] = S.nrml[3 * o + 1];
    hnz[p] = S.nrml[3 * o + 2];
    ha[p] = S.area[o];
  }
  x.upload(hx, st);
  y.upload(hy, st);
  z.upload(hz, st);
  nx.upload(hnx, st);
  ny.upload(hny, st);
  nz.upload(hnz, st);
  a.upload(ha, st);
  perm.upload(host.perm, st);
  tcheb.upload(host.tcheb, st);
  qx.alloc(n);
  qy.alloc(n);
  qz.alloc(n);
  pk.alloc(12 * (size_t)n);
  if (fp32) {
    std::vector<float> b0(n), b1(n), b2(n), c0(n);
    for (int p = 0; p < n; p++) {
      b0[p] = (float)hnx[p];
      b1[p] = (float)hny[p];
      b2[p] = (float)hnz[p];
      c0[p] = (float)ha[p];
    }
    fnx.upload(b0, st);
    fny.upload(b1, st);
    fnz.upload(b2, st);
    fa.upload(c0, st);
    fqx.alloc(n);
    fqy.alloc(n);
    fqz.alloc(n);
  }
  if (direct) return;  // no far field
  // upward-pass items: every non-root node (the root's moments stay zero, as
  // in the reference, which skips it: 2S/KITC.cpp:1446), in chunks of sources.
  // Chunks of at most 512 sources, smaller when the tree is small so that the
  // items fill about four CTAs per SM (a multiple of the 32-source K tile).
  std::vector<MomItem> it;
  std::vector<int> start(nn + 1, 0);
  long long members = 0;
  for (int c = 1; c < nn; c++) members += host.m1[c] - host.m0[c] + 1;
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long want = (members + 4LL * sms - 1) / (4LL * sms);
  const int chunk = (int)std::min(512LL, std::max(64LL, (want + 31) / 32 * 32));
  moment_terms = 0;
  for (int c = 0; c < nn; c++) {
    start[c] = (int)it.size();
    if (c == 0) continue;
    for (int s = host.m0[c]; s <= host.m1[c]; s += chunk) {
      MomItem m;
      m.node = c;
      m.s0 = s;
      m.s1 = std::min(host.m1[c] + 1, s + chunk);
      m.out = (int)it.size();
      it.push_back(m);
    }
    moment_terms += (long long)Pf * (host.m1[c] - host.m0[c] + 1);
  }
  start[nn] = (int)it.size();
  nitems = (int)it.size();
  items.upload(it, st);
  item_start.upload(start, st);
  partial.alloc((size_t)std::max(1, nitems) * 12 * Pf);
  mom.alloc((size_t)nn * 12 * Pf);
  mom.zero(st);
  momf.alloc((size_t)nn * momf_stride(host.P + 1, 20));
  momf.zero(st);
}

void Ctx::check_tc() {
  if (!tc_err.p) return;
  int e = 0;
  HR_CHECK_CUDA(cudaMemcpyAsync(&e, tc_err.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
  HR_CHECK_CUDA(cudaStreamSynchronize(stream));
  if (e) {
    tc_err.zero(stream);
    throw Error(HR_ERR_CUDA, "a tensor-core upward pass gave up waiting for its MMAs (bounded wait ran out)");
  }
}

MomTree DevTree::mom_tree() const {
  return {items.p, nitems, nn, item_start.p, tcheb.p, x.p, y.p, z.p, nx.p, ny.p, nz.p, a.p, qx.p, qy.p, qz.p,
          partial.p, mom.p, momf.p};
}

void DevTree::set_density(Ctx& C, const double* q3_dev, int pack, bool moments, bool tc) {
  set_densities(C, this, nullptr, q3_dev, nullptr, pack, moments, tc);
}

void set_densities(Ctx& C, DevTree* t0, DevTree* t1, const double* q0, const double* q1, int pack, bool moments,
                   bool tc) {
  const bool dl = pack == PACK_DL;
  // the packed records are what the FP64 sums read
  auto perm = [&](DevTree* t, const double* q) -> PermTree {
    if (!t) return PermTree{};
    return {t->n,    t->perm.p, q,       t->x.p,  t->y.p,   t->z.p,   t->nx.p,  t->ny.p,
            t->nz.p, t->a.p,    t->qx.p, t->qy.p, t->qz.p,  t->fqx.p, t->fqy.p, t->fqz.p,
            tc ? nullptr : t->pk.p};
  };
  launch_permute(perm(t0, q0), perm(t1, q1), pack, C.stream);
  C.launches++;
  if (!moments || t0->nitems + (t1 ? t1->nitems : 0) == 0) return;
  const MomTree m0 = t0->mom_tree(), m1 = t1 ? t1->mom_tree() : MomTree{};
  int ch = dl ? 9 : 6;
  if (tc && moments_tc_supported(t0->P1)) {
    for (DevTree* t : {t0, t1}) {
      if (!t || t->nitems == 0) continue;
      launch_moments_tc(dl ? 1 : 0, t->items.p, t->nitems, t->P1, t->tcheb.p, t->x.p, t->y.p, t->z.p, t->nx.p, t->ny.p,
                        t->nz.p, t->a.p, t->qx.p, t->qy.p, t->qz.p, t->partial.p, C.tc_err.p, C.stream);
      C.launches++;
    }
    ch = dl ? 12 : 6;
  } else {
    launch_moments(ch, t0->P1, m0, m1, C.stream);
    C.launches++;
  }
  launch_moments_reduce(ch, t0->P1, m0, m1, C.stream);
  C.launches++;
}

void DevLists::build(const Tree& T, int nt, const double* txyz, const uint8_t* near,
                     cudaStream_t st, const std::vector<int>* morton) {
  host = build_lists(T, nt, txyz, near, morton);
  tord.upload(host.tord, st);
  entries.upload(host.entries, st);
}

void DevStencils::build(const Stencils& S, cudaStream_t st) {
  ne = (int)S.tgt.size();
  tgt.upload(S.tgt, st);
  idx.upload(S.idx, st);
  pq.upload(S.pq, st);
}

EvalTask make_task(int kind, double DEL, double scale, const DevTree& T, const DevLists& L,
                   const DevTargets& tg, double* out) {
  EvalTask k;
  memset(&k, 0, sizeof(k));
  k.kind = kind;
  k.jump_mode = 0;
  k.P1 = T.P1;
  k.Pf = T.Pf;
  k.C = (kind == K_DL_ON || kind == K_DL_OFF) ? 10 : 6;
  k.nt = tg.n;
  k.mixed = 0;
  k.DEL = DEL;
  k.scale = scale;
  k.sx = T.x.p;
  k.sy = T.y.p;
  k.sz = T.z.p;
  k.snx = T.nx.p;
  k.sny = T.ny.p;
  k.snz = T.nz.p;
  k.sa = T.a.p;
  k.qx = T.qx.p;
  k.qy = T.qy.p;
  k.qz = T.qz.p;
  k.pk = T.pk.p;
  k.fnx = T.fnx.p;
  k.fny = T.fny.p;
  k.fnz = T.fnz.p;
  k.fa = T.fa.p;
  k.fqx = T.fqx.p;
  k.fqy = T.fqy.p;
  k.fqz = T.fqz.p;
  k.tcheb = T.tcheb.p;
  k.mom = T.mom.p;
  k.momf = T.momf.p;
  k.tord = L.tord.p;
  k.txyz = tg.xyz.p;
  k.tb = tg.b.p;
  k.tnear = tg.near.p;
  k.tf0 = tg.f0.p;
  k.tx0 = tg.x0.p;
  k.tn0 = tg.n0.p;
  k.tg0 = tg.g0.p;
  k.tq = nullptr;
  k.tnrm = tg.nrm.p;
  k.out = out;
  k.entries = L.entries.p;
  k.counters = nullptr;
  return k;
}

namespace {

// Lean kinds (their own launch): on-surface sums, the extend-to-grid box-face sums.
bool lean_kind(int k) {
  return k == K_SL_ON || k == K_DL_ON || k == K_E2G_SL_AWAY || k == K_E2G_P_AWAY || k == K_E2G_UP_AWAY;
}

// Cost of one target-source pair and of one target-proxy pair for a warp, in
// FP64 instructions of the kernels of hr_eval64.cu, or issue slots of the
// reduced-precision two-surface kernels of hr_eval.cu (an off-surface pair: the
// mean of the singular kernel and of the regularized forms). The off-surface
// stresslet's pairs cost 30 or 75, or both where lanes differ; 100 leaves its
// items short (operator at h = 1/32 with 55 / 75 / 100 / 130: 0.760 / 0.752 /
// 0.743 / 0.746 ms).
struct PairCost {
  double direct, proxy;
};
PairCost pair_cost(int kind, int mixed) {
  const bool dl = kind == K_DL_ON || kind == K_DL_OFF, sl = kind == K_SL_ON || kind == K_SL_OFF;
  if (mixed) {
    if (dl || sl) return {kind == K_DL_ON || kind == K_SL_ON ? 24.0 : 60.0, 15.0};
    return {2.0, 1.5};  // the extend-to-grid sums, in relative units
  }
  switch (kind) {
    case K_DL_ON: return {36, 25};
    case K_DL_OFF: return {100, 25};
    case K_SL_ON: return {40, 22};
    case K_SL_OFF: return {50, 22};
    case K_E2G_SL_AWAY:
    case K_E2G_P_AWAY:
    case K_E2G_UP_AWAY: return {28, 0};
    default: return {60, 0};  // the extend-to-grid band
  }
}

}  // namespace

std::vector<int> item_order(const std::vector<double>& cost, const std::vector<uint8_t>& lean) {
  // Stable LSD radix sort, 11 bits per pass, of 2 cost (an integer, cut to 31
  // bits) downwards below a bit for the others, the item's number in the low half.
  // A comparison sort of the items took half of finalize; with it and larger
  // records the first reduced-precision application at h = 1/32 (17,822 items)
  // was 1.62 ms instead of 1.20.
  const size_t n = cost.size();
  double most = 0.0;
  for (double c : cost) most = std::max(most, c);
  uint64_t top = (uint64_t)(2.0 * most);
  int drop = 0, bits = 0;
  while (top >> drop >> 31) drop++;
  top >>= drop;
  while (top >> bits) bits++;
  std::vector<uint64_t> a(n), b(n);
  for (size_t i = 0; i < n; i++)
    a[i] = ((top - ((uint64_t)(2.0 * cost[i]) >> drop)) | (uint64_t)(lean[i] ? 0 : 1) << bits) << 32 | i;
  for (int shift = 32; shift <= 32 + bits; shift += 11) {
    int cnt[2049] = {0};
    for (uint64_t r : a) cnt[((r >> shift) & 2047) + 1]++;
    for (int d = 0; d < 2048; d++) cnt[d + 1] += cnt[d];
    for (uint64_t r : a) b[cnt[(r >> shift) & 2047]++] = r;
    a.swap(b);
  }
  std::vector<int> order(n);
  for (size_t i = 0; i < n; i++) order[i] = (int)(uint32_t)a[i];
  return order;
}

void Batch::finalize(cudaStream_t st, int num_sms) {
  struct HSeg {
    Seg s;
    double cost;
  };
  // The two-surface kernels and the FP64 extend-to-grid ones take work by the
  // warp; the reduced-precision extend-to-grid ones by the CTA.
  const bool mixed = !tasks.empty() && tasks[0].mixed, by_warp = !mixed || family != F_E2G;
  auto entry_warps = [](const Entry& E) {
    int warps = 0;
    for (int w = 0; w < 4; w++) warps += E.mask[w] != 0u;
    return warps;
  };
  // 1. the cost of each launch (lean items, the others)
  double total[2] = {0.0, 0.0};
  for (size_t t = 0; t < tasks.size(); t++) {
    const Lists& L = *lists[t];
    const Tree& T = *trees[t];
    const double Pf = (double)(T.P + 1) * (T.P + 1) * (T.P + 1);
    const PairCost pc = pair_cost(tasks[t].kind, tasks[t].mixed);
    double sum = 0.0;
    // every cost is a multiple of 1/2 far below 2^52: exact in any order
#pragma omp parallel for schedule(dynamic, 16) reduction(+ : sum)
    for (int b = 0; b < L.nblocks(); b++)
      for (int e = L.blk_start[b]; e < L.blk_start[b + 1]; e++) {
        const Entry& E = L.entries[e];
        sum += entry_warps(E) * (E.type == 0 ? Pf * pc.proxy : (T.m1[E.node] + 1 - T.m0[E.node]) * pc.direct);
      }
    total[lean_kind(tasks[t].kind) ? 0 : 1] += sum;
  }
  // 2. the cost of an item (a run of consecutive segments of one block).
  //    Small items keep the tail short. By the CTA: total / (SMs x 4 resident
  //    CTAs x 16 waves), never below two tiles. By the warp: each launch on its
  //    own and with its kinds' costs, in segments no longer than an item and
  //    never below min_src sources (stresslet batch at h = 1/64, P = 6, with
  //    kWaves = 8 / 16 / 24 / 48: FP64 4.06 / 3.87 / 3.89 / 3.92 ms; one
  //    partition for both launches 4.14 ms; the reduced-precision operator 8 /
  //    16 / 32 / 64: 2.80 / 2.61 / 2.64 / 2.68 ms).
  //    The least item: FP64 128 sources, where that leaves a warp fewer than
  //    kFew items fewer, down to 64 (operator at h = 1/14 / 1/18 / 1/24 / 1/32
  //    with 128 throughout 0.174 / 0.220 / 0.343 / 0.738 ms, so 0.136 / 0.192 /
  //    0.322 / 0.740; 64 throughout 0.760 at h = 1/32; kFew = 3 0.341 at h =
  //    1/24, 8 the same as 5). Reduced precision 64: 128 took the operator at h
  //    = 1/16 / 1/24 / 1/32 / 1/64 0.305 / 0.427 / 0.666 / 2.47 ms, 64 0.223 /
  //    0.330 / 0.644 / 2.46 (a near target's FP64 pairs make long units).
  constexpr double kWaves = 16, kFew = 5;
  int min_src[2];
  // Segment lengths are a multiple of this. Reduced precision: of its tiles, so
  // that the FP32 sums of 16 sources do not depend on how the work is cut.
  const int cut = mixed ? 64 : 32;
  double target[2];
  for (int c = 0; c < 2; c++) target[c] = std::max((total[0] + total[1]) / (num_sms * 4.0 * 16.0), 2.0 * 256.0 * 2.0);
  for (int c = 0; c < 2; c++) {
    const double few = 4.0 * total[c] / (num_sms * 16.0 * kFew) / (4.0 * 36.0);  // sources
    min_src[c] = mixed ? 64 : std::max(64, (int)std::min(128.0, few) / 32 * 32);
    if (by_warp)
      target[c] = std::max(4.0 * total[c] / (num_sms * 16.0 * kWaves), 4.0 * min_src[c] * (mixed ? 24.0 : 36.0));
  }
  // 3. segments: a far entry whole, a near entry cut into source ranges of at
  //    most 512; cost ~ active warps x pair evaluations.
  std::vector<std::vector<std::vector<HSeg>>> per(tasks.size());
  for (size_t t = 0; t < tasks.size(); t++) {
    const Lists& L = *lists[t];
    const Tree& T = *trees[t];
    const double Pf = (double)(T.P + 1) * (T.P + 1) * (T.P + 1);
    const PairCost pc = pair_cost(tasks[t].kind, tasks[t].mixed);
    const double want = target[lean_kind(tasks[t].kind) ? 0 : 1];
    const int least = min_src[lean_kind(tasks[t].kind) ? 0 : 1];
    const int seg = by_warp ? std::min(512, std::max(least, (int)(want / (4.0 * pc.direct)) / cut * cut)) : 512;
    per[t].resize(L.nblocks());
#pragma omp parallel for schedule(dynamic, 16)
    for (int b = 0; b < L.nblocks(); b++) {
      per[t][b].reserve(2 * (L.blk_start[b + 1] - L.blk_start[b]));
      for (int e = L.blk_start[b]; e < L.blk_start[b + 1]; e++) {
        const Entry& E = L.entries[e];
        const int warps = entry_warps(E);
        if (E.type == 0) {
          per[t][b].push_back({Seg{e, 0, 0}, warps * Pf * pc.proxy});
        } else {
          for (int s0 = T.m0[E.node]; s0 <= T.m1[E.node]; s0 += seg) {
            const int s1 = std::min(T.m1[E.node] + 1, s0 + seg);
            per[t][b].push_back({Seg{e, s0, s1}, warps * (double)(s1 - s0) * pc.direct});
          }
        }
      }
    }
  }
  // Blocks in task order; each block's runs are formed on its own (in
  // parallel), then offsets give every segment and item (slot) the position
  // a serial pass over the blocks would give it.
  std::vector<int2> tblocks;
  for (size_t t = 0; t < tasks.size(); t++)
    for (int b = 0; b < (int)per[t].size(); b++) tblocks.push_back(make_int2((int)t, b));
  const long nbt = (long)tblocks.size();
  std::vector<std::vector<std::pair<int, double>>> runs(nbt);  // per block: (segments, cost) per item
#pragma omp parallel for schedule(dynamic, 64)
  for (long q = 0; q < nbt; q++) {
    const auto& v = per[tblocks[q].x][tblocks[q].y];
    const double want = target[lean_kind(tasks[tblocks[q].x].kind) ? 0 : 1];
    size_t i = 0;
    while (i < v.size()) {
      double c = 0.0;
      int n = 0;
      do {
        c += v[i].cost;
        i++;
        n++;
      } while (i < v.size() && c + v[i].cost <= want);
      runs[q].push_back({n, c});
    }
    // a block without work still gets one (empty) item so that its partial
    // slot is written
    if (v.empty()) runs[q].push_back({0, 0.0});
  }
  std::vector<long> seg_off(nbt + 1, 0), slot_off(nbt + 1, 0);
  for (long q = 0; q < nbt; q++) {
    seg_off[q + 1] = seg_off[q] + (long)per[tblocks[q].x][tblocks[q].y].size();
    slot_off[q + 1] = slot_off[q] + (long)runs[q].size();
  }
  HR_REQUIRE(seg_off[nbt] < (1L << 31) && slot_off[nbt] < (1L << 31), "batch too large for 32-bit segment indices");
  std::vector<Seg> segs(seg_off[nbt]);
  std::vector<BlockRef> items(slot_off[nbt]);
  std::vector<double> cost(slot_off[nbt]);
  std::vector<uint8_t> lean(slot_off[nbt]);
#pragma omp parallel for schedule(dynamic, 64)
  for (long q = 0; q < nbt; q++) {
    const int t = tblocks[q].x, b = tblocks[q].y;
    const auto& v = per[t][b];
    int sg = (int)seg_off[q], it = (int)slot_off[q];
    size_t i = 0;
    for (const auto& r : runs[q]) {
      BlockRef ref{t, b, sg, sg + r.first, it};
      for (int k = 0; k < r.first; k++) segs[sg++] = v[i++].s;
      items[it] = ref;
      lean[it] = lean_kind(tasks[t].kind);
      cost[it++] = r.second;
    }
  }
  // per task: the slot of each block's first item, then the task's end
  std::vector<int> starts;
  std::vector<size_t> start_off(tasks.size());
  int slot = (int)slot_off[nbt];
  {
    long q = 0;
    for (size_t t = 0; t < tasks.size(); t++) {
      start_off[t] = starts.size();
      for (int b = 0; b < (int)per[t].size(); b++, q++) starts.push_back((int)slot_off[q]);
      starts.push_back((int)slot_off[q]);
    }
  }
  // lean items first (their own launch: on-surface kinds, or the extend-to-grid
  // box-face sums), each part by decreasing cost
  const std::vector<int> order = item_order(cost, lean);
  std::vector<BlockRef> br(items.size());
  for (size_t i = 0; i < items.size(); i++) br[i] = items[order[i]];
  n_on = (int)std::count(lean.begin(), lean.end(), 1);
  nitems = (int)br.size();
  ntask_blocks = (int)tblocks.size();
  d_items.upload(br, st);
  d_segs.upload(segs, st);
  d_item_start.upload(starts, st);
  d_task_blocks.upload(tblocks, st);
  d_partial.alloc((size_t)std::max(1, slot) * kTB * kPartComps);
  d_next.alloc(2);
  d_next.zero(st);
  // the FP64 kernels stage one smoothing table per launch
  for (const EvalTask& t : tasks) HR_REQUIRE(t.DEL == tasks[0].DEL, "the tasks of a batch share one delta");
  for (size_t t = 0; t < tasks.size(); t++) {
    tasks[t].item_start = d_item_start.p + start_off[t];
    tasks[t].partial = d_partial.p;
  }
  d_tasks.upload(tasks, st);
  ready = true;
}

void Batch::launch(Ctx& C) {
  const bool two = n_on > 0 && nitems > n_on;
  cudaStream_t side = two ? C.side : C.stream;
  if (two) {
    HR_CHECK_CUDA(cudaEventRecord(C.ev_fork, C.stream));
    HR_CHECK_CUDA(cudaStreamWaitEvent(C.side, C.ev_fork, 0));
  }
  if (!tasks.empty() && tasks[0].mixed) launch_eval(family, d_tasks.p, d_items.p, d_segs.p, nitems, n_on, d_next.p, C.num_sms, C.stream, side);
  else
    launch_eval64(family, d_tasks.p, d_items.p, d_segs.p, nitems, n_on, d_next.p, C.num_sms, C.stream, side,
                  C.count_work);
  if (two) {
    HR_CHECK_CUDA(cudaEventRecord(C.ev_join, C.side));
    HR_CHECK_CUDA(cudaStreamWaitEvent(C.stream, C.ev_join, 0));
  }
  launch_reduce(d_tasks.p, ntask_blocks, d_task_blocks.p, d_next.p, C.stream);
  C.launches += 1 + (n_on > 0 ? 1 : 0) + (nitems > n_on ? 1 : 0);
}

}  // namespace hr
