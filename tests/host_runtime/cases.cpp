// Host logic of csrc/hr_runtime.{h,cu} against fake_cudart.cpp; one case per run.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>

#include "../../high-order-regularization_b200/csrc/hr_runtime.h"
#include "fake_cudart.h"

using namespace hr;

#define CHECK(c)                                                    \
  do {                                                              \
    if (!(c)) {                                                     \
      printf("%s:%d: %s\n", __FILE__, __LINE__, #c);                \
      exit(1);                                                      \
    }                                                               \
  } while (0)

template <class F>
bool throws(F&& f) {
  try {
    f();
  } catch (const Error&) {
    return true;
  }
  return false;
}

// Buffers whose growth fails half way are allocated again by the next call, of
// whatever size, and the failure is reported once.
void failed_growth() {
  DBuf<double> a, b;
  int cap = 0;
  auto ensure = [&](int n) {
    grow(cap, n, [&] {
      a.alloc(n);
      b.alloc(1000 * (size_t)n);
    });
  };
  ensure(10);
  CHECK(a.n == 10 && b.n == 10000 && cap == 10);
  double* p = b.p;
  ensure(7);
  CHECK(b.p == p);
  fake.device_limit = 1000000;
  CHECK(throws([&] { ensure(1000); }));
  CHECK(!b.p && cap == 0);
  CHECK(cudaGetLastError() == cudaSuccess);
  ensure(7);
  CHECK(a.p && b.p && b.n == 7000 && cap == 7);
}

// A copy between page-locked memory and the device is one copy, of pageable memory
// one per chunk; what arrives is the same.
void page_locked_copies() {
  Ctx C;
  const size_t n = size_t(5) << 20;
  void *a, *b, *d;
  cudaMallocHost(&a, n);
  cudaMallocHost(&b, n);
  d = dev_alloc(n);
  std::vector<char> u(n), v(n);
  for (size_t i = 0; i < n; i++) u[i] = static_cast<char*>(a)[i] = (char)(i * 7 + i / 1000);
  auto copies = [&](const void* src, void* dst) {
    memset(d, 0, n);
    memset(dst, 0, n);
    const int c0 = fake.copies;
    h2d_staged(C, d, src, n);
    const int c1 = fake.copies;
    d2h_staged(C, dst, d, n);
    CHECK(!memcmp(dst, u.data(), n));
    return std::make_pair(c1 - c0, fake.copies - c1);
  };
  CHECK(copies(a, b) == std::make_pair(1, 1));
  CHECK(copies(u.data(), v.data()).first > 1 && copies(u.data(), v.data()).second > 1);
  CHECK(copies(a, v.data()).first == 1 && copies(u.data(), b).second == 1);
}

// Without page-locked memory large copies are plain ones; once there is some
// they are staged.
void no_page_locked_memory() {
  Ctx C;
  const size_t n = size_t(3) << 20;
  std::vector<char> u(n, 5), v(n);
  void* d = dev_alloc(n);
  fake.no_pinned = true;
  h2d_staged(C, d, u.data(), n);
  d2h_staged(C, v.data(), d, n);
  CHECK(u == v && fake.copies == 2);
  CHECK(cudaGetLastError() == cudaSuccess);
  fake.no_pinned = false;
  v.assign(n, 0);
  d2h_staged(C, v.data(), d, n);
  CHECK(u == v && fake.copies > 4);
}

// The workspace grows to what a call's buffers can use of it, not for those that
// no workspace holds; the others fit it from the next call on.
void workspace_growth() {
  Ctx C;
  const size_t big = Workspace::kDevMax + 1, mid = size_t(40) << 20;
  auto call = [&](std::vector<size_t> sizes, bool up = false) {
    WorkspaceScope scope(C);
    std::vector<DBuf<char>> b(sizes.size());
    std::vector<char> h(1000000);
    std::vector<bool> borrowed;
    for (size_t i = 0; i < sizes.size(); i++) {
      if (up) b[i].upload(h.data(), sizes[i], 0);
      else b[i].alloc(sizes[i]);
      borrowed.push_back(b[i].borrowed);
    }
    return borrowed;
  };
  const std::vector<bool> none(1, false), yes(1, true);
  CHECK(call({big}) == none && C.ws.dev_cap == 0 && fake.device == 0);
  CHECK(call({big, 1000}) == std::vector<bool>(2, false) && C.ws.dev_cap == size_t(1) << 20);
  CHECK(call({big, 1000}) == std::vector<bool>({false, true}));
  CHECK(call({mid, big, mid}) == std::vector<bool>(3, false) && C.ws.dev_cap == size_t(128) << 20);
  CHECK(call({mid, big, mid}) == std::vector<bool>({true, false, true}));
  // seven of 40 MB: six fit
  CHECK(call(std::vector<size_t>(7, mid)).back() == false && C.ws.dev_cap == Workspace::kDevMax);
  CHECK(call(std::vector<size_t>(7, mid)) == std::vector<bool>({true, true, true, true, true, true, false}));
  // uploads need page-locked room as well: 33 of 1 MB fit its 32 MB
  call(std::vector<size_t>(40, 1000000), true);
  CHECK(C.ws.pin_cap == Workspace::kPinMax);
  auto b = call(std::vector<size_t>(40, 1000000), true);
  CHECK(std::count(b.begin(), b.end(), true) == 33 && b[0] && !b[39]);
  CHECK(fake.device == C.ws.dev_cap);
  C.ws.free_all();
  CHECK(fake.device == 0 && fake.locked.empty());
}

// An allocation that does not fit gets the memory of the contexts between calls,
// not that of one in a call; the next call has its workspace again.
void workspace_given_back() {
  Ctx A, B;
  const size_t mb = size_t(1) << 20;
  auto call = [&](Ctx& C, auto&& inside) {
    WorkspaceScope scope(C);
    DBuf<char> b;
    b.alloc(3 * mb);
    b.zero(0);
    inside();
    return b.borrowed;
  };
  auto nothing = [] {};
  for (Ctx* C : {&A, &B})
    for (int i = 0; i < 2; i++) call(*C, nothing);
  CHECK(fake.device == 8 * mb && call(A, nothing) && call(B, nothing));
  fake.device_limit = 10 * mb;
  void* p = nullptr;
  const bool had = call(B, [&] { p = dev_alloc(5 * mb); });  // takes A's, leaves B's
  CHECK(had && p && !A.ws.dev && B.ws.dev && fake.device == 9 * mb);
  CHECK(throws([&] { call(B, [&] { dev_alloc(5 * mb); }); }));
  CHECK(B.ws.dev && cudaGetLastError() == cudaSuccess);
  dev_free(p);
  CHECK(!call(A, nothing) && call(A, nothing) && call(B, nothing));
  A.ws.free_all();
  B.ws.free_all();
  CHECK(fake.device == 0);
  CHECK(throws([&] { dev_alloc(11 * mb); }));
}

// The items' order is that of a stable comparison sort.
void order_of_items() {
  unsigned r = 1;
  auto next = [&] { return r = r * 1664525u + 1013904223u, r >> 8; };
  for (int n : {0, 1, 2, 17, 5000})
    for (double most : {0.5, 3.0, 2047.5, 2048.0, 1e6, 1e9}) {
      std::vector<double> cost(n);
      std::vector<uint8_t> lean(n);
      for (int i = 0; i < n; i++) {
        cost[i] = i % 5 ? 0.5 * std::floor(2.0 * most * ((next() % 1000) / 999.0)) : 0.0;
        lean[i] = next() % 3 == 0;
      }
      std::vector<int> want(n);
      for (int i = 0; i < n; i++) want[i] = i;
      std::stable_sort(want.begin(), want.end(),
                       [&](int x, int y) { return lean[x] != lean[y] ? lean[x] > lean[y] : cost[x] > cost[y]; });
      CHECK(item_order(cost, lean) == want);
    }
}

int main(int, char** argv) {
  const std::string c = argv[1];
  if (c == "failed_growth") failed_growth();
  else if (c == "page_locked_copies") page_locked_copies();
  else if (c == "no_page_locked_memory") no_page_locked_memory();
  else if (c == "workspace_growth") workspace_growth();
  else if (c == "workspace_given_back") workspace_given_back();
  else if (c == "order_of_items") order_of_items();
  else return 2;
  return 0;
}
