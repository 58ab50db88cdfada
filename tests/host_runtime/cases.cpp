// Host logic of csrc/hr_runtime.{h,cu} against fake_cudart.cpp; one case per run.
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

int main(int, char** argv) {
  const std::string c = argv[1];
  if (c == "failed_growth") failed_growth();
  else return 2;
  return 0;
}
