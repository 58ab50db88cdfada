#pragma once
#include <cuda_runtime.h>

#include <map>

struct Fake {
  size_t device = 0, device_limit = size_t(1) << 40;  // bytes of device memory in use and in all
  bool no_pinned = false;                             // page-locked allocations fail
  int copies = 0;                                     // cudaMemcpyAsync calls so far
  std::map<const void*, size_t> size, locked;         // device and page-locked blocks
};
extern Fake fake;
