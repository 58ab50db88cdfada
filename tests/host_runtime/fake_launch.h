#pragma once
#include <cuda_runtime.h>

#include <functional>
#include <map>

struct FakeLaunch {
  std::map<const void*, size_t> limit;  // dynamic shared memory that a kernel may be launched with
  int launches = 0, refused = 0;
  size_t most = 0;                    // largest dynamic shared memory of a launch
  std::function<void()> between;      // run once, after the next limit is set
};
extern FakeLaunch fake_launch;
