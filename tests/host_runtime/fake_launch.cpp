// Kernel launches without a GPU: nothing runs, but a launch with more dynamic shared
// memory than its kernel's limit is refused, as by the CUDA runtime. The limit
// belongs to the kernel (on a device), whichever thread or plan set it last.
#include "fake_launch.h"

#include <utility>

FakeLaunch fake_launch;

namespace {
struct Config {
  dim3 grid, block;
  size_t shared;
  cudaStream_t stream;
} config;
}  // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* handle;
  return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
  config = {grid, block, shared, stream};
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, cudaStream_t* stream) {
  *grid = config.grid;
  *block = config.block;
  *shared = config.shared;
  *stream = config.stream;
  return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int value) {
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fake_launch.limit[fn] = value;
  if (fake_launch.between) std::exchange(fake_launch.between, nullptr)();
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3, dim3, void**, size_t shared, cudaStream_t) {
  const auto l = fake_launch.limit.find(fn);
  fake_launch.launches++;
  fake_launch.most = shared > fake_launch.most ? shared : fake_launch.most;
  if (shared <= (l == fake_launch.limit.end() ? size_t(48) << 10 : l->second)) return cudaSuccess;
  fake_launch.refused++;
  return cudaErrorInvalidValue;
}
}
