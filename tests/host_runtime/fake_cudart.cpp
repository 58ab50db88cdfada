// The CUDA runtime calls of csrc/hr_runtime.cu on host memory, for tests of its
// host logic without a GPU: every stream is in order, "device" memory is
// malloc'd, allocations fail on request.
#include "fake_cudart.h"

#include <cstdlib>
#include <cstring>

Fake fake;

namespace {
cudaError_t last = cudaSuccess;
cudaError_t fail(cudaError_t e) { return last = e; }
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { return *p = (cudaMemPool_t)1, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? cudaSuccess : fail(cudaErrorInvalidResourceHandle); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : fail(cudaErrorInvalidResourceHandle); }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }

cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) {
  if (fake.device + n > fake.device_limit) return fail(cudaErrorMemoryAllocation);
  *p = malloc(n);
  fake.device += n;
  fake.size[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeUnregistered;
  for (const auto& m : fake.size)
    if (p >= m.first && p < (const char*)m.first + m.second) a->type = cudaMemoryTypeDevice;
  for (const auto& m : fake.locked)
    if (p >= m.first && p < (const char*)m.first + m.second) a->type = cudaMemoryTypeHost;
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
  fake.device -= fake.size[p];
  fake.size.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  if (fake.no_pinned) return fail(cudaErrorMemoryAllocation);
  *p = malloc(n);
  fake.locked[*p] = n;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  fake.locked.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  fake.copies++;
  memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return cudaSuccess;
}
}

// the kernels, which these tests never reach
#include "../../high-order-regularization_b200/csrc/hr_device.h"
namespace hr {
void launch_eval(int, const EvalTask*, const BlockRef*, const Seg*, int, int, unsigned*, int, cudaStream_t, cudaStream_t) { abort(); }
void launch_eval64(int, const EvalTask*, const BlockRef*, const Seg*, int, int, unsigned*, int, cudaStream_t, cudaStream_t, bool) { abort(); }
void launch_reduce(const EvalTask*, int, const int2*, unsigned*, cudaStream_t) { abort(); }
bool moments_tc_supported(int) { abort(); }
void launch_moments_tc(int, const MomItem*, int, int, const double*, const double*, const double*, const double*, const double*,
                       const double*, const double*, const double*, const double*, const double*, const double*, double*, int*,
                       cudaStream_t) { abort(); }
void launch_moments(int, int, const MomTree&, const MomTree&, cudaStream_t) { abort(); }
void launch_moments_reduce(int, int, const MomTree&, const MomTree&, cudaStream_t) { abort(); }
void launch_permute(const PermTree&, const PermTree&, int, cudaStream_t) { abort(); }
}  // namespace hr
