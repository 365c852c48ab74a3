// A CUDA runtime on the host, for tests of what the library's host code asks of it: kernels are counted and not run,
// allocations are zeroed host memory whose total is kept, and copies to and from the device take place as late as a
// runtime may do them, when their stream is next synchronised. Linked with the library's object files in place of the
// CUDA runtime (tests/test_host_runtime.py); one thread, and all streams are one queue.
#pragma once

#include <cuda_runtime_api.h>

#include <math.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

template <class T> T __ldg(T const * p) { return *p; }  // (the library's headers name it)

namespace fake {

struct State {
  size_t now = 0, peak = 0;                  // device bytes allocated
  int allocations = 0;
  std::map<void *, size_t> sizes;            // live device allocations
  std::vector<std::function<void()>> queue;  // work not yet done
  std::map<void const *, std::string> names; // kernels by host entry point
  std::vector<std::string> launches;         // mangled names, in order
  std::function<void(std::string const &, void **)> on_launch;  // sees each launch's name and arguments
};
inline State & state() {
  static State s;
  return s;
}
inline void drain() {
  for (auto & f : state().queue) f();
  state().queue.clear();
}
inline cudaError_t allocate(void ** p, size_t n) {
  *p = std::calloc(std::max<size_t>(n, 1) + 256, 1);
  if (!*p) return cudaErrorMemoryAllocation;
  State & s = state();
  s.sizes[*p] = n;
  ++s.allocations;
  s.now += n;
  s.peak = std::max(s.peak, s.now);
  return cudaSuccess;
}
inline cudaError_t release(void * p) {
  State & s = state();
  auto it = s.sizes.find(p);
  if (it == s.sizes.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  s.now -= it->second;
  s.sizes.erase(it);
  s.queue.push_back([p] { std::free(p); });  // stream-ordered: after the work queued so far
  return cudaSuccess;
}
inline int launches_of(char const * name) {
  int n = 0;
  for (auto const & l : state().launches) n += l.find(name) != std::string::npos;
  return n;
}

}  // namespace fake

extern "C" {

cudaError_t cudaMalloc(void ** p, size_t n) { return fake::allocate(p, n); }
cudaError_t cudaMallocHost(void ** p, size_t n) { return (*p = std::calloc(n, 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void * p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void ** p, size_t n, cudaMemPool_t, cudaStream_t) { return fake::allocate(p, n); }
cudaError_t cudaMallocAsync(void ** p, size_t n, cudaStream_t) { return fake::allocate(p, n); }
cudaError_t cudaFreeAsync(void * p, cudaStream_t) { return fake::release(p); }
cudaError_t cudaFree(void * p) { return fake::release(p); }
cudaError_t cudaMemcpyAsync(void * dst, void const * src, size_t n, cudaMemcpyKind, cudaStream_t) {
  fake::state().queue.push_back([=] { std::memcpy(dst, src, n); });
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void * p, int v, size_t n, cudaStream_t) {
  fake::state().queue.push_back([=] { std::memset(p, v, n); });
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { fake::drain(); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { fake::drain(); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { fake::drain(); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t * e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float * ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaGetDevice(int * d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
char const * cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int * v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int * n, void const *, int, size_t) { *n = 4; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int * n, void const *, int, size_t, unsigned) {
  *n = 4;
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus * s) {
  *s = cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t * p, cudaMemPoolProps const *) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
// every pointer counts as device memory
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes * a, void const *) {
  std::memset(a, 0, sizeof(*a));
  a->type = cudaMemoryTypeDevice;
  return cudaSuccess;
}

// what the compiler's launch code calls
static dim3 fake_grid, fake_block;
void ** __cudaRegisterFatBinary(void *) { static void * h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, char const * host, char *, char const * name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
  fake::state().names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, char const *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 * g, dim3 * b, size_t * m, void * s) {
  *g = fake_grid;
  *b = fake_block;
  *m = 0;
  *(void **)s = nullptr;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t * k, void const * host) { *k = (cudaKernel_t)host; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void ** args, size_t, cudaStream_t) {
  std::string const & name = fake::state().names[(void const *)k];
  fake::state().launches.push_back(name);
  if (fake::state().on_launch) fake::state().on_launch(name, args);
  return cudaSuccess;
}

}  // extern "C"
