// The few CUDA runtime calls of csrc/lib/transfer.cu on the host, with two
// devices: a current device per thread, streams and events that belong to a
// device, and page-locked allocations that can be made to fail.
#pragma once

#include <stddef.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorInvalidResourceHandle = 400 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
constexpr unsigned cudaEventDisableTiming = 2;
struct FakeStream { int device; };
struct FakeEvent { int device; };
typedef FakeStream* cudaStream_t;
typedef FakeEvent* cudaEvent_t;

namespace fake {
inline thread_local int current = 0;
inline std::atomic<int> host_allocs{0}, host_live{0}, fail_host{0}, copies{0};
}  // namespace fake

inline cudaError_t cudaGetDevice(int* d) { *d = fake::current; return cudaSuccess; }
inline cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d > 1) return cudaErrorInvalidValue;
  fake::current = d;
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
template <class T>
cudaError_t cudaMallocHost(T** p, size_t n) {
  ++fake::host_allocs;
  if (fake::fail_host) { *p = nullptr; return cudaErrorMemoryAllocation; }
  ++fake::host_live;
  *p = static_cast<T*>(malloc(n));
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
  --fake::host_live;
  free(p);
  return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = new FakeEvent{fake::current}; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  return e->device == s->device ? cudaSuccess : cudaErrorInvalidResourceHandle;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  ++fake::copies;
  memcpy(d, s, n);
  return cudaSuccess;
}
