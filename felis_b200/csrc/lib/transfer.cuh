// Large copies between the device and pageable host memory.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace felis {

// A host table to the device ahead of work on `st`: copied on that stream, and
// there when the call returns.  cudaMemcpy runs on the default stream, for which
// the non-blocking streams of handles, ensembles and networks do not wait, and
// from pageable memory it returns once the bytes are staged.
inline cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
}

struct CopyPart {
  const void* src;
  void* dst;
  size_t bytes;  // at the source (a multiple of 4)
};

// Page-locked slots of one handle, ensemble or network, made when its copies
// have come to kLockAfter bytes and freed with it (16 MB at most).  One call at
// a time, like its owner.
class HostStage {
 public:
  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;
  ~HostStage();
  // Copies every part to the host, FP32 values widened to FP64 when `widen`
  // (the destination then holds twice the bytes).  Returns when all is there.
  cudaError_t download(const CopyPart* parts, int nparts, bool widen, int device, cudaStream_t st);
  // Copies every part to the device.  Returns when all is there.
  cudaError_t upload(const CopyPart* parts, int nparts, int device, cudaStream_t st);

 private:
  static constexpr int kThreads = 8, kSlots = 2;
  static constexpr size_t kChunk = (size_t)1 << 20;
  // bytes at the destination for which plain copies cost what the slots do
  static constexpr size_t kLockAfter = (size_t)64 << 20;
  char* pinned_ = nullptr;  // [threads_][kSlots][kChunk]
  cudaEvent_t ev_[kThreads][kSlots] = {};
  int threads_ = 0;
  size_t moved_ = 0;  // bytes at the destination so far
  cudaError_t reserve(int threads);
  enum Mode { kDown, kDownWiden, kUp };
  cudaError_t run(const CopyPart* parts, int nparts, Mode mode, int device, cudaStream_t st);
};

}  // namespace felis
