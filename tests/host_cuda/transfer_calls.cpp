// C calls for the host tests of HostStage (csrc/lib/transfer.cuh).
#include "transfer.cuh"

extern "C" {
void* stage_new() { return new felis::HostStage(); }
void stage_free(void* s) { delete static_cast<felis::HostStage*>(s); }
// Copies bytes0 and bytes1 (at the source) from src0 and src1 with the handle
// on `device`, the caller's thread on `current`; how: 0 down, 1 down and
// widened, 2 up.  Returns the status, and the thread's device afterwards.
int stage_copy(void* s, int how, int device, int current, const void* src0, void* dst0, size_t bytes0, const void* src1,
               void* dst1, size_t bytes1, int* after) {
  FakeStream st{device};
  cudaSetDevice(current);
  const felis::CopyPart parts[2] = {{src0, dst0, bytes0}, {src1, dst1, bytes1}};
  auto* h = static_cast<felis::HostStage*>(s);
  const cudaError_t e = how == 2 ? h->upload(parts, 2, device, &st) : h->download(parts, 2, how == 1, device, &st);
  cudaGetDevice(after);
  cudaSetDevice(0);
  return e;
}
void fail_host_allocations(int on) { fake::fail_host = on; }
int host_allocations() { return fake::host_allocs; }
int host_live() { return fake::host_live; }
}
