// Large copies between the device and pageable host memory.
//
// The driver moves them through its own bounce buffer on one thread, which
// also takes the destination's page faults: 171 MB of field planes took 30 ms
// that way, and 140 ms with a copy and a conversion per slice.  Here several
// threads each move 1 MB chunks through two page-locked slots of their own: one
// chunk crosses the link while the thread copies (or widens) another, and the
// page faults spread over the threads.
#include "transfer.cuh"

#include <string.h>

#include <algorithm>
#include <atomic>
#include <system_error>
#include <thread>
#include <vector>

namespace felis {

namespace {

// `device` current in this thread (the events are made on it and belong to it),
// and the caller's device current again at the end.
struct OnDevice {
  int was = -1;
  cudaError_t status;
  explicit OnDevice(int device) {
    status = cudaGetDevice(&was);
    if (status != cudaSuccess) was = -1;
    else if (was == device) was = -1;
    else status = cudaSetDevice(device);
  }
  ~OnDevice() {
    if (was >= 0) cudaSetDevice(was);
  }
  OnDevice(const OnDevice&) = delete;
  OnDevice& operator=(const OnDevice&) = delete;
};

}  // namespace

HostStage::~HostStage() {
  for (auto& t : ev_)
    for (cudaEvent_t e : t)
      if (e) cudaEventDestroy(e);
  if (pinned_) cudaFreeHost(pinned_);
}

cudaError_t HostStage::reserve(int threads) {
  if (threads <= threads_) return cudaSuccess;
  if (pinned_) cudaFreeHost(pinned_);
  pinned_ = nullptr;
  threads_ = 0;
  cudaError_t e = cudaMallocHost(&pinned_, (size_t)threads * kSlots * kChunk);
  for (int t = 0; t < threads; ++t)
    for (int s = 0; s < kSlots; ++s)
      if (e == cudaSuccess && !ev_[t][s]) e = cudaEventCreateWithFlags(&ev_[t][s], cudaEventDisableTiming);
  if (e == cudaSuccess) threads_ = threads;
  return e;
}

cudaError_t HostStage::run(const CopyPart* parts, int nparts, Mode mode, int device, cudaStream_t st) {
  std::vector<CopyPart> chunks;
  size_t total = 0;
  for (int p = 0; p < nparts; ++p)
    for (size_t o = 0; o < parts[p].bytes; o += kChunk) {
      const size_t n = std::min(kChunk, parts[p].bytes - o);
      chunks.push_back({static_cast<const char*>(parts[p].src) + o,
                        static_cast<char*>(parts[p].dst) + (mode == kDownWiden ? 2 * o : o), n});
      total += n;
    }
  if (!total) return cudaSuccess;
  const OnDevice here(device);
  if (here.status != cudaSuccess) return here.status;
  if (!pinned_ && total < kChunk && mode != kDownWiden) {
    // too little to page-lock memory for (2 ms)
    for (const CopyPart& c : chunks) {
      const cudaError_t x = mode == kUp ? cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyHostToDevice, st)
                                        : cudaMemcpyAsync(c.dst, c.src, c.bytes, cudaMemcpyDeviceToHost, st);
      if (x != cudaSuccess) return x;
    }
    return cudaStreamSynchronize(st);
  }
  // one thread per 4 MB, as far as the machine has cores
  const int cores = std::max(1, (int)std::thread::hardware_concurrency());
  const int threads = (int)std::min<size_t>(std::min(kThreads, cores), (total >> 22) + 1);
  cudaError_t e = reserve(threads);
  if (e != cudaSuccess) return e;
  std::atomic<size_t> next{0};
  std::atomic<int> status{cudaSuccess};
  auto work = [&](int t) {
    char* slot = pinned_ + (size_t)t * kSlots * kChunk;
    size_t held[kSlots] = {};
    bool busy[kSlots] = {};  // a copy through the slot is in flight
    auto fail = [&](cudaError_t x) {
      int ok = cudaSuccess;
      if (x != cudaSuccess) status.compare_exchange_strong(ok, x);
      return x != cudaSuccess;
    };
    // waits for the slot's copy; a download then goes on to its destination
    auto finish = [&](int s) {
      busy[s] = false;
      if (fail(cudaEventSynchronize(ev_[t][s])) || mode == kUp) return;
      const CopyPart& c = chunks[held[s]];
      const char* from = slot + (size_t)s * kChunk;
      if (mode == kDown) {
        memcpy(c.dst, from, c.bytes);
      } else {
        const float* f = reinterpret_cast<const float*>(from);
        double* d = static_cast<double*>(c.dst);
        for (size_t k = 0; k < c.bytes / sizeof(float); ++k) d[k] = f[k];
      }
    };
    if (t && fail(cudaSetDevice(device))) return;
    int s = 0;
    for (size_t i; status == cudaSuccess && (i = next++) < chunks.size(); s = (s + 1) % kSlots) {
      if (busy[s]) finish(s);
      const CopyPart& c = chunks[i];
      char* at = slot + (size_t)s * kChunk;
      held[s] = i;
      if (mode == kUp) memcpy(at, c.src, c.bytes);
      if (fail(mode == kUp ? cudaMemcpyAsync(c.dst, at, c.bytes, cudaMemcpyHostToDevice, st)
                           : cudaMemcpyAsync(at, c.src, c.bytes, cudaMemcpyDeviceToHost, st)))
        break;
      if (fail(cudaEventRecord(ev_[t][s], st))) break;
      busy[s] = true;
      // the other slot's copy was issued before this one
      const int o = (s + 1) % kSlots;
      if (mode != kUp && busy[o]) finish(o);
    }
    for (int k = 0; k < kSlots; ++k)
      if (busy[k]) finish(k);
  };
  std::vector<std::thread> pool;
  try {
    for (int t = 1; t < threads; ++t) pool.emplace_back(work, t);
  } catch (const std::system_error&) {
    // fewer threads: the chunks go to those that started
  }
  work(0);
  for (std::thread& t : pool) t.join();
  if (status != cudaSuccess) cudaStreamSynchronize(st);  // nothing stays in flight through the slots
  return (cudaError_t)status.load();
}

cudaError_t HostStage::download(const CopyPart* parts, int nparts, bool widen, int device, cudaStream_t st) {
  return run(parts, nparts, widen ? kDownWiden : kDown, device, st);
}

cudaError_t HostStage::upload(const CopyPart* parts, int nparts, int device, cudaStream_t st) {
  return run(parts, nparts, kUp, device, st);
}

}  // namespace felis
