// Large copies between the device and pageable host memory.
//
// The driver moves them through its own bounce buffer on one thread, which
// also takes the destination's page faults: 171 MB of field planes took 30 ms
// that way, and 140 ms with a copy and a conversion per slice.  Here several
// threads each move 1 MB chunks through two page-locked slots of their own: one
// chunk crosses the link while the thread copies (or widens) another, and the
// page faults spread over the threads.
//
// Page-locking the slots takes 1 to 2.5 ms for one thread's and 10 ms for eight
// threads', and freeing them 0.4 to 1.8; the driver's own copy takes 0.06 to
// 0.1 ms per MB into memory that is there and 0.2 with its page faults, the
// staged one 0.05.  So an object's first kLockAfter bytes go through the driver,
// a widening download in pageable chunks of as many threads.  First download
// of a new ensemble: 0.01 MB 0.08 ms with the driver's copies alone, 1.2 to 2.7
// with slots made at once, 0.06 so; 7.8 MB 16, 3.7 to 6.3 and 1.5 ms.
#include "transfer.cuh"

#include <string.h>

#include <algorithm>
#include <atomic>
#include <exception>
#include <memory>
#include <new>
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

void widen_to(double* d, const float* f, size_t n) {
  for (size_t k = 0; k < n; ++k) d[k] = f[k];
}

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
  if (e == cudaSuccess) {
    threads_ = threads;
  } else {
    cudaGetLastError();  // the copies go without slots
    if (pinned_) cudaFreeHost(pinned_);
    pinned_ = nullptr;
  }
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
  moved_ += mode == kDownWiden ? 2 * total : total;
  // one thread per 4 MB (written, where that is more), as far as the machine has cores
  const int cores = std::max(1, (int)std::thread::hardware_concurrency());
  auto threads_for = [&](size_t bytes) { return (int)std::min<size_t>(std::min(kThreads, cores), (bytes >> 22) + 1); };
  int threads = threads_for(total);
  // without slots while they would cost more than they give (a call of less than
  // one chunk makes none, however often it comes), and where the machine has no
  // page-locked memory for them
  const bool small = total < kChunk && mode != kDownWiden;
  const bool plain = (!pinned_ && (small || moved_ < kLockAfter)) || reserve(threads) != cudaSuccess;
  if (plain) threads = threads_for(2 * total);
  if (plain && mode != kDownWiden) {
    for (int p = 0; p < nparts; ++p) {
      if (!parts[p].bytes) continue;
      const cudaError_t e = cudaMemcpyAsync(parts[p].dst, parts[p].src, parts[p].bytes,
                                            mode == kUp ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st);
      if (e != cudaSuccess) return e;
    }
    return cudaStreamSynchronize(st);
  }
  std::atomic<size_t> next{0};
  std::atomic<int> status{cudaSuccess};
  auto fail = [&](cudaError_t x) {
    int ok = cudaSuccess;
    if (x != cudaSuccess) status.compare_exchange_strong(ok, x);
    return x != cudaSuccess;
  };
  // the driver's copies of a widening download, a pageable chunk per thread
  auto widen_plain = [&](int t) {
    const std::unique_ptr<float[]> at(new (std::nothrow) float[kChunk / sizeof(float)]);
    if (!at) fail(cudaErrorMemoryAllocation);
    if (t && fail(cudaSetDevice(device))) return;
    for (size_t i; status == cudaSuccess && (i = next++) < chunks.size();) {
      const CopyPart& c = chunks[i];
      if (fail(cudaMemcpyAsync(at.get(), c.src, c.bytes, cudaMemcpyDeviceToHost, st))) break;
      if (fail(cudaStreamSynchronize(st))) break;
      widen_to(static_cast<double*>(c.dst), at.get(), c.bytes / sizeof(float));
    }
  };
  auto staged = [&](int t) {
    char* slot = pinned_ + (size_t)t * kSlots * kChunk;
    size_t held[kSlots] = {};
    bool busy[kSlots] = {};  // a copy through the slot is in flight
    // waits for the slot's copy; a download then goes on to its destination
    auto finish = [&](int s) {
      busy[s] = false;
      if (fail(cudaEventSynchronize(ev_[t][s])) || mode == kUp) return;
      const CopyPart& c = chunks[held[s]];
      const char* from = slot + (size_t)s * kChunk;
      if (mode == kDown) {
        memcpy(c.dst, from, c.bytes);
      } else {
        widen_to(static_cast<double*>(c.dst), reinterpret_cast<const float*>(from), c.bytes / sizeof(float));
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
  auto spread = [&](auto work) {
    std::thread pool[kThreads];
    int made = 0;
    try {
      for (; made < threads - 1; ++made) pool[made] = std::thread(work, made + 1);
    } catch (const std::exception&) {
      // fewer threads: the chunks go to those that started
    }
    work(0);
    for (int t = 0; t < made; ++t) pool[t].join();
  };
  if (plain) spread(widen_plain);
  else spread(staged);
  if (status != cudaSuccess) cudaStreamSynchronize(st);  // nothing stays in flight through the slots
  return (cudaError_t)status.load();
}

cudaError_t HostStage::download(const CopyPart* parts, int nparts, bool widen, int device, cudaStream_t st) {
  try {
    return run(parts, nparts, widen ? kDownWiden : kDown, device, st);
  } catch (const std::bad_alloc&) {
    return cudaErrorMemoryAllocation;
  }
}

cudaError_t HostStage::upload(const CopyPart* parts, int nparts, int device, cudaStream_t st) {
  try {
    return run(parts, nparts, kUp, device, st);
  } catch (const std::bad_alloc&) {
    return cudaErrorMemoryAllocation;
  }
}

}  // namespace felis
