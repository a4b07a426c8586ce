// Stable integer key sort of particles by slice.
//
// The reference never moves particles between slices in its live loop
// (rearrangeParticles.cpp:7-75 is commented out); slice order matters when
// particles are binned on restart (restoreParticleHDF.cpp:166-214 keeps file
// order inside a slice) and when they are written slice-major
// (saveParticleHDF.cpp:95-109).  This sort reproduces that binning: the
// output permutation equals a stable CPU sort of the slice keys.
//
// LSD radix sort, 8-bit digits, 4096-element tiles.  Per pass:
//   1. per-tile digit counts
//   2. exclusive scan of each digit's counts over the tiles (one block per
//      digit) and the digits' totals
//   3. per tile: every element's rank among the equal digits before it, the
//      tile laid out by digit in shared memory, then written in runs.  A warp
//      takes 256 neighbouring elements, 32 at a time; eight ballots give each
//      lane the lanes with its digit, a counter per warp and digit carries the
//      ranks on.  Elements keep their order at every level: stable.
// Bound by memory traffic (16 B per element and pass, the values 32 bits wide;
// the first pass makes them, the last widens them).  Eight million keys of
// 1024 slices: 2.7 ms on the device with a bitonic sort of every tile, one block
// scanning all counts and 64-bit values; now 0.18, and the copies of the
// caller's pageable arrays around it take most of the 18 ms of a call.
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <cuda.h>
#include <mutex>
#include <vector>

#include "../../../include/felis_b200.h"

namespace {

constexpr int kTile = 4096;
constexpr int kThreads = 512, kWarps = kThreads / 32, kPerWarp = kTile / kWarps;

// Lanes that hold a key and the same digit as this one (those that hold none,
// for a lane without a key).
__device__ __forceinline__ unsigned same_digit(unsigned d, bool valid) {
  const unsigned vb = __ballot_sync(0xffffffffu, valid);
  unsigned m = valid ? vb : ~vb;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned x = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    m &= ((d >> b) & 1u) ? x : ~x;
  }
  return m;
}

// Exclusive scan of one value per thread of the first 256 threads.
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t* wsum) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31 && w < 8) wsum[w] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int q = 0; q < 8; ++q) before += q < w ? wsum[q] : 0u;
  __syncthreads();
  return before + x - v;
}

// The largest key, as an unsigned number.
__global__ void __launch_bounds__(256) k_key_max(const uint32_t* keys, int64_t n, uint32_t* out) {
  uint32_t m = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    m = max(m, keys[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void __launch_bounds__(kThreads) k_hist(const uint32_t* keys, int64_t n, int shift, int ntiles,
                                                   uint32_t* hist) {
  __shared__ uint32_t h[256];
  for (int d = threadIdx.x; d < 256; d += blockDim.x) h[d] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kTile;
#pragma unroll
  for (int r = 0; r < kTile / kThreads; ++r) {
    const int64_t e = base + r * kThreads + threadIdx.x;
    if (e < n) atomicAdd(&h[(keys[e] >> shift) & 255u], 1u);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < 256; d += blockDim.x) hist[(size_t)d * ntiles + blockIdx.x] = h[d];
}

// Exclusive scan of one digit's counts over the tiles, in place; its total.
__global__ void __launch_bounds__(256) k_scan(uint32_t* hist, int ntiles, uint32_t* total) {
  __shared__ uint32_t wsum[8], last;
  uint32_t* a = hist + (size_t)blockIdx.x * ntiles;
  uint32_t run = 0;
  for (int64_t t0 = 0; t0 < ntiles; t0 += 256) {
    const int64_t t = t0 + threadIdx.x;
    const uint32_t v = t < ntiles ? a[t] : 0u, x = scan256(v, wsum);
    if (t < ntiles) a[t] = run + x;
    if (threadIdx.x == 255) last = x + v;
    __syncthreads();
    run += last;
    __syncthreads();
  }
  if (threadIdx.x == 0) total[blockIdx.x] = run;
}

// vin null: the values are the element numbers.  perm set: the last pass, which
// writes the values only.
__global__ void __launch_bounds__(kThreads) k_scatter(const uint32_t* kin, const uint32_t* vin, int64_t n, int shift,
                                                      int ntiles, const uint32_t* offs, const uint32_t* total,
                                                      uint32_t* kout, uint32_t* vout, int64_t* perm) {
  __shared__ uint16_t cnt[kWarps][256];         // counts, then starts, of a warp's digits
  __shared__ uint32_t sk[kTile], sv[kTile];     // the tile by digit
  __shared__ uint32_t first[256], to[256];      // a digit's start in the tile; its output minus that
  __shared__ uint32_t wsum[8];
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  for (int k = tid; k < kWarps * 256; k += kThreads) cnt[k >> 8][k & 255] = 0;
  const int64_t base = (int64_t)blockIdx.x * kTile;
  constexpr int R = kPerWarp / 32;
  uint32_t key[R], val[R], rank[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int64_t e = base + w * kPerWarp + r * 32 + lane;
    key[r] = e < n ? kin[e] : 0u;
    val[r] = e < n ? (vin ? vin[e] : (uint32_t)e) : 0u;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const bool valid = base + w * kPerWarp + r * 32 + lane < n;
    const unsigned d = (key[r] >> shift) & 255u, m = same_digit(d, valid), below = m & ((1u << lane) - 1u);
    const uint32_t c = valid ? cnt[w][d] : 0u;
    rank[r] = c + __popc(below);
    __syncwarp();
    if (valid && !below) cnt[w][d] = (uint16_t)(c + __popc(m));
    __syncwarp();
  }
  __syncthreads();
  uint32_t mine = 0;
  if (tid < 256)
    for (int q = 0; q < kWarps; ++q) {
      const uint32_t c = cnt[q][tid];
      cnt[q][tid] = (uint16_t)mine;
      mine += c;
    }
  const uint32_t f = scan256(mine, wsum), all = scan256(tid < 256 ? total[tid] : 0u, wsum);
  if (tid < 256) {
    first[tid] = f;
    to[tid] = all + offs[(size_t)tid * ntiles + blockIdx.x] - f;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (base + w * kPerWarp + r * 32 + lane < n) {
      const uint32_t d = (key[r] >> shift) & 255u, q = first[d] + cnt[w][d] + rank[r];
      sk[q] = key[r];
      sv[q] = val[r];
    }
  __syncthreads();
  const int m = (int)(n - base < kTile ? n - base : kTile);
  for (int q = tid; q < m; q += kThreads) {
    const uint32_t k = sk[q], dst = to[(k >> shift) & 255u] + (uint32_t)q;
    if (perm) {
      perm[dst] = (int64_t)sv[q];
    } else {
      kout[dst] = k;
      vout[dst] = sv[q];
    }
  }
}

// Sorts by the low 8 * passes bits, stable: perm[k] = the element at place k.
// K and V hold two buffers of n words each (the first of K may be the keys when
// they may be overwritten), hist 256 (ntiles + 1) words.
void sort_passes(const uint32_t* keys, int64_t n, int passes, uint32_t* const K[2], uint32_t* const V[2],
                 uint32_t* hist, int64_t* perm, cudaStream_t st) {
  const int ntiles = (int)((n + kTile - 1) / kTile);
  uint32_t* total = hist + (size_t)256 * ntiles;
  const uint32_t *kin = keys, *vin = nullptr;
  for (int p = 0; p < passes; ++p) {
    const bool last = p == passes - 1;
    uint32_t *ko = K[(p + 1) & 1], *vo = V[(p + 1) & 1];
    k_hist<<<ntiles, kThreads, 0, st>>>(kin, n, 8 * p, ntiles, hist);
    k_scan<<<256, 256, 0, st>>>(hist, ntiles, total);
    k_scatter<<<ntiles, kThreads, 0, st>>>(kin, vin, n, 8 * p, ntiles, hist, total, ko, vo, last ? perm : nullptr);
    kin = ko;
    vin = vo;
  }
}

}  // namespace

extern "C" felis_status felis_sort_by_slice(const int32_t* keys, int64_t n, int64_t* perm) {
  if (n < 0 || (n > 0 && (!keys || !perm))) return FELIS_BAD_ARG;
  if (n == 0) return FELIS_OK;
  if (n > ((int64_t)1 << 32)) return FELIS_UNSUPPORTED;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    for (int64_t i = 0; i < n; ++i)
      if (keys[i] < 0 || keys[i] >= (1 << 30)) return FELIS_BAD_ARG;
    return FELIS_NO_DEVICE;
  }
  const int64_t ntiles = (n + kTile - 1) / kTile;
  // one allocation: perm | two key and two value buffers | counts, totals, largest key
  const size_t words = (size_t)4 * n + (size_t)256 * (ntiles + 1) + 1;
  char* mem = nullptr;
  cudaStream_t st = nullptr;
  felis_status rc = FELIS_OK;
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&mem, (size_t)n * sizeof(int64_t) + words * sizeof(uint32_t));
  if (e == cudaSuccess) {
    int64_t* out = reinterpret_cast<int64_t*>(mem);
    uint32_t* K0 = reinterpret_cast<uint32_t*>(out + n);
    uint32_t* const K[2] = {K0, K0 + n};
    uint32_t* const V[2] = {K0 + 2 * n, K0 + 3 * n};
    uint32_t *hist = K0 + 4 * n, *kmax_d = hist + 256 * (ntiles + 1);
    e = cudaMemcpyAsync(K0, keys, n * sizeof(int32_t), cudaMemcpyHostToDevice, st);
    // the range of the keys, checked on the device: it sets the number of passes
    if (e == cudaSuccess) e = cudaMemsetAsync(kmax_d, 0, sizeof(uint32_t), st);
    uint32_t kmax = 0;
    if (e == cudaSuccess) {
      k_key_max<<<1184, 256, 0, st>>>(K0, n, kmax_d);
      e = cudaMemcpyAsync(&kmax, kmax_d, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && kmax >= (1u << 30)) rc = FELIS_BAD_ARG;
    if (e == cudaSuccess && rc == FELIS_OK) {
      int bits = 0;
      while ((kmax >> bits) != 0) ++bits;
      sort_passes(K0, n, bits == 0 ? 1 : (bits + 7) / 8, K, V, hist, out, st);
      e = cudaGetLastError();
      if (e == cudaSuccess) e = cudaMemcpyAsync(perm, out, n * sizeof(int64_t), cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
  }
  if (e != cudaSuccess) rc = FELIS_CUDA_ERROR;
  if (mem) cudaFree(mem);
  if (st) cudaStreamDestroy(st);
  return rc;
}

// ---------------------------------------------------------------------------
// Allocation-free variant.  Its scratch lives in one file-scope device array:
// two 32-bit key buffers, two 32-bit index buffers, the per-tile digit
// histogram and its totals, sized for FELIS_SORT_NOALLOC_MAX_KEYS keys.  Every GPU that
// loads this library holds the array until the process exits.  Each pass
// writes every scratch word it later reads, so nothing has to be cleared
// between calls; calls that overlap on the GPU share the array and race.
namespace {

constexpr int64_t kNaMax = FELIS_SORT_NOALLOC_MAX_KEYS;
constexpr int64_t kNaTiles = (kNaMax + kTile - 1) / kTile;
constexpr size_t kNaBytes = (size_t)4 * kNaMax * 4 + (size_t)256 * (kNaTiles + 1) * 4;

static __device__ __align__(256) unsigned char g_sort_scratch[kNaBytes];

// Device address of g_sort_scratch per CUDA context.  The address belongs to
// the context that loaded the module: it is resolved again on every call made
// outside stream capture (so a context recreated after cudaDeviceReset, or
// another context made current on the device, gets its own), and a call made
// during capture uses the address last resolved in the current context.
std::mutex g_na_mu;
struct NaEntry {
  CUcontext ctx;
  void* ptr;
};
NaEntry g_na_cache[64];
int g_na_count = 0;
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
CtxGetCurrentFn g_ctx_get_current = nullptr;

CUcontext current_context() {
  if (!g_ctx_get_current) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return nullptr;
    g_ctx_get_current = reinterpret_cast<CtxGetCurrentFn>(fn);
  }
  CUcontext c = nullptr;
  return g_ctx_get_current(&c) == CUDA_SUCCESS ? c : nullptr;
}

// Caller-owned buffers must be device (or managed) memory of device `dev`.
bool on_device(const void* p, int dev) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

}  // namespace

extern "C" felis_status felis_sort_by_slice_noalloc(const int32_t* keys_dev, int64_t n, int64_t* perm_dev,
                                                    void* stream) {
  if (n < 0 || (n > 0 && (!keys_dev || !perm_dev))) return FELIS_BAD_ARG;
  if (n > kNaMax) {
    fprintf(stderr, "felis_sort_by_slice_noalloc: %lld keys exceed the fixed scratch of %lld keys\n",
            (long long)n, (long long)kNaMax);
    return FELIS_BAD_ARG;
  }
  if (n == 0) return FELIS_OK;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return FELIS_NO_DEVICE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) return FELIS_CUDA_ERROR;
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  if (!capturing && (!on_device(keys_dev, dev) || !on_device(perm_dev, dev))) {
    fprintf(stderr, "felis_sort_by_slice_noalloc: keys_dev and perm_dev must be device memory of the current "
                    "device (%d)\n", dev);
    return FELIS_BAD_ARG;
  }
  void* base = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_na_mu);
    const CUcontext ctx = current_context();
    if (!ctx) return FELIS_CUDA_ERROR;
    int slot = -1;
    for (int i = 0; i < g_na_count; ++i)
      if (g_na_cache[i].ctx == ctx) slot = i;
    if (!capturing) {
      // resolve the array's device address in this context (the host-side
      // symbol is only a stand-in, not a device address)
      void* p = nullptr;
      if (cudaGetSymbolAddress(&p, g_sort_scratch) != cudaSuccess || !p) return FELIS_CUDA_ERROR;
      if (slot < 0) {
        if (g_na_count == 64) return FELIS_UNSUPPORTED;
        slot = g_na_count++;
        g_na_cache[slot].ctx = ctx;
      }
      g_na_cache[slot].ptr = p;
    } else if (slot < 0) {
      fprintf(stderr, "felis_sort_by_slice_noalloc: the first call in a context must come before stream capture\n");
      return FELIS_BAD_ARG;
    }
    base = g_na_cache[slot].ptr;
  }
  uint32_t* K0 = reinterpret_cast<uint32_t*>(base);
  uint32_t* const K[2] = {K0, K0 + kNaMax};
  uint32_t* const V[2] = {K0 + 2 * kNaMax, K0 + 3 * kNaMax};
  // four 8-bit passes: keys ordered as unsigned 32-bit values, stable
  sort_passes(reinterpret_cast<const uint32_t*>(keys_dev), n, 4, K, V, K0 + 4 * kNaMax, perm_dev, st);
  return cudaGetLastError() == cudaSuccess ? FELIS_OK : FELIS_CUDA_ERROR;
}
