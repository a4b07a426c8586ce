// BF16 GEMM of the taper surrogate on the 5th-generation tensor cores:
// C[M][N] = A[M][K] . B[N][K]^T, FP32 accumulation in tensor memory, with the
// epilogue of mlp.cuh (bias, GELU or its derivative, FP32 and/or BF16 outputs,
// a transposed copy for the next GEMM that contracts over the rows).
//
// One launch computes one or two independent products (the weight gradient of
// a layer and the gradient of its input, which use the same dz): one
// persistent CTA per SM walks the tiles of both, 128 rows by up to 256
// columns.  A training batch has a handful of rows of tiles, and a 256-column
// epilogue (GELU, two or three outputs) takes its SM 15 us, so small products
// are cut into narrower tiles until they cover the SMs.  Warp roles:
//   warp 0     one lane issues the TMA loads: the A tile (128 x 64) and the
//              B tile (N x 64) of every 64-column K chunk, 128-byte swizzle,
//              into a ring of kStages shared-memory stages (full / empty
//              mbarriers per stage)
//   warp 1     allocates tensor memory (two accumulators of N columns, 32-column
//              aligned); one lane issues tcgen05.mma (M = 128, N, K = 16; four
//              per chunk) and commits each stage back to the producer and each
//              finished accumulator to the epilogue
//   warps 2-9  the epilogue: warp w reads lanes 32 (w % 4) .. + 31 of the
//              accumulator (tcgen05.ld, one row per thread), two warps per
//              lane quarter taking alternate 32-column chunks; each thread
//              applies bias / GELU to its 32 values and writes them with
//              16-byte stores, then the warps free the accumulator
// The two accumulators alternate, so a tile's epilogue overlaps the next
// tile's loads and MMAs.  Every mbarrier wait is bounded: one that runs out
// sets the error word and the flag that stops the other roles; the MMA lane
// then waits (bounded) for its MMAs in flight before the tensor memory is
// freed.  The TMA loads read this GPU's own memory, without multicast.
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mlp.cuh"
#include "tc.cuh"

namespace felis {

namespace {

using namespace tc;

constexpr int kBM = 128;          // rows of a C tile (the MMA M)
constexpr int kBK = 64;           // K columns per stage: 128 bytes of BF16, the swizzle span
constexpr int kStages = 4;
constexpr int kEpiWarps = 8;
constexpr int kThreads = 32 * (2 + kEpiWarps);
constexpr uint32_t kABytes = kBM * kBK * 2;  // 16 KB

struct TmaGemm {
  int M, N, K;  // M a multiple of 128, N a multiple of 16 (<= 256), K a multiple of 16
  const float* bias;
  const float* z;  // multiply by GELU'(z)
  float* out_f32;
  bf16* out_bf16;
  bf16* out_t;
  int ldc, ldt, n_valid, gelu;
  int bn, nt;  // columns of a tile, tiles per 128 rows
};
struct TmaPair {
  TmaGemm g[2];
  CUtensorMap a[2], b[2];
  int tiles0, tiles;     // tiles of the first product, of both
  int tmem_cols;         // allocated tensor-memory columns
  int acc_stride;        // column offset of the second accumulator (the wider tile rounded up to 32)
  uint32_t stage_bytes;  // of the wider tile
  int* err;
};

// Two neighbouring columns as BF16, through GELU where the product has it.
__device__ __forceinline__ uint32_t pack(const TmaGemm& g, int col, float x0, float x1) {
  if (g.gelu) {
    if (col < g.n_valid) x0 = gelu_f(x0);
    if (col + 1 < g.n_valid) x1 = gelu_f(x1);
  }
  const __nv_bfloat162 p2 = __floats2bfloat162_rn(x0, x1);
  return *reinterpret_cast<const uint32_t*>(&p2);
}

// ONE: a single product of whole rows without z and out_t (inference by the
// layer chain, whose epilogues bound it: the four layers of a million rows
// take 3.31 ms in the general instance, 2.27 in this one).
template <bool ONE>
__global__ void __launch_bounds__(kThreads, 1) k_gemm_tma(const __grid_constant__ TmaPair P) {
  extern __shared__ unsigned char smraw[];
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  // the swizzled operand tiles start on 1024-byte boundaries of the shared window
  unsigned char* sm = smraw + ((1024u - (sa(smraw) & 1023u)) & 1023u);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t stage_bytes = P.stage_bytes;
  const int ntiles = P.tiles;
  volatile int* abort_v = &abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(sa(&full[s]), 1);
      mbar_init(sa(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(sa(&tfull[b]), 1);
      mbar_init(sa(&tempty[b]), kEpiWarps * 32);
    }
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(sa(&tmem_slot)),
                 "r"(P.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = tmem_slot;

  auto give_up = [&]() {
    *abort_v = 1;
    if (P.err) atomicOr(P.err, 1);
  };

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        const int p = !ONE && t >= P.tiles0, tp = p ? t - P.tiles0 : t, m = (ONE ? tp : tp / P.g[p].nt) * kBM;
        const int n0 = ONE ? 0 : tp % P.g[p].nt * P.g[p].bn;
        const int nk = (P.g[p].K + kBK - 1) / kBK;
        const uint32_t bytes = kABytes + (uint32_t)P.g[p].bn * kBK * 2;
        for (int k = 0; k < nk && ok; ++k) {
          // a fresh stage passes at once (the phase before the first counts as complete)
          if (!mbar_wait(sa(&empty[s]), ph ^ 1u, abort_v)) { give_up(); ok = false; break; }
          const uint32_t a_s = sa(sm + (size_t)s * stage_bytes);
          mbar_expect_tx(sa(&full[s]), bytes);
          tma_load_2d(a_s, &P.a[p], k * kBK, m, sa(&full[s]));
          tma_load_2d(a_s + kABytes, &P.b[p], k * kBK, n0, sa(&full[s]));
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      int s = 0, it = 0;
      uint32_t ph = 0;
      uint32_t last_bar = 0, last_par = 0;  // last commit, waited for on the way out
      bool ok = true;
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++it) {
        const int b = it & 1;
        const uint32_t bph = (uint32_t)(it >> 1) & 1u;
        if (!mbar_wait(sa(&tempty[b]), bph ^ 1u, abort_v)) { give_up(); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(b * P.acc_stride);
        const TmaGemm& g = P.g[!ONE && t >= P.tiles0];
        const uint32_t idesc = idesc_bf16(kBM, g.bn);
        const int nk = (g.K + kBK - 1) / kBK;
        for (int k = 0; k < nk; ++k) {
          if (!mbar_wait(sa(&full[s]), ph, abort_v)) { give_up(); ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint32_t a_s = sa(sm + (size_t)s * stage_bytes), b_s = a_s + kABytes;
#pragma unroll
          for (int kk = 0; kk < kBK / 16; ++kk)
            mma_bf16(d, desc_sw128(a_s + 32u * kk), desc_sw128(b_s + 32u * kk), idesc, (k | kk) ? 1u : 0u);
          mma_commit(sa(&empty[s]));
          last_bar = sa(&empty[s]);
          last_par = ph;
          if (++s == kStages) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        mma_commit(sa(&tfull[b]));
        last_bar = sa(&tfull[b]);
        last_par = bph;
      }
      // the tensor memory is freed below: wait for the last MMAs issued
      if (last_bar) {
        for (int i = 0; i < kWaitTries && !mbar_try(last_bar, last_par); ++i) {
        }
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3;            // tensor-memory lane quarter this warp may read
    const int half = (warp - 2) >> 2;  // which of the two warps of that quarter
    const TmaGemm g0 = P.g[0];  // in registers: through P they are read again after every store
    int it = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
      const int b = it & 1;
      const uint32_t bph = (uint32_t)(it >> 1) & 1u;
      if (!mbar_wait(sa(&tfull[b]), bph, abort_v)) { give_up(); break; }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * P.acc_stride);
      const int p = !ONE && t >= P.tiles0;
      const TmaGemm& g = ONE ? g0 : P.g[p];
      const int tp = p ? t - P.tiles0 : t, n0 = ONE ? 0 : tp % g.nt * g.bn;
      const int N = ONE ? g.N : min(g.N, n0 + g.bn);
      const size_t row = (size_t)(ONE ? tp : tp / g.nt) * kBM + (size_t)q * 32 + lane;
      auto columns = [&](int c0) {
        uint32_t r[32];
        TMEM_LD32X32(tbase + (uint32_t)(c0 - n0), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        const int ncol = N - c0 < 32 ? N - c0 : 32;  // 16 or 32 (N is a multiple of 16)
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int col = c0 + j;
          const bool valid = col < g.n_valid;
          v[j] = valid ? __uint_as_float(r[j]) + (g.bias ? __ldg(g.bias + col) : 0.f) : 0.f;
        }
        const size_t o = row * (size_t)g.ldc + c0;
        if (g.out_f32) {
          float4* dst = reinterpret_cast<float4*>(g.out_f32 + o);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (4 * j < ncol) dst[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        if (!ONE && g.z) {
          const float4* zs = reinterpret_cast<const float4*>(g.z + o);
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (4 * j < ncol) {
              const float4 z = zs[j];
              v[4 * j] *= gelu_grad(z.x);
              v[4 * j + 1] *= gelu_grad(z.y);
              v[4 * j + 2] *= gelu_grad(z.z);
              v[4 * j + 3] *= gelu_grad(z.w);
            }
        }
        if (ONE && g.out_bf16) {
          uint4* dst = reinterpret_cast<uint4*>(g.out_bf16 + o);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (8 * j >= ncol) break;
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = pack(g, c0 + 8 * j + 2 * k, v[8 * j + 2 * k], v[8 * j + 2 * k + 1]);
            dst[j] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        if (!ONE && (g.out_bf16 || g.out_t)) {
          uint32_t w[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) w[k] = pack(g, c0 + 2 * k, v[2 * k], v[2 * k + 1]);
          if (g.out_bf16) {
            uint4* dst = reinterpret_cast<uint4*>(g.out_bf16 + o);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (8 * j < ncol) dst[j] = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
          }
          if (g.out_t) {
            // 32 neighbouring rows of one column by a warp: 64 bytes
            uint16_t* dst = reinterpret_cast<uint16_t*>(g.out_t) + (size_t)c0 * g.ldt + row;
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < ncol) dst[(size_t)j * g.ldt] = (uint16_t)(w[j >> 1] >> (16 * (j & 1)));
          }
        }
      };
      if constexpr (ONE) {
        for (int c0 = n0 + 32 * half; c0 < N; c0 += 64) columns(c0);
      } else {
#pragma unroll 1
        for (int c0 = n0 + 32 * half; c0 < N; c0 += 64) columns(c0);
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      mbar_arrive(sa(&tempty[b]));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(P.tmem_cols) : "memory");
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn g_encode = nullptr;
int g_sms = 0;

size_t tma_smem(int N) { return 1024 + (size_t)kStages * (kABytes + (size_t)N * kBK * 2); }

}  // namespace

bool tma_encode_bf16(CUtensorMap* map, const bf16* base, int rows, int cols, int ld, int box_rows) {
  if (!g_encode) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  const cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return g_encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int gemm_sm_count() { return g_sms; }

cudaError_t gemm_tma_prepare() {
  if (!g_encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
    if (e != cudaSuccess) return e;
    if (q != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    g_encode = reinterpret_cast<EncodeTiledFn>(fn);
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_gemm_tma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tma_smem(256));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_gemm_tma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tma_smem(256));
  return e;
}

cudaError_t launch_gemm_tma(const GemmArgs* a, int n, cudaStream_t st) {
  if (!g_encode || g_sms <= 0) return cudaErrorNotReady;
  if (n < 1 || n > 2) return cudaErrorInvalidValue;
  TmaPair P{};
  int wide = 0;
  for (int i = 0; i < n; ++i) {
    const GemmArgs& x = a[i];
    if (x.M % kBM || x.N % 16 || x.N < 16 || x.N > 256 || x.K % 16 || x.K < 16 || x.lda % 8 || x.ldb % 8 ||
        (reinterpret_cast<uintptr_t>(x.A) & 15) || (reinterpret_cast<uintptr_t>(x.B) & 15))
      return cudaErrorInvalidValue;
    // rows of A past rows_a read as zero
    const int rows_a = x.rows_a ? x.rows_a : x.M;
    TmaGemm& g = P.g[i];
    // tiles as wide as the product while the launch fills the SMs, else 64 or
    // 32 columns (rows of B past N count as zero).  512 x 256 with GELU and
    // both outputs: 31 us as four tiles of 256 columns, 10.3 us as 32 of 32
    g.bn = x.N;
    for (int bn : {64, 32})
      if (g.bn > bn && (x.M / kBM) * ((x.N + g.bn - 1) / g.bn) * 2 <= g_sms) g.bn = bn;
    g.nt = (x.N + g.bn - 1) / g.bn;
    if (!tma_encode_bf16(&P.a[i], x.A, rows_a, x.K, x.lda, kBM) || !tma_encode_bf16(&P.b[i], x.B, x.N, x.K, x.ldb, g.bn))
      return cudaErrorInvalidValue;
    g.M = x.M; g.N = x.N; g.K = x.K;
    g.bias = x.bias; g.z = x.z; g.out_f32 = x.out_f32; g.out_bf16 = x.out_bf16; g.out_t = x.out_t;
    g.ldc = x.ldc; g.ldt = x.ldt; g.n_valid = x.n_valid; g.gelu = x.gelu;
    P.tiles += x.M / kBM * g.nt;
    if (i == 0) P.tiles0 = P.tiles;
    if (g.bn > wide) wide = g.bn;
  }
  // two accumulators 32-column aligned (the epilogue reads 32 columns at a
  // time), in a power-of-two allocation of at least 32 columns
  P.acc_stride = (wide + 31) & ~31;
  P.tmem_cols = 32;
  while (P.tmem_cols < 2 * P.acc_stride) P.tmem_cols <<= 1;
  P.stage_bytes = kABytes + (uint32_t)wide * kBK * 2;
  P.err = a[0].err;
  const int grid = P.tiles < g_sms ? P.tiles : g_sms;
  if (grid == 0) return cudaSuccess;
  const bool one = n == 1 && P.g[0].nt == 1 && !a[0].z && !a[0].out_t;
  (one ? k_gemm_tma<true> : k_gemm_tma<false>)<<<grid, kThreads, tma_smem(wide), st>>>(P);
  return cudaGetLastError();
}

}  // namespace felis
