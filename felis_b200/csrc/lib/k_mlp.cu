// Elementwise kernels of the taper-surrogate MLP (its GEMMs are in
// k_gemm.cu) and the self-test of the library's bounded mbarrier wait.
#include <math.h>

#include "mlp.cuh"
#include "tc.cuh"

namespace felis {

namespace {

constexpr int kWaitLimit = 1 << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Bounded wait for the phase `parity` of an mbarrier; false when it ran out.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit = kWaitLimit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The bounded wait on an mbarrier that nothing arrives on: phase 0 never
// completes, so every thread's wait runs out after `limit` tries and the
// kernel records that, then returns with nothing in flight.
__global__ void __launch_bounds__(128) k_wait_selftest(int limit, int* timed_out) {
  __shared__ __align__(8) uint64_t bar;
  const uint32_t b = smem_u32(&bar);
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  const bool done = mbar_wait(b, 0u, limit);
  const int all_ran_out = __syncthreads_and(done ? 0 : 1);
  if (threadIdx.x == 0) *timed_out = all_ran_out;
}

__global__ void k_f32_to_bf16(const float* in, bf16* out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __float2bfloat16_rn(in[i]);
}

__global__ void k_pack_rows(const float* __restrict__ in, int rows, int cols, int rows_pad, int cols_pad,
                            __nv_bfloat162* __restrict__ out) {
  const int half = cols_pad >> 1;
  const int64_t n = (int64_t)rows_pad * half;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / half), c = 2 * (int)(i - (int64_t)r * half);
    const float* p = in + (size_t)r * cols + c;
    const float a = r < rows && c < cols ? p[0] : 0.f, b = r < rows && c + 1 < cols ? p[1] : 0.f;
    out[i] = __floats2bfloat162_rn(a, b);
  }
}

__global__ void k_pad_rows(const float* __restrict__ in, int rows, int cols, int ld, float* __restrict__ out) {
  const int64_t n = (int64_t)rows * ld;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / ld), c = (int)(i - (int64_t)r * ld);
    out[i] = c < cols ? in[(size_t)r * cols + c] : 0.f;
  }
}

__global__ void k_unpad_rows(const float* __restrict__ in, int rows, int ld, int cols, float* __restrict__ out) {
  const int64_t n = (int64_t)rows * cols;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int r = (int)(i / cols);
    out[i] = in[(size_t)r * ld + (i - (int64_t)r * cols)];
  }
}

__global__ void k_transpose_bf16(const bf16* in, int rows, int cols, int ld_in, bf16* out, int rows_pad,
                                 int cols_pad) {
  const int64_t n = (int64_t)rows_pad * cols_pad;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i / rows_pad), r = (int)(i % rows_pad);
    out[i] = (r < rows && c < cols) ? in[(size_t)r * ld_in + c] : __float2bfloat16_rn(0.f);
  }
}

// 32 rows per block, a lane per row, a warp per column in turn
__global__ void __launch_bounds__(512) k_batch_rows(const bf16* data_x, const float* data_t, const int* idx, int n,
                                                    int rows, int in_p, int out_p, bf16* x, bf16* xt, float* t) {
  const int r = blockIdx.x * 32 + (threadIdx.x & 31), w = threadIdx.x >> 5;
  if (r >= rows) return;
  const bool real = r < n;
  const int64_t s = real ? (idx ? idx[r] : r) : 0;
#pragma unroll 4
  for (int c = w; c < in_p; c += 16) {
    const bf16 v = real ? data_x[s * in_p + c] : __float2bfloat16_rn(0.f);
    x[(size_t)r * in_p + c] = v;
    xt[(size_t)c * rows + r] = v;
  }
#pragma unroll 4
  for (int c = w; c < out_p; c += 16) t[(size_t)r * out_p + c] = real ? data_t[s * out_p + c] : 0.f;
}

constexpr int kMseRows = 32;  // rows per block of the loss kernel

__global__ void __launch_bounds__(256) k_mse_grad(const float* y, const float* t, int rows, int rows_real,
                                                  int cols_pad, int cols_real, float scale, bf16* dy, bf16* dyt,
                                                  double* part) {
  __shared__ double red[8];
  double acc = 0.0;
  const int r0 = blockIdx.x * kMseRows;
  for (int k = threadIdx.x; k < kMseRows * cols_pad; k += blockDim.x) {
    const int r = r0 + k / cols_pad, c = k % cols_pad;
    if (r >= rows) continue;
    const size_t i = (size_t)r * cols_pad + c;
    float d = 0.f;
    if (r < rows_real && c < cols_real) {
      d = y[i] - t[i];
      acc += (double)d * d;
    }
    const bf16 v = __float2bfloat16_rn(scale * d);
    dy[i] = v;
    dyt[(size_t)c * rows + r] = v;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    part[blockIdx.x] = s;
  }
}

// One thread per column, along its row of dz^T: eight rows to a load, eight
// loads in flight, added in row order (the same sums as walking the columns of
// dz, which waited for memory at every fourth row).  All layers: 6 us at 512
// rows, 28 at 3072; the walk took 12 us for each layer at 512.
__global__ void __launch_bounds__(32) k_bias_grads(MlpLayers L, int M, float* grad) {
  const int l = blockIdx.y, c = blockIdx.x * 32 + threadIdx.x;
  if (c >= L.rows[l]) return;
  const uint4* col = reinterpret_cast<const uint4*>(L.dzt[l] + (size_t)c * M);
  float s = 0.f;
  for (int r = 0; r < M / 8; r += 8) {  // M is a multiple of 128
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = __ldg(col + r + u);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        s += __uint_as_float(w[k] << 16);
        s += __uint_as_float(w[k] & 0xffff0000u);
      }
    }
  }
  grad[L.b_off[l] + c] = s;
}

__global__ void __launch_bounds__(256) k_adamw(MlpLayers L, float* w, const float* g, float* m, float* v, float lr,
                                               float b1, float b2, float eps, float wd, float bc1, float bc2) {
  const int l = blockIdx.y, rows = L.rows[l], cols = L.cols[l], nw = rows * cols;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nw + rows; i += gridDim.x * blockDim.x) {
    const bool weight = i < nw;
    const size_t k = weight ? L.w_off[l] + i : L.b_off[l] + (i - nw);
    const float gi = g[k];
    const float mi = b1 * m[k] + (1.f - b1) * gi;
    const float vi = b2 * v[k] + (1.f - b2) * gi * gi;
    m[k] = mi;
    v[k] = vi;
    const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps) + (weight ? wd : 0.f) * w[k];
    const float wi = w[k] - lr * upd;
    w[k] = wi;
    if (weight) {
      const bf16 h = __float2bfloat16_rn(wi);
      L.wb[l][i] = h;
      if (l > 0) {
        const int r = i / cols;
        L.wt[l][(size_t)(i - r * cols) * rows + r] = h;
      }
    }
  }
}

int grid_for(int64_t n) { return (int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096); }

}  // namespace

void launch_f32_to_bf16(const float* in, bf16* out, int64_t n, cudaStream_t st) {
  if (n > 0) k_f32_to_bf16<<<grid_for(n), 256, 0, st>>>(in, out, n);
}

void launch_pack_rows(const float* in, int rows, int cols, int rows_pad, int cols_pad, bf16* out, cudaStream_t st) {
  const int64_t n = (int64_t)rows_pad * (cols_pad >> 1);
  if (n > 0) k_pack_rows<<<grid_for(n), 256, 0, st>>>(in, rows, cols, rows_pad, cols_pad, reinterpret_cast<__nv_bfloat162*>(out));
}

void launch_pad_rows(const float* in, int rows, int cols, int ld, float* out, cudaStream_t st) {
  const int64_t n = (int64_t)rows * ld;
  if (n > 0) k_pad_rows<<<grid_for(n), 256, 0, st>>>(in, rows, cols, ld, out);
}

void launch_unpad_rows(const float* in, int rows, int ld, int cols, float* out, cudaStream_t st) {
  const int64_t n = (int64_t)rows * cols;
  if (n > 0) k_unpad_rows<<<grid_for(n), 256, 0, st>>>(in, rows, ld, cols, out);
}

void launch_transpose_bf16(const bf16* in, int rows, int cols, int ld_in, bf16* out, int rows_pad, int cols_pad,
                           cudaStream_t st) {
  const int64_t n = (int64_t)rows_pad * cols_pad;
  if (n > 0) k_transpose_bf16<<<grid_for(n), 256, 0, st>>>(in, rows, cols, ld_in, out, rows_pad, cols_pad);
}

void launch_batch_rows(const bf16* data_x, const float* data_t, const int* idx, int n, int rows, int in_p, int out_p,
                       bf16* x, bf16* xt, float* t, cudaStream_t st) {
  k_batch_rows<<<(rows + 31) / 32, 512, 0, st>>>(data_x, data_t, idx, n, rows, in_p, out_p, x, xt, t);
}

int mse_blocks(int rows) { return (rows + kMseRows - 1) / kMseRows; }

void launch_mse_grad(const float* y, const float* t, int rows, int rows_real, int cols_pad, int cols_real,
                     float scale, bf16* dy, bf16* dyt, double* loss_part, cudaStream_t st) {
  k_mse_grad<<<mse_blocks(rows), 256, 0, st>>>(y, t, rows, rows_real, cols_pad, cols_real, scale, dy, dyt, loss_part);
}

void launch_bias_grads(const MlpLayers& l, int M, float* grad, cudaStream_t st) {
  int most = 0;
  for (int k = 0; k < 4; ++k) most = l.rows[k] > most ? l.rows[k] : most;
  k_bias_grads<<<dim3((most + 31) / 32, 4), 32, 0, st>>>(l, M, grad);
}

void launch_adamw(const MlpLayers& l, float* w, const float* g, float* m, float* v, float lr, float b1, float b2,
                  float eps, float wd, float bc1, float bc2, cudaStream_t st) {
  int most = 0;
  for (int k = 0; k < 4; ++k) most = l.rows[k] * (l.cols[k] + 1) > most ? l.rows[k] * (l.cols[k] + 1) : most;
  k_adamw<<<dim3((most + 255) / 256, 4), 256, 0, st>>>(l, w, g, m, v, lr, b1, b2, eps, wd, bc1, bc2);
}

void launch_wait_selftest(int limit, int* timed_out, cudaStream_t st) {
  k_wait_selftest<<<1, 128, 0, st>>>(limit, timed_out);
}

}  // namespace felis
