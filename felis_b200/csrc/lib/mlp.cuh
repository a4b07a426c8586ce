// Taper-surrogate MLP: tensor-core GEMM and the elementwise kernels of its
// forward pass, backward pass and AdamW update.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace felis {

typedef __nv_bfloat16 bf16;

// C[M][N] = A[M][K] . B[N][K]^T on the 5th-generation tensor cores (BF16
// operands, FP32 accumulation in tensor memory), with an optional epilogue:
//   v = C + bias[n]                        (bias may be null)
//   out_f32[m][n] = v                      (may be null)
//   w = gelu ? GELU(v) : z ? v GELU'(z[m][n]) : v, rounded to BF16
//   out_bf16[m][n] = w, out_t[n][m] = w    (each may be null)
// A and B are row-major with leading dimensions lda, ldb (elements, multiples
// of 8); M is a multiple of 128, N a multiple of 16, K a multiple of 16.
// Columns n >= n_valid of the outputs are written as 0.  err (may be null)
// receives 1 when a tensor-core wait ran out.
struct GemmArgs {
  const bf16* A;
  const bf16* B;
  int M, N, K, lda, ldb;
  const float* bias;
  float* out_f32;
  bf16* out_bf16;
  int ldc;       // leading dimension of both outputs and of z
  int n_valid;
  int gelu;
  int* err;
  bf16* out_t = nullptr;
  int ldt = 0;             // leading dimension of out_t
  const float* z = nullptr;
  int rows_a = 0;          // rows that A has, when fewer than M (the others count as zero)
};
// Computed by the TMA-fed, warp-specialised persistent kernel of k_gemm.cu
// (N <= 256; 16-byte aligned A and B); cudaErrorInvalidValue for shapes
// outside that.  gemm_tma_prepare() once per device before use.
// n: one product, or two that are independent of each other in one launch.
cudaError_t launch_gemm_tma(const GemmArgs* g, int n, cudaStream_t st);
cudaError_t gemm_tma_prepare();
// 2-D tensor map of a row-major BF16 matrix [rows][ld] read in (64 x
// box_rows) tiles of its first `cols` columns, 128-byte swizzle; elements
// outside the matrix read as zero.  Valid after gemm_tma_prepare().
bool tma_encode_bf16(CUtensorMap* map, const bf16* base, int rows, int cols, int ld, int box_rows);
int gemm_sm_count();

// The whole inference pass x -> W1 -> GELU -> W2 -> GELU -> W3 -> GELU -> W4
// in one kernel (k_mlp_fused.cu): y[m][n] = (network)(x[m]) in FP32 for M rows
// (a multiple of 128), hidden width 256; x [M][in_k] BF16; W_l row-major
// [rows][cols] BF16 (W1 [256][in_k], W2 and W3 [256][256], W4 [out_n][256]);
// bias_l FP32; in_k and out_n multiples of 16, in_k <= 64, out_n <= 256;
// 16-byte aligned pointers.  Same rounding points as the layer-by-layer
// chain (BF16 hidden activations, FP32 accumulation).
struct MlpFusedArgs {
  const bf16* x;
  int M, width, in_k, out_n;
  const bf16* w[4];
  const float* bias[4];
  float* y;
  int* err;
};
bool mlp_fused_supported(int width, int in_k, int out_n);
cudaError_t mlp_fused_prepare();
cudaError_t launch_mlp_fused(const MlpFusedArgs& a, cudaStream_t st);

// Elementwise and reduction helpers (row-major [rows][cols] unless stated).
void launch_f32_to_bf16(const float* in, bf16* out, int64_t n, cudaStream_t st);
// out[r][c] = in[r][c] in BF16, rows x cols of a dense matrix into a padded one
// of rows_pad x cols_pad (cols_pad even), zeros around them
void launch_pack_rows(const float* in, int rows, int cols, int rows_pad, int cols_pad, bf16* out, cudaStream_t st);
// out[r][c] = in[r][c] for c < cols, 0 up to ld columns
void launch_pad_rows(const float* in, int rows, int cols, int ld, float* out, cudaStream_t st);
// out[r][c] = in[r][c], the first cols of ld columns, densely packed
void launch_unpad_rows(const float* in, int rows, int ld, int cols, float* out, cudaStream_t st);
// out[c][r] = in[r][c] for r < rows, c < cols; rows_pad / cols_pad zero padding
// of the destination ([cols_pad][rows_pad])
void launch_transpose_bf16(const bf16* in, int rows, int cols, int ld_in, bf16* out, int rows_pad, int cols_pad,
                           cudaStream_t st);
// The rows of one batch: row r of x (BF16, in_p columns) and of t (FP32, out_p
// columns) is row idx[r] of the data (idx null: row r), zero for r >= n; xt is
// x transposed, rows columns.
void launch_batch_rows(const bf16* data_x, const float* data_t, const int* idx, int n, int rows, int in_p, int out_p,
                       bf16* x, bf16* xt, float* t, cudaStream_t st);
// dy = scale * (y - t) on real rows / columns, 0 elsewhere (y, t, dy all
// [rows][cols_pad]) and its transpose dyt; loss_part[b] = sum of (y - t)^2 of
// block b, blocks = mse_blocks(rows)
int mse_blocks(int rows);
void launch_mse_grad(const float* y, const float* t, int rows, int rows_real, int cols_pad, int cols_real,
                     float scale, bf16* dy, bf16* dyt, double* loss_part, cudaStream_t st);
// The four layers' parameters, as one launch sees them: weights [rows][cols] at
// w_off and biases at b_off of the flat FP32 arrays, BF16 weights and their
// transposes (not of the first layer), and the batch's dz transposed [rows][M].
struct MlpLayers {
  size_t w_off[4], b_off[4];
  int rows[4], cols[4];
  bf16* wb[4];
  bf16* wt[4];
  const bf16* dzt[4];
};
// grad[b_off + c] = sums of dz over the M rows, in row order (M a multiple of 128)
void launch_bias_grads(const MlpLayers& l, int M, float* grad, cudaStream_t st);
// AdamW on every parameter (no weight decay on biases); refreshes the BF16 copies
void launch_adamw(const MlpLayers& l, float* w, const float* g, float* m, float* v, float lr, float b1, float b2,
                  float eps, float wd, float bc1, float bc2, cudaStream_t st);

// The library's bounded mbarrier wait (the one the GEMM uses) on a barrier
// phase that nothing completes: *timed_out = 1 when every thread's wait gave
// up after `limit` tries.
void launch_wait_selftest(int limit, int* timed_out, cudaStream_t st);

}  // namespace felis
