// Host side of the taper-surrogate MLP (felis_mlp_*).
//
// Four linear layers n_in -> W -> W -> W -> n_out with GELU after the first
// three.  FP32 master parameters and AdamW state; BF16 weights and
// activations feed the tensor-core GEMMs (FP32 accumulation).  Shapes are
// padded to the GEMM's granules: inputs and outputs to multiples of 16,
// batches to multiples of 128 (padding rows and columns are zero and carry
// no loss).
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <random>
#include <string>
#include <vector>

#include "../../../include/felis_b200.h"
#include "mlp.cuh"
#include "transfer.cuh"

using namespace felis;

namespace {

constexpr int kLayers = 4;
constexpr int kChunk = 65536;  // rows per device pass (a multiple of 128)
constexpr int kFwdChunk = 1 << 20;  // rows per inference pass (felis_mlp_forward)

int round_up(int v, int m) { return (v + m - 1) / m * m; }

}  // namespace

struct felis_mlp {
  int n_in = 0, width = 0, n_out = 0;
  int in_p = 0, out_p = 0, out_rows = 0;  // padded sizes; out_rows: out_p rounded to 128
  cudaStream_t st = nullptr;
  std::string err;
  int* d_err = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;  // around the inference kernels of the last forward chunk
  bool fused = false;                        // inference by the fused kernel (k_mlp_fused.cu)
  double fwd_ms = 0.0, fwd_flops = 0.0;
  // per layer: rows (outputs) x cols (inputs), padded
  int rows[kLayers], cols[kLayers], rows_real[kLayers], cols_real[kLayers];
  size_t w_off[kLayers], b_off[kLayers], n_param = 0;
  float* p = nullptr;        // FP32 master parameters (padded layout)
  float* grad = nullptr;     // gradients, same layout (W4 block has out_rows rows)
  float* m = nullptr;        // AdamW moments
  float* v = nullptr;
  bf16* wb[kLayers] = {};    // BF16 weights [rows][cols]
  bf16* wt[kLayers] = {};    // BF16 transposed weights [cols][rows] (layers 2..4)
  int64_t steps = 0;
  // activations of one chunk
  int cap = 0, layer_cap = 0, train_cap = 0;
  char* layer_buf = nullptr;  // holds tgt and the hidden layers' z and a
  bf16* train_buf = nullptr;  // holds dz, dzt and at
  bf16* xb = nullptr;        // [cap][in_p]
  float* xf = nullptr;       // staging for uploads [cap][max(in_p, out_p)]
  float* z[kLayers] = {};    // pre-activations [cap][rows]
  bf16* a[kLayers] = {};     // hidden activations [cap][rows]
  float* tgt = nullptr;      // targets [cap][out_p]
  bf16* dz[kLayers] = {};    // [cap][rows]
  bf16* dzt[kLayers] = {};   // transposed [rows][batch rows]
  bf16* at[kLayers] = {};    // transposed inputs of the layers [cols][batch rows]
  double* loss_part = nullptr;
  int64_t loss_cap = 0;
  // training set
  bf16* dx = nullptr;
  float* dt = nullptr;
  int64_t n_data = 0;
  int* d_idx = nullptr;
  int device = 0;
  HostStage stage;  // rows of inference and gradient calls
};

namespace {

#define MCK(call)                                                                    \
  do {                                                                               \
    cudaError_t e_ = (call);                                                         \
    if (e_ != cudaSuccess) {                                                         \
      m->err = std::string(#call) + ": " + cudaGetErrorString(e_);                   \
      return FELIS_CUDA_ERROR;                                                       \
    }                                                                                \
  } while (0)

felis_status mfail(felis_mlp* m, felis_status s, const std::string& e) {
  if (m) m->err = e;
  return s;
}

// Host rows [n][c_real] (FP32) -> device padded rows [n][c_pad].
felis_status upload_rows(felis_mlp* m, const float* h, int64_t n, int c_real, int c_pad, float* d) {
  std::vector<float> buf((size_t)n * c_pad, 0.f);
  for (int64_t r = 0; r < n; ++r) memcpy(&buf[(size_t)r * c_pad], h + (size_t)r * c_real, c_real * sizeof(float));
  MCK(cudaMemcpyAsync(d, buf.data(), buf.size() * sizeof(float), cudaMemcpyHostToDevice, m->st));
  MCK(cudaStreamSynchronize(m->st));
  return FELIS_OK;
}

// Buffers of an inference pass over `rows` rows; the hidden layers' and the
// targets' only where `layers` (the fused kernel keeps them on chip).
felis_status ensure_cap(felis_mlp* m, int rows, bool layers) {
  if (rows > m->cap) {
    void** bufs[] = {(void**)&m->xb, (void**)&m->xf, (void**)&m->z[kLayers - 1]};
    for (auto b : bufs) { if (*b) cudaFree(*b); *b = nullptr; }
    m->cap = 0;
    MCK(cudaMalloc(&m->xb, (size_t)rows * m->in_p * sizeof(bf16)));
    MCK(cudaMalloc(&m->xf, (size_t)rows * std::max(m->in_p, m->out_p) * sizeof(float)));
    MCK(cudaMalloc(&m->z[kLayers - 1], (size_t)rows * m->out_p * sizeof(float)));
    m->cap = rows;
  }
  if (layers && rows > m->layer_cap) {
    // one allocation: every part is a multiple of 128 rows by 16 columns
    if (m->layer_buf) cudaFree(m->layer_buf);
    m->layer_buf = nullptr;
    m->layer_cap = 0;
    size_t bytes = (size_t)rows * m->out_p * sizeof(float);
    for (int l = 0; l < kLayers - 1; ++l) bytes += (size_t)rows * m->rows[l] * (sizeof(float) + sizeof(bf16));
    MCK(cudaMalloc(&m->layer_buf, bytes));
    char* at = m->layer_buf;
    auto take = [&](size_t n) { char* q = at; at += n; return q; };
    m->tgt = (float*)take((size_t)rows * m->out_p * sizeof(float));
    for (int l = 0; l < kLayers - 1; ++l) {
      m->z[l] = (float*)take((size_t)rows * m->rows[l] * sizeof(float));
      m->a[l] = (bf16*)take((size_t)rows * m->rows[l] * sizeof(bf16));
    }
    m->layer_cap = rows;
  }
  return FELIS_OK;
}

// What training needs besides: dz and the transposed operands of `rows` rows,
// and `parts` partial losses.
felis_status ensure_train(felis_mlp* m, int rows, int64_t parts) {
  felis_status s = ensure_cap(m, rows, true);
  if (s != FELIS_OK) return s;
  if (rows > m->train_cap) {
    if (m->train_buf) cudaFree(m->train_buf);
    m->train_buf = nullptr;
    m->train_cap = 0;
    size_t n = 0;
    for (int l = 0; l < kLayers; ++l) n += (size_t)rows * (2 * m->rows[l] + m->cols[l]);
    MCK(cudaMalloc(&m->train_buf, n * sizeof(bf16)));
    bf16* at = m->train_buf;
    auto take = [&](size_t k) { bf16* q = at; at += k; return q; };
    for (int l = 0; l < kLayers; ++l) {
      m->dz[l] = take((size_t)rows * m->rows[l]);
      m->dzt[l] = take((size_t)rows * m->rows[l]);
      m->at[l] = take((size_t)rows * m->cols[l]);
    }
    m->train_cap = rows;
  }
  if (parts > m->loss_cap) {
    if (m->loss_part) cudaFree(m->loss_part);
    m->loss_part = nullptr;
    m->loss_cap = 0;
    MCK(cudaMalloc(&m->loss_part, (size_t)parts * sizeof(double)));
    m->loss_cap = parts;
  }
  return FELIS_OK;
}

// One product, or two independent ones, in a launch.
void gemm(felis_mlp* m, const GemmArgs* g, int n) {
  if (launch_gemm_tma(g, n, m->st) != cudaSuccess) {
    // shapes the network never produces (M % 128, N > 256, unaligned rows):
    // reported through the error word like a device failure
    cudaMemsetAsync(m->d_err, 0xff, sizeof(int), m->st);
  }
}

// Forward pass of rows [0, M) of xb (M a multiple of 128).  Training keeps
// every layer's FP32 pre-activation z (the backward pass needs it) and the
// hidden activations both ways round; inference writes the hidden layers' BF16
// activations and the last layer's FP32 output only.
void forward(felis_mlp* m, int M, bool train = true) {
  const bf16* in = m->xb;
  int ld_in = m->in_p;
  for (int l = 0; l < kLayers; ++l) {
    const bool last = l == kLayers - 1;
    GemmArgs g{in, m->wb[l], M, m->rows[l], m->cols[l], ld_in, m->cols[l], m->p + m->b_off[l],
               (train || last) ? m->z[l] : nullptr, last ? nullptr : m->a[l],
               m->rows[l], m->rows_real[l], last ? 0 : 1, m->d_err};
    if (train && !last) {
      g.out_t = m->at[l + 1];
      g.ldt = M;
    }
    gemm(m, &g, 1);
    in = m->a[l];
    ld_in = m->rows[l];
  }
}

// The inference pass of rows [0, M) of xb as one fused kernel; the output
// goes where forward() leaves it (z of the last layer).
void forward_fused(felis_mlp* m, int M) {
  MlpFusedArgs a;
  a.x = m->xb;
  a.M = M; a.width = m->width; a.in_k = m->in_p; a.out_n = m->out_p;
  for (int l = 0; l < kLayers; ++l) {
    a.w[l] = m->wb[l];
    a.bias[l] = m->p + m->b_off[l];
  }
  a.y = m->z[kLayers - 1];
  a.err = m->d_err;
  if (launch_mlp_fused(a, m->st) != cudaSuccess) cudaMemsetAsync(m->d_err, 0xff, sizeof(int), m->st);
}

MlpLayers layers_of(const felis_mlp* m) {
  MlpLayers L{};
  for (int l = 0; l < kLayers; ++l) {
    L.w_off[l] = m->w_off[l]; L.b_off[l] = m->b_off[l];
    L.rows[l] = m->rows[l]; L.cols[l] = m->cols[l];
    L.wb[l] = m->wb[l]; L.wt[l] = m->wt[l]; L.dzt[l] = m->dzt[l];
  }
  return L;
}

// Gradients of the mean squared error over the first n_real rows of the
// chunk (targets in tgt, inputs both ways round in xb and at[0]) into m->grad;
// the squared errors' block sums go to loss_part.
void backward(felis_mlp* m, int M, int n_real, double* loss_part) {
  const int L = kLayers;
  const float scale = 2.f / ((float)n_real * (float)m->n_out);
  launch_mse_grad(m->z[L - 1], m->tgt, M, n_real, m->out_p, m->n_out, scale, m->dz[L - 1], m->dzt[L - 1], loss_part, m->st);
  for (int l = L - 1; l >= 0; --l) {
    const int R = m->rows[l], Cc = m->cols[l];
    const int Rt = l == L - 1 ? m->out_rows : R;  // dW rows (a multiple of 128; dz^T has R of them)
    GemmArgs g[2];
    // dW = dz^T . a_{l-1}: A = dz^T [R][M], B = a_{l-1}^T [Cc][M]
    g[0] = GemmArgs{m->dzt[l], m->at[l], Rt, Cc, M, M, M, nullptr, m->grad + m->w_off[l], nullptr, Cc, Cc, 0, m->d_err};
    g[0].rows_a = R;
    if (l > 0) {
      // dz_{l-1} = (dz . W_l) GELU'(z_{l-1}): A = dz [M][R], B = W_l^T [Cc][R]
      g[1] = GemmArgs{m->dz[l], m->wt[l], M, Cc, R, R, R, nullptr, nullptr, m->dz[l - 1], Cc, Cc, 0, m->d_err};
      g[1].z = m->z[l - 1];
      g[1].out_t = m->dzt[l - 1];
      g[1].ldt = M;
    }
    gemm(m, g, l > 0 ? 2 : 1);
  }
  launch_bias_grads(layers_of(m), M, m->grad, m->st);
}

felis_status refresh_bf16(felis_mlp* m) {
  for (int l = 0; l < kLayers; ++l) {
    const int64_t n = (int64_t)m->rows[l] * m->cols[l];
    launch_f32_to_bf16(m->p + m->w_off[l], m->wb[l], n, m->st);
    if (l > 0) launch_transpose_bf16(m->wb[l], m->rows[l], m->cols[l], m->cols[l], m->wt[l], m->rows[l], m->cols[l], m->st);
  }
  MCK(cudaGetLastError());
  return FELIS_OK;
}

felis_status adamw_step(felis_mlp* m, float lr, float wd) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  m->steps += 1;
  const float bc1 = 1.f - powf(b1, (float)m->steps), bc2 = 1.f - powf(b2, (float)m->steps);
  launch_adamw(layers_of(m), m->p, m->grad, m->m, m->v, lr, b1, b2, eps, wd, bc1, bc2, m->st);
  MCK(cudaGetLastError());
  return FELIS_OK;
}

felis_status check_err(felis_mlp* m) {
  int e = 0;
  MCK(cudaMemcpyAsync(&e, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->st));
  MCK(cudaStreamSynchronize(m->st));
  if (e) {
    MCK(cudaMemsetAsync(m->d_err, 0, sizeof(int), m->st));
    return mfail(m, FELIS_TIMEOUT, "tensor-core wait ran out");
  }
  return FELIS_OK;
}

// Padded parameter layout <-> flat unpadded layout W1, b1, ..., W4, b4.
int64_t flat_count(const felis_mlp* m) {
  int64_t n = 0;
  for (int l = 0; l < kLayers; ++l) n += (int64_t)m->rows_real[l] * m->cols_real[l] + m->rows_real[l];
  return n;
}

}  // namespace

extern "C" {

felis_status felis_mlp_create(int32_t n_in, int32_t width, int32_t n_out, uint64_t seed, felis_mlp** out) {
  if (!out || n_in < 1 || n_out < 1 || (width != 128 && width != 256) || n_in > 256 || n_out > width)
    return FELIS_BAD_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return FELIS_NO_DEVICE;
  felis_mlp* m = new felis_mlp();
  m->n_in = n_in; m->width = width; m->n_out = n_out;
  m->in_p = round_up(n_in, 16);
  m->out_p = round_up(n_out, 16);
  m->out_rows = round_up(m->out_p, 128);
  m->fused = mlp_fused_supported(width, m->in_p, m->out_p);
  const int r[kLayers] = {width, width, width, m->out_p};
  const int c[kLayers] = {m->in_p, width, width, width};
  const int rr[kLayers] = {width, width, width, n_out};
  const int cr[kLayers] = {n_in, width, width, width};
  size_t off = 0;
  for (int l = 0; l < kLayers; ++l) {
    m->rows[l] = r[l]; m->cols[l] = c[l]; m->rows_real[l] = rr[l]; m->cols_real[l] = cr[l];
    m->w_off[l] = off;
    // the last layer's gradient block is written as out_rows rows by the GEMM
    off += (size_t)(l == kLayers - 1 ? m->out_rows : r[l]) * c[l];
    m->b_off[l] = off;
    off += round_up(r[l], 4);
  }
  m->n_param = off;
  auto bad = [&](felis_status s, const char* msg) {
    fprintf(stderr, "felis_mlp_create: %s\n", msg);
    felis_mlp_destroy(m);
    return s;
  };
  cudaGetDevice(&m->device);
  cudaError_t e = cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&m->d_err, sizeof(int));
  if (e == cudaSuccess) e = cudaMemsetAsync(m->d_err, 0, sizeof(int), m->st);
  float** fb[] = {&m->p, &m->grad, &m->m, &m->v};
  for (auto f : fb) {
    if (e == cudaSuccess) e = cudaMalloc(f, m->n_param * sizeof(float));
    if (e == cudaSuccess) e = cudaMemsetAsync(*f, 0, m->n_param * sizeof(float), m->st);
  }
  for (int l = 0; l < kLayers && e == cudaSuccess; ++l) {
    e = cudaMalloc(&m->wb[l], (size_t)r[l] * c[l] * sizeof(bf16));
    if (e == cudaSuccess) e = cudaMalloc(&m->wt[l], (size_t)r[l] * c[l] * sizeof(bf16));
  }
  if (e == cudaSuccess) e = gemm_tma_prepare();
  if (e == cudaSuccess) e = mlp_fused_prepare();
  if (e == cudaSuccess) e = cudaEventCreate(&m->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&m->ev1);
  if (e != cudaSuccess) return bad(FELIS_CUDA_ERROR, cudaGetErrorString(e));
  // He-style initialisation for GELU layers (std sqrt(2 / fan_in)), zero biases
  std::mt19937_64 rng(seed ? seed : 1);
  std::vector<float> h(m->n_param, 0.f);
  for (int l = 0; l < kLayers; ++l) {
    std::normal_distribution<float> nd(0.f, sqrtf((l == kLayers - 1 ? 1.f : 2.f) / (float)m->cols_real[l]));
    for (int i = 0; i < m->rows_real[l]; ++i)
      for (int j = 0; j < m->cols_real[l]; ++j) h[m->w_off[l] + (size_t)i * c[l] + j] = nd(rng);
  }
  e = to_device(m->p, h.data(), h.size() * sizeof(float), m->st);
  if (e != cudaSuccess) return bad(FELIS_CUDA_ERROR, cudaGetErrorString(e));
  if (refresh_bf16(m) != FELIS_OK) return bad(FELIS_CUDA_ERROR, m->err.c_str());
  *out = m;
  return FELIS_OK;
}

void felis_mlp_destroy(felis_mlp* m) {
  if (!m) return;
  if (m->st) cudaStreamSynchronize(m->st);
  void* ptrs[] = {m->d_err, m->p, m->grad, m->m, m->v, m->xb, m->xf, m->z[kLayers - 1],
                  m->layer_buf, m->train_buf, m->loss_part, m->dx, m->dt, m->d_idx};
  for (void* q : ptrs) if (q) cudaFree(q);
  for (int l = 0; l < kLayers; ++l) {
    void* q[] = {m->wb[l], m->wt[l]};
    for (void* x : q) if (x) cudaFree(x);
  }
  if (m->ev0) cudaEventDestroy(m->ev0);
  if (m->ev1) cudaEventDestroy(m->ev1);
  if (m->st) cudaStreamDestroy(m->st);
  delete m;
}

const char* felis_mlp_last_error(const felis_mlp* m) { return m ? m->err.c_str() : "null network"; }

felis_status felis_mlp_param_count(const felis_mlp* m, int64_t* count) {
  if (!m || !count) return FELIS_BAD_ARG;
  *count = flat_count(m);
  return FELIS_OK;
}

felis_status felis_mlp_get_params(felis_mlp* m, float* out) {
  if (!m || !out) return FELIS_BAD_ARG;
  std::vector<float> h(m->n_param);
  MCK(cudaStreamSynchronize(m->st));
  MCK(cudaMemcpy(h.data(), m->p, h.size() * sizeof(float), cudaMemcpyDeviceToHost));
  int64_t k = 0;
  for (int l = 0; l < kLayers; ++l) {
    for (int i = 0; i < m->rows_real[l]; ++i)
      for (int j = 0; j < m->cols_real[l]; ++j) out[k++] = h[m->w_off[l] + (size_t)i * m->cols[l] + j];
    for (int i = 0; i < m->rows_real[l]; ++i) out[k++] = h[m->b_off[l] + i];
  }
  return FELIS_OK;
}

felis_status felis_mlp_set_params(felis_mlp* m, const float* in) {
  if (!m || !in) return FELIS_BAD_ARG;
  std::vector<float> h(m->n_param, 0.f);
  int64_t k = 0;
  for (int l = 0; l < kLayers; ++l) {
    for (int i = 0; i < m->rows_real[l]; ++i)
      for (int j = 0; j < m->cols_real[l]; ++j) h[m->w_off[l] + (size_t)i * m->cols[l] + j] = in[k++];
    for (int i = 0; i < m->rows_real[l]; ++i) h[m->b_off[l] + i] = in[k++];
  }
  MCK(cudaStreamSynchronize(m->st));
  MCK(to_device(m->p, h.data(), h.size() * sizeof(float), m->st));
  MCK(cudaMemsetAsync(m->m, 0, m->n_param * sizeof(float), m->st));
  MCK(cudaMemsetAsync(m->v, 0, m->n_param * sizeof(float), m->st));
  m->steps = 0;
  return refresh_bf16(m);
}

felis_status felis_mlp_forward(felis_mlp* m, const float* x, int64_t n, float* y) {
  if (!m || n < 0 || (n > 0 && (!x || !y))) return mfail(m, FELIS_BAD_ARG, "bad argument");
  felis_status s =
      ensure_cap(m, (int)std::min<int64_t>(round_up((int)std::min<int64_t>(n, kFwdChunk), 128), kFwdChunk), !m->fused);
  if (s != FELIS_OK) return s;
  for (int64_t r0 = 0; r0 < n; r0 += kFwdChunk) {
    const int nr = (int)std::min<int64_t>(kFwdChunk, n - r0);
    const int M = round_up(nr, 128);
    // the rows cross the link as they are, in and out; padding and rounding
    // are done on the device
    const CopyPart in{x + (size_t)r0 * m->n_in, m->xf, (size_t)nr * m->n_in * sizeof(float)};
    MCK(m->stage.upload(&in, 1, m->device, m->st));
    launch_pack_rows(m->xf, nr, m->n_in, M, m->in_p, m->xb, m->st);
    MCK(cudaEventRecord(m->ev0, m->st));
    if (m->fused) forward_fused(m, M);
    else forward(m, M, false);
    MCK(cudaEventRecord(m->ev1, m->st));
    launch_unpad_rows(m->z[kLayers - 1], nr, m->out_p, m->n_out, m->xf, m->st);
    MCK(cudaGetLastError());
    const CopyPart out{m->xf, y + (size_t)r0 * m->n_out, (size_t)nr * m->n_out * sizeof(float)};
    MCK(m->stage.download(&out, 1, false, m->device, m->st));
    MCK(cudaStreamSynchronize(m->st));
    float ms = 0.f;
    MCK(cudaEventElapsedTime(&ms, m->ev0, m->ev1));
    m->fwd_ms = ms;
    double fl = 0.0;
    for (int l = 0; l < kLayers; ++l) fl += 2.0 * M * m->rows[l] * m->cols[l];
    m->fwd_flops = fl;
  }
  return check_err(m);
}

felis_status felis_mlp_set_fused(felis_mlp* m, int32_t enable) {
  if (!m) return FELIS_BAD_ARG;
  if (enable && !mlp_fused_supported(m->width, m->in_p, m->out_p))
    return mfail(m, FELIS_UNSUPPORTED, "the fused inference kernel needs width 256, n_in <= 64, n_out <= 256");
  m->fused = enable != 0;
  return FELIS_OK;
}

felis_status felis_mlp_gradients(felis_mlp* m, const float* x, const float* t, int64_t n, float* grads,
                                 double* loss) {
  if (!m || !x || !t || n < 1 || n > kChunk) return mfail(m, FELIS_BAD_ARG, "bad argument (1 <= n <= 65536)");
  const int M = round_up((int)n, 128), parts = mse_blocks(M);
  felis_status s = ensure_train(m, M, parts);
  if (s != FELIS_OK) return s;
  // rows and targets as they are, padded on the device by way of the first
  // and the last layer's z, which the forward pass has not written yet (a row
  // of z is at least 128 floats or the padded outputs; of inputs at most 256
  // 16-bit values)
  bf16* rows = reinterpret_cast<bf16*>(m->z[0]);
  const CopyPart in{x, m->xf, (size_t)n * m->n_in * sizeof(float)};
  MCK(m->stage.upload(&in, 1, m->device, m->st));
  launch_pack_rows(m->xf, (int)n, m->n_in, M, m->in_p, rows, m->st);
  const CopyPart tg{t, m->xf, (size_t)n * m->n_out * sizeof(float)};
  MCK(m->stage.upload(&tg, 1, m->device, m->st));
  launch_pad_rows(m->xf, (int)n, m->n_out, m->out_p, m->z[kLayers - 1], m->st);
  launch_batch_rows(rows, m->z[kLayers - 1], nullptr, (int)n, M, m->in_p, m->out_p, m->xb, m->at[0], m->tgt, m->st);
  forward(m, M);
  backward(m, M, (int)n, m->loss_part);
  std::vector<double> part(parts);
  MCK(cudaMemcpyAsync(part.data(), m->loss_part, parts * sizeof(double), cudaMemcpyDeviceToHost, m->st));
  MCK(cudaStreamSynchronize(m->st));
  double sse = 0.0;
  for (double v : part) sse += v;
  if ((s = check_err(m)) != FELIS_OK) return s;
  std::vector<float> h(m->n_param);
  MCK(cudaMemcpy(h.data(), m->grad, h.size() * sizeof(float), cudaMemcpyDeviceToHost));
  int64_t k = 0;
  for (int l = 0; l < kLayers; ++l) {
    for (int i = 0; i < m->rows_real[l]; ++i)
      for (int j = 0; j < m->cols_real[l]; ++j) grads[k++] = h[m->w_off[l] + (size_t)i * m->cols[l] + j];
    for (int i = 0; i < m->rows_real[l]; ++i) grads[k++] = h[m->b_off[l] + i];
  }
  if (loss) *loss = sse / ((double)n * m->n_out);
  return FELIS_OK;
}

felis_status felis_mlp_set_data(felis_mlp* m, const float* x, const float* t, int64_t n) {
  if (!m || !x || !t || n < 1) return mfail(m, FELIS_BAD_ARG, "bad argument");
  if (m->dx) cudaFree(m->dx);
  if (m->dt) cudaFree(m->dt);
  if (m->d_idx) cudaFree(m->d_idx);
  m->dx = nullptr; m->dt = nullptr; m->d_idx = nullptr;
  float* tmp = nullptr;
  MCK(cudaMalloc(&m->dx, (size_t)n * m->in_p * sizeof(bf16)));
  MCK(cudaMalloc(&m->dt, (size_t)n * m->out_p * sizeof(float)));
  MCK(cudaMalloc(&m->d_idx, (size_t)n * sizeof(int)));
  MCK(cudaMalloc(&tmp, (size_t)n * m->in_p * sizeof(float)));
  felis_status s = upload_rows(m, x, n, m->n_in, m->in_p, tmp);
  if (s == FELIS_OK) {
    launch_f32_to_bf16(tmp, m->dx, n * m->in_p, m->st);
    s = upload_rows(m, t, n, m->n_out, m->out_p, m->dt);
  }
  cudaStreamSynchronize(m->st);
  cudaFree(tmp);
  m->n_data = n;
  return s;
}

felis_status felis_mlp_train(felis_mlp* m, int32_t epochs, int32_t batch, float lr, float weight_decay,
                             uint64_t seed, double* loss_per_epoch) {
  if (!m || epochs < 1 || batch < 128 || batch % 128 || batch > kChunk || m->n_data < 1)
    return mfail(m, FELIS_BAD_ARG, "bad argument (batch a multiple of 128, data set first)");
  const int64_t batches = (m->n_data + batch - 1) / batch;
  const int parts = mse_blocks(batch);
  felis_status s = ensure_train(m, batch, batches * parts);
  if (s != FELIS_OK) return s;
  std::mt19937_64 rng(seed ? seed : 1);
  std::vector<int> perm(m->n_data);
  std::vector<double> part((size_t)(batches * parts));
  for (int64_t i = 0; i < m->n_data; ++i) perm[i] = (int)i;
  for (int ep = 0; ep < epochs; ++ep) {
    std::shuffle(perm.begin(), perm.end(), rng);
    MCK(cudaMemcpyAsync(m->d_idx, perm.data(), perm.size() * sizeof(int), cudaMemcpyHostToDevice, m->st));
    // the batches of an epoch follow one another on the stream; their losses
    // are read once at its end
    for (int64_t b = 0; b < batches; ++b) {
      const int64_t b0 = b * batch;
      const int nr = (int)std::min<int64_t>(batch, m->n_data - b0);
      const int M = round_up(nr, 128);
      launch_batch_rows(m->dx, m->dt, m->d_idx + b0, nr, M, m->in_p, m->out_p, m->xb, m->at[0], m->tgt, m->st);
      forward(m, M);
      backward(m, M, nr, m->loss_part + b * parts);
      if ((s = adamw_step(m, lr, weight_decay)) != FELIS_OK) return s;
    }
    MCK(cudaMemcpyAsync(part.data(), m->loss_part, part.size() * sizeof(double), cudaMemcpyDeviceToHost, m->st));
    MCK(cudaStreamSynchronize(m->st));
    double sse = 0.0;
    for (int64_t b = 0; b < batches; ++b) {
      const int nr = (int)std::min<int64_t>(batch, m->n_data - b * batch), np = mse_blocks(round_up(nr, 128));
      double sum = 0.0;
      for (int k = 0; k < np; ++k) sum += part[(size_t)(b * parts + k)];
      sse += sum;
    }
    if (loss_per_epoch) loss_per_epoch[ep] = sse / ((double)m->n_data * m->n_out);
  }
  return check_err(m);
}

felis_status felis_mlp_last_forward(const felis_mlp* m, double* ms, double* flops) {
  if (!m || !ms || !flops) return FELIS_BAD_ARG;
  *ms = m->fwd_ms;
  *flops = m->fwd_flops;
  return FELIS_OK;
}

felis_status felis_wait_selftest(int32_t limit, int32_t* timed_out) {
  if (limit < 1 || !timed_out) return FELIS_BAD_ARG;
  int* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(int));
  if (e == cudaSuccess) {
    launch_wait_selftest(limit, d, 0);
    e = cudaGetLastError();
  }
  int h = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(int), cudaMemcpyDeviceToHost);
  if (d) cudaFree(d);
  if (e != cudaSuccess) return FELIS_CUDA_ERROR;
  *timed_out = h;
  return h ? FELIS_TIMEOUT : FELIS_OK;
}

}  // extern "C"
