// The distance model's training passes (mlp.cuh has the model): forward and
// backward as sequences of tensor-core products with every activation kept.
// Adam's first steps divide a gradient by its own size, so sums in another order
// end in other parameters: a pass fused over 128-row tiles, which added its tiles'
// weight gradients with atomics, was three to five times faster and moved an
// epoch's parameters by up to 2e-4 of their norm (both are 4e-3 of it from 64 bits).
// Here a weight gradient is one accumulation over the batch (two from 1024 rows on);
// the head's adds 64-row parts and the bias sums 256-row parts with atomics.
#pragma once
#include <cuda_bf16.h>

#include <vector>

#include "automaton.hpp"
#include "common.cuh"
#include "mlp.cuh"

namespace sw {
namespace train {
using namespace mlp;

// A bf16 matrix view: element (i, k) at p[i * si + k * sk].
struct View {
  const __nv_bfloat16* p;
  long long si, sk;
};

// C[i*ldc + j] (= or +=) sum_k A(i,k) B(k,j) for i < M, j < N <= 128; `atomic`
// accumulates with atomicAdd (required when split > 1: K is cut in `split`
// slices, one per grid z).
void gemm(View A, View B, float* C, int ldc, int M, int N, int K, bool atomic, int split, cudaStream_t s);
// True once a product's bounded wait for its tensor-core work ran out (its
// results are then incomplete); synchronises with the device.
bool tc_error();

// Set rows (device layout, W words) -> dense 0/1 bf16 rows of width ld (>= n).
void bits_to_dense(const u64* rows, int W, int n, u32 count, __nv_bfloat16* out, int ld, cudaStream_t s);

// act = bf16(relu(in + bias)); keeps `in + bias` in `pre` when pre != nullptr.
// With relu == false only the bias is added.
void bias_act(const float* in, const float* bias, int rows, int cols, bool relu, float* pre, __nv_bfloat16* act,
              cudaStream_t s);

// y[b] = sum_j H[b][j] * w3[j] + b3 (w3, b3 from the fp32 parameters).
void head(const __nv_bfloat16* H, const float* params, int rows, float* y, cudaStream_t s);

// Loss 1/B sum (y - t)^2 (loss[0] += ...) and dy = 2 (y - t) / B.
void mse(const float* y, const float* t, int rows, float* dy, float* loss, cudaStream_t s);
// Adds w/B sum over pairs of one group with t_a < t_b of softplus(y_a - y_b)
// to the loss and its gradient to dy (a within-layer ranking term).
void rank_add(const float* y, const float* t, const uint32_t* grp, int rows, float w, float* dy, float* loss,
              cudaStream_t s);

// From dy: grad of w3 and b3 (grad vector, accumulated), and the masked
// hidden gradient dH = dy w3^T * [pre > 0] (fp32 and bf16).
void head_back(const float* dy, const __nv_bfloat16* H, const float* pre, const float* params, int rows, float* grad,
               float* dH, __nv_bfloat16* dHb, cudaStream_t s);

// d = d * [pre > 0] in place, bf16 copy in db (nullptr: none).
void relu_back(float* d, const float* pre, int count, __nv_bfloat16* db, cudaStream_t s);

// out[j] += sum_i M[i*cols + j].
void col_sum(const float* M, int rows, int cols, float* out, cudaStream_t s);

// fp32 -> bf16.
void to_bf16(const float* in, __nv_bfloat16* out, int count, cudaStream_t s);

// Adam step (t = 1-based step count) on the parameter vector.
void adam(float* p, const float* g, float* m, float* v, int count, float lr, int t, cudaStream_t s);

}  // namespace train

class Trainer {
 public:
  explicit Trainer(cudaStream_t s) : stream_(s) {}

  // Parameters: mlp::kParams floats on the device (layout in mlp.cuh); no moments.
  void set_params(const float* device);
  void get_params(float* host);
  bool has_params() const { return loaded_; }

  // Embedding table of automaton A (its state features through Phi, c, relu).
  void prepare(const Automaton& A);

  // y[i] = predicted distance of rows[i] (device layout, W words per row),
  // for the automaton last prepared.  Activations stay for backward().
  void forward(const u64* rows, int W, u32 count, float* y);

  // After forward() on the same rows: gradient of the mean squared error
  // against targets t (device) added into grad(); loss added into loss().
  // With `grp` (a group id per row, e.g. its BFS layer) and rank_w > 0 the
  // loss adds rank_w times a pairwise ranking term within each group.
  void backward(const float* t, u32 count, const uint32_t* grp = nullptr, float rank_w = 0.0f);

  void zero_grad();
  void adam_step(float lr);  // then refreshes the bf16 weight copies
  float* grad() { return grad_.as<float>(); }
  float* loss() { return loss_.as<float>(); }

 private:
  cudaStream_t stream_;
  bool loaded_ = false;
  int n_ = 0, step_ = 0;
  std::vector<uint32_t> feat_key_;  // automaton whose features are in feat_ (n, k, table)
  u32 count_ = 0;
  DevBuf params_, grad_, m_, v_, loss_;
  DevBuf phi_b_, w1_b_, w2_b_, feat_, feat_b_, epre_, e_b_;
  DevBuf bits_, x_, xb_, h1_, h1b_, h2_, h2b_, dy_, dh2_, dh2b_, dh1_, dh1b_, dx_, dxb_, de_, deb_;
  void refresh_bf16();
  void reserve_batch(u32 count);
};


}  // namespace sw
