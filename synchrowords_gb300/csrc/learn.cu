// MlpRunner (learn.hpp): the forward and backward passes of the learned
// distance model as sequences of the launches of mlp.cu.
#include "learn.hpp"

namespace sw {

using mlp::bf16;

void MlpRunner::set_params(const float* host) {
  params_.reserve(sizeof(float) * mlp::kParams);
  grad_.reserve(sizeof(float) * mlp::kParams);
  m_.reserve(sizeof(float) * mlp::kParams);
  v_.reserve(sizeof(float) * mlp::kParams);
  loss_.reserve(sizeof(float) * 4);
  weights_.reserve(sizeof(bf16) * mlp::kStagedWeights);
  SW_CUDA(cudaMemcpyAsync(params_.p, host, sizeof(float) * mlp::kParams, cudaMemcpyHostToDevice, stream_));
  SW_CUDA(cudaMemsetAsync(m_.p, 0, sizeof(float) * mlp::kParams, stream_));
  SW_CUDA(cudaMemsetAsync(v_.p, 0, sizeof(float) * mlp::kParams, stream_));
  step_ = 0;
  mlp::stage_weights(params_.as<float>(), weights_.as<bf16>(), stream_);
  SW_CUDA(cudaStreamSynchronize(stream_));
  loaded_ = true;
}

void MlpRunner::get_params(float* host) {
  SW_CUDA(cudaMemcpyAsync(host, params_.p, sizeof(float) * mlp::kParams, cudaMemcpyDeviceToHost, stream_));
  SW_CUDA(cudaStreamSynchronize(stream_));
}

void MlpRunner::prepare(const Automaton& A) {
  if (!loaded_) throw std::runtime_error("no distance model loaded");
  n_ = (int)A.n;
  std::vector<uint32_t> key{A.n, A.k};
  key.insert(key.end(), A.t.begin(), A.t.end());
  if (key != feat_key_) {  // features depend on the automaton only: computed once per automaton
    const std::vector<float> f = state_features(A);
    feat_.reserve(sizeof(float) * f.size());
    SW_CUDA(cudaMemcpyAsync(feat_.p, f.data(), sizeof(float) * f.size(), cudaMemcpyHostToDevice, stream_));
    SW_CUDA(cudaStreamSynchronize(stream_));  // f is released at the end of this block
    feat_key_ = std::move(key);
  }
  epre_.reserve(sizeof(float) * n_ * mlp::kEmb);
  e_.reserve(sizeof(bf16) * mlp::staged_embeddings(n_));
  mlp::embed(feat_.as<float>(), params_.as<float>(), n_, epre_.as<float>(), e_.as<bf16>(), stream_);
}

void MlpRunner::forward(const u64* rows, int W, u32 count, float* y) {
  mlp::forward(rows, W, n_, count, e_.as<bf16>(), weights_.as<bf16>(), params_.as<float>(), y, mlp::Activations{},
               stream_);
}

void MlpRunner::zero_grad() {
  SW_CUDA(cudaMemsetAsync(grad_.p, 0, sizeof(float) * mlp::kParams, stream_));
  SW_CUDA(cudaMemsetAsync(loss_.p, 0, sizeof(float), stream_));
}

void MlpRunner::gradient(const u64* rows, int W, u32 count, const float* t, const uint32_t* grp, float rank_w,
                         float* loss) {
  if (!count) return;
  const size_t c = count;
  x_.reserve(sizeof(bf16) * c * mlp::kEmb);
  h1_.reserve(sizeof(bf16) * c * mlp::kHidden);
  h2_.reserve(sizeof(bf16) * c * mlp::kHidden);
  open_.reserve(sizeof(u32) * c * 8);
  y_.reserve(sizeof(float) * c * 2);
  const size_t de_bytes = sizeof(float) * mlp::kEmb * (size_t)n_;
  if (de_.cap < de_bytes) {  // the backward launches leave it zero
    de_.reserve(de_bytes);
    SW_CUDA(cudaMemsetAsync(de_.p, 0, de_.cap, stream_));
  }
  const mlp::Activations act{x_.as<bf16>(), h1_.as<bf16>(), h2_.as<bf16>(), open_.as<u32>(), open_.as<u32>() + 4 * c};
  float *y = y_.as<float>(), *dy = y + c;
  mlp::forward(rows, W, n_, count, e_.as<bf16>(), weights_.as<bf16>(), params_.as<float>(), y, act, stream_);
  mlp::loss(y, t, grp, (int)count, grp ? rank_w : 0.0f, dy, loss, stream_);
  mlp::backward(rows, W, n_, count, dy, weights_.as<bf16>(), params_.as<float>(), act, grad_.as<float>(),
                de_.as<float>(), stream_);
  mlp::embed_back(feat_.as<float>(), epre_.as<float>(), n_, de_.as<float>(), grad_.as<float>(), stream_);
}

void MlpRunner::adam_step(float lr) {
  ++step_;
  mlp::adam(params_.as<float>(), grad_.as<float>(), m_.as<float>(), v_.as<float>(), weights_.as<bf16>(), lr, step_,
            stream_);
}

}  // namespace sw
