// MlpRunner (learn.hpp): scoring with the learned distance model (mlp.cu).
#include "learn.hpp"

namespace sw {

using mlp::bf16;

void MlpRunner::set_params(const float* host) {
  params_.reserve(sizeof(float) * mlp::kParams);
  weights_.reserve(sizeof(bf16) * mlp::kStagedWeights);
  SW_CUDA(cudaMemcpyAsync(params_.p, host, sizeof(float) * mlp::kParams, cudaMemcpyHostToDevice, stream_));
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
    feat_key_.clear();  // until they are there: growing the buffer gives up the ones it holds
    const std::vector<float> f = state_features(A);
    feat_.reserve(sizeof(float) * f.size());
    SW_CUDA(cudaMemcpyAsync(feat_.p, f.data(), sizeof(float) * f.size(), cudaMemcpyHostToDevice, stream_));
    SW_CUDA(cudaStreamSynchronize(stream_));  // f is released at the end of this block
    feat_key_ = std::move(key);
  }
  e_.reserve(sizeof(bf16) * mlp::staged_embeddings(n_));
  mlp::embed(feat_.as<float>(), params_.as<float>(), n_, e_.as<bf16>(), error_, stream_);
}

void MlpRunner::forward(const u64* rows, int W, u32 count, float* y) {
  mlp::forward(rows, W, n_, count, e_.as<bf16>(), weights_.as<bf16>(), params_.as<float>(), y, error_,
               stream_);
}

}  // namespace sw
