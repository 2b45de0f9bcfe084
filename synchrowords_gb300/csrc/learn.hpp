// Host side of the learned distance model (mlp.cuh): parameters, the
// per-automaton embedding table and scoring (train.hpp trains).
#pragma once
#include <cuda_bf16.h>

#include <vector>

#include "automaton.hpp"
#include "common.cuh"
#include "mlp.cuh"

namespace sw {

class MlpRunner {
 public:
  // error: device word that a launch whose tensor-core wait ran out sets
  // (mlp::kErrorWait); whoever reads a launch's results back reads it with them.
  MlpRunner(cudaStream_t s, u32* error) : stream_(s), error_(error) {}

  // Parameters: host vector of mlp::kParams floats (layout in mlp.cuh).
  void set_params(const float* host);
  void get_params(float* host);
  bool has_params() const { return loaded_; }
  const float* params() const { return params_.as<float>(); }  // on the device

  // Embedding table of automaton A (its state features through Phi, c, relu).
  void prepare(const Automaton& A);

  // y[i] = predicted distance of rows[i] (device layout, W words per row),
  // for the automaton last prepared.
  void forward(const u64* rows, int W, u32 count, float* y);

 private:
  cudaStream_t stream_;
  u32* error_;
  bool loaded_ = false;
  int n_ = 0;
  std::vector<uint32_t> feat_key_;  // automaton whose features are in feat_ (n, k, table)
  DevBuf params_, weights_;
  DevBuf feat_, e_;                 // features, embeddings (staged bf16)
};

}  // namespace sw
