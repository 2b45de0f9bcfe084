// Host side of the learned distance model (mlp.cuh): parameters, the
// per-automaton embedding table, forward scoring, the backward pass and Adam.
#pragma once
#include <cuda_bf16.h>

#include <vector>

#include "automaton.hpp"
#include "common.cuh"
#include "mlp.cuh"

namespace sw {

class MlpRunner {
 public:
  explicit MlpRunner(cudaStream_t s) : stream_(s) {}

  // Parameters: host vector of mlp::kParams floats (layout in mlp.cuh).
  void set_params(const float* host);
  void get_params(float* host);
  bool has_params() const { return loaded_; }

  // Embedding table of automaton A (its state features through Phi, c, relu).
  void prepare(const Automaton& A);

  // y[i] = predicted distance of rows[i] (device layout, W words per row),
  // for the automaton last prepared.
  void forward(const u64* rows, int W, u32 count, float* y);

  // Adds the gradient of the mean squared error against targets t (device)
  // into grad() and the error into *loss (device).  With `grp` (a group id per row, e.g.
  // its BFS layer) and rank_w > 0 the loss adds rank_w times a pairwise
  // ranking term within each group.
  void gradient(const u64* rows, int W, u32 count, const float* t, const uint32_t* grp, float rank_w, float* loss);

  void zero_grad();          // clears grad() and loss()
  void adam_step(float lr);  // also refreshes the bf16 weight copies and clears grad()
  float* grad() { return grad_.as<float>(); }
  float* loss() { return loss_.as<float>(); }

 private:
  cudaStream_t stream_;
  bool loaded_ = false;
  int n_ = 0, step_ = 0;
  std::vector<uint32_t> feat_key_;  // automaton whose features are in feat_ (n, k, table)
  DevBuf params_, grad_, m_, v_, loss_, weights_;
  DevBuf feat_, epre_, e_;               // features, embeddings before and after the relu (staged bf16)
  DevBuf x_, h1_, h2_, open_, y_, de_;  // one batch
};

}  // namespace sw
