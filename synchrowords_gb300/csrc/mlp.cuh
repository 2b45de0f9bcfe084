// Learned distance model: a set S of states is scored by
//   E   = relu(feat · Phi + c)                  per-state embeddings, n x 64 (bf16)
//   x   = sum over q in S of E[q]                (= bits(S) · E, a tensor-core product)
//   h1  = relu(x · W1 + b1),  h2 = relu(h1 · W2 + b2)   (64 -> 128 -> 128)
//   y   = h2 · w3 + b3                            predicted shortest merge length
// feat is a fixed per-state feature vector of the automaton (automaton.cpp),
// so one trained model applies to automata of any size.  The products over a
// batch run on the tensor cores (tcgen05.mma, bf16 inputs, fp32 accumulation in
// TMEM); master weights, gradients and Adam moments are fp32.  Scoring is one launch
// (mlp.cu); training runs every product, bias, conversion and sum as a launch of its
// own (train.hpp).
#pragma once
#include <cuda_bf16.h>

#include "common.cuh"

namespace sw {
namespace mlp {

constexpr int kFeat = 16;    // per-state features
constexpr int kEmb = 64;     // embedding width
constexpr int kHidden = 128; // hidden width

// Offsets (floats) into the flat parameter vector.
constexpr int kOffPhi = 0;                            // [kFeat][kEmb]
constexpr int kOffC = kOffPhi + kFeat * kEmb;         // [kEmb]
constexpr int kOffW1 = kOffC + kEmb;                  // [kEmb][kHidden]
constexpr int kOffB1 = kOffW1 + kEmb * kHidden;       // [kHidden]
constexpr int kOffW2 = kOffB1 + kHidden;              // [kHidden][kHidden]
constexpr int kOffB2 = kOffW2 + kHidden * kHidden;    // [kHidden]
constexpr int kOffW3 = kOffB2 + kHidden;              // [kHidden]
constexpr int kOffB3 = kOffW3 + kHidden;              // [1]
constexpr int kParams = kOffB3 + 1;

using bf16 = __nv_bfloat16;

// The dense layers' weights in bf16, in the layout their products read from
// shared memory (mlp.cu); element counts.
constexpr int kStagedW1 = kEmb * kHidden, kStagedW2 = kHidden * kHidden;
constexpr int kOffW1F = 0, kOffW2F = kOffW1F + kStagedW1, kStagedWeights = kOffW2F + kStagedW2;

// Elements of the staged embeddings of n states (whole 64-state slices).
inline size_t staged_embeddings(int n) { return (size_t)((n + 63) / 64) * 64 * kEmb; }

// What a launch leaves in the error word it was given when a bounded wait for its
// tensor-core work ran out (its results are then incomplete).
constexpr u32 kErrorWait = 4;

// staged = bf16(relu(feat · Phi + c)).
void embed(const float* feat, const float* params, int n, bf16* staged, u32* err, cudaStream_t s);
// y of `count` sets (device rows of W words).
void forward(const u64* rows, int W, int n, u32 count, const bf16* staged_e, const bf16* weights, const float* params,
             float* y, u32* err, cudaStream_t s);
void stage_weights(const float* p, bf16* weights, cudaStream_t s);

}  // namespace mlp
}  // namespace sw
