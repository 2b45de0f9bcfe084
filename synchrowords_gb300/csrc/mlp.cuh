// Learned distance model: a set S of states is scored by
//   E   = relu(feat · Phi + c)                  per-state embeddings, n x 64 (bf16)
//   x   = sum over q in S of E[q]                (= bits(S) · E, a tensor-core product)
//   h1  = relu(x · W1 + b1),  h2 = relu(h1 · W2 + b2)   (64 -> 128 -> 128)
//   y   = h2 · w3 + b3                            predicted shortest merge length
// feat is a fixed per-state feature vector of the automaton (automaton.cpp),
// so one trained model applies to automata of any size.  The products over a
// batch run on the tensor cores (tcgen05.mma, bf16 inputs, fp32 accumulation in
// TMEM); master weights, gradients and Adam moments are fp32.  A training step is
// six launches (mlp.cu): embeddings, forward, loss, backward, the embeddings'
// gradient, Adam.
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
// shared memory (mlp.cu), as the forward pass and as the backward pass needs
// them; element counts.
constexpr int kStagedW1 = kEmb * kHidden, kStagedW2 = kHidden * kHidden;
constexpr int kOffW1F = 0, kOffW1B = kOffW1F + kStagedW1, kOffW2F = kOffW1B + kStagedW1,
              kOffW2B = kOffW2F + kStagedW2, kStagedWeights = kOffW2B + kStagedW2;

// Elements of the staged embeddings of n states (whole 64-state slices).
inline size_t staged_embeddings(int n) { return (size_t)((n + 63) / 64) * 64 * kEmb; }

// Activations a backward pass needs (null pointers: scoring only).
struct Activations {
  bf16 *x = nullptr, *h1 = nullptr, *h2 = nullptr;  // [rows][64], [rows][128], [rows][128]
  u32 *open1 = nullptr, *open2 = nullptr;           // [rows][4]: bit c of word c / 32 = pre-activation above zero
};

// What a launch leaves in the error word it was given when a bounded wait for its
// tensor-core work ran out (its results are then incomplete).
constexpr u32 kErrorWait = 4;

// epre = feat · Phi + c (fp32, n x 64), staged = bf16(relu(epre)).
void embed(const float* feat, const float* params, int n, float* epre, bf16* staged, u32* err, cudaStream_t s);
// y of `count` sets (device rows of W words).
void forward(const u64* rows, int W, int n, u32 count, const bf16* staged_e, const bf16* weights, const float* params,
             float* y, const Activations& act, u32* err, cudaStream_t s);
void stage_weights(const float* p, bf16* weights, cudaStream_t s);

}  // namespace mlp
}  // namespace sw
