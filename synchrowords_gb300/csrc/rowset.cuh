// Device helpers shared by the kernels that expand layers and keep sets of
// rows in open-addressing hash tables (kernels.cu, batch_cluster.cu).
#pragma once
#include "common.cuh"

namespace sw {

__device__ __forceinline__ u32 ld_volatile(const u32* p) { return *(const volatile u32*)p; }
__device__ __forceinline__ u64 ld_volatile64(const u64* p) { return *(const volatile u64*)p; }

template <int W>
__device__ __forceinline__ u64 row_hash(const u64* x) {
  u64 h = 0x243F6A8885A308D3ULL;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    h ^= x[w];
    h *= 0x9E3779B97F4A7C15ULL;
    h ^= h >> 29;
  }
  h *= 0xD6E8FEB86659FD93ULL;
  return h ^ (h >> 32);
}

// Row at p (possibly written by another block in this launch) equals x.
template <int W>
__device__ __forceinline__ bool row_eq_volatile(const u64* p, const u64* x) {
  bool e = true;
#pragma unroll
  for (int w = 0; w < W; ++w) e = e && ld_volatile64(p + w) == x[w];
  return e;
}

// 32 x 32 bit transpose across a warp: bit l of lane i's result is bit i of
// lane l's value (five exchange stages, each swapping the off-diagonal halves).
__device__ __forceinline__ u32 transpose32(u32 v) {
  const u32 lane = threadIdx.x & 31u;
  const u32 low[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const u32 s = 16u >> i;
    const u32 o = __shfl_xor_sync(0xffffffffu, v, s);
    v = (lane & s) ? (v & ~low[i]) | ((o >> s) & low[i]) : (v & low[i]) | ((o & low[i]) << s);
  }
  return v;
}

// 32 rows, one per lane, as columns: col[q] has bit l set when lane l's row
// holds state q (q < 64 W).
template <int W>
__device__ __forceinline__ void rows_to_columns(const u64* x, u32* col) {
  const u32 lane = threadIdx.x & 31u;
#pragma unroll
  for (int w = 0; w < W; ++w) {  // lane i gets the column of bit i: state 31 - i of the half
    col[64 * w + 31 - lane] = transpose32((u32)(x[w] >> 32));
    col[64 * w + 63 - lane] = transpose32((u32)x[w]);
  }
}

// Children of 32 parents (columns `col`) under one letter, one per lane, into
// x.  Preimages: child state s is parent state delta[s * ds].  Images: child
// state t is the OR of the parent states src[beg[t] .. beg[t + 1]).
template <int W, bool kImage, class Idx, class Off>
__device__ __forceinline__ void expand_columns(const u32* col, u32 n, const Idx* delta, u32 ds, const Off* beg,
                                               const Idx* src, u64* x) {
  const u32 lane = threadIdx.x & 31u;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    u32 half[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const u32 s = 64 * w + 32 * h + lane;
      u32 v = 0;
      if (s < n) {
        if (!kImage) {
          v = col[delta[s * ds]];
        } else {
          const u32 b = beg[s], e = beg[s + 1];
          for (u32 j = b; j < e; ++j) v |= col[src[j]];
        }
      }
      half[h] = __brev(transpose32(v));
    }
    x[w] = ((u64)half[0] << 32) | half[1];
  }
}

}  // namespace sw
