// Dominance checks of one side's layer, bit-sliced: which sets of a list X lie
// inside which sets of a list T (x ⊆ t, or x ⊊ t).
//
// The searches drop a child that a visited set or a sibling dominates
// (synchrolib/algorithm/exact/meet_in_the_middle.cpp:195-237, 264-337; the
// reference asks its implicit trie, subsets_implicit_trie.hpp:29-266).
// Forward, a child is dropped when it contains such a set (T = children, the
// hits are rows of T); backward, when such a set contains it (T = the visited or
// sibling sets, the hits are rows of X; rows are complements, so sets are the
// rows' complements).  Both come down to sparse sets x and the question which t
// hold every state of x:
//   * a block turns a chunk of T into columns in shared memory: for every state
//     a bitmap over the chunk's rows (32 x 32 bit transposes);
//   * a warp takes one x at a time and ANDs the bitmaps of its states until
//     no row is left; the rows left when the states run out hold x.
// A random set of 10 to 30 states dies within four to five ANDs, 4096 rows each.
// The masks of the tiled check (subset_check.cu) reject little here, because
// a child and the sets around it share most of their leading states: counted on
// layers of 45 000 to 48 000 backward sets (n = 200, 256) its tests covered 10
// pairs per instruction, these cover 40 to 50.  Bound by the bitmaps' way
// through shared memory (128 bytes per 1024 rows and state).
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"
#include "rowset.cuh"

namespace sw {

namespace {
constexpr u32 kFullWarp = 0xffffffffu;

// Bitmap words per lane: a chunk is 1024 V rows.  Column stride in words: padded
// so that a group's 32 columns (one per lane) are stored with at most four lanes
// to a bank, and kept 16-byte aligned for V = 4 (8-byte for V = 2).
template <int V>
constexpr u32 col_stride() {
  return V == 1 ? 33 : 32 * V + (V == 4 ? 4 : 2);
}
template <int W, int V>
constexpr size_t dom_smem() {
  return sizeof(u32) * 64 * W * col_stride<V>() + sizeof(uint16_t) * 1024 * V;
}
template <int V>
constexpr int dom_threads() {
  return V == 1 ? 256 : 1024;
}

template <int V>
__device__ __forceinline__ void and_column(u32* acc, const u32* col) {
  if constexpr (V == 4) {
    const uint4 c = *reinterpret_cast<const uint4*>(col);
    acc[0] &= c.x;
    acc[1] &= c.y;
    acc[2] &= c.z;
    acc[3] &= c.w;
  } else if constexpr (V == 2) {
    const uint2 c = *reinterpret_cast<const uint2*>(col);
    acc[0] &= c.x;
    acc[1] &= c.y;
  } else {
    acc[0] &= *col;
  }
}
}  // namespace

// Block (chunk of T, slice of X).  kHitT: flags[t] = 1 for every row t of T
// that holds some x; else flags[x] = 1 for every row x of X that some t holds.
// kComp: rows are complements of the sets.  decided (may be null): rows of T
// (kHitT) or X whose answer is not wanted.
template <int W, int V, bool kComp, bool kHitT>
__global__ void __launch_bounds__(dom_threads<V>()) k_dominance(const u64* __restrict__ T, u32 tm,
                                                               const u64* __restrict__ X, u32 xm, int n, int proper,
                                                               u32 per_slice, const u32* __restrict__ decided,
                                                               u32* flags) {
  extern __shared__ __align__(16) u32 s_dom[];
  constexpr u32 kStride = col_stride<V>();
  constexpr u32 kWarps = dom_threads<V>() / 32;
  uint16_t* const s_size = reinterpret_cast<uint16_t*>(s_dom + 64 * W * kStride);
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const u32 r0 = blockIdx.x * 1024u * V, rows = min(1024u * V, tm - r0);
  for (u32 g = warp; g < 32 * V; g += kWarps) {
    const u32 r = 32 * g + lane;
    u32 size = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      u64 b = 0;
      if (r < rows) {
        b = T[(size_t)(r0 + r) * W + w];
        if (kComp) b = ~b & valid_mask(n, w);
      }
      size += __popcll(b);
      s_dom[(64 * w + 31 - lane) * kStride + g] = transpose32((u32)(b >> 32));
      s_dom[(64 * w + 63 - lane) * kStride + g] = transpose32((u32)b);
    }
    s_size[r] = (uint16_t)size;
  }
  __syncthreads();
  // the lane's rows: 32 (V lane + i) + bit; those past the chunk or decided take no part
  u32 open[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const u32 b = 32 * (V * lane + i);
    open[i] = b >= rows ? 0u : (rows - b >= 32 ? 0xffffffffu : (1u << (rows - b)) - 1u);
    if (kHitT && decided)
      for (u32 left = open[i]; left; left &= left - 1)
        if (decided[r0 + b + __ffs(left) - 1]) open[i] &= ~(left & -left);
  }
  const u32 x_end = min(xm, (blockIdx.y + 1) * per_slice);
  for (u32 x0 = blockIdx.y * per_slice + warp * 32; x0 < x_end; x0 += kWarps * 32) {
    const u32 xi = x0 + lane;
    u64 x[W];
    u32 size = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      u64 b = xi < x_end ? X[(size_t)xi * W + w] : 0ULL;
      if (kComp && xi < x_end) b = ~b & valid_mask(n, w);
      x[w] = b;
      size += __popcll(b);
    }
    bool want = xi < x_end;
    if (!kHitT && want) want = !*(volatile u32*)(flags + xi) && !(decided && decided[xi]);
    u32 todo = __ballot_sync(kFullWarp, want);
    while (todo) {
      const int j = __ffs(todo) - 1;
      todo &= todo - 1;
      u32 acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i) acc[i] = open[i];
      bool alive = true;
      // states are numbered by falling frequency in images: the last ones first,
      // whose columns are the emptiest
#pragma unroll
      for (int w = W - 1; w >= 0; --w) {
        u64 v = __shfl_sync(kFullWarp, x[w], j);
        const u32* const last = s_dom + (u32)(64 * w + 63) * kStride + V * lane;  // column of bit 0
        while (v && alive) {  // two states a turn
          and_column<V>(acc, last - (u32)(__ffsll((long long)v) - 1) * kStride);
          v &= v - 1;
          if (v) {
            and_column<V>(acc, last - (u32)(__ffsll((long long)v) - 1) * kStride);
            v &= v - 1;
          }
          u32 any = 0;
#pragma unroll
          for (int i = 0; i < V; ++i) any |= acc[i];
          alive = __any_sync(kFullWarp, any != 0);
        }
      }
      if (!alive) continue;
      // rows still set hold x; a row of x's own size is x itself
      const u32 sx = __shfl_sync(kFullWarp, size, j);
      bool hit = false;
#pragma unroll
      for (int i = 0; i < V; ++i)
        for (u32 left = acc[i]; left; left &= left - 1) {
          const u32 r = 32 * (V * lane + i) + __ffs(left) - 1;
          if (proper && s_size[r] == sx) continue;
          if (kHitT) {
            flags[r0 + r] = 1u;
            open[i] &= ~(left & -left);
          } else {
            hit = true;
            break;
          }
        }
      if (!kHitT && __any_sync(kFullWarp, hit) && lane == 0) flags[x0 + j] = 1u;
    }
  }
}

namespace {
template <int W, int V>
void launch_dom(bool comp, bool hit_t, const u64* T, u32 tm, const u64* X, u32 xm, int n, bool proper,
                const u32* decided, u32* flags, cudaStream_t s) {
  const u32 chunks = (tm + 1024 * V - 1) / (1024 * V);
  constexpr u32 kThreads = dom_threads<V>();
  // about two blocks an SM and chunk set, at least one pass of a block's warps
  // (one round of 32 sets each; 8 at V = 1 would only add staging) per slice
  u32 slices = std::max<u32>(1, (u32)device_sm_count() * (V == 1 ? 8 : 2) / chunks);
  slices = std::min<u32>({slices, (xm + kThreads - 1) / kThreads, 65535u});
  u32 per = (xm + slices - 1) / slices;
  per = (per + 31) / 32 * 32;
  slices = (xm + per - 1) / per;
  const dim3 grid(chunks, slices);
  constexpr size_t smem = dom_smem<W, V>();
#define SW_DOM(C, H)                                                                                      \
  {                                                                                                       \
    ensure_smem_limit((const void*)k_dominance<W, V, C, H>, (int)smem);                                   \
    k_dominance<W, V, C, H><<<grid, kThreads, smem, s>>>(T, tm, X, xm, n, proper ? 1 : 0, per, decided, flags); \
  }
  if (comp) {
    if (hit_t) SW_DOM(true, true) else SW_DOM(true, false)
  } else {
    if (hit_t) SW_DOM(false, true) else SW_DOM(false, false)
  }
#undef SW_DOM
  SW_LAUNCH_CHECK();
}
template <int W>
void launch_dom_w(bool comp, bool hit_t, const u64* T, u32 tm, const u64* X, u32 xm, int n, bool proper,
                  const u32* decided, u32* flags, cudaStream_t s) {
  // small lists: 1024-row chunks, so that they spread over more blocks
  if (tm <= kDomSmallRows)
    launch_dom<W, 1>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
  else
    launch_dom<W, (W < 7 ? 4 : 2)>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
}
}  // namespace

void launch_dominance(int W, bool comp, bool hit_t, const u64* T, u32 tm, const u64* X, u32 xm, int n, bool proper,
                      const u32* decided, u32* flags, cudaStream_t s) {
  if (!tm || !xm) return;
  switch (W) {
    case 1: return launch_dom_w<1>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 2: return launch_dom_w<2>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 3: return launch_dom_w<3>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 4: return launch_dom_w<4>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 5: return launch_dom_w<5>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 6: return launch_dom_w<6>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 7: return launch_dom_w<7>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    case 8: return launch_dom_w<8>(comp, hit_t, T, tm, X, xm, n, proper, decided, flags, s);
    default: throw std::runtime_error("dominance: unsupported width");
  }
}

}  // namespace sw
