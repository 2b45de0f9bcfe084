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
constexpr size_t dom_smem() {  // columns, open rows, row sizes
  return sizeof(u32) * (64 * W * col_stride<V>() + 32 * V) + sizeof(uint16_t) * 1024 * V;
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
// kComp: rows are complements of the sets.  Rows flagged before are left out.
// index (may be null): what row t of T is called in flags.
template <int W, int V, bool kComp, bool kHitT>
__global__ void __launch_bounds__(dom_threads<V>()) k_dominance(const u64* __restrict__ T, u32 tm,
                                                               const u32* __restrict__ index,
                                                               const u64* __restrict__ X, u32 xm, int n, int proper,
                                                               u32 per_slice, u32 per_warp, u32* flags,
                                                               const u32* t_live, const u32* x_live) {
  extern __shared__ __align__(16) u32 s_dom[];
  __shared__ u32 s_max;
  constexpr u32 kStride = col_stride<V>();
  constexpr u32 kWarps = dom_threads<V>() / 32;
  u32* const s_open = s_dom + 64 * W * kStride;
  uint16_t* const s_size = reinterpret_cast<uint16_t*>(s_open + 32 * V);
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  tm = live_count(tm, t_live);
  xm = live_count(xm, x_live);
  const u32 r0 = blockIdx.x * 1024u * V;
  if (r0 >= tm || blockIdx.y * per_slice >= xm) return;
  const u32 rows = min(1024u * V, tm - r0);
  if (threadIdx.x == 0) s_max = 0;
  __syncthreads();
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
      // column c of a word holds bit c: its states from the last to the first
      s_dom[(64 * w + 32 + lane) * kStride + g] = transpose32((u32)(b >> 32));
      s_dom[(64 * w + lane) * kStride + g] = transpose32((u32)b);
    }
    s_size[r] = (uint16_t)size;
    bool in = r < rows;
    if (kHitT && in) in = !*(volatile u32*)(flags + (index ? index[r0 + r] : r0 + r));
    const u32 open = __ballot_sync(kFullWarp, in);
    const u32 most = __reduce_max_sync(kFullWarp, size);
    if (lane == 0) {
      s_open[g] = open;
      atomicMax(&s_max, most);
    }
  }
  __syncthreads();
  u32 open[V];  // the lane's rows that take part: 32 (V lane + i) + bit
#pragma unroll
  for (int i = 0; i < V; ++i) open[i] = s_open[V * lane + i];
  const u32 most = s_max;
  const u32 x_end = min(xm, (blockIdx.y + 1) * per_slice);
  for (u32 x0 = blockIdx.y * per_slice + warp * per_warp; x0 < x_end; x0 += kWarps * per_warp) {
    const u32 xi = x0 + lane;
    const bool valid = lane < per_warp && xi < x_end;
    u32 x[2 * W];  // the set in 32-bit halves
    u32 size = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      u64 b = valid ? X[(size_t)xi * W + w] : 0ULL;
      if (kComp && valid) b = ~b & valid_mask(n, w);
      x[2 * w] = (u32)(b >> 32);
      x[2 * w + 1] = (u32)b;
      size += __popcll(b);
    }
    // no row of the chunk is as large as a larger set (nor, for a proper subset, larger than one as large)
    bool want = valid && (proper ? size < most : size <= most);
    if (!kHitT && want) want = !*(volatile u32*)(flags + xi);
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
      for (int h = 2 * W - 1; h >= 0; --h) {
        u32 v = __shfl_sync(kFullWarp, x[h], j);
        const u32* const base = s_dom + (u32)(64 * (h >> 1) + ((h & 1) ? 0 : 32)) * kStride + V * lane;
        while (v && alive) {  // two states a turn
          const u32 b0 = __ffs(v) - 1;
          v &= v - 1;
          and_column<V>(acc, base + b0 * kStride);
          if (v) {
            const u32 b1 = __ffs(v) - 1;
            v &= v - 1;
            and_column<V>(acc, base + b1 * kStride);
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
            flags[index ? index[r0 + r] : r0 + r] = 1u;
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

// ---- rows by falling size, so that a chunk's sizes are alike ----
template <int W, bool kComp>
__global__ void __launch_bounds__(256) k_size_rank(const u64* __restrict__ T, u32 m, int n, u32* __restrict__ counts,
                                                   uint2* __restrict__ place, const u32* live) {
  m = live_count(m, live);
  const u32 e = blockIdx.x * blockDim.x + threadIdx.x;
  u32 size = 0;
  if (e < m)
#pragma unroll
    for (int w = 0; w < W; ++w) size += __popcll(T[(size_t)e * W + w]);
  const u32 bucket = kComp ? size : (u32)n - size;  // largest sets first
  const u32 in = __ballot_sync(kFullWarp, e < m);
  if (e >= m) return;
  const u32 lane = threadIdx.x & 31;
  const u32 peers = __match_any_sync(in, bucket);
  const int leader = __ffs(peers) - 1;
  u32 first = 0;
  if (lane == (u32)leader) first = atomicAdd(&counts[bucket], (u32)__popc(peers));
  place[e] = make_uint2(__shfl_sync(peers, first, leader) + __popc(peers & ((1u << lane) - 1u)), bucket);
}

template <int W>
__global__ void __launch_bounds__(256) k_size_scatter(const u64* __restrict__ T, u32 m, const uint2* __restrict__ place,
                                                      const u32* __restrict__ first, u64* __restrict__ out,
                                                      u32* __restrict__ index, const u32* live) {
  const u32 e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= live_count(m, live)) return;
  const uint2 pl = place[e];
  const u32 d = first[pl.y] + pl.x;
#pragma unroll
  for (int w = 0; w < W; ++w) out[(size_t)d * W + w] = T[(size_t)e * W + w];
  index[d] = e;
}

namespace {
template <int W, int V>
void launch_dom(bool comp, bool hit_t, const u64* T, u32 tm, const u32* index, const u64* X, u32 xm, int n, bool proper,
                u32* flags, cudaStream_t s, const u32* t_live, const u32* x_live) {
  const u32 chunks = (tm + 1024 * V - 1) / (1024 * V);
  constexpr u32 kThreads = dom_threads<V>(), kWarps = kThreads / 32;
  // slices of X: as many blocks as fit the GPU a few times over, while a warp keeps eight sets or more
  u32 slices = std::max<u32>(1, (u32)device_sm_count() * (V == 1 ? 8 : 2) / chunks);
  slices = std::min<u32>({slices, (xm + 8 * kWarps - 1) / (8 * kWarps), 65535u});
  u32 per = (xm + slices - 1) / slices;
  const u32 per_warp = std::min<u32>(32, (per + kWarps - 1) / kWarps);
  slices = (xm + per - 1) / per;
  const dim3 grid(chunks, slices);
  constexpr size_t smem = dom_smem<W, V>();
#define SW_DOM(C, H)                                                                                          \
  {                                                                                                           \
    ensure_smem_limit((const void*)k_dominance<W, V, C, H>, (int)smem);                                       \
    k_dominance<W, V, C, H><<<grid, kThreads, smem, s>>>(T, tm, index, X, xm, n, proper ? 1 : 0, per, per_warp, \
                                                         flags, t_live, x_live);                     \
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
                  u32* flags, const DominanceScratch& sc, cudaStream_t s, const u32* t_live, const u32* x_live) {
  constexpr int V = W < 7 ? 4 : 2;
  // small lists: 1024-row chunks, so that they spread over more blocks
  if (tm <= kDomSmallRows) return launch_dom<W, 1>(comp, hit_t, T, tm, nullptr, X, xm, n, proper, flags, s, t_live, x_live);
  if (tm <= kDomOrderRows) return launch_dom<W, V>(comp, hit_t, T, tm, nullptr, X, xm, n, proper, flags, s, t_live, x_live);
  const u32 blocks = (tm + 255) / 256;
  if (comp)
    k_size_rank<W, true><<<blocks, 256, 0, s>>>(T, tm, n, sc.bucket.counts, sc.bucket.place, t_live);
  else
    k_size_rank<W, false><<<blocks, 256, 0, s>>>(T, tm, n, sc.bucket.counts, sc.bucket.place, t_live);
  launch_bucket_scan(BucketScratch{kBucketBitsSmall, sc.bucket.counts, sc.bucket.first, sc.bucket.place, nullptr,
                                   sc.bucket.met},
                     sc.total, s);
  k_size_scatter<W><<<blocks, 256, 0, s>>>(T, tm, sc.bucket.place, sc.bucket.first, sc.rows, sc.index, t_live);
  SW_LAUNCH_CHECK();
  launch_dom<W, V>(comp, hit_t, sc.rows, tm, sc.index, X, xm, n, proper, flags, s, t_live, x_live);
}
}  // namespace

void launch_dominance(int W, bool comp, bool hit_t, const u64* T, u32 tm, const u64* X, u32 xm, int n, bool proper,
                      u32* flags, const DominanceScratch& sc, cudaStream_t s, const u32* t_live, const u32* x_live) {
  if (!tm || !xm) return;
  switch (W) {
    case 1: return launch_dom_w<1>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 2: return launch_dom_w<2>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 3: return launch_dom_w<3>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 4: return launch_dom_w<4>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 5: return launch_dom_w<5>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 6: return launch_dom_w<6>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 7: return launch_dom_w<7>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    case 8: return launch_dom_w<8>(comp, hit_t, T, tm, X, xm, n, proper, flags, sc, s, t_live, x_live);
    default: throw std::runtime_error("dominance: unsupported width");
  }
}

}  // namespace sw
