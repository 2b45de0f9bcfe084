// Tiled subset check: for every query row c, does some row s of S satisfy
// s ⊆ c (proper: s ⊊ c; disjoint: s ∩ c = ∅)?
//
// Replaces the reference's subset tests (SubsetsImplicitTrie::check_contains_subset,
// synchrolib/data_structures/subsets_implicit_trie.hpp:29-266, and its GPU leaf
// kernel cuda/subsets_implicit_trie_kernel.cu:13-92).  The trie's pruning is
// re-expressed as a prefix-partitioned candidate filter:
//   * S comes ordered by its leading word (most frequent states first) and is
//     cut into tiles of 64 consecutive rows, grouped 16 to a super-tile (the
//     default ScanShape; tile rows, tiles per super-tile, warps per block and
//     the grid's S chunking are runtime parameters that the kernel autotuner
//     picks per row width and list size);
//   * every tile and super-tile keeps the AND of its rows — the states all of
//     its sets contain: the range's common prefix (the trie node's path) plus
//     incidental shared states — and the size of its smallest row; every group
//     of four rows the AND of its first words;
//   * a query that lacks one of those states, or has fewer states than the
//     range's smallest row, cannot contain any set of the range.
// One warp owns 32 consecutive (hence similar) queries, one per lane, and
// descends: its lanes test 32 super-tiles at a time, then a super-tile's
// tiles, against the union of the warp's open queries; a tile that passes is
// tested by every lane against its own query; then the lanes test the tile's
// groups against the union, and a group that passes is tested, and at last its
// rows read, by every lane for its own query.  Ranges are rejected 32 at a
// time from coalesced loads, and rows are read from global memory (L2) only
// where a query passed every mask above them, so nothing is staged and no
// barrier is taken.  In meet mode the first hit stops the grid.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.cuh"

namespace sw {

namespace {
constexpr int kMaxScanWarps = 16;
constexpr int kMaxTilesPerSuper = 32;
// Units up to which a check takes every (32 queries, super-tile) pair as a unit;
// above, the pairs are tested first (one more launch, about 4 us) and listed.
constexpr u64 kDirectUnits = 1u << 14;
// Checks of fewer units than this split them below super-tiles: the heaviest units
// end such a check.  Milliseconds by 2^12 / 2^14 / 2^16 / 2^18: four solves at n = 200
// 11.9 / 11.5 / 11.9 / 13.7 (12.5 unsplit), eight in a batch 14.2 / 15.2 / 18.6 / 25.7,
// 65 536 x 32 768 sets 0.91 / 0.91 / 0.83 / 0.85, n = 100 reduced 18.1 / 17.0 / 16.7 /
// 16.8.
constexpr u32 kSplitUnits = 1u << 14;
// Queries needing a tile up to which they are taken one at a time.
constexpr int kFewTakers = 6;
constexpr u32 kFullMask = 0xffffffffu;

int sm_count_sc() { return device_sm_count(); }

u32 n_tiles(u32 m, const ScanShape& sh) { return (m + sh.tile_rows - 1) / (u32)sh.tile_rows; }
u32 n_supers(u32 m, const ScanShape& sh) {
  const u32 rows = (u32)sh.tile_rows * (u32)sh.tiles_per_super;
  return (m + rows - 1) / rows;
}
}  // namespace

bool scan_shape_valid(int W, const ScanShape& sh) {
  const bool pow2_tr = sh.tile_rows == 32 || sh.tile_rows == 64 || sh.tile_rows == 128;
  const bool warps = sh.warps == 4 || sh.warps == 8 || sh.warps == 16;
  const bool tps = sh.tiles_per_super == 4 || sh.tiles_per_super == 8 || sh.tiles_per_super == 16 ||
                   sh.tiles_per_super == 32;
  const bool grid = sh.grid_factor >= 1 && sh.grid_factor <= 64;
  return W >= 1 && W <= 8 && pow2_tr && warps && tps && grid && scan_smem_bytes(W, sh) <= kMaxScanSmem;
}

// The rule's bound on a shape: two tiles per warp in kMaxScanSmem bytes (the
// scan stages no tiles, but what the rule refuses stays refused).
size_t scan_smem_bytes(int W, const ScanShape& sh) {
  return sizeof(u64) * (size_t)W * (size_t)sh.tile_rows * 2 * (size_t)sh.warps;
}

// ---- masks ----
// One buffer: tile ANDs (W words each), super-tile ANDs (W words each), one word
// per group of kGroupRows rows (the AND of their first words), then the smallest
// row size of every tile and of every super-tile (u32).
namespace {
constexpr u32 kGroupRows = 4;

struct MaskLayout {
  size_t super_and, group_and, tile_min, super_min, words;  // offsets and total in u64 words
};
__host__ __device__ inline MaskLayout mask_layout(int W, u32 m, u32 tiles, u32 supers) {
  MaskLayout L;
  L.super_and = (size_t)tiles * W;
  L.group_and = L.super_and + (size_t)supers * W;
  L.tile_min = L.group_and + (m + kGroupRows - 1) / kGroupRows;
  L.super_min = L.tile_min + (tiles + 1) / 2;
  L.words = L.super_min + (supers + 1) / 2;
  return L;
}
}  // namespace

// One block per super-tile, one warp per tile: each lane takes the tile's rows
// lane, lane + 32, ..., a butterfly combines the lanes (four adjacent lanes
// hold a group), and warp 0 folds the block's tile masks into the super-tile's.
// *size_floor becomes at least ~(size of the smallest row) (it starts at 0).
// Bound by the one read of S.
template <int W>
__global__ void __launch_bounds__(kMaxTilesPerSuper * 32) k_range_and(const u64* __restrict__ S, u32 m,
                                                                      u64* __restrict__ masks, u32 tile_rows,
                                                                      u32* size_floor, const u32* m_live) {
  __shared__ u64 s_and[kMaxTilesPerSuper][W];
  __shared__ u32 s_min[kMaxTilesPerSuper];
  const u32 tiles = (m + tile_rows - 1) / tile_rows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tps = blockDim.x >> 5;
  const u32 t = blockIdx.x * tps + warp;
  const MaskLayout L = mask_layout(W, m, tiles, gridDim.x);
  m = live_count(m, m_live);
  if (blockIdx.x * tps * tile_rows >= m) return;
  u64 a[W];
#pragma unroll
  for (int w = 0; w < W; ++w) a[w] = ~0ULL;
  u32 mn = 0xffffffffu;
  for (u32 i = lane; i < tile_rows; i += 32) {
    const u64 r = (u64)t * tile_rows + i;
    u64 x[W];
    u32 c = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      x[w] = r < m ? S[(size_t)r * W + w] : ~0ULL;
      a[w] &= x[w];
      c += __popcll(x[w]);
    }
    if (r < m) mn = min(mn, c);
    u64 g = x[0];
    g &= __shfl_xor_sync(kFullMask, g, 1);
    g &= __shfl_xor_sync(kFullMask, g, 2);
    if (r < m && (lane & 3) == 0) masks[L.group_and + r / kGroupRows] = g;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) {
#pragma unroll
    for (int o = 16; o; o >>= 1) a[w] &= __shfl_xor_sync(kFullMask, a[w], o);
    if (lane == 0) {
      if (t < tiles) masks[(size_t)t * W + w] = a[w];
      s_and[warp][w] = a[w];  // ~0 for tiles past the end
    }
  }
  mn = __reduce_min_sync(kFullMask, mn);
  if (lane == 0) {
    if (t < tiles) reinterpret_cast<u32*>(masks + L.tile_min)[t] = mn;
    s_min[warp] = mn;
  }
  __syncthreads();
  if (warp == 0) {
    if (lane < W) {
      u64 v = ~0ULL;
      for (int x = 0; x < tps; ++x) v &= s_and[x][lane];
      masks[L.super_and + (size_t)blockIdx.x * W + lane] = v;
    }
    const u32 v = __reduce_min_sync(kFullMask, lane < tps ? s_min[lane] : 0xffffffffu);
    if (lane == 0) {
      reinterpret_cast<u32*>(masks + L.super_min)[blockIdx.x] = v;
      atomicMax(size_floor, ~v);
    }
  }
}

// ---- scan ----
// A unit of work is one warp's 32 queries against a few super-tiles.  Queries
// differ by orders of magnitude in the tiles they need (a large set needs most
// of S), so a warp that kept its queries for all of S left the SMs waiting for
// the heaviest warps (achieved occupancy 15%, 1.1 ms where the work of an even
// spread is 0.2 ms: 155 000 x 159 000 sets, n = 200).  Units are therefore spread over
// the grid's warps: all (queries, super-tiles) units of a small check directly, and
// for larger ones the (queries, super-tile) pairs that the union test of
// k_scan_candidates leaves.
namespace {
// The lane's query: complement nc (a row or mask is inside the query when it
// shares no state with nc) and the size of the largest row it can hold.
template <int W, int MODE>
__device__ __forceinline__ int load_query(const u64* __restrict__ Q, u32 qi, bool valid, int n, u64* nc) {
  int size = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    u64 c = valid ? Q[(size_t)qi * W + w] : 0ULL;
    if (MODE == kQueryDisjoint) c = ~c & valid_mask(n, w);
    size += __popcll(c);
    nc[w] = ~c;
  }
  return MODE == kQueryProperSubset ? size - 1 : size;
}

// Complement of the union of the warp's open queries, and the largest row any
// of them can hold (-1: none).  Every lane takes part.
template <int W>
__device__ __forceinline__ int query_union(const u64* nc, int room, bool done, u64* nu) {
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const u64 c = done ? 0ULL : ~nc[w];
    nu[w] = ~(((u64)__reduce_or_sync(kFullMask, (u32)(c >> 32)) << 32) | __reduce_or_sync(kFullMask, (u32)c));
  }
  return __reduce_max_sync(kFullMask, done ? -1 : room);
}
}  // namespace

// items[0 .. *count) = (query group, super-tile) pairs whose super-tile's mask and
// smallest row fit the union of the group's queries; warp per group of 32
// queries, 32 super-tiles tested at a time.
template <int W, int MODE>
__global__ void __launch_bounds__(256) k_scan_candidates(const u64* __restrict__ super_and,
                                                         const u32* __restrict__ super_min, u32 m, u32 super_rows,
                                                         const u64* __restrict__ Q, u32 q, u32 group0, u32 groups, int n,
                                                         const u32* __restrict__ flags, const u32* witness,
                                                         const u32* __restrict__ size_floor, int stop,
                                                         uint2* __restrict__ items, u32* count, const u32* m_live,
                                                         const u32* q_live) {
  const u32 supers = (live_count(m, m_live) + super_rows - 1) / super_rows;
  q = live_count(q, q_live);
  const u32 lane = threadIdx.x & 31, g = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (g >= groups) return;
  if (stop) {  // met in an earlier slice of the queries
    const u32 f = lane == 0 ? *(const volatile u32*)witness : 0u;
    if (__shfl_sync(kFullMask, f, 0) != 0) return;
  }
  const u32 qi = (group0 + g) * 32 + lane;
  const bool valid = qi < q;
  u64 nc[W], nu[W];
  const int room = load_query<W, MODE>(Q, qi, valid, n, nc);
  const bool done = !valid || room < (int)~*size_floor || (!stop && flags[qi]);
  const int most = query_union<W>(nc, room, done, nu);
  if (most < 0) return;
  for (u32 b0 = 0; b0 < supers; b0 += 1024) {  // one reservation per 1024 super-tiles
    u32 mine = 0;  // lane i: which of super-tiles b0 + 32 i .. + 31 are candidates
    for (u32 i = 0; i < 32 && b0 + 32 * i < supers; ++i) {
      const u32 s = b0 + 32 * i + lane;
      bool cand = s < supers;
      if (cand) {
        cand = (int)super_min[s] <= most;
#pragma unroll
        for (int w = 0; w < W; ++w)
          if (super_and[(size_t)s * W + w] & nu[w]) cand = false;
      }
      const u32 mask = __ballot_sync(kFullMask, cand);
      if (lane == i) mine = mask;
    }
    u32 incl = __popc(mine);
#pragma unroll
    for (u32 d = 1; d < 32; d *= 2) {
      const u32 o = __shfl_up_sync(kFullMask, incl, d);
      if (lane >= d) incl += o;
    }
    u32 at = 0;
    if (lane == 31 && incl) at = atomicAdd(count, incl);
    at = __shfl_sync(kFullMask, at, 31);
    u32 left = __ballot_sync(kFullMask, mine != 0);
    while (left) {
      const int i = __ffs(left) - 1;
      left &= left - 1;
      const u32 mask = __shfl_sync(kFullMask, mine, i), before = __shfl_sync(kFullMask, incl, i) - __popc(mask);
      if ((mask >> lane) & 1u)
        items[at + before + __popc(mask & ((1u << lane) - 1u))] = make_uint2(group0 + g, b0 + 32 * i + lane);
    }
  }
}

// Units: items[0 .. counts[0]), or without items every (query group, `chunk`
// super-tiles) pair; where these are fewer than `split_units`, parts of them.
// Warps fetch items one by one, the next while they work on one, from
// kSubsetQueues counters: class c of the warps takes the items c, c + 64, ... (one
// counter served ~0.6 fetches a ns, and 19 456 warps starting on it were 30 us of a
// 77 us launch).  Instructions per launch against rows of needed tiles tested by the
// whole warp one query at a time: 237 -> 88 M and 309 -> 155 M at two levels
// of an n = 200 search.
// Registers are held to 40 up to four words a row (48 warps an SM): the loads a
// unit waits for are what the other warps hide.
template <int W, int MODE>
__global__ void __launch_bounds__(kMaxScanWarps * 32, W <= 4 ? 3 : 2) k_subset_scan(const u64* __restrict__ S, u32 m,
                                                                    const u64* __restrict__ masks, u32 tile_rows,
                                                                    u32 tps, const u64* __restrict__ Q, u32 q, int n,
                                                                    u32* flags, u32* witness,
                                                                    const u32* __restrict__ size_floor, int stop,
                                                                    const uint2* __restrict__ items,
                                                                    u32* counts, u32 chunk, u32 split_units,
                                                                    u64* __restrict__ bytes_ctr, const u32* m_live,
                                                                    const u32* q_live) {
  const u32 lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  u32 tiles = (m + tile_rows - 1) / tile_rows, supers = (tiles + tps - 1) / tps;
  const MaskLayout L = mask_layout(W, m, tiles, supers);
  m = live_count(m, m_live);
  q = live_count(q, q_live);
  tiles = (m + tile_rows - 1) / tile_rows;
  supers = (tiles + tps - 1) / tps;
  const u64* const super_and = masks + L.super_and;
  const u64* const group_and = masks + L.group_and;
  const u32* const tile_min = reinterpret_cast<const u32*>(masks + L.tile_min);
  const u32* const super_min = reinterpret_cast<const u32*>(masks + L.super_min);
  const u32 gpt = tile_rows / kGroupRows;  // groups per tile: 8, 16 or 32
  const u32 chunks = (supers + chunk - 1) / chunk;
  const u64 whole = items ? *(volatile u32*)counts : (u64)((q + 31) / 32) * chunks;
  u32 split = 1;
  if (items || chunk == 1)
    while (split < tps && whole * split < split_units) split *= 2;
  const u64 units = whole * split;
  const u32 me = blockIdx.x * warps + (threadIdx.x >> 5), queue = me % kSubsetQueues;
  // the class's warps start on its first items, one each
  const u32 started = (gridDim.x * warps - queue + kSubsetQueues - 1) / kSubsetQueues;
  auto fetch = [&]() -> u32 { return lane == 0 ? atomicAdd(counts + 32 * (queue + 1), 1u) : 0u; };
  const int floor_size = (int)~*size_floor;
  u32 rows_read = 0, ahead = 0;
  bool first = true;
  for (u64 u = me;; u += gridDim.x * warps) {
    if (items && !first) u = (u64)(__shfl_sync(kFullMask, ahead, 0) + started) * kSubsetQueues + queue;
    first = false;
    if (u >= units) break;
    if (items) ahead = fetch();
    if (stop) {  // leave once any warp met
      const u32 f = lane == 0 ? *(volatile u32*)witness : 0u;
      if (__shfl_sync(kFullMask, f, 0) != 0) break;
    }
    u32 g, s0, s1, lo = 0, hi = tps;  // tiles lo .. hi - 1 of the super-tiles s0 .. s1 - 1
    if (split > 1) {
      lo = (u32)(u % split) * (tps / split);
      hi = lo + tps / split;
    }
    const u64 v = u / split;
    if (items) {
      const uint2 it = items[v];
      g = it.x;
      s0 = it.y;
      s1 = s0 + 1;
    } else {
      g = (u32)(v / chunks);
      s0 = (u32)(v - (u64)g * chunks) * chunk;
      s1 = min(supers, s0 + chunk);
    }
    const u32 qi = g * 32 + lane;
    const bool valid = qi < q;
    u64 nc[W], nu[W];
    const int room = load_query<W, MODE>(Q, qi, valid, n, nc);
    bool done = !valid || room < floor_size || (!stop && *(volatile u32*)(flags + qi));
    bool hit = false;
    u32 hit_idx = 0;
    const int most = query_union<W>(nc, room, done, nu);
    if (most < 0) continue;
    bool cand = s0 + lane < s1;
    if (cand) {
      cand = (int)super_min[s0 + lane] <= most;
#pragma unroll
      for (int w = 0; w < W; ++w)
        if (super_and[(size_t)(s0 + lane) * W + w] & nu[w]) cand = false;
    }
    u32 s_todo = __ballot_sync(kFullMask, cand);
    while (s_todo) {
      const u32 t0 = (s0 + __ffs(s_todo) - 1) * tps;
      s_todo &= s_todo - 1;
      bool tc = lane >= lo && lane < hi && t0 + lane < tiles;
      if (tc) {
        tc = (int)tile_min[t0 + lane] <= most;
#pragma unroll
        for (int w = 0; w < W; ++w)
          if (masks[(size_t)(t0 + lane) * W + w] & nu[w]) tc = false;
      }
      u32 t_todo = __ballot_sync(kFullMask, tc);
      while (t_todo) {
        const u32 t = t0 + __ffs(t_todo) - 1;
        t_todo &= t_todo - 1;
        bool need = !done && (int)tile_min[t] <= room && !(masks[(size_t)t * W] & nc[0]);
        if (!__any_sync(kFullMask, need)) continue;
#pragma unroll
        for (int w = 1; w < W; ++w)
          if (masks[(size_t)t * W + w] & nc[w]) need = false;
        if (!__any_sync(kFullMask, need)) continue;
        const u32 g0 = t * gpt;
        const bool gin = lane < gpt && (g0 + lane) * kGroupRows < m;
        const u64 gm = gin ? group_and[g0 + lane] : ~0ULL;
        u32 takers = __ballot_sync(kFullMask, need);
        if (__popc(takers) <= kFewTakers) {
          // few queries need the tile: one at a time, the lanes testing its
          // groups' masks at once, then the words of a passing group's rows
          while (takers) {
            const int j = __ffs(takers) - 1;
            takers &= takers - 1;
            const u64 first = __shfl_sync(kFullMask, nc[0], j);  // every lane takes part
            u32 g_todo = __ballot_sync(kFullMask, gin && !(gm & first));
            if (!g_todo) continue;
            u64 mine = 0;  // word lane % W of query j's complement
#pragma unroll
            for (int w = 0; w < W; ++w) {
              const u64 v = __shfl_sync(kFullMask, nc[w], j);
              if (lane % W == (u32)w) mine = v;
            }
            while (g_todo) {
              const u32 r0 = (g0 + __ffs(g_todo) - 1) * kGroupRows;
              g_todo &= g_todo - 1;
              const bool in = lane < kGroupRows * W && r0 + lane / W < m;
              const u64 x = in ? S[(size_t)r0 * W + lane] : 0ULL;
              rows_read += kGroupRows;
              const u32 bad = __ballot_sync(kFullMask, !in || (x & mine));
              const u32 same = MODE == kQueryProperSubset ? __ballot_sync(kFullMask, in && x == ~mine) : 0u;
              int row = -1;
#pragma unroll
              for (int r = (int)kGroupRows - 1; r >= 0; --r) {
                constexpr u32 kRow = (1u << W) - 1u;
                if (((bad >> (r * W)) & kRow) == 0 && (MODE != kQueryProperSubset || ((same >> (r * W)) & kRow) != kRow))
                  row = r;
              }
              if (row >= 0) {
                if (lane == (u32)j) {
                  hit = done = true;
                  hit_idx = r0 + (u32)row;
                }
                break;
              }
            }
          }
          continue;
        }
        u32 g_todo = __ballot_sync(kFullMask, gin && !(gm & nu[0]));
        while (g_todo) {
          const int i = __ffs(g_todo) - 1;
          g_todo &= g_todo - 1;
          const u64 gmask = __shfl_sync(kFullMask, gm, i);  // every lane takes part
          const bool p = need && !(gmask & nc[0]);
          if (!__any_sync(kFullMask, p)) continue;
          const u32 r0 = (g0 + i) * kGroupRows, rn = min(kGroupRows, m - r0);
          rows_read += rn;
          for (u32 r = 0; r < rn; ++r) {
            const u64* const row = S + (size_t)(r0 + r) * W;
            const u64 x0 = row[0];
            bool sub = p && need && !(x0 & nc[0]);
            if (!__any_sync(kFullMask, sub)) continue;
            bool eq = x0 == ~nc[0];
#pragma unroll
            for (int w = 1; w < W; ++w) {
              const u64 x = row[w];
              if (x & nc[w]) sub = false;
              eq = eq && x == ~nc[w];
            }
            if (MODE == kQueryProperSubset && eq) sub = false;
            if (sub) {
              hit = done = true;
              need = false;
              hit_idx = r0 + r;
            }
          }
        }
      }
      if (__all_sync(kFullMask, done)) break;
    }
    if (hit) {
      if (!stop) {
        flags[qi] = 1u;
      } else if (atomicCAS(witness, 0u, 1u) == 0u) {
        witness[1] = qi;
        witness[2] = hit_idx;
      }
    }
  }
  if (bytes_ctr && lane == 0 && rows_read) atomicAdd(bytes_ctr, rows_read * 8ULL * W);
}

size_t subset_check_temp_bytes(int W, u32 m, const ScanShape& sh) {
  const u32 mm = std::max<u32>(m, 1);
  return sizeof(u64) * mask_layout(W, mm, n_tiles(mm, sh), n_supers(mm, sh)).words;
}

u64 subset_check_items(u32 m, u32 q, const ScanShape& sh) {
  const u64 pairs = (u64)((q + 31) / 32) * n_supers(m, sh);
  return pairs > kDirectUnits ? std::min(pairs, kSubsetItems) : 0;
}

void launch_tile_and(int W, const u64* S, u32 m, u64* masks, u32* size_floor, const ScanShape& sh, cudaStream_t s,
                     const u32* m_live) {
  if (!m) return;
  if (!scan_shape_valid(W, sh)) throw std::invalid_argument("range_and: invalid scan shape");
  const u32 blocks = n_supers(m, sh);
  const int threads = sh.tiles_per_super * 32;
#define SW_RA(WW) \
  case WW: k_range_and<WW><<<blocks, threads, 0, s>>>(S, m, masks, (u32)sh.tile_rows, size_floor, m_live); break;
  switch (W) {
    SW_RA(1)
    SW_RA(2)
    SW_RA(3)
    SW_RA(4)
    SW_RA(5)
    SW_RA(6)
    SW_RA(7)
    SW_RA(8)
    default: throw std::runtime_error("range_and: unsupported width");
  }
#undef SW_RA
  SW_LAUNCH_CHECK();
}

void launch_subset_check(int W, int mode, const u64* S, u32 m, const u64* masks, const u32* size_floor, const u64* Q,
                         u32 q, int n, u32* flags, u32* witness, bool stop, const ScanShape& sh, cudaStream_t s,
                         u64* bytes_ctr, uint2* items, u32* item_counts, const u32* m_live, const u32* q_live) {
  if (!m || !q) return;
  if (!scan_shape_valid(W, sh)) throw std::invalid_argument("subset check: invalid scan shape");
  const u32 tiles = n_tiles(m, sh), supers = n_supers(m, sh);
  const MaskLayout L = mask_layout(W, m, tiles, supers);
  const u32 super_rows = (u32)(sh.tile_rows * sh.tiles_per_super);
  const u32 groups = (q + 31) / 32, warps = (u32)sh.warps;
  const u64 pairs = (u64)groups * supers;
  // no more blocks than are resident (the launch bounds): the others only find the
  // units gone (eight n = 200 solves in a batch 15.2 -> 14.5 ms)
  const u32 most_blocks = (u32)sm_count_sc() * std::min<u32>((u32)sh.grid_factor, (W <= 4 ? 48u : 32u) / warps);
  // without a list: few enough units for one each, else up to 32 super-tiles a unit
  const bool listed = items && pairs > kDirectUnits && supers <= kSubsetItems;
  u32 chunk = 1;
  if (!listed)
    while (chunk < 32 && (u64)groups * ((supers + chunk - 1) / chunk) > kDirectUnits) chunk *= 2;
  const u32 slice = listed ? std::max<u32>(1, std::min<u32>(groups, (u32)(kSubsetItems / supers))) : groups;
  for (u32 g0 = 0; g0 < groups; g0 += slice) {
    const u32 gs = std::min(slice, groups - g0);
    u64 units = listed ? (u64)gs * supers : (u64)groups * ((supers + chunk - 1) / chunk);
    if (listed || chunk == 1) units = std::max(units, std::min<u64>(units * sh.tiles_per_super, kSplitUnits));
    const u32 blocks = (u32)std::min<u64>((units + warps - 1) / warps, most_blocks);
    if (listed) SW_CUDA(cudaMemsetAsync(item_counts, 0, sizeof(u32) * kSubsetCounterWords, s));
#define SW_SC_ONE(WW, MM)                                                                                             \
  {                                                                                                                   \
    if (listed)                                                                                                       \
      k_scan_candidates<WW, MM><<<(gs + 7) / 8, 256, 0, s>>>(                                                         \
          masks + L.super_and, reinterpret_cast<const u32*>(masks + L.super_min), m, super_rows, Q, q, g0, gs, n,     \
          flags, witness, size_floor, stop, items, item_counts, m_live, q_live);                                       \
    k_subset_scan<WW, MM><<<blocks, warps * 32, 0, s>>>(S, m, masks, (u32)sh.tile_rows, (u32)sh.tiles_per_super, Q,   \
                                                        q, n, flags, witness, size_floor, stop,                       \
                                                        listed ? items : nullptr, item_counts, chunk, kSplitUnits, bytes_ctr,       \
                                                        m_live, q_live);                                              \
  }
#define SW_SC(WW)                                                           \
  case WW:                                                                  \
    if (mode == kQuerySubset) SW_SC_ONE(WW, kQuerySubset)                   \
    else if (mode == kQueryProperSubset) SW_SC_ONE(WW, kQueryProperSubset)  \
    else SW_SC_ONE(WW, kQueryDisjoint)                                      \
    break;
    switch (W) {
      SW_SC(1)
      SW_SC(2)
      SW_SC(3)
      SW_SC(4)
      SW_SC(5)
      SW_SC(6)
      SW_SC(7)
      SW_SC(8)
      default:
        throw std::runtime_error("subset check: unsupported width");
    }
#undef SW_SC
#undef SW_SC_ONE
    SW_LAUNCH_CHECK();
  }
}

}  // namespace sw
