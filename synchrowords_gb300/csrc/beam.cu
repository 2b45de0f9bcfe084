// The Beam algorithm's levels in one launch, for beams whose children fit in
// one CTA's shared memory.
//
// Reference: Beam::run (synchrolib/algorithm/beam/beam.hpp:88-188): each level
// expands the kept sets by every letter, orders the preimages by cardinality
// (ties by raw words), drops duplicates and keeps the `beam` largest.
#include <algorithm>

#include "algos.cuh"
#include "rowset.cuh"

namespace sw {

namespace {
constexpr u32 kBeamThreads = 1024;
constexpr u32 kBeamBins = 2 * kBeamThreads;
constexpr u32 kDuplicate = 0x8000u;  // in a child's key: an earlier child is the same set
// Pairs a child, within the bins, above which a level's children are sorted instead:
// us a level by 16 / 64 / 128 / 256 / never, random automata n=256 beam 2048 62 / 53 /
// 54 / 66 / 67, n=60 k=16 beam 500 107 / 69 / 64 / 64 / 82; letters that permute all
// states but one, whose sets differ in few states, n=128 beam 3000 101 / 100 / 100 /
// 101 / 1730, n=60 k=16 beam 500 118 / 101 / 97 / 101 / 520 (launches over the whole GPU
// 113 and 116).
constexpr u32 kBeamPairs = 128;

struct BeamLayout {
  size_t child, col, delta, bins, key, list, kept, bytes;
};
__host__ __device__ inline BeamLayout beam_layout(int W, u32 n, u32 k, u32 parents) {
  BeamLayout L;
  const size_t groups = (parents + 31) / 32, children = (size_t)parents * k;
  L.child = 0;                                     // u64[W][children]
  L.col = L.child + 8 * (size_t)W * children;      // u32[groups][64 W]
  L.list = L.col;                                  // u16[children], while no columns are held
  L.bins = L.col + std::max(256 * groups * (size_t)W, (2 * children + 3) / 4 * 4);  // u32[2][kBeamBins + 1]
  L.delta = L.bins + 8 * (size_t)(kBeamBins + 1);  // u16[k][n]
  L.key = L.delta + 2 * (size_t)n * k;             // u16[children]
  L.kept = L.key + 2 * children;                   // u16[parents]
  L.bytes = L.kept + 2 * (size_t)parents;
  return L;
}

// out[b] = count[b] = the sum of the first b counts, for b <= kBeamBins; the
// whole block, two bins per thread.  The caller synchronises before and after.
__device__ __forceinline__ void scan_bins(u32* count, u32* out, u32* s_sum) {
  const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const u32 c0 = count[2 * tid], c1 = count[2 * tid + 1];
  u32 incl = c0 + c1;
#pragma unroll
  for (u32 d = 1; d < 32; d *= 2) {
    const u32 o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  if (lane == 31) s_sum[warp] = incl;
  __syncthreads();
  const u32 other = s_sum[lane];
  const u32 before = __reduce_add_sync(0xffffffffu, lane < warp ? other : 0u);
  const u32 at = before + incl - c0 - c1;
  out[2 * tid] = count[2 * tid] = at;
  out[2 * tid + 1] = count[2 * tid + 1] = at + c0;
  if (tid == kBeamThreads - 1) out[kBeamBins] = count[kBeamBins] = at + c0 + c1;
}

template <int W>
__device__ __forceinline__ bool same_child(const u64* child, size_t cap, u32 i, u32 j) {
  if (child[i] != child[j]) return false;
  bool same = true;
#pragma unroll
  for (int w = 1; w < W; ++w) same = same && child[w * cap + i] == child[w * cap + j];
  return same;
}

// list[0 .. N) = the children by (key, set in the beam's order, number): a bitonic
// network whose exchanges all ascend, so that places past N (larger than any
// child) need no storage.  The whole block.
template <int W>
__device__ __forceinline__ void sort_children(uint16_t* list, const uint16_t* key, const u64* child, size_t cap,
                                              u32 N) {
  const auto less = [&](u32 i, u32 j) {
    if (key[i] != key[j]) return key[i] < key[j];
    u64 d = child[i] ^ child[j], y = child[j];
#pragma unroll
    for (int w = 1; w < W; ++w)
      if (!d) {
        y = child[w * cap + j];
        d = child[w * cap + i] ^ y;
      }
    return d ? (y & (d & (~d + 1))) != 0 : i < j;  // the lowest differing bit decides
  };
  const auto exchange = [&](u32 a, u32 b) {
    if (b >= N) return;
    const uint16_t i = list[a], j = list[b];
    if (less(j, i)) {
      list[a] = j;
      list[b] = i;
    }
  };
  u32 half = 1;  // exchanges of a stage
  while (2 * half < N) half *= 2;
  for (u32 p = threadIdx.x; p < N; p += kBeamThreads) list[p] = (uint16_t)p;
  for (u32 size = 1; size <= half; size *= 2) {  // merges runs of `size`
    __syncthreads();
    for (u32 t = threadIdx.x; t < half; t += kBeamThreads) {
      const u32 at = 2 * (t & ~(size - 1)), o = t & (size - 1);
      exchange(at + o, at + 2 * size - 1 - o);
    }
    for (u32 step = size / 2; step; step /= 2) {
      __syncthreads();
      for (u32 t = threadIdx.x; t < half; t += kBeamThreads) {
        const u32 a = 2 * (t & ~(step - 1)) + (t & (step - 1));
        exchange(a, a + step);
      }
    }
  }
  __syncthreads();
}
}  // namespace

// Every level of the beam in one CTA: over the whole GPU a level of a few
// thousand children costs its 14 launches and two synchronisations (73 us at 30
// children, 107-127 us at thousands), not its work.  Children stay in shared
// memory word by word (lane = child, no bank conflicts), the kept sets as
// columns of 32 (one letter's preimages of 32 sets are then 2 W table reads and
// transposes per lane).  Ordering: a counting sort by cardinality and the next
// bits of the order, then each child counts the smaller ones in its bin; bins by
// cardinality alone were 2-3x slower from 1500 children, and where bins hold too
// many (kBeamPairs) the level is sorted by a bitonic network.  What bounds a level
// is that count (shared memory) and ~14 barriers, or the network's stages.  Per level, launches over the
// whole GPU -> here: n=100 k=3 beam 10 73 -> 6.2 us, n=64 beam 4000 105 -> 31,
// n=128 beam 896 114 -> 17, n=200 beam 1528 121 -> 43.
template <int W>
__global__ void __launch_bounds__(kBeamThreads, 1) k_beam(const uint16_t* __restrict__ delta, u32 n, u32 k, u32 beam,
                                                          u32 m, u32 parents, u32 levels, u64* __restrict__ rows,
                                                          u32* __restrict__ log, u32* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t s_raw[];
  const BeamLayout L = beam_layout(W, n, k, parents);
  u64* const child = (u64*)(s_raw + L.child);
  u32* const col = (u32*)(s_raw + L.col);
  uint16_t* const s_delta = (uint16_t*)(s_raw + L.delta);
  u32* const count = (u32*)(s_raw + L.bins);
  u32* const first = count + (kBeamBins + 1);
  uint16_t* const key = (uint16_t*)(s_raw + L.key);
  uint16_t* const list = (uint16_t*)(s_raw + L.list);
  uint16_t* const kept = (uint16_t*)(s_raw + L.kept);
  __shared__ u32 s_full, s_least, s_most, s_pairs, s_sum[32];
  const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, warps = kBeamThreads / 32;
  const u32 cap = parents * k;
  const u32 low = W == 1 ? 64 - n : 0;  // the first word's last state, whose bit leads the order
  for (u32 e = tid; e < n * k; e += kBeamThreads) s_delta[e] = delta[e];
  for (u32 g = warp; g < (m + 31) / 32; g += warps) {
    u64 x[W];
#pragma unroll
    for (int w = 0; w < W; ++w) x[w] = 32 * g + lane < m ? rows[(size_t)(32 * g + lane) * W + w] : 0;
    rows_to_columns<W>(x, col + (size_t)g * 64 * W);
  }
  u32 done = 0, found = 0;
  for (; done < levels; ++done) {
    const u32 N = m * k, groups = (m + 31) / 32;
    for (u32 b = tid; b <= kBeamBins; b += kBeamThreads) count[b] = 0;
    if (tid == 0) {
      s_full = s_least = ~0u;
      s_most = s_pairs = 0;
    }
    __syncthreads();
    for (u32 t = warp; t < k * groups; t += warps) {
      const u32 a = t / groups, g = t % groups, p = 32 * g + lane;
      u64 x[W];
      expand_columns<W, false>(col + (size_t)g * 64 * W, n, s_delta + a * n, 1u, (const uint16_t*)nullptr,
                               (const uint16_t*)nullptr, x);
      u32 missing = ~0u;
      if (p < m) {
        const u32 i = a * m + p;
        u32 c = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
          child[(size_t)w * cap + i] = x[w];
          c += __popcll(x[w]);
        }
        missing = n - c;
        key[i] = (uint16_t)missing;
        if (c == n) atomicMin(&s_full, i);
      }
      const u32 least = __reduce_min_sync(0xffffffffu, missing);
      const u32 most = __reduce_max_sync(0xffffffffu, p < m ? missing : 0u);
      if (lane == 0) {
        atomicMin(&s_least, least);
        atomicMax(&s_most, most);
      }
    }
    __syncthreads();
    if (tid == 0) out[kBeamHeader + kBeamLevels + done] = m;
    if (s_full != ~0u) {  // beam.hpp:173-177: the largest set is all states
      found = 1;
      break;
    }
    // bins: cardinality, then as many leading bits of the order as there is room for
    const u32 least = s_least, range = s_most - least + 1;
    const u32 bits = 31 - __clz(kBeamBins / range);
    for (u32 i = tid; i < N; i += kBeamThreads) {
      const u32 lead = bits ? __brev((u32)(child[i] >> low)) >> (32 - bits) : 0;
      const u32 b = ((key[i] - least) << bits) | lead;
      key[i] = (uint16_t)b;
      atomicAdd(&count[b], 1u);
    }
    __syncthreads();
    // pairs that ranking within the bins would compare
    const u32 c0 = count[2 * tid], c1 = count[2 * tid + 1];
    const u32 pairs = __reduce_add_sync(0xffffffffu, c0 * c0 + c1 * c1);
    if (lane == 0) atomicAdd(&s_pairs, pairs);
    scan_bins(count, first, s_sum);
    __syncthreads();
    u32 unique;
    if (s_pairs > kBeamPairs * N) {
      sort_children<W>(list, key, child, cap, N);
      // runs of `run` places: the first of equal sets is kept, in order
      const u32 run = (N + kBeamThreads - 1) / kBeamThreads, p0 = min(tid * run, N), p1 = min(p0 + run, N);
      const auto fresh = [&](u32 p) { return p == 0 || !same_child<W>(child, cap, list[p], list[p - 1]); };
      u32 mine = 0;
      for (u32 p = p0; p < p1; ++p) mine += fresh(p);
      count[2 * tid] = mine;
      count[2 * tid + 1] = 0;
      __syncthreads();
      scan_bins(count, count, s_sum);
      __syncthreads();
      u32 r = count[2 * tid];
      for (u32 p = p0; p < p1 && r < beam; ++p)
        if (fresh(p)) kept[r++] = list[p];
      unique = count[kBeamBins];
    } else {
      for (u32 i = tid; i < N; i += kBeamThreads) list[atomicAdd(&count[key[i]], 1u)] = (uint16_t)i;
      __syncthreads();
      for (u32 b = tid; b <= kBeamBins; b += kBeamThreads) count[b] = 0;
      __syncthreads();
      for (u32 p = tid; p < N; p += kBeamThreads) {
        const u32 i = list[p], b = key[i], end = first[b + 1];
        u64 x[W];
#pragma unroll
        for (int w = 0; w < W; ++w) x[w] = child[(size_t)w * cap + i];
        bool dup = false;
        for (u32 j = first[b]; j < end && !dup; ++j) {
          const u32 o = list[j];
          if (child[o] != x[0] || o >= i) continue;
          bool same = true;
#pragma unroll
          for (int w = 1; w < W; ++w) same = same && child[(size_t)w * cap + o] == x[w];
          dup = same;
        }
        if (dup)
          key[i] = (uint16_t)(b | kDuplicate);
        else
          atomicAdd(&count[b], 1u);
      }
      __syncthreads();
      scan_bins(count, count, s_sum);  // distinct sets before each bin; first keeps the bins' places
      __syncthreads();
      unique = count[kBeamBins];
      for (u32 p = tid; p < N; p += kBeamThreads) {
        const u32 i = list[p], b = key[i];
        if (b & kDuplicate) continue;
        u32 r = count[b];
        if (r >= beam) continue;
        u64 x[W];
#pragma unroll
        for (int w = 0; w < W; ++w) x[w] = child[(size_t)w * cap + i];
        const u32 end = first[b + 1];
        for (u32 j = first[b]; j < end; ++j) {
          const u32 o = list[j];
          // order of the bit-reversed words: the lowest differing bit decides
          u64 d = child[o] ^ x[0], y = x[0];
#pragma unroll
          for (int w = 1; w < W; ++w)
            if (!d) {
              y = x[w];
              d = child[(size_t)w * cap + o] ^ y;
            }
          r += (y & (d & (~d + 1))) != 0 && !(key[o] & kDuplicate);
        }
        if (r < beam) kept[r] = (uint16_t)i;
      }
    }
    __syncthreads();
    m = min(unique, beam);
    const bool last = done + 1 == levels;
    for (u32 g = warp; g < (m + 31) / 32; g += warps) {
      const u32 p = 32 * g + lane, i = p < m ? kept[p] : 0;
      u64 x[W];
#pragma unroll
      for (int w = 0; w < W; ++w) x[w] = p < m ? child[(size_t)w * cap + i] : 0;
      rows_to_columns<W>(x, col + (size_t)g * 64 * W);
      if (p < m) {
        log[(size_t)done * parents + p] = i;
        if (last) {
#pragma unroll
          for (int w = 0; w < W; ++w) rows[(size_t)p * W + w] = x[w];
        }
      }
    }
    __syncthreads();
  }
  if (tid == 0) {
    u32 at = 0;
    if (found) {  // letters of this launch's levels, the last applied first
      u32 val = s_full;
      for (u32 d = done;; --d) {
        const u32 pm = out[kBeamHeader + kBeamLevels + d];
        out[kBeamHeader + done - d] = val / pm;
        at = val % pm;
        if (d == 0) break;
        val = log[(size_t)(d - 1) * parents + at];
      }
    }
    out[0] = found;
    out[1] = done + found;  // levels expanded
    out[2] = m;
    out[3] = at;  // the found set's ancestor among the rows this launch started from
  }
}

bool beam_fits(int W, u32 n, u32 k, u64 parents) {
  return parents * k < kDuplicate && beam_layout(W, n, k, (u32)parents).bytes <= kBeamSmemBytes;
}

void launch_beam(int W, const uint16_t* delta, u32 n, u32 k, u32 beam, u32 m, u32 parents, u32 levels, u64* rows,
                 u32* log, u32* out, cudaStream_t s) {
  const size_t bytes = beam_layout(W, n, k, parents).bytes;
  const auto go = [&](auto kernel) {
    SW_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBeamSmemBytes));
    kernel<<<1, kBeamThreads, bytes, s>>>(delta, n, k, beam, m, parents, levels, rows, log, out);
  };
  switch (W) {
    case 1: go(k_beam<1>); break;
    case 2: go(k_beam<2>); break;
    case 3: go(k_beam<3>); break;
    case 4: go(k_beam<4>); break;
    case 5: go(k_beam<5>); break;
    case 6: go(k_beam<6>); break;
    case 7: go(k_beam<7>); break;
    case 8: go(k_beam<8>); break;
    default: throw std::runtime_error("unsupported set width");
  }
  SW_LAUNCH_CHECK();
}

}  // namespace sw
