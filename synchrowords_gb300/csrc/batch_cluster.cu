// Device-resident exact search: one thread-block cluster per automaton of up
// to 256 states, the meet-in-the-middle search in one persistent launch.
//
// The streamed path (exact.cu) drives every BFS level from the host: an
// expansion, a sort, a compaction, a merge and a subset check per level, each
// a launch, with the counts read back in between.  While the lists hold up to
// a few thousand sets those launches are latency-bound (about 90 us a level
// whatever its size).  Here a cluster of CTAs keeps the level loop on the
// device:
//   * the lists of both sides live in a per-cluster global region (L2
//     resident at these sizes); the CTAs of the cluster split every phase and
//     meet at hardware cluster barriers (barrier.cluster, release/acquire), two
//     per level;
//   * expansion and duplicate removal are one phase.  Child e = letter * m +
//     parent is written to the side's row slot `used + e`, then looked up and
//     inserted in the side's open-addressing hash table in one probe sequence
//     (a row equal to one of an earlier layer or to a sibling is found there and
//     dropped).  A layer is the list of the slots it kept, so nothing is copied
//     or compacted, and a kept row's slot names its letter and parent;
//   * slots carry a tag unique to the search, so no table is cleared between
//     automata;
//   * the meet check f ⊆ B (f ∩ b' = ∅) tests small layers pair by pair (lane
//     per backward row, 32 forward rows per warp in shared memory) and stages
//     the backward rows of large ones bit-sliced: for every state q a bitmap
//     over the layer's rows (bit j set when q lies in B_j).  A warp then takes
//     one forward set f at a time and ANDs the bitmaps of f's states, 32 rows
//     per lane-word, stopping as soon as every word is zero; a word still
//     nonzero when f's states run out names a B_j ⊇ f;
//   * the word is traced back through the layers' slot lists.
// Exactness: one side grows by one layer per step, every total
// length is checked once, and a set equal to one of an earlier layer of its
// side is dropped (a shorter prefix reaches it).  An automaton whose lists
// outgrow the capacities, or whose search reaches the depth or length limit,
// is reported with the reason and solved again by the streamed path.  A launch
// may also stop at a level boundary once a level passes the work limits it was
// given: the streamed search then goes on from the region's lists
// (launch_cluster_export).
//
// Replaces, for these sizes, the reference's MeetInTheMiddle::run loop
// (synchrolib/algorithm/exact/meet_in_the_middle.cpp:58-107) with its BFS /
// IBFS steps (:179-344) and goal check (:90).
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <set>
#include <utility>

#include "algos.cuh"
#include "rowset.cuh"

namespace sw {

namespace {
constexpr int kCtThreads = 1024;
constexpr int kCtWarps = kCtThreads / 32;
constexpr u32 kCtMaxDepth = 1024;   // layers per side
constexpr u32 kCtChunkRows = 4096;  // backward rows per bit-sliced meet-check chunk
constexpr u32 kCtGroups = kCtChunkRows / 32;  // 32-row bitmap words per state and chunk
constexpr u32 kCtFSlice = 32 * kCtWarps;  // forward sets per meet-check unit (32 per warp)
constexpr u32 kCtMaxNK = 4096;      // n * k of the transition table staged per CTA
constexpr u32 kRunning = 255;

__device__ __forceinline__ u32 cluster_rank() {
  u32 r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ u32 cluster_ctas() {
  u32 r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ u32 cluster_index() {
  u32 r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
// Every thread of every CTA of the cluster arrives and waits; the arrive
// releases and the wait acquires at cluster scope, so global-memory writes made
// before the barrier by any CTA of the cluster are visible after it.
// A row's words before its table slot, for the CTAs of the cluster.
__device__ __forceinline__ void cluster_fence() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A table slot: the search's tag (26 bits), a fingerprint of the row (16), its
// row slot (22).
constexpr int kSlotTagShift = 38, kSlotRowBits = 22;
constexpr u32 kSlotRowMask = (1u << kSlotRowBits) - 1;

// Looks x (stored in the side's row slot r) up and inserts it: true when no
// equal row was there.  Every probe sequence is bounded by the table size.
template <int W>
__device__ __forceinline__ bool table_insert(u64* vt, u32 vmask, u64 tag, const u64* V, const u64* x, u32 r,
                                             u32* overflow) {
  const u64 h = row_hash<W>(x);
  const u64 mine = (tag << kSlotTagShift) | ((h >> 48) << kSlotRowBits) | r;
  u32 slot = (u32)h & vmask;
  for (u32 it = 0; it <= vmask; ++it) {
    u64 v = ld_volatile64(&vt[slot]);
    if ((v >> kSlotTagShift) != tag) {  // empty, or left by an earlier search
      const u64 old = atomicCAS(&vt[slot], v, mine);
      if (old == v) return true;
      v = old;  // taken meanwhile, by a row of this search
    }
    if (((v ^ mine) >> kSlotRowBits) == 0) {  // same tag and fingerprint
      cluster_fence();                        // the row was written before its slot
      if (row_eq_volatile<W>(V + (size_t)((u32)v & kSlotRowMask) * W, x)) return false;
    }
    slot = (slot + 1) & vmask;
  }
  atomicOr(overflow, 1u);
  return false;
}

__device__ __forceinline__ uint4 ld_volatile128(const void* p) {
  uint4 v;
  asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}

// Per-cluster control words (one 256-byte block per cluster index; the first
// four are read together).
struct ClusterCtl {
  u32 fcount[2];  // kept children of the step (by step parity)
  u32 overflow;   // bit 0: a table probe ran out (never expected: tables hold more slots than rows); bit 1: given up
  u32 found;      // meet flag
  u32 inst;       // automaton being solved
  u32 vtag;       // tag of this search's table slots
  u32 fi, bj;     // meeting pair: index in the current F layer, in the current B layer
  ClusterExit exit;  // how the last search ended
  u32 pad[64 - 8 - sizeof(ClusterExit) / 4];
};
static_assert(sizeof(ClusterCtl) == 256, "control block is one 256-byte line");
static_assert(offsetof(ClusterCtl, exit) == kClusterExitOffset - 256, "the exit record's place in the scratch");

}  // namespace

// Byte offsets of one cluster's region (set width W, capacities c).  The hash
// tables come first, at offsets that depend on the capacities only: a launch of
// any width and any cluster count finds every table slot either zero or holding
// a tag an earlier search took, never row data of another layout read as a tag.
// meta: per side the first row slot, the first list entry and the row count of
// every layer.
struct ClusterRegion {
  size_t vtab[2], meta, vis[2], lst[2], bytes;
};
static_assert(kClusterMetaStride == kCtMaxDepth + 1, "one table entry per layer and one for the seeds");

template <int W>
__host__ __device__ inline ClusterRegion cluster_region(const ClusterCaps& c) {
  ClusterRegion r{};
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o += (bytes + 255) & ~(size_t)255;
    return at;
  };
  r.vtab[0] = take(sizeof(u64) << c.vtab_bits);
  r.vtab[1] = take(sizeof(u64) << c.vtab_bits);
  r.meta = take(sizeof(u32) * kClusterMetaWords);
  r.vis[0] = take(sizeof(u64) * W * (size_t)c.vis);
  r.vis[1] = take(sizeof(u64) * W * (size_t)c.vis);
  r.lst[0] = take(sizeof(u32) * (size_t)c.vis);
  r.lst[1] = take(sizeof(u32) * (size_t)c.vis);
  r.bytes = o;
  return r;
}

// Scratch = header (tag counter, then one control block per cluster index, for
// kCtMaxClusters clusters) + one region per cluster, every region as large as
// the widest (W = 4) layout needs.
constexpr u32 kCtMaxClusters = 512;
constexpr size_t kCtHeaderBytes = 256 + 256 * (size_t)kCtMaxClusters;

// Level of pairs above which the meet check goes bit-sliced: staging a chunk
// costs a CTA about as much as testing 2^18 pairs one by one.
constexpr u64 kCtDirectPairs = 1ull << 21;

template <int W>
__global__ void __launch_bounds__(kCtThreads, 1)
    k_cluster_batch(const SmallInstance* __restrict__ inst, u32 count, const uint8_t* __restrict__ delta_pool,
                    const uint8_t* __restrict__ seed_pool, SmallResult* results, uint8_t* words, u32 word_stride,
                    uint8_t* scratch, size_t region_stride, ClusterCaps caps, ClusterLimits lim, u32* counter,
                    u64* stats) {
  // meet check: bitmaps s_col[q * kCtGroups + g], q < 64 W, or 32 forward rows
  // per warp; expansion: one warp's parents as columns, 64 W words per warp
  extern __shared__ __align__(16) u32 s_col[];
  __shared__ uint8_t s_delta[kCtMaxNK];          // delta[q * k + a]
  __shared__ uint8_t s_isrc[kCtMaxNK];           // preimage lists, letter-major CSR
  __shared__ u32 s_ibeg[kCtMaxNK + 16 + 1];      // list of (a, t): [s_ibeg[a*(n+1)+t], s_ibeg[a*(n+1)+t+1])
  __shared__ u32 s_fill[kCtMaxNK];
  __shared__ u64 s_par[kCtWarps][W];
  __shared__ u32 s_flag;

  const u32 rank = cluster_rank(), CS = cluster_ctas();
  const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u32 gtid = rank * kCtThreads + tid, G = CS * kCtThreads;
  const u32 NW = G >> 5;
  // consecutive warp indices alternate between the CTAs, so that few warps' work spreads over all of them
  const u32 gwarp = warp * CS + rank;

  u32* tag_counter = reinterpret_cast<u32*>(scratch);
  ClusterCtl* ctl = reinterpret_cast<ClusterCtl*>(scratch + 256) + cluster_index();
  uint8_t* base = scratch + lim.header_bytes + (size_t)cluster_index() * region_stride;
  const ClusterRegion R = cluster_region<W>(caps);
  u32* const meta = reinterpret_cast<u32*>(base + R.meta);
  auto m_voff = [&](int side) { return meta + side * (kCtMaxDepth + 1); };
  auto m_loff = [&](int side) { return meta + (2 + side) * (kCtMaxDepth + 1); };
  auto m_cnt = [&](int side) { return meta + (4 + side) * (kCtMaxDepth + 1); };
  u64* const V0 = reinterpret_cast<u64*>(base + R.vis[0]);
  u64* const V1 = reinterpret_cast<u64*>(base + R.vis[1]);
  u32* const L0 = reinterpret_cast<u32*>(base + R.lst[0]);
  u32* const L1 = reinterpret_cast<u32*>(base + R.lst[1]);
  u64* const vt0 = reinterpret_cast<u64*>(base + R.vtab[0]);
  u64* const vt1 = reinterpret_cast<u64*>(base + R.vtab[1]);
  const u32 vmask = (1u << caps.vtab_bits) - 1;

  for (;;) {
    if (rank == 0 && tid == 0) {
      ctl->inst = atomicAdd(counter, 1u);
      ctl->vtag = atomicAdd(tag_counter, 1u) + 1u;
      ctl->fcount[0] = ctl->fcount[1] = 0;
      ctl->overflow = 0;
      ctl->found = 0;
    }
    cluster_barrier();
    const u32 id = ld_volatile(&ctl->inst);
    if (id >= count) break;  // the same value in every CTA: the cluster leaves together
    const u64 vtag = ld_volatile(&ctl->vtag);
    const SmallInstance I = inst[id];
    const u32 n = I.n, k = I.k, sc = I.seed_count;
    // transition table and its inverse lists, per CTA: the preimages of t
    // under a are s_isrc[s_ibeg[a*(n+1)+t] .. s_ibeg[a*(n+1)+t+1])
    for (u32 e = tid; e < n * k; e += kCtThreads) s_delta[e] = delta_pool[I.delta_off + e];
    for (u32 e = tid; e < k * (n + 1); e += kCtThreads) s_ibeg[e] = 0;
    for (u32 e = tid; e < n * k; e += kCtThreads) s_fill[e] = 0;
    __syncthreads();
    for (u32 e = tid; e < n * k; e += kCtThreads) {
      const u32 q = e / k, a = e - q * k;
      atomicAdd(&s_ibeg[a * (n + 1) + s_delta[e] + 1], 1u);  // in-degree of t, one entry to the right
    }
    __syncthreads();
    if (warp < k) {  // warp per letter: start of every list, from a * n
      u32 run = warp * n;
      for (u32 t0 = 0; t0 <= n; t0 += 32) {
        const u32 t = t0 + lane;
        u32 v = t <= n ? s_ibeg[warp * (n + 1) + t] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const u32 y = __shfl_up_sync(0xffffffffu, v, o);
          if (lane >= (u32)o) v += y;
        }
        if (t <= n) s_ibeg[warp * (n + 1) + t] = run + v;
        run += __shfl_sync(0xffffffffu, v, 31);
      }
    }
    __syncthreads();
    for (u32 e = tid; e < n * k; e += kCtThreads) {
      const u32 q = e / k, a = e - q * k, t = s_delta[e];
      const u32 slot = atomicAdd(&s_fill[a * n + t], 1u);
      s_isrc[s_ibeg[a * (n + 1) + t] + slot] = (uint8_t)q;
    }
    __syncthreads();
    u32 status = kRunning, why = 0, length = 0;
    if (sc == 0 || sc > caps.vis) {
      status = 1;
      why = 3;
    }
    // seeds: F = {Q}, B = complements of the seed singletons, entered in the tables
    if (status == kRunning) {
      for (u32 i = gtid; i < 1 + sc; i += G) {
        const int s = i == 0 ? -1 : (int)seed_pool[I.seed_off + i - 1];
        const u32 r = i == 0 ? 0 : i - 1;
        u64* const V = i == 0 ? V0 : V1;
        u64 x[W];
#pragma unroll
        for (int w = 0; w < W; ++w) {
          x[w] = valid_mask((int)n, w) & ~(s >= 0 && state_word(s) == w ? state_bit(s) : 0ULL);
          V[(size_t)r * W + w] = x[w];
        }
        (i == 0 ? L0 : L1)[r] = r;
        cluster_fence();
        table_insert<W>(i == 0 ? vt0 : vt1, vmask, vtag, V, x, r, &ctl->overflow);
      }
      if (rank == 0 && tid == 0) {
        m_voff(0)[0] = m_voff(1)[0] = m_loff(0)[0] = m_loff(1)[0] = 0;
        m_cnt(0)[0] = 1;
        m_cnt(1)[0] = sc;
      }
    }
    cluster_barrier();
    // per-side counters, identical in every thread of the cluster: rows of the
    // current layer, row slots and list entries used, first list entry of the
    // current layer, depth
    u32 cnt0 = 1, cnt1 = sc, used0 = 1, used1 = sc, ll0 = 1, ll1 = sc, cur0 = 0, cur1 = 0, depth0 = 0, depth1 = 0;
    u64 my_pairs = 0, my_children = 0, my_staged = 0, my_queries = 0;
    u32 steps = 0, rt = 0;
    // cycles between the cluster barriers, per phase (rank 0, thread 0): stats[4..8]
    long long clk = clock64();
    u64 ph[3] = {0, 0, 0};
    auto lap = [&](int i) {
      const long long t = clock64();
      ph[i] += (u64)(t - clk);
      clk = t;
    };
    for (; status == kRunning; ++rt) {
      if (rt >= I.max_len) {
        status = 2;
        why = 9;
        break;
      }
      const int X = cnt0 <= cnt1 ? 0 : 1;  // expand the smaller frontier
      u64* const VX = X ? V1 : V0;
      u32* const LX = X ? L1 : L0;
      u64* const vtX = X ? vt1 : vt0;
      const u32 m = X ? cnt1 : cnt0;
      const u32 usedX = X ? used1 : used0;
      const u32 llX = X ? ll1 : ll0;
      const u32 curX = X ? cur1 : cur0;
      const u32 depthX = X ? depth1 : depth0;
      const u64 c64 = (u64)m * k;
      if (c64 > caps.ch || usedX + c64 > caps.vis || depthX + 1 > kCtMaxDepth) {
        status = 1;
        why = c64 > caps.ch ? 1u : (depthX + 1 > kCtMaxDepth ? 4u : 3u);
        break;
      }
      const u32 c = (u32)c64;
      if (c > lim.max_children || (u64)cnt0 * cnt1 > lim.max_pairs ||
          4 * (((u64)cnt0 + ll0 + cnt1 + ll1) * 8 * W + (u64)c * (24 * W + 16)) > lim.budget) {
        status = 3;  // a level of this size belongs to the whole GPU
        break;
      }
      // read now, used at the level's end: the word lies in host memory, a microsecond away
      u32 given_up = 0;
      if (lim.cancel && rank == 0 && tid == 0 && rt % kClusterPoll == kClusterPoll - 1) given_up = ld_volatile(lim.cancel);
      // ---- expansion and duplicate removal ----
      const u32* const P = LX + curX;  // the parents' row slots
      const u32 par = rt & 1u;
      auto insert = [&](const u64* x, bool valid, u32 e) {
        const u32 r = usedX + e;
        if (valid) {
#pragma unroll
          for (int w = 0; w < W; ++w) VX[(size_t)r * W + w] = x[w];
        }
        cluster_fence();  // the row before its slot
        const bool keep = valid && table_insert<W>(vtX, vmask, vtag, VX, x, r, &ctl->overflow);
        const u32 kmask = __ballot_sync(0xffffffffu, keep);
        u32 pos0 = 0;
        if (lane == 0 && kmask) pos0 = atomicAdd(&ctl->fcount[par], (u32)__popc(kmask));
        pos0 = __shfl_sync(0xffffffffu, pos0, 0);
        if (keep) LX[llX + pos0 + __popc(kmask & ((1u << lane) - 1u))] = r;
      };
      if (c <= 2 * NW) {
        // few children: a warp decides one child's states by ballots
        for (u32 e = gwarp; e < c; e += NW) {
          const u32 a = e / m, p = e - a * m;
          if (lane < (u32)W) s_par[warp][lane] = VX[(size_t)P[p] * W + lane];
          __syncwarp();
          u64 x[W];
#pragma unroll
          for (int w = 0; w < W; ++w) {
            u32 b[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const u32 s = 64 * w + 32 * h + lane;
              bool bit = false;
              if (s < n) {
                if (X == 1) {  // preimage of a complement row: s with δ(s, a) in the row
                  const u32 d = s_delta[s * k + a];
                  bit = (s_par[warp][d >> 6] >> (63 - (d & 63))) & 1ULL;
                } else {  // image: some preimage of s under a lies in the row
                  const u32 b0 = s_ibeg[a * (n + 1) + s], b1 = s_ibeg[a * (n + 1) + s + 1];
                  for (u32 j = b0; j < b1 && !bit; ++j) {
                    const u32 q = s_isrc[j];
                    bit = (s_par[warp][q >> 6] >> (63 - (q & 63))) & 1ULL;
                  }
                }
              }
              b[h] = __ballot_sync(0xffffffffu, bit);
            }
            // lane l decided state 64w + l (bit 63 - l) and 64w + 32 + l (bit 31 - l)
            x[w] = ((u64)__brev(b[0]) << 32) | (u64)__brev(b[1]);
          }
          __syncwarp();
          insert(x, lane == 0, e);
        }
      } else {
        // a warp takes 32 parents under one letter as columns (a word per
        // state, a bit per parent): a child's column is a gather of the
        // parents', and two bit transposes lead in and out; about 12
        // instructions a child instead of 100 by ballots (rowset.cuh)
        u32* const col = s_col + warp * 64 * W;
        const u32 groups = (m + 31) / 32;
        for (u32 u = gwarp; u < groups * k; u += NW) {
          const u32 a = u / groups, p = 32 * (u - a * groups) + lane;
          const bool valid = p < m;
          const u64* const row = VX + (size_t)(valid ? P[p] : 0u) * W;
          u64 x[W];
#pragma unroll
          for (int w = 0; w < W; ++w) x[w] = valid ? row[w] : 0ULL;
          rows_to_columns<W>(x, col);
          __syncwarp();
          if (X == 1)
            expand_columns<W, false>(col, n, s_delta + a, k, s_ibeg, s_isrc, x);
          else
            expand_columns<W, true>(col, n, s_delta, 0u, s_ibeg + a * (n + 1), s_isrc, x);
          __syncwarp();
          insert(x, valid, a * m + p);
        }
      }
      my_children += c;
      if (given_up) atomicOr(&ctl->overflow, 2u);
      cluster_barrier();
      lap(0);
      const uint4 now = ld_volatile128(ctl);  // both counts, overflow, meet flag
      const u32 f = par ? now.y : now.x;
      if (rank == 0 && tid == 0) {
        ctl->fcount[par ^ 1u] = 0;
        m_voff(X)[depthX + 1] = usedX;
        m_loff(X)[depthX + 1] = llX;
        m_cnt(X)[depthX + 1] = f;
      }
      if (X) {
        cur1 = llX;
        ll1 = llX + f;
        used1 = usedX + c;
        cnt1 = f;
        depth1 = depthX + 1;
      } else {
        cur0 = llX;
        ll0 = llX + f;
        used0 = usedX + c;
        cnt0 = f;
        depth0 = depthX + 1;
      }
      ++steps;
      if (now.z) {
        status = 1;
        why = now.z & 1u ? 6 : 7;
        break;
      }
      if (f == 0) {  // a side died out: no reset word within reach
        status = 2;
        why = 8;
        ++rt;
        break;
      }
      // ---- meet check of the current layers: some f ⊆ B_j (f ∩ b'_j = ∅) ----
      const u32 nF = cnt0, nB = cnt1;
      const u32* const lF = L0 + cur0;
      const u32* const lB = L1 + cur1;  // rows are complements b' = Q \ B
      my_pairs += (u64)nF * nB;
      my_queries += nB;
      if ((u64)nF * nB <= kCtDirectPairs) {
        u64* const s_f = reinterpret_cast<u64*>(s_col) + warp * 32 * W;
        const u32 fgs = (nF + 31) / 32, tasks = ((nB + 31) / 32) * fgs;
        for (u32 t = gwarp; t < tasks; t += NW) {
          const u32 bg = t / fgs, fg = t - bg * fgs;
          const u32 bi = 32 * bg + lane, fi = 32 * fg + lane, nf = min(32u, nF - 32 * fg);
          u64 b[W];
#pragma unroll
          for (int w = 0; w < W; ++w) b[w] = ~0ULL;
          if (bi < nB) {
            const u64* const row = V1 + (size_t)lB[bi] * W;
#pragma unroll
            for (int w = 0; w < W; ++w) b[w] = row[w];
          }
          const u64* const frow = V0 + (size_t)(fi < nF ? lF[fi] : 0u) * W;
#pragma unroll
          for (int w = 0; w < W; ++w) s_f[lane * W + w] = fi < nF ? frow[w] : ~0ULL;
          __syncwarp();
          for (u32 j0 = 0; j0 < nf; j0 += 4) {  // entries past nf are full words: never disjoint from a row
            u32 open = 0;
#pragma unroll
            for (u32 i = 0; i < 4; ++i) open |= (s_f[(j0 + i) * W] & b[0]) ? 0u : 1u << i;
            if (!__any_sync(0xffffffffu, open)) continue;
#pragma unroll
            for (u32 i = 0; i < 4; ++i)
#pragma unroll
              for (int w = 1; w < W; ++w)
                if (s_f[(j0 + i) * W + w] & b[w]) open &= ~(1u << i);
            if (open && j0 + __ffs(open) - 1 < nf && atomicCAS(&ctl->found, 0u, 1u) == 0u) {
              ctl->fi = 32 * fg + j0 + __ffs(open) - 1;
              ctl->bj = bi;
            }
          }
          __syncwarp();
        }
      } else {
        const u32 chunks = (nB + kCtChunkRows - 1) / kCtChunkRows;
        const u32 fslices = (nF + kCtFSlice - 1) / kCtFSlice;
        const u32 units = chunks * fslices;
        u32 staged = 0xffffffffu;
        // Block barriers only around restaging a chunk (every warp of the CTA
        // walks the same unit sequence); a warp that sees the meet flag set
        // skips its remaining work but still takes part in those barriers.
        bool met = false;
        for (u32 u = rank; u < units; u += CS) {
          const u32 chunk = u / fslices, fs = u - chunk * fslices;
          const u32 r0 = chunk * kCtChunkRows;
          const u32 rows = min(kCtChunkRows, nB - r0);
          const u32 groups = (rows + 31) / 32;
          if (chunk != staged) {
            if (tid == 0) s_flag = ld_volatile(&ctl->found);
            __syncthreads();  // every warp is done with the previous chunk
            if (s_flag != 0) break;  // block-uniform: the meet was found
            // transpose: bit j of s_col[q * kCtGroups + g] says state q lies in
            // B_{r0 + 32 g + j}; warp per 32-row group
            for (u32 g = warp; g < groups; g += kCtWarps) {
              const u32 r = 32 * g + lane;
              const u64* const row = V1 + (size_t)(r < rows ? lB[r0 + r] : 0u) * W;
#pragma unroll
              for (int w = 0; w < W; ++w) {
                const u64 b = r < rows ? ~row[w] & valid_mask((int)n, w) : 0ULL;
                s_col[(64 * w + 31 - lane) * kCtGroups + g] = transpose32((u32)(b >> 32));
                s_col[(64 * w + 63 - lane) * kCtGroups + g] = transpose32((u32)b);
              }
            }
            staged = chunk;
            my_staged += (u64)rows * W * 8;
            __syncthreads();
          }
          // warp per 32 forward sets: lane l fetches set f0 + 32 warp + l, then
          // the warp takes them one by one (broadcast by shuffle) and ANDs the
          // bitmaps of each set's states; lane l owns the chunk's 32-row words
          // 4l .. 4l + 3 (one 16-byte shared load per state)
          if (!met) {
            u32 fl = lane == 0 ? ld_volatile(&ctl->found) : 0u;
            met = __shfl_sync(0xffffffffu, fl, 0) != 0;
          }
          if (met) continue;
          const u32 fw0 = fs * kCtFSlice + warp * 32;
          const u32 fw1 = min(nF, fw0 + 32);
          const u64* const frow = V0 + (size_t)(fw0 + lane < fw1 ? lF[fw0 + lane] : 0u) * W;
          u64 myf[W];
#pragma unroll
          for (int w = 0; w < W; ++w) myf[w] = fw0 + lane < fw1 ? frow[w] : 0ULL;
          u32 acc0[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const u32 g = 4 * lane + i;
            acc0[i] = g < groups ? (32 * g + 32 <= rows ? 0xffffffffu : (1u << (rows - 32 * g)) - 1u) : 0u;
          }
          for (u32 t = 0; fw0 + t < fw1; ++t) {
            u32 acc[4] = {acc0[0], acc0[1], acc0[2], acc0[3]};
            bool alive = true;
#pragma unroll
            for (int w = W - 1; w >= 0; --w) {
              u64 v = __shfl_sync(0xffffffffu, myf[w], t);
              while (v && alive) {
                const u32 j = 63 - (__ffsll((long long)v) - 1);  // state 64 w + j (bit 63 - j)
                v &= v - 1;
                const uint4 col = reinterpret_cast<const uint4*>(s_col + (64 * w + j) * kCtGroups)[lane];
                acc[0] &= col.x;
                acc[1] &= col.y;
                acc[2] &= col.z;
                acc[3] &= col.w;
                alive = __any_sync(0xffffffffu, (acc[0] | acc[1] | acc[2] | acc[3]) != 0u);
              }
            }
            if (alive) {  // some B_j contains every state of f
              u32 hit = 0xffffffffu;
#pragma unroll
              for (int i = 3; i >= 0; --i)
                if (acc[i]) hit = 32 * (4 * lane + i) + __ffs(acc[i]) - 1;
              const u32 who = __ballot_sync(0xffffffffu, hit != 0xffffffffu);
              const u32 bj = __shfl_sync(0xffffffffu, hit, __ffs(who) - 1);
              if (lane == 0 && atomicCAS(&ctl->found, 0u, 1u) == 0u) {
                ctl->fi = fw0 + t;
                ctl->bj = r0 + bj;
              }
              break;
            }
          }
        }
      }
      cluster_barrier();
      lap(1);
      if (ld_volatile(&ctl->found)) {
        status = 0;
        length = rt + 1;
      }
    }
    // ---- result and word (forward letters from depth 1 up, then backward letters from the top down) ----
    if (rank == 0 && tid == 0) {
      SmallResult res;
      res.status = status;
      res.length = status == 0 ? length : rt;
      res.word_len = 0;
      res.why = why | ((depth0 + depth1) << 8);
      if (status == 0 && length <= word_stride) {
        uint8_t* wout = words + (size_t)id * word_stride;
        // a kept row's slot is its layer's first slot + letter * parents + parent
        u32 idx = ld_volatile(&ctl->fi);
        for (u32 d = depth0; d >= 1; --d) {
          const u32 e = L0[m_loff(0)[d] + idx] - m_voff(0)[d], pc = m_cnt(0)[d - 1];
          wout[d - 1] = (uint8_t)(e / pc);
          idx = e % pc;
        }
        idx = ld_volatile(&ctl->bj);
        u32 wpos = depth0;
        for (u32 d = depth1; d >= 1; --d) {
          const u32 e = L1[m_loff(1)[d] + idx] - m_voff(1)[d], pc = m_cnt(1)[d - 1];
          wout[wpos++] = (uint8_t)(e / pc);
          idx = e % pc;
        }
        res.word_len = wpos;
      } else if (status == 0) {
        res.status = 1;  // word longer than the buffer: solved again by the streamed path
        res.why = 5 | ((depth0 + depth1) << 8);
      }
      results[id] = res;
      ctl->exit = ClusterExit{my_pairs, my_children, my_queries, {depth0, depth1}, {ll0, ll1}, {cnt0, cnt1}};
      if (stats) {
        atomicAdd(&stats[0], (unsigned long long)my_pairs);
        atomicAdd(&stats[1], (unsigned long long)my_children);
        atomicAdd(&stats[3], (unsigned long long)steps);
        lap(2);
        for (int i = 0; i < 3; ++i) atomicAdd(&stats[4 + i], (unsigned long long)ph[i]);
      }
    }
    if (stats && tid == 0 && my_staged) atomicAdd(&stats[2], (unsigned long long)my_staged);
    cluster_barrier();  // the trace has read this search's records before the next one overwrites them
  }
}

// The lists a stopped search left in its region, for the streamed search to go
// on from: side X's kept rows (every layer, in order), the origin (letter *
// parents + parent position) of each, and nothing else; thread per kept row.
template <int W>
__global__ void k_cluster_export(const uint8_t* __restrict__ region, ClusterCaps caps, int side, u32 kept, u32 depth,
                                 u64* __restrict__ rows, u32* __restrict__ origin) {
  const u32 j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= kept) return;
  const ClusterRegion R = cluster_region<W>(caps);
  const u32* meta = reinterpret_cast<const u32*>(region + R.meta);
  const u32* voff = meta + side * (kCtMaxDepth + 1);
  const u32* loff = meta + (2 + side) * (kCtMaxDepth + 1);
  const u64* V = reinterpret_cast<const u64*>(region + R.vis[side]);
  const u32 r = reinterpret_cast<const u32*>(region + R.lst[side])[j];
  u32 lo = 0, hi = depth;  // last layer that starts at or before list entry j
  while (lo < hi) {
    const u32 mid = (lo + hi + 1) >> 1;
    if (loff[mid] <= j) lo = mid;
    else hi = mid - 1;
  }
#pragma unroll
  for (int w = 0; w < W; ++w) rows[(size_t)j * W + w] = V[(size_t)r * W + w];
  origin[j] = r - voff[lo];
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
namespace {
const void* cluster_fn_w(int W) {
  switch (W) {
    case 1: return (const void*)k_cluster_batch<1>;
    case 2: return (const void*)k_cluster_batch<2>;
    case 3: return (const void*)k_cluster_batch<3>;
    case 4: return (const void*)k_cluster_batch<4>;
  }
  throw std::runtime_error("cluster batch: unsupported width");
}
// bitmaps of 64 W states x kCtGroups words
size_t col_smem(int W) { return sizeof(u32) * 64 * (size_t)W * kCtGroups; }

std::mutex g_cluster_mu;
std::set<std::pair<int, const void*>> g_nonportable;  // (device, kernel) pairs opted in to clusters above 8

// Sets the kernel's attributes once per device, so that a launch issued
// while a stream is being captured makes no attribute call.
void prepare(const void* fn, int W, int cs) {
  std::lock_guard<std::mutex> g(g_cluster_mu);
  ensure_smem_limit(fn, (int)col_smem(W));
  if (cs > 8) {
    int dev = 0;
    SW_CUDA(cudaGetDevice(&dev));
    if (g_nonportable.insert({dev, fn}).second)
      SW_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
}
}  // namespace

ClusterCaps cluster_default_caps() {
  ClusterCaps c;
  c.vis = 3u << 20;
  c.ch = 1u << 20;
  c.vtab_bits = 22;  // at least four slots per three rows
  return c;
}

ClusterCaps cluster_single_caps() {
  ClusterCaps c;
  c.vis = 1u << 18;
  c.ch = 1u << 17;
  c.vtab_bits = 19;
  return c;
}

ClusterCaps cluster_tiny_caps() {
  ClusterCaps c;
  c.vis = 1u << 16;
  c.ch = 1u << 15;
  c.vtab_bits = 17;
  return c;
}

size_t cluster_scratch_bytes(u32 clusters, const ClusterCaps& c) {
  return kCtHeaderBytes + (size_t)clusters * cluster_region<4>(c).bytes;
}

size_t cluster_single_scratch_bytes(const ClusterCaps& c) { return kClusterSingleHeader + cluster_region<4>(c).bytes; }

u32 cluster_max_clusters_supported() { return kCtMaxClusters; }

u32 cluster_batch_max_clusters(int W, int cs) {
  const void* fn = cluster_fn_w(W);
  prepare(fn, W, cs);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)cs * 64, 1, 1);
  cfg.blockDim = dim3(kCtThreads, 1, 1);
  cfg.dynamicSmemBytes = col_smem(W);
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int clusters = 0;
  SW_CUDA(cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg));
  return (u32)std::max(clusters, 0);
}

void launch_cluster_batch(int W, int cs, u32 clusters, const SmallInstance* inst, u32 count,
                          const uint8_t* delta_pool, const uint8_t* seed_pool, SmallResult* results, uint8_t* words,
                          u32 word_stride, void* scratch, const ClusterCaps& caps, const ClusterLimits& limits,
                          u32* counter, u64* stats, cudaStream_t s) {
  if (!count || !clusters) return;
  if (cs < 1 || cs > 16) throw std::invalid_argument("cluster size must be 1..16");
  if (clusters > kCtMaxClusters) throw std::invalid_argument("too many clusters for the scratch header");
  if (caps.vtab_bits > 30 || caps.vis > kSlotRowMask || 3 * (1ull << caps.vtab_bits) < 4ull * caps.vis)
    throw std::invalid_argument("cluster batch: hash tables must hold four slots per three rows");
  ClusterLimits lim = limits;
  if (!lim.header_bytes) lim.header_bytes = kCtHeaderBytes;
  if (lim.header_bytes < 256 + sizeof(ClusterCtl) * (size_t)clusters)
    throw std::invalid_argument("cluster batch: scratch header too small for the clusters");
  const void* fn = cluster_fn_w(W);
  prepare(fn, W, cs);
  if (!lim.counter_ready) SW_CUDA(cudaMemsetAsync(counter, 0, sizeof(u32), s));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cs;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(cs * clusters), 1, 1);
  cfg.blockDim = dim3(kCtThreads, 1, 1);
  cfg.dynamicSmemBytes = col_smem(W);
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const size_t stride = cluster_region<4>(caps).bytes;  // every width uses the widest region
  uint8_t* sc = static_cast<uint8_t*>(scratch);
  switch (W) {
    case 1:
      SW_CUDA(cudaLaunchKernelEx(&cfg, k_cluster_batch<1>, inst, count, delta_pool, seed_pool, results, words,
                                 word_stride, sc, stride, caps, lim, counter, stats));
      break;
    case 2:
      SW_CUDA(cudaLaunchKernelEx(&cfg, k_cluster_batch<2>, inst, count, delta_pool, seed_pool, results, words,
                                 word_stride, sc, stride, caps, lim, counter, stats));
      break;
    case 3:
      SW_CUDA(cudaLaunchKernelEx(&cfg, k_cluster_batch<3>, inst, count, delta_pool, seed_pool, results, words,
                                 word_stride, sc, stride, caps, lim, counter, stats));
      break;
    case 4:
      SW_CUDA(cudaLaunchKernelEx(&cfg, k_cluster_batch<4>, inst, count, delta_pool, seed_pool, results, words,
                                 word_stride, sc, stride, caps, lim, counter, stats));
      break;
    default:
      throw std::runtime_error("cluster batch: unsupported width");
  }
  SW_LAUNCH_CHECK();
}

size_t cluster_meta_offset(int W, size_t header_bytes, const ClusterCaps& c) {
  switch (W) {
    case 1: return header_bytes + cluster_region<1>(c).meta;
    case 2: return header_bytes + cluster_region<2>(c).meta;
    case 3: return header_bytes + cluster_region<3>(c).meta;
    case 4: return header_bytes + cluster_region<4>(c).meta;
  }
  throw std::runtime_error("cluster meta: unsupported width");
}

void launch_cluster_export(int W, const void* scratch, size_t header_bytes, const ClusterCaps& caps, int side, u32 kept,
                           u32 depth, u64* rows, u32* origin, cudaStream_t s) {
  if (!kept) return;
  const uint8_t* region = static_cast<const uint8_t*>(scratch) + header_bytes;
  const u32 blocks = (kept + 255) / 256;
  switch (W) {
    case 1: k_cluster_export<1><<<blocks, 256, 0, s>>>(region, caps, side, kept, depth, rows, origin); break;
    case 2: k_cluster_export<2><<<blocks, 256, 0, s>>>(region, caps, side, kept, depth, rows, origin); break;
    case 3: k_cluster_export<3><<<blocks, 256, 0, s>>>(region, caps, side, kept, depth, rows, origin); break;
    case 4: k_cluster_export<4><<<blocks, 256, 0, s>>>(region, caps, side, kept, depth, rows, origin); break;
    default: throw std::runtime_error("cluster export: unsupported width");
  }
  SW_LAUNCH_CHECK();
}

}  // namespace sw
