// Device parts of the reference's small algorithms: the Eppstein greedy upper
// bound (pairs.cu) and the power-set BFS `Brute` (brute.cu).  Launchers are
// asynchronous on the given stream; scratch comes from the caller.
#pragma once
#include "common.cuh"
#include "kernels.cuh"

namespace sw {

// ---- Eppstein (synchrolib/algorithm/eppstein/eppstein.hpp:82-114 over the
// pairs tree of synchrolib/data_structures/pairs_tree.hpp:25-62) ----------

// Result words written by launch_eppstein into `out` (u32[8]).
enum EppsteinStatus : u32 {
  kEppFound = 0,       // out[1..2] = length (lo, hi), out[3] = letters written
  kEppOverBound = 1,   // the greedy word grew past `upper` (eppstein.hpp:104-106)
  kEppNonSynchro = 2,  // some pair never reaches the diagonal (pairs_tree.hpp:95-100)
  kEppWordCapacity = 3,
};

size_t eppstein_scratch_bytes(int n);

// One block: breadth-first pair tree (per pair {p, q} the length of the
// shortest word merging it and that word's first letter, the same first
// letter the reference's queue order records), then the greedy walk that
// repeatedly merges the closest pair of the current image.  Letters go to
// `word` (capacity `word_cap`).
void launch_eppstein(const TransTables& t, u64 upper, void* scratch, u32* out, uint8_t* word, u64 word_cap,
                     cudaStream_t s);

// ---- Brute (synchrolib/algorithm/brute/brute.hpp:88-122), n <= 32 --------

// Bitmap of visited subsets: 2^n bits.
size_t brute_visited_bytes(int n);

// One BFS level: every image of every frontier mask under every letter that
// was not visited yet is marked and appended to `next` (next_count[0] counts,
// capped at next_cap: the excess is counted but not stored).  found[0] = 1 and
// found[1] = the mask when a singleton is produced.
void launch_brute_level(const uint16_t* delta, int n, int k, const u32* frontier, u32 count, u32* visited,
                        u32* next, u32 next_cap, u32* next_count, u32* found, cudaStream_t s);

// Word back-tracking: best[0] = min over (i, a) with image(level[i], a) ==
// target of i * k + a (caller initialises best[0] to ~0).
void launch_brute_parent(const uint16_t* delta, int n, int k, const u32* level, u32 count, u32 target, u64* best,
                         cudaStream_t s);

// ---- Beam in one CTA (beam.cu) -------------------------------------------

// Levels per launch, and the words of `out`: found, levels expanded, sets kept,
// ancestor; kBeamLevels letters; kBeamLevels parent counts.
constexpr u32 kBeamLevels = 256, kBeamHeader = 8, kBeamOutWords = kBeamHeader + 2 * kBeamLevels;
constexpr size_t kBeamSmemBytes = 226 * 1024;
// Whether `parents` sets (the larger of the beam and the seeds) and their
// children fit.
bool beam_fits(int W, u32 n, u32 k, u64 parents);
// Up to `levels` (<= kBeamLevels) levels from the m sets in `rows` (room for
// `parents`; after a launch that found nothing it holds the kept sets), each
// kept set's letter * m + parent position in log[level * parents + position].
void launch_beam(int W, const uint16_t* delta, u32 n, u32 k, u32 beam, u32 m, u32 parents, u32 levels, u64* rows,
                 u32* log, u32* out, cudaStream_t s);

// ---- Device-resident exact search (batch_cluster.cu) ----------------------

// One automaton of a batch: n <= 64 W states; delta[q*k + a]
// (u8) at delta_off of the delta pool, its backward seeds (ascending) at
// seed_off of the seed pool; lengths 1..max_len are searched.
struct SmallInstance {
  u32 n, k, delta_off, seed_off, seed_count, max_len;
};
// status: 0 solved, 1 over a capacity, 2 no meeting within max_len.
// why (status 1): bits 0-7 the capacity (1 children, 2 layer, 3 visited,
// 4 depth, 5 word buffer), bits 8+ the layers searched when it stopped.
struct SmallResult {
  u32 status, length, word_len, why;
};

// Device-resident search on thread-block clusters (batch_cluster.cu): one
// cluster of `cs` CTAs per automaton (n <= 256, n * k <= 4096), lists in a
// per-cluster global region.  Status 1 may also report why 6 (a hash-table probe ran out) or 7 (given up), status 2 why 8
// (a side died out) or 9 (max_len reached), and status 3 says that the search
// stopped at a work limit; where no word was found, `length` counts the
// lengths excluded so far.
struct ClusterCaps {
  u32 vis = 0;        // row slots per side (one per child ever expanded on that side)
  u32 ch = 0;         // children of one step
  u32 vtab_bits = 0;  // log2 slots of a side's hash table (at least 4/3 of vis)
};
// Work limits of a launch: a search stops before a level of more than
// max_children children, after a level of more than max_pairs meet pairs, and
// once its lists and the next level pass a quarter of `budget` bytes by the
// streamed search's count (which then changes its reductions).
constexpr u32 kClusterPoll = 4;
struct ClusterLimits {
  u64 max_pairs = ~0ull;
  u64 budget = ~0ull;
  u32 max_children = ~0u;
  u32 counter_ready = 0;    // the caller zeroed the counter on the launch's stream
  size_t header_bytes = 0;  // bytes before the first region; 0: room for every cluster index
  // Word in pinned host memory (may be null) that the host sets to have the search
  // given up at one of its next kClusterPoll levels (status 1, why 7).
  const u32* cancel = nullptr;
};
// How a single search ended (written at kClusterExitOffset of its scratch):
// meet pairs, children and meet queries (backward rows, summed over levels),
// then per side (forward, backward) depth, kept rows and current layer size.
struct ClusterExit {
  u64 pairs, children, queries;
  u32 depth[2], kept[2], cnt[2];
};
constexpr size_t kClusterExitOffset = 256 + 32;
// Scratch of a single search: tag counter, control block, its SmallResult, its
// word (up to kClusterSingleWord letters); then the region.
constexpr size_t kClusterSingleResult = 512, kClusterSingleWords = 576, kClusterSingleHeader = 2048;
constexpr u32 kClusterSingleWord = 1024;
ClusterCaps cluster_default_caps();
ClusterCaps cluster_single_caps();
ClusterCaps cluster_tiny_caps();
// Bytes of scratch for `clusters` clusters.  It must be zero-filled before its
// first launch, and again before the tags the launches take from its counter
// (cluster_tags_per_launch) could pass kClusterTagLimit.
size_t cluster_scratch_bytes(u32 clusters, const ClusterCaps& c);
size_t cluster_single_scratch_bytes(const ClusterCaps& c);
u32 cluster_max_clusters_supported();
// Clusters of `cs` CTAs that fit on the current device at once.
u32 cluster_batch_max_clusters(int W, int cs);
// Tags a launch of `count` automata can take: one per search and one per
// cluster that finds the batch done.
constexpr u64 cluster_tags_per_launch(u32 count) { return (u64)count + 512; }
constexpr u64 kClusterTagLimit = 1ull << 26;
void launch_cluster_batch(int W, int cs, u32 clusters, const SmallInstance* inst, u32 count,
                          const uint8_t* delta_pool, const uint8_t* seed_pool, SmallResult* results, uint8_t* words,
                          u32 word_stride, void* scratch, const ClusterCaps& caps, const ClusterLimits& limits,
                          u32* counter, u64* stats, cudaStream_t s);
// Kept rows of one side (0 forward, 1 backward complements) of a search that
// stopped, layer after layer, and each row's origin (letter * parents +
// parent position; a seed's entry is its seed index).
// The layer table a search left (host copy of it: kClusterMetaWords words from
// cluster_meta_offset): per side the first row slot, the first list entry and
// the row count of every layer, each kClusterMetaStride words.
constexpr size_t kClusterMetaStride = 1025, kClusterMetaWords = 6 * kClusterMetaStride;
size_t cluster_meta_offset(int W, size_t header_bytes, const ClusterCaps& c);
void launch_cluster_export(int W, const void* scratch, size_t header_bytes, const ClusterCaps& caps, int side, u32 kept,
                           u32 depth, u64* rows, u32* origin, cudaStream_t s);

}  // namespace sw
