// Launchers for the device kernels of the exact search (kernels.cu).
//
// Every launcher is asynchronous on the given stream; scratch buffers come
// from the caller (no allocation inside).  Kernel roles and the reference
// functions they replace:
//   expand        PreprocessedTransition::apply
//                 (synchrolib/data_structures/preprocessed_transitions.cpp:56-93,
//                  cuda/preprocessed_transition_kernel.cu:19-88)
//   radix sort +  sort_keep_unique (synchrolib/utils/vector.hpp:13-27)
//   unique
//   subset check  SubsetsImplicitTrie::check_contains_subset / reduce
//   (subset_      (synchrolib/data_structures/subsets_implicit_trie.hpp:29-266,
//   check.cu)      cuda/subsets_implicit_trie_kernel.cu:13-92) and
//                 SubsetsTrie::contains_subset_of (subsets_trie.hpp:78-90)
#pragma once
#include "common.cuh"

namespace sw {

// Per-letter transition tables as staged into shared memory by `expand`.
// Layout (all u16): delta[a*n + q]; inv_beg[a*(n+1) + t] ..inv_beg[..+1] index
// inv_src[a*n + e] (CSR of preimages).
// Counts that only the device knows yet: a launcher's `live` pointers (null: the
// host's count holds) name the word that holds how many of a list's first m rows
// there are; grids and scratch are sized for m.
#ifdef __CUDACC__
__device__ __forceinline__ u32 live_count(u32 m, const u32* live) { return live ? min(m, *live) : m; }
#endif

struct TransTables {
  const uint16_t* delta = nullptr;   // k*n
  const uint16_t* inv_beg = nullptr; // k*(n+1)
  const uint16_t* inv_src = nullptr; // k*n
  int n = 0, k = 0;
};

// Sort key of a side: the 64 states whose pattern leads the key (identity =
// states 0..63, i.e. word 0 of the row).
struct KeyMap {
  uint16_t q[64];
  int identity = 1;
};

// out[(a*m + i)] = image (kImage) or preimage of in[i] under letter a.  With
// keys (and vals) given, each child o = a*m + i also gets its layer key
// keys[2o..2o+1] (as launch_layer_keys with `map`) and vals[o] = o.
void launch_expand(int W, bool image, const u64* in, u32 m, const TransTables& t, u64* out, cudaStream_t s,
                   u64* keys = nullptr, u32* vals = nullptr, const KeyMap& map = KeyMap{});

// Duplicate removal by hash table and bucket order (kernels.cu).  A layer is
// expanded into C (child a*m + i) and what is new — no row of V[0, base) that
// the table holds, no other child of this layer — is ranked within its bucket,
// the leading `bits` bits of word 0; launch_bucket_scatter then moves the kept
// rows to out_rows (bucket order), their child indices to out_vals, and points
// their slots at rows base .. of V (tab given; V + base * W is then out_rows).
// Table: tmask + 1 slots of u64, zero = empty, more slots than rows; *err is
// set to 3 if a probe runs out.  counts: 2^bits words, zero before the first
// launch (the scatter clears them); first: 2^bits words; place: one entry per
// child.
struct BucketScratch {
  int bits = 12;
  u32* counts = nullptr;
  u32* first = nullptr;
  uint2* place = nullptr;
  void* scan = nullptr;  // launch_scan's scratch, above kBucketBitsLarge
  u32* met = nullptr;  // two words, the first zero before the first launch; the second gets the children found in V
};
// Leading bits by the layer's children: up to 4096 buckets take one round of the
// bucket scan; above 2^20 children 16 bits leave tiles of the subset check and the
// dominance checks with few shared states, and the checks, which grow with the
// square, cost more than any scan (launch_scan's three launches).  Sums of searches
// in ms by bits above 2^20 children, 16 / 20 / 22 / 24 (sorted lists): plain Exact n = 200
// 31 / 31 / 31 / 31 (84), n = 280 1572 / 909 / 735 / 629 (760), n = 320 381 / 256 / 227 / 211
// (505); Beam + Exact n = 340 7125 / 4268 / 3882 / 3646 (7821), n = 384 14040 / 8715 /
// 7476 / 6740 (10882).  22 below 2^22 children keeps the counts small against the rows.
constexpr int kBucketBitsSmall = 12, kBucketBitsLarge = 16, kBucketBitsHuge = 22, kBucketBitsMost = 24;
inline int bucket_bits(u64 children) {
  if (children < (1u << 16)) return kBucketBitsSmall;
  if (children < (1u << 20)) return kBucketBitsLarge;
  return children < (1u << 22) ? kBucketBitsHuge : kBucketBitsMost;
}
void launch_expand_hash(int W, bool image, const u64* in, u32 m, const TransTables& t, u64* C, const u64* V, u32 base,
                        u64* tab, u32 tmask, const BucketScratch& b, u32* err, cudaStream_t s);
// Ranks m rows that are all kept.
void launch_bucket_rank(int W, const u64* C, u32 m, const BucketScratch& b, cudaStream_t s);
void launch_bucket_scatter(int W, const u64* C, u32 m, const BucketScratch& b, u32 base, u64* out_rows, u32* out_vals,
                           u64* tab, u32* total, cudaStream_t s);
// Enters rows [0, m) of V in a zeroed table.
void launch_hash_build(int W, const u64* V, u32 m, u64* tab, u32 tmask, u32* err, cudaStream_t s);

// Scratch sizing for the sort / scan helpers.
size_t scan_temp_bytes(u32 n);
size_t sort_temp_bytes(int R, u32 m);

// Exclusive prefix sum of in[0..n) into out; *total_dev receives the sum.
void launch_scan(const u32* in, u32* out, u32 n, u32* total_dev, void* temp, cudaStream_t s);

// Stable sort of m rows of R words (word 0 most significant) with a u32
// payload.  Result lands in (keys, vals); (keys_alt, vals_alt) are scratch of
// the same size.  Up to 2^20 rows: 2048-row chunks sorted in shared memory,
// then pairwise merges; beyond: LSD radix passes over 8-bit digits, digits
// constant over all rows skipped.  Returns the number of kernels launched;
// *data_passes (optional) = full read+write passes over the rows.
int radix_sort_rows(int R, u64* keys, u32* vals, u64* keys_alt, u32* vals_alt, u32 m, void* temp,
                     cudaStream_t s, int* data_passes = nullptr);

// flags[i] = 1 if row i differs from row i-1 (rows sorted).
void launch_unique_flags(int W, const u64* rows, u32 m, u32* flags, cudaStream_t s);

// Stream compaction of rows (+ optional payload) by flags; pos = exclusive scan of flags.
void launch_compact(int W, const u64* rows, const u32* vals, const u32* flags, const u32* pos, u32 m, u64* out_rows,
                    u32* out_vals, cudaStream_t s);

enum QueryMode : int {
  kQuerySubset = 0,        // hit(c) = exists s in S, s ⊆ c
  kQueryProperSubset = 1,  // hit(c) = exists s in S, s ⊊ c
  kQueryDisjoint = 2,      // hit(c) = exists s in S, s ∩ c = ∅  (s ⊆ ~c)
};

// Tiled subset check (subset_check.cu): for each query row c, flags[c] |=
// hit(c) (or, with `stop`, record one witness pair and let all warps exit
// early: witness[0] = found flag, witness[1] = query index, witness[2] = set
// index).  S is cut into tiles of sh.tile_rows rows and super-tiles of
// sh.tiles_per_super tiles; `masks` (subset_check_temp_bytes) and *size_floor
// (zero beforehand) come from launch_tile_and with the same shape.  `flags`
// must start zeroed (non-stop mode).  `items` (subset_check_items entries) and
// item_counts (kSubsetCounterWords words) list the parts of S that a large check's queries need; without them
// (nullptr) it goes over all of S.  `bytes_ctr` (optional) accumulates the
// bytes of S rows tested.
constexpr u64 kSubsetItems = 1u << 22;
constexpr u32 kSubsetQueues = 64, kSubsetCounterWords = 32 * (kSubsetQueues + 1);  // counters a cache line apart
// Launch shape of the subset check: rows of S per tile mask (32, 64, 128),
// warps of 32 queries per block (4, 8, 16), tiles per super-tile mask (4, 8,
// 16, 32) and the grid's target blocks per SM (1..64), which sets how finely
// S is chunked over blockIdx.y.  Results do not depend on it.
struct ScanShape {
  int tile_rows = 64;
  int warps = 8;
  int tiles_per_super = 16;
  int grid_factor = 16;
};
// Shapes per row width W (1..8) and list size class: class 0 for lists S of
// fewer than kScanLargeRows rows, class 1 for larger ones.
constexpr int kScanSizeClasses = 2;
constexpr u32 kScanLargeRows = 1u << 15;
constexpr size_t kMaxScanSmem = 200 * 1024;
struct ScanShapes {
  ScanShape s[8][kScanSizeClasses];
  const ScanShape& pick(int W, u32 m) const { return s[W - 1][m >= kScanLargeRows ? 1 : 0]; }
};
bool scan_shape_valid(int W, const ScanShape& sh);
size_t scan_smem_bytes(int W, const ScanShape& sh);
size_t subset_check_temp_bytes(int W, u32 m, const ScanShape& sh);
// Entries of `items` that a check of q queries against m rows can use.
u64 subset_check_items(u32 m, u32 q, const ScanShape& sh);
void launch_tile_and(int W, const u64* S, u32 m, u64* masks, u32* size_floor, const ScanShape& sh, cudaStream_t s,
                     const u32* m_live = nullptr);
void launch_subset_check(int W, int mode, const u64* S, u32 m, const u64* masks, const u32* size_floor, const u64* Q,
                         u32 q, int n, u32* flags, u32* witness, bool stop, const ScanShape& sh, cudaStream_t s,
                         u64* bytes_ctr, uint2* items, u32* item_counts, const u32* m_live = nullptr,
                         const u32* q_live = nullptr);

// Dominance (dominance.cu): with hit_t, flags[t] = 1 for every row t of T that
// holds some row x of X (x ⊆ t; proper: x ⊊ t), else flags[x] = 1 for every x that
// some t holds.  comp: rows are complements of the sets meant.  Rows whose flag
// is set already are left out.  T up to kDomSmallRows rows is cut into 1024-row
// chunks (a level of 5 000 against 4 000 sets: 16 us), above into chunks of 4096
// (2048 at seven words a row and more), which cost a quarter of the instructions
// a pair; above kDomOrderRows its rows are first ordered by falling size (three
// launches), so that most sets are too large for most chunks, and only then is the
// scratch used.
constexpr u32 kDomSmallRows = 1u << 13, kDomOrderRows = 1u << 15;
struct DominanceScratch {
  BucketScratch bucket;   // as for launch_bucket_scatter, with room for T's rows
  u64* rows = nullptr;    // T's rows again
  u32* index = nullptr;   // one word per row of T
  u32* total = nullptr;   // one word
};
void launch_bucket_scan(const BucketScratch& b, u32* total, cudaStream_t s);
void launch_dominance(int W, bool comp, bool hit_t, const u64* T, u32 tm, const u64* X, u32 xm, int n, bool proper,
                      u32* flags, const DominanceScratch& sc, cudaStream_t s, const u32* t_live = nullptr,
                      const u32* x_live = nullptr);

// In-place conversion of `count` rows between the reference bit layout (state
// q = bit q % 64 of word q / 64) and the device layout (bit 63 - q % 64); bits
// of states >= n come out zero.
void launch_convert_rows(int W, u64* rows, u64 count, int n, bool to_device, cudaStream_t s);

// out[i] = popcount of row i.
// sum[0..W) |= every row; ~(index of the first single-state row) is maxed into
// *single (zero: none).  The caller zeroes both.
void launch_list_summary(int W, const u64* rows, u32 m, u64* sum, u32* single, cudaStream_t s,
                         const u32* live = nullptr);
// Row i of `out` (Wo words) holds state t where row i of `in` (Wi words) holds
// state src[t], for t < n.
void launch_relabel_rows(const u64* in, int Wi, u32 m, const uint16_t* src, int n, u64* out, int Wo, cudaStream_t s);
void launch_popcount(int W, const u64* rows, u32 m, u32* out, cudaStream_t s);

// flags[i] = AND/OR combine: out[i] = (a[i] == 0 && b[i] == 0).
void launch_keep_flags(const u32* a, const u32* b, u32 m, u32* out, cudaStream_t s);

// Layer keys keys[2i..2i+1] = (the map's 64 states of row i packed MSB-first,
// 32-bit mix of the row in the high half): sort order of a layer and of the
// visited list of one side.
void launch_layer_keys(int W, const u64* rows, u32 m, u64* keys, cudaStream_t s, const KeyMap& map = KeyMap{});
// Merge of two row arrays sorted by the same layer key.
void launch_merge_key(int W, const u64* A, u32 na, const u64* B, u32 nb, u64* out, cudaStream_t s,
                      const KeyMap& map = KeyMap{});
// flags[i] = 1 if row i of C equals a row of V (flags untouched otherwise);
// V and C sorted by the same layer key.
// Duplicate removal of a key-sorted layer and compaction in one launch
// (decoupled look-back over tiles): child vals[i] of C is kept when it
// differs from child vals[i-1] and equals no row of the key-sorted visited
// list V (keys = the children's sorted layer keys); out_rows / out_vals
// receive the kept children in sort order, *total their count.  `status`
// holds dedup_compact_status_words(m) words (zero-filled when first
// allocated), `ctr` one word that is zero before the first launch (each
// launch leaves it zero); `epoch` is 1..2^30-1 and must differ from the
// previous launch's on the same status array.  *err is set to 2 if a bounded
// wait ran out.
size_t dedup_compact_status_words(u32 m);
void launch_dedup_compact(int W, const u64* C, const u32* vals, const u64* keys, u32 m, const u64* V, u32 nv,
                          const KeyMap& map, u64* out_rows, u32* out_vals, u32* total, u64* status, u32* ctr,
                          u32 epoch, u32* err, cudaStream_t s);
// The rows whose flag is zero, in order, and their vals: one launch, compacted as
// by launch_dedup_compact (same status, ctr and epoch).
void launch_keep_compact(int W, const u64* rows, const u32* vals, const u32* flags, u32 m, u64* out_rows, u32* out_vals,
                         u32* total, u64* status, u32* ctr, u32 epoch, u32* err, cudaStream_t s, const u32* live = nullptr);
// counts[q] += rows containing state q (counts: 64*W entries, caller-zeroed).
void launch_state_counts(int W, const u64* rows, u32 m, u32* counts, cudaStream_t s);

// p[i] = i.
void launch_iota(u32* p, u32 m, cudaStream_t s);

// dst[i] = src[idx[i]] (rows of W words).
void launch_gather_rows(int W, const u64* src, const u32* idx, u32 m, u64* dst, cudaStream_t s);

// Beam sort keys: keys[i] = [n - |row i|, bit-reversed words of row i] (R words).
void launch_beam_keys(int W, const u64* rows, u32 m, int n, int R, u64* keys, cudaStream_t s);

// dst[i] = src[idx[i]] (u32 payloads).
void launch_gather_u32(const u32* src, const u32* idx, u32 m, u32* dst, cudaStream_t s);

// Ascending sort keys of beam candidates: keys[i] = primary << 32 | i with
// primary = the order-preserving bits of score[i] (counts null), counts[i]
// (score null), or counts[i] << 16 | leading 16 bits of score[i] (both).
void launch_score_keys(const float* score, const u32* counts, u32 m, u64* keys, cudaStream_t s);
// sel[0 .. width) = positions, ascending, of the `width` rows with the smallest
// score keys (upper halves; ties by layer key); 0 < width <= m <= kSelectMax.
constexpr u32 kSelectMax = 1u << 14;
void launch_select(int W, const u64* keys, u32 m, u32 width, const u64* rows, u32* sel, cudaStream_t s);

// Walks a word back: step i reads o = steps[i].origin[idx], emits the letter
// out[i] = o / parents and goes on at idx = o % parents; out[count] = the last idx.
struct TraceStep {
  const u32* origin;
  u32 parents;
};
void launch_trace(const TraceStep* steps, u32 count, u32 idx, u32* out, cudaStream_t s);

// Fill u32 array with a value.
void launch_fill_u32(u32* p, u32 value, u32 m, cudaStream_t s);

}  // namespace sw
