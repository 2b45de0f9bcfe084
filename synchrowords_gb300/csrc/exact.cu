// Host driver of the GPU exact search and beam (see exact.hpp).
//
// Exact (synchrolib/algorithm/exact/exact.cpp:37-97, meet_in_the_middle.cpp:58-344):
// two frontiers live on the device,
//   F: forward images  delta(Q, w), seeded with {Q}           (exact.cpp:130-146)
//   B: inverse preimages, seeded with sink singletons whose
//      state has some letter of in-degree > 1                (exact.cpp:149-164)
// B is stored as complements: the preimage of a complement is the complement
// of the preimage, so the same expansion, dedup and dominance code serves both
// sides.  One step expands the smaller side (meet_in_the_middle.cpp:355-358),
// drops duplicates by hash table (or by sorting, past its limits), drops where it
// pays every child that has a visited set inside it or a proper subset in its own
// layer (meet_in_the_middle.cpp:179-344 on complements for B), and then asks
// whether some F is disjoint from some B-complement (F ⊆ B,
// meet_in_the_middle.cpp:90).  Each kept child records (letter, parent) so the
// meeting pair yields a word, which is verified on the host before it is
// returned.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <stdexcept>
#include <string>

#include "algos.cuh"
#include "exact.hpp"
#include "kernels.cuh"
#include "learn.hpp"
#include "search_rules.hpp"
#include "train.hpp"

namespace sw {

namespace {

struct Layer {
  DevBuf origin;        // per kept set: child position a*parent_count + parent
  const u32* view = nullptr;  // the same, in a buffer this layer shares with others (then `origin` is unused)
  const u32* org() const { return view ? view : origin.as<u32>(); }
  u32 count = 0;
  u32 parent_count = 0;
};

struct Side {
  DevBuf rows, rows_alt;
  u32 count = 0;
  DevBuf vis, vis_alt;
  u32 vis_count = 0;
  // Hashed sides (Engine::step_hashed) append each layer to the visited list,
  // whose tail the current layer then is (in_vis; else it is `rows`), and keep a
  // hash table of every distinct row met.  Its slots name rows of vis until a
  // reduction drops one; from then on (split) they name rows of `met`, which
  // keeps the dropped ones too.
  bool hashed = false, sorted_only = false, in_vis = false, split = false;
  u32 cur_off = 0;  // first row of the current layer in vis
  DevBuf table, met;
  u32 met_count = 0;    // rows of met (split)
  u64 table_slots = 0;  // 0: to be built
  // The last hashed step, and where its layer's count is while only the device
  // knows it (count is then an upper bound).
  struct Step {
    u32 parents = 0, children = 0, base = 0, visited = 0, distinct = 0, kept = 0;
    bool forward = false, reduce = false, compacted = false, deferred = false, counted = false;
    double t0 = 0;
  } step;
  const u32* live = nullptr;
  size_t list_bytes() const { return vis.cap + vis_alt.cap + met.cap + table.cap; }
  const u64* cur_rows(int W) const { return in_vis ? vis.as<u64>() + (size_t)cur_off * W : rows.as<u64>(); }
  std::vector<std::unique_ptr<Layer>> layers;
  double unique_growth = 0;      // distinct children per parent at the last step
  KeyMap keymap;                 // sort key of this side's layers and visited list
  bool keymap_chosen = false;
  // Layers of earlier solves, kept with their device buffers, so that a
  // solve's layers reuse them instead of allocating: a new layer takes the
  // spare whose origin buffer holds `origin_bytes` with the least room to
  // spare, else the largest (which then grows).
  std::vector<std::unique_ptr<Layer>> spare;
  std::unique_ptr<Layer> new_layer(size_t origin_bytes) {
    if (spare.empty()) return std::make_unique<Layer>();
    size_t best = 0;
    for (size_t i = 1; i < spare.size(); ++i) {
      const size_t c = spare[i]->origin.cap, cb = spare[best]->origin.cap;
      const bool fits = c >= origin_bytes, best_fits = cb >= origin_bytes;
      if (fits ? (!best_fits || c < cb) : (!best_fits && c > cb)) best = i;
    }
    std::unique_ptr<Layer> L = std::move(spare[best]);
    spare[best] = std::move(spare.back());
    spare.pop_back();
    L->count = L->parent_count = 0;
    L->view = nullptr;
    return L;
  }
  void reset() {
    count = vis_count = 0;
    hashed = sorted_only = in_vis = split = false;
    live = nullptr;
    table_slots = 0;
    unique_growth = 0;
    keymap = KeyMap{};
    keymap_chosen = false;
    for (auto& L : layers) spare.push_back(std::move(L));
    layers.clear();
  }
};

// Where a search leaves the single cluster it starts on (Engine::run_single).
// CTAs of that cluster, and the children and meet pairs of a level above which
// the level goes to the whole GPU.  Four solves at n = 200 in ms, by children
// (pairs = children^2 / 4): 2^11 15.1, 2^12 15.1, 2^13 14.8, 2^14 15.3; with 4
// CTAs and 2^13 15.4, with 16 (a size not every GPU part can place) 14.5.
constexpr int kSingleClusterCtas = 8;
constexpr u32 kSingleMaxChildren = 1u << 13;
constexpr u64 kSingleMaxPairs = 1ull << 24;

// One level of the bounded inverse phase (a chunk of parents' children).
struct DLevel {
  DevBuf rows, origin;
  u32 count = 0;
  u32 chunk_off = 0, chunk_cnt = 0;  // parent slice this level was expanded from
};

}  // namespace

class Engine {
 public:
  explicit Engine(int device) {
    SW_CUDA(cudaSetDevice(device));
    SW_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    pinned.reserve(4096);
    SW_CUDA(cudaMalloc(&d_misc, 64 * sizeof(u32)));
    SW_CUDA(cudaMemset(d_misc, 0, 64 * sizeof(u32)));
    mlp = std::make_unique<MlpRunner>(stream, d_misc + kScanErrWord);
  }
  ~Engine() {
    for (auto e : ev_pool) cudaEventDestroy(e);
    for (auto* p : {&reduce_span, &meet_span})
      for (auto e : p->ev)
        if (e) cudaEventDestroy(e);
    if (d_query_bytes) cudaFree(d_query_bytes);
    if (d_misc) cudaFree(d_misc);
    if (stream) cudaStreamDestroy(stream);
  }

  cudaStream_t stream = nullptr;
  HostPinned pinned;
  std::unique_ptr<MlpRunner> mlp;
  std::unique_ptr<Trainer> trainer;  // of the first training call; its buffers are kept

  // ---- optional per-kernel-class timing (CUDA events on `stream`) ----
  // class 0: subset-query tree walks, 1: layer expansion, 2: radix sorts,
  // 3: everything else (unique/compaction/tree build/merge).
  struct ProfClass {
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev;
    u64 launches = 0;
    double bytes = 0;
  };
  bool prof_on = false;
  ProfClass prof[4];
  std::vector<cudaEvent_t> ev_pool;
  size_t ev_next = 0;
  u64* d_query_bytes = nullptr;
  cudaEvent_t next_event() {
    if (ev_next == ev_pool.size()) {
      cudaEvent_t e;
      SW_CUDA(cudaEventCreate(&e));
      ev_pool.push_back(e);
    }
    return ev_pool[ev_next++];
  }
  template <class Fn>
  void timed(int cls, double bytes, Fn&& fn) {
    if (!prof_on) {
      fn();
      return;
    }
    cudaEvent_t a = next_event(), b = next_event();
    SW_CUDA(cudaEventRecord(a, stream));
    fn();
    SW_CUDA(cudaEventRecord(b, stream));
    prof[cls].ev.emplace_back(a, b);
    prof[cls].launches++;
    prof[cls].bytes += bytes;
  }
  void profile_begin() {
    if (!d_query_bytes) SW_CUDA(cudaMalloc(&d_query_bytes, sizeof(u64)));
    SW_CUDA(cudaMemsetAsync(d_query_bytes, 0, sizeof(u64), stream));
    for (auto& c : prof) c = ProfClass{};
    scan_ev.clear();
    ev_next = 0;
    prof_on = true;
  }
  void profile_end(sw_kernel_profile out[4]) {
    SW_CUDA(cudaStreamSynchronize(stream));
    u64 qb = 0;
    SW_CUDA(cudaMemcpy(&qb, d_query_bytes, sizeof(u64), cudaMemcpyDeviceToHost));
    prof[0].bytes += (double)qb;
    for (int c = 0; c < 4; ++c) {
      double ms = 0;
      for (auto& pr : prof[c].ev) {
        float t = 0;
        SW_CUDA(cudaEventElapsedTime(&t, pr.first, pr.second));
        ms += t;
      }
      out[c].launches = prof[c].launches;
      out[c].ms = ms;
      out[c].bytes = prof[c].bytes;
    }
    for (int i = 0; i < 8 * kScanSizeClasses; ++i) {
      scan_ms[i] = 0;
      scan_launches[i] = 0;
    }
    for (auto& kv : scan_ev) {
      float t = 0;
      SW_CUDA(cudaEventElapsedTime(&t, kv.second.first, kv.second.second));
      scan_ms[kv.first] += t;
      scan_launches[kv.first]++;
    }
    prof_on = false;
  }
  u32* d_misc = nullptr;  // [0..2] witness, [3] the subset check's size floor, [6, 7] children met before, [8] scan total, [9] rows kept by the reductions, [kScanErrWord] bounded-wait timeouts
  static constexpr int kScanErrWord = 4;  // read back with the witness, never cleared by it
  // Throws, and clears the word, if a launch reported a bounded wait that ran out:
  // 2 = a compaction tile's look-back never saw its predecessor, 3 = a hash
  // table's probe found no slot, mlp::kErrorWait; `w` is the pinned copy of
  // d_misc[kScanErrWord].
  void check_scan_error(u32 w) {
    if (!w) return;
    SW_CUDA(cudaMemsetAsync(d_misc + kScanErrWord, 0, sizeof(u32), stream));
    if (w == mlp::kErrorWait) throw CudaError("distance model: a tensor-core wait ran out");
    if (w == 2) throw CudaError("layer compaction: a look-back wait ran out");
    if (w == 3) throw CudaError("duplicate removal: a hash table ran out of slots");
    throw CudaError("a launch reported error " + std::to_string(w));
  }
  // Single-pass duplicate removal (launch_dedup_compact): its tile status
  // words (zero-filled when allocated), tile counter and launch epoch.
  DevBuf dc_status, dc_ctr;
  size_t dc_status_zeroed = 0;
  u32 dc_epoch = 0;
  u32 next_dc_epoch(u32 m) {
    const size_t words = dedup_compact_status_words(m);
    if (!dc_ctr.p) {
      dc_ctr.reserve(sizeof(u32));
      SW_CUDA(cudaMemsetAsync(dc_ctr.p, 0, sizeof(u32), stream));
    }
    if (++dc_epoch >= (1u << 30)) dc_epoch = 0;  // wrapped: every word back to "unpublished"
    if (dc_status.cap < sizeof(u64) * words || dc_epoch == 0) {
      dc_status.reserve(sizeof(u64) * std::max<size_t>(words, (size_t)1 << 16));
      SW_CUDA(cudaMemsetAsync(dc_status.p, 0, dc_status.cap, stream));
      if (dc_epoch == 0) dc_epoch = 1;
    }
    return dc_epoch;
  }
  // The compaction's count and the timeout word in one read-back.
  u32 read_total_checked() {
    SW_CUDA(cudaMemcpyAsync(pinned.p, d_misc + kScanErrWord, 5 * sizeof(u32), cudaMemcpyDeviceToHost, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    const u32* w = pinned.as<u32>();
    check_scan_error(w[0]);
    return w[8 - kScanErrWord];
  }
  // tables
  DevBuf t_delta, t_beg, t_src;
  TransTables tables;
  // scratch
  DevBuf ch_rows, ch_vals, alt_rows, alt_vals, uq_rows, uq_vals, new_vals;
  DevBuf epp_scratch, epp_word, br_visited, br_arena;
  DevBuf flags_a, flags_b, keep, pos, sort_tmp, scan_tmp, keys, keys_alt, sorted_rows;

  // Sort m rows in place by layer key (word 0, then a mix of the other words).
  void sort_by_layer_key(int W, u64* rows, u32 m, const KeyMap& map = KeyMap{}) {
    if (m < 2) return;
    keys.reserve(sizeof(u64) * 2 * m);
    ch_vals.reserve(sizeof(u32) * m);
    sorted_rows.reserve(sizeof(u64) * W * m);
    launch_layer_keys(W, rows, m, keys.as<u64>(), stream, map);
    launch_iota(ch_vals.as<u32>(), m, stream);
    sort_rows(2, keys.as<u64>(), ch_vals.as<u32>(), m);
    launch_gather_rows(W, rows, ch_vals.as<u32>(), m, sorted_rows.as<u64>(), stream);
    SW_CUDA(cudaMemcpyAsync(rows, sorted_rows.p, sizeof(u64) * W * m, cudaMemcpyDeviceToDevice, stream));
    count_launch(4);
  }
  Side F, B;
  Side R;  // the list of the last Reduce, from which a search of the reduced automaton starts
  // Where the running call counts; the caller's record, so only for that long.
  sw_stats* st = nullptr;
  struct Counting {
    Engine& E;
    Counting(Engine& e, sw_stats& st) : E(e) { E.st = &st; }
    ~Counting() {
      E.st = nullptr;
      E.list_budget = ~(size_t)0;
      E.states_ordered = false;
    }
  };
  std::vector<std::unique_ptr<DLevel>> dlevel_pool;  // the bounded phase's per-depth levels
  // scratch of the beams and of Reduce, kept across calls
  DevBuf lb_counts, lb_scores, lb_keys, lb_vals, lb_alt_k, lb_alt_v, lb_sel_rows, lb_sel_origin, red_states;
  DevBuf beam_log, beam_out;

  void upload_tables(const Automaton& A) {
    HostTables h = build_tables(A);
    t_delta.reserve(h.delta.size() * 2);
    t_beg.reserve(h.inv_beg.size() * 2);
    t_src.reserve(h.inv_src.size() * 2);
    SW_CUDA(cudaMemcpyAsync(t_delta.p, h.delta.data(), h.delta.size() * 2, cudaMemcpyHostToDevice, stream));
    SW_CUDA(cudaMemcpyAsync(t_beg.p, h.inv_beg.data(), h.inv_beg.size() * 2, cudaMemcpyHostToDevice, stream));
    SW_CUDA(cudaMemcpyAsync(t_src.p, h.inv_src.data(), h.inv_src.size() * 2, cudaMemcpyHostToDevice, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    tables.delta = t_delta.as<uint16_t>();
    tables.inv_beg = t_beg.as<uint16_t>();
    tables.inv_src = t_src.as<uint16_t>();
    tables.n = (int)A.n;
    tables.k = (int)A.k;
  }

  u32 read_u32(const u32* dptr) {
    SW_CUDA(cudaMemcpyAsync(pinned.p, dptr, sizeof(u32), cudaMemcpyDeviceToHost, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    return *pinned.as<u32>();
  }

  void count_launch(u64 c = 1) {
    if (st) st->kernel_launches += c;
  }

  // Compact rows/vals by flags; returns kept count.
  u32 compact(int W, const u64* rows, const u32* vals, const u32* flags, u32 m, u64* out_rows, u32* out_vals) {
    pos.reserve(sizeof(u32) * (size_t)m);
    scan_tmp.reserve(scan_temp_bytes(m));
    u32* total = d_misc + 8;
    timed(3, (double)m * (4 + 4 + 4 + 8.0 * W + 4), [&] {
      launch_scan(flags, pos.as<u32>(), m, total, scan_tmp.p, stream);
      launch_compact(W, rows, vals, flags, pos.as<u32>(), m, out_rows, out_vals, stream);
    });
    count_launch(4);
    return read_u32(total);
  }

  void sort_rows(int R, u64* rows, u32* vals, u32 m) {
    alt_rows.reserve(sizeof(u64) * R * (size_t)m);
    alt_vals.reserve(sizeof(u32) * (size_t)m);
    sort_tmp.reserve(sort_temp_bytes(R, m));
    int launches = 0, passes = 0;
    // algorithmic bytes: every pass reads and writes each (row, payload) once
    timed(2, 0.0, [&] {
      launches =
          radix_sort_rows(R, rows, vals, alt_rows.as<u64>(), alt_vals.as<u32>(), m, sort_tmp.p, stream, &passes);
    });
    if (prof_on) prof[2].bytes += (double)m * passes * 2.0 * (8.0 * R + 4);
    count_launch(launches);
  }

  // Subset queries run on the tiled check (subset_check.cu), in the launch
  // shape the context holds for the row width and the list's size class.
  DevBuf tile_and, scan_items;
  ScanShapes scan_shapes;
  // while profiling: events around each check's mask build + scan, keyed by
  // (W - 1) * kScanSizeClasses + size class
  std::vector<std::pair<int, std::pair<cudaEvent_t, cudaEvent_t>>> scan_ev;
  double scan_ms[8 * kScanSizeClasses] = {};
  u64 scan_launches[8 * kScanSizeClasses] = {};

  void query(int W, int mode, const u64* S, u32 m, const u64* Q, u32 q, int n, u32* flags, bool stop,
             const u32* m_live = nullptr, const u32* q_live = nullptr) {
    if (!m || !q) return;
    const ScanShape& sh = scan_shapes.pick(W, m);
    tile_and.reserve(subset_check_temp_bytes(W, m, sh));
    static_assert(kSubsetCounterWords % 2 == 0, "the list lies behind the counters");
    scan_items.reserve(sizeof(u32) * kSubsetCounterWords + sizeof(uint2) * subset_check_items(m, q, sh));
    cudaEvent_t e0 = nullptr;
    if (prof_on) {
      e0 = next_event();
      SW_CUDA(cudaEventRecord(e0, stream));
    }
    u32* const size_floor = d_misc + 3;  // zeroed with the witness in meet mode
    if (!stop) SW_CUDA(cudaMemsetAsync(size_floor, 0, sizeof(u32), stream));
    timed(3, (double)m * 8.0 * W, [&] { launch_tile_and(W, S, m, tile_and.as<u64>(), size_floor, sh, stream, m_live); });
    // algorithmic bytes: the query rows plus every row of S a query is tested against
    timed(0, (double)q * 8.0 * W, [&] {
      launch_subset_check(W, mode, S, m, tile_and.as<u64>(), size_floor, Q, q, n, flags, d_misc, stop, sh, stream,
                          prof_on ? d_query_bytes : nullptr,
                          reinterpret_cast<uint2*>(scan_items.as<u32>() + kSubsetCounterWords), scan_items.as<u32>(),
                          m_live, q_live);
    });
    if (prof_on) {
      cudaEvent_t e1 = next_event();
      SW_CUDA(cudaEventRecord(e1, stream));
      scan_ev.push_back({(W - 1) * kScanSizeClasses + (m >= kScanLargeRows ? 1 : 0), {e0, e1}});
    }
    count_launch(2);
    if (!m_live && !q_live) count_query(m, q);
  }
  void count_query(u32 m, u32 q) {
    if (!st) return;
    st->trie_queries += q;
    st->logical_pairs += (u64)m * q;
  }

  // flags[i] = 1 where a row of S (a proper one) is inside child row i of Q, on
  // the forward side or on complement rows; children flagged already are left out.
  // Forward, children are the rows that hold: large sets, which take many bitmaps
  // to rule out.  Above kMaskedChildren of them the tiled check's masks leave less
  // to test.  ms masked / bitmaps, S x children: n = 42 22K x 37K 0.12 / 0.15, 53K x
  // 89K 0.35 / 0.69, 1.1M x 1.1M 28 / 105; n = 60 random 59K x 59K 0.24 / 0.24, near-
  // permutations 0.39 / 0.63; n = 128 50K x 50K 0.21 / 0.21, 170K x 170K 0.66 / 1.1; n =
  // 300 50K x 50K 0.28 / 0.28, 1.1M x 1.1M 22 / 34.  Backward the bitmaps are
  // faster throughout (n = 42 283K 2.7 / 1.4, n = 300 280K 27 / 2.5).
  // That is with states ordered by how often images hold them, as in the exact
  // search.  In the caller's order (distance_pairs) the masks say less: from 2^18
  // children, and not among siblings once the layers shrink against the visited
  // list: n = 130 839K x 1228K 8.4 / 34, siblings 10 / 24, at the end 822K x 5851K 52 /
  // 109, siblings 26 / 18; n = 160 129K 0.5 / 0.9; n = 200 168K x 414K 3.5 / 1.9,
  // siblings 3.8 / 0.9.
  static constexpr u32 kMaskedChildren = 1u << 16, kMaskedChildrenOneWord = 1u << 15, kMaskedUnordered = 1u << 18;
  bool states_ordered = false;
  bool masked_check(bool forward, int W, u32 q, bool siblings, u32 visited) const {
    if (!forward) return false;
    if (states_ordered) return q > (W == 1 ? kMaskedChildrenOneWord : kMaskedChildren);
    return q > kMaskedUnordered && (!siblings || 2 * (u64)q > visited);
  }
  // Siblings (proper) are checked beside `visited` visited rows.  `order`: scratch
  // for the rows in the order the check takes them.
  DevBuf dom_rows, dom_index;
  void dominated(bool forward, int W, const u64* S, u32 m, const u64* Q, u32 q, int n, bool proper, u32 visited, u32* flags,
                 DevBuf& order, const u32* m_live = nullptr, const u32* q_live = nullptr) {
    if (!m || !q) return;
    if (masked_check(forward, W, q, proper, visited))
      return query(W, proper ? kQueryProperSubset : kQuerySubset, S, m, Q, q, n, flags, false, m_live, q_live);
    cudaEvent_t e0 = nullptr;
    if (prof_on) {
      e0 = next_event();
      SW_CUDA(cudaEventRecord(e0, stream));
    }
    DominanceScratch sc;
    const u32 tm = forward ? q : m;  // rows that hold: children forward, visited or siblings backward
    if (tm > kDomOrderRows) {
      sc.bucket = buckets(tm);
      sc.bucket.met = d_misc + 14;  // not the step's
      order.reserve(sizeof(u64) * W * (size_t)tm);
      dom_index.reserve(sizeof(u32) * (size_t)tm);
      sc.rows = order.as<u64>();
      sc.index = dom_index.as<u32>();
      sc.total = d_misc + 10;
      count_launch(3);
    }
    timed(0, (double)(m + q) * 8.0 * W, [&] {
      if (forward)  // sets s ⊆ c: the children hold them
        launch_dominance(W, false, true, Q, q, S, m, n, proper, flags, sc, stream, q_live, m_live);
      else  // complements: the set of c lies in the set of s
        launch_dominance(W, true, false, S, m, Q, q, n, proper, flags, sc, stream, m_live, q_live);
    });
    if (tm > kDomOrderRows) scanned();
    if (prof_on) {
      cudaEvent_t e1 = next_event();
      SW_CUDA(cudaEventRecord(e1, stream));
      scan_ev.push_back({(W - 1) * kScanSizeClasses + (m >= kScanLargeRows ? 1 : 0), {e0, e1}});
    }
    count_launch();
    if (!m_live && !q_live) count_query(m, q);
  }

  // Device time of a level's dominance checks and of its meet check.
  struct Span {
    cudaEvent_t ev[2] = {nullptr, nullptr};
    void mark(int i, cudaStream_t s) {
      if (!ev[i]) SW_CUDA(cudaEventCreate(&ev[i]));
      SW_CUDA(cudaEventRecord(ev[i], s));
    }
    double seconds() const {
      float ms = 0;
      SW_CUDA(cudaEventElapsedTime(&ms, ev[0], ev[1]));
      return 1e-3 * ms;
    }
  } reduce_span, meet_span;

  // Step log on stderr when SYNCHRO_VERBOSE is set (synchronises per phase).
  const bool verbose = std::getenv("SYNCHRO_VERBOSE") != nullptr;
  double vclock() {
    if (!verbose) return 0.0;
    SW_CUDA(cudaStreamSynchronize(stream));
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
  }

  // One BFS layer on side X (forward = image, backward = preimage of complements).
  // With `dominance` false only duplicates are removed and the visited list is
  // left alone (the bounded inverse phase, see Solver::exact).
  // Dominance reductions (the reference's self and visited reductions): drop
  // children that hold a visited set or a proper subset in their own layer.
  // Solver::exact runs them only where they pay: each removes ~15% of a layer for a
  // check of the layer, which repays itself when the lists are large or feed the
  // bounded phase.  Lengths are the same either way: every kept set is still a set
  // of its layer and the meet check is exact.
  bool reductions = true;

  // ---- duplicate removal by hash table ----
  DevBuf bk_counts, bk_first, bk_place, bk_scan, level_table;
  // Bucket counts are zero between steps: the scan that reads them clears them.
  // A step that ends before that scan (its buffers did not fit) leaves counts
  // behind, and the next step would move its rows past their list; so every use
  // starts with buckets(), which zeroes what such a step left, and ends with
  // scanned() once the scan is launched.
  bool bk_open = true;
  BucketScratch buckets(u64 children) {
    const int bits = bucket_bits(children);
    const size_t bytes = sizeof(u32) << std::max(bits, kBucketBitsLarge);
    if (bk_counts.cap < bytes) bk_open = true;
    bk_counts.reserve(bytes);
    bk_first.reserve(bytes);
    bk_place.reserve(sizeof(uint2) * children);
    bk_scan.reserve(scan_temp_bytes(1u << bits));
    if (bk_open) {
      SW_CUDA(cudaMemsetAsync(bk_counts.p, 0, bk_counts.cap, stream));
      SW_CUDA(cudaMemsetAsync(d_misc + 6, 0, 2 * sizeof(u32), stream));
      SW_CUDA(cudaMemsetAsync(d_misc + 14, 0, 2 * sizeof(u32), stream));
    }
    bk_open = true;
    return BucketScratch{bits, bk_counts.as<u32>(), bk_first.as<u32>(), bk_place.as<uint2>(), bk_scan.p, d_misc + 6};
  }
  void scanned() { bk_open = false; }
  // Power-of-two slots, two to four per row.
  static u64 slots_for(u64 rows) {
    u64 s = 1024;
    while (s < 2 * rows) s *= 2;
    return s;
  }
  // Room for `rows` more rows behind the first `count` of `buf`, which are kept.
  void grow_rows(DevBuf& buf, int W, u64 count, u64 rows) {
    const size_t need = sizeof(u64) * W * (count + rows);
    if (buf.cap >= need) return;
    DevBuf larger;
    larger.reserve(need);
    SW_CUDA(cudaMemcpyAsync(larger.p, buf.p, sizeof(u64) * W * (size_t)count, cudaMemcpyDeviceToDevice, stream));
    std::swap(buf.p, larger.p);
    std::swap(buf.cap, larger.cap);
    larger.release();
  }
  // Lists up to this size are hashed; larger ones, whose table and second list
  // would take several times as much again, are kept sorted.  So are lists that,
  // with table and second list, would pass the search's memory budget, which
  // counts rows only.
  static constexpr u64 kHashBytes = 16ull << 30;
  size_t list_budget = ~(size_t)0;
  bool hashable(const Side& X, int W, u64 children) const {
    const u64 rows = (X.split ? X.met_count : X.vis_count) + children + 1;
    if (X.sorted_only || 2 * rows > 1ull << 32 || rows * 8 * W > kHashBytes) return false;
    if (list_budget == ~(size_t)0) return true;
    // what the step's buffers come to, and the list that is copied while it grows
    size_t copied = 0;
    const auto list = [&](const DevBuf& b, u64 count) {
      const size_t need = sizeof(u64) * W * (count + children);
      if (b.cap >= need) return b.cap;
      copied = std::max(copied, b.cap);
      return need + need / 4;
    };
    size_t bytes = list(X.vis, X.vis_count);
    if (X.split || reductions) bytes += list(X.met, X.split ? X.met_count : X.vis_count);
    bytes += 2 * X.table_slots < 3 * rows ? sizeof(u64) * slots_for(rows) / 4 * 5 : X.table.cap;
    return bytes + copied + X.vis_alt.cap + (&X == &F ? B : F).list_bytes() <= list_budget;
  }
  // Gives back what the bounded phase, whose levels are counted row by row, has no use for.
  void release_tables() {
    for (Side* X : {&F, &B}) {
      X->table.release();
      X->met.release();
      X->table_slots = 0;
    }
  }
  // One layer on a hashed side: children equal to a row met before or to a sibling
  // are dropped by the table, then, with the reductions on, those that a visited
  // set or a sibling dominates.
  // With `defer` the counts stay on the device (X.live) until finish_step():
  // the launches that follow are sized for every child.
  void step_hashed(Side& X, bool forward, int W, int n, int k, bool defer) {
    const u32 m = X.count, Nc = m * (u32)k;
    const bool reduce = reductions;
    Side::Step& P = X.step;
    P = Side::Step{};
    P.t0 = vclock();
    P.forward = forward;
    P.reduce = reduce;
    P.parents = m;
    P.children = Nc;
    X.hashed = true;
    if (reduce && !X.split) {
      X.split = true;
      X.met_count = X.vis_count;
      X.met.reserve(sizeof(u64) * W * ((size_t)X.vis_count + Nc));
      SW_CUDA(cudaMemcpyAsync(X.met.p, X.vis.p, sizeof(u64) * W * (size_t)X.vis_count, cudaMemcpyDeviceToDevice,
                              stream));
    }
    DevBuf& list = X.split ? X.met : X.vis;
    const u32 base = X.split ? X.met_count : X.vis_count;
    grow_rows(list, W, base, Nc);
    if (2 * X.table_slots < 3 * ((u64)base + Nc)) {  // fewer than 1.5 slots a row: rebuild
      X.table_slots = slots_for((u64)base + Nc);
      X.table.reserve(sizeof(u64) * X.table_slots);
      SW_CUDA(cudaMemsetAsync(X.table.p, 0, sizeof(u64) * X.table_slots, stream));
      timed(3, (double)base * (8.0 * W + 8), [&] {
        launch_hash_build(W, list.as<u64>(), base, X.table.as<u64>(), (u32)(X.table_slots - 1), d_misc + kScanErrWord,
                          stream);
      });
      count_launch();
    }
    ch_rows.reserve(sizeof(u64) * W * (size_t)Nc);
    const BucketScratch bk = buckets(Nc);
    // reads each parent row, writes k child rows, a table slot and a place each
    timed(1, (double)m * 8.0 * W * (1 + k) + (double)Nc * 16.0, [&] {
      launch_expand_hash(W, forward, X.cur_rows(W), m, tables, ch_rows.as<u64>(), list.as<u64>(), base,
                         X.table.as<u64>(), (u32)(X.table_slots - 1), bk, d_misc + kScanErrWord, stream);
    });
    std::unique_ptr<Layer> L = X.new_layer(sizeof(u32) * (size_t)std::max<u32>(Nc, 1));
    L->origin.reserve(sizeof(u32) * (size_t)std::max<u32>(Nc, 1));
    if (X.split) uq_vals.reserve(sizeof(u32) * (size_t)std::max<u32>(Nc, 1));
    u64* const fresh = list.as<u64>() + (size_t)base * W;  // the new rows, in bucket order
    u32* const fresh_origin = X.split ? uq_vals.as<u32>() : L->origin.as<u32>();
    timed(3, (double)Nc * (2 * 8.0 * W + 8 + 4), [&] {
      launch_bucket_scatter(W, ch_rows.as<u64>(), Nc, bk, base, fresh, fresh_origin, X.table.as<u64>(), d_misc + 8,
                            stream);
    });
    scanned();
    count_launch(3);
    // The checks of a reduced level are cut for the rows they are told of, and
    // where most children are duplicates few of those rows are there: from
    // kDomOrderRows children on the count is read back first (searches whose
    // letters permute all states but one: n = 60, k = 16 55 -> 26 ms, n = 40, k = 8
    // 35 -> 20; below, a read-back costs more than it saves: n = 100, k = 3 plans
    // of ten levels of 10 000 to 30 000 children 2.4 -> 2.6 ms)
    defer = defer && Nc && (reduce || !X.split);
    P.counted = reduce && Nc > kDomOrderRows;
    u32 u = Nc;
    if (!defer || P.counted) u = read_total_checked();
    defer = defer && u;
    const u32* const fresh_live = defer && !P.counted ? d_misc + 8 : nullptr;
    if (X.split) {
      P.visited = X.vis_count;
      grow_rows(X.vis, W, X.vis_count, u);
      u64* const out = X.vis.as<u64>() + (size_t)X.vis_count * W;
      if (reduce && u) {
        flags_a.reserve(sizeof(u32) * (size_t)u);
        SW_CUDA(cudaMemsetAsync(flags_a.p, 0, sizeof(u32) * (size_t)u, stream));
        reduce_span.mark(0, stream);
        if (X.vis_count)
          dominated(forward, W, X.vis.as<u64>(), X.vis_count, fresh, u, n, false, X.vis_count, flags_a.as<u32>(),
                    dom_rows, nullptr, fresh_live);
        dominated(forward, W, fresh, u, fresh, u, n, true, X.vis_count, flags_a.as<u32>(), dom_rows, fresh_live,
                  fresh_live);
        reduce_span.mark(1, stream);
        const u32 epoch = next_dc_epoch(u);
        timed(3, (double)u * (4 + 2 * (8.0 * W + 4)), [&] {
          launch_keep_compact(W, fresh, fresh_origin, flags_a.as<u32>(), u, out, L->origin.as<u32>(), d_misc + 9,
                              dc_status.as<u64>(), dc_ctr.as<u32>(), epoch, d_misc + kScanErrWord, stream, fresh_live);
        });
        count_launch();
      } else if (u) {
        SW_CUDA(cudaMemcpyAsync(out, fresh, sizeof(u64) * W * (size_t)u, cudaMemcpyDeviceToDevice, stream));
        SW_CUDA(cudaMemcpyAsync(L->origin.p, fresh_origin, sizeof(u32) * (size_t)u, cudaMemcpyDeviceToDevice, stream));
      }
    }
    L->parent_count = m;
    X.layers.push_back(std::move(L));
    X.in_vis = true;
    X.cur_off = X.vis_count;
    X.count = u;
    P.base = base;
    P.compacted = X.split && reduce && u;
    P.deferred = defer;
    if (defer) {
      X.live = d_misc + (P.compacted ? 9 : 8);
      return;
    }
    SW_CUDA(cudaMemcpyAsync(pinned.p, d_misc, sizeof(u32) * kStepWords, cudaMemcpyDeviceToHost, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    finish_step(X, pinned.as<u32>());
  }
  // The step's counts from a host copy of d_misc's first kStepWords words.
  static constexpr int kStepWords = 10;
  void finish_step(Side& X, const u32* w) {
    Side::Step& P = X.step;
    check_scan_error(w[kScanErrWord]);
    const u32 u = w[8], f = P.compacted ? w[9] : u;
    // branching of a level that drops siblings only (the bounded phase's)
    if (P.parents) X.unique_growth = (double)(u + w[7]) / P.parents;
    if (st) {
      st->subsets_expanded += P.children;
      st->subsets_kept += f;
    }
    if (P.deferred && P.compacted && !P.counted) {
      if (P.visited) count_query(P.visited, u);
      count_query(u, u);
    }
    if (X.split) X.met_count = P.base + u;
    P.distinct = u;
    P.kept = f;
    X.layers.back()->count = f;
    X.count = f;
    X.vis_count += f;
    X.live = nullptr;
    if (verbose)
      std::fprintf(stderr, "[sw] %s parents=%u children=%u unique=%u kept=%u (%s) | %.3f ms\n",
                   P.forward ? "BFS " : "IBFS", P.parents, P.children, u, f, P.reduce ? "reduced" : "duplicates only",
                   vclock() - P.t0);
  }
  // X's children without duplicates among themselves, in bucket order, as its next
  // layer, whose count is left in d_misc[8].
  void step_distinct(Side& X, int W, int k) {
    const u32 m = X.count, Nc = m * (u32)k;
    const u64 slots = slots_for(Nc);
    level_table.reserve(sizeof(u64) * slots);
    ch_rows.reserve(sizeof(u64) * W * (size_t)Nc);
    X.rows_alt.reserve(sizeof(u64) * W * (size_t)Nc);
    const BucketScratch bk = buckets(Nc);
    SW_CUDA(cudaMemsetAsync(level_table.p, 0, sizeof(u64) * slots, stream));
    timed(1, (double)m * 8.0 * W * (1 + k) + (double)Nc * 16.0, [&] {
      launch_expand_hash(W, true, X.rows.as<u64>(), m, tables, ch_rows.as<u64>(), nullptr, 0, level_table.as<u64>(),
                         (u32)(slots - 1), bk, d_misc + kScanErrWord, stream);
    });
    std::unique_ptr<Layer> L = X.new_layer(sizeof(u32) * (size_t)Nc);
    L->origin.reserve(sizeof(u32) * (size_t)Nc);
    timed(3, (double)Nc * (2 * 8.0 * W + 8 + 4), [&] {
      launch_bucket_scatter(W, ch_rows.as<u64>(), Nc, bk, 0, X.rows_alt.as<u64>(), L->origin.as<u32>(), nullptr,
                            d_misc + 8, stream);
    });
    scanned();
    count_launch(3);
    if (st) st->subsets_expanded += Nc;
    std::swap(X.rows.p, X.rows_alt.p);
    std::swap(X.rows.cap, X.rows_alt.cap);
    L->parent_count = m;
    X.layers.push_back(std::move(L));
    X.count = Nc;
  }
  // Back to a current layer of its own and a visited list in key order.
  void unhash(Side& X, int W) {
    if (!X.hashed) return;
    if (X.in_vis) {
      X.rows.reserve(sizeof(u64) * W * (size_t)std::max<u32>(X.count, 1));
      SW_CUDA(cudaMemcpyAsync(X.rows.p, X.cur_rows(W), sizeof(u64) * W * (size_t)X.count, cudaMemcpyDeviceToDevice,
                              stream));
    }
    X.hashed = X.in_vis = X.split = false;
    X.table_slots = 0;
    X.table.release();
    X.met.release();
    dom_rows.release();
    sort_by_layer_key(W, X.vis.as<u64>(), X.vis_count, X.keymap);
  }

  // `ordered`: the layer's rows come in key order, the same on every run
  // (samples of a layer, and beams whose ties go by it, depend on that).
  // `defer`: the counts of a hashed step may stay on the device until the caller's
  // next read-back (X.live then names the layer's, and finish_step() is called).
  void step(Side& X, bool forward, int W, int n, int k, bool dominance = true, bool ordered = false,
            bool defer = false) {
    const u32 m = X.count;
    const u64 N = (u64)m * k;
    if (N > 0xffffffffULL) throw std::runtime_error("layer exceeds 2^32 children");
    const u32 Nc = (u32)N;
    if (dominance && !ordered && !sort_key_option() && hashable(X, W, N)) 
      return step_hashed(X, forward, W, n, k, defer && !verbose && !prof_on);
    unhash(X, W);
    X.sorted_only = true;
    ch_rows.reserve(sizeof(u64) * W * N);
    ch_vals.reserve(sizeof(u32) * N);
    uq_rows.reserve(sizeof(u64) * W * N);
    uq_vals.reserve(sizeof(u32) * N);
    flags_a.reserve(sizeof(u32) * N);
    flags_b.reserve(sizeof(u32) * N);
    keep.reserve(sizeof(u32) * N);
    const double t_step0 = vclock();
    keys.reserve(sizeof(u64) * 2 * N);
    sorted_rows.reserve(sizeof(u64) * W * N);
    // expansion reads each parent row and writes k child rows, each with its
    // layer key (2 words) and its index as the sort payload
    timed(1, (double)m * 8.0 * W * (1 + k) + (double)N * 20.0, [&] {
      launch_expand(W, forward, X.rows.as<u64>(), m, tables, ch_rows.as<u64>(), stream, keys.as<u64>(),
                    ch_vals.as<u32>(), X.keymap);
    });
    count_launch(1);
    if (st) st->subsets_expanded += N;
    // sort the children by layer key
    sort_rows(2, keys.as<u64>(), ch_vals.as<u32>(), Nc);
    if (dominance && !reductions) {
      // duplicates only: a child is dropped when it equals its predecessor in
      // the sorted layer or a visited set.  One launch flags the children in
      // sort order (rows read through the sort's permutation), counts the
      // kept ones before each tile by decoupled look-back, and gathers the
      // kept rows and their origins into the new layer.
      X.rows_alt.reserve(sizeof(u64) * W * (size_t)std::max<u32>(Nc, 1));
      std::unique_ptr<Layer> L = X.new_layer(sizeof(u32) * (size_t)std::max<u32>(Nc, 1));
      L->origin.reserve(sizeof(u32) * (size_t)std::max<u32>(Nc, 1));
      u32* total = d_misc + 8;
      const u32 epoch = next_dc_epoch(Nc);
      timed(3, (double)Nc * (4 + 16 + 8.0 * W) + (double)Nc * (8.0 * W + 4), [&] {
        launch_dedup_compact(W, ch_rows.as<u64>(), ch_vals.as<u32>(), keys.as<u64>(), Nc, X.vis.as<u64>(),
                             X.vis_count, X.keymap, X.rows_alt.as<u64>(), L->origin.as<u32>(), total,
                             dc_status.as<u64>(), dc_ctr.as<u32>(), epoch, d_misc + kScanErrWord, stream);
      });
      count_launch();
      const u32 f = read_total_checked();
      if (m) X.unique_growth = (double)f / m;
      if (verbose)
        std::fprintf(stderr, "[sw] %s parents=%u children=%u kept=%u (duplicates only) | %.3f ms\n",
                     forward ? "BFS " : "IBFS", m, Nc, f, vclock() - t_step0);
      finish_layer(X, W, n, m, f, std::move(L));
      return;
    }
    // the other reductions work on the rows in sorted order
    launch_gather_rows(W, ch_rows.as<u64>(), ch_vals.as<u32>(), Nc, sorted_rows.as<u64>(), stream);
    launch_unique_flags(W, sorted_rows.as<u64>(), Nc, flags_a.as<u32>(), stream);
    count_launch(2);
    const u32 u = compact(W, sorted_rows.as<u64>(), ch_vals.as<u32>(), flags_a.as<u32>(), Nc, uq_rows.as<u64>(),
                          uq_vals.as<u32>());
    if (m) X.unique_growth = (double)u / m;  // branching before dominance pruning
    if (!dominance) {
      // bounded phase: the deduplicated layer is the new frontier as is
      std::swap(X.rows.p, uq_rows.p);
      std::swap(X.rows.cap, uq_rows.cap);
      X.count = u;
      if (st) {
        st->subsets_kept += u;
        st->dfs_sets += u;
      }
      auto L = X.new_layer(sizeof(u32) * std::max<u32>(u, 1));
      L->origin.reserve(sizeof(u32) * std::max<u32>(u, 1));
      if (u) SW_CUDA(cudaMemcpyAsync(L->origin.p, uq_vals.p, sizeof(u32) * u, cudaMemcpyDeviceToDevice, stream));
      L->count = u;
      L->parent_count = m;
      X.layers.push_back(std::move(L));
      if (verbose)
        std::fprintf(stderr, "[sw] %s (bounded) parents=%u children=%u unique=%u | %.3f ms\n",
                     forward ? "BFS " : "IBFS", m, Nc, u, vclock() - t_step0);
      return;
    }
    // dominance: visited set inside the child, or a proper subset in the layer
    launch_fill_u32(flags_a.as<u32>(), 0, u, stream);
    launch_fill_u32(flags_b.as<u32>(), 0, u, stream);
    count_launch(2);
    const double t_sort = vclock();
    if (X.vis_count)  // the list the layer is merged into afterwards is free until then
      dominated(forward, W, X.vis.as<u64>(), X.vis_count, uq_rows.as<u64>(), u, n, false, X.vis_count,
                flags_a.as<u32>(), X.vis_alt);
    const double t_vis = vclock();
    dominated(forward, W, uq_rows.as<u64>(), u, uq_rows.as<u64>(), u, n, true, X.vis_count, flags_b.as<u32>(),
                X.vis_alt);
    const double t_self = vclock();
    if (verbose) {
      std::vector<u32> fa(u), fb(u);
      SW_CUDA(cudaMemcpy(fa.data(), flags_a.p, sizeof(u32) * u, cudaMemcpyDeviceToHost));
      SW_CUDA(cudaMemcpy(fb.data(), flags_b.p, sizeof(u32) * u, cudaMemcpyDeviceToHost));
      size_t cv = 0, cs = 0;
      for (u32 i = 0; i < u; ++i) {
        cv += fa[i] != 0;
        cs += fb[i] != 0;
      }
      std::fprintf(stderr,
                   "[sw] %s parents=%u children=%u unique=%u visited=%u dropped_by_visited=%zu dropped_by_self=%zu "
                   "| expand+sort+unique %.3f ms, visited check %.3f ms, self check %.3f ms\n",
                   forward ? "BFS " : "IBFS", m, Nc, u, X.vis_count, cv, cs, t_sort - t_step0, t_vis - t_sort,
                   t_self - t_vis);
    }
    launch_keep_flags(flags_a.as<u32>(), flags_b.as<u32>(), u, keep.as<u32>(), stream);
    count_launch();
    X.rows_alt.reserve(sizeof(u64) * W * (size_t)std::max<u32>(u, 1));
    new_vals.reserve(sizeof(u32) * (size_t)std::max<u32>(u, 1));
    const u32 f = compact(W, uq_rows.as<u64>(), uq_vals.as<u32>(), keep.as<u32>(), u, X.rows_alt.as<u64>(),
                          new_vals.as<u32>());
    finish_layer(X, W, n, m, f);
  }

  // The kept children (X.rows_alt, f of them) become the new layer of X:
  // recorded for word tracing and merged into the visited list.  Their origins
  // are in `L` when given, else in new_vals.
  void finish_layer(Side& X, int W, int n, u32 m, u32 f, std::unique_ptr<Layer> L = nullptr) {
    std::swap(X.rows.p, X.rows_alt.p);
    std::swap(X.rows.cap, X.rows_alt.cap);
    X.count = f;
    if (st) st->subsets_kept += f;
    if (!L) {
      L = X.new_layer(sizeof(u32) * std::max<u32>(f, 1));
      L->origin.reserve(sizeof(u32) * std::max<u32>(f, 1));
      if (f)
        SW_CUDA(cudaMemcpyAsync(L->origin.p, new_vals.p, sizeof(u32) * f, cudaMemcpyDeviceToDevice, stream));
    }
    L->count = f;
    L->parent_count = m;
    X.layers.push_back(std::move(L));
    // visited := visited ∪ layer (both sorted, disjoint)
    X.vis_alt.reserve(sizeof(u64) * W * ((size_t)X.vis_count + f + 1));
    timed(3, (double)(X.vis_count + f) * 8.0 * W * 2, [&] {
      launch_merge_key(W, X.vis.as<u64>(), X.vis_count, X.rows.as<u64>(), f, X.vis_alt.as<u64>(), stream,
                       X.keymap);
    });
    count_launch();
    std::swap(X.vis.p, X.vis_alt.p);
    std::swap(X.vis.cap, X.vis_alt.cap);
    X.vis_count += f;
    if (!X.keymap_chosen && X.count >= 2048) choose_keymap(X, W, n);
  }

  // Optionally, once a side's layers are large enough to matter, lead its
  // sort key with 64 chosen states of its current layer (for the backward
  // side, states of the complements) and re-sort its visited list.
  DevBuf d_counts;
  static const char* sort_key_option() {
    static const char* opt = std::getenv("SW_SORT_KEY");
    return opt && (std::string(opt) == "frequent" || std::string(opt) == "balanced") ? opt : nullptr;
  }
  void choose_keymap(Side& X, int W, int n) {
    X.keymap_chosen = true;
    if (n <= 64) return;  // the identity map already covers every state
    // Measured on random binary DFAs (n = 200 and 320), re-keying made the
    // subset checks slower than the identity key, so it is opt-in:
    // SW_SORT_KEY=frequent or SW_SORT_KEY=balanced.
    const char* opt = sort_key_option();
    if (!opt) return;
    d_counts.reserve(sizeof(u32) * 64 * W);
    SW_CUDA(cudaMemsetAsync(d_counts.p, 0, sizeof(u32) * 64 * W, stream));
    launch_state_counts(W, X.rows.as<u64>(), X.count, d_counts.as<u32>(), stream);
    std::vector<u32> cnt(64 * W);
    SW_CUDA(cudaMemcpyAsync(cnt.data(), d_counts.p, sizeof(u32) * cnt.size(), cudaMemcpyDeviceToHost, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    std::vector<int> idx(n);
    std::iota(idx.begin(), idx.end(), 0);
    // column q of the device row holds state q (word q/64, bit 63 - q%64).
    // "balanced" leads with the states closest to half the layer (the most
    // even splits), "frequent" with the most frequent.
    if (std::string(opt) == "balanced") {
      const long long half = X.count / 2;
      std::stable_sort(idx.begin(), idx.end(),
                       [&](int a, int b) { return std::llabs(cnt[a] - half) < std::llabs(cnt[b] - half); });
    } else {
      std::stable_sort(idx.begin(), idx.end(), [&](int a, int b) { return cnt[a] > cnt[b]; });
    }
    KeyMap km;
    km.identity = 0;
    for (int j = 0; j < 64; ++j) km.q[j] = (uint16_t)idx[j];
    X.keymap = km;
    sort_by_layer_key(W, X.vis.as<u64>(), X.vis_count, X.keymap);
    count_launch(2);
  }

  // Bounded phase helpers.  expand_dedup: preimages (complement rows) of m
  // parents, duplicates removed, into out_rows / out_origin (origin = letter *
  // m + parent) — no dominance, no visited update.
  void expand_dedup(const u64* parents, u32 m, int W, int k, DevBuf& out_rows, DevBuf& out_origin, u32& out_count) {
    const u64 N = (u64)m * k;
    if (N > 0xffffffffULL) throw std::runtime_error("level exceeds 2^32 children");
    const u32 Nc = (u32)N;
    const u64 slots = slots_for(N);
    if (slots > 1ull << 32) throw std::runtime_error("level exceeds 2^31 children");
    ch_rows.reserve(sizeof(u64) * W * N);
    level_table.reserve(sizeof(u64) * slots);
    out_rows.reserve(sizeof(u64) * W * std::max<u64>(N, 1));
    out_origin.reserve(sizeof(u32) * std::max<u64>(N, 1));
    const BucketScratch bk = buckets(N);
    const double t0 = vclock();
    SW_CUDA(cudaMemsetAsync(level_table.p, 0, sizeof(u64) * slots, stream));
    timed(1, (double)m * 8.0 * W * (1 + k) + (double)N * 16.0, [&] {
      launch_expand_hash(W, false, parents, m, tables, ch_rows.as<u64>(), nullptr, 0, level_table.as<u64>(),
                         (u32)(slots - 1), bk, d_misc + kScanErrWord, stream);
    });
    timed(3, (double)N * (2 * 8.0 * W + 8 + 4), [&] {
      launch_bucket_scatter(W, ch_rows.as<u64>(), Nc, bk, 0, out_rows.as<u64>(), out_origin.as<u32>(), nullptr,
                            d_misc + 8, stream);
    });
    scanned();
    count_launch(3);
    if (st) st->subsets_expanded += N;
    out_count = read_total_checked();
    if (verbose)
      std::fprintf(stderr, "[sw] IBFS (bounded) parents=%u children=%u unique=%u | %.3f ms\n", m, Nc, out_count,
                   vclock() - t0);
  }

  // Meet check of q complement rows against F; on a hit returns true with the
  // query index and the F index.
  bool meet(int W, int n, const u64* Q, u32 q, u32* qi, u32* si) {
    SW_CUDA(cudaMemsetAsync(d_misc, 0, 4 * sizeof(u32), stream));
    query(W, kQueryDisjoint, F.cur_rows(W), F.count, Q, q, n, nullptr, true);
    if (st) st->meet_pairs += (u64)F.count * q;
    SW_CUDA(cudaMemcpyAsync(pinned.p, d_misc, 5 * sizeof(u32), cudaMemcpyDeviceToHost, stream));  // witness + error
    SW_CUDA(cudaStreamSynchronize(stream));
    const u32* w = pinned.as<u32>();
    check_scan_error(w[4]);
    if (!w[0]) return false;
    *qi = w[1];
    *si = w[2];
    return true;
  }

  // Trace letters of set `idx` at the top layer of side X down to depth 0.
  DevBuf trace_dev;
  HostPinned trace_host;
  std::vector<uint32_t> trace(const Side& X, u32 idx, u32* seed_index) {
    const size_t L = X.layers.size();  // letters come from the top layer down
    const size_t steps_bytes = sizeof(TraceStep) * L, out_bytes = sizeof(u32) * (L + 1);
    trace_dev.reserve(steps_bytes + out_bytes);
    trace_host.reserve(steps_bytes + out_bytes);
    TraceStep* h = trace_host.as<TraceStep>();
    for (size_t i = 0; i < L; ++i) h[i] = TraceStep{X.layers[L - 1 - i]->org(), X.layers[L - 1 - i]->parent_count};
    SW_CUDA(cudaMemcpyAsync(trace_dev.p, h, steps_bytes, cudaMemcpyHostToDevice, stream));
    u32* d_out = reinterpret_cast<u32*>(trace_dev.as<uint8_t>() + steps_bytes);
    launch_trace(trace_dev.as<TraceStep>(), (u32)L, idx, d_out, stream);
    u32* out = reinterpret_cast<u32*>(trace_host.as<uint8_t>() + steps_bytes);
    SW_CUDA(cudaMemcpyAsync(out, d_out, out_bytes, cudaMemcpyDeviceToHost, stream));
    SW_CUDA(cudaStreamSynchronize(stream));
    if (seed_index) *seed_index = out[L];
    return std::vector<uint32_t>(out, out + L);
  }

  // ---- the first levels in one launch (batch_cluster.cu) ----
  // A search starts on one thread-block cluster, which runs it level by level
  // on the device: to its end where the lists stay small, else until a level
  // is worth the whole GPU; import_single() then turns the cluster's lists into
  // the two sides' layers.
  DevBuf single_scratch, single_in, single_org[2];
  HostPinned single_host;
  u64 single_tags = 0;
  size_t single_zeroed = 0;
  struct Single {
    SmallResult res;
    ClusterExit exit;
    const uint8_t* word;
  };
  // `meanwhile` runs on the host while the cluster searches; when it returns false
  // the search is given up (a search without an end took up to 5.5 ms of its
  // hundreds of levels, where the host knows after 0.05).
  template <class Fn>
  Single run_single(const Automaton& A, const std::vector<uint32_t>& seeds, u32 max_len, u64 budget, Fn&& meanwhile) {
    const int W = words_for((int)A.n);
    const ClusterCaps caps = cluster_single_caps();
    single_scratch.reserve(cluster_single_scratch_bytes(caps));
    if (single_zeroed < single_scratch.cap || single_tags + cluster_tags_per_launch(1) >= kClusterTagLimit) {
      SW_CUDA(cudaMemsetAsync(single_scratch.p, 0, single_scratch.cap, stream));
      single_zeroed = single_scratch.cap;
      single_tags = 0;
    }
    single_tags += cluster_tags_per_launch(1);
    // input: the launch's counter (zero), the instance, its table and seeds
    const size_t inst_off = 32, pool_off = 64, seeds_off = pool_off + A.t.size();
    const size_t in_bytes = seeds_off + seeds.size();
    const size_t out_bytes = kClusterSingleWords + kClusterSingleWord - 256;
    single_in.reserve(in_bytes);
    single_host.reserve(16384 + sizeof(u32) * kClusterMetaWords);
    uint8_t* h = single_host.as<uint8_t>();
    std::memset(h, 0, pool_off);
    const SmallInstance I{A.n, A.k, (u32)pool_off, (u32)seeds_off, (u32)seeds.size(), max_len};
    std::memcpy(h + inst_off, &I, sizeof(I));
    for (size_t i = 0; i < A.t.size(); ++i) h[pool_off + i] = (uint8_t)A.t[i];
    for (size_t i = 0; i < seeds.size(); ++i) h[seeds_off + i] = (uint8_t)seeds[i];
    SW_CUDA(cudaMemcpyAsync(single_in.p, h, in_bytes, cudaMemcpyHostToDevice, stream));
    ClusterLimits lim;
    lim.max_children = kSingleMaxChildren;
    lim.max_pairs = kSingleMaxPairs;
    lim.budget = budget;
    lim.counter_ready = 1;
    lim.header_bytes = kClusterSingleHeader;
    volatile u32* const cancel = reinterpret_cast<volatile u32*>(h + 12288);
    *cancel = 0;
    lim.cancel = const_cast<const u32*>(cancel);
    uint8_t* sc = single_scratch.as<uint8_t>();
    const uint8_t* in = single_in.as<uint8_t>();
    timed(3, 0.0, [&] {
      launch_cluster_batch(W, kSingleClusterCtas, 1, reinterpret_cast<const SmallInstance*>(in + inst_off), 1, in, in,
                           reinterpret_cast<SmallResult*>(sc + kClusterSingleResult), sc + kClusterSingleWords,
                           kClusterSingleWord, sc, caps, lim, single_in.as<u32>(), nullptr, stream);
    });
    count_launch();
    uint8_t* out = h + 8192;
    SW_CUDA(cudaMemcpyAsync(out, sc + 256, out_bytes, cudaMemcpyDeviceToHost, stream));
    if (!meanwhile()) *cancel = 1;
    SW_CUDA(cudaStreamSynchronize(stream));
    Single r;
    std::memcpy(&r.res, out + kClusterSingleResult - 256, sizeof(r.res));
    std::memcpy(&r.exit, out + kClusterExitOffset - 256, sizeof(r.exit));
    r.word = out + kClusterSingleWords - 256;
    if (st) {
      st->bfs_steps += r.exit.depth[0];
      st->ibfs_steps += r.exit.depth[1];
      st->subsets_expanded += r.exit.children;
      st->subsets_kept += r.exit.kept[0] + r.exit.kept[1] - 1 - seeds.size();
      st->trie_queries += r.exit.queries;
      st->logical_pairs += r.exit.pairs;
      st->meet_pairs += r.exit.pairs;
    }
    return r;
  }
  void import_single(int W, const ClusterExit& ex) {
    const ClusterCaps caps = cluster_single_caps();
    u32* meta = reinterpret_cast<u32*>(single_host.as<uint8_t>() + 16384);
    SW_CUDA(cudaMemcpyAsync(meta, single_scratch.as<uint8_t>() + cluster_meta_offset(W, kClusterSingleHeader, caps),
                            sizeof(u32) * kClusterMetaWords, cudaMemcpyDeviceToHost, stream));
    for (int side = 0; side < 2; ++side) {
      Side& X = side ? B : F;
      const u32 kept = ex.kept[side], cnt = ex.cnt[side], depth = ex.depth[side];
      ch_rows.reserve(sizeof(u64) * W * kept);
      single_org[side].reserve(sizeof(u32) * kept);
      launch_cluster_export(W, single_scratch.p, kClusterSingleHeader, caps, side, kept, depth, ch_rows.as<u64>(),
                            single_org[side].as<u32>(), stream);
      // the visited list: the earlier layers as they are, then the current one in bucket order
      const u32 base = kept - cnt;
      X.vis.reserve(sizeof(u64) * W * (size_t)kept);
      SW_CUDA(cudaMemcpyAsync(X.vis.p, ch_rows.p, sizeof(u64) * W * (size_t)base, cudaMemcpyDeviceToDevice, stream));
      const u64* cur = ch_rows.as<u64>() + (size_t)(kept - cnt) * W;
      const BucketScratch bk = buckets(cnt);
      ch_vals.reserve(sizeof(u32) * cnt);
      launch_bucket_rank(W, cur, cnt, bk, stream);
      launch_bucket_scatter(W, cur, cnt, bk, base, X.vis.as<u64>() + (size_t)base * W, ch_vals.as<u32>(), nullptr,
                            d_misc + 8, stream);
      scanned();
      count_launch(4);
      X.hashed = X.in_vis = true;
      X.cur_off = base;
      X.count = cnt;
      X.vis_count = base + cnt;
      std::unique_ptr<Layer> top;
      if (depth) {  // the current layer's origins in the order of its rows
        top = X.new_layer(sizeof(u32) * cnt);
        top->origin.reserve(sizeof(u32) * cnt);
        launch_gather_u32(single_org[side].as<u32>() + (kept - cnt), ch_vals.as<u32>(), cnt, top->origin.as<u32>(),
                          stream);
        count_launch();
      }
      if (side == 0) SW_CUDA(cudaStreamSynchronize(stream));  // the layer table has arrived
      const u32* loff = meta + (2 + side) * kClusterMetaStride;
      const u32* lcnt = meta + (4 + side) * kClusterMetaStride;
      for (u32 d = 1; d <= depth; ++d) {
        std::unique_ptr<Layer> L = d == depth ? std::move(top) : X.new_layer(0);
        if (d < depth) L->view = single_org[side].as<u32>() + loff[d];
        L->count = lcnt[d];
        L->parent_count = lcnt[d - 1];
        X.layers.push_back(std::move(L));
      }
    }
  }
};

// ---------------------------------------------------------------------------
// Bounded inverse phase with chunking (the reference's memory-bounded DFS,
// dfs.cpp:161-218, on device levels).  F is frozen; B levels are expanded
// with duplicate removal only and meet-checked against F.  A level whose
// children fit the budget is expanded whole (plain BFS); otherwise its
// parents are taken in chunks and each chunk's subtree is explored depth
// first.  A hit at length L makes every other branch search only lengths
// below L (dfs.cpp:179-189), so the smallest length found is the answer.
// ---------------------------------------------------------------------------
namespace {

struct BoundedSearch {
  Engine& E;
  const Automaton& A;
  int W, n, k;
  size_t budget, row_bytes;
  u64 min_chunk;
  u64 max_len;  // longest length still worth examining
  u64 best = 0;
  std::vector<uint32_t> best_tail;  // letters after the forward part, for the best hit
  u32 best_f = 0;
  std::vector<DLevel*> levels;                // levels[0] stands for E.B (nullptr)
  std::vector<std::unique_ptr<DLevel>> pool;  // one reusable level per depth
  sw_stats& st;

  size_t held() const {
    size_t s = (size_t)(E.F.count + E.F.vis_count + E.B.count + E.B.vis_count) * row_bytes;
    for (size_t i = 1; i < levels.size(); ++i) s += (size_t)levels[i]->count * (row_bytes + 4);
    return s;
  }

  const u64* level_rows(size_t li) const {
    return li == 0 ? E.B.cur_rows(W) : levels[li]->rows.as<u64>();
  }

  // Letters from level `li` index x back to the B frontier, plus the MITM B trace.
  std::vector<uint32_t> tail_word(size_t li, u32 x) {
    std::vector<uint32_t> letters;
    for (size_t l = li; l >= 1; --l) {
      const DLevel& L = *levels[l];
      const u32 o = E.read_u32(L.origin.as<u32>() + x);
      letters.push_back(o / L.chunk_cnt);
      x = L.chunk_off + o % L.chunk_cnt;
    }
    std::vector<uint32_t> bw = E.trace(E.B, x, nullptr);
    letters.insert(letters.end(), bw.begin(), bw.end());
    return letters;
  }

  // Explore the children of parents [off, off+cnt) of level li (at length len).
  void explore(size_t li, u32 off, u32 cnt, u64 len) {
    if (len + 1 > max_len || cnt == 0) return;
    const double per_child = (double)k * (3.0 * row_bytes + 32) + (double)k * (row_bytes + 4);
    const size_t have = budget > held() ? budget - held() : 0;
    u64 chunk = (u64)((double)have / per_child);
    if (chunk < min_chunk) chunk = min_chunk;
    if (chunk > cnt) chunk = cnt;
    for (u32 pos = 0; pos < cnt && len + 1 <= max_len; pos += (u32)chunk) {
      const u32 c = (u32)std::min<u64>(chunk, cnt - pos);
      const size_t me = levels.size();
      while (pool.size() <= me) pool.push_back(std::make_unique<DLevel>());
      DLevel* L = pool[me].get();
      L->chunk_off = off + pos;
      L->chunk_cnt = c;
      E.expand_dedup(level_rows(li) + (size_t)(off + pos) * W, c, W, k, L->rows, L->origin, L->count);
      st.dfs_sets += L->count;
      levels.push_back(L);
      u32 q = 0, s = 0;
      if (E.meet(W, n, levels[me]->rows.as<u64>(), levels[me]->count, &q, &s)) {
        best = len + 1;
        best_f = s;
        best_tail = tail_word(me, q);
        max_len = len;  // only shorter words are of interest from now on
        if (E.verbose)
          std::fprintf(stderr, "[sw] bounded search: word of length %llu found; searching below\n",
                       (unsigned long long)best);
      } else if (len + 1 < max_len) {
        explore(me, 0, levels[me]->count, len + 1);
      }
      levels.pop_back();
    }
  }
};
}  // namespace

Solver::Solver(int device) : device_(device), eng_(new Engine(device)) {}
Solver::~Solver() = default;

void* Solver::stream() const { return (void*)eng_->stream; }
void Solver::profile_begin() {
  SW_CUDA(cudaSetDevice(device_));
  eng_->profile_begin();
}
void Solver::profile_end(sw_kernel_profile out[4]) {
  SW_CUDA(cudaSetDevice(device_));
  eng_->profile_end(out);
}
void Solver::set_scan_shapes(const ScanShapes& s) { eng_->scan_shapes = s; }
const ScanShapes& Solver::scan_shapes() const { return eng_->scan_shapes; }
void Solver::last_scan_profile(double ms[8 * kScanSizeClasses], uint64_t checks[8 * kScanSizeClasses]) const {
  for (int i = 0; i < 8 * kScanSizeClasses; ++i) {
    ms[i] = eng_->scan_ms[i];
    checks[i] = eng_->scan_launches[i];
  }
}

// ---------------------------------------------------------------------------
// Exact::run (exact.cpp:37-97) on the device.
// ---------------------------------------------------------------------------
// State order for the device search: states most likely to lie in forward
// images first (descending stationary mass of the random walk that applies a
// uniform random letter, with a 1% uniform restart).  Images are then most
// often separated by their first word, and the subset check's tile filter
// sees the shared states of a tile early.  The reference orders by stationary
// mass too (synchrolib/algorithm/exact/exact.cpp:108-127, ascending there, for
// its CPU trie); the order changes the work done, never the result.
static std::vector<uint32_t> image_frequency_order(const Automaton& A) {
  const uint32_t n = A.n, k = A.k;
  std::vector<double> pi(n, 1.0 / n), nx(n);
  const double share = 0.99 / k;
  for (int it = 0; it < 200; ++it) {
    std::fill(nx.begin(), nx.end(), 0.01 / n);
    for (uint32_t q = 0; q < n; ++q) {
      const double w = share * pi[q];
      for (uint32_t a = 0; a < k; ++a) nx[A.at(q, a)] += w;
    }
    double moved = 0;
    for (uint32_t q = 0; q < n; ++q) moved += std::abs(nx[q] - pi[q]);
    pi.swap(nx);
    if (moved < 1e-9) break;  // settled (random automata: after 30 to 60 rounds)
  }
  std::vector<uint32_t> idx(n);
  std::iota(idx.begin(), idx.end(), 0u);
  std::stable_sort(idx.begin(), idx.end(), [&](uint32_t x, uint32_t y) { return pi[x] > pi[y]; });
  std::vector<uint32_t> order(n);
  for (uint32_t r = 0; r < n; ++r) order[idx[r]] = r;
  return order;
}

void Solver::exact(const Automaton& A0, const sw_exact_config& cfg, Bounds& b, sw_stats& st,
                   const ReduceState* red) {
  const std::vector<uint32_t> order = image_frequency_order(A0);
  const Automaton A = permute(A0, order);
  if (b.non_synchro || b.lower == b.upper) return;  // exact.cpp:45-47
  if (A.n == 1) {                                   // exact.cpp:49-53
    b.lower = b.upper = 0;
    b.has_word = true;
    b.word.clear();
    return;
  }
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  AllocScope alloc_scope(E.stream);  // buffer growth ordered on this solve's stream only
  const Engine::Counting counting(E, st);
  auto t0 = std::chrono::steady_clock::now();
  const int n = (int)A.n, k = (int)A.k, W = words_for(n);
  const size_t budget = (size_t)cfg.max_memory_mb * 1024 * 1024;
  const size_t row_bytes = sizeof(u64) * W;
  // exact.cpp:65 searches lengths below the upper bound; when no word backs
  // that bound (it came from the plan's upper_bound), length == bound is
  // searched too so that a word can be returned.
  const u64 max_rt = b.has_word ? b.upper - 1 : b.upper;
  u64 rt = 0;
  const std::vector<uint32_t> seeds = backward_seeds(A);
  E.F.reset();
  E.B.reset();
  E.list_budget = budget;
  E.states_ordered = true;
  if (E.F.list_bytes() + E.B.list_bytes() > budget)  // left by a search of a larger budget
    for (DevBuf* b : {&E.F.vis, &E.F.vis_alt, &E.F.met, &E.F.table, &E.B.vis, &E.B.vis_alt, &E.B.met, &E.B.table})
      b->release();
  auto finish = [&] {
    st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  };
  // A search with duplicate removal only starts on one thread-block cluster
  // (the other reductions and reduced forward seeds are the streamed path's).
  bool imported = false, checked = false, synchronizing = false;
  ClusterExit single_exit{};
  if (!red && !b.has_word && cfg.reductions != SW_REDUCE_ALWAYS && !Engine::sort_key_option() && n <= 256 && n * k <= 4096 && !seeds.empty() &&
      max_rt > 0) {
    const Engine::Single S = E.run_single(A, seeds, (u32)std::min<u64>(max_rt, kClusterSingleWord), budget, [&] {
      synchronizing = is_synchronizing(A);
      checked = true;
      return synchronizing;
    });
    if (E.verbose)
      std::fprintf(stderr, "[sw] first levels on a cluster: status %u why %u, len %u, |F|=%u |B|=%u, %llu children\n",
                   S.res.status, S.res.why & 255u, S.res.length, S.exit.cnt[0], S.exit.cnt[1], S.exit.children);
    if (S.res.status == 0) {
      std::vector<uint32_t> word(S.word, S.word + S.res.word_len);
      if (word.size() != S.res.length || apply_word(A, word).size() != 1)
        throw std::runtime_error("internal error: the cluster search's word does not synchronize");
      b.lower = std::max<u64>(b.lower, S.res.length);
      b.upper = S.res.length;
      b.has_word = true;
      b.word = std::move(word);
      finish();
      return;
    }
    const u32 why = S.res.why & 255u;
    imported = S.res.status == 3 || (S.res.status == 1 && (why == 1 || why == 3 || why == 4)) ||
               (S.res.status == 2 && why == 9);
    if (imported) {
      single_exit = S.exit;
      rt = S.res.length;
    }
  }
  if (!(checked ? synchronizing : is_synchronizing(A))) {
    // The reference's Exact has no such check and runs until its bound; a
    // non-synchronizing automaton is reported as such instead.
    b.non_synchro = true;
    finish();
    return;
  }
  E.upload_tables(A);
  if (imported) {
    E.import_single(W, single_exit);
  } else {  // seeds
    const u32 nf = red ? red->seeds : 1;
    E.F.rows.reserve(sizeof(u64) * W * std::max<u32>(nf, 1));
    std::vector<u64> full(W, 0);
    std::vector<uint16_t> from(n);
    if (red) {
      // exact.cpp:130-146: the forward side starts from the reduced BFS list
      for (int q = 0; q < n; ++q) from[order[q]] = (uint16_t)red->states[q];
      E.red_states.reserve(sizeof(uint16_t) * n);
      SW_CUDA(cudaMemcpyAsync(E.red_states.p, from.data(), sizeof(uint16_t) * n, cudaMemcpyHostToDevice, E.stream));
      const int Wr = words_for((int)red->original.n);
      launch_relabel_rows(E.R.cur_rows(Wr), Wr, nf, E.red_states.as<uint16_t>(), n, E.F.rows.as<u64>(), W, E.stream);
      E.count_launch();
    } else {
      for (int q = 0; q < n; ++q) full[q >> 6] |= state_bit(q);
      SW_CUDA(cudaMemcpyAsync(E.F.rows.p, full.data(), sizeof(u64) * W, cudaMemcpyHostToDevice, E.stream));
    }
    E.F.count = nf;
    std::vector<u64> rows((size_t)W * std::max<size_t>(seeds.size(), 1), 0);
    for (size_t i = 0; i < seeds.size(); ++i) {
      for (int q = 0; q < n; ++q)
        if ((uint32_t)q != seeds[i]) rows[i * W + (q >> 6)] |= state_bit(q);  // complement of {seed}
    }
    E.B.rows.reserve(sizeof(u64) * rows.size());
    SW_CUDA(cudaMemcpyAsync(E.B.rows.p, rows.data(), sizeof(u64) * W * seeds.size(), cudaMemcpyHostToDevice,
                            E.stream));
    E.B.count = (u32)seeds.size();
    // visited starts with the seeds (the reference's visited lists start empty;
    // a seed can never be dominated by its own descendants' check either way)
    E.F.vis.reserve(sizeof(u64) * W);
    E.B.vis.reserve(sizeof(u64) * W * std::max<size_t>(seeds.size(), 1));
    SW_CUDA(cudaMemcpyAsync(E.F.vis.p, E.F.rows.p, sizeof(u64) * W, cudaMemcpyDeviceToDevice, E.stream));
    E.F.vis_count = red ? 0 : 1;  // a reduced list starts with an empty visited list, as the reference's does
    if (!seeds.empty()) {
      // seeds are already sorted ascending by state = descending by row value
      // for complements; sort them properly via the row sort.
      SW_CUDA(cudaMemcpyAsync(E.B.vis.p, E.B.rows.p, sizeof(u64) * W * seeds.size(), cudaMemcpyDeviceToDevice,
                              E.stream));
      E.sort_by_layer_key(W, E.B.vis.as<u64>(), (u32)seeds.size());
      E.B.vis_count = (u32)seeds.size();
    }
  }
  bool found = false, oom = false;
  u32 wit_q = 0, wit_s = 0;
  // Bounded inverse phase (the device counterpart of the reference's DFS
  // shortcut, dfs.cpp:64-218 and meet_in_the_middle.cpp:466-511): when the
  // upper bound is backed by a word, only lengths < bound remain to be
  // excluded.  F is then frozen and B is expanded level by level with
  // duplicate removal only, each level meet-checked against F.  The switch is
  // taken when the projected cost of those levels (measured per-query meet
  // time, B growing by the last observed branching) is below that of
  // continuing the dominance-pruned search (last step's time growing 1.5x per
  // step), and the widest projected level fits the memory budget.
  bool bounded = false;
  // Seconds of a step's and a meet check's launches, which do not grow with the
  // lists; below kSwitchRows rows they are all of it, and neither the times nor
  // the branching say anything about later levels (a switch at 145 rows, 29
  // levels before the bound, took 190 ms where 35 was enough).
  constexpr double kStepLaunch = 8e-5, kMeetLaunch = 1.5e-5;
  constexpr u32 kSwitchRows = 4096;
  Reduction reductions[2];
  double rest = 0;  // projected seconds to the end of the search (0: not known)
  double t_iter_last = 0, t_meet_per_query = 0, b_growth = k * 0.95;
  while (rt < max_rt) {  // meet_in_the_middle.cpp:73
    const auto t_iter0 = std::chrono::steady_clock::now();
    const bool fwd = bounded ? false : E.F.count <= E.B.count;
    Side& X = fwd ? E.F : E.B;
    size_t live = (size_t)(E.F.count + E.F.vis_count + E.B.count + E.B.vis_count) * row_bytes;
    size_t next = (size_t)X.count * k * (3 * row_bytes + 4 * sizeof(u32));
    if (live + next > budget) {
      // meet_in_the_middle.cpp:98-101 + exact.cpp:139-145: out of memory, the
      // search continues in the memory-bounded inverse phase when DFS is
      // enabled and the remaining depth is bounded (word-backed bound or at
      // most 64 levels); otherwise only a lower bound results.  Plans that reduce
      // for memory only and have a word behind the bound switch there by cost at
      // any level, DFS or not, and so go on at the budget too: while the switch
      // still came within the first levels of such plans (below kSwitchRows) they
      // never met the budget
      const bool goes_on = cfg.dfs || (b.has_word && cfg.reductions == SW_REDUCE_MEMORY);
      if (goes_on && !bounded && E.B.count && (b.has_word || max_rt - rt <= 64)) {
        bounded = true;
        if (E.verbose)
          std::fprintf(stderr, "[sw] memory budget reached at length %llu: bounded phase\n", (unsigned long long)rt);
        break;
      }
      oom = true;
      break;
    }
    rt++;
    const u32 parents_before = X.count;
    const bool pressure = 4 * (live + next) > budget;
    Reduction& red_last = reductions[fwd];
    const LevelRule level =
        reductions_of_level((int)cfg.reductions, b.has_word, cfg.dfs != 0, pressure, red_last, X.count, rest);
    E.reductions = level.reduce;
    E.step(X, fwd, W, n, k, /*dominance=*/!bounded, false, /*defer=*/true);
    if (fwd) {
      st.bfs_steps++;
    } else {
      st.ibfs_steps++;
    }
    // meet check: some F disjoint from some B-complement (F ⊆ B)
    const double t_meet0 = E.vclock();
    // the switch to the bounded phase prices the meet check per query: it is timed
    // while that switch is possible
    const bool time_meet = !bounded && b.has_word;
    if (time_meet) E.meet_span.mark(0, E.stream);
    SW_CUDA(cudaMemsetAsync(E.d_misc, 0, 4 * sizeof(u32), E.stream));
    E.query(W, kQueryDisjoint, E.F.cur_rows(W), E.F.count, E.B.cur_rows(W), E.B.count, n, nullptr, true, E.F.live,
            E.B.live);
    if (time_meet) E.meet_span.mark(1, E.stream);
    // the one read-back of a level: witness, error, the step's counts (a reduced
    // level read back four times: n=100 plans of ~19 levels 2.7 -> 2.4 ms, plain
    // n=200 levels twice: 3.1 -> 2.9 ms)
    SW_CUDA(cudaMemcpyAsync(E.pinned.p, E.d_misc, Engine::kStepWords * sizeof(u32), cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    const auto t_end = std::chrono::steady_clock::now();
    u32 w[Engine::kStepWords];
    std::copy(E.pinned.as<u32>(), E.pinned.as<u32>() + Engine::kStepWords, w);
    E.check_scan_error(w[Engine::kScanErrWord]);
    if (X.live) {
      E.finish_step(X, w);
      E.count_query(E.F.count, E.B.count);
    }
    st.meet_pairs += (u64)E.F.count * E.B.count;
    if (X.hashed && X.step.compacted && X.step.distinct && time_meet)
      red_last = Reduction{E.reduce_span.seconds(), 1.0 - (double)X.step.kept / X.step.distinct, X.step.parents};
    // projected branching of the bounded levels: distinct children per parent
    // before pruning, never below 1.2
    if (!fwd && parents_before) b_growth = std::max(1.2, E.B.unique_growth);
    t_iter_last = std::chrono::duration<double>(t_end - t_iter0).count();
    if (E.B.count && time_meet) t_meet_per_query = E.meet_span.seconds() / (double)E.B.count;
    if (!bounded && b.has_word && !w[0] && rt < max_rt && rt >= 4 && E.B.count >= kSwitchRows) {
      const u64 R = max_rt - rt;  // levels still to exclude
      // per child: expansion and hash table (0.12-0.25 ns measured at 10^7
      // rows) + the meet check's cost per query.  Continuing costs 1.5x more
      // per length: the sides alternate, each list grows ~1.7x when its turn
      // comes and the dominance checks with its square (0.8, 1.5, 3.4, 6, 10 ms
      // measured for five lengths at n=300).  With the 2 ns and 1.35x that the
      // sorted levels cost, the switch came one or two lengths later: n=256
      // 70.8 -> 56 ms, n=300 within 5% either way.
      const double per_row = std::max(t_meet_per_query - kMeetLaunch / (double)E.B.count, 0.0) + 2.5e-10;
      t_iter_last = std::max(t_iter_last - kStepLaunch, 0.0);
      double lvl = E.B.count, total = 0, mitm = 0, grow = 1.0;
      bool fits = true;
      for (u64 i = 1; i <= R && fits; ++i) {
        const double children = lvl * k;
        total += children * per_row;
        grow *= 1.5;
        mitm += kStepLaunch + t_iter_last * grow;
        // children rows + their sorted copy + the kept level, keys and payloads
        if (children * (3.0 * row_bytes + 32) + (lvl + (double)E.F.count) * row_bytes > (double)budget)
          fits = false;
        lvl *= b_growth;
      }
      // without the checks' own time, which is what the rest is held against
      const double checks = X.hashed && X.step.compacted ? std::min(red_last.seconds, t_iter_last) : 0.0;
      const double plain = mitm * (1.0 - checks / std::max(t_iter_last, 1e-9));
      const double lists =
          (double)(E.F.count + E.F.vis_count + E.B.count + E.B.vis_count) * (double)row_bytes;
      rest = fits ? std::min(total, plain) : lists_stay_small(lists, R, (double)budget) ? plain : 0.0;
      // voluntary switch only when every projected level fits; chunking is the
      // safety net for an exhausted budget, not a plan
      if (fits && total * (level.left_out ? kSwitchUnreduced : 1.0) < mitm) {
        bounded = true;
        if (E.verbose)
          std::fprintf(stderr, "[sw] bounded phase from length %llu: %llu levels left, |F|=%u |B|=%u, "
                       "projected %.1f ms vs %.1f ms\n", (unsigned long long)rt, (unsigned long long)R, E.F.count,
                       E.B.count, 1e3 * total, 1e3 * mitm);
      }
    }
    if (E.verbose)
      std::fprintf(stderr, "[sw] len %llu: |F|=%u |B|=%u meet check %.3f ms%s\n", (unsigned long long)rt, E.F.count,
                   E.B.count, E.vclock() - t_meet0, w[0] ? " -> found" : "");
    if (w[0]) {
      found = true;
      wit_q = w[1];
      wit_s = w[2];
      break;
    }
    if (E.F.count == 0 || E.B.count == 0) break;  // a side died out: no reset word within reach
    if (bounded) break;
  }
  std::vector<uint32_t> bounded_tail;
  if (bounded && !found) {
    BoundedSearch S{E, A, W, n, k, budget, row_bytes, std::max<u64>(cfg.dfs_min_list_size, 1), max_rt, 0, {}, 0,
                    {}, {}, st};
    if (4 * (E.F.list_bytes() + E.B.list_bytes()) > budget) E.release_tables();
    S.pool.swap(E.dlevel_pool);  // levels (and their device buffers) kept across solves
    S.levels.push_back(nullptr);
    S.explore(0, 0, E.B.count, rt);
    E.dlevel_pool.swap(S.pool);
    if (S.best) {
      found = true;
      rt = S.best;
      wit_s = S.best_f;
      bounded_tail = S.best_tail;
    } else {
      rt = max_rt;  // every length up to the bound minus one is excluded
    }
  }
  if (red) {  // exact.cpp:83-87: lengths count the reduction's BFS steps
    rt += red->bfs_steps;
    b.lower += red->bfs_steps;
    b.upper += red->bfs_steps;
  }
  if (found) {
    // word = (reduction prefix) forward letters (depth 1..df) then backward
    // letters (depth db..1)
    u32 fseed = 0;
    std::vector<uint32_t> fw = E.trace(E.F, wit_s, &fseed);
    std::reverse(fw.begin(), fw.end());
    u32 seed_idx = 0;
    std::vector<uint32_t> bw = bounded_tail.empty() ? E.trace(E.B, wit_q, &seed_idx) : bounded_tail;
    std::vector<uint32_t> word;
    if (red) {
      word = E.trace(E.R, fseed, nullptr);
      std::reverse(word.begin(), word.end());
    }
    word.insert(word.end(), fw.begin(), fw.end());
    word.insert(word.end(), bw.begin(), bw.end());
    std::vector<uint32_t> img = apply_word(red ? red->original : A, word);
    if (img.size() != 1 || word.size() != rt)
      throw std::runtime_error("internal error: reconstructed word does not synchronize (length " +
                               std::to_string(word.size()) + ", image " + std::to_string(img.size()) + ")");
    b.lower = std::max<u64>(b.lower, rt);
    b.upper = rt;
    b.has_word = true;
    b.word = word;
  } else {
    // exact.cpp:148-164: every length <= rt is excluded; if that reaches the
    // upper bound, the bound is the answer (its word, if any, came from the
    // algorithm that set it).  Otherwise (memory budget) only a lower bound.
    (void)oom;
    if (rt + 1 >= b.upper) {
      b.lower = std::max<u64>(b.lower, b.upper);
    } else {
      b.lower = std::max<u64>(b.lower, rt + 1);
    }
  }
  finish();
}

// ---------------------------------------------------------------------------
// Beam (beam.hpp:31-188): inverse BFS from the backward seeds keeping the
// `beam_size` largest sets, ties by the reference's raw word order.
// ---------------------------------------------------------------------------
namespace {
struct BeamRun {
  u64 bound = 0;
  bool has_word = false;
  std::vector<uint32_t> word;
};
}  // namespace

static BeamRun beam_cutoff(Engine& E, const Automaton& A, u32 beam_size, u64 max_mlsw, int64_t max_iter, sw_stats& st) {
  const int n = (int)A.n, k = (int)A.k, W = words_for(n);
  const int R = (n + 63) / 64 + 1;
  BeamRun out;
  out.bound = max_mlsw;
  std::vector<uint32_t> seeds = backward_seeds(A);
  Side& X = E.B;  // beam rows are plain (not complemented) preimages
  X.reset();
  std::vector<u64> rows((size_t)W * std::max<size_t>(seeds.size(), 1), 0);
  for (size_t i = 0; i < seeds.size(); ++i) rows[i * W + (seeds[i] >> 6)] |= state_bit((int)seeds[i]);
  const u64 parents = std::max<u64>(beam_size, seeds.size());
  const bool one_cta = beam_fits(W, (u32)n, (u32)k, parents);
  X.rows.reserve(sizeof(u64) * std::max<size_t>(rows.size(), one_cta ? W * parents : 0));
  SW_CUDA(cudaMemcpyAsync(X.rows.p, rows.data(), sizeof(u64) * W * seeds.size(), cudaMemcpyHostToDevice, E.stream));
  X.count = (u32)seeds.size();
  if (X.count == 0 || beam_size == 0 || max_mlsw == 0) return out;
  if (one_cta) {
    // Beams whose children fit in one CTA's shared memory run there (still the
    // faster side at the largest that fit: n=256 beam 2048 123 us a level over
    // the whole GPU, 64 here; n=100 beam 3000 127 and 54), up to kBeamLevels
    // levels a launch; earlier launches' origins are kept on the host.
    const u64 most = max_iter >= 0 ? std::min<u64>(max_mlsw - 1, (u64)max_iter) : max_mlsw - 1;
    E.beam_log.reserve(sizeof(u32) * parents * kBeamLevels);
    E.beam_out.reserve(sizeof(u32) * kBeamOutWords);
    struct Part {
      std::vector<u32> log, parents;  // per level: kept origins, parent count
    };
    std::vector<Part> parts;
    u32 m = X.count;
    for (u64 len = 0; len < most;) {
      const u32 levels = (u32)std::min<u64>(most - len, kBeamLevels);
      launch_beam(W, E.tables.delta, (u32)n, (u32)k, beam_size, m, (u32)parents, levels, X.rows.as<u64>(),
                  E.beam_log.as<u32>(), E.beam_out.as<u32>(), E.stream);
      E.count_launch();
      SW_CUDA(cudaMemcpyAsync(E.pinned.p, E.beam_out.p, sizeof(u32) * kBeamOutWords, cudaMemcpyDeviceToHost, E.stream));
      SW_CUDA(cudaStreamSynchronize(E.stream));
      const u32 *o = E.pinned.as<u32>(), *counts = o + kBeamHeader + kBeamLevels;
      for (u32 l = 0; l < o[1]; ++l) st.subsets_expanded += (u64)counts[l] * k;
      len += o[1];
      if (o[0]) {
        // word: letters from this layer down to the first, applied in that order
        out.word.assign(o + kBeamHeader, o + kBeamHeader + o[1]);
        u32 idx = o[3];
        for (size_t i = parts.size(); i-- > 0;)
          for (size_t d = parts[i].parents.size(); d-- > 0;) {
            const u32 v = parts[i].log[d * parents + idx];
            out.word.push_back(v / parts[i].parents[d]);
            idx = v % parts[i].parents[d];
          }
        out.bound = len;
        std::vector<uint32_t> img = apply_word(A, out.word);
        out.has_word = img.size() == 1 && out.word.size() == len;
        return out;
      }
      m = o[2];
      if (len < most) {
        parts.emplace_back();
        parts.back().parents.assign(counts, counts + levels);
        parts.back().log.resize((size_t)levels * parents);
        SW_CUDA(cudaMemcpyAsync(parts.back().log.data(), E.beam_log.p, sizeof(u32) * levels * parents,
                                cudaMemcpyDeviceToHost, E.stream));
        SW_CUDA(cudaStreamSynchronize(E.stream));
      }
    }
    return out;
  }
  for (u64 len = 1; len < max_mlsw; ++len) {
    if (max_iter >= 0 && (int64_t)len > max_iter) break;
    const u32 m = X.count;
    const u64 N = (u64)m * k;
    if (N > 0xffffffffULL) throw std::runtime_error("beam layer exceeds 2^32 children");
    const u32 Nc = (u32)N;
    E.ch_rows.reserve(sizeof(u64) * W * N);
    E.keys.reserve(sizeof(u64) * R * N);
    E.ch_vals.reserve(sizeof(u32) * N);
    E.flags_a.reserve(sizeof(u32) * N);
    E.uq_vals.reserve(sizeof(u32) * N);
    E.keys_alt.reserve(sizeof(u64) * R * N);
    E.timed(1, (double)m * 8.0 * W * (1 + k), [&] {
      launch_expand(W, false, X.rows.as<u64>(), m, E.tables, E.ch_rows.as<u64>(), E.stream);
    });
    launch_beam_keys(W, E.ch_rows.as<u64>(), Nc, n, R, E.keys.as<u64>(), E.stream);
    launch_iota(E.ch_vals.as<u32>(), Nc, E.stream);
    E.count_launch(3);
    st.subsets_expanded += N;
    E.sort_rows(R, E.keys.as<u64>(), E.ch_vals.as<u32>(), Nc);
    // beam.hpp:173-177: the largest set is first; Q means done
    SW_CUDA(cudaMemcpyAsync(E.pinned.p, E.keys.p, sizeof(u64), cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    if (*E.pinned.as<u64>() == 0) {
      u32 first_val = 0;
      SW_CUDA(cudaMemcpy(&first_val, E.ch_vals.p, sizeof(u32), cudaMemcpyDeviceToHost));
      // word: letters from this layer down to the first, applied in that order
      std::vector<uint32_t> letters;
      letters.push_back(first_val / m);
      u32 idx = first_val % m;
      for (size_t d = X.layers.size(); d-- > 0;) {
        const Layer& L = *X.layers[d];
        u32 o = E.read_u32(L.org() + idx);
        letters.push_back(o / L.parent_count);
        idx = o % L.parent_count;
      }
      out.bound = len;
      out.word = letters;
      std::vector<uint32_t> img = apply_word(A, out.word);
      out.has_word = img.size() == 1 && out.word.size() == len;
      return out;
    }
    // keep_unique + truncate (beam.hpp:179-182)
    launch_unique_flags(R, E.keys.as<u64>(), Nc, E.flags_a.as<u32>(), E.stream);
    E.count_launch();
    E.uq_rows.reserve(sizeof(u64) * R * N);
    u32 u = E.compact(R, E.keys.as<u64>(), E.ch_vals.as<u32>(), E.flags_a.as<u32>(), Nc, E.uq_rows.as<u64>(),
                      E.uq_vals.as<u32>());
    u32 keep = std::min<u32>(u, beam_size);
    X.rows_alt.reserve(sizeof(u64) * W * std::max<u32>(keep, 1));
    launch_gather_rows(W, E.ch_rows.as<u64>(), E.uq_vals.as<u32>(), keep, X.rows_alt.as<u64>(), E.stream);
    E.count_launch();
    std::swap(X.rows.p, X.rows_alt.p);
    std::swap(X.rows.cap, X.rows_alt.cap);
    auto L = X.new_layer(sizeof(u32) * std::max<u32>(keep, 1));
    L->origin.reserve(sizeof(u32) * std::max<u32>(keep, 1));
    SW_CUDA(cudaMemcpyAsync(L->origin.p, E.uq_vals.p, sizeof(u32) * keep, cudaMemcpyDeviceToDevice, E.stream));
    L->count = keep;
    L->parent_count = m;
    X.layers.push_back(std::move(L));
    X.count = keep;
  }
  return out;
}

void Solver::beam(const Automaton& A0, const sw_beam_config& cfg, Bounds& b, sw_stats& st) {
  if (b.non_synchro || b.lower == b.upper) return;  // beam.hpp:34-40
  if (A0.n == 1) {                                  // beam.hpp:42-46
    b.lower = b.upper = 0;
    b.has_word = true;
    b.word.clear();
    return;
  }
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  AllocScope alloc_scope(E.stream);  // buffer growth ordered on this solve's stream only
  const Engine::Counting counting(E, st);
  auto t0 = std::chrono::steady_clock::now();
  // presort (beam.hpp:54-63, 351-369): states ordered by in-degree ascending
  std::vector<uint32_t> perm(A0.n);
  std::iota(perm.begin(), perm.end(), 0u);
  if (cfg.presort_indeg) {
    std::vector<std::pair<double, int>> d(A0.n);
    for (uint32_t q = 0; q < A0.n; ++q) d[q] = {0.0, (int)q};
    for (uint32_t q = 0; q < A0.n; ++q)
      for (uint32_t a = 0; a < A0.k; ++a) d[A0.at(q, a)].first++;
    std::sort(d.begin(), d.end());
    for (uint32_t q = 0; q < A0.n; ++q) perm[d[q].second] = q;
  }
  Automaton A = permute(A0, perm);
  E.upload_tables(A);
  BeamRun run;
  if (cfg.dynamic) {  // beam.hpp:66-86
    using cost_t = long double;
    const uint32_t minb = (uint32_t)cfg.min_beam_size, maxb = (uint32_t)cfg.max_beam_size;
    run = beam_cutoff(E, A, minb, b.upper, cfg.max_iter, st);
    uint32_t bound = (uint32_t)run.bound;
    cost_t exact_cost = 2 * std::pow(static_cast<cost_t>(A.k), (bound + 1) / 2);
    cost_t proposed = std::round(exact_cost * (cost_t)cfg.beam_exact_ratio / bound);
    uint32_t bs = (uint32_t)std::clamp<cost_t>(proposed, (cost_t)minb, (cost_t)maxb);
    if (bs > minb) {
      // the second run searches below the first bound; it returns that bound
      // unchanged (and no word) when it finds nothing shorter
      BeamRun second = beam_cutoff(E, A, bs, bound, cfg.max_iter, st);
      if (second.bound < bound) run = second;
    }
  } else {
    run = beam_cutoff(E, A, (uint32_t)cfg.beam_size, b.upper, cfg.max_iter, st);
  }
  const uint32_t bound = (uint32_t)run.bound;  // the reference stores the bound in a uint
  b.upper = bound;
  if (run.has_word && run.word.size() == bound) {
    b.has_word = true;
    b.word = run.word;
  } else if (b.has_word && b.word.size() != b.upper) {
    b.has_word = false;
  }
  st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// ---------------------------------------------------------------------------
// Kernel-level helpers.
// ---------------------------------------------------------------------------
void Solver::apply_transition(const Automaton& A, uint32_t letter, bool inverse, const uint64_t* from, uint64_t* to,
                              uint64_t count) {
  if (letter >= A.k) throw std::invalid_argument("letter out of range");
  if (count == 0) return;
  if (count > 0xffffffffULL) throw std::invalid_argument("count exceeds 2^32");
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const int n = (int)A.n, W = words_for(n);
  // single-letter automaton view so the kernel writes one block
  Automaton one;
  one.n = A.n;
  one.k = 1;
  one.t.resize(A.n);
  for (uint32_t q = 0; q < A.n; ++q) one.t[q] = A.at(q, letter);
  E.upload_tables(one);
  const size_t bytes = sizeof(u64) * (size_t)W * count;
  E.uq_rows.reserve(bytes);
  E.ch_rows.reserve(bytes);
  SW_CUDA(cudaMemcpyAsync(E.uq_rows.p, from, bytes, cudaMemcpyHostToDevice, E.stream));
  launch_convert_rows(W, E.uq_rows.as<u64>(), count, n, true, E.stream);
  launch_expand(W, !inverse, E.uq_rows.as<u64>(), (u32)count, E.tables, E.ch_rows.as<u64>(), E.stream);
  launch_convert_rows(W, E.ch_rows.as<u64>(), count, n, false, E.stream);
  SW_CUDA(cudaMemcpyAsync(to, E.ch_rows.p, bytes, cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
}

void Solver::subsets_check(uint32_t n, const uint64_t* sets, uint64_t set_count, const uint64_t* checks,
                           uint64_t check_count, bool proper, uint8_t* results) {
  if (n == 0 || n > (uint32_t)kMaxStates) throw std::invalid_argument("n out of range");
  if (set_count > 0xffffffffULL || check_count > 0xffffffffULL) throw std::invalid_argument("count exceeds 2^32");
  std::fill(results, results + check_count, 0);
  if (!set_count || !check_count) return;
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const int W = words_for((int)n);
  const u32 m = (u32)set_count, q = (u32)check_count;
  const size_t sbytes = sizeof(u64) * (size_t)W * m, qbytes = sizeof(u64) * (size_t)W * q;
  E.uq_rows.reserve(sbytes);
  E.uq_vals.reserve(sizeof(u32) * m);
  E.ch_rows.reserve(qbytes);
  E.flags_a.reserve(sizeof(u32) * m);
  E.flags_b.reserve(sizeof(u32) * q);
  E.keys.reserve(sbytes);
  SW_CUDA(cudaMemcpyAsync(E.uq_rows.p, sets, sbytes, cudaMemcpyHostToDevice, E.stream));
  SW_CUDA(cudaMemcpyAsync(E.ch_rows.p, checks, qbytes, cudaMemcpyHostToDevice, E.stream));
  launch_convert_rows(W, E.uq_rows.as<u64>(), m, (int)n, true, E.stream);
  launch_convert_rows(W, E.ch_rows.as<u64>(), q, (int)n, true, E.stream);
  // sort + unique the set list (check_contains_subset sorts both, :30-33)
  launch_iota(E.uq_vals.as<u32>(), m, E.stream);
  E.sort_rows(W, E.uq_rows.as<u64>(), E.uq_vals.as<u32>(), m);
  launch_unique_flags(W, E.uq_rows.as<u64>(), m, E.flags_a.as<u32>(), E.stream);
  u32 u = E.compact(W, E.uq_rows.as<u64>(), E.uq_vals.as<u32>(), E.flags_a.as<u32>(), m, E.keys.as<u64>(), nullptr);
  launch_fill_u32(E.flags_b.as<u32>(), 0, q, E.stream);
  E.query(W, proper ? kQueryProperSubset : kQuerySubset, E.keys.as<u64>(), u,
          E.ch_rows.as<u64>(), q, (int)n, E.flags_b.as<u32>(), false);
  std::vector<u32> flags(q);
  SW_CUDA(cudaMemcpyAsync(flags.data(), E.flags_b.p, sizeof(u32) * q, cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
  for (u32 i = 0; i < q; ++i) results[i] = flags[i] ? 1 : 0;
}

uint64_t Solver::sort_unique(uint32_t n, uint64_t* sets, uint64_t count) {
  if (n == 0 || n > (uint32_t)kMaxStates) throw std::invalid_argument("n out of range");
  if (count > 0xffffffffULL) throw std::invalid_argument("count exceeds 2^32");
  if (count == 0) return 0;
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const int W = words_for((int)n);
  const u32 m = (u32)count;
  const size_t bytes = sizeof(u64) * (size_t)W * m;
  E.uq_rows.reserve(bytes);
  E.uq_vals.reserve(sizeof(u32) * m);
  E.keys.reserve(bytes);
  E.flags_a.reserve(sizeof(u32) * m);
  SW_CUDA(cudaMemcpyAsync(E.uq_rows.p, sets, bytes, cudaMemcpyHostToDevice, E.stream));
  launch_convert_rows(W, E.uq_rows.as<u64>(), m, (int)n, true, E.stream);
  launch_iota(E.uq_vals.as<u32>(), m, E.stream);
  E.sort_rows(W, E.uq_rows.as<u64>(), E.uq_vals.as<u32>(), m);
  launch_unique_flags(W, E.uq_rows.as<u64>(), m, E.flags_a.as<u32>(), E.stream);
  u32 u = E.compact(W, E.uq_rows.as<u64>(), E.uq_vals.as<u32>(), E.flags_a.as<u32>(), m, E.keys.as<u64>(), nullptr);
  launch_convert_rows(W, E.keys.as<u64>(), u, (int)n, false, E.stream);
  SW_CUDA(cudaMemcpyAsync(sets, E.keys.p, sizeof(u64) * W * u, cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
  return u;
}

// ---------------------------------------------------------------------------
// Eppstein (synchrolib/algorithm/eppstein/eppstein.hpp:26-76).
// ---------------------------------------------------------------------------
void Solver::eppstein(const Automaton& A, const sw_eppstein_config&, Bounds& b, sw_stats& st) {
  if (b.non_synchro || b.lower == b.upper) return;  // eppstein.hpp:28-34
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  auto t0 = std::chrono::steady_clock::now();
  E.upload_tables(A);
  const u64 n = A.n;
  E.epp_scratch.reserve(eppstein_scratch_bytes((int)n));
  // the greedy word is at most (n^3 - n) / 6 letters long (Eppstein 1990)
  const u64 cap = std::min<u64>(b.upper, n * n * n / 6 + n) + 1;
  E.epp_word.reserve(cap);
  u32* out = E.d_misc + 16;
  SW_CUDA(cudaMemsetAsync(out, 0, 8 * sizeof(u32), E.stream));
  launch_eppstein(E.tables, b.upper, E.epp_scratch.p, out, E.epp_word.as<uint8_t>(), cap, E.stream);
  ++st.kernel_launches;
  u32* h = E.pinned.as<u32>();
  SW_CUDA(cudaMemcpyAsync(h, out, 8 * sizeof(u32), cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
  const u32 status = h[0];
  const u64 len = (u64)h[1] | ((u64)h[2] << 32);
  const u64 letters = h[3];
  st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  if (status == kEppNonSynchro) {  // eppstein.hpp:53-57
    b.non_synchro = true;
    return;
  }
  if (status == kEppOverBound) return;  // eppstein.hpp:60-62: bound unchanged
  if (status != kEppFound) throw std::runtime_error("internal: Eppstein word buffer too small");
  const u64 old_upper = b.upper;
  b.upper = len;
  if (letters == len) {
    std::vector<uint8_t> w8(letters);
    if (letters) SW_CUDA(cudaMemcpy(w8.data(), E.epp_word.p, letters, cudaMemcpyDeviceToHost));
    std::vector<uint32_t> word(w8.begin(), w8.end());
    if (apply_word(A, word).size() != 1) throw std::runtime_error("internal: Eppstein word does not synchronize");
    if (!b.has_word || len < old_upper) {
      b.has_word = true;
      b.word = std::move(word);
    }
  }
  if (b.has_word && b.word.size() != b.upper) b.has_word = false;
}

// ---------------------------------------------------------------------------
// Brute (synchrolib/algorithm/brute/brute.hpp:28-71).
// ---------------------------------------------------------------------------
void Solver::brute(const Automaton& A, const sw_brute_config& cfg, Bounds& b, sw_stats& st) {
  if (b.non_synchro || b.lower == b.upper) return;  // brute.hpp:30-36
  if (cfg.max_n > 32) return;                       // brute.hpp:44-47: refused, bounds unchanged
  if (A.n > cfg.max_n) return;                      // brute.hpp:49-52
  if (A.n == 1) {
    b.lower = b.upper = 0;
    b.has_word = true;
    b.word.clear();
    return;
  }
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  auto t0 = std::chrono::steady_clock::now();
  E.upload_tables(A);
  const int n = (int)A.n, k = (int)A.k;
  const u64 space = 1ULL << n;  // masks; every level holds new masks only, so all levels fit in `space`
  const u32 full = n == 32 ? 0xffffffffu : ((1u << n) - 1u);
  E.br_visited.reserve(brute_visited_bytes(n));
  SW_CUDA(cudaMemsetAsync(E.br_visited.p, 0, brute_visited_bytes(n), E.stream));
  const u32 full_bit = 1u << (full & 31u);
  SW_CUDA(cudaMemcpyAsync(E.br_visited.as<u32>() + (full >> 5), &full_bit, sizeof(u32), cudaMemcpyHostToDevice,
                          E.stream));
  E.br_arena.reserve(sizeof(u32) * std::min<u64>(space, 1ULL << 20));
  SW_CUDA(cudaMemcpyAsync(E.br_arena.p, &full, sizeof(u32), cudaMemcpyHostToDevice, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
  std::vector<u64> off{0, 1};  // level j = arena[off[j], off[j+1])
  u32* ctrl = E.d_misc + 24;   // [0] next count, [1] found, [2] singleton
  u32* h = E.pinned.as<u32>();
  u64 length = 0;
  u32 target = 0;
  for (u64 depth = 0;; ++depth) {
    const u64 begin = off[depth], end = off[depth + 1], count = end - begin;
    const u64 room = std::min<u64>(count * (u64)k, space - end);
    const size_t need = sizeof(u32) * (end + room);
    if (need > E.br_arena.cap) {  // grow, keeping the stored levels
      DevBuf bigger;
      bigger.reserve(std::max(need, 2 * E.br_arena.cap));
      SW_CUDA(cudaMemcpyAsync(bigger.p, E.br_arena.p, sizeof(u32) * end, cudaMemcpyDeviceToDevice, E.stream));
      SW_CUDA(cudaStreamSynchronize(E.stream));
      std::swap(bigger.p, E.br_arena.p);
      std::swap(bigger.cap, E.br_arena.cap);
    }
    u32* arena = E.br_arena.as<u32>();
    SW_CUDA(cudaMemsetAsync(ctrl, 0, 3 * sizeof(u32), E.stream));
    launch_brute_level(E.t_delta.as<uint16_t>(), n, k, arena + begin, (u32)count, E.br_visited.as<u32>(), arena + end,
                       (u32)room, ctrl, ctrl + 1, E.stream);
    ++st.kernel_launches;
    SW_CUDA(cudaMemcpyAsync(h, ctrl, 3 * sizeof(u32), cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    st.subsets_expanded += count * (u64)k;
    st.subsets_kept += h[0];
    if (h[0] > room) throw std::runtime_error("internal: Brute level overflow");
    if (h[1]) {
      length = depth + 1;
      target = h[2];
      break;
    }
    if (h[0] == 0) {  // brute.hpp:61-65: BFS exhausted without a singleton
      b.non_synchro = true;
      st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
      return;
    }
    off.push_back(end + h[0]);
  }
  // walk back through the stored levels: a parent of `target` in level j
  std::vector<uint32_t> word(length);
  u64* best = reinterpret_cast<u64*>(E.d_misc + 32);
  for (u64 j = length; j-- > 0;) {
    const u64 begin = off[j], count = off[j + 1] - begin;
    SW_CUDA(cudaMemsetAsync(best, 0xff, sizeof(u64), E.stream));
    launch_brute_parent(E.t_delta.as<uint16_t>(), n, k, E.br_arena.as<u32>() + begin, (u32)count, target, best,
                        E.stream);
    ++st.kernel_launches;
    u64 hb = 0;
    SW_CUDA(cudaMemcpyAsync(h, best, sizeof(u64), cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    std::memcpy(&hb, h, sizeof(u64));
    if (hb == ~0ULL) throw std::runtime_error("internal: Brute parent not found");
    word[j] = (uint32_t)(hb % (u64)k);
    SW_CUDA(cudaMemcpy(&target, E.br_arena.as<u32>() + begin + hb / (u64)k, sizeof(u32), cudaMemcpyDeviceToHost));
  }
  if (apply_word(A, word).size() != 1) throw std::runtime_error("internal: Brute word does not synchronize");
  b.lower = b.upper = length;  // brute.hpp:66-70
  b.has_word = true;
  b.word = std::move(word);
  st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// ---------------------------------------------------------------------------
// Reduce (synchrolib/algorithm/reduce/reduce.hpp:31-91).  The BFS steps are
// the forward side of the exact search (expansion, duplicate removal, the two
// dominance checks, visited merge); the reachability closure and relabelling
// of the small final list are host bookkeeping.
// ---------------------------------------------------------------------------
void Solver::reduce(const Automaton& A, const sw_reduce_config& cfg, Bounds& b, sw_stats& st, ReduceState& red) {
  if (b.non_synchro || b.lower == b.upper) return;  // reduce.hpp:40-46
  if (A.n < cfg.min_n) return;                      // reduce.hpp:48-50
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const Engine::Counting counting(E, st);
  auto t0 = std::chrono::steady_clock::now();
  const int n = (int)A.n, k = (int)A.k, W = words_for(n);
  E.upload_tables(A);
  E.reductions = true;  // the reference's step (reduce.hpp:186-187): its list sizes decide the reduction
  E.R.reset();
  std::vector<u64> full(W, 0);
  for (int q = 0; q < n; ++q) full[q >> 6] |= state_bit(q);
  E.R.rows.reserve(sizeof(u64) * W);
  SW_CUDA(cudaMemcpyAsync(E.R.rows.p, full.data(), sizeof(u64) * W, cudaMemcpyHostToDevice, E.stream));
  E.R.count = 1;
  E.R.vis_count = 0;  // reduce.hpp:128: the visited list starts empty
  const u64 max_mlsw = b.upper - 1;
  u64 mlsw = 0;
  bool found = false;
  std::vector<uint32_t> word;
  auto done = [&] {
    st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  };
  u64* const sum = reinterpret_cast<u64*>(E.d_misc + 32);  // the list's union, then ~(its first single-state set)
  const size_t sum_bytes = 8 * sizeof(u64) + sizeof(u32);
  // reduce.hpp:96-109 (process_short_bfs) with bfs_step :171-198
  while (mlsw < max_mlsw) {
    if (E.R.count > cfg.list_size_threshold) break;
    mlsw++;
    st.bfs_steps++;
    if (E.R.count == 0) continue;  // an exhausted list stays empty up to the bound, as in the reference
    E.step(E.R, true, W, n, k, true, false, /*defer=*/true);
    if (!E.R.count) continue;
    SW_CUDA(cudaMemsetAsync(sum, 0, sum_bytes, E.stream));
    launch_list_summary(W, E.R.cur_rows(W), E.R.count, sum, reinterpret_cast<u32*>(sum + 8), E.stream, E.R.live);
    E.count_launch();
    SW_CUDA(cudaMemcpyAsync(E.pinned.p, E.d_misc, 32 * sizeof(u32) + sum_bytes, cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    if (E.R.live) E.finish_step(E.R, E.pinned.as<u32>());
    if (!E.R.count) continue;
    std::copy(E.pinned.as<u64>() + 16, E.pinned.as<u64>() + 16 + W, full.begin());
    const u32 single = E.pinned.as<u32>()[48];
    if (single) {
      word = E.trace(E.R, ~single, nullptr);
      std::reverse(word.begin(), word.end());
      found = true;
      break;
    }
  }
  if (!found && mlsw == max_mlsw) {  // reduce.hpp:60-63: every shorter length is excluded
    mlsw++;
    if (b.has_word && b.word.size() != mlsw) b.has_word = false;
    b.lower = b.upper = mlsw;
    return done();
  }
  if (found) {  // reduce.hpp:65-70
    if (apply_word(A, word).size() != 1 || word.size() != mlsw)
      throw std::runtime_error("internal: Reduce word does not synchronize");
    b.lower = b.upper = mlsw;
    b.has_word = true;
    b.word = word;
    return done();
  }
  // reduce.hpp:112-143 (try_to_reduce): states reachable from the list
  std::vector<char> reach(n, 0);
  std::vector<uint32_t> stack;
  for (int q = 0; q < n && E.R.count; ++q)
    if (full[q >> 6] & state_bit(q)) {
      reach[q] = 1;
      stack.push_back((uint32_t)q);
    }
  while (!stack.empty()) {  // reduce.hpp:145-169
    const uint32_t q = stack.back();
    stack.pop_back();
    for (int a = 0; a < k; ++a) {
      const uint32_t p = A.at(q, (uint32_t)a);
      if (!reach[p]) {
        reach[p] = 1;
        stack.push_back(p);
      }
    }
  }
  uint32_t rn = 0;
  std::vector<uint32_t> map(n, 0);
  for (int q = 0; q < n; ++q)
    if (reach[q]) map[q] = rn++;
  if (rn == (uint32_t)n || rn == 0) return done();  // reduce.hpp:72-75: skipping reduction
  red = ReduceState{};
  red.active = true;
  red.bfs_steps = mlsw;
  red.original = A;
  red.reduced.n = rn;
  red.reduced.k = A.k;
  red.reduced.t.assign((size_t)rn * A.k, 0);
  for (int q = 0; q < n; ++q)
    if (reach[q])
      for (uint32_t a = 0; a < A.k; ++a) red.reduced.t[(size_t)map[q] * A.k + a] = map[A.at((uint32_t)q, a)];
  for (int q = 0; q < n; ++q)
    if (reach[q]) red.states.push_back((uint32_t)q);
  red.seeds = E.R.count;
  st.reduce_bfs_steps = mlsw;
  st.reduced_states = rn;
  // reduce.hpp:77-84: the remaining search works on reduced lengths
  b.lower = b.lower > mlsw ? b.lower - mlsw : 0;
  b.upper -= mlsw;
  done();
}

// ---------------------------------------------------------------------------
// Learned distance model: training pairs, scoring, training, learned beam.
// ---------------------------------------------------------------------------
namespace {
// device rows of W words -> the 8-word reference layout of the model's sets
void rows_to_ref8(const u64* rows, uint64_t count, uint32_t n, int W, uint64_t* out) {
  for (uint64_t i = 0; i < count; ++i) {
    for (int w = 0; w < 8; ++w) out[i * 8 + w] = 0;
    for (uint32_t q = 0; q < n; ++q)
      if (rows[(size_t)i * W + (q >> 6)] & state_bit((int)q)) out[i * 8 + (q >> 6)] |= 1ULL << (q & 63);
  }
}
}  // namespace

void Solver::set_model(const float* params) {
  SW_CUDA(cudaSetDevice(device_));
  eng_->mlp->set_params(params);
}
void Solver::get_model(float* params) {
  if (!eng_->mlp->has_params()) throw std::runtime_error("no distance model loaded");
  SW_CUDA(cudaSetDevice(device_));
  eng_->mlp->get_params(params);
}
bool Solver::has_model() const { return eng_->mlp->has_params(); }

uint32_t Solver::distance_pairs(const Automaton& A, uint32_t per_layer, uint64_t max_inverse_sets,
                                std::vector<uint64_t>& sets, std::vector<float>& labels,
                                std::vector<uint32_t>& depths) {
  sets.clear();
  labels.clear();
  depths.clear();
  if (A.n < 2 || per_layer == 0) return 0;
  // the reset length bounds the depths worth labelling
  Bounds b;
  b.upper = std::max<u64>(1, (u64)A.n * A.n * A.n / 6);
  sw_exact_config cfg{1, 1, 0, 2048, 10000, (uint64_t)A.n * 16};
  sw_stats st0{};
  exact(A, cfg, b, st0);
  if (b.non_synchro || b.lower != b.upper) return 0;
  const u64 L = b.upper;
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const int n = (int)A.n, k = (int)A.k, W = words_for(n);
  E.upload_tables(A);
  E.reductions = true;  // labelled layers are the fully reduced ones
  // inverse layers (complements of the maximal preimage sets), depth 0..D
  E.B.reset();
  std::vector<uint32_t> seeds = backward_seeds(A);
  if (seeds.empty()) return 0;
  {
    std::vector<u64> rows((size_t)W * seeds.size(), 0);
    for (size_t i = 0; i < seeds.size(); ++i)
      for (int q = 0; q < n; ++q)
        if ((uint32_t)q != seeds[i]) rows[i * W + (q >> 6)] |= state_bit(q);
    E.B.rows.reserve(sizeof(u64) * rows.size());
    E.B.vis.reserve(sizeof(u64) * rows.size());
    SW_CUDA(cudaMemcpyAsync(E.B.rows.p, rows.data(), sizeof(u64) * rows.size(), cudaMemcpyHostToDevice, E.stream));
    SW_CUDA(cudaMemcpyAsync(E.B.vis.p, rows.data(), sizeof(u64) * rows.size(), cudaMemcpyHostToDevice, E.stream));
    E.B.count = E.B.vis_count = (u32)seeds.size();
    E.sort_by_layer_key(W, E.B.vis.as<u64>(), E.B.vis_count);
  }
  std::vector<std::unique_ptr<DevBuf>> inv;
  std::vector<u32> inv_count;
  u64 inv_total = 0;
  auto keep_layer = [&] {
    inv.push_back(std::make_unique<DevBuf>());
    inv.back()->reserve(sizeof(u64) * W * std::max<u32>(E.B.count, 1));
    SW_CUDA(cudaMemcpyAsync(inv.back()->p, E.B.rows.p, sizeof(u64) * W * E.B.count, cudaMemcpyDeviceToDevice,
                            E.stream));
    inv_count.push_back(E.B.count);
    inv_total += E.B.count;
  };
  keep_layer();
  for (u64 j = 1; j <= L && inv_total < max_inverse_sets; ++j) {
    E.step(E.B, false, W, n, k, true, true);
    if (!E.B.count) break;
    keep_layer();
  }
  const u32 D = (u32)inv.size() - 1;
  // forward layers, sampled and labelled
  E.F.reset();
  {
    std::vector<u64> full(W, 0);
    for (int q = 0; q < n; ++q) full[q >> 6] |= state_bit(q);
    E.F.rows.reserve(sizeof(u64) * W);
    E.F.vis.reserve(sizeof(u64) * W);
    SW_CUDA(cudaMemcpyAsync(E.F.rows.p, full.data(), sizeof(u64) * W, cudaMemcpyHostToDevice, E.stream));
    SW_CUDA(cudaMemcpyAsync(E.F.vis.p, full.data(), sizeof(u64) * W, cudaMemcpyHostToDevice, E.stream));
    E.F.count = E.F.vis_count = 1;
  }
  DevBuf idx_d, sample, flags;
  for (u64 i = 0; i <= L; ++i) {
    const u32 c = E.F.count;
    const u32 s = std::min<u32>(c, per_layer);
    std::vector<u32> idx(s);
    for (u32 t = 0; t < s; ++t) idx[t] = (u32)(((u64)t * c) / s);
    idx_d.reserve(sizeof(u32) * s);
    sample.reserve(sizeof(u64) * W * s);
    flags.reserve(sizeof(u32) * s);
    SW_CUDA(cudaMemcpyAsync(idx_d.p, idx.data(), sizeof(u32) * s, cudaMemcpyHostToDevice, E.stream));
    launch_gather_rows(W, E.F.rows.as<u64>(), idx_d.as<u32>(), s, sample.as<u64>(), E.stream);
    std::vector<float> lab(s, (float)(D + 1));
    std::vector<u32> fl(s);
    u32 open = s;
    for (u32 j = 0; j <= D && open; ++j) {
      launch_fill_u32(flags.as<u32>(), 0, s, E.stream);
      E.query(W, kQueryDisjoint, inv[j]->as<u64>(), inv_count[j], sample.as<u64>(), s, n, flags.as<u32>(), false);
      SW_CUDA(cudaMemcpyAsync(fl.data(), flags.p, sizeof(u32) * s, cudaMemcpyDeviceToHost, E.stream));
      SW_CUDA(cudaStreamSynchronize(E.stream));
      for (u32 t = 0; t < s; ++t)
        if (fl[t] && lab[t] > (float)j) {
          lab[t] = (float)j;
          --open;
        }
    }
    std::vector<u64> rows((size_t)s * W);
    SW_CUDA(cudaMemcpy(rows.data(), sample.p, sizeof(u64) * W * s, cudaMemcpyDeviceToHost));
    const size_t base = sets.size();
    sets.resize(base + (size_t)s * 8);
    rows_to_ref8(rows.data(), s, (uint32_t)n, W, sets.data() + base);
    labels.insert(labels.end(), lab.begin(), lab.end());
    depths.insert(depths.end(), s, (uint32_t)i);
    if (i == L) break;
    E.step(E.F, true, W, n, k, true, true);
    if (!E.F.count) break;
  }
  return (uint32_t)L;
}

void Solver::mlp_forward(const Automaton& A, const uint64_t* sets, uint64_t count, float* out) {
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  if (!count) return;
  DevBuf d_rows, d_y;
  d_rows.reserve(sizeof(u64) * 8 * count);
  d_y.reserve(sizeof(float) * count);
  SW_CUDA(cudaMemcpyAsync(d_rows.p, sets, sizeof(u64) * 8 * count, cudaMemcpyHostToDevice, E.stream));
  launch_convert_rows(8, d_rows.as<u64>(), count, (int)A.n, true, E.stream);
  E.mlp->prepare(A);
  E.mlp->forward(d_rows.as<u64>(), 8, (u32)count, d_y.as<float>());
  SW_CUDA(cudaMemcpyAsync(out, d_y.p, sizeof(float) * count, cudaMemcpyDeviceToHost, E.stream));
  E.check_scan_error(E.read_u32(E.d_misc + Engine::kScanErrWord));
}

float Solver::check_dominated(uint32_t n, bool forward, bool proper, const uint64_t* S, uint32_t m, const uint64_t* Q,
                              uint32_t q, bool live, bool masked, uint32_t* flags) {
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const int W = words_for((int)n);
  // with live counts the lists are announced half as long again, and hold garbage there
  const u32 mm = live ? m + m / 2 : m, qq = live ? q + q / 2 : q;
  DevBuf s_rows, q_rows, d_flags;
  s_rows.reserve(sizeof(u64) * W * (size_t)mm);
  q_rows.reserve(sizeof(u64) * W * (size_t)qq);
  d_flags.reserve(sizeof(u32) * (size_t)qq);
  SW_CUDA(cudaMemsetAsync(s_rows.p, 0, s_rows.cap, E.stream));
  SW_CUDA(cudaMemsetAsync(q_rows.p, 0xff, q_rows.cap, E.stream));
  SW_CUDA(cudaMemcpyAsync(s_rows.p, S, sizeof(u64) * W * (size_t)m, cudaMemcpyHostToDevice, E.stream));
  SW_CUDA(cudaMemcpyAsync(q_rows.p, Q, sizeof(u64) * W * (size_t)q, cudaMemcpyHostToDevice, E.stream));
  u32* const counts = E.d_misc + 50;
  launch_fill_u32(counts, m, 1, E.stream);
  launch_fill_u32(counts + 1, q, 1, E.stream);
  float ms = 0;
  E.states_ordered = true;
  for (int run = 0; run < 2; ++run) {  // the first grows the buffers
    SW_CUDA(cudaMemcpyAsync(d_flags.p, flags, sizeof(u32) * (size_t)q, cudaMemcpyHostToDevice, E.stream));
    E.reduce_span.mark(0, E.stream);
    if (masked)
      E.query(W, proper ? kQueryProperSubset : kQuerySubset, s_rows.as<u64>(), mm, q_rows.as<u64>(), qq, (int)n,
              d_flags.as<u32>(), false, live ? counts : nullptr, live ? counts + 1 : nullptr);
    else
      E.dominated(forward, W, s_rows.as<u64>(), mm, q_rows.as<u64>(), qq, (int)n, proper, mm, d_flags.as<u32>(),
                  E.dom_rows, live ? counts : nullptr, live ? counts + 1 : nullptr);
    E.reduce_span.mark(1, E.stream);
    SW_CUDA(cudaStreamSynchronize(E.stream));
    ms = (float)(1e3 * E.reduce_span.seconds());
  }
  E.states_ordered = false;
  SW_CUDA(cudaMemcpy(flags, d_flags.p, sizeof(u32) * (size_t)q, cudaMemcpyDeviceToHost));
  return ms;
}

void Solver::plant_error(uint32_t code) {
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  launch_fill_u32(E.d_misc + Engine::kScanErrWord, code, 1, E.stream);
  SW_CUDA(cudaStreamSynchronize(E.stream));
}

// The trainer, with the loaded parameters and no moments.
static Trainer& training(Engine& E) {
  if (!E.mlp->has_params()) throw std::runtime_error("no distance model loaded");
  if (!E.trainer) E.trainer = std::make_unique<Trainer>(E.stream);
  E.trainer->set_params(E.mlp->params());
  return *E.trainer;
}

float Solver::mlp_gradient(const Automaton& A, const uint64_t* sets, const float* labels, uint64_t count,
                           float* grad) {
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  if (!count) throw std::invalid_argument("empty batch");
  DevBuf d_rows, d_y, d_t;
  d_rows.reserve(sizeof(u64) * 8 * count);
  d_y.reserve(sizeof(float) * count);
  d_t.reserve(sizeof(float) * count);
  SW_CUDA(cudaMemcpyAsync(d_rows.p, sets, sizeof(u64) * 8 * count, cudaMemcpyHostToDevice, E.stream));
  launch_convert_rows(8, d_rows.as<u64>(), count, (int)A.n, true, E.stream);
  SW_CUDA(cudaMemcpyAsync(d_t.p, labels, sizeof(float) * count, cudaMemcpyHostToDevice, E.stream));
  Trainer& T = training(E);
  T.prepare(A);
  T.zero_grad();
  T.forward(d_rows.as<u64>(), 8, (u32)count, d_y.as<float>());
  T.backward(d_t.as<float>(), (u32)count);
  float loss = 0;
  SW_CUDA(cudaMemcpyAsync(grad, T.grad(), sizeof(float) * mlp::kParams, cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaMemcpyAsync(&loss, T.loss(), sizeof(float), cudaMemcpyDeviceToHost, E.stream));
  SW_CUDA(cudaStreamSynchronize(E.stream));
  if (train::tc_error()) throw CudaError("distance model: a tensor-core wait ran out");
  return loss;
}

float Solver::mlp_train(const std::vector<Automaton>& autos, const uint64_t* offsets, const uint64_t* sets,
                        const float* labels, uint32_t epochs, uint32_t batch, float lr, uint64_t seed,
                        const uint32_t* groups, float rank_w) {
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const size_t A_n = autos.size();
  const uint64_t total = offsets[A_n];
  if (!total || !batch) throw std::invalid_argument("no training pairs");
  // all pairs resident on the device as 8-word rows
  Trainer& T = training(E);
  DevBuf d_rows, d_lab, d_grp, d_y;
  d_y.reserve(sizeof(float) * batch);
  d_rows.reserve(sizeof(u64) * 8 * total);
  d_lab.reserve(sizeof(float) * total);
  SW_CUDA(cudaMemcpyAsync(d_rows.p, sets, sizeof(u64) * 8 * total, cudaMemcpyHostToDevice, E.stream));
  for (size_t a = 0; a < A_n; ++a)
    launch_convert_rows(8, d_rows.as<u64>() + offsets[a] * 8, offsets[a + 1] - offsets[a], (int)autos[a].n, true,
                        E.stream);
  SW_CUDA(cudaMemcpyAsync(d_lab.p, labels, sizeof(float) * total, cudaMemcpyHostToDevice, E.stream));
  if (groups && rank_w > 0.0f) {
    d_grp.reserve(sizeof(uint32_t) * total);
    SW_CUDA(cudaMemcpyAsync(d_grp.p, groups, sizeof(uint32_t) * total, cudaMemcpyHostToDevice, E.stream));
  }
  std::vector<size_t> order(A_n);
  for (size_t a = 0; a < A_n; ++a) order[a] = a;
  uint64_t state = seed;
  auto next = [&] {  // SplitMix64
    uint64_t z = (state += 0x9E3779B97F4A7C15ULL);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
  };
  double last = 0;
  for (uint32_t ep = 0; ep < epochs; ++ep) {
    for (size_t a = A_n; a > 1; --a) std::swap(order[a - 1], order[next() % a]);
    double sum = 0;
    uint64_t steps = 0;
    for (size_t oi = 0; oi < A_n; ++oi) {
      const size_t a = order[oi];
      for (uint64_t o = offsets[a]; o < offsets[a + 1]; o += batch) {
        const u32 c = (u32)std::min<uint64_t>(batch, offsets[a + 1] - o);
        T.prepare(autos[a]);
        T.zero_grad();
        T.forward(d_rows.as<u64>() + o * 8, 8, c, d_y.as<float>());
        T.backward(d_lab.as<float>() + o, c, d_grp.p ? d_grp.as<uint32_t>() + o : nullptr, rank_w);
        T.adam_step(lr);
        float l = 0;
        SW_CUDA(cudaMemcpyAsync(&l, T.loss(), sizeof(float), cudaMemcpyDeviceToHost, E.stream));
        SW_CUDA(cudaStreamSynchronize(E.stream));
        sum += l;
        ++steps;
      }
    }
    last = steps ? sum / steps : 0.0;
  }
  if (train::tc_error()) throw CudaError("distance model: a tensor-core wait ran out");
  std::vector<float> trained(mlp::kParams);
  T.get_params(trained.data());
  E.mlp->set_params(trained.data());
  return (float)last;
}

void Solver::learned_beam(const Automaton& A, const sw_learned_beam_config& cfg, Bounds& b, sw_stats& st) {
  if (b.non_synchro || b.lower == b.upper) return;
  const bool use_model = cfg.order != SW_ORDER_SIZE;
  if (use_model && !has_model()) throw std::runtime_error("LearnedBeam: no distance model loaded");
  if (A.n == 1) {
    b.lower = b.upper = 0;
    b.has_word = true;
    b.word.clear();
    return;
  }
  SW_CUDA(cudaSetDevice(device_));
  Engine& E = *eng_;
  const Engine::Counting counting(E, st);
  auto t0 = std::chrono::steady_clock::now();
  const int n = (int)A.n, k = (int)A.k, W = words_for(n);
  E.upload_tables(A);
  if (use_model) E.mlp->prepare(A);
  E.F.reset();
  {
    std::vector<u64> full(W, 0);
    for (int q = 0; q < n; ++q) full[q >> 6] |= state_bit(q);
    E.F.rows.reserve(sizeof(u64) * W);
    SW_CUDA(cudaMemcpyAsync(E.F.rows.p, full.data(), sizeof(u64) * W, cudaMemcpyHostToDevice, E.stream));
    E.F.count = 1;
    E.F.vis_count = 0;
  }
  const u32 width = (u32)std::min<uint64_t>(cfg.beam_size, 1u << 26);
  // engine-owned, kept across calls: freeing device memory would synchronise the device
  DevBuf &counts = E.lb_counts, &scores = E.lb_scores, &keys = E.lb_keys, &vals = E.lb_vals;
  DevBuf &alt_k = E.lb_alt_k, &alt_v = E.lb_alt_v, &sel_rows = E.lb_sel_rows, &sel_origin = E.lb_sel_origin;
  u64* const sum = reinterpret_cast<u64*>(E.d_misc + 32);  // as in reduce(): ~(the first single-state set) follows
  const size_t sum_bytes = 8 * sizeof(u64) + sizeof(u32);
  u64 found_len = 0;
  std::vector<uint32_t> word;
  for (u64 depth = 1; depth < b.upper && (cfg.max_iter < 0 || depth <= (u64)cfg.max_iter); ++depth) {
    // Layers of up to kSelectMax children scored by the model: duplicates dropped by
    // the hash table and the kept sets selected, where the others are sorted twice.
    // Ordering by size stays sorted: most of its keys are equal.
    const bool select = use_model && (u64)E.F.count * k <= kSelectMax;
    if (select)
      E.step_distinct(E.F, W, k);
    else
      E.step(E.F, true, W, n, k, /*dominance=*/false);  // children, duplicates removed, origins recorded
    SW_CUDA(cudaMemsetAsync(sum, 0, sum_bytes, E.stream));
    launch_list_summary(W, E.F.rows.as<u64>(), E.F.count, sum, reinterpret_cast<u32*>(sum + 8), E.stream,
                        select ? E.d_misc + 8 : nullptr);
    SW_CUDA(cudaMemcpyAsync(E.pinned.p, E.d_misc, 32 * sizeof(u32) + sum_bytes, cudaMemcpyDeviceToHost, E.stream));
    SW_CUDA(cudaStreamSynchronize(E.stream));
    E.check_scan_error(E.pinned.as<u32>()[Engine::kScanErrWord]);
    const u32 single = E.pinned.as<u32>()[48];
    if (select) {
      E.F.count = E.F.layers.back()->count = E.pinned.as<u32>()[8];
      st.subsets_kept += E.F.count;
    }
    const u32 m = E.F.count;
    if (!m) break;
    if (single) {
      word = E.trace(E.F, ~single, nullptr);
      std::reverse(word.begin(), word.end());
      found_len = depth;
      break;
    }
    if (m <= width) continue;
    // keep the `width` children with the smallest score (ties: child order)
    keys.reserve(sizeof(u64) * m);
    vals.reserve(sizeof(u32) * m);
    if (use_model) {
      scores.reserve(sizeof(float) * m);
      E.mlp->forward(E.F.rows.as<u64>(), W, m, scores.as<float>());
    }
    if (cfg.order != SW_ORDER_MODEL) {
      counts.reserve(sizeof(u32) * m);
      launch_popcount(W, E.F.rows.as<u64>(), m, counts.as<u32>(), E.stream);
    }
    launch_score_keys(use_model ? scores.as<float>() : nullptr,
                      cfg.order != SW_ORDER_MODEL ? counts.as<u32>() : nullptr, m, keys.as<u64>(), E.stream);
    if (select) {
      launch_select(W, keys.as<u64>(), m, width, E.F.rows.as<u64>(), vals.as<u32>(), E.stream);
      E.count_launch();
    } else {
      launch_iota(vals.as<u32>(), m, E.stream);
      E.sort_rows(1, keys.as<u64>(), vals.as<u32>(), m);
    }
    sel_rows.reserve(sizeof(u64) * W * width);
    sel_origin.reserve(sizeof(u32) * width);
    launch_gather_rows(W, E.F.rows.as<u64>(), vals.as<u32>(), width, sel_rows.as<u64>(), E.stream);
    Layer& top = *E.F.layers.back();
    launch_gather_u32(top.origin.as<u32>(), vals.as<u32>(), width, sel_origin.as<u32>(), E.stream);
    std::swap(E.F.rows.p, sel_rows.p);
    std::swap(E.F.rows.cap, sel_rows.cap);
    std::swap(top.origin.p, sel_origin.p);
    std::swap(top.origin.cap, sel_origin.cap);
    top.count = width;
    E.F.count = width;
    E.count_launch(5);
  }
  if (found_len && found_len < b.upper) {
    if (apply_word(A, word).size() != 1 || word.size() != found_len)
      throw std::runtime_error("internal: learned beam word does not synchronize");
    b.upper = found_len;
    b.has_word = true;
    b.word = word;
  }
  st.device_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

}  // namespace sw
