// kernels.cuh -- sm_103a device code of the blocking engine.
//
// Pipeline per run (all on one stream; the batched form is a CUDA graph):
//   1. k_join_count   join key of every row per rule (partition bucket and
//                     equality dictionary codes in mixed radix, or a dense
//                     composite id) + histogram of keys per side.
//   2. k_join_scan    exclusive scans: row offsets per key, and work items
//                     per key (a work item = one left row x up to TR right rows
//                     of one candidate block).
//   3. k_join_scatter rows grouped by key (counting sort) -> candidate blocks
//                     L_key x R_key.
//   4. k_peq_build    Peq bitmask table of every left string (built with
//                     __match_any), in device memory.
//   5. k_eval         persistent, warp-granular work stealing over the items
//                     of every rule: a warp filters an item's right rows
//                     (staged by bulk copies, the next item's copies in
//                     flight) against the first similarity predicate and
//                     queues the pairs that need a scan in a shared-memory
//                     ring; lanes take the next queued pair, of whatever
//                     item, as soon as theirs is decided (bit-parallel Jaro
//                     from the left string's table, exact early-fail bound),
//                     and go on with the rule's next predicate in the same
//                     lane; matches leave by warp-aggregated atomics.
//   6. k_eval_long    where some left string has over 256 symbols (no table):
//                     the items of those strings, and the pairs that met one
//                     at a later predicate, by whole warps.
//   7. k_report       counters, and a small result's pairs, to the host.
//
// Semantics reproduced (reference = HyperBlocker):
//   * pairs are compared only inside a partition (data_mngr.h:150-216, the
//     bucket is part of every join key);
//   * a pair matches when some rule has all equalities true and all
//     similarities !(JW < (double)threshold) (global_func.cuh:120-167);
//   * Jaro match count m of device_func.cuh:54-132 equals the size of a
//     maximum matching between equal characters at distance <= h,
//     h = (min(len1, len2) + 1) / 2, whenever the shorter string has at most
//     256 bytes; longer pairs run the reference's own loop order (jaro_m_ref);
//   * the Jaro value is (float)(((double)(m/ls + m/ll) + 1.0) / 3.0) with IEEE
//     float quotients, and JW = fma((1 - j) * p, 0.1, j) clamped to 1 with an
//     uncapped common prefix p (device_func.cuh:210-231).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <vector>

namespace hbx {
namespace dev {

constexpr int kMaxEq = 8;
constexpr int kMaxSim = 8;
constexpr int kWarpsPerCta = 8;
// words per symbol row of a Peq table for a left string of w 32-bit words
__host__ __device__ constexpr int row_words(int w) { return w <= 1 ? 1 : w <= 2 ? 2 : w <= 4 ? 4 : 8; }
constexpr float kDecisionMargin = 1e-4f;  // |approx JW - thr| below this -> exact path

// Count signature of a string: byte k (of 32) counts the string's symbols in
// bucket k (at most 255), where the 31 most frequent symbols have a bucket
// each and the rest share the last one.  For any two strings a, b the Jaro
// match count (any matching between equal symbols) is at most
//     sum_k min(count_a[k], count_b[k])
//         = (len_a + len_b - sum_k |count_a[k] - count_b[k]|) / 2,
// and pooling symbols into one bucket only raises that sum.  Counts cut off
// at 255 only lower the differences, so the signatures still give an upper
// bound.
constexpr uint32_t kSigBuckets = 32;
__host__ __device__ inline uint32_t sig_bucket(uint32_t sym) {  // sym >= 1
  return sym >= kSigBuckets ? kSigBuckets - 1 : sym - 1;
}

// Metadata of one string: where it is, how long, its first 16 symbols (0 past
// the end) and its count signature, so that one 64-byte record gives the
// length, the common prefix with another string (up to 16), the first chunk
// of a scan and an upper bound on the matches with any other string.
struct __align__(16) StrMeta {
  uint4 loc;     // {offset / 16, length, 0, 0}
  uint4 head;    // symbols 0-3, 4-7, 8-11, 12-15 (little endian)
  uint4 sig[2];  // bucket counts 0-15, 16-31, one byte each (little endian)
};

// Host form of the signature of a string of symbols.
inline void make_sig(const uint8_t* s, uint32_t len, uint4 out[2]) {
  uint32_t w[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  uint32_t c[kSigBuckets] = {0};
  for (uint32_t i = 0; i < len; i++)
    if (s[i]) c[sig_bucket(s[i])]++;
  for (uint32_t k = 0; k < kSigBuckets; k++) w[k / 4] |= (c[k] < 255u ? c[k] : 255u) << (8 * (k % 4));
  out[0] = make_uint4(w[0], w[1], w[2], w[3]);
  out[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// A record of Rule::sorted_meta_r holds its four 16-byte pieces (loc, head,
// sig[0], sig[1]) in an order that depends on its position: piece p of record
// pos is at index p ^ meta_turn(pos).  Lanes that read the same piece of
// consecutive records from shared memory then spread over all banks (in
// record order they would use two of eight 16-byte columns).
__host__ __device__ inline uint32_t meta_turn(uint32_t pos) { return (pos >> 1) & 3u; }

struct Side {
  const uint32_t* bucket;
  const int32_t* eq_codes;    // [n_eq_slots][n_rows]
  const int32_t* comp_codes;  // [n_comp][n_rows]
  const uint8_t* arena;       // symbol strings, 16-byte aligned, zero padded
  const StrMeta* str_meta;    // [n_str_slots][n_rows]
  uint32_t n_rows;
};

// A rule evaluated as a member of a group (see Rule): its threshold on the
// group's first similarity column, the extra equality slots it needs beyond
// the group root's (bits of Rule::xslot), and its other similarity
// predicates in evaluation order.
constexpr uint32_t kMaxMembers = 8;
constexpr uint32_t kMaxDup = 4;
struct Member {
  float thr_first;
  uint32_t xmask;
  uint32_t n_rest;
  uint32_t rest_l[kMaxSim], rest_r[kMaxSim];
  float rest_thr[kMaxSim];
};

struct Rule {
  uint32_t n_eq, n_sim, composite, comp_index;
  uint32_t eq_slot[kMaxEq];
  uint32_t radix[kMaxEq];
  uint32_t sim_l[kMaxSim], sim_r[kMaxSim];
  float thr[kMaxSim];
  uint32_t domain;    // D: join keys
  // Where some left string has no Peq table (more than kMaxTableLen symbols),
  // left rows are grouped by (class, key): class 1 holds the rows whose
  // string of the first similarity predicate is that long.  Their work items
  // follow all items of class 0 and are evaluated by k_eval_long.  The left
  // keys of class 1 follow the D of class 0: one per join key, or, where there
  // are at least twice as many join keys as left rows, one per row of the
  // class (ranked: in the order of arrival, *n_long so far, with their join
  // keys in long_key), so that few long strings do not double the state of a
  // large key domain (20 bytes a key).
  uint32_t n_classes;   // 1, or 2 with long left strings
  uint32_t class_slot;  // left string slot that decides the class
  uint32_t ranked;
  uint32_t domain_l;    // left keys of all classes
  uint32_t* long_key;   // [left rows], ranked only
  uint32_t* n_long;
  uint32_t* key_l;
  uint32_t* key_r;
  uint32_t* cnt_l;  // [domain_l]
  uint32_t* cnt_r;  // [domain]
  uint32_t* off_l;  // [domain_l]
  uint32_t* off_r;  // [domain]
  uint32_t* cur_l;
  uint32_t* cur_r;
  unsigned long long* item_off;  // [domain_l + 1]
  uint32_t* sorted_l;
  uint32_t* sorted_r;  // [n_rows + 4]: the tail pads 16-byte bulk copies
  // right-row string metadata of the first similarity predicate in sorted_r
  // order (the pieces of a record turned, meta_turn), so that a work item's
  // metadata is one contiguous, 16-byte-aligned block for a bulk copy into
  // shared memory (null without similarities)
  StrMeta* sorted_meta_r;
  // Group evaluation.  The work items of this rule's join are evaluated for
  // n_members rules at once: member 0 is this rule, the others are rules whose
  // equality slots contain this rule's (their candidates are this join's
  // candidates whose extra slots xslot[] also hold) and whose similarity
  // predicates include this rule's first column (sim_l[0], sim_r[0]).  The
  // first column is filtered and scanned once per pair, at the smallest
  // threshold of the members still live, and decided per member from the
  // match count; members that pass go on with their other predicates, and
  // the pair matches when one member passes them all (OR across rules).
  // n_members == 0: the rule is a member of another rule's group and has no
  // work items of its own; its pair-comparisons are still counted.
  uint32_t n_members;
  // Rules whose pair-comparisons this rule's join counts: itself and, in a
  // grouped rule array, the rules with the same equality slots that have no
  // join of their own (their cmp_weight is 0).
  uint32_t cmp_weight;
  uint32_t n_xslots;
  uint32_t xslot[kMaxEq];
  float thr_min;  // smallest member threshold on the first column
  Member mem[kMaxMembers];
  // Groups with at most two extra slots: for each pattern of the extra slots
  // that hold (bit j: xslot[j]), the members still live and the smallest of
  // their first-column thresholds (fill_extras_table), so that the filter
  // looks them up instead of walking the members for every pair.
  uint32_t x_live[4];
  float x_thr[4];
  // A pair can be reported by another rule of the launch too only where that
  // rule's equalities also hold.  dup_always: it may at any pair (or there are
  // more such rules than kMaxDup); else entry k: another rule and up to two of
  // its equality slots that this rule's do not imply (set_overlaps).
  uint32_t dup_always, n_dup;
  uint32_t dup_slot[kMaxDup][2];
};

// Host: fills Rule::x_live / x_thr from the members, with the device's
// live-threshold rule (the smallest threshold; NaN when any is NaN).
inline void fill_extras_table(Rule* g) {
  for (uint32_t eqm = 0; eqm < 4; eqm++) {
    uint32_t live = 0;
    float t = 3.0e38f;
    for (uint32_t k = 0; k < g->n_members; k++) {
      if (g->mem[k].xmask & ~eqm) continue;
      live |= 1u << k;
      const float u = g->mem[k].thr_first;
      t = (u != u || t != t) ? __builtin_nanf("") : (u < t ? u : t);
    }
    g->x_live[eqm] = live;
    g->x_thr[eqm] = t;
  }
}

// Host: a rule as the only member of its own group (the plain form, serving,
// and any rule no group takes in).
inline void make_singleton(Rule* d) {
  d->n_members = 1;
  d->cmp_weight = 1;
  d->dup_always = d->n_dup = 0;
  d->n_xslots = 0;
  Member& m = d->mem[0];
  m = Member{};
  m.thr_first = d->n_sim ? d->thr[0] : 0.0f;
  m.xmask = 0;
  m.n_rest = d->n_sim > 1 ? d->n_sim - 1 : 0;
  for (uint32_t k = 1; k < d->n_sim; k++) {
    m.rest_l[k - 1] = d->sim_l[k];
    m.rest_r[k - 1] = d->sim_r[k];
    m.rest_thr[k - 1] = d->thr[k];
  }
  d->thr_min = m.thr_first;
  fill_extras_table(d);
}

// Host: fills dup_always and dup_slot of the rules [0, n) that are evaluated
// (those with members) over the same rows.
inline void set_overlaps(Rule* rules, size_t n) {
  auto has = [](const Rule& r, uint32_t slot) {
    for (uint32_t e = 0; e < r.n_eq; e++)
      if (r.eq_slot[e] == slot) return true;
    return false;
  };
  for (size_t g = 0; g < n; g++) {
    Rule& G = rules[g];
    G.dup_always = G.n_dup = 0;
    for (size_t h = 0; h < n && G.n_members; h++) {
      const Rule& H = rules[h];
      if (h == g || !H.n_members) continue;
      uint32_t extra[2], k = 0;  // a slot may come twice: no harm
      for (uint32_t e = 0; e < H.n_eq && k < 2; e++)
        if (!has(G, H.eq_slot[e])) extra[k++] = H.eq_slot[e];
      if (k == 0 || G.n_dup == kMaxDup) {
        G.dup_always = 1;
        break;
      }
      G.dup_slot[G.n_dup][0] = extra[0];
      G.dup_slot[G.n_dup][1] = extra[k - 1];
      G.n_dup++;
    }
  }
}

constexpr uint32_t kMaxTableLen = 256;
__host__ __device__ inline uint32_t left_class(uint32_t len) { return len > kMaxTableLen ? 1u : 0u; }

// Host: the left keys of a rule over n_left rows, in two classes when some left
// string is longer than kMaxTableLen.  After domain, n_sim and sim_l are set.
inline void set_classes(Rule* d, bool long_left, uint32_t n_left) {
  d->n_classes = long_left && d->n_sim ? 2u : 1u;
  d->class_slot = d->n_sim ? d->sim_l[0] : 0u;
  d->ranked = d->n_classes > 1 && d->domain / 2 >= n_left ? 1u : 0u;
  d->domain_l = d->domain + (d->n_classes == 1 ? 0u : d->ranked ? n_left : d->domain);
}
#ifdef __CUDACC__
// Left key of a row with join key `key`; class 1 ranks are handed out here.
__device__ __forceinline__ uint32_t left_key(const Rule& R, const Side& L, uint32_t row,
                                             uint32_t key) {
  if (R.n_classes == 1 || !left_class(L.str_meta[(size_t)R.class_slot * L.n_rows + row].loc.y))
    return key;
  if (!R.ranked) return R.domain + key;
  const uint32_t k = atomicAdd(R.n_long, 1u);
  R.long_key[k] = key;
  return R.domain + k;
}
// Join key of left key j, which holds rows.
__device__ __forceinline__ uint32_t join_key(const Rule& R, uint32_t j) {
  if (j < R.domain) return j;
  return R.ranked ? R.long_key[j - R.domain] : j - R.domain;
}
#endif
constexpr uint32_t kMaxSegments = 1;
constexpr uint32_t kRingEntries = 64;
constexpr uint32_t kRingWords = 12;  // words per ring entry (three 16-byte records)

// Peq tables of the left strings, in device memory: one per (left string
// slot, left row), tab_words 32-bit words each; row `sym` (peq_s words) has
// bit j of word k set when a[32k + j] == sym.  Strings of 1 to fast_max
// symbols have a table; fast_max = 32 * peq_w <= 256.
struct PeqShape {
  uint32_t w;          // words the scans run on: 1, 2, 3, 4 or 8
  uint32_t s;          // words per symbol row: row_words(w)
  uint32_t tab_words;  // words per table (a multiple of 4: tables are 16-byte aligned)
  uint32_t fast_max;   // longest left string with a table
};

// Shape for left strings up to max_len symbols (capped at 256) over an
// alphabet of n_symbols symbols.
inline PeqShape peq_shape(uint32_t max_len, uint32_t n_symbols) {
  const uint32_t len = max_len < 1 ? 1 : (max_len > 256 ? 256 : max_len);
  const uint32_t w0 = (len + 31) / 32;
  PeqShape p;
  p.w = w0 <= 4 ? w0 : 8;
  p.s = (uint32_t)row_words((int)p.w);
  p.tab_words = (n_symbols * p.s + 3) / 4 * 4;
  p.fast_max = 32 * p.w;
  return p;
}

// Shared memory of one warp of k_eval, in 32-bit words: the ring of pairs
// waiting for a scan (kRingEntries x kRingWords), n_bufs staging buffers
// (while the warp filters one work item, the bulk copies of the next
// n_bufs - 1 fill the others) and one mbarrier per buffer.  A staging buffer holds the item's right-row
// metadata (tile_right StrMeta records), its right rows (tile_right + 8: a
// 16-byte-aligned copy starts up to 3 rows early and rounds up) and the
// metadata of its left string.  Every offset is a multiple of 4 words (16
// bytes) when tile_right is a multiple of 32.  A control block of
// kWarpCtlWords words follows.
constexpr uint32_t kMaxStageBufs = 4;
struct WarpLayout {
  uint32_t n_bufs, buf_off, buf_words, buf_rows_off, buf_lmeta_off, mbar_off, ctl_off, warp_words;
};
constexpr uint32_t kWarpCtlWords = 512;  // the warp's control block (kernels.cu: WarpCtl)

inline WarpLayout warp_layout(uint32_t tile_right, uint32_t n_bufs) {
  WarpLayout w;
  w.n_bufs = n_bufs < 1 ? 1 : (n_bufs > kMaxStageBufs ? kMaxStageBufs : n_bufs);
  const uint32_t meta_words = (uint32_t)(sizeof(StrMeta) / 4) * tile_right;
  w.buf_rows_off = meta_words;
  w.buf_lmeta_off = meta_words + (tile_right + 8 + 3) / 4 * 4;
  // (64-byte multiples: a record's turned pieces stay inside it)
  w.buf_words = (w.buf_lmeta_off + (uint32_t)(sizeof(StrMeta) / 4) + 15) / 16 * 16;
  w.buf_off = kRingWords * kRingEntries;
  w.mbar_off = w.buf_off + w.n_bufs * w.buf_words;
  w.ctl_off = w.mbar_off + (2 * w.n_bufs + 3) / 4 * 4;
  w.warp_words = (w.ctl_off + kWarpCtlWords + 15) / 16 * 16;
  return w;
}

// The deepest staging (up to kMaxStageBufs buffers) that keeps two blocks of
// kWarpsPerCta warps on an SM within smem_cap bytes of shared memory; one
// buffer when none does (with one buffer the next item's copies start once
// the current item is filtered, and other warps cover their latency).
inline WarpLayout warp_layout_fit(uint32_t tile_right, size_t smem_cap) {
  for (uint32_t n = kMaxStageBufs; n > 1; n--) {
    const WarpLayout c = warp_layout(tile_right, n);
    if ((size_t)c.warp_words * 4 * kWarpsPerCta * 2 <= smem_cap) return c;
  }
  return warp_layout(tile_right, 1);
}

struct Counters {
  unsigned long long out_count;
  unsigned long long comparisons;
  unsigned long long ambiguous;
  unsigned long long long_pairs;
  unsigned long long work_next;
  unsigned long long watchdog_trips;
  unsigned long long items_done;
  unsigned long long jw_word_ops;  // algorithmic work of the JW evaluations
  unsigned long long seen_overflow;  // nonzero: the duplicate set had no room (run repeats)
  unsigned long long passes;  // matches taken through the duplicate set (first_report)
  unsigned long long firsts;  // those of them that were reported (k_count_firsts, after an overflow)
  unsigned long long scans;       // pairs that reached a bit-parallel scan
  unsigned long long scan_steps;  // scan steps of 4 symbols
  unsigned long long items_total; // work items of the run (written by the join)
  unsigned long long scan_warp_steps;  // warp-level scan steps (any lane scanning)
  unsigned long long rest_scans;       // scans of predicates after a rule's or group's first
  unsigned long long work_next_long;   // k_eval_long's work_next
  unsigned long long deferred;       // pairs put on EvalParams::defer (and those it had no room for)
  unsigned long long deferred_next;  // and taken from it
};

static_assert(sizeof(Counters) % 8 == 0, "reported in 8-byte words");

// Distinct pairs of a run; with a full duplicate set an upper bound: the pairs
// that did not go through it, and every match that did (after read_firsts).
inline unsigned long long pair_count(const Counters& c) {
  return c.seen_overflow ? c.out_count - c.firsts + c.passes : c.out_count;
}

struct EvalParams {
  Side L, R;
  const Rule* rules;
  uint32_t n_rules;
  uint32_t n_symbols;
  // [n_rules + 1], global item space of the class this launch evaluates (the
  // two halves of ItemBases)
  const unsigned long long* rule_item_base;
  // Work list of the launch: every item (n_seg == 0, the batched form), or the
  // concatenation of item ranges [seg_begin[k], seg_end[k]) (the plain form:
  // one partition of one rule).
  uint32_t n_seg;
  unsigned long long seg_begin[kMaxSegments];
  unsigned long long seg_end[kMaxSegments];
  uint32_t tile_right;  // TR: right rows per work item
  uint32_t stage_rows;  // right rows per staging buffer (a multiple of 32)
  // shared-memory words per warp and offsets inside a warp's region (warp_layout)
  uint32_t warp_words, n_bufs, buf_off, buf_words, buf_rows_off, buf_lmeta_off, mbar_off, ctl_off;
  // Peq tables of the left strings (PeqShape): [left string slot][left row]
  const uint32_t* peq;
  uint32_t peq_w, tab_words, fast_max;
  uint32_t* out_l;
  uint32_t* out_r;
  unsigned long long capacity;
  Counters* ctr;
  unsigned long long watchdog_cycles;  // 0 = no budget
  // Pairs that reached a predicate whose left string has no Peq table, for
  // k_eval_long: {left row, right row, rule, live members}; null: decided in
  // the lane, as are those it has no room for
  uint4* defer;
  uint32_t defer_cap;
  uint32_t long_what;  // k_eval_long: bit 0 = work items, bit 1 = deferred pairs
  // set of the reported (left, right) keys that another rule may report too
  // (plans with several rules, else null)
  unsigned long long* seen;
  unsigned long long seen_mask;  // slots - 1 (a power of two minus one)
};

// Host: the shared-memory layout and Peq tables of a launch.
inline void set_layout(EvalParams* P, const WarpLayout& w, const PeqShape& s, const uint32_t* peq) {
  P->warp_words = w.warp_words;
  P->n_bufs = w.n_bufs;
  P->buf_off = w.buf_off;
  P->buf_words = w.buf_words;
  P->buf_rows_off = w.buf_rows_off;
  P->buf_lmeta_off = w.buf_lmeta_off;
  P->mbar_off = w.mbar_off;
  P->ctl_off = w.ctl_off;
  P->peq = peq;
  P->peq_w = s.w;
  P->tab_words = s.tab_words;
  P->fast_max = s.fast_max;
}

// ------------------------------------------------------------------ join
__global__ void k_keys_hist(Side S, const Rule* rules, uint32_t rule, int side);
__global__ void k_scatter(Side S, const Rule* rules, uint32_t rule, int side);
__global__ void k_scan_partial_u32(const uint32_t* in, uint32_t n, uint32_t* partial);
__global__ void k_scan_top_u32(uint32_t* partial, uint32_t nb);
__global__ void k_scan_final_u32(const uint32_t* in, uint32_t n, const uint32_t* partial,
                                 uint32_t* out);
// The same in one launch for up to kScanOnceChunks chunks: a block per chunk
// (taken from a ticket) adds the totals of the chunks before its own, as
// k_join_scan does; sync: one word per chunk and the ticket, zero before the
// launch.
constexpr uint32_t kScanOnceChunks = 2048;
// Polls (some 100 ns each) after which a single-launch scan or the sort gives
// up waiting for a chunk before its own and counts what lies before it itself;
// 0 with HBX_TEST_SCAN_GIVE_UP=1 in the environment: they count at once.
uint32_t scan_polls();
__global__ void k_scan_once_u32(const uint32_t* in, uint32_t n, uint32_t* out,
                                unsigned long long* sync, uint32_t polls);
__global__ void k_items_partial(const Rule* rules, uint32_t rule, uint32_t tile_right,
                                unsigned long long* partial, unsigned long long* comparisons);
__global__ void k_scan_top_u64(unsigned long long* partial, uint32_t nb);
__global__ void k_items_final(const Rule* rules, uint32_t rule, uint32_t tile_right,
                              const unsigned long long* partial);
// Item bases of a rule array: n_rules + 1 words for the items of class 0 (the
// first item of each rule, then their number), the same for class 1, then
// the number of all items.
inline size_t item_base_words(size_t n_rules) { return 2 * (n_rules + 1) + 1; }
#ifdef __CUDACC__
// Writes them; returns the number of all items.  A rule evaluated in another
// rule's group has no items of its own.
__device__ __forceinline__ unsigned long long item_bases(const Rule* rules, uint32_t n_rules,
                                                         unsigned long long* base) {
  unsigned long long acc = 0, acc1 = 0;
  for (uint32_t r = 0; r < n_rules; r++) {
    base[r] = acc;
    base[n_rules + 1 + r] = acc1;
    if (!rules[r].n_members) continue;
    const unsigned long long n0 = rules[r].item_off[rules[r].domain];
    acc += n0;
    acc1 += rules[r].item_off[rules[r].domain_l] - n0;
  }
  base[n_rules] = acc;
  base[2 * n_rules + 1] = acc1;
  base[2 * n_rules + 2] = acc + acc1;
  return acc + acc1;
}
#endif
__global__ void k_rule_base(const Rule* rules, uint32_t n_rules, unsigned long long* base);
// One launch for a run's resets: the counters and histograms to 0, the
// duplicate set (n_seen slots, may be 0) to empty.
__global__ void k_reset(Counters* ctr, uint32_t* counts, uint64_t n_counts,
                        unsigned long long* seen, uint64_t n_seen, unsigned long long* zero64,
                        uint64_t n_zero64);
// The join of a rule array in three launches, whatever the key domains.
// k_join_count and k_join_scatter run on grid (blocks, tasks): a task is one
// table of one rule (join_task).  Count: both tables of the rules with work
// items, the right one of the members that only count their comparisons;
// kSharedHistKeys * 4 bytes of dynamic shared memory, or 4 bytes per key of
// the largest domain when that is less.  Scatter: both tables of the rules
// with work items, the left one of the members.  k_join_scan runs
// a block per chunk of keys of each ScanTask; sync holds one word per block of
// its grid, then one ticket per task, zero before the launch (k_reset).
constexpr uint32_t kSharedHistKeys = 8192;
constexpr uint32_t kTaskRight = 1u << 31;
__host__ __device__ inline uint32_t join_task(uint32_t rule, int side) {
  return rule | (side ? kTaskRight : 0u);
}
// One scan of a rule's join: 0 = row offsets per left key, 1 = row offsets
// per right key, 2 = work items per left key with the rule's comparisons.
struct ScanTask {
  uint32_t rule, what, first_block, n_chunks;
};
// Keys of k_join_scan's chunks: kJoinChunk as long as all of them run at once
// (two blocks per SM), kWideJoinChunk above.
constexpr uint32_t kJoinChunk = 4096, kWideJoinChunk = 8192;
// Lays out the tasks' chunks (n_chunks holds their keys on entry); block_task
// gets the task of every block.  Returns the chunk.
inline uint32_t scan_chunks(int n_sm, std::vector<ScanTask>* tasks,
                            std::vector<uint32_t>* block_task) {
  uint64_t n = 0;
  for (const ScanTask& t : *tasks) n += ((uint64_t)t.n_chunks + kJoinChunk - 1) / kJoinChunk;
  const uint32_t chunk = n <= 2ull * (uint64_t)n_sm ? kJoinChunk : kWideJoinChunk;
  for (size_t i = 0; i < tasks->size(); i++) {
    ScanTask& t = (*tasks)[i];
    t.first_block = (uint32_t)block_task->size();
    t.n_chunks = (uint32_t)(((uint64_t)t.n_chunks + chunk - 1) / chunk);
    block_task->insert(block_task->end(), t.n_chunks, (uint32_t)i);
  }
  return chunk;
}
__global__ void k_join_count(Side L, Side R, const Rule* rules, const uint32_t* tasks);
// comparisons: rule r's pair-comparisons are added to comparisons[r *
// cmp_stride].
struct JoinScan {
  void (*kernel)(const Rule* rules, uint32_t tile_right, const ScanTask* tasks,
                 const uint32_t* block_task, unsigned long long* sync,
                 unsigned long long* comparisons, uint32_t cmp_stride, uint32_t polls);
  int threads;
};
JoinScan join_scan(uint32_t chunk);  // k_join_scan for a chunk of scan_chunks
__global__ void k_join_scatter(Side L, Side R, const Rule* rules, uint32_t n_rules,
                               const uint32_t* tasks, unsigned long long* rule_base,
                               Counters* ctr);
// ------------------------------------------------------------------ evaluation
// The planner's sample: for row pair k (x: left row, y: right row) and each
// pair of string columns (blockIdx.y; string metadata of the whole columns)
// {left length, right length, match count, common prefix} into out[column *
// n + k]; count 0xffffffff, not counted here, when both strings are longer
// than kMaxTableLen symbols.  A warp per pair.
constexpr uint32_t kSampleBatch = 8;
struct SampleCols {
  const StrMeta *l[kSampleBatch], *r[kSampleBatch];
};
__global__ void k_sample(const __grid_constant__ SampleCols cols, const uint8_t* arena_l,
                         const uint8_t* arena_r, const uint2* rows, uint32_t n, uint4* out);
// Peq tables of every left string of n_slots string slots (PeqShape).
__global__ void k_peq_build(Side L, uint32_t n_slots, PeqShape shape, uint32_t* peq);
// The evaluation kernel for masks of peq_w words (PeqShape::w): k_eval<W>
// (3 CTAs per SM, register-limited) or k_eval_wide<W> (2 CTAs per SM, more
// registers), or the same two over rule groups (k_eval_groups<W>,
// k_eval_groups_wide<W>: launches where some rule evaluates others).
using EvalKernel = void (*)(EvalParams);
// The work items of left strings without a Peq table (class 1; rule_item_base
// points at their bases) and the pairs that the evaluation kernels deferred
// (EvalParams::long_what), for groups and rules alike: grid long_grid(number
// of SMs), kWarpsPerCta * 32 threads.
__global__ void k_eval_long(const __grid_constant__ EvalParams P);
inline int long_grid(int n_sm) { return n_sm * 4; }
constexpr uint32_t kDeferPairs = 1u << 20;  // most room for deferred pairs of a run
EvalKernel eval_kernel(int wide, bool groups, uint32_t peq_w);
// Counts the reports that went through a duplicate set, its taken slots (a run
// whose set overflowed only: the evaluation itself does not count them, which
// would cost it 0.6 %).
__global__ void k_count_firsts(const unsigned long long* seen, uint64_t n_seen, Counters* ctr);
// words and, if there are at most limit of them (and capacity), the pairs to
// page-locked host memory: h_out holds the left rows, then the right rows.
__global__ void k_report(const unsigned long long* words, uint32_t n_words, const Counters* ctr,
                         const uint32_t* l, const uint32_t* r, unsigned long long capacity,
                         unsigned long long limit, unsigned long long* h_words, uint32_t* h_out);
constexpr uint32_t kPeqWidths[] = {1, 2, 3, 4, 8};  // every PeqShape::w

constexpr uint32_t kScanChunk = 4096;  // elements per CTA in the scans (1024 threads x 4)

}  // namespace dev
}  // namespace hbx
