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
  PairCount count(const char* a, size_t la, const char* b, size_t lb) {
    PairCount c{(uint32_t)la, (uint32_t)lb, 0, 0};
    if (la == 0 || lb == 0) return c;
    if (la > lb) {
      std::swap(a, b);
      std::swap(la, lb);
    }
    const size_t h = (la + 1) / 2, words = (la + 63) / 64;
    if (mask_.size() < 256 * words) mask_.assign(256 * words, 0);
    free_.assign(words, ~0ull);
    for (size_t j = 0; j < la; j++) mask_[(uint8_t)a[j] * words + j / 64] |= 1ull << (j % 64);
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
        c.m++;
        break;
      }
    }
    for (size_t j = 0; j < la; j++) mask_[(uint8_t)a[j] * words + j / 64] = 0;
    while (c.p < la && a[c.p] == b[c.p]) c.p++;
    return c;
  }

 private:
  std::vector<uint64_t> mask_, free_;  // mask_: zero between calls
};

double jaro_winkler(const PairCount& c) {
  if (c.la == 0 || c.lb == 0) return (c.la == 0 && c.lb == 0) ? 1.0 : 0.0;
  if (!c.m) return 0.0;
  const size_t ls = std::min(c.la, c.lb), ll = std::max(c.la, c.lb);
  double j = ((double)c.m / ls + (double)c.m / ll + 1.0) / 3.0;
  j += (1.0 - j) * (double)c.p * 0.1;
  return j > 1.0 ? 1.0 : j;
}

}  // namespace

PlanSample sample_plan(const Plan& plan, const Table& left, const Table& right) {
  PlanSample out;
  if (left.n_rows == 0 || right.n_rows == 0) return out;
  // rules test the same few columns at different thresholds: each pair of
  // columns is sampled once
  for (auto& cr : plan.compiled) {
    if (cr.sims.size() < 2) continue;
    for (auto& p : cr.sims) {
      const std::pair<int, int> c(p.col_l, p.col_r);
      if (p.col_l < left.n_cols() && p.col_r < right.n_cols() &&
          std::find(out.cols.begin(), out.cols.end(), c) == out.cols.end())
        out.cols.push_back(c);
    }
  }
  if (out.cols.empty()) return out;
  const int kSamples = 2048;
  uint64_t state = 0x48594250ull;
  auto next = [&]() {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return state >> 17;
  };
  for (int i = 0; i < kSamples; i++) {
    const int64_t l = (int64_t)(next() % (uint64_t)left.n_rows);
    out.rows.emplace_back(l, (int64_t)(next() % (uint64_t)right.n_rows));
  }
  return out;
}

ColumnSample column_sample(const PlanSample& sample, std::pair<int, int> cols, const Table& left,
                           const Table& right, const PairCount* counts) {
  const Column& cl = left.cols[(size_t)cols.first];
  const Column& cr = right.cols[(size_t)cols.second];
  ColumnSample s;
  Sampler sampler;
  for (size_t k = 0; k < sample.rows.size(); k++) {
    const auto& pr = sample.rows[k];
    PairCount c = counts ? counts[k] : PairCount{0, 0, kNotCounted, 0};
    if (c.m == kNotCounted)
      c = sampler.count(cl.ptr(pr.first), c_len(cl, pr.first), cr.ptr(pr.second), c_len(cr, pr.second));
    s.cost += (double)c.lb * (double)((std::min<size_t>(c.la, 256) + 31) / 32 + 2);
    s.jw.push_back(jaro_winkler(c));
  }
  s.cost /= (double)sample.rows.size();
  return s;
}

void rank_predicates(Plan* plan, const PlanSample& sample, const std::vector<ColumnSample>& values) {
  if (sample.cols.empty()) return;
  for (auto& cr : plan->compiled) {
    if (cr.sims.size() < 2) continue;
    std::vector<double> rank(cr.sims.size());
    for (size_t s = 0; s < cr.sims.size(); s++) {
      const Pred& p = cr.sims[s];
      const auto it = std::find(sample.cols.begin(), sample.cols.end(), std::make_pair(p.col_l, p.col_r));
      if (it == sample.cols.end()) {
        rank[s] = 1e30;
        continue;
      }
      const ColumnSample& c = values[(size_t)(it - sample.cols.begin())];
      double pass = 0;
      for (double v : c.jw)
        if (v >= (double)p.thr) pass += 1;
      pass /= (double)c.jw.size();
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

void order_predicates(Plan* plan, const Table& left, const Table& right) {
  const PlanSample sample = sample_plan(*plan, left, right);
  std::vector<ColumnSample> values;
  for (auto& c : sample.cols) values.push_back(column_sample(sample, c, left, right, nullptr));
  rank_predicates(plan, sample, values);
}

}  // namespace hbx
