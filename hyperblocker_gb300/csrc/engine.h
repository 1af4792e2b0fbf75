// engine.h -- engine entry points used by other translation units.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>
#include <vector>

#include "../../include/hbx.h"

namespace hbx {

// Runs a session (batched or plain) on its context's stream and copies its
// pairs, exactly sized, into host vectors.
void run_to_host(hbx_session* s, hbx_mode mode, std::vector<uint32_t>* l, std::vector<uint32_t>* r);
// Grows a session's own output (and duplicate set) to at least `pairs`
// slots before a run, so that a run expected to produce that many pairs
// does not overflow and repeat.
void reserve_output(hbx_session* s, uint64_t pairs);
struct Table;
struct Plan;
struct PlanSample;
struct PairCount;
struct Encoded;
struct SideBufs;
// The planner's sample counted on encoded tables (rows: x left, y right), and
// the order of *plan's predicates from those counts.
std::vector<PairCount> count_samples(const Encoded& E, const SideBufs& L, const SideBufs& R,
                                     const std::vector<std::pair<int, int>>& columns,
                                     const std::vector<uint2>& rows, cudaStream_t st);
void rank_by_counts(Plan* plan, const PlanSample& sample, const Table& left, const Table& right,
                    const std::vector<PairCount>& counts);
// After a run whose duplicate set (n_seen slots) overflowed: c->firsts, counted
// on st and waited for.
void read_firsts(const unsigned long long* seen, uint64_t n_seen, dev::Counters* d_ctr,
                 dev::Counters* c, int n_sm, cudaStream_t st);
// sort.cu: sorts n device pairs by (left row, right row) in place; the first
// form queues it on st.
void queue_pair_sort(int n_sm, cudaStream_t st, uint32_t* l, uint32_t* r, uint64_t n,
                     uint32_t n_left, uint32_t n_right);
// Device memory that takes besides the pairs, while it runs.
uint64_t pair_sort_bytes(int n_sm, uint64_t n, uint32_t n_left, uint32_t n_right);
void sort_pairs_device(hbx_ctx* ctx, uint32_t* l, uint32_t* r, uint64_t n, uint32_t n_left,
                       uint32_t n_right);
// writer.cu: appends the id lines of n device pairs to path.
void write_pairs_device(hbx_ctx* ctx, const Table& left, const Table& right, const uint32_t* l_row,
                        const uint32_t* r_row, uint64_t n, const char* path);

}  // namespace hbx
