// kernels.cu -- sm_103a kernels of the blocking engine (see kernels.cuh).
#include <cstdlib>
#include <cstring>

#include "kernels.cuh"
#include "bitscan.cuh"

namespace hbx {
namespace dev {

constexpr unsigned kFull = 0xffffffffu;

// =====================================================================
// Join: keys, histograms, scans, scatter
// =====================================================================

__device__ __forceinline__ uint32_t row_key(const Side& S, const Rule& R, uint32_t row) {
  if (R.composite) return (uint32_t)S.comp_codes[(size_t)R.comp_index * S.n_rows + row];
  uint32_t key = S.bucket[row];
  for (uint32_t e = 0; e < R.n_eq; e++)
    key = key * R.radix[e] + (uint32_t)S.eq_codes[(size_t)R.eq_slot[e] * S.n_rows + row];
  return key;
}

__global__ void k_keys_hist(Side S, const Rule* rules, uint32_t rule, int side) {
  const Rule& R = rules[rule];
  uint32_t* keys = side ? R.key_r : R.key_l;
  uint32_t* cnt = side ? R.cnt_r : R.cnt_l;
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < S.n_rows;
       row += gridDim.x * blockDim.x) {
    uint32_t k = row_key(S, R, row);
    if (!side) k = left_key(R, S, row, k);
    keys[row] = k;
    atomicAdd(cnt + k, 1u);
  }
}

// Stores a right row's metadata at position pos of sorted_meta_r (its pieces
// turned, meta_turn): the string metadata of the rule's first similarity
// column, with the row's dictionary codes of the group's first two extra
// equality slots in loc.z and loc.w (unused words of the string record), so
// that the filter compares them from the staged copy.
__device__ __forceinline__ void store_meta(const Side& S, const Rule& Q, const StrMeta* meta_in,
                                           uint32_t row, uint32_t pos) {
  StrMeta m = meta_in[row];
  if (Q.n_xslots > 0) m.loc.z = (uint32_t)S.eq_codes[(size_t)Q.xslot[0] * S.n_rows + row];
  if (Q.n_xslots > 1) m.loc.w = (uint32_t)S.eq_codes[(size_t)Q.xslot[1] * S.n_rows + row];
  uint4* out = reinterpret_cast<uint4*>(Q.sorted_meta_r + pos);
  const uint32_t t = meta_turn(pos);
  out[t] = m.loc;
  out[1u ^ t] = m.head;
  out[2u ^ t] = m.sig[0];
  out[3u ^ t] = m.sig[1];
}

__global__ void k_scatter(Side S, const Rule* rules, uint32_t rule, int side) {
  const Rule& R = rules[rule];
  if (!R.n_members) return;  // evaluated in another rule's group: no items of its own
  const uint32_t* keys = side ? R.key_r : R.key_l;
  const uint32_t* off = side ? R.off_r : R.off_l;
  uint32_t* cur = side ? R.cur_r : R.cur_l;
  uint32_t* sorted = side ? R.sorted_r : R.sorted_l;
  StrMeta* meta_out = side ? R.sorted_meta_r : nullptr;
  const StrMeta* meta_in = S.str_meta + (size_t)R.sim_r[0] * S.n_rows;
  for (uint32_t row = blockIdx.x * blockDim.x + threadIdx.x; row < S.n_rows;
       row += gridDim.x * blockDim.x) {
    const uint32_t k = keys[row];
    const uint32_t pos = off[k] + atomicAdd(cur + k, 1u);
    sorted[pos] = row;
    if (meta_out) store_meta(S, R, meta_in, row, pos);
  }
}

// Block-wide exclusive scan of a value per thread.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* s_warp, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(kFull, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = (lane < (int)(blockDim.x >> 5)) ? s_warp[lane] : T(0);
    T z = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(kFull, z, o);
      if (lane >= o) z += y;
    }
    s_warp[lane] = z - w;  // exclusive prefix of warp sums
    if (lane == 31) *total = z;
  }
  __syncthreads();
  const T r = s_warp[warp] + x - v;
  __syncthreads();
  return r;
}

// A chunk's word in a single-launch scan: the chunk's total, or the sum of it
// and of all chunks before (kScanSum has the bit of kScanCount too).
constexpr unsigned long long kScanCount = 1ull << 63, kScanSum = 3ull << 62;
constexpr unsigned long long kScanValue = ~kScanSum;

uint32_t scan_polls() {
  const char* e = std::getenv("HBX_TEST_SCAN_GIVE_UP");
  return e && std::strcmp(e, "1") == 0 ? 0u : 1u << 20;
}

// Publishes chunk c's total and sums the chunks before it into *s_base
// (shared; complete when this returns): a window of blockDim.x chunks at a
// time, a thread each, back to the nearest that has published its sum, which
// is one window as long as fewer blocks run at once.  (Adding up every chunk
// before, by atomic reads, was most of the join's scans at large domains:
// 5,860 chunks of three rules' scans took 227 us, with this and vector
// accesses 203.)  Every thread of the block calls it; false in all of them: a
// wait gave up after `polls` polls (scan_polls), and the caller adds up what
// lies before the chunk itself (scan_recount).  The caller publishes the sum.
__device__ __forceinline__ bool scan_lookback(unsigned long long* words, uint32_t c,
                                              unsigned long long total, uint32_t polls,
                                              unsigned long long* s_base) {
  __shared__ uint32_t s_near;
  volatile unsigned long long* w = words;
  bool ok = true;
  if (threadIdx.x == 0) {
    *s_base = 0;
    w[c] = total | (c ? kScanCount : kScanSum);
  }
  for (uint32_t end = c; end != 0; end = end > blockDim.x ? end - blockDim.x : 0u) {
    if (threadIdx.x == 0) s_near = ~0u;
    __syncthreads();
    unsigned long long f = 0;
    if (threadIdx.x < end) {
      uint32_t left = polls;
      while (left && !((f = w[end - 1 - threadIdx.x]) & kScanCount)) {
        left--;
        __nanosleep(64);
      }
      ok = ok && (f & kScanCount);
    }
    const unsigned sums = __ballot_sync(kFull, (f & kScanSum) == kScanSum);
    if (sums && (int)(threadIdx.x & 31) == __ffs(sums) - 1) atomicMin(&s_near, threadIdx.x);
    __syncthreads();
    const uint32_t near = s_near;
    unsigned long long t = threadIdx.x <= near ? f & kScanValue : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(s_base, t);
    __syncthreads();
    if (near != ~0u) break;
  }
  return !__syncthreads_or(!ok);
}

// The block's sum of value(k) for k below n, into *s_base (complete when this
// returns).
template <class F>
__device__ __forceinline__ void scan_recount(uint64_t n, unsigned long long* s_base, F&& value) {
  if (threadIdx.x == 0) *s_base = 0;
  __syncthreads();
  unsigned long long t = 0;
  for (uint64_t k = threadIdx.x; k < n; k += blockDim.x) t += value(k);
  atomicAdd(s_base, t);
  __syncthreads();
}

// Four consecutive values from index b on, those at n and above 0; in one
// access where they lie on a 16-byte boundary.
__device__ __forceinline__ uint4 load4(const uint32_t* p, uint32_t b, uint32_t n) {
  if (b + 3 < n && ((uintptr_t)(p + b) & 15) == 0) return *reinterpret_cast<const uint4*>(p + b);
  return make_uint4(b < n ? p[b] : 0u, b + 1 < n ? p[b + 1] : 0u, b + 2 < n ? p[b + 2] : 0u,
                    b + 3 < n ? p[b + 3] : 0u);
}
__device__ __forceinline__ void store4(uint32_t* p, uint32_t b, uint32_t n, uint4 v) {
  if (b + 3 < n && ((uintptr_t)(p + b) & 15) == 0) {
    *reinterpret_cast<uint4*>(p + b) = v;
    return;
  }
  if (b < n) p[b] = v.x;
  if (b + 1 < n) p[b + 1] = v.y;
  if (b + 2 < n) p[b + 2] = v.z;
  if (b + 3 < n) p[b + 3] = v.w;
}

__global__ void k_scan_once_u32(const uint32_t* in, uint32_t n, uint32_t* out,
                                unsigned long long* sync, uint32_t polls) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_total, s_chunk;
  __shared__ unsigned long long s_base;
  if (threadIdx.x == 0) s_chunk = (uint32_t)atomicAdd(sync + gridDim.x, 1ull);
  __syncthreads();
  const uint32_t c = s_chunk;
  const uint32_t b = c * kScanChunk + threadIdx.x * 4u;
  const uint4 v = load4(in, b, n);
  uint32_t ex = block_excl_scan<uint32_t>(v.x + v.y + v.z + v.w, s_warp, &s_total);
  if (!scan_lookback(sync, c, s_total, polls, &s_base))
    scan_recount((uint64_t)c * kScanChunk, &s_base, [&](uint64_t k) { return in[k]; });
  if (threadIdx.x == 0)
    *static_cast<volatile unsigned long long*>(sync + c) = (s_base + s_total) | kScanSum;
  ex += (uint32_t)s_base;
  store4(out, b, n, make_uint4(ex, ex + v.x, ex + v.x + v.y, ex + v.x + v.y + v.z));
}

__global__ void k_scan_partial_u32(const uint32_t* in, uint32_t n, uint32_t* partial) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_total;
  const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + threadIdx.x * 4u;
  uint32_t v = 0;
  for (int k = 0; k < 4; k++)
    if (base + k < n) v += in[base + k];
  block_excl_scan<uint32_t>(v, s_warp, &s_total);
  if (threadIdx.x == 0) partial[blockIdx.x] = s_total;
}

template <typename T>
__device__ void scan_top(T* partial, uint32_t nb) {
  __shared__ T s_warp[32];
  __shared__ T s_total;
  T carry = 0;
  for (uint32_t b0 = 0; b0 < nb; b0 += blockDim.x) {
    const uint32_t i = b0 + threadIdx.x;
    const T v = i < nb ? partial[i] : T(0);
    const T ex = block_excl_scan<T>(v, s_warp, &s_total);
    if (i < nb) partial[i] = carry + ex;
    carry += s_total;
    __syncthreads();
  }
}

__global__ void k_scan_top_u32(uint32_t* partial, uint32_t nb) { scan_top<uint32_t>(partial, nb); }
__global__ void k_scan_top_u64(unsigned long long* partial, uint32_t nb) {
  scan_top<unsigned long long>(partial, nb);
}

__global__ void k_scan_final_u32(const uint32_t* in, uint32_t n, const uint32_t* partial,
                                 uint32_t* out) {
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_total;
  const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + threadIdx.x * 4u;
  uint32_t v[4];
  uint32_t sum = 0;
  for (int k = 0; k < 4; k++) {
    v[k] = (base + k < n) ? in[base + k] : 0u;
    sum += v[k];
  }
  uint32_t ex = block_excl_scan<uint32_t>(sum, s_warp, &s_total) + partial[blockIdx.x];
  for (int k = 0; k < 4; k++) {
    if (base + k < n) out[base + k] = ex;
    ex += v[k];
  }
}

// Work items of a key with nl left and nr right rows, and its pairs.
__device__ __forceinline__ unsigned long long n_items(uint32_t nl, uint32_t nr, uint32_t tile_right,
                                                      unsigned long long* pairs) {
  *pairs = (unsigned long long)nl * nr;
  if (!nl || !nr) return 0;
  return (unsigned long long)nl * ((nr + tile_right - 1) / tile_right);
}

// Work items of left key j.
__device__ __forceinline__ unsigned long long key_items(const Rule& R, uint32_t j,
                                                        uint32_t tile_right,
                                                        unsigned long long* pairs) {
  const uint32_t nl = R.cnt_l[j];
  return n_items(nl, nl ? R.cnt_r[join_key(R, j)] : 0u, tile_right, pairs);
}

__global__ void k_items_partial(const Rule* rules, uint32_t rule, uint32_t tile_right,
                                unsigned long long* partial, unsigned long long* comparisons) {
  __shared__ unsigned long long s_warp[32];
  __shared__ unsigned long long s_total;
  const Rule& R = rules[rule];
  const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + threadIdx.x * 4u;
  unsigned long long v = 0, pr = 0;
  for (int k = 0; k < 4; k++)
    if (base + k < R.domain_l) {
      unsigned long long p;
      v += key_items(R, (uint32_t)(base + k), tile_right, &p);
      pr += p;
    }
  block_excl_scan<unsigned long long>(v, s_warp, &s_total);
  if (threadIdx.x == 0) partial[blockIdx.x] = s_total;
  __shared__ unsigned long long s_pairs;
  block_excl_scan<unsigned long long>(pr, s_warp, &s_pairs);
  if (threadIdx.x == 0 && s_pairs) atomicAdd(comparisons, s_pairs);
}

__global__ void k_items_final(const Rule* rules, uint32_t rule, uint32_t tile_right,
                              const unsigned long long* partial) {
  __shared__ unsigned long long s_warp[32];
  __shared__ unsigned long long s_total;
  const Rule& R = rules[rule];
  const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + threadIdx.x * 4u;
  unsigned long long v[4], sum = 0, p;
  for (int k = 0; k < 4; k++) {
    v[k] = (base + k < R.domain_l) ? key_items(R, (uint32_t)(base + k), tile_right, &p) : 0ull;
    sum += v[k];
  }
  unsigned long long ex =
      block_excl_scan<unsigned long long>(sum, s_warp, &s_total) + partial[blockIdx.x];
  for (int k = 0; k < 4; k++) {
    if (base + k < R.domain_l) R.item_off[base + k] = ex;
    ex += v[k];
    if (base + k + 1 == R.domain_l) R.item_off[R.domain_l] = ex;
  }
}

// Programmatic dependent launch: a kernel launched with the programmatic
// stream serialization attribute (launch_dependent) may start while the
// kernel before it still runs; it waits here before it reads anything that
// kernel writes (every write of the earlier grid is visible after the wait).
// Without the attribute both are no-ops.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel in the stream start its blocks (they wait in
// pdl_wait); called once every block of this grid has started.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;"); }

// ---- the join of every rule of a session: one launch for keys + histograms,
// one for offsets + work items, one for the scatter, each covering every
// rule and both tables.  The row kernels run one block row per task
// (blockIdx.y: one table of one rule), so the rules' and tables' dependent
// load -> atomic -> store chains run side by side.
//
// A rule evaluated in another rule's group needs no offsets, only its number
// of pair-comparisons, sum over left rows of the right rows with their key:
// its right rows are counted with the others' and its left rows add up their
// counts in the scatter launch, so no pass runs over its key domain (8 rules,
// 30,012 x 29,990 rows: the key + venue rules have 64 partitions x 250 keys x
// 500 venues = 8M keys).  Bound by launches and memory latency: reset, count,
// scan and scatter take 36 us there and 115 us at 150k x 150k rows, against
// 1.57 and 1.83 ms with a scan of every rule's domain, times 5 length
// classes, in launches per rule; 35 us against 44 us for 2 rules, 2,601 x
// 64,264 rows.

// Keys and key histograms of every task's rule and table; histograms of
// domains up to kSharedHistKeys are kept per block in shared memory.
__global__ void k_join_count(Side L, Side R, const Rule* rules, const uint32_t* tasks) {
  extern __shared__ uint32_t s_cnt[];
  pdl_trigger();
  pdl_wait();  // the histograms are cleared (k_reset)
  const uint32_t task = tasks[blockIdx.y];
  const int side = task & kTaskRight ? 1 : 0;
  const Side& S = side ? R : L;
  if ((unsigned long long)blockIdx.x * blockDim.x >= S.n_rows) return;  // whole block
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const Rule& Q = rules[task & ~kTaskRight];
  const uint32_t D = side ? Q.domain : Q.domain_l;
  uint32_t* keys = !Q.n_members ? nullptr : side ? Q.key_r : Q.key_l;
  uint32_t* cnt = side ? Q.cnt_r : Q.cnt_l;
  const bool sh = D <= kSharedHistKeys;
  if (sh) {
    for (uint32_t k = threadIdx.x; k < D; k += blockDim.x) s_cnt[k] = 0;
    __syncthreads();
  }
  for (uint32_t row = t0; row < S.n_rows; row += stride) {
    uint32_t k = row_key(S, Q, row);
    if (!side) k = left_key(Q, S, row, k);
    if (keys) keys[row] = k;
    atomicAdd(sh ? s_cnt + k : cnt + k, 1u);
  }
  if (sh) {
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < D; k += blockDim.x)
      if (s_cnt[k]) atomicAdd(cnt + k, s_cnt[k]);
  }
}

// The rows of keys below n, and the work items of left keys below n, for a
// block whose wait gave up (out of line: the scans' registers are for their keys).
__device__ __noinline__ void recount_rows(const uint32_t* cnt, uint32_t n, unsigned long long* s_base) {
  scan_recount(n, s_base, [&](uint64_t k) { return cnt[k]; });
}
__device__ __noinline__ void recount_items(const Rule& R, uint32_t tile_right, uint32_t n,
                                           unsigned long long* s_base) {
  scan_recount(n, s_base, [&](uint64_t k) {
    unsigned long long pairs;
    return key_items(R, (uint32_t)k, tile_right, &pairs);
  });
}

// The scans of every rule with work items (ScanTask), one block per
// chunk of keys, in one launch.  A block takes its
// chunk from its task's ticket counter when it starts, publishes the chunk's
// total before it reads anything of the other chunks, and looks back over
// those before its own: their blocks took their tickets earlier, so they are
// running or done, and every wait ends (bounded all the same: a block whose
// wait gave up adds up the counts before its chunk itself).
// A block takes some 10 us whatever it holds (its task, its ticket, the look
// back), so where there are more chunks than blocks run at once a block holds
// 8,192 keys, 16 a thread, instead of 4,096, eight a thread (scan_chunks):
// three scans of 8 million keys each take 108 us against 203, but 1 to 2 us
// more where all chunks run at once (2,617 x 2,295 rows: 17.6 against 15.6 us
// of join, measured with 1,024 threads of four keys; 512 of eight take the same
// and have the registers for the recount without spills).
template <int kThreads, int kKeys>
__global__ void __launch_bounds__(kThreads, 2) k_join_scan(
    const Rule* rules, uint32_t tile_right, const ScanTask* tasks, const uint32_t* block_task,
    unsigned long long* sync, unsigned long long* comparisons, uint32_t cmp_stride, uint32_t polls) {
  __shared__ unsigned long long s_w64[32];
  __shared__ unsigned long long s_t64, s_base;
  __shared__ uint32_t s_chunk;
  constexpr int kVec = kKeys / 4;
  pdl_trigger();
  pdl_wait();  // the histograms are complete (k_join_count)
  const uint32_t ti = block_task[blockIdx.x];
  if (threadIdx.x == 0) s_chunk = (uint32_t)atomicAdd(sync + gridDim.x + ti, 1ull);
  const ScanTask T = tasks[ti];
  unsigned long long* totals = sync + T.first_block;
  const Rule& Q = rules[T.rule];
  const uint32_t D = T.what == 1 ? Q.domain : Q.domain_l;
  __syncthreads();
  const uint32_t c = s_chunk;
  const uint32_t chunk0 = c * (kThreads * kKeys), b = chunk0 + threadIdx.x * kKeys;
  if (T.what != 2) {  // row counts
    const uint32_t* cnt = T.what == 1 ? Q.cnt_r : Q.cnt_l;
    uint4 v[kVec];
    uint32_t ex;
    for (bool again = false;; again = true) {
      unsigned long long sum = 0;
#pragma unroll
      for (int k = 0; k < kVec; k++) v[k] = load4(cnt, b + 4 * k, D);
#pragma unroll
      for (int k = 0; k < kVec; k++) sum += v[k].x + v[k].y + v[k].z + v[k].w;
      ex = (uint32_t)block_excl_scan<unsigned long long>(sum, s_w64, &s_t64);
      // (after a recount the keys are loaded again: nothing is kept across it)
      if (again || scan_lookback(totals, c, s_t64, polls, &s_base)) break;
      recount_rows(cnt, chunk0, &s_base);
    }
    if (threadIdx.x == 0)
      *static_cast<volatile unsigned long long*>(totals + c) = (s_base + s_t64) | kScanSum;
    ex += (uint32_t)s_base;
    uint32_t* off = T.what == 1 ? Q.off_r : Q.off_l;
#pragma unroll
    for (int k = 0; k < kVec; k++) {
      const uint4 o = make_uint4(ex, ex + v[k].x, ex + v[k].x + v[k].y, ex + v[k].x + v[k].y + v[k].z);
      store4(off, b + 4 * k, D, o);
      ex = o.w + v[k].w;
    }
    return;
  }
  // work items
  uint4 nl[kVec], nr[kVec];
  const uint32_t m = Q.domain;
  unsigned long long pairs, ex, p;
  for (bool again = false;; again = true) {
#pragma unroll
    for (int k = 0; k < kVec; k++) {
      const uint32_t j = b + 4 * k;
      nl[k] = load4(Q.cnt_l, j, D);
      if (j + 3 < m) {
        nr[k] = load4(Q.cnt_r, j, m);
      } else {  // class 1, or beyond the keys (0 left rows)
        nr[k].x = nl[k].x ? Q.cnt_r[join_key(Q, j)] : 0u;
        nr[k].y = nl[k].y ? Q.cnt_r[join_key(Q, j + 1)] : 0u;
        nr[k].z = nl[k].z ? Q.cnt_r[join_key(Q, j + 2)] : 0u;
        nr[k].w = nl[k].w ? Q.cnt_r[join_key(Q, j + 3)] : 0u;
      }
    }
    unsigned long long items = 0;
    pairs = 0;
#pragma unroll
    for (int k = 0; k < kVec; k++) {
      items += n_items(nl[k].x, nr[k].x, tile_right, &p);
      pairs += p;
      items += n_items(nl[k].y, nr[k].y, tile_right, &p);
      pairs += p;
      items += n_items(nl[k].z, nr[k].z, tile_right, &p);
      pairs += p;
      items += n_items(nl[k].w, nr[k].w, tile_right, &p);
      pairs += p;
    }
    ex = block_excl_scan<unsigned long long>(items, s_w64, &s_t64);
    if (again || scan_lookback(totals, c, s_t64, polls, &s_base)) break;
    recount_items(Q, tile_right, chunk0, &s_base);
  }
  if (threadIdx.x == 0) {
    const unsigned long long sum = s_base + s_t64;
    *static_cast<volatile unsigned long long*>(totals + c) = sum | kScanSum;
    if (c + 1 == T.n_chunks) Q.item_off[D] = sum;
  }
  ex += s_base;
#pragma unroll
  for (int k = 0; k < kVec; k++) {
    const uint32_t j = b + 4 * k;
    const unsigned long long e1 = ex + n_items(nl[k].x, nr[k].x, tile_right, &p);
    const unsigned long long e2 = e1 + n_items(nl[k].y, nr[k].y, tile_right, &p);
    const unsigned long long e3 = e2 + n_items(nl[k].z, nr[k].z, tile_right, &p);
    if (j + 3 < D && ((uintptr_t)(Q.item_off + j) & 15) == 0) {
      ulonglong2* to = reinterpret_cast<ulonglong2*>(Q.item_off + j);
      to[0] = make_ulonglong2(ex, e1);
      to[1] = make_ulonglong2(e2, e3);
    } else {
      if (j < D) Q.item_off[j] = ex;
      if (j + 1 < D) Q.item_off[j + 1] = e1;
      if (j + 2 < D) Q.item_off[j + 2] = e2;
      if (j + 3 < D) Q.item_off[j + 3] = e3;
    }
    ex = e3 + n_items(nl[k].w, nr[k].w, tile_right, &p);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(kFull, pairs, o);
  if ((threadIdx.x & 31) == 0 && pairs)
    atomicAdd(comparisons + (size_t)T.rule * cmp_stride, pairs * Q.cmp_weight);
}

JoinScan join_scan(uint32_t chunk) {
  if (chunk == kJoinChunk) return {k_join_scan<512, 8>, 512};
  return {k_join_scan<512, 16>, 512};
}

// Rows of every rule with work items grouped by key (counting-sort scatter,
// right rows with their first similarity column's metadata), the
// pair-comparisons of the others, and the rules' item bases.
__global__ void k_join_scatter(Side L, Side R, const Rule* rules, uint32_t n_rules,
                               const uint32_t* tasks, unsigned long long* rule_base,
                               Counters* ctr) {
  pdl_trigger();
  pdl_wait();  // offsets and work items are complete (k_join_scan)
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    ctr->items_total = item_bases(rules, n_rules, rule_base);
  }
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t task = tasks[blockIdx.y];
  const Rule& Q = rules[task & ~kTaskRight];
  if (task & kTaskRight) {
    const StrMeta* meta_in = R.str_meta + (size_t)Q.sim_r[0] * R.n_rows;
    for (uint32_t row = t0; row < R.n_rows; row += stride) {
      const uint32_t k = Q.key_r[row];
      const uint32_t pos = Q.off_r[k] + atomicAdd(Q.cur_r + k, 1u);
      Q.sorted_r[pos] = row;
      if (Q.sorted_meta_r) store_meta(R, Q, meta_in, row, pos);
    }
  } else if (Q.n_members) {
    for (uint32_t row = t0; row < L.n_rows; row += stride) {
      const uint32_t k = Q.key_l[row];
      Q.sorted_l[Q.off_l[k] + atomicAdd(Q.cur_l + k, 1u)] = row;
    }
  } else {
    unsigned long long pairs = 0;
    for (uint32_t row = t0; row < L.n_rows; row += stride) pairs += Q.cnt_r[row_key(L, Q, row)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(kFull, pairs, o);
    if ((threadIdx.x & 31) == 0 && pairs) atomicAdd(&ctr->comparisons, pairs * Q.cmp_weight);
  }
}

__global__ void k_rule_base(const Rule* rules, uint32_t n_rules, unsigned long long* base) {
  if (threadIdx.x == 0 && blockIdx.x == 0) item_bases(rules, n_rules, base);
}

__global__ void k_reset(Counters* ctr, uint32_t* counts, uint64_t n_counts,
                        unsigned long long* seen, uint64_t n_seen, unsigned long long* zero64,
                        uint64_t n_zero64) {
  // launched in stream order (after the previous run); lets the join's first
  // kernel start its blocks early
  pdl_trigger();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  constexpr uint64_t kCtrWords = sizeof(Counters) / 8;
  for (uint64_t i = t0; i < kCtrWords; i += stride) reinterpret_cast<unsigned long long*>(ctr)[i] = 0;
  for (uint64_t i = t0; i < n_counts; i += stride) counts[i] = 0;
  for (uint64_t i = t0; i < n_seen; i += stride) seen[i] = ~0ull;
  for (uint64_t i = t0; i < n_zero64; i += stride) zero64[i] = 0ull;
}

// =====================================================================
// Jaro-Winkler
// =====================================================================

// One symbol row of a Peq table in device memory (plain loads: they need
// fewer registers around the scan than the read-only path's).
template <int S>
__device__ __forceinline__ void load_row(const uint32_t* row, uint32_t (&pe)[S]) {
  if constexpr (S == 1) {
    pe[0] = *row;
  } else if constexpr (S == 2) {
    const uint2 v = *reinterpret_cast<const uint2*>(row);
    pe[0] = v.x;
    pe[1] = v.y;
  } else if constexpr (S == 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(row);
    pe[0] = v.x;
    pe[1] = v.y;
    pe[2] = v.z;
    pe[3] = v.w;
  } else {
    const uint4 v = *reinterpret_cast<const uint4*>(row);
    const uint4 u = *reinterpret_cast<const uint4*>(row + 4);
    pe[0] = v.x;
    pe[1] = v.y;
    pe[2] = v.z;
    pe[3] = v.w;
    pe[4] = u.x;
    pe[5] = u.y;
    pe[6] = u.z;
    pe[7] = u.w;
  }
}

// The reference's Jaro loops (device_func.cuh:71-111) on symbol strings, with
// position 256 usable like any other (the reference's uint16_t idx[256] is
// indexed at 256 there).  Used for the predicates after the first of a pair
// whose left string there is longer than a Peq table covers.
__device__ __noinline__ uint32_t jaro_m_ref(const uint8_t* s1, uint32_t l1, const uint8_t* s2,
                                            uint32_t l2) {
  const uint8_t* s = s1;
  const uint8_t* t = s2;
  uint32_t ls = l1, lt = l2;
  if (l1 > l2) {
    s = s2;
    t = s1;
    ls = l2;
    lt = l1;
  }
  const uint32_t h = (ls + 1u) / 2u;
  uint32_t used[9];
#pragma unroll
  for (int k = 0; k < 9; k++) used[k] = 0;
  uint32_t m = 0;
  for (uint32_t i = 0; i < h; i++) {
    const uint8_t ti = t[i];
    for (uint32_t j = 0; j <= i + h; j++) {
      if (j >= 256) break;
      const uint8_t sj = j < ls ? s[j] : (uint8_t)0;
      if (sj == ti && !((used[j >> 5] >> (j & 31)) & 1u)) {
        used[j >> 5] |= 1u << (j & 31);
        m++;
        break;
      }
    }
  }
  const uint32_t to = (ls + h < lt) ? ls + h : lt;
  for (uint32_t i = h; i < to; i++) {
    const uint8_t ti = t[i];
    for (uint32_t j = i - h; j < ls; j++) {
      if (j > 256) break;
      if (s[j] == ti && !((used[j >> 5] >> (j & 31)) & 1u)) {
        used[j >> 5] |= 1u << (j & 31);
        m++;
        break;
      }
    }
  }
  return m;
}

// jaro_m_ref for one pair by a whole warp (every lane calls it with the same
// arguments): lane k holds positions 8k .. 8k + 7 of the shorter string as
// bytes of a 64-bit word, with a byte mask of those in the window and not yet
// matched; a symbol of the longer string takes the lowest candidate position,
// found by one ballot.  Position 256 (used by the reference's second loop
// only) is kept beside it.
// A step is about 30 instructions and one vote; one lane alone searches up to
// 256 bytes per symbol (jaro_m_ref).
__device__ __noinline__ uint32_t jaro_m_warp(const uint8_t* s1, uint32_t l1, const uint8_t* s2,
                                             uint32_t l2) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint8_t* s = s1;
  const uint8_t* t = s2;
  uint32_t ls = l1, lt = l2;
  if (l1 > l2) {
    s = s2;
    t = s1;
    ls = l2;
    lt = l1;
  }
  const uint32_t h = (ls + 1u) / 2u;
  constexpr unsigned long long kHigh = 0x8080808080808080ull;
  // strings are padded to 16 bytes with zeros, which equal no symbol
  const uint2 own = lane * 8u < ls ? *reinterpret_cast<const uint2*>(s + lane * 8u) : make_uint2(0, 0);
  const uint32_t s256 = ls > 256u ? s[256] : 0u;
  unsigned long long avail = kHigh;
  // byte mask of the lane's positions below n
  auto below = [&](uint32_t n) {
    const uint32_t b = lane * 8u;
    if (n >= b + 8u) return kHigh;
    return n <= b ? 0ull : kHigh & ((1ull << (8u * (n - b))) - 1ull);
  };
  auto zero_bytes = [](uint32_t x) {  // 0x80 in every byte of x that is 0
    return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
  };
  auto candidates = [&](uint32_t c) {
    const uint32_t cc = c * 0x01010101u;
    return (unsigned long long)zero_bytes(own.y ^ cc) << 32 | zero_bytes(own.x ^ cc);
  };
  const uint32_t to = min(ls + h, lt);
  uint32_t m = 0;
  bool free256 = true;
  unsigned long long win = below(h + 1u);
  uint32_t w = 0;
  for (uint32_t i = 0; i < to; i++) {
    if ((i & 3u) == 0) w = *reinterpret_cast<const uint32_t*>(t + i);
    const uint32_t c = w & 0xffu;
    w >>= 8;
    if (i == h) win = kHigh;  // second loop: from position i - h on
    const unsigned long long cand = candidates(c) & avail & win;
    const unsigned v = __ballot_sync(kFull, cand != 0ull);
    if (v) {
      m++;
      if (lane == (uint32_t)__ffs(v) - 1u) avail &= ~(cand & (0ull - cand));
    } else if (i >= h && i - h <= 256u && free256 && s256 == c) {
      m++;
      free256 = false;
    }
    // the position that enters (first loop) or leaves (second) for the next symbol
    const uint32_t j = i < h ? i + h + 1u : i - h;
    if ((j >> 3) == lane) {
      const unsigned long long bit = 0x80ull << (8u * (j & 7u));
      win = i < h ? win | bit : win & ~bit;
    }
  }
  return m;
}

// Common prefix of two 16-byte-aligned, zero-padded symbol strings, capped at mn.
__device__ __forceinline__ uint32_t prefix_len(const uint8_t* a, const uint8_t* b, uint32_t mn) {
  const uint4* ap = reinterpret_cast<const uint4*>(a);
  const uint4* bp = reinterpret_cast<const uint4*>(b);
  for (uint32_t k = 0; k < mn; k += 16) {
    const uint4 x = __ldg(ap + (k >> 4));
    const uint4 y = __ldg(bp + (k >> 4));
    const uint32_t d[4] = {x.x ^ y.x, x.y ^ y.y, x.z ^ y.z, x.w ^ y.w};
#pragma unroll
    for (int q = 0; q < 4; q++)
      if (d[q]) return min(mn, k + 4u * q + ((uint32_t)(__ffs(d[q]) - 1) >> 3));
  }
  return mn;
}

// Exact threshold decision with the reference's arithmetic.  Returns pass.
__device__ __noinline__ bool jw_exact(uint32_t m, uint32_t ls, uint32_t ll, uint32_t p, float thr,
                                      unsigned long long* ambiguous) {
  float jf;
  if (ls == 0 || ll == 0) {
    jf = (ls == 0 && ll == 0) ? 1.0f : 0.0f;
  } else if (m == 0) {
    jf = 0.0f;
  } else {
    const float md = (float)m;
    const float q = __fadd_rn(__fdiv_rn(md, (float)ls), __fdiv_rn(md, (float)ll));
    const double t = __dadd_rn((double)q, 1.0);
    jf = __double2float_rn(__ddiv_rn(t, 3.0));
  }
  const double j = (double)jf;
  const double a = __dmul_rn(__dsub_rn(1.0, j), (double)p);
  double jw_fma = __fma_rn(a, 0.1, j);
  double jw_sep = __dadd_rn(j, __dmul_rn(a, 0.1));
  jw_fma = jw_fma > 1.0 ? 1.0 : jw_fma;
  jw_sep = jw_sep > 1.0 ? 1.0 : jw_sep;
  const double t = (double)thr;
  const bool fail_fma = jw_fma < t;
  const bool fail_sep = jw_sep < t;
  if (fail_fma != fail_sep) atomicAdd(ambiguous, 1ull);
  return !fail_fma;
}

// Decision from the match count m and the common prefix p: a float estimate
// settles every pair whose JW lies farther than kDecisionMargin from the
// threshold (the estimate's error is below 2e-6 up to p = 10); the rest take
// the exact path.  The prefix has no cap, so from p = 10 on the sum reaches 1
// and more: cut at 1 like the value it stands for, it is 1 but for the rounding.
__device__ __forceinline__ bool jw_decide(uint32_t m, uint32_t ls, uint32_t ll, uint32_t p,
                                          float thr, unsigned long long* ambiguous) {
  const float fm = (float)m;
  const float ja = m ? (__fdividef(fm, (float)ls) + __fdividef(fm, (float)ll) + 1.0f) * (1.0f / 3.0f)
                     : 0.0f;
  const float jwa = fminf(ja + (1.0f - ja) * (0.1f * (float)p), 1.0f);
  if (jwa >= thr + kDecisionMargin) return true;
  if (jwa < thr - kDecisionMargin) return false;
  return jw_exact(m, ls, ll, p, thr, ambiguous);
}

// Smallest match count that can still reach the threshold, lowered by a
// safety margin: every m below the returned value gives JW < thr exactly.
// JW >= thr needs j >= (thr - c) / (1 - c) with c = 0.1 p, and
// j = (m/ls + m/ll + 1) / 3.  JW grows with m by at least
// 0.1 * (1/ls) / 3 >= 1.3e-4 per match (c <= 0.9, shorter length ls <= 256 on
// the path that uses this), so staying 0.05 matches below the real-valued
// bound keeps a 6.5e-6 gap, far above the float rounding of j (6e-8) and of
// this computation (< 3e-4 matches).  For shorter lengths up to kReachMaxLen
// = 1024 (can_reach) the gap is 0.05 / 3 / 1024 = 1.6e-5 of j, against the same
// 6e-8, and the computation errs by less than 3e-3 matches.  p >= 10 reaches
// 1.0: no bound.  A NaN threshold never fails a pair in the reference, so it
// gives no bound either.
__device__ __forceinline__ int m_need_lo(uint32_t ls, uint32_t ll, uint32_t p, float thr) {
  if (p >= 10u) return 0;
  const float c = 0.1f * (float)p;
  // every quotient here is __fdividef (at most 2 ulp off): the relative error
  // of mr stays below 1e-6, under 3e-4 matches for ls <= 256, far inside the
  // 0.05 margin below
  const float jn = __fdividef(thr - c, 1.0f - c);
  // m = (3 jn - 1) / (1/ls + 1/ll) = (3 jn - 1) ls ll / (ls + ll): one
  // quotient, each factor within an ulp or two, so the bound's error stays
  // far inside the margin below as well
  const float mr = __fdividef((3.0f * jn - 1.0f) * (float)ls * (float)ll, (float)ls + (float)ll);
  const float v = ceilf(mr - 0.05f);
  if (!(v > 0.0f)) return 0;
  return v > 1.0e6f ? 1000000 : (int)v;
}

// Threshold decision on one similarity column of a pair from its match
// count m and common prefix p (la, lb: left and right lengths); an empty
// string takes the reference's rule for empty strings (device_func.cuh:65-69).
__device__ __forceinline__ bool decide(uint32_t m, uint32_t la, uint32_t lb, uint32_t p, float thr,
                                       unsigned long long* ambiguous) {
  if (la == 0 || lb == 0) return jw_exact(0, la, lb, 0, thr, ambiguous);
  return jw_decide(m, min(la, lb), max(la, lb), p, thr, ambiguous);
}

// Members of `live` whose threshold on the group's first column the pair
// reaches.
__device__ __forceinline__ uint32_t first_pass(const Rule* R, uint32_t live, uint32_t m,
                                               uint32_t la, uint32_t lb, uint32_t p,
                                               unsigned long long* ambiguous) {
  uint32_t out = 0;
  for (uint32_t x = live; x; x &= x - 1) {
    const uint32_t k = (uint32_t)__ffs(x) - 1u;
    if (decide(m, la, lb, p, R->mem[k].thr_first, ambiguous)) out |= 1u << k;
  }
  return out;
}

// Does a member of `pass` have no predicate left (the pair matches)?
__device__ __forceinline__ bool member_done(const Rule* R, uint32_t pass) {
  for (uint32_t x = pass; x; x &= x - 1)
    if (R->mem[__ffs(x) - 1].n_rest == 0) return true;
  return false;
}

// Smallest first-column threshold of the live members: the threshold the
// filters and the scan's early stop use.  A NaN threshold never fails a pair
// (the reference compares JW < thr), so it makes the bound NaN: no bound.
__device__ __forceinline__ float live_thr(const Rule* R, uint32_t live) {
  float t = 3.0e38f;
  for (uint32_t x = live; x; x &= x - 1) {
    const float u = R->mem[__ffs(x) - 1].thr_first;
    t = (u != u || t != t) ? __int_as_float(0x7fc00000) : fminf(t, u);
  }
  return t;
}

__device__ __forceinline__ uint32_t find_key(const unsigned long long* item_off, uint32_t domain,
                                             unsigned long long local) {
  uint32_t lo = 0, hi = domain;  // item_off[lo] <= local < item_off[hi]
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (item_off[mid] <= local)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Algorithmic work of one Jaro-Winkler evaluation (one pair, one similarity
// predicate) in 64-bit word operations, the per-unit figure the roofline uses:
// 6 per scanned character per 64-bit word of the shorter string (Peq lookup,
// window AND, ANDNOT matched, lowest-bit isolate x2, OR) over
// to = min(ls + h, ll) characters, the prefix compare in 32-bit steps and 16
// for the count and the formula.  It is counted for every evaluation, also
// for pairs the bound settles without a scan.
__device__ __forceinline__ unsigned long long jw_eval_ops(uint32_t ls, uint32_t ll) {
  const uint32_t h = (ls + 1u) >> 1;
  const uint32_t to = min(ls + h, ll);
  return 6ull * to * ((ls + 63u) >> 6) + 2ull * ((ls + 3u) >> 2) + 16ull;
}

// The same below 2^32 (shorter lengths up to kMaxTableLen: at most 384 * 4 * 6
// + 144).
__device__ __forceinline__ uint32_t jw_eval_ops32(uint32_t ls, uint32_t ll) {
  const uint32_t h = (ls + 1u) >> 1;
  const uint32_t to = min(ls + h, ll);
  return 6u * to * ((ls + 63u) >> 6) + 2u * ((ls + 3u) >> 2) + 16u;
}

// One character step of the bit-parallel match count: x = the unmatched
// positions of the left string equal to `sym` inside the window; the lowest
// one becomes matched; the window [i - h, i + h] moves one position right
// (and only grows while i < h).
template <int W, int S>
__device__ __forceinline__ void bp_step(const uint32_t* __restrict__ tab, uint32_t sym,
                                        uint32_t (&win)[W], uint32_t (&mt)[W], uint32_t grow) {
  uint32_t pe[S];
  load_row<S>(tab + sym * S, pe);
  bp_update<W, S>(pe, win, mt, grow);
}

// May another rule of the launch report the pair too (Rule::dup_slot)?
__device__ __forceinline__ bool shared_pair(const EvalParams& P, const Rule* R, uint32_t lrow,
                                            uint32_t rrow) {
  bool any = R->dup_always != 0;
  for (uint32_t k = 0; k < R->n_dup && !any; k++) {
    const size_t a = R->dup_slot[k][0], b = R->dup_slot[k][1];
    any = P.L.eq_codes[a * P.L.n_rows + lrow] == P.R.eq_codes[a * P.R.n_rows + rrow] &&
          (a == b || P.L.eq_codes[b * P.L.n_rows + lrow] == P.R.eq_codes[b * P.R.n_rows + rrow]);
  }
  return any;
}

// First report of a pair that several rules may report?  With several rules a
// pair can match more than one of them (the reference stops at the first rule
// that passes, global_func.cuh:161-165); a device hash set of emitted (left,
// right) keys keeps exactly one report.  Open addressing with linear probing over
// seen_mask + 1 slots (all ones = empty).  The set is sized for a load of at
// most one half, where probe runs stay far below kMaxProbes; a run past it
// means the set is too small for this run's distinct pairs: seen_overflow is
// set, the host repeats the run with a set sized from the pass count
// (Counters::passes, an upper bound on the distinct pairs of the set).  Reports whose
// probe run reaches kCheckProbe look at the overflow flag first and give up
// once it is set, so an overflowing run costs a few probes per report; runs
// of a set sized as intended rarely get that far and never read the flag.
constexpr unsigned long long kMaxProbes = 4096;
constexpr unsigned long long kCheckProbe = 8;
__device__ __forceinline__ bool first_report(const EvalParams& P, uint32_t lrow, uint32_t rrow) {
  const unsigned long long key = ((unsigned long long)lrow << 32) | rrow;
  unsigned long long h = key * 0x9E3779B97F4A7C15ull;
  h ^= h >> 29;
  for (unsigned long long probe = 0; probe <= P.seen_mask && probe < kMaxProbes; probe++) {
    if (probe == kCheckProbe && *(volatile unsigned long long*)&P.ctr->seen_overflow) return false;
    const unsigned long long slot = (h + probe) & P.seen_mask;
    const unsigned long long prev = atomicCAS(P.seen + slot, ~0ull, key);
    if (prev == ~0ull) return true;
    if (prev == key) return false;
  }
  atomicAdd(&P.ctr->seen_overflow, 1ull);
  return false;
}

// Writes up to one match per lane to the output with one atomic per warp,
// the matches that another rule may report too after the duplicate set.  Most
// matches of rules with different equalities are no other rule's candidates:
// two loads each instead of a probe of a set larger than L2, which also had to
// be cleared and, in a first run, grown (8 rules in two groups, 150k x 150k
// rows, 7.9M matches: a run's reset and join 118 against 158 us; 30k x 30k
// rows, the first run of a session 0.96 against 3.8 ms).
__device__ __forceinline__ void flush_pairs(const EvalParams& P, bool pass, uint32_t lrow,
                                            uint32_t rrow, uint32_t rule, int lane) {
  if (P.seen) {
    const bool shared = pass && shared_pair(P, P.rules + rule, lrow, rrow);
    const unsigned cm = __ballot_sync(kFull, shared);
    if (cm) {
      if (lane == 0) atomicAdd(&P.ctr->passes, (unsigned long long)__popc(cm));
      if (shared) pass = first_report(P, lrow, rrow);
    }
  }
  const unsigned pm = __ballot_sync(kFull, pass);
  if (!pm) return;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(&P.ctr->out_count, (unsigned long long)__popc(pm));
  base = __shfl_sync(kFull, base, 0);
  if (pass) {
    const unsigned long long pos = base + __popc(pm & ((1u << lane) - 1u));
    if (pos < P.capacity) {
      P.out_l[pos] = lrow;
      P.out_r[pos] = rrow;
    }
  }
}

// Twice an upper bound on the Jaro matches of two strings of lengths la and lb
// from their count signatures (dev::StrMeta): the lengths less the sum of the
// counts' differences, one vabsdiff4 per word (four minima per word, summed,
// take five times as many instructions: 123 against 42 issue slots for a
// bound and its operands in a loop).
__device__ __forceinline__ int sig_bound2(uint32_t la, uint32_t lb, const uint4& a0,
                                          const uint4& a1, const uint4& b0, const uint4& b1) {
  uint32_t d = 0;
  auto add = [&d](uint32_t a, uint32_t b) {
    asm("vabsdiff4.u32.u32.u32.add %0, %1, %2, %0;" : "+r"(d) : "r"(a), "r"(b));
  };
  add(a0.x, b0.x);
  add(a0.y, b0.y);
  add(a0.z, b0.z);
  add(a0.w, b0.w);
  add(a1.x, b1.x);
  add(a1.y, b1.y);
  add(a1.z, b1.z);
  add(a1.w, b1.w);
  return (int)(la + lb - d);
}

// Common prefix of two 16-symbol little-endian heads; 16 when they agree.
__device__ __forceinline__ uint32_t prefix16(const uint4& a, const uint4& b) {
  const uint32_t d0 = a.x ^ b.x, d1 = a.y ^ b.y, d2 = a.z ^ b.z, d3 = a.w ^ b.w;
  const uint32_t d = d0 ? d0 : d1 ? d1 : d2 ? d2 : d3;  // the first word that differs
  const uint32_t k = d0 ? 0u : d1 ? 4u : d2 ? 8u : 12u;
  return k + ((uint32_t)__clz((int)__brev(d)) >> 3);  // 12 + 32 / 8 when none does
}

// Can a pair of non-empty strings whose left one has no Peq table reach thr?
// The filters of the scanned pairs, in front of the reference's own loops:
// the loops match each position of either string at most once, so lengths
// and count signatures bound their count too.  false = JW < thr for certain.
// Longer strings than kReachMaxLen and prefixes of 16 and more are not
// decided here.
constexpr uint32_t kReachMaxLen = 1024;
__device__ __forceinline__ bool can_reach(const StrMeta* am, const uint4& b_head, const uint4& b_s0,
                                          const uint4& b_s1, uint32_t la, uint32_t lb, float thr) {
  const uint32_t ls = min(la, lb), ll = max(la, lb);
  if (ls > kReachMaxLen) return true;
  const uint32_t p16 = prefix16(am->head, b_head);
  if (p16 == 16u && ls > 16u) return true;
  const int need = m_need_lo(ls, ll, min(p16, ls), thr);
  if (need > (int)ls) return false;
  return need <= 0 || sig_bound2(la, lb, am->sig[0], am->sig[1], b_s0, b_s1) >= 2 * need;
}

// Slow exact similarity check of one pair (any lengths).  Out of line and
// with plain pointer/scalar arguments only: passing the kernel parameters by
// reference would copy them into local memory for the whole kernel.
__device__ __noinline__ bool sim_pass_slow(const StrMeta* am, const StrMeta* bm, const uint8_t* a,
                                           const uint8_t* b, float thr, Counters* ctr) {
  const uint32_t la = am->loc.y, lb = bm->loc.y;
  if (la == 0 || lb == 0) return jw_exact(0, la, lb, 0, thr, &ctr->ambiguous);
  const uint32_t mn = min(la, lb);
  if (mn > 256) atomicAdd(&ctr->long_pairs, 1ull);
  if (!can_reach(am, bm->head, bm->sig[0], bm->sig[1], la, lb, thr)) return false;
  const uint32_t m = jaro_m_ref(a, la, b, lb);
  const uint32_t p = prefix_len(a, b, mn);
  return jw_exact(m, mn, max(la, lb), p, thr, &ctr->ambiguous);
}

// The same for a pair inside the evaluation loop: one lane's loops over two
// long strings hold up its warp for half a millisecond, so a pair that can
// reach the threshold is left to k_eval_long where the launch has room for it.
// 0 = fails, 1 = passes, 2 + k = the caller puts it on the list at k (< cap).
__device__ __noinline__ uint32_t sim_slow_or_defer(const StrMeta* am, const StrMeta* bm,
                                                   const uint8_t* a, const uint8_t* b, float thr,
                                                   Counters* ctr, uint32_t cap) {
  const uint32_t la = am->loc.y, lb = bm->loc.y;
  if (cap && la && lb && can_reach(am, bm->head, bm->sig[0], bm->sig[1], la, lb, thr)) {
    const unsigned long long at = atomicAdd(&ctr->deferred, 1ull);
    if (at < cap) return 2u + (uint32_t)at;
  }
  return sim_pass_slow(am, bm, a, b, thr, ctr) ? 1u : 0u;
}

// Per-lane work counts of the evaluation loop, summed into Counters at exit:
// algorithmic JW word operations (every evaluation, scanned or not), pairs
// that reached a bit-parallel scan, and scan steps (4 symbols each).
struct WorkTally {
  unsigned long long ops;
  uint32_t scans, steps;
  uint32_t wsteps;  // warp-level scan steps (counted by lane 0)
  uint32_t rest;    // scans of predicates after the first (advance_rule / advance_group)
};

// Does the left string of length la have a Peq table (PeqShape)?
__device__ __forceinline__ bool has_table(const EvalParams& P, uint32_t la) {
  return la > 0u && la <= P.fast_max;
}

__device__ __forceinline__ const uint32_t* peq_table(const EvalParams& P, uint32_t slot,
                                                     uint32_t lrow) {
  return P.peq + ((size_t)slot * P.L.n_rows + lrow) * P.tab_words;
}

// Ring of pairs waiting for a scan, kRingEntries entries of three 16-byte
// records per warp:
//   {right row, right offset / 16, right length, tag}
//   {first 16 symbols of the right string}
//   {left row, left length | Peq slot << 9 | rule << 16, left offset / 16,
//   threshold bits} for a plain entry (its left string has a Peq table:
//   length <= 256; slot 127 = read it from the rule; plans hold at most 64
//   rules), with the threshold its need was computed for; {left row, left
//   length, left offset / 16, rule} for a kAdvance entry.
// tag = need | p << 10 | s << 15 | kAdvance? | live << 19 | member << 27.
// A plain entry waits for the scan of its group's first column: `live` holds
// the members whose extra equalities hold, need the matches the smallest of
// their thresholds needs and p the common prefix (or kPrefixUnknown).  A
// kAdvance entry passed the first column (live = the members that passed):
// the lane that takes it goes on with predicate s of member `member`.
constexpr uint32_t kRing = kRingEntries;
constexpr uint32_t kPrefixUnknown = 31u;  // common prefix longer than 16: measured at the scan
constexpr uint32_t kAdvance = 1u << 18;

__device__ __forceinline__ uint32_t ring_tag(uint32_t need, uint32_t p, uint32_t s, uint32_t live,
                                             uint32_t member) {
  return need | (p << 10) | (s << 15) | (live << 19) | (member << 27);
}
__device__ __forceinline__ uint32_t tag_live(uint32_t t) { return (t >> 19) & 0xffu; }
__device__ __forceinline__ uint32_t tag_member(uint32_t t) { return (t >> 27) & 7u; }
__device__ __forceinline__ uint32_t tag_s(uint32_t t) { return (t >> 15) & 7u; }

// Bit-parallel scan state of one lane: the pair's Peq table and right
// string, the symbols in hand (cur) and the next 16 (nxt), the window and
// matched masks, lengths, position, common prefix, the mismatches it can
// still afford and the threshold.
template <int W>
struct Scan {
  const uint32_t* tab;
  const uint8_t* b;
  uint4 cur, nxt;
  uint32_t win[W], mt[W];
  uint32_t ls, ll, i, n_iter, h, p;
  int allowed;
  float thr;
};

// Starts the scan of a pair (la, lb: lengths; p: common prefix or
// kPrefixUnknown; need: matches the threshold needs).  false = decided
// (fails) without a scan.
template <int W>
__device__ __forceinline__ bool scan_begin(Scan<W>& z, const uint32_t* tab, const uint8_t* a,
                                           const uint8_t* b, const uint4& head_b, uint32_t la,
                                           uint32_t lb, uint32_t p, int need, float thr,
                                           WorkTally* ops) {
  z.ls = min(la, lb);
  z.ll = max(la, lb);
  z.h = (z.ls + 1u) >> 1;
  z.n_iter = min(lb, la + z.h);
  if (p == kPrefixUnknown) {
    p = prefix_len(a, b, z.ls);
    need = m_need_lo(z.ls, z.ll, p, thr);
  }
  if (need > (int)min(z.n_iter, z.ls)) return false;
  z.p = p;
  z.thr = thr;
  z.allowed = (int)z.n_iter - need;
  z.i = 0;
  z.tab = tab;
  z.b = b;
  z.cur = head_b;
  if (z.n_iter > 16u) z.nxt = __ldg(reinterpret_cast<const uint4*>(b + 16));
#pragma unroll
  for (int k = 0; k < W; k++) {
    const int nb = (int)z.h + 1 - 32 * k;
    z.win[k] = nb >= 32 ? 0xffffffffu : (nb <= 0 ? 0u : ((1u << nb) - 1u));
    z.mt[k] = 0u;
  }
  ops->scans++;
  return true;
}

// One scan step of 16 symbols, the chunk in hand (the next chunk was asked
// for one step earlier); after each, the pair stops once even matching every
// remaining symbol stays below its bound.  Returns 0 (not decided yet), 1
// (the scan is complete: *m = the match count) or 2 (the pair cannot reach
// the scan's threshold).
constexpr int kScanQuadUnroll = 1;
// A loop turn scans until fewer than this many lanes are still scanning, then
// decides the finished pairs and hands out the next ones: deciding and
// picking up cost as much as two to three scan steps, whether one lane or all
// take part.  8 rules, 150k x 150k rows, evaluation: 13.97 ms with one step
// per turn, 12.18, 11.75, 11.74, 11.59, 11.34 ms with 24, 20, 16, 12, 8 lanes.
constexpr uint32_t kTurnLanes = 8;
template <int W>
__device__ __forceinline__ int scan_step(Scan<W>& z, uint32_t* m_out, WorkTally* ops) {
  constexpr int S = row_words(W);
  if (z.i) {
    // chunk i/16 arrived one chunk ago; ask for the one after it
    z.cur = z.nxt;
    if (z.i + 16u < z.n_iter) z.nxt = __ldg(reinterpret_cast<const uint4*>(z.b + z.i + 16u));
  }
  // four symbols per 32-bit word of the chunk, one word per loop turn: the
  // smaller loop body runs faster than the fully unrolled chunk (C3, 300k
  // rows: 98.5 ms of evaluation against 102.4 ms with two words per turn and
  // 113 ms with four), which stalled on instruction fetch
  uint4 c4 = z.cur;
#pragma unroll(kScanQuadUnroll)
  for (uint32_t q = 0; q < 4; q++) {
    const uint32_t wd = c4.x;
#pragma unroll
    for (int c = 0; c < 4; c++)
      bp_step<W, S>(z.tab, (wd >> (8 * c)) & 0xffu, z.win, z.mt,
                    (z.i + 4u * q + (uint32_t)c) < z.h ? 1u : 0u);
    c4 = make_uint4(c4.y, c4.z, c4.w, 0u);
  }
  z.i += 16;
  ops->steps += 4;
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < W; k++) m += __popc(z.mt[k]);
  *m_out = m;
  if (z.i >= z.n_iter) return 1;
  if ((int)(z.i - m) > z.allowed) return 2;  // even matching every remaining symbol stays below
  return 0;
}

// The similarity predicates after predicate s of a pair that passed it, in
// order, until one needs a scan (returns 2, the scan state set up and s its
// index), one fails (0) or all pass (1).  Each predicate first goes through
// the filters of the first one: length bound, common prefix, count
// signatures.  (A launch without rule groups: every rule evaluated alone.)
template <int W>
__device__ __forceinline__ int advance_rule(const EvalParams& P, uint32_t rule, uint32_t* s,
                                            uint32_t lrow, uint32_t rrow, Scan<W>& z,
                                            WorkTally* ops) {
  const Rule* R = P.rules + rule;
  const uint32_t n_sim = R->n_sim;
  for (uint32_t k = *s + 1; k < n_sim; k++) {
    *s = k;
    const uint32_t sl = R->sim_l[k], sr = R->sim_r[k];
    const float thr = R->thr[k];
    const StrMeta* am = P.L.str_meta + (size_t)sl * P.L.n_rows + lrow;
    const StrMeta* bm = P.R.str_meta + (size_t)sr * P.R.n_rows + rrow;
    const uint4 al = am->loc, bl = bm->loc;
    const uint32_t la = al.y, lb = bl.y;
    const uint8_t* a = P.L.arena + 16ull * al.x;
    const uint8_t* b = P.R.arena + 16ull * bl.x;
    if (la == 0 || lb == 0) {
      if (!jw_exact(0, la, lb, 0, thr, &P.ctr->ambiguous)) return 0;
      continue;
    }
    if constexpr (W == kMaxTableLen / 32) {  // narrower masks: every string has a table
      if (!has_table(P, la)) {
        const uint32_t st = sim_slow_or_defer(am, bm, a, b, thr, P.ctr, P.defer_cap);
        if (st >= 2u) {
          P.defer[st - 2u] = make_uint4(lrow, rrow, rule, 1u);
          return 0;
        }
        ops->ops += jw_eval_ops(min(la, lb), max(la, lb));
        if (!st) return 0;
        continue;
      }
    }
    const uint32_t ls = min(la, lb), ll = max(la, lb);
    ops->ops += jw_eval_ops(ls, ll);
    const uint4 bh = bm->head;
    const uint32_t p16 = prefix16(am->head, bh);
    uint32_t p = kPrefixUnknown;
    int need = 0;
    if (!(p16 == 16u && ls > 16u)) {
      p = min(p16, ls);
      need = m_need_lo(ls, ll, p, thr);
      const uint32_t n_iter = min(lb, la + ((ls + 1u) >> 1));
      if (need > (int)min(n_iter, ls)) return 0;
      if (need > 0 &&
          sig_bound2(la, lb, am->sig[0], am->sig[1], bm->sig[0], bm->sig[1]) < 2 * need)
        return 0;
    }
    ops->rest++;
    return scan_begin<W>(z, peq_table(P, sl, lrow), a, b, bh, la, lb, p, need, thr, ops) ? 2 : 0;
  }
  return 1;
}

// The similarity predicates after the group's first column, for the live
// members of a pair's group in member order, from predicate *s of member
// *mi: until one needs a scan (returns 2, the scan state set up for (*mi,
// *s)), a member passes all of its predicates (1: the pair matches) or no
// member is left (0).  A member drops out at its first failing predicate.
// Each predicate first goes through the filters of the first column: length
// bound, common prefix, count signatures.
//
// A member that needs a scan of a column scans it at the smallest threshold
// among itself and the live members after it that test the same column, so
// that one scan serves them all: *memo then names the column (left slot <<
// 16 | right slot) and memo_m holds its match count (the scan state z still
// holds the pair's lengths and prefix) or kMemoBelow (the scan stopped below
// that smallest threshold, so every one of those members fails the column).
// Each member decides at its own threshold.  Starting a scan ends the memo.
constexpr uint32_t kNoMemo = 0xffffffffu;
constexpr uint32_t kMemoBelow = 0xffffffffu;

// Smallest threshold on column (sl, sr) of member mi (threshold thr) and of
// the live members after it that test that column; NaN (no bound) when one
// of them has a NaN threshold.
__device__ __forceinline__ float shared_thr(const Rule* R, uint32_t live, uint32_t mi, uint32_t sl,
                                            uint32_t sr, float thr) {
  float t = thr;
  for (uint32_t x = live & ~((2u << mi) - 1u); x; x &= x - 1) {
    const Member* M = R->mem + (__ffs(x) - 1);
    for (uint32_t j = 0; j < M->n_rest; j++)
      if (M->rest_l[j] == sl && M->rest_r[j] == sr) {
        const float u = M->rest_thr[j];
        t = (u != u || t != t) ? __int_as_float(0x7fc00000) : fminf(t, u);
        break;
      }
  }
  return t;
}

template <int W>
__device__ __forceinline__ int advance_group(const EvalParams& P, uint32_t rule, uint32_t* live,
                                             uint32_t* mi, uint32_t* s, uint32_t lrow,
                                             uint32_t rrow, Scan<W>& z, uint32_t* memo,
                                             uint32_t memo_m, WorkTally* ops) {
  const Rule* R = P.rules + rule;
  while (*live) {
    const Member* M = R->mem + *mi;
    const uint32_t n_rest = M->n_rest;
    uint32_t k = *s;
    for (; k < n_rest; k++) {
      const uint32_t sl = M->rest_l[k], sr = M->rest_r[k];
      const float thr = M->rest_thr[k];
      if (*memo == (sl << 16 | sr)) {
        if (memo_m == kMemoBelow || !jw_decide(memo_m, z.ls, z.ll, z.p, thr, &P.ctr->ambiguous))
          break;
        continue;
      }
      const StrMeta* am = P.L.str_meta + (size_t)sl * P.L.n_rows + lrow;
      const StrMeta* bm = P.R.str_meta + (size_t)sr * P.R.n_rows + rrow;
      const uint4 al = am->loc, bl = bm->loc;
      const uint32_t la = al.y, lb = bl.y;
      const uint8_t* a = P.L.arena + 16ull * al.x;
      const uint8_t* b = P.R.arena + 16ull * bl.x;
      if (la == 0 || lb == 0) {
        if (!jw_exact(0, la, lb, 0, thr, &P.ctr->ambiguous)) break;
        continue;
      }
      if constexpr (W == kMaxTableLen / 32) {  // narrower masks: every string has a table
        if (!has_table(P, la)) {
          const uint32_t st = sim_slow_or_defer(am, bm, a, b, thr, P.ctr, P.defer_cap);
          if (st >= 2u) {  // with the members still live
            P.defer[st - 2u] = make_uint4(lrow, rrow, rule, *live);
            return 0;
          }
          ops->ops += jw_eval_ops(min(la, lb), max(la, lb));
          if (!st) break;
          continue;
        }
      }
      const uint32_t ls = min(la, lb), ll = max(la, lb);
      ops->ops += jw_eval_ops(ls, ll);
      const uint4 bh = bm->head;
      const uint32_t p16 = prefix16(am->head, bh);
      uint32_t p = kPrefixUnknown;
      int need = 0;
      if (!(p16 == 16u && ls > 16u)) {
        p = min(p16, ls);
        need = m_need_lo(ls, ll, p, thr);
        const uint32_t n_iter = min(lb, la + ((ls + 1u) >> 1));
        if (need > (int)min(n_iter, ls)) break;
        if (need > 0 &&
            sig_bound2(la, lb, am->sig[0], am->sig[1], bm->sig[0], bm->sig[1]) < 2 * need)
          break;
      }
      // member *mi may pass: one scan for it and the later members testing
      // this column, at the smallest of their thresholds
      const float ts = shared_thr(R, *live, *mi, sl, sr, thr);
      if (p != kPrefixUnknown && ts != thr) need = m_need_lo(ls, ll, p, ts);
      *memo = kNoMemo;  // z is about to hold another pair's scan
      ops->rest++;
      if (scan_begin<W>(z, peq_table(P, sl, lrow), a, b, bh, la, lb, p, need, ts, ops)) {
        *s = k;
        return 2;
      }
      break;
    }
    if (k >= n_rest) return 1;
    *live &= ~(1u << *mi);  // member *mi failed predicate k
    if (!*live) return 0;
    *mi = (uint32_t)__ffs(*live) - 1u;
    *s = 0;
  }
  return 0;
}

// Warp-uniform state of the evaluation loop kept in shared memory (every
// lane reads it; every lane writes the same values, after a __syncwarp when
// the values were read in the same step): the work items the warp has
// claimed, the claim in each staging buffer, and the item being filtered.
constexpr uint32_t kMaxClaimChunk = 16;
// Kind of a claimed item: its rule has similarity predicates, and some
// member of its group has extra equality slots; bits 8-11 hold the group's
// member count.
constexpr uint32_t kItemSim = 1u, kItemExtras = 2u, kItemMore = 4u;  // more: n_sim > 1
constexpr uint32_t kItemLast = 8u;  // of a staged piece: the item's last one
__device__ __forceinline__ uint32_t item_members(uint32_t kind) { return (kind >> 8) & 15u; }
// A claimed work item: the sources of its bulk copies (right-row metadata
// from the block's first row, right rows from the 16-byte boundary at or
// before it, the left string's metadata), left row, rule, rows, the first
// row's position in sorted_r modulo 8 (modulo 4: past the boundary; meta_turn
// needs the rest), its kind and the group's smallest first-column threshold.
struct ItemDesc {
  const StrMeta* meta_src;
  const uint32_t* rows_src;
  const StrMeta* lm_src;
  uint32_t lrow, rule, n, pos, kind, slot;
  float thr0;
  int32_t lcode[2];  // the left row's codes of the group's first two extra slots
};
constexpr uint32_t kOutBuf = 64;  // matches a warp holds before writing them out
struct OutBuf {  // matches not yet written out (emit): fewer than 32 between calls
  uint2 pair[kOutBuf];
  uint32_t rule[kOutBuf];
  uint32_t n;
};
struct WarpCtl {
  ItemDesc desc[kMaxClaimChunk];  // claimed items not yet staged
  uint32_t c_rule[kMaxStageBufs], c_lrow[kMaxStageBufs];  // claim per staging buffer
  uint32_t c_n[kMaxStageBufs], c_pos[kMaxStageBufs];      // (n = 0: none)
  uint32_t c_kind[kMaxStageBufs], c_slot[kMaxStageBufs];
  float c_thr[kMaxStageBufs];
  int32_t c_lcode[kMaxStageBufs][2];
  // the item being filtered; i_lcode: its left row's codes of the group's
  // extra equality slots
  uint32_t i_rule, i_lrow, i_kind, i_all, i_slot;  // i_slot: its first column's left slot
  float i_thr;
  int32_t i_lcode[kMaxEq];
  uint32_t i_live[4];  // its group's Rule::x_live, x_thr (groups with extra slots)
  float i_xthr[4];
  OutBuf out;
};
static_assert(sizeof(WarpCtl) <= kWarpCtlWords * 4, "warp control block outgrows its words");

// Collects the warp's final matches of one step; every 32 of them go out
// together (flush_pairs), so the duplicate-set probes and the output
// reservation pay their round trips once per 32 matches instead of once per
// step with a match.
__device__ __forceinline__ void emit(const EvalParams& P, OutBuf* O, bool pass, uint32_t lrow,
                                     uint32_t rrow, uint32_t rule, int lane) {
  const unsigned pm = __ballot_sync(kFull, pass);
  if (!pm) return;
  const uint32_t n0 = O->n;
  if (pass) {
    const uint32_t at = n0 + __popc(pm & ((1u << lane) - 1u));
    O->pair[at] = make_uint2(lrow, rrow);
    O->rule[at] = rule;
  }
  const uint32_t n = n0 + __popc(pm);
  __syncwarp();
  if (n < 32) {
    if (lane == 0) O->n = n;
    __syncwarp();
    return;
  }
  const uint2 e = O->pair[lane];
  const uint32_t er = O->rule[lane];
  const bool more = (uint32_t)lane + 32u < n;
  const uint2 t = more ? O->pair[32 + lane] : make_uint2(0u, 0u);
  const uint32_t tr = more ? O->rule[32 + lane] : 0u;
  __syncwarp();
  if (more) {
    O->pair[lane] = t;
    O->rule[lane] = tr;
  }
  if (lane == 0) O->n = n - 32u;
  __syncwarp();
  flush_pairs(P, true, e.x, e.y, er, lane);
}

// Writes out the matches emit still holds (at the end of the warp's loop).
__device__ __forceinline__ void emit_drain(const EvalParams& P, OutBuf* O, int lane) {
  const uint32_t n = O->n;
  const bool have = (uint32_t)lane < n;
  const uint2 e = have ? O->pair[lane] : make_uint2(0u, 0u);
  const uint32_t er = have ? O->rule[lane] : 0u;
  __syncwarp();
  if (lane == 0) O->n = 0;
  __syncwarp();
  flush_pairs(P, have, e.x, e.y, er, lane);
}

// Filter one batch of 32 right rows of the item against its group's first
// similarity column: first the members whose extra equalities hold for the
// pair (live), then one staged metadata record per right row gives its
// length and first 16 symbols, hence the common prefix p (when below 16) and
// the match count the smallest live threshold needs, and its count
// signature, an upper bound on the matches; pairs that cannot reach it are
// decided here, the rest go to the ring with their first 16 symbols.  Pairs
// decided without a scan that pass go to the ring for their members' further
// predicates, or match at once when a passing member has none.  lm: the
// item's left string metadata; pos0: the item's first position in sorted_r
// modulo 8.  Returns the entries appended.
// G: the launch has rule groups; without, every rule is its own group of one
// and its predicates take the plain path (one threshold per predicate).
//
// A chain of shared-memory loads and arithmetic, every candidate pair once:
// issue slots and shared-memory wavefronts bound it.  With the bound from
// differences (sig_bound2), the records turned (meta_turn) and the group's
// table in shared memory a batch takes 1,620 cycles of its warp against
// 2,150 (8 rules, 150k x 150k rows; evaluation 9.90 against 11.34 ms) and
// 1,130 against 1,690 without groups (2,601 x 64,264 rows; 145 against
// 179 us).
template <bool G>
__device__ __forceinline__ uint32_t filter_batch(const EvalParams& P, WarpCtl* C,
                                                 const StrMeta* lm, const uint32_t* rows,
                                                 const StrMeta* meta, uint32_t pos0, uint32_t n,
                                                 uint32_t e0, uint4* q, uint32_t tail,
                                                 WorkTally* ops) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const uint32_t e = e0 + (uint32_t)lane;
  const bool act = e < n;
  const uint32_t rrow = act ? rows[e] : 0u;
  const uint32_t la = lm->loc.y, a_off = lm->loc.x;
  const uint32_t all = C->i_all;
  uint32_t live = act ? all : 0u;
  float thr = C->i_thr;
  const uint4* rec = reinterpret_cast<const uint4*>(meta + e);
  const uint32_t turn = meta_turn(pos0 + e);
  uint4 loc = make_uint4(0, 0, 0, 0), head = make_uint4(0, 0, 0, 0);
  if (act) loc = rec[turn];
  if (G && act && (C->i_kind & kItemExtras)) {
    // the right row's codes of the extra slots: the first two staged with
    // its metadata (store_meta), the others from device memory
    uint32_t eqm = 0;
    const uint32_t nx = (C->i_kind >> 12) & 15u;
    if ((int32_t)loc.z == C->i_lcode[0]) eqm |= 1u;
    if (nx > 1 && (int32_t)loc.w == C->i_lcode[1]) eqm |= 2u;
    if (nx <= 2u) {  // the group's table (Rule::x_live, x_thr)
      live = C->i_live[eqm];
      if (live != all) thr = C->i_xthr[eqm];
    } else {
      const Rule* R = P.rules + C->i_rule;
      for (uint32_t j = 2; j < nx; j++)
        if (P.R.eq_codes[(size_t)R->xslot[j] * P.R.n_rows + rrow] == C->i_lcode[j]) eqm |= 1u << j;
      for (uint32_t x = all; x; x &= x - 1) {
        const uint32_t k = (uint32_t)__ffs(x) - 1u;
        if (R->mem[k].xmask & ~eqm) live &= ~(1u << k);
      }
      if (live != all) thr = live_thr(R, live);
    }
  }
  uint32_t pass1 = 0;  // members that passed the first column without a scan
  bool scan = false;
  uint32_t p = 0;
  int need = 0;
  if (live) {
    head = rec[1u ^ turn];
    const uint32_t lb = loc.y;
    if (la == 0 || lb == 0) {
      if constexpr (G)
        pass1 = first_pass(P.rules + C->i_rule, live, 0, la, lb, 0, &P.ctr->ambiguous);
      else
        pass1 = jw_exact(0, la, lb, 0, thr, &P.ctr->ambiguous) ? 1u : 0u;
    } else {
      const uint32_t ls = min(la, lb), ll = max(la, lb);
      ops->ops += jw_eval_ops32(ls, ll);
      const uint32_t p16 = prefix16(lm->head, head);
      if (p16 == 16u && ls > 16u) {
        scan = true;  // prefix longer than 16: measured exactly before the scan
        p = kPrefixUnknown;
      } else {
        // out of reach when the need is above the shorter length, or above
        // what the count signatures leave
        p = min(p16, ls);
        need = m_need_lo(ls, ll, p, thr);
        scan = need <= (int)ls &&
               sig_bound2(la, lb, lm->sig[0], lm->sig[1], rec[2u ^ turn], rec[3u ^ turn]) >= 2 * need;
      }
    }
  }
  bool done;
  if constexpr (G)
    done = pass1 && member_done(P.rules + C->i_rule, pass1);
  else
    done = pass1 && !(C->i_kind & kItemMore);
  const bool push = scan || (pass1 && !done);
  const unsigned qm = __ballot_sync(kFull, push);
  const uint32_t lrow = C->i_lrow;
  if (push) {
    const uint32_t slot = (tail + __popc(qm & lt)) & (kRing - 1);
    uint4* en = q + kRingWords / 4 * slot;
    const uint32_t tag = scan ? ring_tag((uint32_t)need, p, 0, live, 0)
                              : (ring_tag(0, 0, 0, pass1, (uint32_t)__ffs(pass1) - 1u) | kAdvance);
    en[0] = make_uint4(rrow, loc.x, loc.y, tag);
    en[1] = head;
    en[2] = scan ? make_uint4(lrow, la | (min(C->i_slot, 127u) << 9) | (C->i_rule << 16), a_off,
                              __float_as_uint(thr))
                 : make_uint4(lrow, la, a_off, C->i_rule);
  }
  emit(P, &C->out, done, lrow, rrow, C->i_rule, lane);
  return __popc(qm);
}

// Maps a position of the launch's work list to a global work item: the list
// is the concatenation of the segments [seg_begin[k], seg_end[k]).
__device__ __forceinline__ unsigned long long seg_item(const EvalParams& P, unsigned long long v) {
  for (uint32_t k = 0; k < P.n_seg; k++) {
    const unsigned long long len = P.seg_end[k] - P.seg_begin[k];
    if (v < len) return P.seg_begin[k] + v;
    v -= len;
  }
  return ~0ull;
}

// ---- bulk copies (TMA) into shared memory, completed on an mbarrier --------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .b64 st;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes)
      : "memory");
}

// Global -> shared bulk copy: both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity, at most kMaxWaitSpins tries
// (each try suspends the thread for a while).  false = gave up.
constexpr uint32_t kMaxWaitSpins = 1u << 22;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t k = 0; k < kMaxWaitSpins; k++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}


// Key of the item at position `local` of a rule's item space, searched in
// [lo, hi): item_off[lo] <= local < item_off[hi].
__device__ __forceinline__ uint32_t find_key_in(const unsigned long long* item_off, uint32_t lo,
                                                uint32_t hi, unsigned long long local) {
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (__ldg(item_off + mid) <= local)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// The left row and the rows [rb0, rb1) of sorted_r of item `local` of a rule's
// item space, under left key jl with join key `key`.
__device__ __forceinline__ void item_rows(const EvalParams& P, const Rule& R, uint32_t jl,
                                          uint32_t key, unsigned long long local, uint32_t* lrow,
                                          uint32_t* rb0, uint32_t* rb1) {
  const unsigned long long in_key = local - R.item_off[jl];
  const uint32_t nl = R.cnt_l[jl];
  const uint32_t ri = (uint32_t)(in_key / nl);
  const uint32_t li = (uint32_t)(in_key - (unsigned long long)ri * nl);
  *lrow = R.sorted_l[R.off_l[jl] + li];
  const uint32_t offr = R.off_r[key];
  *rb0 = offr + ri * P.tile_right;
  *rb1 = min(*rb0 + P.tile_right, offr + R.cnt_r[key]);
}

// Claims up to `chunk` consecutive work positions with one atomic and
// computes their item descriptors into C->desc, one lane per item, so the
// dependent loads of every item (rule fields included) overlap.  Within one rule, the first and
// last lanes find their keys over the whole key space and the others search
// only between those two.  Returns the count (0: the work list is exhausted).
__device__ __forceinline__ uint32_t claim_chunk(const EvalParams& P, WarpCtl* C,
                                                unsigned long long n_work, uint32_t chunk) {
  const int lane = threadIdx.x & 31;
  unsigned long long v0 = 0;
  if (lane == 0) v0 = atomicAdd(&P.ctr->work_next, (unsigned long long)chunk);
  v0 = __shfl_sync(kFull, v0, 0);
  if (v0 >= n_work) return 0;
  const uint32_t n = (uint32_t)min((unsigned long long)chunk, n_work - v0);
  const uint32_t k = min((uint32_t)lane, n - 1);  // lanes past n repeat the last item
  const unsigned long long v = v0 + k;
  const unsigned long long it = P.n_seg ? seg_item(P, v) : v;
  uint32_t r = 0;
  while (r + 1 < P.n_rules && P.rule_item_base[r + 1] <= it) r++;
  const Rule& R = P.rules[r];
  const unsigned long long local = it - P.rule_item_base[r];
  const uint32_t r_first = __shfl_sync(kFull, r, 0), r_last = __shfl_sync(kFull, r, n - 1);
  uint32_t jl;  // left key (items of class 0 only: the join key)
  if (r_first == r_last) {
    uint32_t kb = 0;
    if (k == 0 || k == n - 1) kb = find_key(R.item_off, R.domain, local);
    const uint32_t k0 = __shfl_sync(kFull, kb, 0), k1 = __shfl_sync(kFull, kb, n - 1);
    jl = find_key_in(R.item_off, k0, k1 + 1, local);
  } else {
    jl = find_key(R.item_off, R.domain, local);
  }
  uint32_t lrow, rb0, rb1;
  item_rows(P, R, jl, jl, local, &lrow, &rb0, &rb1);
  const uint32_t a0 = rb0 & ~3u;
  ItemDesc d;
  const bool sim = R.n_sim != 0;
  d.kind = (sim ? kItemSim : 0u) | (R.n_xslots ? kItemExtras : 0u) |
           (R.n_sim > 1 ? kItemMore : 0u) | (R.n_members << 8) | (R.n_xslots << 12);
  // loaded here, a claim ahead of the item's filtering
  d.lcode[0] = R.n_xslots > 0 ? P.L.eq_codes[(size_t)R.xslot[0] * P.L.n_rows + lrow] : 0;
  d.lcode[1] = R.n_xslots > 1 ? P.L.eq_codes[(size_t)R.xslot[1] * P.L.n_rows + lrow] : 0;
  d.meta_src = sim ? R.sorted_meta_r + rb0 : nullptr;
  d.rows_src = R.sorted_r + a0;
  d.lm_src = sim ? P.L.str_meta + (size_t)R.sim_l[0] * P.L.n_rows + lrow : nullptr;
  d.lrow = lrow;
  d.rule = r;
  d.n = rb1 - rb0;
  d.pos = rb0 & 7u;
  d.slot = sim ? R.sim_l[0] : 0u;
  d.thr0 = sim ? R.thr_min : 0.0f;
  __syncwarp();  // earlier reads of the descriptors are done
  if ((uint32_t)lane < n) C->desc[lane] = d;
  __syncwarp();
  return n;
}

// Claims the next work item whose rule has similarity predicates and starts
// the bulk copies of its right rows, their metadata and its left string's
// metadata into staging buffer b (completing on bar).  Items of rules with
// equalities only are emitted on the spot.  Items come from the warp's
// claimed descriptors C->desc[*d_pos, *d_n), refilled by claim_chunk.  Once
// the work list is exhausted or the cycle budget has run out, *stop is set
// and this and every later claim leave c_n[b] = 0.
__device__ __forceinline__ void claim_item(const EvalParams& P, WarpCtl* C, uint32_t b,
                                           uint32_t* buf, uint64_t* bar, unsigned long long n_work,
                                           uint32_t chunk, long long t_start, bool* stop,
                                           uint32_t* d_pos, uint32_t* d_n, uint32_t* d_off,
                                           unsigned long long* done) {
  const int lane = threadIdx.x & 31;
  while (!*stop) {
    if (*d_pos >= *d_n) {
      *d_n = claim_chunk(P, C, n_work, chunk);
      *d_pos = 0;
      if (*d_n == 0) {
        *stop = true;
        break;
      }
    }
    if (P.watchdog_cycles && (unsigned long long)(clock64() - t_start) > P.watchdog_cycles) {
      if (lane == 0) atomicAdd(&P.ctr->watchdog_trips, 1ull);
      *stop = true;
      break;
    }
    ItemDesc d = C->desc[*d_pos];
    if (!(d.kind & kItemSim)) {  // equalities only: every candidate matches
      for (uint32_t e = 0; e < d.n; e += 32) {
        const uint32_t k = e + (uint32_t)lane;
        const uint32_t rrow = k < d.n ? d.rows_src[(d.pos & 3u) + k] : 0u;
        emit(P, &C->out, k < d.n, d.lrow, rrow, d.rule, lane);
      }
      (*done)++;
      (*d_pos)++;
      continue;
    }
    // the next piece of the item that a buffer holds
    const uint32_t off = *d_off, left = d.n - off;
    d.n = min(left, P.stage_rows);
    if (left > P.stage_rows) {
      *d_off = off + d.n;
    } else {
      *d_off = 0;
      (*d_pos)++;
      d.kind |= kItemLast;
    }
    d.meta_src += off;
    d.rows_src += off;
    if (lane == 0) {
      const uint32_t mbytes = d.n * (uint32_t)sizeof(StrMeta);
      const uint32_t rbytes = ((d.n + (d.pos & 3u)) * 4u + 15u) & ~15u;
      // earlier reads of this buffer are done (__syncwarp before the claim);
      // order them before the asynchronous writes
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(bar, mbytes + rbytes + (uint32_t)sizeof(StrMeta));
      bulk_g2s(buf, d.meta_src, mbytes, bar);
      bulk_g2s(buf + P.buf_rows_off, d.rows_src, rbytes, bar);
      bulk_g2s(buf + P.buf_lmeta_off, d.lm_src, (uint32_t)sizeof(StrMeta), bar);
    }
    C->c_rule[b] = d.rule;
    C->c_lrow[b] = d.lrow;
    C->c_n[b] = d.n;
    C->c_pos[b] = d.pos;
    C->c_kind[b] = d.kind;
    C->c_slot[b] = d.slot;
    C->c_thr[b] = d.thr0;
    C->c_lcode[b][0] = d.lcode[0];
    C->c_lcode[b][1] = d.lcode[1];
    return;
  }
  C->c_n[b] = 0;
}

// The evaluation loop of one warp, for scans over W-word masks.  Work items
// (one left row x up to tile_right right rows of one candidate block) are
// claimed one ahead, so the bulk copies of the next item run while the
// current one is filtered.  Filtered pairs queue in the warp's ring; lanes
// take the next queued pair as soon as theirs is decided, whichever item it
// came from, since every pair reads its left string's Peq table from device
// memory; the ring is refilled from the current item, then the next ones, as
// it drains.  A pair that passes its group's first column goes on with the
// further predicates of the members that passed, member by member, in the
// same lane; matches leave by warp-aggregated atomics.
template <int W, bool G>
__device__ __forceinline__ void eval_loop(const EvalParams& P, uint32_t* region,
                                          unsigned long long n_work, WorkTally* ops,
                                          unsigned long long* done) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint4* q = reinterpret_cast<uint4*>(region);
  WarpCtl* C = reinterpret_cast<WarpCtl*>(region + P.ctl_off);
  uint64_t* bar0 = reinterpret_cast<uint64_t*>(region + P.mbar_off);
  const long long t_start = clock64();
  if (lane == 0) C->out.n = 0;
  __syncwarp();
  // work positions per claim: every warp gets about eight claims, at most
  // kMaxClaimChunk items each
  const unsigned long long n_warps = (unsigned long long)gridDim.x * kWarpsPerCta;
  const uint32_t chunk =
      (uint32_t)max(1ull, min((unsigned long long)kMaxClaimChunk, n_work / (n_warps * 8ull)));
  bool stop = false;
  // the warp's claimed descriptors not yet taken, and the rows of the first one
  // already staged
  uint32_t d_pos = 0, d_n = 0, d_off = 0;
  for (uint32_t b = 0; b < P.n_bufs; b++)
    claim_item(P, C, b, region + P.buf_off + b * P.buf_words, bar0 + b, n_work, chunk, t_start,
               &stop, &d_pos, &d_n, &d_off, done);
  uint32_t cb = 0;      // buffer of the current item (buffer cb + k holds the k-th next)
  uint32_t phs = 0;     // bit b: mbarrier phase of buffer b
  bool active = false;  // current item waited for and being filtered
  uint32_t in_pos = 0, cur_n = C->c_n[0];
  uint32_t head = 0, tail = 0;
  // lane state: the pair, its group's live members, the member and predicate
  // in hand (first = the group's first column)
  bool busy = false, first = false;
  uint32_t rrow = 0, lrow = 0, rule = 0, s = 0, live = 0, mi = 0;
  uint32_t memo = kNoMemo, memo_m = 0;  // the last finished column scan (advance_group)
  Scan<W> z;
  z.tab = nullptr;
  z.b = nullptr;
  z.cur = z.nxt = make_uint4(0, 0, 0, 0);
  z.ls = z.ll = z.i = z.n_iter = z.h = z.p = 0;
  z.allowed = 0;
  z.thr = 0.0f;
#pragma unroll
  for (int k = 0; k < W; k++) z.win[k] = z.mt[k] = 0u;

  for (;;) {
    const unsigned idle = __ballot_sync(kFull, !busy);
    const uint32_t n_idle = __popc(idle);
    // refill the ring until it holds a pair for every idle lane
    while (tail - head < n_idle && tail - head <= kRing - 32) {
      uint32_t* buf = region + P.buf_off + cb * P.buf_words;
      if (active) {
        if (in_pos < cur_n) {
          tail += filter_batch<G>(P, C, reinterpret_cast<const StrMeta*>(buf + P.buf_lmeta_off),
                                  buf + P.buf_rows_off + (C->c_pos[cb] & 3u),
                                  reinterpret_cast<const StrMeta*>(buf), C->c_pos[cb], cur_n,
                                  in_pos, q, tail, ops);
          in_pos += 32;
          continue;
        }
        // the item is filtered: its buffer takes the item after the next one
        active = false;
        __syncwarp();
        claim_item(P, C, cb, buf, bar0 + cb, n_work, chunk, t_start, &stop, &d_pos, &d_n, &d_off, done);
        cb = cb + 1u == P.n_bufs ? 0u : cb + 1u;
        buf = region + P.buf_off + cb * P.buf_words;
        cur_n = C->c_n[cb];
      }
      if (cur_n == 0) break;  // no work left (claims run in order)
      const bool ok = mbar_wait(bar0 + cb, (phs >> cb) & 1u);
      phs ^= 1u << cb;
      if (!__all_sync(kFull, ok)) {
        // a copy never completed: report, wait once more (bounded) for it
        // and for the other buffers' copies, stop
        if (lane == 0) atomicAdd(&P.ctr->watchdog_trips, 1ull);
        mbar_wait(bar0 + cb, ((phs >> cb) & 1u) ^ 1u);
        for (uint32_t b = 0; b < P.n_bufs; b++)
          if (b != cb && C->c_n[b]) mbar_wait(bar0 + b, (phs >> b) & 1u);
        emit_drain(P, &C->out, lane);
        return;
      }
      active = true;
      in_pos = 0;
      const uint32_t ir = C->c_rule[cb], il = C->c_lrow[cb], kind = C->c_kind[cb];
      if (kind & kItemLast) (*done)++;
      const float thr = C->c_thr[cb];
      __syncwarp();  // the previous item's fields are read
      C->i_rule = ir;
      C->i_lrow = il;
      C->i_thr = thr;
      C->i_kind = kind;
      C->i_all = (1u << item_members(kind)) - 1u;
      C->i_slot = C->c_slot[cb];
      if (G && (kind & kItemExtras)) {  // the left row's codes of the extra equality slots
        const uint32_t nx = (kind >> 12) & 15u;
        if (lane >= 28) {
          C->i_live[lane - 28] = P.rules[ir].x_live[lane - 28];
          C->i_xthr[lane - 28] = P.rules[ir].x_thr[lane - 28];
        } else if (lane < 2) {
          C->i_lcode[lane] = C->c_lcode[cb][lane];  // loaded with the claim
        } else if ((uint32_t)lane < nx) {
          const Rule* R = P.rules + ir;
          C->i_lcode[lane] = P.L.eq_codes[(size_t)R->xslot[lane] * P.L.n_rows + il];
        }
      }
      __syncwarp();
    }
    // idle lanes take the next queued pairs
    bool fin = false, pass = false;
    const uint32_t avail = tail - head;
    const uint32_t rank = __popc(idle & lt);
    if (!busy && rank < avail) {
      const uint4* en = q + kRingWords / 4 * ((head + rank) & (kRing - 1));
      const uint4 e0 = en[0], e2 = en[2];
      rrow = e0.x;
      lrow = e2.x;
      live = tag_live(e0.w);
      memo = kNoMemo;
      int st = 0;
      if (e0.w & kAdvance) {
        rule = e2.w;
        first = false;
        mi = tag_member(e0.w);
        s = tag_s(e0.w);
        if constexpr (G)
          st = advance_group<W>(P, rule, &live, &mi, &s, lrow, rrow, z, &memo, memo_m, ops);
        else
          st = advance_rule<W>(P, rule, &s, lrow, rrow, z, ops);
      } else {
        // the group's first column at the smallest live threshold (without
        // groups: the rule's first predicate), as the filter computed it
        rule = e2.y >> 16;
        first = true;
        s = 0;
        uint32_t sl0 = (e2.y >> 9) & 127u;  // 127: the slot did not fit, read it from the rule
        if (sl0 == 127u) sl0 = P.rules[rule].sim_l[0];
        const uint32_t p = (e0.w >> 10) & 31u;
        st = scan_begin<W>(z, peq_table(P, sl0, lrow), P.L.arena + 16ull * e2.z,
                           P.R.arena + 16ull * e0.y, en[1], e2.y & 511u, e0.z, p,
                           (int)(e0.w & 1023u), __uint_as_float(e2.w), ops)
                 ? 2
                 : 0;
      }
      if (st == 2) {
        busy = true;
      } else {
        fin = true;
        pass = st == 1;
      }
    }
    head += min(n_idle, avail);
    // scan steps until fewer than kTurnLanes lanes are left scanning (or, when
    // fewer had a pair, one of them is decided): every lane votes
    uint32_t m = 0;
    int sc = 0;
    {
      uint32_t on = __popc(__ballot_sync(kFull, busy));
      const uint32_t few = min(on, kTurnLanes);
      while (on && on >= few) {
        if (lane == 0) ops->wsteps++;
        if (busy && !sc) sc = scan_step<W>(z, &m, ops);
        on = __popc(__ballot_sync(kFull, busy && !sc));
      }
    }
    if (busy) {
      if (sc) {
        busy = false;
        int st = 0;
        if constexpr (!G) {
          // one rule: the scanned predicate s decides, then its next ones
          if (sc == 1 && jw_decide(m, z.ls, z.ll, z.p, z.thr, &P.ctr->ambiguous))
            st = advance_rule<W>(P, rule, &s, lrow, rrow, z, ops);
        } else if (first) {
          // decided per live member; the scan stopped early only when even
          // the smallest threshold is out of reach
          const Rule* R = P.rules + rule;
          const uint32_t pass1 =
              sc == 1 ? first_pass(R, live, m, z.ls, z.ll, z.p, &P.ctr->ambiguous) : 0u;
          if (pass1 && member_done(R, pass1)) {
            st = 1;
          } else if (pass1) {
            first = false;
            live = pass1;
            mi = (uint32_t)__ffs(pass1) - 1u;
            s = 0;
            memo = kNoMemo;
            st = advance_group<W>(P, rule, &live, &mi, &s, lrow, rrow, z, &memo, memo_m, ops);
          }
        } else {
          // the scan ran at the smallest threshold of the members testing
          // this column (advance_group): remembered for them, and member mi
          // decides at its own threshold
          const Member* M = P.rules[rule].mem + mi;
          memo = M->rest_l[s] << 16 | M->rest_r[s];
          memo_m = sc == 1 ? m : kMemoBelow;
          if (sc == 1 && jw_decide(m, z.ls, z.ll, z.p, M->rest_thr[s], &P.ctr->ambiguous)) {
            s++;  // member mi passed predicate s
          } else {
            live &= ~(1u << mi);
            mi = live ? (uint32_t)__ffs(live) - 1u : 0u;
            s = 0;
          }
          if (live)
            st = advance_group<W>(P, rule, &live, &mi, &s, lrow, rrow, z, &memo, memo_m, ops);
        }
        if (st == 2) {
          busy = true;
        } else {
          fin = true;
          pass = st == 1;
        }
      }
    }
    emit(P, &C->out, fin && pass, lrow, rrow, rule, lane);
    if (!__any_sync(kFull, busy) && head == tail && !active && cur_n == 0) break;
  }
  emit_drain(P, &C->out, lane);
}

// The evaluation kernel body for masks of W words, instantiated below with
// two register budgets (k_eval / k_eval_wide) and for rule groups.  One
// kernel per mask width: a kernel holding every width's scan loop is
// register-allocated for the widest and spills in the narrow ones too.
template <int W, bool G>
__device__ __forceinline__ void eval_body(const EvalParams& P) {
  extern __shared__ __align__(16) uint32_t smem[];
  pdl_wait();  // nothing to wait for: launched in stream order, after the join
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  uint32_t* region = smem + (size_t)warp * P.warp_words;
  if (lane == 0) {
    uint64_t* bar = reinterpret_cast<uint64_t*>(region + P.mbar_off);
    for (uint32_t b = 0; b < P.n_bufs; b++) mbar_init(bar + b);
  }
  __syncwarp();
  unsigned long long n_work = 0;  // length of this launch's work list
  if (P.n_seg == 0) {
    n_work = P.rule_item_base[P.n_rules];
  } else {
    for (uint32_t k = 0; k < P.n_seg; k++) n_work += P.seg_end[k] - P.seg_begin[k];
  }
  unsigned long long done = 0;
  WorkTally tally{0ull, 0u, 0u, 0u, 0u};
  eval_loop<W, G>(P, region, n_work, &tally, &done);
  if (lane == 0 && done) atomicAdd(&P.ctr->items_done, done);
  unsigned long long ops = tally.ops, scans = tally.scans, steps = tally.steps, rest = tally.rest;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ops += __shfl_down_sync(kFull, ops, o);
    scans += __shfl_down_sync(kFull, scans, o);
    steps += __shfl_down_sync(kFull, steps, o);
    rest += __shfl_down_sync(kFull, rest, o);
  }
  if (lane == 0) {
    if (ops) atomicAdd(&P.ctr->jw_word_ops, ops);
    if (scans) atomicAdd(&P.ctr->scans, scans);
    if (steps) atomicAdd(&P.ctr->scan_steps, steps);
    if (rest) atomicAdd(&P.ctr->rest_scans, rest);
    if (tally.wsteps) atomicAdd(&P.ctr->scan_warp_steps, (unsigned long long)tally.wsteps);
  }
}

// One pair, by the whole warp (arguments the same in every lane): does a
// member of `pass`, the members whose threshold on the group's first column
// the pair reaches, pass all its other predicates?
__device__ __noinline__ bool long_pair_rest(const EvalParams& P, const Rule* R, uint32_t pass,
                                            uint32_t lrow, uint32_t rrow) {
  const int lane = threadIdx.x & 31;
  uint32_t memo = 0xffffffffu, m = 0, p = 0;  // the last column counted (advance_group)
  for (uint32_t x = pass; x; x &= x - 1) {
    const Member* M = R->mem + (__ffs(x) - 1);
    uint32_t k = 0;
    for (; k < M->n_rest; k++) {
      const uint32_t sl = M->rest_l[k], sr = M->rest_r[k];
      const float thr = M->rest_thr[k];
      const StrMeta* am = P.L.str_meta + (size_t)sl * P.L.n_rows + lrow;
      const StrMeta* bm = P.R.str_meta + (size_t)sr * P.R.n_rows + rrow;
      const uint4 al = am->loc, bl = bm->loc;
      const uint32_t la = al.y, lb = bl.y, mn = min(la, lb), mx = max(la, lb);
      if (mn && memo != (sl << 16 | sr)) {
        if (lane == 0) {
          atomicAdd(&P.ctr->jw_word_ops, jw_eval_ops(mn, mx));
          if (mn > kMaxTableLen) atomicAdd(&P.ctr->long_pairs, 1ull);
        }
        if (!can_reach(am, bm->head, bm->sig[0], bm->sig[1], la, lb, thr)) break;
        const uint8_t* a = P.L.arena + 16ull * al.x;
        const uint8_t* b = P.R.arena + 16ull * bl.x;
        m = jaro_m_warp(a, la, b, lb);
        p = prefix_len(a, b, mn);
        memo = sl << 16 | sr;
      }
      bool ok = false;
      if (lane == 0) ok = mn ? jw_exact(m, mn, mx, p, thr, &P.ctr->ambiguous)
                             : jw_exact(0, la, lb, 0, thr, &P.ctr->ambiguous);
      if (!__shfl_sync(kFull, ok ? 1 : 0, 0)) break;
    }
    if (k == M->n_rest) return true;
  }
  return false;
}

// Work items whose left string has no Peq table (longer than kMaxTableLen).
// A warp takes one item at a time from the class-1 item space and goes over
// its right rows 32 at a time: a lane per row tests the extra equalities and
// the filters of the scanned pairs (can_reach), and the few pairs left are
// counted one after the other by the whole warp (jaro_m_warp).  As items
// of the evaluation kernels -- a lane per pair, every pair through the
// reference's loops -- they were most of the time: 40,014 x 60,000 rows of
// 64-256 characters, 2 % of the authors over 256 symbols, evaluation 37.5 ms
// against 2.51 ms; and the evaluation kernels without that path need fewer
// registers (8 rules, 150k x 150k rows: 14.06 against 13.91 ms).  Pairs that
// meet such a string at a later predicate (EvalParams::defer) follow: left to
// their lanes they kept a few warps busy for 1.2 ms after all others (2.29
// against 1.03 ms).
__global__ void __launch_bounds__(kWarpsPerCta * 32, 4) k_eval_long(
    const __grid_constant__ EvalParams P) {
  __shared__ OutBuf s_out[kWarpsPerCta];
  const int lane = threadIdx.x & 31;
  OutBuf* O = s_out + (threadIdx.x >> 5);
  if (lane == 0) O->n = 0;
  __syncwarp();
  const unsigned long long n_work = !(P.long_what & 1u) ? 0ull
                                    : P.n_seg ? P.seg_end[0] - P.seg_begin[0]
                                              : P.rule_item_base[P.n_rules];
  const long long t_start = clock64();
  unsigned long long done = 0, word_ops = 0;
  for (;;) {
    unsigned long long v = 0;
    if (lane == 0) v = atomicAdd(&P.ctr->work_next_long, 1ull);
    v = __shfl_sync(kFull, v, 0);
    if (v >= n_work) break;
    if (P.watchdog_cycles && (unsigned long long)(clock64() - t_start) > P.watchdog_cycles) {
      if (lane == 0) atomicAdd(&P.ctr->watchdog_trips, 1ull);
      break;
    }
    const unsigned long long it = P.n_seg ? P.seg_begin[0] + v : v;
    uint32_t r = 0;
    while (r + 1 < P.n_rules && P.rule_item_base[r + 1] <= it) r++;
    const Rule* R = P.rules + r;
    const unsigned long long local = it - P.rule_item_base[r] + R->item_off[R->domain];
    const uint32_t jl =
        R->domain + find_key(R->item_off + R->domain, R->domain_l - R->domain, local);
    uint32_t lrow, rb0, rb1;
    item_rows(P, *R, jl, join_key(*R, jl), local, &lrow, &rb0, &rb1);
    const StrMeta* lm = P.L.str_meta + (size_t)R->sim_l[0] * P.L.n_rows + lrow;
    const uint32_t la = lm->loc.y;
    const uint8_t* a = P.L.arena + 16ull * lm->loc.x;
    const uint32_t all = (1u << R->n_members) - 1u, nx = R->n_xslots;
    for (uint32_t e0 = rb0; e0 < rb1; e0 += 32) {
      const uint32_t e = e0 + (uint32_t)lane;
      const bool act = e < rb1;
      const uint32_t rrow = act ? R->sorted_r[e] : 0u;
      const uint32_t at = act ? e : e0, turn = meta_turn(at);
      const uint4* rm = reinterpret_cast<const uint4*>(R->sorted_meta_r + at);
      const uint4 loc = rm[turn];
      const uint32_t lb = loc.y;
      uint32_t live = act ? all : 0u, pass1 = 0;
      if (act && nx) {  // members whose extra equalities hold
        uint32_t eqm = 0;
        for (uint32_t j = 0; j < nx; j++) {
          const size_t xs = R->xslot[j];
          if (P.R.eq_codes[xs * P.R.n_rows + rrow] == P.L.eq_codes[xs * P.L.n_rows + lrow])
            eqm |= 1u << j;
        }
        for (uint32_t x = all; x; x &= x - 1) {
          const uint32_t k = (uint32_t)__ffs(x) - 1u;
          if (R->mem[k].xmask & ~eqm) live &= ~(1u << k);
        }
      }
      bool count = false;
      if (live) {
        if (lb == 0) {
          pass1 = first_pass(R, live, 0, la, 0, 0, &P.ctr->ambiguous);
        } else {
          word_ops += jw_eval_ops(min(la, lb), max(la, lb));
          if (lb > kMaxTableLen) atomicAdd(&P.ctr->long_pairs, 1ull);
          count = can_reach(lm, rm[1u ^ turn], rm[2u ^ turn], rm[3u ^ turn], la, lb,
                            live_thr(R, live));
        }
      }
      for (unsigned x = __ballot_sync(kFull, count); x; x &= x - 1) {
        const int src = __ffs(x) - 1;
        const uint8_t* b = P.R.arena + 16ull * __shfl_sync(kFull, loc.x, src);
        const uint32_t m = jaro_m_warp(a, la, b, __shfl_sync(kFull, lb, src));
        if (lane == src)
          pass1 = first_pass(R, live, m, la, lb, prefix_len(a, b, min(la, lb)), &P.ctr->ambiguous);
        __syncwarp();
      }
      bool match = pass1 && member_done(R, pass1);
      for (unsigned x = __ballot_sync(kFull, pass1 && !match); x; x &= x - 1) {
        const int src = __ffs(x) - 1;
        const bool ok = long_pair_rest(P, R, __shfl_sync(kFull, pass1, src), lrow,
                                       __shfl_sync(kFull, rrow, src));
        if (lane == src) match = ok;
      }
      emit(P, O, match, lrow, rrow, r, lane);
    }
    done++;
  }
  // the deferred pairs, one at a time by a warp
  const unsigned long long n_def =
      P.long_what & 2u ? min(P.ctr->deferred, (unsigned long long)P.defer_cap) : 0ull;
  for (;;) {
    unsigned long long v = n_def;
    if (lane == 0 && n_def) v = atomicAdd(&P.ctr->deferred_next, 1ull);
    v = __shfl_sync(kFull, v, 0);
    if (v >= n_def) break;
    if (P.watchdog_cycles && (unsigned long long)(clock64() - t_start) > P.watchdog_cycles) {
      if (lane == 0) atomicAdd(&P.ctr->watchdog_trips, 1ull);
      break;
    }
    const uint4 e = P.defer[v];
    const bool ok = long_pair_rest(P, P.rules + e.z, e.w, e.x, e.y);
    emit(P, O, ok && lane == 0, e.x, e.y, e.z, lane);
  }
  emit_drain(P, O, lane);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) word_ops += __shfl_xor_sync(kFull, word_ops, o);
  if (lane == 0 && done) atomicAdd(&P.ctr->items_done, done);
  if (lane == 0 && word_ops) atomicAdd(&P.ctr->jw_word_ops, word_ops);
}

__global__ void k_count_firsts(const unsigned long long* seen, uint64_t n_seen, Counters* ctr) {
  uint32_t k = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n_seen;
       i += (uint64_t)gridDim.x * blockDim.x)
    k += seen[i] != ~0ull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(kFull, k, o);
  if ((threadIdx.x & 31) == 0 && k) atomicAdd(&ctr->firsts, (unsigned long long)k);
}

// What the host reads after an evaluation, written to its page-locked memory
// by one launch; few pairs need no copy of their own then, nor the host a
// second wait.  Bound by the latency of one pass of stores over the link: a
// serving request of 16 records takes 174 us, with copies of the counters and
// then of the pairs 257 us; hbx_block of 2,077 pairs 388 against 417 us.
__global__ void k_report(const unsigned long long* words, uint32_t n_words, const Counters* ctr,
                         const uint32_t* l, const uint32_t* r, unsigned long long capacity,
                         unsigned long long limit, unsigned long long* h_words, uint32_t* h_out) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
  for (uint32_t i = t; i < n_words; i += step) h_words[i] = words[i];
  const unsigned long long n = ctr->out_count;
  if (n > limit || n > capacity) return;
  for (uint32_t i = t; i < (uint32_t)n; i += step) {
    h_out[i] = l[i];
    h_out[n + i] = r[i];
  }
}

// A few thousand strings, once per pair of tables and plan: latency, a few
// microseconds.  (The host's bit-parallel count of the same pairs takes 1.2 ms
// per pair of columns, mostly cache misses: CSV files to pair file, 8 rules, 25k
// x 40k rows, 8.7 against 12.8 ms; streamed windows of 40k x 60k long rows
// 30.4 against 35.9 ms.)
__global__ void k_sample(const __grid_constant__ SampleCols cols, const uint8_t* arena_l,
                         const uint8_t* arena_r, const uint2* rows, uint32_t n, uint4* out) {
  const uint32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= n) return;  // whole warps
  const uint2 at = rows[k];
  const uint4 al = cols.l[blockIdx.y][at.x].loc, bl = cols.r[blockIdx.y][at.y].loc;
  const uint8_t* a = arena_l + 16ull * al.x;
  const uint8_t* b = arena_r + 16ull * bl.x;
  const uint32_t la = al.y, lb = bl.y, mn = min(la, lb);
  uint32_t m = 0, p = 0;
  if (mn > kMaxTableLen) {
    m = 0xffffffffu;
  } else if (mn) {
    m = jaro_m_warp(a, la, b, lb);
    p = prefix_len(a, b, mn);
  }
  if ((threadIdx.x & 31) == 0) out[(size_t)blockIdx.y * n + k] = make_uint4(la, lb, m, p);
}

// Peq tables (PeqShape): one warp per (slot, row); the table is cleared,
// then every symbol's mask per 32-symbol word is built with __match_any_sync
// (lanes holding the same symbol agree on it; the lowest of them stores it).
__global__ void k_peq_build(Side L, uint32_t n_slots, PeqShape shape, uint32_t* peq) {
  const int lane = threadIdx.x & 31;
  const unsigned long long n_tasks = (unsigned long long)n_slots * L.n_rows;
  const unsigned long long n_warps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
  for (unsigned long long t = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
       t < n_tasks; t += n_warps) {
    const uint4 loc = L.str_meta[t].loc;  // slot-major: t = slot * n_rows + row
    const uint32_t la = loc.y;
    if (la == 0 || la > shape.fast_max) continue;
    uint32_t* tab = peq + t * shape.tab_words;
    uint4* t4 = reinterpret_cast<uint4*>(tab);
    for (uint32_t w = (uint32_t)lane; w < shape.tab_words / 4; w += 32)
      t4[w] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    const uint8_t* a = L.arena + 16ull * loc.x;
    const uint32_t nw = (la + 31u) >> 5;
    for (uint32_t k = 0; k < nw; k++) {
      const uint32_t j = k * 32u + (uint32_t)lane;
      const uint32_t sym = j < la ? (uint32_t)a[j] : 0xffffffffu;
      const unsigned mm = __match_any_sync(kFull, sym);
      if (j < la && lane == __ffs(mm) - 1) tab[sym * shape.s + k] = mm;
    }
    __syncwarp();
  }
}

// Dense variant: 3 CTAs (24 warps) per SM, at most 85 registers per thread.
template <int W>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 3) k_eval(EvalParams P) {
  eval_body<W, false>(P);
}

// Wide variant: 2 CTAs (16 warps) per SM, up to 128 registers per thread, so
// the longer-string scan variants keep their state in registers.
template <int W>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 2) k_eval_wide(EvalParams P) {
  eval_body<W, false>(P);
}

// The same two over rule groups (Rule: "Group evaluation").
template <int W>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 3) k_eval_groups(EvalParams P) {
  eval_body<W, true>(P);
}
template <int W>
__global__ void __launch_bounds__(kWarpsPerCta * 32, 2) k_eval_groups_wide(EvalParams P) {
  eval_body<W, true>(P);
}

namespace {
template <int W>
EvalKernel pick(int wide, bool groups) {
  return groups ? (wide ? k_eval_groups_wide<W> : k_eval_groups<W>)
                : (wide ? k_eval_wide<W> : k_eval<W>);
}
}  // namespace

EvalKernel eval_kernel(int wide, bool groups, uint32_t peq_w) {
  switch (peq_w) {
    case 1: return pick<1>(wide, groups);
    case 2: return pick<2>(wide, groups);
    case 3: return pick<3>(wide, groups);
    case 4: return pick<4>(wide, groups);
    default: return pick<8>(wide, groups);
  }
}

}  // namespace dev
}  // namespace hbx
