// sort.cu -- (left row, right row) pairs sorted on the device, for output in
// row order: a least-significant-digit radix sort of keys left << b | right
// (b bits hold a right row), 8 bits per pass.
//
// One launch counts every pass's digits.  A pass is then one launch: a block
// ranks a tile of keys, publishes its counts per digit, adds the counts
// of the tiles before it (looking back tile by tile, as far as the first that
// has published its sum) and scatters: the published one-sweep radix sort
// (Adinets and Merrill) with decoupled look-back (Merrill and Garland).  The
// first pass reads the pairs and the last one writes them back, so that no
// launch only converts.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "context.h"
#include "device_buffers.h"
#include "hbx_core.h"
#include "ingest.h"

namespace hbx {
namespace srt {

constexpr uint32_t kThreads = 256, kWarps = kThreads / 32;
constexpr uint32_t kMaxPasses = 8;
constexpr uint32_t kBack = 8;  // tiles read at once when looking back
constexpr unsigned kFull = 0xffffffffu;

struct Pairs {
  uint32_t *l, *r;
  uint64_t n;
  uint32_t bits_r;
  __device__ unsigned long long key(uint64_t i) const {
    return (unsigned long long)l[i] << bits_r | r[i];
  }
};

// count[pass * 256 + digit] over all keys.
__global__ void __launch_bounds__(kThreads) k_digits(Pairs p, uint32_t n_passes, uint32_t* count) {
  __shared__ uint32_t h[kMaxPasses * 256];
  for (uint32_t k = threadIdx.x; k < n_passes * 256; k += kThreads) h[k] = 0;
  __syncthreads();
  for (uint64_t i = blockIdx.x * (uint64_t)kThreads + threadIdx.x; i < p.n;
       i += (uint64_t)gridDim.x * kThreads) {
    const unsigned long long v = p.key(i);
    for (uint32_t q = 0; q < n_passes; q++)
      atomicAdd(&h[q * 256 + ((uint32_t)(v >> (8 * q)) & 0xffu)], 1u);
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < n_passes * 256; k += kThreads)
    if (h[k]) atomicAdd(&count[k], h[k]);
}

// A tile's word per digit: the keys of the tile (kCount) or of it and all
// tiles before it (kSum) with that digit, the state in the two highest bits.
template <class T>
struct State {
  static constexpr int kShift = 8 * sizeof(T) - 2;
  static constexpr T kCount = (T)1 << kShift, kSum = (T)2 << kShift, kValue = kCount - 1;
};

// One pass.  What bounds it at 10^5 pairs is latency: a launch, the ranks (a
// warp ranks 8 rounds of its own 256 keys without a block barrier), the look
// back (8 tiles at a time: their words arrive together).  100,000 pairs take
// 8.7 us a pass and 43 us a sort; a histogram, a scan and a scatter launch per
// pass took 24 us, and 126 us a sort with the packing launches.  Above what
// four blocks per SM hold, a thread takes 16 keys instead of 8: half as many
// tiles look back over half as many (24.5 million pairs: 255 us a pass and
// 1.12 ms a sort, 300 us and 1.30 ms with 8 keys, 282 us and 1.27 ms with
// three launches a pass).
// Tiles are handed out by a ticket, so the tiles before a block's own are
// running or done; a wait for their counts ends after max_polls polls
// (dev::scan_polls), and the block counts the keys before its tile itself.
// next: the other pass's words, cleared for it.
template <class T, uint32_t kKeys>
__global__ void __launch_bounds__(kThreads) k_pass(Pairs p, const unsigned long long* src,
                                                   unsigned long long* dst, uint32_t shift,
                                                   const uint32_t* count, uint32_t* ticket, T* state,
                                                   T* next, uint32_t max_polls) {
  using S = State<T>;
  constexpr uint32_t kTile = kThreads * kKeys;
  __shared__ uint32_t s_cnt[kWarps][256];  // a warp's keys per digit, then where they start
  __shared__ uint32_t s_base[256];         // the tile's first position per digit
  __shared__ uint32_t s_warp[kWarps];
  __shared__ uint32_t s_tile;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  if (t == 0) s_tile = atomicAdd(ticket, 1u);
  for (uint32_t k = lane; k < 256; k += 32) s_cnt[warp][k] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = (uint64_t)tile * kTile + warp * (32 * kKeys) + lane;
  unsigned long long v[kKeys];
  uint32_t rank[kKeys];
#pragma unroll
  for (uint32_t k = 0; k < kKeys; k++) {
    const uint64_t i = base + 32 * k;
    v[k] = i >= p.n ? 0ull : src ? src[i] : p.key(i);
  }
#pragma unroll
  for (uint32_t k = 0; k < kKeys; k++) {
    const bool act = base + 32 * k < p.n;
    const uint32_t d = act ? (uint32_t)(v[k] >> shift) & 0xffu : 256u + lane;  // inactive: unique
    const unsigned peers = __match_any_sync(kFull, d);
    const uint32_t before = (uint32_t)__popc(peers & ((1u << lane) - 1u));
    const uint32_t had = act ? s_cnt[warp][d] : 0u;
    __syncwarp();
    if (act && before == 0) s_cnt[warp][d] = had + (uint32_t)__popc(peers);
    __syncwarp();
    rank[k] = had + before;
  }
  __syncthreads();
  // thread t: digit t
  uint32_t mine = 0;
#pragma unroll
  for (uint32_t w = 0; w < kWarps; w++) {
    const uint32_t c = s_cnt[w][t];
    s_cnt[w][t] = mine;
    mine += c;
  }
  volatile T* words = state;
  const uint64_t at = (uint64_t)tile * 256 + t;
  words[at] = (T)mine | (tile ? S::kCount : S::kSum);
  next[at] = 0;
  // where the digit starts: all keys with smaller digits
  const uint32_t all = count[t];
  uint32_t inc = all;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, inc, o);
    if ((int)lane >= o) inc += y;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t first = inc - all;
  for (uint32_t w = 0; w < warp; w++) first += s_warp[w];
  // the tiles before this one
  T sum = 0;
  int64_t j = (int64_t)tile - 1;
  uint32_t polls = 0;
  bool done = tile == 0;
  while (!done && polls < max_polls) {
    T w[kBack];
#pragma unroll
    for (uint32_t u = 0; u < kBack; u++)
      w[u] = j >= (int64_t)u ? (T)words[(uint64_t)(j - u) * 256 + t] : S::kSum;
    uint32_t got = 0;
#pragma unroll
    for (uint32_t u = 0; u < kBack; u++) {
      if (done || got != u || !(w[u] & ~S::kValue)) continue;
      sum += w[u] & S::kValue;
      got++;
      done = (w[u] & S::kSum) != 0;
    }
    j -= got;
    if (got == 0) {
      polls++;
      __nanosleep(32);
    }
  }
  if (__syncthreads_or(!done)) {  // a wait gave up: the keys themselves
    s_base[t] = 0;
    __syncthreads();
    for (uint64_t i = t; i < (uint64_t)tile * kTile; i += kThreads)
      atomicAdd(&s_base[(uint32_t)((src ? src[i] : p.key(i)) >> shift) & 0xffu], 1u);
    __syncthreads();
    sum = s_base[t];
    __syncthreads();
  }
  if (tile) words[at] = (sum + (T)mine) | S::kSum;
  s_base[t] = first + (uint32_t)sum;
  __syncthreads();
#pragma unroll
  for (uint32_t k = 0; k < kKeys; k++) {
    if (base + 32 * k >= p.n) continue;
    const uint32_t d = (uint32_t)(v[k] >> shift) & 0xffu;
    const uint32_t to = s_base[d] + s_cnt[warp][d] + rank[k];
    if (dst) {
      dst[to] = v[k];
    } else {
      p.l[to] = (uint32_t)(v[k] >> p.bits_r);
      p.r[to] = (uint32_t)(v[k] & ((1ull << p.bits_r) - 1));
    }
  }
}

template <class T, uint32_t kKeys>
void queue_passes(Pairs p, uint32_t n_passes, int n_sm, cudaStream_t st) {
  constexpr uint32_t kTile = kThreads * kKeys;
  const uint32_t n_tiles = (uint32_t)((p.n + kTile - 1) / kTile);
  const uint64_t words = 256ull * n_tiles;
  // two passes and more: the first reads the pairs that the last overwrites
  DBuf<unsigned long long> a, b;
  a.alloc(p.n);
  if (n_passes > 2) b.alloc(p.n);
  DBuf<uint32_t> count;  // digit counts, tickets
  DBuf<T> state;
  count.alloc((size_t)kMaxPasses * 256 + kMaxPasses);
  state.alloc(2 * words);
  HBX_CUDA(cudaMemsetAsync(count.p, 0, count.n * 4, st));
  HBX_CUDA(cudaMemsetAsync(state.p, 0, words * sizeof(T), st));
  k_digits<<<std::min<uint32_t>(n_tiles, (uint32_t)n_sm * 4), kThreads, 0, st>>>(p, n_passes, count.p);
  for (uint32_t q = 0; q < n_passes; q++) {
    const unsigned long long* src = q == 0 ? nullptr : q & 1 ? a.p : b.p;
    unsigned long long* dst = q + 1 == n_passes ? nullptr : q & 1 ? b.p : a.p;
    k_pass<T, kKeys><<<n_tiles, kThreads, 0, st>>>(p, src, dst, 8 * q, count.p + 256 * q,
                                            count.p + 256 * kMaxPasses + q, state.p + (q & 1) * words,
                                            state.p + (~q & 1) * words, dev::scan_polls());
  }
  check_launch("pair sort");
}

}  // namespace srt

namespace {

struct SortShape {
  uint32_t bits_r, n_passes, keys;  // keys a thread
  bool wide;                        // 64-bit words
};

SortShape sort_shape(int n_sm, uint64_t n, uint32_t n_left, uint32_t n_right) {
  auto bits_of = [](uint32_t rows) {
    uint32_t b = 0;
    while ((uint64_t)rows > (1ull << b)) b++;
    return b;  // bits that hold row indices below rows
  };
  SortShape s;
  s.bits_r = bits_of(n_right);
  s.n_passes = std::max(2u, (bits_of(n_left) + s.bits_r + 7) / 8);
  // the words' values go up to n; 64-bit words at any n for a test
  const char* wide = std::getenv("HBX_TEST_SORT_WIDE");
  s.wide = n >= (1ull << 30) || (wide && std::strcmp(wide, "1") == 0);
  s.keys = !s.wide && n <= 4ull * n_sm * 8 * srt::kThreads ? 8 : 16;
  return s;
}

}  // namespace

uint64_t pair_sort_bytes(int n_sm, uint64_t n, uint32_t n_left, uint32_t n_right) {
  if (n < 2) return 0;
  const SortShape s = sort_shape(n_sm, n, n_left, n_right);
  const uint64_t tile = (uint64_t)srt::kThreads * s.keys, words = 512 * ((n + tile - 1) / tile);
  return 8 * n * (s.n_passes > 2 ? 2 : 1) + words * (s.wide ? 8 : 4) +
         4 * (srt::kMaxPasses * 257) + 4 * 1024;
}

// Queues the sort of n pairs by (left row, right row) in place on st; rows
// are below n_left / n_right, and bits of the keys beyond those take no pass.
// Its buffers come from the calling thread's pool on st.
void queue_pair_sort(int n_sm, cudaStream_t st, uint32_t* l, uint32_t* r, uint64_t n,
                     uint32_t n_left, uint32_t n_right) {
  if (n < 2) return;
  if (n >= (1ull << 32)) fail(HBX_ERR_UNSUPPORTED, "more than 2^32 pairs to sort");
  const SortShape s = sort_shape(n_sm, n, n_left, n_right);
  const srt::Pairs p{l, r, n, s.bits_r};
  if (s.wide)
    srt::queue_passes<unsigned long long, 16>(p, s.n_passes, n_sm, st);
  else if (s.keys == 8)
    srt::queue_passes<uint32_t, 8>(p, s.n_passes, n_sm, st);
  else
    srt::queue_passes<uint32_t, 16>(p, s.n_passes, n_sm, st);
}

// The same on the context's stream; returns when the pairs are sorted.
void sort_pairs_device(hbx_ctx* C, uint32_t* l, uint32_t* r, uint64_t n, uint32_t n_left,
                       uint32_t n_right) {
  PoolScope scope(C->pool, C->stream);
  queue_pair_sort(C->n_sm, C->stream, l, r, n, n_left, n_right);
  HBX_CUDA(cudaStreamSynchronize(C->stream));
}

}  // namespace hbx
