// ingest.cu -- device-side encoding of two host tables (see ingest.h).
//
// Only the columns a plan reads are copied: per column its cell bytes and
// int64 cell offsets, as the host table holds them.  Then, on the device:
//   k_buckets        partition bucket of every row: std::hash of the
//                    partition cell (and of the prefix cell's first byte)
//                    modulo n_partitions, exactly as data_mngr.h:150-202
//                    computes it; a per-side histogram of buckets;
//   k_pairs_covered  sum over partitions of |L_p| * |R_p|;
//   dictionaries     per equality slot, both tables' cells go into one
//                    open-addressing table keyed by the 64-bit hash of the
//                    cell (up to its first NUL, as equalities_kernel
//                    compares); the row that fills a slot represents it and
//                    numbers it; every cell is then compared byte by byte
//                    with its slot's representative, so a hash collision is
//                    always detected;
//   k_byte_hist +    the frequency-ordered symbol alphabet of the string
//   k_symbol_map     columns (ties by byte value), as the host encoder;
//   k_units + scan + the arenas: string k of slot s starts at the 16-byte
//   k_pack           unit given by the scan of the padded lengths in
//                    (slot, row) order, one warp per string translating
//                    bytes to symbols and writing the string's metadata.
// Each launch covers all columns of its kind and both tables: about fifteen
// launches, clears and copies for a session instead of seventy-five, which is
// what small tables cost (a session's creation: 0.29 against 0.53 ms for 2,601
// x 64,264 rows, 0.17 against 0.32 ms for 2,617 x 2,295).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <map>
#include <string>
#include <vector>

#include "ingest.h"
#include "kernels.cuh"
#include "std_hash.h"

namespace hbx {
namespace ing {

constexpr uint32_t kSharedHist = 4096;  // partitions counted in shared memory

// One table's rows: its partition (and prefix) column, buckets and histogram.
struct BucketJob {
  ColDev part, pre;
  uint32_t use_part, use_pre, n;
  uint32_t* bucket;
  unsigned long long* hist;
};
struct BucketJobs {
  BucketJob side[2];
};
__global__ void k_buckets(const __grid_constant__ BucketJobs jobs, unsigned long long n_part) {
  extern __shared__ uint32_t s_hist[];
  const BucketJob& J = jobs.side[blockIdx.y];
  const bool sh = n_part <= kSharedHist;
  if ((unsigned long long)blockIdx.x * blockDim.x >= J.n) return;  // whole block
  if (sh)
    for (uint32_t k = threadIdx.x; k < n_part; k += blockDim.x) s_hist[k] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < J.n; i += gridDim.x * blockDim.x) {
    unsigned long long b = 0;
    if (J.use_part) {
      const int64_t a = J.part.off[i];
      const uint64_t len = (uint64_t)(J.part.off[i + 1] - a);
      b = std_hash_bytes(J.part.bytes + a, len) % n_part;
    }
    if (J.use_pre) {
      const int64_t a = J.pre.off[i];
      const uint64_t len = (uint64_t)(J.pre.off[i + 1] - a);
      if (len > 2) {
        const unsigned long long two_d = (std_hash_bytes(J.pre.bytes + a, 1) + b) % n_part;
        b = (b + two_d) % n_part;
      }
    }
    J.bucket[i] = (uint32_t)b;
    if (sh)
      atomicAdd(&s_hist[b], 1u);
    else
      atomicAdd(&J.hist[b], 1ull);
  }
  __syncthreads();
  if (sh)
    for (uint32_t k = threadIdx.x; k < n_part; k += blockDim.x)
      if (s_hist[k]) atomicAdd(&J.hist[k], (unsigned long long)s_hist[k]);
}

// Host memory that the device can read (page-locked, or pageable where the
// device goes through the host's page tables) into device memory, a piece per
// blockIdx.y: one launch instead of two copies per column.
struct Piece {
  const uint8_t* src;
  uint8_t* dst;
  uint64_t bytes;
};
constexpr uint32_t kFetchBatch = 32;
struct Pieces {
  Piece p[kFetchBatch];
};
__global__ void k_fetch(const __grid_constant__ Pieces pieces) {
  const Piece& p = pieces.p[blockIdx.y];
  const uint64_t t0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t done = 0;
  if ((((uintptr_t)p.src | (uintptr_t)p.dst) & 15) == 0) {
    const uint64_t n = p.bytes / 16;
    for (uint64_t i = t0; i < n; i += stride)
      reinterpret_cast<uint4*>(p.dst)[i] = reinterpret_cast<const uint4*>(p.src)[i];
    done = n * 16;
  }
  for (uint64_t i = done + t0; i < p.bytes; i += stride) p.dst[i] = p.src[i];
}

__global__ void k_pairs_covered(const unsigned long long* hl, const unsigned long long* hr,
                                unsigned long long n_part, unsigned long long* sum) {
  unsigned long long pairs = 0, used = 0;
  for (unsigned long long p = blockIdx.x * blockDim.x + threadIdx.x; p < n_part;
       p += gridDim.x * blockDim.x) {
    pairs += hl[p] * hr[p];
    used += (hl[p] && hr[p]) ? 1ull : 0ull;
  }
  for (int o = 16; o; o >>= 1) {
    pairs += __shfl_xor_sync(0xffffffffu, pairs, o);
    used += __shfl_xor_sync(0xffffffffu, used, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (pairs) atomicAdd(&sum[kSumPairs], pairs);
    if (used) atomicAdd(&sum[kSumUsed], used);
  }
}

// Rows of a dictionary job: [0, n_left) of the left column, then the right's.
__device__ __forceinline__ uint32_t job_cell(const DictBatch& B, const DictJob& J, uint32_t gid,
                                             const uint8_t** bytes) {
  int64_t a;
  const bool left = gid < B.n_left;
  const ColDev& c = left ? J.l : J.r;
  const uint32_t len = cell_len(c, left ? gid : gid - B.n_left, &a);
  *bytes = c.bytes + a;
  return len;
}

// Places every cell's hash in the job's table; the row that fills a slot
// represents it and gives it the next code (one addition per warp).  The
// row's slot goes where its code will be.  A slot that already holds the
// hash is seen by a plain load: columns of few values then cost no atomics.
__global__ void k_dict_insert(const __grid_constant__ DictBatch B, unsigned long long* sum,
                              unsigned long long seed) {
  const DictJob& J = B.job[blockIdx.y];
  // seed bit 63 set: the test build of kDictSeed that keeps 3 bits of the hash
  const unsigned long long hmask = (seed >> 63) ? 7ull : ~0ull;
  seed &= ~(1ull << 63);
  const uint32_t n = B.n_left + B.n_right, lane = threadIdx.x & 31u;
  for (uint64_t w0 = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); w0 < n;
       w0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t gid = w0 + lane;
    bool fresh = false;
    uint32_t slot = 0;
    if (gid < n) {
      const uint8_t* p;
      const uint32_t len = job_cell(B, J, (uint32_t)gid, &p);
      unsigned long long h = hash_bytes_seeded(p, len, seed) & hmask;
      if (h == kEmpty) h = kEmpty - 1;  // the empty marker; verification keeps this exact
      slot = (uint32_t)(h ^ (h >> 32)) & B.mask;
      bool placed = false;
      for (uint32_t probe = 0; probe <= B.mask; probe++) {
        unsigned long long k = *(volatile unsigned long long*)&J.keys[slot];
        if (k == kEmpty) {
          k = atomicCAS(&J.keys[slot], kEmpty, h);
          fresh = k == kEmpty;
        }
        if (fresh || k == h) {
          placed = true;
          break;
        }
        slot = (slot + 1) & B.mask;
      }
      if (!placed) {
        slot = 0;
        atomicOr(&sum[kSumFlags], (unsigned long long)kFlagTableFull);
      }
      if (gid < B.n_left)
        J.out_l[gid] = (int32_t)slot;
      else
        J.out_r[gid - B.n_left] = (int32_t)slot;
    }
    const unsigned f = __ballot_sync(0xffffffffu, fresh);
    if (!f) continue;
    unsigned long long base = 0;
    if (lane == (uint32_t)__ffs(f) - 1u) base = atomicAdd(J.card, (unsigned long long)__popc(f));
    base = __shfl_sync(0xffffffffu, base, __ffs(f) - 1);
    if (fresh) {
      J.code[slot] = (uint32_t)base + (uint32_t)__popc(f & ((1u << lane) - 1u));
      J.rep[slot] = (uint32_t)gid;
    }
  }
}

// code of each row, and the exact check against the slot's representative
__global__ void k_dict_assign(const __grid_constant__ DictBatch B, unsigned long long* sum) {
  const DictJob& J = B.job[blockIdx.y];
  const uint32_t n = B.n_left + B.n_right;
  for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < n;
       g += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t gid = (uint32_t)g;
    int32_t* out = gid < B.n_left ? J.out_l + gid : J.out_r + (gid - B.n_left);
    const uint32_t slot = (uint32_t)*out;
    *out = (int32_t)J.code[slot];
    const uint32_t r = J.rep[slot];
    if (r == gid) continue;
    const uint8_t *pa, *pb;
    const uint32_t la = job_cell(B, J, gid, &pa), lb = job_cell(B, J, r, &pb);
    bool same = la == lb;
    for (uint32_t k = 0; same && k < la; k++) same = pa[k] == pb[k];
    if (!same) atomicOr(&sum[kSumFlags], (unsigned long long)kFlagCollision);
  }
}

// Composite join keys.  Row i's tuple: its bucket, then its dictionary code
// of each of the rule's equality slots, as 4-byte little-endian words (a
// fixed-width cell for the dictionary kernels).
struct TupleSlots {
  uint32_t k;
  uint32_t slot[dev::kMaxEq];
};
__global__ void k_tuples(const uint32_t* bucket, const int32_t* eq, uint32_t n, TupleSlots ts,
                         uint32_t* out) {
  const uint32_t w = ts.k + 1;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t* o = out + (size_t)i * w;
    o[0] = bucket[i];
    for (uint32_t j = 0; j < ts.k; j++) o[1 + j] = (uint32_t)eq[(size_t)ts.slot[j] * n + i];
  }
}

// The bucket of every tuple code (the bucket of its slot's representative
// row), and the tuples per bucket.
__global__ void k_code_bucket(const unsigned long long* keys, const uint32_t* code,
                              const uint32_t* rep, uint32_t cap, const uint32_t* bucket_l,
                              const uint32_t* bucket_r, uint32_t n_left, uint32_t* code_bucket,
                              uint32_t* per_bucket) {
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < cap; s += gridDim.x * blockDim.x) {
    if (keys[s] == kEmpty) continue;
    const uint32_t r = rep[s];
    const uint32_t b = r < n_left ? bucket_l[r] : bucket_r[r - n_left];
    code_bucket[code[s]] = b;
    atomicAdd(per_bucket + b, 1u);
  }
}

// Dense ids grouped by bucket: code c gets start[bucket] + its rank there
// (ranks in any order; only equality and the grouping matter).
__global__ void k_code_remap(const uint32_t* code_bucket, uint32_t n_codes, const uint32_t* start,
                             uint32_t* cursor, uint32_t* remap) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n_codes; c += gridDim.x * blockDim.x) {
    const uint32_t b = code_bucket[c];
    remap[c] = start[b] + atomicAdd(cursor + b, 1u);
  }
}

__global__ void k_apply_remap(const int32_t* codes, uint32_t n, const uint32_t* remap, int32_t* out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = (int32_t)remap[(uint32_t)codes[i]];
}

// dst = scan[n - 1] + in[n - 1] (+ extra): the total of an exclusive scan
__global__ void k_scan_total(const uint32_t* scan, const uint32_t* in, uint32_t n,
                             unsigned long long extra, unsigned long long* dst) {
  if (threadIdx.x == 0 && blockIdx.x == 0)
    *dst = (n ? (unsigned long long)scan[n - 1] + in[n - 1] : 0ull) + extra;
}

// byte counts of a string column (bytes up to each cell's first NUL)
__global__ void k_byte_hist(const __grid_constant__ StrBatch B, unsigned long long* hist) {
  const ColDev& c = B.job[blockIdx.y].c;
  const uint32_t n = B.job[blockIdx.y].n;
  if (!n) return;
  __shared__ uint32_t s[8][256];
  const uint32_t warp = threadIdx.x >> 5;
  for (uint32_t k = threadIdx.x; k < 8 * 256; k += blockDim.x) (&s[0][0])[k] = 0;
  __syncthreads();
  if (!c.has_nul && ((uintptr_t)c.bytes & 15) == 0) {
    const uint64_t total = (uint64_t)c.off[n];  // cells are contiguous from byte 0
    const uint64_t chunks = (total + 15) / 16;
    for (uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; k < chunks;
         k += (uint64_t)gridDim.x * blockDim.x) {
      const uint64_t b0 = k * 16;
      if (b0 + 16 <= total) {
        const uint4 v = *reinterpret_cast<const uint4*>(c.bytes + b0);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
          for (int j = 0; j < 4; j++) atomicAdd(&s[warp][(w[q] >> (8 * j)) & 0xffu], 1u);
      } else {
        for (uint64_t b = b0; b < total; b++) atomicAdd(&s[warp][c.bytes[b]], 1u);
      }
    }
  } else {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      int64_t a;
      const uint32_t len = cell_len(c, i, &a);
      for (uint32_t k = 0; k < len; k++) atomicAdd(&s[warp][c.bytes[a + k]], 1u);
    }
  }
  __syncthreads();
  for (uint32_t b = threadIdx.x; b < 256; b += blockDim.x) {
    uint32_t t = 0;
    for (int w = 0; w < 8; w++) t += s[w][b];
    if (t) atomicAdd(&hist[b], (unsigned long long)t);
  }
}

// symbol of byte b = 1 + (bytes more frequent than b, or as frequent and
// smaller): the host encoder's stable sort by descending frequency
__global__ void k_symbol_map(const unsigned long long* hist, uint8_t* sym,
                             unsigned long long* sum) {
  __shared__ unsigned long long f[256];
  const uint32_t b = threadIdx.x;
  f[b] = b ? hist[b] : 0ull;
  __syncthreads();
  uint32_t rank = 0, nz = 0;
  for (uint32_t k = 1; k < 256; k++) {
    const unsigned long long fk = f[k];
    if (!fk) continue;
    nz++;
    if (fk > f[b] || (fk == f[b] && k < b)) rank++;
  }
  sym[b] = (b && f[b]) ? (uint8_t)(rank + 1) : (uint8_t)0;
  if (b == 0) sum[kSumSymbols] = nz + 1;
}

__global__ void k_units(const __grid_constant__ StrBatch B) {
  const ColDev& c = B.job[blockIdx.y].c;
  const uint32_t n = B.job[blockIdx.y].n;
  uint32_t* units = B.job[blockIdx.y].units;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int64_t a;
    units[i] = (cell_len(c, i, &a) + 15u) / 16u;
  }
}

// One warp per string: symbols into the arena at unit off16[i], metadata
// {offset / 16, length, 0, 0} + the first 16 symbols + the count signature
// (dev::StrMeta); the longest length goes to *maxlen.  256 threads per block.
__global__ void k_pack(const __grid_constant__ StrBatch B, const uint8_t* sym_g) {
  const StrJob& J = B.job[blockIdx.y];
  const ColDev& c = J.c;
  const uint32_t n = J.n;
  const uint32_t* off16 = J.off16;
  uint8_t* arena = J.arena;
  dev::StrMeta* meta = J.meta;
  __shared__ uint8_t sym[256];
  __shared__ uint32_t s_cnt[8][dev::kSigBuckets];
  for (uint32_t k = threadIdx.x; k < 256; k += blockDim.x) sym[k] = sym_g[k];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31;
  uint32_t* cnt = s_cnt[threadIdx.x >> 5];
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  uint32_t mx = 0;
  for (uint32_t i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < n; i += warps) {
    const int64_t a = c.off[i];
    const uint32_t full = (uint32_t)(c.off[i + 1] - a);
    uint32_t len = full;
    if (c.has_nul) {
      for (uint32_t base = 0; base < full; base += 32) {
        const uint32_t z = __ballot_sync(0xffffffffu, base + lane < full && c.bytes[a + base + lane] == 0);
        if (z) {
          len = base + (uint32_t)__ffs(z) - 1;
          break;
        }
      }
    }
    const uint64_t pos = (uint64_t)off16[i] * 16;
    cnt[lane] = 0;
    __syncwarp();
    for (uint32_t base = 0; base < len; base += 32) {
      const uint32_t j = base + lane;
      const uint32_t v = j < len ? sym[c.bytes[a + j]] : 0u;
      if (j < len) arena[pos + j] = (uint8_t)v;
      // one add per (bucket, chunk): the lowest lane of each bucket group
      const uint32_t b = v ? dev::sig_bucket(v) : 0xffffffffu;
      const unsigned grp = __match_any_sync(0xffffffffu, b);
      if (v && lane == (uint32_t)(__ffs(grp) - 1)) cnt[b] += (uint32_t)__popc(grp);
      __syncwarp();
    }
    __syncwarp();
    uint32_t sw = 0;  // signature word `lane` (lanes 0-7)
    if (lane < 8)
      for (int k = 0; k < 4; k++) sw |= min(cnt[4 * lane + k], 255u) << (8 * k);
    const uint32_t s = (lane < 16 && lane < len) ? sym[c.bytes[a + lane]] : 0u;
    uint32_t v = s << (8 * (lane & 3));
    v |= __shfl_xor_sync(0xffffffffu, v, 1);
    v |= __shfl_xor_sync(0xffffffffu, v, 2);
    const uint32_t w0 = __shfl_sync(0xffffffffu, v, 0), w1 = __shfl_sync(0xffffffffu, v, 4);
    const uint32_t w2 = __shfl_sync(0xffffffffu, v, 8), w3 = __shfl_sync(0xffffffffu, v, 12);
    uint32_t g[8];
#pragma unroll
    for (int k = 0; k < 8; k++) g[k] = __shfl_sync(0xffffffffu, sw, k);
    if (lane == 0) {
      dev::StrMeta m;
      m.loc = make_uint4(off16[i], len, 0u, 0u);
      m.head = make_uint4(w0, w1, w2, w3);
      m.sig[0] = make_uint4(g[0], g[1], g[2], g[3]);
      m.sig[1] = make_uint4(g[4], g[5], g[6], g[7]);
      meta[i] = m;
      mx = max(mx, len);
    }
    __syncwarp();
  }
  if (lane == 0 && mx) atomicMax(J.maxlen, (unsigned long long)mx);
}

}  // namespace ing

int grid_for(uint64_t n, int n_sm, int per_sm) {
  const uint64_t g = (n + 255) / 256;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(g, (uint64_t)n_sm * per_sm));
}

void check_launch(const char* what) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) fail(HBX_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

void scan_u32(const uint32_t* in, uint32_t n, uint32_t* out, cudaStream_t st) {
  const uint32_t nb = (n + dev::kScanChunk - 1) / dev::kScanChunk;
  if (nb <= dev::kScanOnceChunks) {
    // one launch and a clear instead of three launches, where launches are
    // what a scan costs; above, the passes take longer than their launches
    DBuf<unsigned long long> sync;
    sync.alloc(nb + 1);
    HBX_CUDA(cudaMemsetAsync(sync.p, 0, (nb + 1) * 8ull, st));
    dev::k_scan_once_u32<<<nb, 1024, 0, st>>>(in, n, out, sync.p, dev::scan_polls());
    check_launch("ingest scan");
    return;
  }
  DBuf<uint32_t> part;
  part.alloc(nb);
  dev::k_scan_partial_u32<<<nb, 1024, 0, st>>>(in, n, part.p);
  dev::k_scan_top_u32<<<1, 1024, 0, st>>>(part.p, nb);
  dev::k_scan_final_u32<<<nb, 1024, 0, st>>>(in, n, part.p, out);
  check_launch("ingest scan");
}

namespace {

// f(batch, jobs in it) for every kStrBatch of the jobs.
template <class F>
void for_str_batches(const std::vector<ing::StrJob>& jobs, F&& f) {
  for (size_t k = 0; k < jobs.size(); k += ing::kStrBatch) {
    ing::StrBatch B{};
    const size_t m = std::min<size_t>(jobs.size() - k, ing::kStrBatch);
    for (size_t q = 0; q < m; q++) B.job[q] = jobs[k + q];
    f(B, (uint32_t)m);
  }
}

uint32_t most_rows(const std::vector<ing::StrJob>& jobs) {
  uint32_t n = 1;
  for (const ing::StrJob& j : jobs) n = std::max(n, j.n);
  return n;
}

}  // namespace

void byte_hist(const std::vector<ing::StrJob>& jobs, uint64_t work, unsigned long long* hist,
               int n_sm, cudaStream_t st) {
  for_str_batches(jobs, [&](const ing::StrBatch& B, uint32_t m) {
    ing::k_byte_hist<<<dim3(grid_for(work, n_sm, 4), m), 256, 0, st>>>(B, hist);
  });
}

void str_units(const std::vector<ing::StrJob>& jobs, int n_sm, cudaStream_t st) {
  for_str_batches(jobs, [&](const ing::StrBatch& B, uint32_t m) {
    ing::k_units<<<dim3(grid_for(most_rows(jobs), n_sm), m), 256, 0, st>>>(B);
  });
}

void str_pack(const std::vector<ing::StrJob>& jobs, const uint8_t* sym, int n_sm, cudaStream_t st) {
  for_str_batches(jobs, [&](const ing::StrBatch& B, uint32_t m) {
    ing::k_pack<<<dim3(grid_for((uint64_t)most_rows(jobs) * 32, n_sm), m), 256, 0, st>>>(B, sym);
  });
}

void build_dictionaries(const ing::DictBatch& B, uint32_t n_jobs, unsigned long long* keys,
                        unsigned long long* sum, unsigned long long seed, int n_sm,
                        cudaStream_t st) {
  HBX_CUDA(cudaMemsetAsync(keys, 0xff, (size_t)n_jobs * (B.mask + 1ull) * 8, st));
  const uint64_t n = (uint64_t)B.n_left + B.n_right;
  if (!n || !n_jobs) return;
  const dim3 grid(grid_for(n, n_sm), n_jobs);
  ing::k_dict_insert<<<grid, 256, 0, st>>>(B, sum, seed);
  ing::k_dict_assign<<<grid, 256, 0, st>>>(B, sum);
  check_launch("ingest dictionary");
}

std::vector<uint32_t> bucket_rows(const Table& t, int part_col, int64_t prefix_idx,
                                  uint64_t n_part, int n_sm, cudaStream_t st) {
  const uint64_t n = (uint64_t)t.n_rows;
  std::vector<uint32_t> out(n, 0);
  const int pre = prefix_idx != INT_MAX ? (int)prefix_idx : -1;
  if (!n || (part_col < 0 && pre < 0)) return out;
  constexpr uint64_t kChunk = 1ull << 22;
  DBuf<unsigned long long> hist;
  hist.alloc(n_part);
  DBuf<uint32_t> d_out;
  d_out.alloc(std::min(n, kChunk));
  const size_t hist_smem = n_part <= ing::kSharedHist ? n_part * sizeof(uint32_t) : 0;
  for (uint64_t r0 = 0; r0 < n; r0 += kChunk) {
    const uint64_t r1 = std::min(n, r0 + kChunk), m = r1 - r0;
    DBuf<uint8_t> b[2];
    DBuf<int64_t> o[2];
    ing::ColDev view[2] = {{nullptr, nullptr, 0}, {nullptr, nullptr, 0}};
    const int cols[2] = {part_col, pre};
    for (int k = 0; k < 2; k++) {
      if (cols[k] < 0) continue;
      const Column& c = t.cols[(size_t)cols[k]];
      const int64_t a = c.off[r0], z = c.off[r1];
      std::vector<int64_t> off(m + 1);
      for (uint64_t i = 0; i <= m; i++) off[i] = c.off[r0 + i] - a;
      b[k].alloc(std::max<int64_t>(z - a, 16));
      o[k].alloc(m + 1);
      if (z > a)
        HBX_CUDA(cudaMemcpyAsync(b[k].p, c.bytes.data() + a, (size_t)(z - a), cudaMemcpyHostToDevice, st));
      HBX_CUDA(cudaMemcpyAsync(o[k].p, off.data(), (m + 1) * 8, cudaMemcpyHostToDevice, st));
      HBX_CUDA(cudaStreamSynchronize(st));  // off is a local vector
      view[k] = ing::ColDev{b[k].p, o[k].p, 0};
    }
    ing::BucketJobs job{};
    job.side[0] = ing::BucketJob{view[0], view[1], part_col >= 0 ? 1u : 0u, pre >= 0 ? 1u : 0u,
                                 (uint32_t)m, d_out.p, hist.p};
    ing::k_buckets<<<grid_for(m, n_sm, 4), 256, hist_smem, st>>>(job, n_part);
    check_launch("bucket_rows");
    HBX_CUDA(cudaMemcpyAsync(out.data() + r0, d_out.p, m * 4, cudaMemcpyDeviceToHost, st));
    HBX_CUDA(cudaStreamSynchronize(st));
  }
  return out;
}

void pin_table(const hbx_table* ct) {
  hbx_table* t = const_cast<hbx_table*>(ct);
  std::lock_guard<std::mutex> lock(t->pin_mu);
  if (t->pin_tried) return;
  t->pin_tried = true;
  auto pin = [&](const void* p, size_t bytes) {
    if (!p || bytes < (1u << 16)) return;  // small buffers copy fast enough pageable
    if (cudaHostRegister(const_cast<void*>(p), bytes, cudaHostRegisterPortable) == cudaSuccess)
      t->pinned.push_back(const_cast<void*>(p));
    else
      cudaGetLastError();  // not fatal: the copy stages through the driver
  };
  for (const Column& c : t->t.cols) {
    pin(c.bytes.data(), c.bytes.size());
    pin(c.off.data(), c.off.size() * sizeof(int64_t));
  }
}

void unpin_table(hbx_table* t) {
  std::lock_guard<std::mutex> lock(t->pin_mu);
  for (void* p : t->pinned) cudaHostUnregister(p);
  t->pinned.clear();
}

bool device_encode(const hbx_table* left, const hbx_table* right, Encoded* Ep, SideBufs* LB,
                   SideBufs* RB, int n_sm, cudaStream_t st, uint64_t* h2d, std::string* why,
                   bool pin, size_t dict_bytes) {
  Encoded& E = *Ep;
  const Table& TL = left->t;
  const Table& TR = right->t;
  const uint32_t nL = (uint32_t)E.L.n_rows, nR = (uint32_t)E.R.n_rows;
  const uint64_t n_part = E.n_partitions;
  if ((uint64_t)nL + nR > (1ull << 30)) {
    *why = "more than 2^30 rows in the two tables";
    return false;
  }
  // host tables that the device reads through the host's page tables need no
  // page-locking
  int direct = 0;
  if (pin) {
    int dev_id = 0;
    HBX_CUDA(cudaGetDevice(&dev_id));
    HBX_CUDA(cudaDeviceGetAttribute(&direct, cudaDevAttrPageableMemoryAccessUsesHostPageTables, dev_id));
    if (!direct) {
      pin_table(left);
      pin_table(right);
    }
  }
  // a failure below leaves no launch reading the host tables
  struct DrainOnError {
    cudaStream_t st;
    int n = std::uncaught_exceptions();
    ~DrainOnError() {
      if (std::uncaught_exceptions() > n) cudaStreamSynchronize(st);
    }
  } drain{st};
  *h2d = 0;

  // ---- the columns the plan reads, in one block (256-byte aligned pieces)
  struct DevCol {
    size_t bytes_at, off_at;
    const Column* c;
  };
  std::map<int, DevCol> cols_l, cols_r;
  size_t col_bytes = 0;
  auto room = [&](size_t bytes) {
    const size_t at = col_bytes;
    col_bytes += (bytes + 255) / 256 * 256;
    return at;
  };
  auto need = [&](const Table& t, std::map<int, DevCol>& m, int col) {
    if (col < 0 || m.count(col)) return;
    const Column& c = t.cols[(size_t)col];
    DevCol& d = m[col];
    d.bytes_at = room(std::max<size_t>(c.bytes.size(), 16));
    d.off_at = room(c.off.size() * sizeof(int64_t));
    d.c = &c;
    *h2d += c.bytes.size() + c.off.size() * sizeof(int64_t);
  };
  const int pre = E.prefix_idx != INT_MAX ? (int)E.prefix_idx : -1;
  for (int col : {E.part_col, pre}) {
    need(TL, cols_l, col);
    need(TR, cols_r, col);
  }
  for (auto& s : E.eq_slots) {
    need(TL, cols_l, s.first);
    need(TR, cols_r, s.second);
  }
  for (int col : E.L.str_col) need(TL, cols_l, col);
  for (int col : E.R.str_col) need(TR, cols_r, col);
  DBuf<uint8_t> cols;
  cols.alloc(std::max<size_t>(col_bytes, 16));
  {
    // one launch reads them all where the device reads host memory itself,
    // else a copy each
    ing::Pieces P{};
    uint32_t m = 0;
    uint64_t most = 0;
    auto launch = [&]() {
      if (m) ing::k_fetch<<<dim3(grid_for((most + 15) / 16, n_sm, 4), m), 256, 0, st>>>(P);
      m = 0;
      most = 0;
    };
    auto fetch = [&](size_t at, const void* src, size_t bytes) {
      if (!bytes) return;
      if (!direct) {
        HBX_CUDA(cudaMemcpyAsync(cols.p + at, src, bytes, cudaMemcpyHostToDevice, st));
        return;
      }
      P.p[m++] = ing::Piece{static_cast<const uint8_t*>(src), cols.p + at, bytes};
      most = std::max<uint64_t>(most, bytes);
      if (m == ing::kFetchBatch) launch();
    };
    for (auto* side : {&cols_l, &cols_r})
      for (auto& kv : *side) {
        const Column& c = *kv.second.c;
        fetch(kv.second.bytes_at, c.bytes.data(), c.bytes.size());
        fetch(kv.second.off_at, c.off.data(), c.off.size() * sizeof(int64_t));
      }
    launch();
    check_launch("ingest columns");
  }
  auto view = [&](std::map<int, DevCol>& m, int col) {
    if (col < 0) return ing::ColDev{nullptr, nullptr, 0, 0};
    const DevCol& d = m.at(col);
    return ing::ColDev{cols.p + d.bytes_at, reinterpret_cast<const int64_t*>(cols.p + d.off_at),
                       d.c->has_nul ? 1u : 0u, 0};
  };

  const size_t n_eq = E.eq_slots.size();
  const size_t n_sl = E.L.str_col.size(), n_sr = E.R.str_col.size();
  // summary: fixed words, eq card, maxlen L, maxlen R; then the symbol map
  // (read back together), the partitions' and the bytes' histograms: one clear
  const size_t i_card = ing::kSumFixed, i_mxl = i_card + n_eq, i_mxr = i_mxl + n_sl,
               n_sum = i_mxr + n_sr, i_sym = n_sum, i_hist = i_sym + 256 / 8,
               i_bhist = i_hist + 2 * n_part;
  DBuf<unsigned long long> sum;
  sum.alloc(i_bhist + 256);
  HBX_CUDA(cudaMemsetAsync(sum.p, 0, (i_bhist + 256) * sizeof(unsigned long long), st));
  unsigned long long* hist = sum.p + i_hist;
  uint8_t* sym = reinterpret_cast<uint8_t*>(sum.p + i_sym);

  // ---- partition buckets
  const size_t hist_smem = n_part <= ing::kSharedHist ? n_part * sizeof(uint32_t) : 0;
  LB->bucket.alloc(nL);
  RB->bucket.alloc(nR);
  {
    auto job = [&](std::map<int, DevCol>& m, uint32_t n, SideBufs* B, unsigned long long* h) {
      return ing::BucketJob{view(m, E.part_col), view(m, pre), E.part_col >= 0 ? 1u : 0u,
                            pre >= 0 ? 1u : 0u, n, B->bucket.p, h};
    };
    const ing::BucketJobs jobs{{job(cols_l, nL, LB, hist), job(cols_r, nR, RB, hist + n_part)}};
    if (nL || nR)
      ing::k_buckets<<<dim3(grid_for(std::max(nL, nR), n_sm, 4), 2), 256, hist_smem, st>>>(jobs, n_part);
  }
  ing::k_pairs_covered<<<grid_for(n_part, n_sm, 2), 256, 0, st>>>(hist, hist + n_part, n_part, sum.p);
  check_launch("ingest buckets");

  // ---- joint dictionaries (rebuilt with a fresh seed after a collision,
  // below), as many slots to a launch as keep their tables within dict_bytes
  LB->eq.alloc(std::max<size_t>(n_eq * nL, 1));
  RB->eq.alloc(std::max<size_t>(n_eq * nR, 1));
  uint32_t cap = 1024;
  while (cap < 2ull * ((uint64_t)nL + nR)) cap <<= 1;
  const size_t n_tab = current_arena() ? 1 : std::max<size_t>(1, std::min<size_t>(
      {n_eq, (size_t)ing::kDictBatch, (size_t)(dict_bytes / (16ull * cap))}));
  DBuf<unsigned long long> keys;
  DBuf<uint32_t> rep, code;
  keys.alloc(n_tab * cap);
  rep.alloc(n_tab * cap);
  code.alloc(n_tab * cap);
  const char* collide_env = std::getenv("HBX_TEST_DICT_COLLIDE");
  const bool collide_test = collide_env && std::strcmp(collide_env, "1") == 0;
  // attempt k hashes with seed kDictSeed + k; the test build of attempt 0
  // keeps 3 bits of each hash (bit 63 of the seed word asks for that)
  auto seed_of = [&](int attempt) {
    unsigned long long sd = kDictSeed + (unsigned long long)attempt;
    if (collide_test && attempt == 0) sd |= 1ull << 63;
    return sd;
  };
  auto job_of = [&](size_t tab, const ing::ColDev& cl, const ing::ColDev& cr, int32_t* out_l,
                    int32_t* out_r, unsigned long long* card) {
    return ing::DictJob{cl, cr, out_l, out_r, keys.p + tab * cap, code.p + tab * cap,
                        rep.p + tab * cap, card};
  };
  auto eq_dictionaries = [&](unsigned long long seed) {
    for (size_t k = 0; k < n_eq; k += n_tab) {
      ing::DictBatch B{};
      B.n_left = nL;
      B.n_right = nR;
      B.mask = cap - 1;
      const size_t m = std::min(n_tab, n_eq - k);
      for (size_t q = 0; q < m; q++)
        B.job[q] = job_of(q, view(cols_l, E.eq_slots[k + q].first), view(cols_r, E.eq_slots[k + q].second),
                          LB->eq.p + (k + q) * nL, RB->eq.p + (k + q) * nR, sum.p + i_card + k + q);
      build_dictionaries(B, (uint32_t)m, keys.p, sum.p, seed, n_sm, st);
    }
  };
  eq_dictionaries(seed_of(0));

  // ---- symbol alphabet
  {
    std::vector<ing::StrJob> jobs;
    uint64_t work = 1;
    auto side = [&](std::map<int, DevCol>& m, const std::vector<int>& str_col, uint32_t n,
                    const Table& t) {
      for (int col : str_col) {
        if (!n) continue;
        const Column& c = t.cols[(size_t)col];
        work = std::max<uint64_t>(work, c.has_nul ? n : (c.bytes.size() + 15) / 16);
        jobs.push_back(ing::StrJob{view(m, col), n, nullptr, nullptr, nullptr, nullptr, nullptr});
      }
    };
    side(cols_l, E.L.str_col, nL, TL);
    side(cols_r, E.R.str_col, nR, TR);
    byte_hist(jobs, work, sum.p + i_bhist, n_sm, st);
    ing::k_symbol_map<<<1, 256, 0, st>>>(sum.p + i_bhist, sym, sum.p);
    check_launch("ingest symbols");
  }

  // ---- arenas and string metadata: both tables in each launch, or one after the
  // other in the scratch of the entry point without allocation, where the
  // units and offsets of a table are given back before the next is placed
  auto strings = [&](bool of_left, bool of_right) {
    std::vector<ing::StrJob> jobs;
    DBuf<uint32_t> tmp_l, tmp_r;  // arena units, then their offsets
    auto side = [&](std::map<int, DevCol>& m, const std::vector<int>& str_col, uint32_t n,
                    const Table& t, SideBufs* B, DBuf<uint32_t>& tmp, size_t i_mx) {
      const size_t ns = str_col.size();
      uint64_t bound = 16;  // the zero block at the end
      for (int col : str_col) bound += t.cols[(size_t)col].bytes.size() + 15ull * n;
      bound = (bound + 15) / 16 * 16;
      if (bound / 16 > UINT32_MAX) fail(HBX_ERR_UNSUPPORTED, "string arena above 64 GiB");
      B->arena.alloc(bound);
      HBX_CUDA(cudaMemsetAsync(B->arena.p, 0, bound, st));
      B->meta.alloc(std::max<size_t>(ns * n, 1));
      if (!ns || !n) return;
      if ((uint64_t)ns * n > UINT32_MAX) fail(HBX_ERR_UNSUPPORTED, "more than 2^32 strings");
      const size_t half = (ns * n + 63) / 64 * 64;  // 256-byte aligned pieces
      tmp.alloc(2 * half);
      for (size_t k = 0; k < ns; k++)
        jobs.push_back(ing::StrJob{view(m, str_col[k]), n, tmp.p + k * n, tmp.p + half + k * n,
                                   B->arena.p, B->meta.p + k * n, sum.p + i_mx + k});
    };
    if (of_left) side(cols_l, E.L.str_col, nL, TL, LB, tmp_l, i_mxl);
    if (of_right) side(cols_r, E.R.str_col, nR, TR, RB, tmp_r, i_mxr);
    str_units(jobs, n_sm, st);
    if (tmp_l.p) scan_u32(tmp_l.p, (uint32_t)(n_sl * nL), tmp_l.p + tmp_l.n / 2, st);
    if (tmp_r.p) scan_u32(tmp_r.p, (uint32_t)(n_sr * nR), tmp_r.p + tmp_r.n / 2, st);
    str_pack(jobs, sym, n_sm, st);
    check_launch("ingest arenas");
  };
  if (current_arena()) {
    strings(true, false);
    strings(false, true);
  } else {
    strings(true, true);
  }

  // ---- summary
  constexpr int kMaxAttempts = 4;
  std::vector<unsigned long long> h(i_hist);  // and the symbol map
  auto read_summary = [&]() {
    HBX_CUDA(cudaMemcpyAsync(h.data(), sum.p, i_hist * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost, st));
    HBX_CUDA(cudaStreamSynchronize(st));
  };
  read_summary();
  std::memcpy(E.sym_of_byte.data(), h.data() + i_sym, 256);
  auto give_up = [&](const std::string& reason) {
    *why = reason;
    *LB = SideBufs{};
    *RB = SideBufs{};
    return false;
  };
  // two distinct cells shared a hash: every dictionary again with the next seed
  for (int attempt = 1; (h[ing::kSumFlags] & ing::kFlagCollision) && attempt < kMaxAttempts;
       attempt++) {
    const unsigned long long clear = h[ing::kSumFlags] & ~(unsigned long long)ing::kFlagCollision;
    HBX_CUDA(cudaMemcpyAsync(sum.p + ing::kSumFlags, &clear, sizeof clear, cudaMemcpyHostToDevice, st));
    HBX_CUDA(cudaMemsetAsync(sum.p + i_card, 0, n_eq * sizeof(unsigned long long), st));
    eq_dictionaries(seed_of(attempt));
    read_summary();
  }
  if (h[ing::kSumFlags] & ing::kFlagCollision)
    return give_up("dictionary cells collide under four hash seeds");
  if (h[ing::kSumFlags] & ing::kFlagTableFull) return give_up("dictionary table full");
  E.pairs_covered = h[ing::kSumPairs];
  E.n_partitions_used = (uint32_t)h[ing::kSumUsed];
  E.n_symbols = (uint32_t)h[ing::kSumSymbols];
  E.eq_card.assign(n_eq, 1);
  for (size_t k = 0; k < n_eq; k++) E.eq_card[k] = (uint32_t)std::max<unsigned long long>(h[i_card + k], 1);
  E.L.str_maxlen.assign(n_sl, 0);
  E.R.str_maxlen.assign(n_sr, 0);
  for (size_t s = 0; s < n_sl; s++) E.L.str_maxlen[s] = (uint32_t)h[i_mxl + s];
  for (size_t s = 0; s < n_sr; s++) E.R.str_maxlen[s] = (uint32_t)h[i_mxr + s];

  // ---- join-key domains; composite ids for rules whose mixed-radix domain
  // is too large: each row's (bucket, codes) tuple through a dictionary of
  // its own, then the tuple ids regrouped by bucket
  std::vector<size_t> comp_rules;
  for (size_t r = 0; r < E.rules.size(); r++)
    if (!rule_mixed_domain(E, &E.rules[r])) comp_rules.push_back(r);
  const size_t n_comp = comp_rules.size();
  LB->comp.alloc(std::max<size_t>(n_comp * nL, 1));
  RB->comp.alloc(std::max<size_t>(n_comp * nR, 1));
  if (n_comp) {
    DBuf<int32_t> tcode_l, tcode_r;
    DBuf<uint32_t> tup_l, tup_r, code_bucket, per_bucket, start, cursor, remap;
    tcode_l.alloc(std::max<uint32_t>(nL, 1));
    tcode_r.alloc(std::max<uint32_t>(nR, 1));
    code_bucket.alloc(cap);
    remap.alloc(cap);
    per_bucket.alloc(n_part + 1);
    start.alloc(n_part + 1);
    cursor.alloc(n_part + 1);
    DBuf<unsigned long long> dsum;
    dsum.alloc(1);
    for (size_t ci = 0; ci < n_comp; ci++) {
      RuleEnc& re = E.rules[comp_rules[ci]];
      ing::TupleSlots ts{};
      ts.k = (uint32_t)re.eq_slot.size();
      for (uint32_t j = 0; j < ts.k; j++) ts.slot[j] = (uint32_t)re.eq_slot[j];
      const uint32_t w = ts.k + 1;
      tup_l.alloc(std::max<size_t>((size_t)nL * w, 1));
      tup_r.alloc(std::max<size_t>((size_t)nR * w, 1));
      if (nL) ing::k_tuples<<<grid_for(nL, n_sm), 256, 0, st>>>(LB->bucket.p, LB->eq.p, nL, ts, tup_l.p);
      if (nR) ing::k_tuples<<<grid_for(nR, n_sm), 256, 0, st>>>(RB->bucket.p, RB->eq.p, nR, ts, tup_r.p);
      const ing::ColDev tl{reinterpret_cast<const uint8_t*>(tup_l.p), nullptr, 0, 4 * w};
      const ing::ColDev tr{reinterpret_cast<const uint8_t*>(tup_r.p), nullptr, 0, 4 * w};
      unsigned long long n_codes = 0;
      for (int attempt = 0;; attempt++) {
        HBX_CUDA(cudaMemsetAsync(sum.p + ing::kSumFlags, 0, sizeof(unsigned long long), st));
        HBX_CUDA(cudaMemsetAsync(dsum.p, 0, sizeof(unsigned long long), st));
        ing::DictBatch B{};
        B.n_left = nL;
        B.n_right = nR;
        B.mask = cap - 1;
        B.job[0] = job_of(0, tl, tr, tcode_l.p, tcode_r.p, dsum.p);
        build_dictionaries(B, 1, keys.p, sum.p, seed_of(attempt), n_sm, st);
        unsigned long long got[2] = {0, 0};
        HBX_CUDA(cudaMemcpyAsync(&got[0], sum.p + ing::kSumFlags, 8, cudaMemcpyDeviceToHost, st));
        HBX_CUDA(cudaMemcpyAsync(&got[1], dsum.p, 8, cudaMemcpyDeviceToHost, st));
        HBX_CUDA(cudaStreamSynchronize(st));
        if (got[0] & ing::kFlagTableFull) return give_up("dictionary table full");
        n_codes = got[1];
        if (!(got[0] & ing::kFlagCollision)) break;
        if (attempt + 1 == kMaxAttempts) return give_up("join-key tuples collide under four hash seeds");
      }
      HBX_CUDA(cudaMemsetAsync(per_bucket.p, 0, (n_part + 1) * 4, st));
      HBX_CUDA(cudaMemsetAsync(cursor.p, 0, (n_part + 1) * 4, st));
      ing::k_code_bucket<<<grid_for(cap, n_sm), 256, 0, st>>>(keys.p, code.p, rep.p, cap,
                                                              LB->bucket.p, RB->bucket.p, nL,
                                                              code_bucket.p, per_bucket.p);
      scan_u32(per_bucket.p, (uint32_t)(n_part + 1), start.p, st);  // start[n_part] = n_codes
      if (n_codes)
        ing::k_code_remap<<<grid_for(n_codes, n_sm), 256, 0, st>>>(code_bucket.p, (uint32_t)n_codes,
                                                                  start.p, cursor.p, remap.p);
      if (nL)
        ing::k_apply_remap<<<grid_for(nL, n_sm), 256, 0, st>>>(tcode_l.p, nL, remap.p,
                                                               LB->comp.p + ci * nL);
      if (nR)
        ing::k_apply_remap<<<grid_for(nR, n_sm), 256, 0, st>>>(tcode_r.p, nR, remap.p,
                                                               RB->comp.p + ci * nR);
      check_launch("ingest composite keys");
      std::vector<uint32_t> hs(n_part + 1);
      HBX_CUDA(cudaMemcpyAsync(hs.data(), start.p, (n_part + 1) * 4, cudaMemcpyDeviceToHost, st));
      HBX_CUDA(cudaStreamSynchronize(st));
      re.composite = true;
      re.comp_index = (int)ci;
      re.domain = std::max<uint64_t>(n_codes, 1);
      re.part_key_begin.assign(hs.begin(), hs.end());
      if (re.domain > (1ull << 31)) fail(HBX_ERR_UNSUPPORTED, "join key domain too large");
    }
  }
  return true;
}

}  // namespace hbx
