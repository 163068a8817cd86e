// ghb_join.cu — device hash equi-join: build (J1) and probe (J2).
//
// Replaces the reference's join, which sorted both inputs' row indices on the
// GPU and merged them single-threaded on the CPU
// (gpu_impl/src/Operator/SortMergeJoinPredicate.cu:8-461), then gathered the
// retained columns on the host (gpu_impl/src/Operator/BaseJoinPredicate.cu:
// 4-97).  Hive's CPU map-join probes a power-of-two open-addressing table
// whose value store holds each build row's retained columns
// (VectorMapJoinFastLongHashTable.java:99-254, VectorMapJoinFastLongHashMap.
// java:71-84).  The device table keeps, per slot, the key, the (first row,
// count) of the rows with that key and the first row's payload words, in
// three arrays (below), under one of two layouts the build chooses on the
// device from the keys' range (join_layout):
//
//   direct  dense keys (a range below twice the rows, the surrogate key of a
//           dimension table): slot = key - min; the probe loads the slot's
//           count, no key array, no bucket scan;
//   hashed  4-slot buckets, Fibonacci-hashed bucket index; slots fill in order
//           inside a bucket and spill to the next bucket (linear probing by
//           buckets), so one 32-byte load of the bucket's keys settles almost
//           every probe.  The key INT64_MIN, whose image is the empty marker,
//           lives in slot 0 of an extra side bucket.
//
// A key that occurs more than once in the build chains its later rows through
// chain[slot] / next[row] (row + 1, 0 ends the chain; pushed with atomicExch)
// and their payloads are read from the build columns.  The default load
// factor is 0.5, below Hive's hive.hashtable.loadfactor (0.75): at 0.75 more
// full buckets send a probe on to the next bucket, and the 60M-row probe
// measured 7% slower.  Keys and results stream with evict-first loads and
// stores.
//
// The probe counts, then writes (two passes over fixed chunks of probe rows,
// no ordering dependency between CTAs):
//   J2a  count: each CTA takes a chunk, loads its keys, issues the table
//        loads of all its rows together, stores each row's slot (-1 = no
//        match) and each warp's output-row count (a warp covers consecutive
//        rows of the chunk);
//   J2b  scan: the warp counts become output offsets (a multi-CTA look-back
//        scan);
//   J2c  write: each warp re-reads its rows' slots, loads each matching
//        slot's payload words, scans its rows' output counts and writes
//        (probe row, build row, payloads) at its offset, in probe-row order.
// Neither pass takes a CTA barrier per chunk.
#include <algorithm>
#include <map>
#include <mutex>

#include "ghb_ctx.hpp"
#include "ghb_log.hpp"

namespace ghb {

// Slot s = bucket * 4 + index (a direct table: key - min).  The slots' fields
// live in three arrays, so each probe pass reads one dense array: the hashed
// count pass only keys (4 per bucket = one 32-byte sector), the direct one
// only the counts, the write pass the payload words and, when it needs them,
// the (first row, count) pairs.
//   key[s]   uint64 key image (flip_i64 of the key, 0 = empty)
//   meta[s]  int2 {first build row + 1, build rows with this key}
//   pay[s]   ulonglong2, the first build row's inline payload words

constexpr int kJThreads = 256;
constexpr int kJItems = 4;
constexpr int kChunk = kJThreads * kJItems;   // probe rows per chunk
constexpr int kMaxPay = GHB_MAX_JOIN_PAYLOAD;
constexpr int kInline = 2;

// Bucket of a key image: Fibonacci (multiplicative) hashing, the top bits of
// u * 2^64/phi.  One 64-bit multiply; consecutive keys land far apart.
__device__ __forceinline__ int64_t bucket_of(unsigned long long u, int shift) {
  return (int64_t)((u * 0x9E3779B97F4A7C15ull) >> shift);
}

struct BuildParams {
  ghb_column key;
  int32_t n_inline;
  ghb_column pay[kInline];
  unsigned long long* kimg;   // key[s] of the layout above
  int2* meta;
  ulonglong2* payw;
  int32_t* chain_p1;     // [slots]
  int32_t* next_p1;      // [build rows]
  int64_t bmask;         // hashed buckets - 1
  int32_t hshift;        // 64 - log2(hashed buckets)
  int64_t side;          // index of the side bucket
  unsigned long long* stats;  // [0] rows stored, [1] max duplicates
  int32_t* status;
  int64_t slots;         // hashed slots allocated (a direct table fits in them)
};

// The table's layout, decided on the device from the build keys' range
// (stats[2] non-NULL keys, stats[3] max of the complemented order images,
// stats[4] max of the order images): dense keys (a range below twice the
// rows and within the allocated slots, the common surrogate key of a
// dimension table) get a direct table, slot = key - min, with no key array
// and no bucket scan on probe; other keys the hashed buckets.  Every thread
// of the build and probe kernels computes the same answer from the same
// words, so no host round trip is needed.
struct JoinLayout {
  bool direct;
  int64_t dmin;
  int64_t drange;
};

__host__ __device__ inline JoinLayout join_layout(const unsigned long long* stats, int64_t build_rows,
                                                  int64_t slots) {
  JoinLayout L{false, 0, 0};
  if (stats[2] == 0) return L;
  const unsigned long long umin = ~stats[3], umax = stats[4];
  const unsigned long long span = umax - umin;   // the images keep the keys' order and distances
  if (span < 2ull * (unsigned long long)build_rows && span < (unsigned long long)slots && span < (1ull << 30)) {
    L.direct = true;
    L.dmin = (int64_t)(umin ^ 0x8000000000000000ull);
    L.drange = (int64_t)span + 1;
  }
  return L;
}

// The build keys' range into stats[2..4] (zeroed with the table).
__global__ void __launch_bounds__(256) join_key_range_kernel(ghb_column key, unsigned long long* stats) {
  unsigned long long cmin = 0, umax = 0, cnt = 0;   // cmin: max of ~image = ~(min image)
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < key.n;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t raw = ld_raw(key, r);
    if (raw_is_null(key, raw, r)) continue;
    const unsigned long long u = flip_i64(raw);
    cmin = max(cmin, ~u);
    umax = max(umax, u);
    cnt++;
  }
  for (int o = 16; o > 0; o >>= 1) {
    cmin = max(cmin, __shfl_down_sync(0xffffffffu, cmin, o));
    umax = max(umax, __shfl_down_sync(0xffffffffu, umax, o));
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  }
  // one set of atomics per CTA (the same three words from every warp would
  // serialise at L2)
  __shared__ unsigned long long s_red[3][8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_red[0][warp] = cmin;
    s_red[1][warp] = umax;
    s_red[2][warp] = cnt;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      cmin = max(cmin, s_red[0][w]);
      umax = max(umax, s_red[1][w]);
      cnt += s_red[2][w];
    }
    if (cnt) {
      atomicMax(&stats[3], cmin);
      atomicMax(&stats[4], umax);
      atomicAdd(&stats[2], cnt);
    }
  }
}

// Zeroes what the chosen layout reads before a build row fills it: a direct
// table's counts and chain heads of the key range, or the hashed table's keys,
// counts and chain heads (the payload words are read only in filled slots).
// 1.5M dense keys: 6 us, where clearing every allocated slot cost 20.
__global__ void __launch_bounds__(256) join_clear_kernel(BuildParams p) {
  const JoinLayout L = join_layout(p.stats, p.key.n, p.slots);
  const int64_t n = L.direct ? (L.drange + 3) / 4 : (p.side + 1);   // groups of four slots
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    uint4* m = (uint4*)(p.meta + i * 4);
    m[0] = zero;
    m[1] = zero;
    *(uint4*)(p.chain_p1 + i * 4) = zero;
    if (!L.direct) {
      uint4* k = (uint4*)(p.kimg + i * 4);
      k[0] = zero;
      k[1] = zero;
    }
  }
}

__global__ void __launch_bounds__(256) join_build_kernel(BuildParams p) {
  const JoinLayout L = join_layout(p.stats, p.key.n, p.slots);
  unsigned long long stored = 0, maxdup = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < p.key.n;
       r += (int64_t)gridDim.x * blockDim.x) {
    int64_t raw = ld_raw(p.key, r);
    if (raw_is_null(p.key, raw, r)) continue;   // NULL keys never join
    unsigned long long u = flip_i64(raw);
    int64_t bk, j = -1;
    if (L.direct) {   // slot = key - dmin: bucket * 4 + j
      const unsigned long long d = (unsigned long long)raw - (unsigned long long)L.dmin;
      bk = (int64_t)(d >> 2);
      j = (int64_t)(d & 3);
    } else if (u == 0) {
      bk = p.side;
      j = 0;
    } else {
      bk = bucket_of(u, p.hshift);
      for (int64_t probes = 0; probes <= p.bmask && j < 0; probes++) {
        for (int q = 0; q < 4; q++) {
          unsigned long long cur = p.kimg[bk * 4 + q];
          if (cur == 0) {
            unsigned long long prev = atomicCAS(&p.kimg[bk * 4 + q], 0ull, u);
            if (prev == 0 || prev == u) { j = q; break; }
            cur = prev;
          }
          if (cur == u) { j = q; break; }
        }
        if (j < 0) bk = (bk + 1) & p.bmask;
      }
      if (j < 0) {   // table full: cannot happen with load factor < 1
        raise_status(p.status, kDevCapacity);
        continue;
      }
    }
    const int64_t slot = bk * 4 + j;
    int old = atomicAdd(&p.meta[slot].y, 1);
    if (old == 0) {
      p.meta[slot].x = (int32_t)(r + 1);
      if (p.n_inline > 0) p.payw[slot].x = (unsigned long long)ld_raw(p.pay[0], r);
      if (p.n_inline > 1) p.payw[slot].y = (unsigned long long)ld_raw(p.pay[1], r);
    } else {
      p.next_p1[r] = atomicExch(&p.chain_p1[slot], (int)(r + 1));
    }
    stored++;
    maxdup = max(maxdup, (unsigned long long)(old + 1));
  }
  // one atomic per CTA for the statistics (per warp, thousands of warps'
  // atomics on two words would serialise at L2)
  for (int o = 16; o > 0; o >>= 1) {
    stored += __shfl_down_sync(0xffffffffu, stored, o);
    maxdup = max(maxdup, __shfl_down_sync(0xffffffffu, maxdup, o));
  }
  __shared__ unsigned long long s_red[2][8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_red[0][warp] = stored;
    s_red[1][warp] = maxdup;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      stored += s_red[0][w];
      maxdup = max(maxdup, s_red[1][w]);
    }
    if (stored) atomicAdd(&p.stats[0], stored);
    if (maxdup) atomicMax(&p.stats[1], maxdup);
  }
}

// ------------------------------------------------------------------ probe
struct ProbeParams {
  const unsigned long long* kimg;
  const int2* meta;
  const ulonglong2* payw;
  const int32_t* chain_p1;
  const int32_t* next_p1;
  const unsigned long long* stats;
  int64_t bmask;
  int32_t hshift;
  int64_t side;
  ghb_column pkey;
  int32_t join_type;
  int32_t nbp, npp, n_inline;
  int32_t lean;            // INNER, no probe payloads, every build payload inline and non-NULL
  ghb_column bpay[kMaxPay];
  ghb_out_column obp[kMaxPay];
  ghb_column ppay[kMaxPay];
  ghb_out_column opp[kMaxPay];
  int32_t* out_prow;
  int32_t* out_brow;
  int32_t prow_base;       // added to every probe row id written (a chunk of a longer probe)
  int64_t n, nchunks, cap;
  int32_t* slot_of_row;    // [n] slot (bucket * 4 + index) of the row's key, -1 = no match
  int64_t* chunk_count;    // [nchunks * warps per CTA] output rows of each warp's rows of a
                           // chunk (a warp covers 32 * IT consecutive rows), then their offset
  int64_t* d_out_rows;
  int32_t* status;
  int64_t build_rows;      // with slots: the table's layout (join_layout of stats)
  int64_t slots;
  int32_t dup_bit;         // set in slot_of_row where the key has several build rows; 0: the slots
                           // leave no bit free
};

// Output rows a probe row produces, from its slot's count (0 = no match).
__device__ __forceinline__ int32_t out_rows_of(int join_type, int32_t count) {
  if (join_type == GHB_LEFT_SEMI_JOIN) return count > 0 ? 1 : 0;
  if (join_type == GHB_LEFT_OUTER_JOIN) return count > 0 ? count : 1;
  return count;
}

__device__ __forceinline__ void load_keys(const unsigned long long* kimg, int64_t bk,
                                          unsigned long long k[4]) {
  const ulonglong2* s = (const ulonglong2*)(kimg + bk * 4);
  ulonglong2 x = s[0], y = s[1];
  k[0] = x.x;
  k[1] = x.y;
  k[2] = y.x;
  k[3] = y.y;
}

// Index (0..3) of `u` among the bucket's keys, -1 when an empty slot ends
// the search, -2 when the bucket is full of other keys.
__device__ __forceinline__ int find_in(const unsigned long long k[4], unsigned long long u) {
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (k[q] == u) return q;
    if (k[q] == 0) return -1;
  }
  return -2;
}

// The count pass over a direct table: one load of the slot's row count per
// probe row, nothing else, so a thread keeps little and many CTAs fit on an
// SM.  It runs beside the hashed count pass; the build's key range chooses
// which of the two does the work and the other returns at once.
template <int TH, int IT, bool KEY_INT, bool NULLABLE>
__global__ void __launch_bounds__(TH) join_count_direct_kernel(ProbeParams p) {
  static_assert(TH * IT == kChunk, "a CTA iteration covers one chunk");
  const JoinLayout L = join_layout(p.stats, p.build_rows, p.slots);
  if (!L.direct) return;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const bool unique = p.stats[1] <= 1;
  // every key of [min, max] present once (a dense surrogate key): a probe key
  // in the range matches, with no table load
  const bool full = unique && p.stats[2] == (unsigned long long)L.drange;
  // the lean write pass recomputes a direct table's slot from the key, so
  // this pass writes no slots for it
  const bool keep_slots = !(p.lean && p.out_brow == nullptr && unique);
  const int woff = warp * (32 * IT) + lane;
  auto load_chunk_keys = [&](int64_t c, long long* raw) {
    const int64_t cbase = c * kChunk;
    const int left = (int)min((int64_t)kChunk, p.n - cbase);
#pragma unroll
    for (int k = 0; k < IT; k++) {
      const int off = woff + k * 32;
      raw[k] = 0;
      if (c < p.nchunks && off < left)
        raw[k] = KEY_INT ? (long long)__ldcs((const int*)p.pkey.data + cbase + off)
                         : __ldcs((const long long*)p.pkey.data + cbase + off);
    }
  };
  long long next_raw[IT];
  load_chunk_keys(blockIdx.x, next_raw);
  for (int64_t c = blockIdx.x; c < p.nchunks; c += gridDim.x) {
    const int64_t cbase = c * kChunk;
    const int left = (int)min((int64_t)kChunk, p.n - cbase);
    long long raw[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) raw[k] = next_raw[k];
    load_chunk_keys(c + gridDim.x, next_raw);
    unsigned long long d[IT];
    int32_t cnt[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) {
      const int off = woff + k * 32;
      const bool valid = off < left && !(NULLABLE && raw_is_null(p.pkey, raw[k], cbase + off));
      d[k] = (unsigned long long)raw[k] - (unsigned long long)L.dmin;
      const bool inr = valid && d[k] < (unsigned long long)L.drange;
      cnt[k] = inr ? (full ? 1 : p.meta[d[k]].y) : 0;
    }
    uint64_t m_sum = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
      const int off = woff + k * 32;
      if (off < left) {
        if (keep_slots)
          p.slot_of_row[cbase + off] = cnt[k] > 0 ? (int32_t)d[k] | (cnt[k] > 1 ? p.dup_bit : 0) : -1;
        m_sum += (uint64_t)out_rows_of(p.join_type, unique ? (cnt[k] > 0 ? 1 : 0) : cnt[k]);
      }
    }
    for (int o = 16; o > 0; o >>= 1) m_sum += __shfl_down_sync(0xffffffffu, m_sum, o);
    if (lane == 0) p.chunk_count[c * (TH / 32) + warp] = (int64_t)m_sum;
  }
}

// TH threads x IT rows per thread = one chunk (kChunk rows) per iteration.
// Four 256-thread CTAs per SM (64 registers): more key and table loads in flight.
template <int TH, int IT, bool KEY_INT, bool NULLABLE>
__global__ void __launch_bounds__(TH, TH == 512 ? 2 : TH == 256 ? 4 : 1) join_count_kernel(ProbeParams p) {
  constexpr int kJThreads = TH, kJItems = IT;
  static_assert(TH * IT == kChunk, "a CTA iteration covers one chunk");
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const bool unique = p.stats[1] <= 1;   // every key once: a match is one output row
  if (join_layout(p.stats, p.build_rows, p.slots).direct) return;   // join_count_direct_kernel's table
  const int woff = warp * (32 * kJItems) + lane;
  // The keys of the CTA's next chunk are loaded while this chunk probes the
  // table, so the DRAM latency of the key stream overlaps the table loads.
  auto load_chunk_keys = [&](int64_t c, long long* raw) {
    const int64_t cbase = c * kChunk;
    const int left = (int)min((int64_t)kChunk, p.n - cbase);
#pragma unroll
    for (int k = 0; k < kJItems; k++) {
      const int off = woff + k * 32;
      raw[k] = 0;
      if (c < p.nchunks && off < left)
        raw[k] = KEY_INT ? (long long)__ldcs((const int*)p.pkey.data + cbase + off)
                         : __ldcs((const long long*)p.pkey.data + cbase + off);
    }
  };
  long long next_raw[kJItems];
  load_chunk_keys(blockIdx.x, next_raw);
  for (int64_t c = blockIdx.x; c < p.nchunks; c += gridDim.x) {
    const int64_t cbase = c * kChunk;
    // rows of this chunk left (a full chunk unless it is the last one)
    const int left = (int)min((int64_t)kChunk, p.n - cbase);
    long long cur_raw[kJItems];
#pragma unroll
    for (int k = 0; k < kJItems; k++) cur_raw[k] = next_raw[k];
    load_chunk_keys(c + gridDim.x, next_raw);
    unsigned long long u[kJItems];
    bool valid[kJItems];
#pragma unroll
    for (int k = 0; k < kJItems; k++) {
      const int off = woff + k * 32;
      const long long raw = cur_raw[k];
      valid[k] = off < left && !(NULLABLE && raw_is_null(p.pkey, raw, cbase + off));
      u[k] = flip_i64(raw);
    }
    uint64_t m_sum = 0;
    int64_t bk[kJItems];
    unsigned long long keys[kJItems][4];
#pragma unroll
    for (int k = 0; k < kJItems; k++) {
      bk[k] = bucket_of(u[k], p.hshift);
      if (valid[k] && u[k] != 0) load_keys(p.kimg, bk[k], keys[k]);
    }
#pragma unroll
    for (int k = 0; k < kJItems; k++) {
      const int off = woff + k * 32;
      const int64_t row = cbase + off;
      int32_t slot = -1, count = 0;
      if (valid[k]) {
        if (u[k] == 0) {
          int32_t cnt = p.meta[p.side * 4].y;
          if (cnt > 0) { slot = (int32_t)(p.side * 4); count = cnt; }
        } else {
          int q = find_in(keys[k], u[k]);
          while (q == -2) {   // bucket full of other keys: continue in the next one
            bk[k] = (bk[k] + 1) & p.bmask;
            load_keys(p.kimg, bk[k], keys[k]);
            q = find_in(keys[k], u[k]);
          }
          if (q >= 0) {
            slot = (int32_t)(bk[k] * 4 + q);
            count = unique ? 1 : p.meta[slot].y;
          }
        }
      }
      if (off < left) {
        p.slot_of_row[row] = count > 1 ? slot | p.dup_bit : slot;
        m_sum += (uint64_t)out_rows_of(p.join_type, count);
      }
    }
    for (int o = 16; o > 0; o >>= 1) m_sum += __shfl_down_sync(0xffffffffu, m_sum, o);
    if (lane == 0) p.chunk_count[c * (kJThreads / 32) + warp] = (int64_t)m_sum;
  }
}

// Chunk counts -> exclusive offsets in place, many CTAs: each claims a tile
// of 1024 counts in order, scans it, and gets the tile's offset from the tiles
// before it by decoupled look-back; the last tile writes the total.
struct ScanParams {
  int64_t* counts;
  int64_t n;
  int64_t ntiles;
  int64_t* d_total;
  uint64_t* lb;
  uint32_t epoch;
  unsigned long long* counters;
  int32_t* status;
  int32_t spin_limit;   // look-back polls before GHB_ERR_TIMEOUT
};

__global__ void __launch_bounds__(1024) join_scan_lb_kernel(ScanParams p) {
  __shared__ int64_t s_tile;
  __shared__ int64_t s_warp[32];
  __shared__ uint64_t s_excl;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  while (true) {
    claim_tile(&p.counters[0], &s_tile);
    const int64_t tile = s_tile;
    if (tile >= p.ntiles) break;
    const int64_t i = tile * 1024 + threadIdx.x;
    const int64_t v = i < p.n ? p.counts[i] : 0;
    int64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      const int64_t w = s_warp[lane];
      int64_t wi = w;
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(0xffffffffu, wi, o);
        if (lane >= o) wi += t;
      }
      s_warp[lane] = wi - w;
      const int64_t total = __shfl_sync(0xffffffffu, wi, 31);
      const uint64_t ex = lookback_exclusive(p.lb, p.epoch, tile, (uint64_t)total, p.status,
                                                    p.spin_limit);
      if (lane == 0) {
        s_excl = ex;
        if (tile == p.ntiles - 1) *p.d_total = (int64_t)(ex + total);
      }
    }
    __syncthreads();
    if (i < p.n) p.counts[i] = (int64_t)s_excl + s_warp[warp] + incl - v;
    __syncthreads();
  }
  claim_finish(p.counters);
}

// One CTA: chunk counts -> exclusive offsets in place; the total to d_out_rows.
__global__ void __launch_bounds__(1024) join_scan_kernel(int64_t* counts, int64_t n, int64_t* d_total) {
  __shared__ int64_t s_part[1024];
  const int t = threadIdx.x;
  const int64_t per = (n + 1023) / 1024;
  const int64_t lo = t * per, hi = min(n, lo + per);
  int64_t sum = 0;
  for (int64_t i = lo; i < hi; i++) sum += counts[i];
  s_part[t] = sum;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int64_t v = t >= o ? s_part[t - o] : 0;
    __syncthreads();
    s_part[t] += v;
    __syncthreads();
  }
  int64_t run = s_part[t] - sum;
  for (int64_t i = lo; i < hi; i++) {
    int64_t c = counts[i];
    counts[i] = run;
    run += c;
  }
  if (t == 1023) *d_total = s_part[1023];
}

// The payload descriptors and output pointers of a probe, copied to shared
// memory once per CTA for the general emit path below.
struct EmitDesc {
  ghb_column bpay[kMaxPay];
  ghb_out_column obp[kMaxPay];
  ghb_column ppay[kMaxPay];
  ghb_out_column opp[kMaxPay];
  int32_t* out_prow;
  int32_t* out_brow;
  int32_t prow_base;
  int32_t nbp, npp;
};

__device__ __forceinline__ void load_emit_desc(const ProbeParams& p, EmitDesc* d) {
  if (threadIdx.x < kMaxPay) {
    const int j = threadIdx.x;
    d->bpay[j] = p.bpay[j];
    d->obp[j] = p.obp[j];
    d->ppay[j] = p.ppay[j];
    d->opp[j] = p.opp[j];
  }
  if (threadIdx.x == 0) {
    d->out_prow = p.out_prow;
    d->out_brow = p.out_brow;
    d->prow_base = p.prow_base;
    d->nbp = p.nbp;
    d->npp = p.npp;
  }
  __syncthreads();
}

// Writes raw[k] (NULL: bit k of `nulls`) to row base + pos[k], k with bit k of
// `live`.
template <int N>
__device__ __forceinline__ void put_words(const ghb_out_column& o, int type, const int64_t (&raw)[N], uint32_t nulls,
                                          int64_t base, const int64_t (&pos)[N], uint32_t live) {
  if (type == GHB_INT) {
    int* dst = (int*)o.data + base;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) __stcs(dst + pos[k], nulls >> k & 1 ? INT32_MAX : (int)raw[k]);
  } else {
    const long long none = type == GHB_LONG ? (long long)INT64_MAX : 0x7ff8000000000000ll;
    long long* dst = (long long*)o.data + base;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) __stcs(dst + pos[k], nulls >> k & 1 ? none : (long long)raw[k]);
  }
  if (o.is_null) {
    uint8_t* dst = o.is_null + base;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) dst[pos[k]] = nulls >> k & 1;
  }
}

// Writes IT output rows of a thread (k with bit k of `live`) at wpos + pos[k]:
// probe row row(k) with build row brow[k] (bit k of `hit`; else an outer miss or
// a semi join's row), whose inline payload words are w[k] when INL.  One column
// at a time, its loads issued before its stores.
template <int IT, bool INL, typename ROW>
__device__ __forceinline__ void emit_rows(const EmitDesc& d, int n_inline, uint32_t live, uint32_t hit, int64_t wpos,
                                          const int64_t (&pos)[IT], const ROW& row, const int32_t (&brow)[IT],
                                          const ulonglong2 (&w)[IT]) {
  int64_t raw[IT];
  if (d.out_prow) {
#pragma unroll
    for (int k = 0; k < IT; k++)
      if (live >> k & 1) __stcs(d.out_prow + wpos + pos[k], (int)row(k) + d.prow_base);
  }
  if (d.out_brow) {
#pragma unroll
    for (int k = 0; k < IT; k++)
      if (live >> k & 1) __stcs(d.out_brow + wpos + pos[k], hit >> k & 1 ? brow[k] : -1);
  }
  for (int j = 0; j < d.nbp; j++) {
    const ghb_column& col = d.bpay[j];
    if (INL && j < n_inline) {   // not a BYTEMAP column
#pragma unroll
      for (int k = 0; k < IT; k++) raw[k] = (int64_t)(j == 0 ? w[k].x : w[k].y);
    } else {
#pragma unroll
      for (int k = 0; k < IT; k++) raw[k] = hit >> k & 1 ? ld_raw(col, brow[k]) : 0;
    }
    uint32_t nulls = live & ~hit;
    if (col.null_mode != GHB_NULLS_NONE) {
#pragma unroll
      for (int k = 0; k < IT; k++)
        if (hit >> k & 1) nulls |= (raw_is_null(col, raw[k], brow[k]) ? 1u : 0u) << k;
    }
    put_words<IT>(d.obp[j], col.type, raw, nulls, wpos, pos, live);
  }
  for (int j = 0; j < d.npp; j++) {
    const ghb_column& col = d.ppay[j];
#pragma unroll
    for (int k = 0; k < IT; k++) raw[k] = live >> k & 1 ? ld_raw(col, row(k)) : 0;
    uint32_t nulls = 0;
    if (col.null_mode != GHB_NULLS_NONE) {
#pragma unroll
      for (int k = 0; k < IT; k++)
        if (live >> k & 1) nulls |= (raw_is_null(col, raw[k], row(k)) ? 1u : 0u) << k;
    }
    put_words<IT>(d.opp[j], col.type, raw, nulls, wpos, pos, live);
  }
}

// The write pass of an INNER join on unique build keys whose output is the
// probe row and at most two inline, non-NULL build payloads (p.lean, no build
// row ids): a row's output is its slot's two payload words or nothing.  A warp
// takes units of UNIT rows (the rows of one count): the keys or slots of a
// unit are loaded together, then each 32 rows' words are gathered and stored.
// It runs beside the general write pass; the build's statistics (unique keys)
// choose which of the two does the work and the other returns at once.
//
// Bound by the SM's requests to L2, one per gathered row (57M rows of the 60M
// probe).  432 us there at 40 warps per SM with one gather per thread in
// flight; 487 us with four of a thread's gathers together and the next rows'
// keys loaded ahead (47 registers, which also hold what the stores wait for);
// two together 447-457 us, four 506; 56 or 64 warps 450 and 452; gathers that
// do not allocate in L1 640 us.
template <int UNIT>
__global__ void __launch_bounds__(kJThreads, 5) join_write_lean_kernel(const __grid_constant__ ProbeParams p) {
  if (!(p.lean && p.out_brow == nullptr && p.stats[1] <= 1)) return;
  constexpr int kIt = UNIT / 32;   // rows of a unit per lane
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  // a direct table: the slot is the key's offset from the minimum, read from
  // the key itself (the count pass wrote no slots); a full one (every key of
  // the range present) needs no check of the slot
  const JoinLayout L = join_layout(p.stats, p.build_rows, p.slots);
  const bool from_keys = L.direct;
  const bool full = from_keys && p.stats[2] == (unsigned long long)L.drange;
  const bool kint = p.pkey.type == GHB_INT;
  const int64_t nunits = (p.n + UNIT - 1) / UNIT;
  for (int64_t u = ((int64_t)blockIdx.x * kJThreads + threadIdx.x) >> 5; u < nunits;
       u += (int64_t)gridDim.x * (kJThreads / 32)) {
    const int64_t row0 = u * UNIT + lane;
    int32_t s[kIt];
    if (!from_keys) {
#pragma unroll
      for (int k = 0; k < kIt; k++) s[k] = row0 + k * 32 < p.n ? __ldcs(p.slot_of_row + row0 + k * 32) : -1;
    } else {
      long long r[kIt];
#pragma unroll
      for (int k = 0; k < kIt; k++) {
        const int64_t row = row0 + k * 32;
        r[k] = 0;
        if (row < p.n)
          r[k] = kint ? (long long)__ldcs((const int*)p.pkey.data + row) : __ldcs((const long long*)p.pkey.data + row);
      }
#pragma unroll
      for (int k = 0; k < kIt; k++) {
        const int64_t row = row0 + k * 32;
        const unsigned long long d = (unsigned long long)r[k] - (unsigned long long)L.dmin;
        const bool hit = row < p.n && d < (unsigned long long)L.drange && !raw_is_null(p.pkey, r[k], row);
        s[k] = hit ? (int32_t)d : -1;
      }
      if (!full) {
#pragma unroll
        for (int k = 0; k < kIt; k++)
          if (s[k] >= 0 && p.meta[s[k]].y == 0) s[k] = -1;   // a hole of the key range
      }
    }
    int64_t at = p.chunk_count[u];   // this unit's offset
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      const ulonglong2 w = s[k] >= 0 && p.nbp > 0 ? p.payw[s[k]] : make_ulonglong2(0, 0);
      const unsigned bal = __ballot_sync(0xffffffffu, s[k] >= 0);
      const int64_t pos = at + __popc(bal & lt);
      at += __popc(bal);
      if (s[k] < 0) continue;
      if (pos >= p.cap) {
        raise_status(p.status, kDevCapacity);
        continue;
      }
      if (p.out_prow) __stcs(p.out_prow + pos, (int)row0 + k * 32 + p.prow_base);
#pragma unroll
      for (int j = 0; j < kInline; j++) {
        if (j >= p.nbp) break;
        const unsigned long long x = j == 0 ? w.x : w.y;
        if (p.bpay[j].type == GHB_INT) __stcs((int*)p.obp[j].data + pos, (int)x);
        else __stcs((unsigned long long*)p.obp[j].data + pos, x);
        if (p.obp[j].is_null) p.obp[j].is_null[pos] = 0;
      }
    }
  }
}

// Many output rows to a probe row: join_write_many_kernel writes them.  From two
// on, or from four without payloads, where there is little to write.  8M probe rows
// of 400k build rows, every key 2 / 3 / 4 times (1.8 / 2.7 / 3.6 output rows to a
// probe row), one probe and two build payloads: 626 / 965 / 1465 us by the general
// pass, - / 780 / 878 by this one; row ids alone 198 / 253 / 326 against - / 334 /
// 352; 5M rows of 1000, every key 8 times, row ids alone: 460 against 256.  The
// capacity bounds the output rows, so a call that cannot have as many does not
// launch it (4 us).
__host__ __device__ __forceinline__ int join_many_rows(const ProbeParams& p) { return p.nbp + p.npp > 0 ? 2 : 4; }
__host__ __device__ __forceinline__ bool join_may_be_many(const ProbeParams& p) {
  return p.cap / join_many_rows(p) >= p.n;
}
__device__ __forceinline__ bool join_many(const ProbeParams& p) {
  return join_may_be_many(p) && *p.d_out_rows >= join_many_rows(p) * p.n;
}

constexpr int kFewChains = 4;    // chains of a warp at most that it walks one after another
constexpr int kLongChain = 16;   // further rows of a chain that is worth it

// The write pass of every other join: any type, payloads and NULLs, duplicated
// build keys.  A warp's rows are written one output column at a time, the
// loads of a column issued before its stores; the further build rows of
// duplicated keys follow their chains, a thread's rows together, and a warp left
// with a few long chains walks each with all its lanes (2000 build rows of one
// key: 0.24 ms; a row a round 1.73, and 1.87 without the next row's index loaded
// ahead).  A LEFT OUTER
// probe of 8M rows over 400k spread keys (one in ten twice), one probe and two
// build payloads with NULL maps: 315 us when each row was written by an
// out-of-line loop over the columns, 179 at three CTAs per SM, 168 at four (64
// registers), 149 with the rows of a unique key told by a bit of the slot
// instead of a load of their count; five CTAs 192.  Bound by the latency and the
// requests of its gathers (DRAM 19 %).  One kernel that keeps a claimed range's
// slots in shared memory, looks back a range later and writes measured slower,
// here (449 us against 84 + 179 for the two passes) and for the lean write
// pass on 60M rows (634-687 us against 90 + 16 + 455): the barriers, claims and
// look-backs of a range cost more than reading the keys again.
template <int TH, int IT>
__global__ void __launch_bounds__(TH, TH == 128 ? 4 : 1024 / TH) join_write_kernel(const __grid_constant__ ProbeParams p) {
  static_assert(TH * IT == kChunk, "a CTA iteration covers one chunk");
  if (p.lean && p.out_brow == nullptr && p.stats[1] <= 1) return;   // join_write_lean_kernel's case
  if (join_many(p)) return;                                         // join_write_many_kernel's
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const bool unique = p.stats[1] <= 1;
  // the first build row itself is read or written
  const bool need_first = p.out_brow != nullptr || p.nbp > p.n_inline;
  __shared__ EmitDesc s_desc;
  load_emit_desc(p, &s_desc);
  // the next chunk's slots load while this chunk gathers and writes
  int32_t next_s[IT];
#pragma unroll
  for (int k = 0; k < IT; k++) {
    const int64_t row = (int64_t)blockIdx.x * kChunk + (int64_t)warp * (32 * IT) + k * 32 + lane;
    next_s[k] = row < p.n ? __ldcs(p.slot_of_row + row) : -2;
  }
  for (int64_t c = blockIdx.x; c < p.nchunks; c += gridDim.x) {
    const int64_t row0 = c * kChunk + (int64_t)warp * (32 * IT) + lane;
    int32_t slot[IT], mult[IT], first[IT];   // slot: -1 no match, -2 past the end
    bool dup[IT];                            // the key may have several build rows
    ulonglong2 w[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) {
      slot[k] = next_s[k];
      dup[k] = slot[k] >= 0 && (p.dup_bit == 0 || (slot[k] & p.dup_bit));
      if (slot[k] >= 0) slot[k] &= ~p.dup_bit;
      const int64_t nrow = row0 + (int64_t)gridDim.x * kChunk + k * 32;
      next_s[k] = nrow < p.n ? __ldcs(p.slot_of_row + nrow) : -2;
    }
#pragma unroll
    for (int k = 0; k < IT; k++) {
      first[k] = 0;
      mult[k] = slot[k] >= 0 ? 1 : 0;
      w[k] = make_ulonglong2(0, 0);
      if (slot[k] >= 0) {
        if (p.nbp > 0) w[k] = p.payw[slot[k]];
        if (need_first || (!unique && dup[k])) {
          const int2 m = p.meta[slot[k]];
          first[k] = m.x;
          mult[k] = m.y;
        }
      }
    }
    int64_t pos[IT];              // from the warp's offset on
    int64_t running = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
      if (slot[k] != -2) mult[k] = out_rows_of(p.join_type, mult[k]);
      uint32_t incl, total;
      if (__all_sync(0xffffffffu, mult[k] <= 1)) {
        const unsigned bal = __ballot_sync(0xffffffffu, mult[k] == 1);
        incl = __popc(bal & ((2u << lane) - 1u));
        total = __popc(bal);
      } else {
        incl = (uint32_t)mult[k];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        total = __shfl_sync(0xffffffffu, incl, 31);
      }
      pos[k] = running + incl - (uint32_t)mult[k];
      running += total;
    }
    const int64_t wpos = p.chunk_count[c * (TH / 32) + warp];   // this warp's offset
    uint32_t live = 0, hit = 0;   // bit k: row k has output, and a build row
#pragma unroll
    for (int k = 0; k < IT; k++) {
      if (mult[k] > 0) {
        if (wpos + pos[k] + mult[k] <= p.cap) live |= 1u << k;
        else raise_status(p.status, kDevCapacity);
      }
      if (slot[k] >= 0 && p.join_type != GHB_LEFT_SEMI_JOIN) hit |= 1u << k;
    }
    hit &= live;
#pragma unroll
    for (int k = 0; k < IT; k++) first[k]--;   // the build row
    auto item = [&](int k) -> int64_t { return row0 + k * 32; };
    emit_rows<IT, true>(s_desc, p.n_inline, live, hit, wpos, pos, item, first, w);
    if (unique) continue;
    // the further build rows of the threads' keys, a row of each chain a round
    uint32_t more = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
      if (!(hit >> k & 1) || mult[k] <= 1) continue;
      more |= 1u << k;
      first[k] = p.chain_p1[slot[k]] - 1;
    }
    for (int j = 1;; j++) {
      int chains = __reduce_add_sync(0xffffffffu, __popc(more));
      while (chains > 0 && chains <= kFewChains) {
        // the longest, when it is long: the warp walks it 32 rows at a time and writes
        // those together (a row a round would pay every wait of a round for it)
        int k0 = 0, left = 0;
#pragma unroll
        for (int k = 0; k < IT; k++)
          if (more >> k & 1 && mult[k] - j > left) {
            left = mult[k] - j;
            k0 = k;
          }
        const int longest = __reduce_max_sync(0xffffffffu, left);
        if (longest < kLongChain) break;
        const int src = __ffs(__ballot_sync(0xffffffffu, left == longest)) - 1;
        int32_t cur = 0;
        int64_t at = 0;
#pragma unroll
        for (int k = 0; k < IT; k++)
          if (k == k0) {
            cur = first[k];
            at = pos[k];
          }
        cur = __shfl_sync(0xffffffffu, cur, src);
        at = wpos + __shfl_sync(0xffffffffu, (long long)at, src) + 1;
        const int64_t row = row0 - lane + src + 32 * __shfl_sync(0xffffffffu, k0, src);
        for (int done = 0; done < longest; done += 32) {
          int32_t one[1] = {0};
          const int m = min(32, longest - done);
          for (int i = 0; i < m; i++) {   // cur: further row done + i
            if (lane == i) one[0] = cur;
            if (done + i + 1 < longest) cur = p.next_p1[cur] - 1;
          }
          const int64_t here[1] = {at + done + lane};
          const ulonglong2 none[1] = {};
          const uint32_t mine = lane < m ? 1u : 0u;
          emit_rows<1, false>(s_desc, p.n_inline, mine, mine, 0, here, [&](int) -> int64_t { return row; }, one, none);
        }
        if (lane == src) more &= ~(1u << k0);
        chains--;
      }
      if (chains == 0) break;
      int32_t next[IT];   // on its way while this row is gathered and written
      uint32_t on = 0;
#pragma unroll
      for (int k = 0; k < IT; k++) {
        pos[k]++;
        on |= (more >> k & 1 && j + 1 < mult[k] ? 1u : 0u) << k;
        next[k] = on >> k & 1 ? p.next_p1[first[k]] : 0;
      }
      emit_rows<IT, false>(s_desc, p.n_inline, more, more, wpos, pos, item, first, w);
#pragma unroll
      for (int k = 0; k < IT; k++) first[k] = next[k] - 1;
      more = on;
    }
  }
}

constexpr int kManyTile = 256;   // output rows a warp puts in order at a time
constexpr int kManyStep = 3;     // of each key, as a power of two, when 32 keys have that many

// The write pass where build rows are many to a probe row.  A warp takes 32 probe
// rows, a lane each; every lane walks its key's chain for eight build rows
// (up to 32 when few chains are left) and lists them in shared memory, and the
// warp writes the listed rows side by side, so that the rows of a key fill whole
// sectors of the output columns.  UNIT: the probe rows of one count.
//
// 2M probe rows of 100,000 build rows, every key 16 times (29M output rows): 0.42
// ms with one build payload, 0.83 with two of them and two of the probe's, NULL maps
// among them.  By the general pass, whose rounds write one row of 128 keys each, a
// part of as many sectors per column, 1.59 and 3.94 ms (1.02 and 3.05 when each
// thread wrote one key's rows at a time).  Four rows of each key at a time instead of
// eight: the same.
template <int UNIT>
__global__ void __launch_bounds__(kJThreads, 4) join_write_many_kernel(const __grid_constant__ ProbeParams p) {
  if (!join_many(p)) return;
  constexpr int kIt = UNIT / 32, kWarps = kJThreads / 32;
  __shared__ EmitDesc s_desc;
  __shared__ int32_t s_brow[kWarps][kManyTile];   // listed build rows (-1: none), a chain's together
  __shared__ int64_t s_pos[kWarps][32];           // per chain: output row of its first listed
  __shared__ int32_t s_cnt[kWarps][32];           // listed rows
  __shared__ uint8_t s_lane[kWarps][32];          // probe row
  load_emit_desc(p, &s_desc);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  int32_t* brow = s_brow[warp];
  const int64_t nwork = (p.n + 31) / 32;
  for (int64_t q = (int64_t)blockIdx.x * kWarps + warp; q < nwork; q += (int64_t)gridDim.x * kWarps) {
    // the unit's rows up to this one's 32: their output rows come before
    const int64_t unit = q / kIt;
    const int item = (int)(q % kIt);
    int64_t pos = p.chunk_count[unit], before = 0;
    int32_t slot = -1, left = 0, cur = 0;   // cur: build row + 1, 0 none
#pragma unroll
    for (int k = 0; k < kIt; k++) {
      if (k > item) break;
      const int64_t row = unit * UNIT + k * 32 + lane;
      const int32_t s = row < p.n ? p.slot_of_row[row] : -2;
      slot = s >= 0 ? s & ~p.dup_bit : s;
      int2 m = make_int2(0, 0);
      if (s >= 0 && (k == item || p.dup_bit == 0 || (s & p.dup_bit))) m = p.meta[slot];
      else if (s >= 0) m.y = 1;
      if (k < item) before += s != -2 ? out_rows_of(p.join_type, m.y) : 0;
      left = s != -2 ? out_rows_of(p.join_type, m.y) : 0;
      cur = m.x;
    }
    int64_t incl = left;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xffffffffu, (long long)incl, o);
      before += __shfl_xor_sync(0xffffffffu, (long long)before, o);
      if (lane >= o) incl += t;
    }
    pos += before + incl - left;
    const int64_t row0 = unit * UNIT + item * 32;
    while (true) {
      const unsigned act = __ballot_sync(0xffffffffu, left > 0);
      if (!act) break;
      const int longest = __reduce_max_sync(0xffffffffu, left);
      const int chains = __popc(act);
      int sh = kManyStep;   // rows listed of a chain, as a power of two
      while (sh > 0 && longest <= 1 << (sh - 1)) sh--;
      while (sh < 5 && longest > 1 << sh && chains << (sh + 1) <= kManyTile) sh++;
      if (left > 0) {
        const int r = __popc(act & lt), cnt = min(1 << sh, left);
        s_pos[warp][r] = pos;
        s_cnt[warp][r] = cnt;
        s_lane[warp][r] = (uint8_t)lane;
        for (int i = 0; i < cnt; i++) {
          brow[(r << sh) + i] = cur - 1;
          if (--left > 0) {
            cur = slot >= 0 ? p.chain_p1[slot] : p.next_p1[cur - 1];
            slot = -1;   // the chain's head is taken once
          }
        }
        pos += cnt;
      }
      __syncwarp();
      for (int e = lane; e < chains << sh; e += 128) {
        int32_t b[4], f[4];
        int64_t at[4];
        const ulonglong2 none[4] = {};
        uint32_t in = 0, hit = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int x = e + 32 * k, r = x >> sh, i = x & ((1 << sh) - 1);
          const bool mine = x < chains << sh && i < s_cnt[warp][r];
          b[k] = mine ? brow[x] : -1;
          at[k] = mine ? s_pos[warp][r] + i : 0;
          f[k] = mine ? s_lane[warp][r] : 0;
          if (mine && at[k] >= p.cap) raise_status(p.status, kDevCapacity);
          else in |= (mine ? 1u : 0u) << k;
          hit |= (b[k] >= 0 ? 1u : 0u) << k;
        }
        emit_rows<4, false>(s_desc, p.n_inline, in, hit & in, 0, at, [&](int k) -> int64_t { return row0 + f[k]; }, b,
                            none);
      }
      __syncwarp();   // the lists are the next rows'
    }
  }
}

static int64_t next_pow2(int64_t v) {
  int64_t p = 1;
  while (p < v) p <<= 1;
  return p;
}

// Tables holding an L2 persistence window, per device (`delta` added under a
// lock; returns the new count).
static int l2_window_count(int device, int delta) {
  static std::mutex mu;
  static std::map<int, int> count;
  std::lock_guard<std::mutex> lock(mu);
  return count[device] += delta;
}

int32_t join_build_impl(ghb_ctx* ctx, const ghb_column* build_key, const ghb_column* build_payload,
                        int32_t nbp, const ghb_join_cfg* cfg, ghb_join_table** out,
                        cudaStream_t stream) {
  if (!out) return set_error(ctx, GHB_ERR_INVALID, "out is NULL");
  *out = nullptr;
  int32_t st = validate_columns(ctx, build_key, 1, nullptr);
  if (st) return st;
  if (build_key->type == GHB_DOUBLE)
    return set_error(ctx, GHB_ERR_UNSUPPORTED, "join keys must be LONG or INT");
  if (build_key->n >= INT32_MAX / 2)
    return set_error(ctx, GHB_ERR_UNSUPPORTED, "build side of 2^30 rows or more");
  if (nbp < 0 || nbp > kMaxPay || (nbp > 0 && !build_payload))
    return set_error(ctx, GHB_ERR_INVALID, "n_build_payload=%d outside [0,%d]", nbp, kMaxPay);
  for (int j = 0; j < nbp; j++) {
    if ((st = validate_columns(ctx, &build_payload[j], 1, nullptr))) return st;
    if (build_payload[j].n != build_key->n)
      return set_error(ctx, GHB_ERR_INVALID, "build payload %d has %lld rows, the key %lld", j,
                       (long long)build_payload[j].n, (long long)build_key->n);
  }
  float lf = (cfg && cfg->load_factor > 0.f && cfg->load_factor < 0.95f) ? cfg->load_factor : 0.5f;
  int64_t nb = next_pow2(std::max<int64_t>(16, (int64_t)((double)build_key->n / (4.0 * lf)) + 1));
  ghb_join_table* t = new ghb_join_table();
  t->slots = nb * 4;
  t->build_rows = build_key->n;
  t->key_type = build_key->type;
  t->nbp = nbp;
  for (int j = 0; j < nbp; j++) t->pay[j] = build_payload[j];
  // payloads copied into the slots: the first two non-BYTEMAP columns
  t->n_inline = 0;
  while (t->n_inline < std::min(nbp, kInline) && build_payload[t->n_inline].null_mode != GHB_NULLS_BYTEMAP)
    t->n_inline++;
  const size_t slots = (size_t)(nb + 1) * 4;   // hashed buckets + the side bucket
  auto a256 = [](size_t b) { return (b + 255) & ~(size_t)255; };
  const size_t key_bytes = a256(slots * 8), meta_bytes = a256(slots * 8), pay_bytes = a256(slots * 16);
  size_t bucket_bytes = key_bytes + meta_bytes + pay_bytes;
  size_t chain_bytes = a256(slots * 4);
  size_t next_bytes = a256((size_t)std::max<int64_t>(build_key->n, 1) * 4);
  size_t bytes = bucket_bytes + chain_bytes + next_bytes + 256;
  // stream-ordered allocation: no device-wide sync, and the pool keeps the
  // memory for the next build on this device
  t->stream = stream;
  if (cfg && cfg->block_threads > 0) t->probe_threads = cfg->block_threads;
  if (cudaMallocAsync(&t->alloc, bytes, stream) != cudaSuccess) {
    cudaGetLastError();
    delete t;
    return set_error(ctx, GHB_ERR_OOM, "cannot allocate a %zu-byte join table", bytes);
  }
  t->alloc_bytes = bytes;
  t->kimg = (unsigned long long*)t->alloc;
  t->meta = (int2*)((char*)t->alloc + key_bytes);
  t->payw = (ulonglong2*)((char*)t->alloc + key_bytes + meta_bytes);
  t->chain = (int32_t*)((char*)t->alloc + bucket_bytes);
  t->next = (int32_t*)((char*)t->alloc + bucket_bytes + chain_bytes);
  t->d_stats = (unsigned long long*)((char*)t->alloc + bucket_bytes + chain_bytes + next_bytes);
  // join_clear_kernel zeroes the table's arrays; without a build row nothing
  // chooses a layout, and the hashed one's are cleared here
  if (cudaMemsetAsync(t->d_stats, 0, 256, stream) != cudaSuccess ||
      (build_key->n == 0 && (cudaMemsetAsync(t->alloc, 0, key_bytes + meta_bytes, stream) != cudaSuccess ||
                             cudaMemsetAsync(t->chain, 0, chain_bytes, stream) != cudaSuccess))) {
    cudaFreeAsync(t->alloc, stream);
    delete t;
    return set_error(ctx, GHB_ERR_CUDA, "memset of the join table failed");
  }
  BuildParams p;
  std::memset(&p, 0, sizeof(p));
  p.key = *build_key;
  p.n_inline = t->n_inline;
  for (int j = 0; j < t->n_inline; j++) p.pay[j] = build_payload[j];
  p.kimg = t->kimg;
  p.meta = t->meta;
  p.payw = t->payw;
  p.chain_p1 = t->chain;
  p.next_p1 = t->next;
  p.bmask = nb - 1;
  p.hshift = 64 - __builtin_ctzll((unsigned long long)nb);
  p.side = nb;
  p.stats = t->d_stats;
  p.status = ctx->d_status;
  p.slots = nb * 4;
  if (build_key->n > 0) {
    int grid = (int)std::min<int64_t>((build_key->n + 255) / 256, (int64_t)ctx->num_sms * 8);
    join_key_range_kernel<<<grid, 256, 0, stream>>>(*build_key, t->d_stats);
    ctx->launches++;
    const int cgrid = (int)std::min<int64_t>((nb + 256) / 256, (int64_t)ctx->num_sms * 8);
    join_clear_kernel<<<cgrid, 256, 0, stream>>>(p);
    ctx->launches++;
    join_build_kernel<<<grid, 256, 0, stream>>>(p);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
      cudaFreeAsync(t->alloc, stream);
      delete t;
      return set_error(ctx, GHB_ERR_CUDA, "join build launch failed: %s", cudaGetErrorString(e));
    }
  }
  if (cfg && cfg->l2_persist) {
    int max_persist = 0;
    cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, ctx->device);
    if (max_persist > 0) {
      cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, (size_t)max_persist);
      cudaStreamAttrValue attr;
      std::memset(&attr, 0, sizeof(attr));
      attr.accessPolicyWindow.base_ptr = t->alloc;
      attr.accessPolicyWindow.num_bytes = std::min(bucket_bytes, (size_t)max_persist);
      attr.accessPolicyWindow.hitRatio = 1.0f;
      attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
      attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
      cudaStreamSetAttribute(stream, cudaStreamAttributeAccessPolicyWindow, &attr);
      t->l2_window = true;
      t->device = ctx->device;
      l2_window_count(ctx->device, +1);
    }
  }
  *out = t;
  return GHB_OK;
}

// Scratch one probe of n rows needs (slot per row, count per chunk).
size_t join_probe_scratch_bytes(int64_t n) {
  int64_t nchunks = (n + kChunk - 1) / kChunk;
  // a count per warp of each chunk: 16 warps at most (512-thread CTAs)
  return (((size_t)std::max<int64_t>(n, 1) * 4 + 255) & ~(size_t)255) +
         (((size_t)std::max<int64_t>(nchunks, 1) * 16 * 8 + 255) & ~(size_t)255) + 512;
}

int32_t scan_counts(ghb_ctx* ctx, int64_t* counts, int64_t n, int64_t* d_total, cudaStream_t stream) {
  if (n <= 4096) {
    join_scan_kernel<<<1, 1024, 0, stream>>>(counts, n, d_total);
  } else {
    ScanParams sp;
    sp.counts = counts;
    sp.n = n;
    sp.ntiles = (n + 1023) / 1024;
    sp.d_total = d_total;
    const int32_t st = lookback_prepare(ctx, sp.ntiles, &sp.epoch, stream);
    if (st) return st;
    sp.lb = ctx->lb_status;
    sp.counters = ctx->d_counters;
    sp.status = ctx->d_status;
    sp.spin_limit = ctx->spin_limit;
    const int sgrid = (int)std::min<int64_t>(sp.ntiles, (int64_t)ctx->num_sms);
    join_scan_lb_kernel<<<sgrid, 1024, 0, stream>>>(sp);
  }
  GHB_LAUNCH_CHECK(ctx);
  return GHB_OK;
}

int32_t join_probe_impl(ghb_ctx* ctx, const ghb_join_table* t, const ghb_column* probe_key,
                        int32_t join_type, ghb_out_column* out_build, const ghb_column* probe_payload,
                        int32_t npp, ghb_out_column* out_probe, int32_t* out_probe_rowid,
                        int32_t* out_build_rowid, int64_t out_capacity, int64_t* d_out_rows,
                        cudaStream_t stream, int32_t prow_base) {
  if (!t) return set_error(ctx, GHB_ERR_INVALID, "table is NULL");
  int32_t st = validate_columns(ctx, probe_key, 1, nullptr);
  if (st) return st;
  if (probe_key->type == GHB_DOUBLE)
    return set_error(ctx, GHB_ERR_UNSUPPORTED, "join keys must be LONG or INT");
  if (probe_key->n >= INT32_MAX)
    return set_error(ctx, GHB_ERR_UNSUPPORTED, "probe side above 2^31-1 rows per call");
  if (join_type != GHB_INNER_JOIN && join_type != GHB_LEFT_SEMI_JOIN && join_type != GHB_LEFT_OUTER_JOIN)
    return set_error(ctx, GHB_ERR_UNSUPPORTED, "join type %d", join_type);
  if (npp < 0 || npp > kMaxPay)
    return set_error(ctx, GHB_ERR_INVALID, "n_probe_payload=%d outside [0,%d]", npp, kMaxPay);
  if (!d_out_rows) return set_error(ctx, GHB_ERR_INVALID, "d_out_rows is NULL");
  if (t->nbp > 0 && !out_build) return set_error(ctx, GHB_ERR_INVALID, "out_build is NULL");
  ProbeParams p;
  std::memset(&p, 0, sizeof(p));
  for (int j = 0; j < t->nbp; j++) {
    if (out_build[j].type != t->pay[j].type || !out_build[j].data)
      return set_error(ctx, GHB_ERR_INVALID, "build payload output %d: bad type or data", j);
    p.bpay[j] = t->pay[j];
    p.obp[j] = out_build[j];
  }
  for (int j = 0; j < npp; j++) {
    if ((st = validate_columns(ctx, &probe_payload[j], 1, nullptr))) return st;
    if (probe_payload[j].n != probe_key->n)
      return set_error(ctx, GHB_ERR_INVALID, "probe payload %d row count differs from the key", j);
    if (out_probe[j].type != probe_payload[j].type || !out_probe[j].data)
      return set_error(ctx, GHB_ERR_INVALID, "probe payload output %d: bad type or data", j);
    p.ppay[j] = probe_payload[j];
    p.opp[j] = out_probe[j];
  }
  p.kimg = t->kimg;
  p.meta = t->meta;
  p.payw = t->payw;
  p.chain_p1 = t->chain;
  p.next_p1 = t->next;
  p.stats = t->d_stats;
  p.bmask = t->slots / 4 - 1;
  p.hshift = 64 - __builtin_ctzll((unsigned long long)(t->slots / 4));
  p.side = t->slots / 4;
  p.build_rows = t->build_rows;
  p.slots = t->slots;
  p.pkey = *probe_key;
  p.join_type = join_type;
  p.nbp = t->nbp;
  p.npp = npp;
  p.n_inline = t->n_inline;
  p.lean = join_type == GHB_INNER_JOIN && npp == 0 && t->nbp == t->n_inline;
  for (int j = 0; j < t->n_inline && p.lean; j++) p.lean = t->pay[j].null_mode == GHB_NULLS_NONE;
  p.out_prow = out_probe_rowid;
  p.out_brow = out_build_rowid;
  p.prow_base = prow_base;
  p.n = probe_key->n;
  p.nchunks = (p.n + kChunk - 1) / kChunk;
  p.cap = out_capacity;
  p.d_out_rows = d_out_rows;
  p.status = ctx->d_status;
  if (p.nchunks == 0) {
    GHB_CUDA_TRY(ctx, cudaMemsetAsync(d_out_rows, 0, sizeof(int64_t), stream));
    return GHB_OK;
  }
  // CTA shape (threads x rows per thread, one 1024-row chunk either way),
  // chosen by the build's ghb_join_cfg.block_threads
  const int threads = t->probe_threads == 128 || t->probe_threads == 512 ? t->probe_threads : 256;
  const int64_t nunits = p.nchunks * (threads / 32);   // a count per warp of each chunk
  if ((st = scratch_alloc(ctx, (size_t)p.n * 4, (void**)&p.slot_of_row, stream))) return st;
  if ((st = scratch_alloc(ctx, (size_t)nunits * 8, (void**)&p.chunk_count, stream))) return st;
  const bool kint = probe_key->type == GHB_INT, knull = probe_key->null_mode != GHB_NULLS_NONE;
  void (*count_kernel)(ProbeParams) = nullptr;
  void (*write_kernel)(ProbeParams) = nullptr;
  void (*write_lean)(ProbeParams) = nullptr;
  void (*count_direct)(ProbeParams) = nullptr;
  void (*write_many)(ProbeParams) = nullptr;
#define GHB_COUNT(TH, IT)                                                                   \
  count_kernel = kint ? (knull ? join_count_kernel<TH, IT, true, true> : join_count_kernel<TH, IT, true, false>) \
                      : (knull ? join_count_kernel<TH, IT, false, true> : join_count_kernel<TH, IT, false, false>); \
  count_direct = kint ? (knull ? join_count_direct_kernel<TH, IT, true, true> : join_count_direct_kernel<TH, IT, true, false>) \
                      : (knull ? join_count_direct_kernel<TH, IT, false, true> : join_count_direct_kernel<TH, IT, false, false>); \
  write_kernel = join_write_kernel<TH, IT>;                                                  \
  write_lean = join_write_lean_kernel<32 * IT>;                                              \
  write_many = join_write_many_kernel<32 * IT>
  if (threads == 128) { GHB_COUNT(128, 8); }
  else if (threads == 512) { GHB_COUNT(512, 2); }
  else { GHB_COUNT(256, 4); }
#undef GHB_COUNT
  p.dup_bit = t->slots + 4 <= (1ll << 30) ? 1 << 30 : 0;
  int per_sm = 0;
  if ((st = resident_ctas(ctx, (const void*)count_kernel, threads, 0, &per_sm))) return st;
  int grid = (int)std::min<int64_t>(p.nchunks, (int64_t)ctx->num_sms * std::max(1, per_sm));
  count_kernel<<<grid, threads, 0, stream>>>(p);
  GHB_LAUNCH_CHECK(ctx);
  // the count pass of a direct table (the build decided on the device which one works)
  if ((st = resident_ctas(ctx, (const void*)count_direct, threads, 0, &per_sm))) return st;
  grid = (int)std::min<int64_t>(p.nchunks, (int64_t)ctx->num_sms * std::max(1, per_sm));
  count_direct<<<grid, threads, 0, stream>>>(p);
  GHB_LAUNCH_CHECK(ctx);
  if ((st = scan_counts(ctx, p.chunk_count, nunits, d_out_rows, stream))) return st;
  if ((st = resident_ctas(ctx, (const void*)write_kernel, threads, 0, &per_sm))) return st;
  grid = (int)std::min<int64_t>(p.nchunks, (int64_t)ctx->num_sms * std::max(1, per_sm));
  write_kernel<<<grid, threads, 0, stream>>>(p);
  GHB_LAUNCH_CHECK(ctx);
  if (join_may_be_many(p)) {   // the write pass of many build rows to a probe row, when the count pass finds them
    if ((st = resident_ctas(ctx, (const void*)write_many, kJThreads, 0, &per_sm))) return st;
    grid = (int)std::min<int64_t>((p.n + kJThreads - 1) / kJThreads, (int64_t)ctx->num_sms * std::max(1, per_sm));
    write_many<<<grid, kJThreads, 0, stream>>>(p);
    GHB_LAUNCH_CHECK(ctx);
  }
  if (p.lean && !p.out_brow) {   // the lean write pass, when the build's keys turn out unique
    if ((st = resident_ctas(ctx, (const void*)write_lean, kJThreads, 0, &per_sm))) return st;
    grid = (int)std::min<int64_t>((nunits * 32 + kJThreads - 1) / kJThreads, (int64_t)ctx->num_sms * std::max(1, per_sm));
    write_lean<<<grid, kJThreads, 0, stream>>>(p);
  }
  GHB_LAUNCH_CHECK(ctx);
  return GHB_OK;
}

}  // namespace ghb

using namespace ghb;

extern "C" {

int32_t ghb_join_build(ghb_ctx* ctx, const ghb_column* build_key, const ghb_column* build_payload,
                       int32_t n_build_payload, const ghb_join_cfg* cfg, ghb_join_table** out,
                       void* stream) {
  if (!ctx) return GHB_ERR_INVALID;
  CallScope cs(ctx, "join_build", (cudaStream_t)stream);
  cs.rows(build_key ? build_key->n : 0);
  cs.bytes(cols_bytes(build_key, build_key ? 1 : 0) + cols_bytes(build_payload, n_build_payload));
  return cs.done(join_build_impl(ctx, build_key, build_payload, n_build_payload, cfg, out,
                                 (cudaStream_t)stream));
}

int32_t ghb_join_table_free(ghb_ctx* ctx, ghb_join_table* table) {
  if (!ctx || !table) return GHB_ERR_INVALID;
  if (table->l2_window) {
    cudaStreamSynchronize(table->stream);
    // the build stream's window, if it still points at this table, goes
    cudaStreamAttrValue attr;
    std::memset(&attr, 0, sizeof(attr));
    if (cudaStreamGetAttribute(table->stream, cudaStreamAttributeAccessPolicyWindow, &attr) == cudaSuccess &&
        attr.accessPolicyWindow.base_ptr == table->alloc) {
      std::memset(&attr, 0, sizeof(attr));
      cudaStreamSetAttribute(table->stream, cudaStreamAttributeAccessPolicyWindow, &attr);
    }
    cudaGetLastError();
    // the persisting carve-out is shared by every resident table of the
    // device: it is released with the last table that holds a window
    if (l2_window_count(table->device, -1) == 0) {
      cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, 0);
      cudaCtxResetPersistingL2Cache();
    }
  }
  // released in the order of the build stream: probes issued on that stream
  // before this call finish first; probes on other streams must be ordered
  // before it by the caller
  if (table->alloc) cudaFreeAsync(table->alloc, table->stream);
  delete table;
  return GHB_OK;
}

int32_t ghb_join_table_info(ghb_ctx* ctx, const ghb_join_table* table, int64_t* rows,
                            int64_t* max_dup, int64_t* slots) {
  if (!ctx || !table) return GHB_ERR_INVALID;
  unsigned long long st[5] = {0, 0, 0, 0, 0};
  GHB_CUDA_TRY(ctx, cudaMemcpy(st, table->d_stats, sizeof(st), cudaMemcpyDeviceToHost));
  if (rows) *rows = (int64_t)st[0];
  if (max_dup) *max_dup = (int64_t)st[1];
  // a direct table reports its key range as its slots
  const JoinLayout L = join_layout(st, table->build_rows, table->slots);
  if (slots) *slots = L.direct ? L.drange : table->slots;
  return GHB_OK;
}

int32_t ghb_join_probe(ghb_ctx* ctx, const ghb_join_table* table, const ghb_column* probe_key,
                       int32_t join_type, ghb_out_column* out_build, const ghb_column* probe_payload,
                       int32_t n_probe_payload, ghb_out_column* out_probe, int32_t* out_probe_rowid,
                       int32_t* out_build_rowid, int64_t out_capacity, int64_t* d_out_rows,
                       void* stream) {
  if (!ctx) return GHB_ERR_INVALID;
  CallScope cs(ctx, "join_probe", (cudaStream_t)stream);
  int64_t n = probe_key ? probe_key->n : 0;
  cs.rows(n);
  cs.bytes(cols_bytes(probe_key, probe_key ? 1 : 0) + cols_bytes(probe_payload, n_probe_payload));
  scratch_reset(ctx);
  int32_t st = scratch_reserve(ctx, join_probe_scratch_bytes(n), (cudaStream_t)stream);
  if (st) return cs.done(st);
  return cs.done(join_probe_impl(ctx, table, probe_key, join_type, out_build, probe_payload, n_probe_payload,
                                 out_probe, out_probe_rowid, out_build_rowid, out_capacity, d_out_rows,
                                 (cudaStream_t)stream, 0));
}

}  // extern "C"
