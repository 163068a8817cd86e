// ghb_sort.cu — stable ORDER BY sort (S1): LSD radix sort on packed keys.
//
// Replaces the Sink sort of the reference (gpu_impl/src/Operator/
// SinkOperator.cu:153-286: H2D of the key columns, thrust::sort of row
// indices with an indirect multi-column comparator, D2H of the index, host
// gather of every column).  The order is Hive's BinarySortable order
// (BinarySortableSerDe.java:921-960 and the null markers at :195-220):
// integers by signed value, doubles by IEEE total order, per key ASC/DESC and
// NULLS FIRST/LAST; ties keep input order (LSD radix sort is stable).
//
// Pipeline (one call):
//   1. analyse   one read of the key columns: per key the min/max of its
//                order image and whether it holds NULLs; and a sample of the
//                packed keys: how many rows share their leading digits;
//   2. plan      (host) each key becomes sub-fields [null flag][value - min]
//                of just the width its range needs, packed least-significant
//                key first into 64-bit segments; and how many leading digits
//                the radix passes sort by;
//   3. histogram one read per segment: 8-bit digit histograms of all of the
//                segment's passes at once; when every digit is sorted by,
//                passes whose digit is constant are skipped;
//   4. passes    onesweep-style: each CTA claims a tile, ranks its keys by
//                digit within each warp (stable: a lane's peers of an item
//                from one shared atomicOr per lane), gets each digit's global
//                offset by decoupled look-back over earlier tiles, reorders
//                the tile in shared memory and writes one run per digit;
//   5. finish    a one-segment key whose leading digits already set all but a
//                few rows apart is sorted by those digits only; the finish
//                puts the rows of each run of equal leading digits in order
//                (each row counts the rows of its run before it, in shared
//                memory) and writes the output columns in order.
// A one-segment key (the common case, e.g. (int32 d, int64 k) with the ranges
// of the sort workload) is packed by the histogram kernel from the user's
// columns and unpacked by the finish, or the last pass, into the output columns; the
// value carried with it is the single payload column, or the row index.  A
// key wider than 64 bits is sorted segment by segment (least significant
// first), each later segment packed from the row order the previous one left,
// and the output is gathered by the final row order.
#include <algorithm>
#include <vector>

#include "ghb_ctx.hpp"
#include "ghb_log.hpp"
#include "ghb_range.cuh"

namespace ghb {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;   // 4096
constexpr int kDigitBits = 8;
constexpr int kBins = 1 << kDigitBits;
constexpr int kMaxPasses = 8;                          // per 64-bit segment
constexpr int kMaxSortKeys = 8;
constexpr int kMaxSortPay = 8;
constexpr int kMaxSub = 2 * kMaxSortKeys;
constexpr int kMaxSeg = kMaxSub;

struct KeyField {
  ghb_column col;
  int32_t desc;
  int32_t nulls_first;
  int32_t has_null;      // the column holds NULLs: the key has a flag sub-field
  int32_t vbits;         // value bits
  uint64_t umin;         // min of the (possibly inverted) order image
};

struct SubField {
  int8_t key;
  int8_t is_flag;        // 1: the NULL flag, 0: the value bits
  int8_t bits;
  int8_t shift;          // within the segment word
};

struct Segment {
  int32_t n;
  int32_t bits;
  SubField f[kMaxSub];
};

struct KeySet {
  int32_t nkeys;
  KeyField k[kMaxSortKeys];
};

__device__ __forceinline__ uint64_t key_image(const ghb_column& c, int64_t raw) {
  return c.type == GHB_DOUBLE ? flip_f64_bits((uint64_t)raw) : flip_i64(raw);
}

// Contribution of one sub-field for row r (value already shifted into place).
__device__ __forceinline__ uint64_t sub_bits(const KeySet& K, const SubField& sf, int64_t r) {
  const KeyField& kf = K.k[sf.key];
  int64_t raw = ld_raw(kf.col, r);
  bool null = kf.has_null && raw_is_null(kf.col, raw, r);
  uint64_t v;
  if (sf.is_flag) {
    v = (null == (bool)kf.nulls_first) ? 0 : 1;   // NULLS FIRST: null 0 / value 1
  } else {
    uint64_t u = key_image(kf.col, raw);
    if (kf.desc) u = ~u;
    v = null ? 0 : u - kf.umin;
  }
  return v << sf.shift;
}

// ---------------------------------------------------------------- analyse
struct MinMaxParams {
  KeySet K;
  int64_t n;
  unsigned long long* out;  // per key: [0] max of ~image (~min), [1] max image, [2] any NULL; zeroed
};

// Reads the key columns once, one after another: (d int32, k int64) of 60M
// rows 191 us when each value went through its order image, 107 now (minima on
// the values themselves, eight 16-byte loads in flight).
__global__ void __launch_bounds__(256) sort_minmax_kernel(const __grid_constant__ MinMaxParams p) {
  for (int j = 0; j < p.K.nkeys; j++) range_to(p.K.k[j].col, p.n, p.K.k[j].desc, p.out + 3 * j);
}

// ---------------------------------------------------------------- sample
// Ordered pairs of sampled rows whose packed keys share their leading q
// digits, for q = first..8 (pairs[q]): each CTA packs S random rows' keys (the
// ranges are on the device already) into shared memory and compares 64 of them
// with all.  pairs[q] / S^2 is the chance that two rows share a run of equal
// leading digits.  Of a key wider than 64 bits the leading 64 are sampled.
constexpr int kSampleMax = 2048;
constexpr int kSampleRows = 64;   // rows a CTA compares with all

struct SampleParams {
  KeySet K;
  int64_t n;
  int32_t S;               // rows sampled: 1024 or 2048
  int32_t first;           // fewest leading digits worth counting, at most 4
  const unsigned long long* mm;
  unsigned long long* pairs;   // [9], zeroed
};

__global__ void __launch_bounds__(256) sort_sample_kernel(const __grid_constant__ SampleParams p) {
  __shared__ uint64_t s_key[kSampleMax];
  __shared__ __align__(16) uint32_t s_hi[kSampleMax];   // the keys' upper halves
  __shared__ uint64_t s_umin[kMaxSortKeys];
  __shared__ int s_vshift[kMaxSortKeys], s_fshift[kMaxSortKeys], s_total;
  __shared__ unsigned int s_pairs[9];
  if (threadIdx.x < 9) s_pairs[threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    int bits = 0;
    for (int j = p.K.nkeys - 1; j >= 0; j--) {
      uint64_t range;
      key_range(p.mm + 3 * j, &s_umin[j], &range);
      s_vshift[j] = bits;
      bits += range == 0 ? 0 : 64 - __clzll((long long)range);
      s_fshift[j] = p.mm[3 * j + 2] ? bits++ : -1;
    }
    s_total = bits;
  }
  __syncthreads();
  const int total = s_total;
  if (total <= 8 * p.first) return;
  const int cut = max(0, total - 64);   // a wider key: its leading 64 bits
  constexpr int U = 4;
  for (int base = threadIdx.x; base < p.S; base += U * blockDim.x) {   // S is a multiple of U * blockDim.x
    int64_t row[U];
    uint64_t k[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      row[u] = (int64_t)__umul64hi(mix64((uint64_t)(base + u * blockDim.x) + 1), (uint64_t)p.n);
      k[u] = 0;
    }
    for (int j = 0; j < p.K.nkeys; j++) {
      const KeyField& f = p.K.k[j];
      int64_t raw[U];
#pragma unroll
      for (int u = 0; u < U; u++) raw[u] = ld_raw(f.col, row[u]);
#pragma unroll
      for (int u = 0; u < U; u++) {
        const bool null = f.col.null_mode != GHB_NULLS_NONE && raw_is_null(f.col, raw[u], row[u]);
        uint64_t v = key_image(f.col, raw[u]);
        if (f.desc) v = ~v;
        const int at = s_vshift[j] - cut;
        if (!null && at > -64 && at < 64) k[u] |= at >= 0 ? (v - s_umin[j]) << at : (v - s_umin[j]) >> -at;
        if (s_fshift[j] >= cut && null != (bool)f.nulls_first) k[u] |= 1ull << (s_fshift[j] - cut);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t x = k[u] << (64 - (total - cut));
      s_key[base + u * blockDim.x] = x;
      s_hi[base + u * blockDim.x] = (uint32_t)(x >> 32);
    }
  }
  __syncthreads();
  unsigned int cnt[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};   // pairs with exactly q equal leading digits
  const int me = blockIdx.x * kSampleRows + threadIdx.x % kSampleRows;
  const uint64_t x = s_key[me];
  const uint32_t xh = (uint32_t)(x >> 32), lead = 0xffffffffu << (32 - 8 * p.first);
  const int span = p.S / (256 / kSampleRows), j0 = (threadIdx.x / kSampleRows) * span;
#pragma unroll 4
  for (int j = j0; j < j0 + span; j += 4) {
    const uint4 y = *(const uint4*)&s_hi[j];
    const bool hit[4] = {((xh ^ y.x) & lead) == 0, ((xh ^ y.y) & lead) == 0, ((xh ^ y.z) & lead) == 0,
                         ((xh ^ y.w) & lead) == 0};
    if (!(hit[0] | hit[1] | hit[2] | hit[3])) continue;
    for (int e = 0; e < 4; e++) {
      if (((xh ^ s_hi[j + e]) & lead) || j + e == me) continue;
      const uint64_t diff = x ^ s_key[j + e];
      const int q = diff == 0 ? 8 : __clzll((long long)diff) / 8;
#pragma unroll
      for (int k = 0; k < 9; k++) cnt[k] += k == q;
    }
  }
#pragma unroll
  for (int k = 0; k < 9; k++)
    if (cnt[k]) atomicAdd(&s_pairs[k], cnt[k]);
  __syncthreads();
  if (threadIdx.x >= (unsigned)p.first && threadIdx.x < 9) {
    unsigned long long v = 0;   // at least q equal leading digits
    for (int k = threadIdx.x; k < 9; k++) v += s_pairs[k];
    if (v) atomicAdd(&p.pairs[threadIdx.x], v);
  }
}

// ---------------------------------------------------------------- histogram
// One sub-field of a packed key with everything its bits need, so a kernel
// packing keys reads it with constant indices.
struct SubPlan {
  ghb_column col;
  uint64_t umin;
  int8_t shift;
  int8_t is_flag;
  int8_t desc;
  int8_t nulls_first;
  int8_t has_null;
};

__device__ __forceinline__ uint64_t sub_bits_plan(const SubPlan& sp, int64_t raw, int64_t r) {
  const bool null = sp.has_null && raw_is_null(sp.col, raw, r);
  uint64_t v;
  if (sp.is_flag) {
    v = (null == (bool)sp.nulls_first) ? 0 : 1;   // NULLS FIRST: null 0 / value 1
  } else {
    uint64_t u = key_image(sp.col, raw);
    if (sp.desc) u = ~u;
    v = null ? 0 : u - sp.umin;
  }
  return sp.shift >= 0 ? v << sp.shift : v >> -sp.shift;   // below 0: its low bits are left out
}

struct HistParams {
  KeySet K;
  Segment seg;
  SubPlan sub[kMaxSub];     // the segment's sub-fields, self-contained
  int64_t n;
  int32_t npasses;
  int32_t shift0;  // the first pass's digit starts here (lower bits are left to the finish)
  uint32_t* hist;  // [npasses][kBins]
  // a one-segment key: the packed keys and carried values are written here
  // too, so every radix pass reads packed keys
  uint64_t* keys_out;        // nullptr: not written
  void* vals_out;
  int32_t vals_wide;         // values are 64-bit (else 32-bit)
  int32_t carry_rowid;       // value = row index (else the single payload's raw bits)
  ghb_column pay_src;
  int32_t vec;               // every column read has 16-byte aligned data and no NULL map
};

__global__ void __launch_bounds__(256) sort_hist_kernel(HistParams p) {
  constexpr int U = 4;
  __shared__ uint32_t sh[kMaxPasses][kBins];
  for (int i = threadIdx.x; i < kMaxPasses * kBins; i += blockDim.x) (&sh[0][0])[i] = 0;
  __syncthreads();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // four consecutive rows per thread by 16-byte loads and stores, then the
  // rows past the last group of four (or all rows) one at a time
  int64_t done = 0;
  if (p.vec) {
    const int64_t ng = p.n / 4;
    for (int64_t g = tid; g < ng; g += stride) {
      const int64_t r = g * 4;
      uint64_t k[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < kMaxSub; i++) {
        if (i >= p.seg.n) break;
        const SubPlan& sp = p.sub[i];
        int64_t raw[4];
        load4(sp.col, r, raw);
#pragma unroll
        for (int u = 0; u < 4; u++) k[u] |= sub_bits_plan(sp, raw[u], r + u);
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        for (int q = 0; q < p.npasses; q++)
          atomicAdd(&sh[q][(k[u] >> (p.shift0 + q * kDigitBits)) & (kBins - 1)], 1u);
      if (p.keys_out) {
        ulonglong2* ko = (ulonglong2*)(p.keys_out + r);
        __stcs(ko, make_ulonglong2(k[0], k[1]));
        __stcs(ko + 1, make_ulonglong2(k[2], k[3]));
        int64_t v[4] = {r, r + 1, r + 2, r + 3};
        if (!p.carry_rowid) load4(p.pay_src, r, v);
        if (p.vals_wide) {
          ulonglong2* vo = (ulonglong2*)p.vals_out + r / 2;
          __stcs(vo, make_ulonglong2((unsigned long long)v[0], (unsigned long long)v[1]));
          __stcs(vo + 1, make_ulonglong2((unsigned long long)v[2], (unsigned long long)v[3]));
        } else {
          __stcs((uint4*)p.vals_out + r / 4,
                 make_uint4((unsigned)v[0], (unsigned)v[1], (unsigned)v[2], (unsigned)v[3]));
        }
      }
    }
    done = ng * 4;
  }
  for (int64_t base = done + tid; base < p.n; base += U * stride) {
    uint64_t k[U];
#pragma unroll
    for (int u = 0; u < U; u++) k[u] = 0;
#pragma unroll
    for (int i = 0; i < kMaxSub; i++) {
      if (i >= p.seg.n) break;
      const SubPlan& sp = p.sub[i];
      int64_t raw[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t r = base + u * stride;
        raw[u] = r < p.n ? ld_raw(sp.col, r) : 0;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t r = base + u * stride;
        if (r < p.n) k[u] |= sub_bits_plan(sp, raw[u], r);
      }
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t r = base + u * stride;
      if (r >= p.n) continue;
      for (int q = 0; q < p.npasses; q++)
        atomicAdd(&sh[q][(k[u] >> (p.shift0 + q * kDigitBits)) & (kBins - 1)], 1u);
      if (p.keys_out) {
        __stcs((unsigned long long*)p.keys_out + r, (unsigned long long)k[u]);
        const uint64_t v = p.carry_rowid ? (uint64_t)r : (uint64_t)ld_raw(p.pay_src, r);
        if (p.vals_wide) __stcs((unsigned long long*)p.vals_out + r, (unsigned long long)v);
        else __stcs((unsigned int*)p.vals_out + r, (unsigned int)v);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < p.npasses * kBins; i += blockDim.x) {
    uint32_t v = (&sh[0][0])[i];
    if (v) atomicAdd(&p.hist[i], v);
  }
}

// ---------------------------------------------------------------- passes
enum SrcMode { kSrcPacked = 0, kSrcCols = 1, kSrcPerm = 2 };
enum DstMode { kDstPacked = 0, kDstDecode = 1, kDstGather = 2 };

struct PassParams {
  KeySet K;
  Segment seg;
  int64_t n;
  int64_t ntiles;
  int32_t shift;
  int32_t carry_rowid;       // value = row index (else the single payload's raw bits)
  const uint64_t* keys_in;
  const void* vals_in;
  uint64_t* keys_out;
  void* vals_out;
  ghb_column pay_src;        // single carried payload (when !carry_rowid)
  ghb_out_column out_keys[kMaxSortKeys];
  int32_t npay;
  ghb_column pay[kMaxSortPay];
  ghb_out_column out_pay[kMaxSortPay];
  int32_t* out_rowid;
  // decoding a one-segment key, per key: value bits and shift, NULL flag
  // shift (-1 none)
  int8_t dec_vbits[kMaxSortKeys];
  int8_t dec_vshift[kMaxSortKeys];
  int8_t dec_fshift[kMaxSortKeys];
  const uint32_t* hist;        // rows of each digit of this pass
  uint32_t* status;            // [ntiles][kBins] look-back words, zero at the start of the pass
  uint32_t* status_next;       // the next pass's, zeroed by this one (nullptr: the last pass)
  unsigned long long* counters;
  int32_t* dev_status;
  unsigned int* gave_up;       // 1: a look-back of this sort gave up, what its passes wrote is not to be used
  int32_t spin_limit;          // look-back polls before GHB_ERR_TIMEOUT
  // a key wider than 64 bits sorted by its leading 64 (the finish): rows equal in
  // those are compared by their columns, the key columns are gathered by row,
  // and a long run with such rows out of order is reported
  int32_t wide;
  unsigned int* ties;
  uint32_t* long_runs;         // the finish: [0] runs it leaves to sort_finish_long_kernel, then their first rows
};

__device__ __forceinline__ void write_raw(const ghb_out_column& o, int64_t pos, int type, int64_t raw,
                                          bool null) {
  if (null) {
    if (o.is_null) o.is_null[pos] = 1;
    if (type == GHB_INT) ((int32_t*)o.data)[pos] = INT32_MAX;
    else if (type == GHB_LONG) ((int64_t*)o.data)[pos] = INT64_MAX;
    else ((long long*)o.data)[pos] = 0x7ff8000000000000ll;
    return;
  }
  if (type == GHB_INT) ((int32_t*)o.data)[pos] = (int32_t)raw;
  else ((long long*)o.data)[pos] = raw;
  if (o.is_null) o.is_null[pos] = 0;
}

// Copies keys and payloads of input row `row` to output position `pos`.
__device__ __forceinline__ void gather_write(const PassParams& p, int64_t row, int64_t pos) {
  for (int j = 0; j < p.K.nkeys; j++) {
    const ghb_column& c = p.K.k[j].col;
    int64_t raw = ld_raw(c, row);
    write_raw(p.out_keys[j], pos, c.type, raw, c.null_mode != GHB_NULLS_NONE && raw_is_null(c, raw, row));
  }
  if (p.out_rowid) p.out_rowid[pos] = (int32_t)row;
  for (int j = 0; j < p.npay; j++) {
    const ghb_column& c = p.pay[j];
    int64_t raw = ld_raw(c, row);
    write_raw(p.out_pay[j], pos, c.type, raw, c.null_mode != GHB_NULLS_NONE && raw_is_null(c, raw, row));
  }
}

// The carried value of a decoded row: its row index (row id output and
// payloads gathered by it), or the single payload itself.
__device__ __forceinline__ void decode_value(const PassParams& p, uint64_t v, int64_t pos) {
  if (p.carry_rowid) {
    int64_t row = (int64_t)v;
    if (p.out_rowid) p.out_rowid[pos] = (int32_t)row;
    for (int j = 0; j < p.npay; j++) {
      const ghb_column& c = p.pay[j];
      int64_t raw = ld_raw(c, row);
      write_raw(p.out_pay[j], pos, c.type, raw, c.null_mode != GHB_NULLS_NONE && raw_is_null(c, raw, row));
    }
  } else if (p.npay == 1) {
    const ghb_column& c = p.pay[0];
    bool null = c.null_mode == GHB_NULLS_SENTINEL && raw_is_null(c, (int64_t)v, 0);
    write_raw(p.out_pay[0], pos, c.type, (int64_t)v, null);
  }
}

// A tile's look-back word of one digit: 0 = not published; kTilePrefix | the
// inclusive count of the digit up to and with this tile (31 bits); else the
// tile's own count + 1.  Each pass of a call has its own zeroed words.
constexpr uint32_t kTilePrefix = 0x80000000u;
constexpr int kTileWindow = 8;   // earlier tiles read at once

__device__ __forceinline__ void tile_store(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t tile_load(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Rows of digit d in the tiles before `tile`: kTileWindow words are loaded
// together, so a walk over many unfinished tiles pays one L2 round trip per
// window and not per tile.  Gives up after `p.spin_limit` windows that brought
// nothing new (GHB_ERR_TIMEOUT; the count so far, no larger than the true one).
// That is told by the sort's own word as well: the status word keeps the first
// error, which may be that of a call before.
__device__ __forceinline__ uint32_t tile_lookback(const uint32_t* words, int64_t tile, int d, const PassParams& p) {
  uint32_t excl = 0;
  int64_t t = tile - 1;
  int spins = 0;
  while (t >= 0) {
    uint32_t v[kTileWindow];
#pragma unroll
    for (int i = 0; i < kTileWindow; i++) v[i] = t - i >= 0 ? tile_load(words + (t - i) * kBins + d) : kTilePrefix;
    int used = 0;
    bool found = false;
#pragma unroll
    for (int i = 0; i < kTileWindow; i++) {
      if (found || used < i || v[i] == 0) continue;   // past the first word not ready
      used = i + 1;
      if (v[i] & kTilePrefix) {
        excl += v[i] & ~kTilePrefix;
        found = true;
      } else {
        excl += v[i] - 1;
      }
    }
    if (found) break;
    t -= used;
    if (used == 0 && ++spins >= p.spin_limit) {
      raise_status(p.dev_status, kDevTimeout);
      *(volatile unsigned int*)p.gave_up = 1;
      break;
    }
  }
  return excl;
}

// Bound by the shared-memory and load/store data path (80 % busy, DRAM 36 %):
// about 40 shared wavefronts per 32 rows, 15 more for the global accesses.
// One pass over 20M packed 64-bit keys with 32-bit values: 148 us (188 us
// when the look-back read one tile's word at a time, rows past the end were
// tested per key, and a key's tile position and destination took two table
// reads each).  Three CTAs per SM (80 registers); measured on the 60M-row
// sort at this form: 3.57 ms, four CTAs at 64 registers 3.76 (the look-back
// walks more unfinished tiles), look-back windows of 2 / 4 / 16 tiles 3.57 /
// 3.50 / 3.9 ms (a 1M-row sort: 0.280 / 0.273 / - against 0.262 ms), ranking
// by eight ballots 4.37 and by __match_any_sync 4.40 ms, 12 / 18 / 20 / 24
// keys per thread 4.26 / 3.75 / 3.95 / 3.86 ms.
template <typename V, int SRC, int DST>
__global__ void __launch_bounds__(kSortThreads, 3) sort_pass_kernel(const __grid_constant__ PassParams p) {
  constexpr int kWarps = kSortThreads / 32;
  // per warp and digit: keys ranked so far << 32 | lanes of the item being
  // ranked, one word so a lane reads both with one load
  __shared__ unsigned long long s_cnt[kWarps][kBins];
  __shared__ uint32_t s_pos[kWarps][kBins];   // the warp's first tile position of each digit
  __shared__ uint32_t s_gb[kBins];       // global destination of each digit's run - its tile position
  __shared__ uint32_t s_base[kBins];     // global exclusive offset of each digit
  __shared__ uint32_t s_wsum[kWarps];
  __shared__ int64_t s_tile;
  extern __shared__ uint64_t s_dyn[];    // reordered tile: its keys, after them its values
  uint64_t* s_keys = s_dyn;
  V* s_vals = (V*)s_dyn;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int d = threadIdx.x;             // kSortThreads == kBins: a digit per thread
  const V* vals_in = (const V*)p.vals_in;
  V* vals_out = (V*)p.vals_out;

  // exclusive sum over the 256 digits of v (all threads, two barriers)
  auto digit_scan = [&](uint32_t v) -> uint32_t {
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) before += w < warp ? s_wsum[w] : 0;
    __syncthreads();
    return before + incl - v;
  };
  s_base[d] = digit_scan(p.hist[d]);

  while (true) {
    if (threadIdx.x == 0) {
      int64_t t = (int64_t)atomicAdd(&p.counters[0], 1ull);
      // a look-back of this sort that gave up left this pass's input invalid
      // (rows at wrong places, some never written): claim no more tiles, so no
      // key or row index read from that input addresses anything
      if (*(volatile unsigned int*)p.gave_up) t = p.ntiles;
      s_tile = t;
      // the tile about one round of claims ahead starts toward L2, so the
      // CTA that claims it finds its keys and values there
      const int64_t ahead = t + gridDim.x;
      if (SRC == kSrcPacked && (ahead + 1) * kSortTile <= p.n) {
        bulk_prefetch_l2((const unsigned long long*)p.keys_in + ahead * kSortTile, kSortTile * 8);
        bulk_prefetch_l2(vals_in + ahead * kSortTile, kSortTile * (uint32_t)sizeof(V));
      }
    }
    for (int i = threadIdx.x; i < kWarps * kBins; i += kSortThreads) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    if (tile >= p.ntiles) break;
    const int64_t wbase = tile * kSortTile + (int64_t)warp * (32 * kSortItems);
    const int tile_n = (int)min((int64_t)kSortTile, p.n - tile * kSortTile);

    // Rows past the end carry the key ~0: they are the last of the last
    // digit, so ranking and reordering take them along at the tile's end and
    // only the published count leaves them out.
    uint64_t key[kSortItems];
    V val[kSortItems];
    if (SRC == kSrcPacked) {
#pragma unroll
      for (int k = 0; k < kSortItems; k++) {
        int64_t row = wbase + k * 32 + lane;
        key[k] = row < p.n ? __ldcs((const unsigned long long*)p.keys_in + row) : ~0ull;
      }
    } else {
      int64_t src[kSortItems];
#pragma unroll
      for (int k = 0; k < kSortItems; k++) {
        int64_t row = wbase + k * 32 + lane;
        key[k] = 0;
        if (SRC == kSrcPerm) src[k] = row < p.n ? (int64_t)vals_in[row] : 0;
        else src[k] = row;
      }
      // one sub-field at a time over all items: the loads are independent
      for (int i = 0; i < p.seg.n; i++) {
        const SubField sf = p.seg.f[i];
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
          int64_t row = wbase + k * 32 + lane;
          if (row < p.n) key[k] |= sub_bits(p.K, sf, src[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < kSortItems; k++) {
        int64_t row = wbase + k * 32 + lane;
        if (row >= p.n) key[k] = ~0ull;
        if (p.carry_rowid) val[k] = (V)src[k];
        else val[k] = row < p.n ? (V)ld_raw(p.pay_src, row) : (V)0;
      }
    }
    // stable rank of each key among the warp's keys with the same digit: the
    // lanes holding digit dk set their bits in the digit's word (one shared
    // atomic, no per-bit ballots), read the word and the running count back,
    // and the lowest of them clears the one and advances the other
    uint32_t rank[kSortItems / 2];   // two 16-bit ranks a word
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      const uint32_t dk = (uint32_t)(key[k] >> p.shift) & (kBins - 1);
      volatile unsigned long long* word = &s_cnt[warp][dk];
      atomicOr((unsigned int*)word, 1u << lane);
      __syncwarp();
      const unsigned long long w = *word;
      const uint32_t peers = (uint32_t)w, before = (uint32_t)(w >> 32);
      __syncwarp();
      if ((peers & lt) == 0) *word = (unsigned long long)(before + __popc(peers)) << 32;
      __syncwarp();
      const uint32_t r = before + __popc(peers & lt);
      rank[k / 2] = k & 1 ? rank[k / 2] | r << 16 : r;
    }
    __syncthreads();
    // per digit (one thread each): exclusive over warps, tile total; publish
    uint32_t excl_w[kWarps];
    uint32_t total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; w++) {
      excl_w[w] = total;
      total += (uint32_t)(s_cnt[w][d] >> 32);
    }
    const uint32_t mine = d == kBins - 1 ? total - (uint32_t)(kSortTile - tile_n) : total;
    uint32_t* words = p.status + tile * kBins + d;
    if (tile == 0) tile_store(words, kTilePrefix | mine);
    else tile_store(words, mine + 1);
    if (p.status_next) p.status_next[tile * kBins + d] = 0;   // the next pass's words
    const uint32_t bexcl = digit_scan(total);
#pragma unroll
    for (int w = 0; w < kWarps; w++) s_pos[w][d] = bexcl + excl_w[w];
    __syncthreads();
    // scatter the keys into shared memory in digit order (stable); rank
    // becomes the tile position
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      const uint32_t dk = (uint32_t)(key[k] >> p.shift) & (kBins - 1);
      const uint32_t at = s_pos[warp][dk] + (rank[k / 2] >> (k & 1 ? 16 : 0) & 0xffffu);
      s_keys[at] = key[k];
      rank[k / 2] = k & 1 ? (rank[k / 2] & 0xffffu) | at << 16 : (rank[k / 2] & 0xffff0000u) | at;
    }
    // the values are loaded here, when the keys' registers are free, and
    // arrive during the look-back
    if (SRC == kSrcPacked) {
#pragma unroll
      for (int k = 0; k < kSortItems; k++) {
        int64_t row = wbase + k * 32 + lane;
        val[k] = row < p.n ? __ldcs(vals_in + row) : (V)0;
      }
    }
    // look back for the digit's rows in earlier tiles (after the scatter, so
    // that more of them have published), then publish the prefix
    uint32_t excl = 0;
    if (tile > 0) {
      excl = tile_lookback(p.status, tile, d, p);
      tile_store(words, kTilePrefix | (excl + mine));
    }
    s_gb[d] = s_base[d] + excl - bexcl;
    __syncthreads();
    // write runs: element i of the reordered tile goes to s_gb[digit] + i,
    // keys first, then the values through the same shared memory
    uint32_t pos[kSortItems];
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      const int i = k * kSortThreads + threadIdx.x;
      const uint64_t x = s_keys[i];
      pos[k] = s_gb[(uint32_t)(x >> p.shift) & (kBins - 1)] + (uint32_t)i;
      if (DST == kDstPacked && i < tile_n) __stcs((unsigned long long*)p.keys_out + pos[k], (unsigned long long)x);
    }
    if (DST == kDstDecode) {
      // one key column at a time, its decoding parameters held in registers
      for (int j = 0; j < p.K.nkeys; j++) {
        const KeyField& kf = p.K.k[j];
        const int vb = p.dec_vbits[j], vs = p.dec_vshift[j], fs = p.dec_fshift[j];
        const uint64_t vmask = vb == 0 ? 0 : (vb >= 64 ? ~0ull : ((1ull << vb) - 1));
        const uint64_t umin = kf.umin;
        const bool desc = kf.desc, nf = kf.nulls_first;
        const int type = kf.col.type;
        const ghb_out_column o = p.out_keys[j];
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
          const int i = k * kSortThreads + threadIdx.x;
          if (i >= tile_n) continue;
          const uint64_t x = s_keys[i];
          const bool null = fs >= 0 && (((x >> fs) & 1ull) == 0) == nf;
          uint64_t u = (vb == 0 ? 0 : (x >> vs) & vmask) + umin;
          if (desc) u = ~u;
          const int64_t raw = type == GHB_DOUBLE ? (int64_t)unflip_f64_bits(u) : (int64_t)(u ^ 0x8000000000000000ull);
          write_raw(o, pos[k], type, raw, null);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) s_vals[rank[k / 2] >> (k & 1 ? 16 : 0) & 0xffffu] = val[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSortItems; k++) {
      const int i = k * kSortThreads + threadIdx.x;
      if (i >= tile_n) continue;
      if (DST == kDstPacked) __stcs(vals_out + pos[k], s_vals[i]);
      else if (DST == kDstDecode) decode_value(p, (uint64_t)s_vals[i], pos[k]);
      else gather_write(p, (int64_t)s_vals[i], pos[k]);
    }
    __syncthreads();
  }
  claim_finish(p.counters);
}

// ---------------------------------------------------------------- finish
// Writes raw[k] (NULL: bit k of `nulls`) to row pos[k] of an output column, k
// with bit k of `live`: the type and the NULL map are tested once per column.
template <int N>
__device__ __forceinline__ void put_rows(const ghb_out_column& o, int type, const int64_t (&raw)[N], uint32_t nulls,
                                         const uint32_t (&pos)[N], uint32_t live) {
  if (type == GHB_INT) {
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) ((int32_t*)o.data)[pos[k]] = nulls >> k & 1 ? INT32_MAX : (int32_t)raw[k];
  } else {
    const int64_t none = type == GHB_LONG ? INT64_MAX : 0x7ff8000000000000ll;
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) ((int64_t*)o.data)[pos[k]] = nulls >> k & 1 ? none : raw[k];
  }
  if (o.is_null) {
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) o.is_null[pos[k]] = nulls >> k & 1;
  }
}

// Bit k: raw[k] of row row[k] is NULL.
template <int N>
__device__ __forceinline__ uint32_t null_bits(const ghb_column& c, const int64_t (&raw)[N], const int64_t (&row)[N],
                                              uint32_t live) {
  uint32_t m = 0;
  if (c.null_mode == GHB_NULLS_NONE) return 0;
#pragma unroll
  for (int k = 0; k < N; k++)
    if (live >> k & 1) m |= (raw_is_null(c, raw[k], row[k]) ? 1u : 0u) << k;
  return m;
}

// Writes N rows of a thread, key[k] and carried value val[k], to output
// positions pos[k] (k with bit k of `live`): one column at a time, every load
// of a gathered column issued before its stores.
template <int N, bool WIDE, typename V>
__device__ __forceinline__ void emit_rows(const PassParams& p, const uint64_t (&key)[N], const V (&val)[N],
                                          const uint32_t (&pos)[N], uint32_t live) {
  int64_t raw[N];
  for (int j = 0; j < p.K.nkeys && WIDE; j++) {
    const ghb_column& c = p.K.k[j].col;
    int64_t r[N];
#pragma unroll
    for (int k = 0; k < N; k++) r[k] = (int64_t)val[k];
#pragma unroll
    for (int k = 0; k < N; k++) raw[k] = live >> k & 1 ? ld_raw(c, r[k]) : 0;
    put_rows<N>(p.out_keys[j], c.type, raw, null_bits<N>(c, raw, r, live), pos, live);
  }
  for (int j = 0; j < p.K.nkeys && !WIDE; j++) {
    const KeyField& kf = p.K.k[j];
    const int vb = p.dec_vbits[j], vs = p.dec_vshift[j] & 63, fs = p.dec_fshift[j];
    const uint64_t vmask = vb == 0 ? 0 : (vb >= 64 ? ~0ull : ((1ull << vb) - 1));
    // order image = field + umin, complemented for DESC; an integer's value is
    // its image with the sign bit flipped, that is 2^63 added; -f = ~f + 1
    const uint64_t neg = kf.desc ? ~0ull : 0ull;
    const uint64_t base = (kf.umin ^ neg) - neg - (kf.desc ? 1 : 0);
    uint32_t nulls = 0;
    if (kf.col.type == GHB_INT) {
      const uint32_t m32 = (uint32_t)vmask, n32 = (uint32_t)neg, b32 = (uint32_t)base - n32;
#pragma unroll
      for (int k = 0; k < N; k++) raw[k] = (int32_t)((((uint32_t)(key[k] >> vs) & m32) ^ n32) + b32);
    } else if (kf.col.type == GHB_LONG) {
      const uint64_t b64 = base - neg + 0x8000000000000000ull;
#pragma unroll
      for (int k = 0; k < N; k++) raw[k] = (int64_t)((((key[k] >> vs) & vmask) ^ neg) + b64);
    } else {
#pragma unroll
      for (int k = 0; k < N; k++) raw[k] = (int64_t)unflip_f64_bits((((key[k] >> vs) & vmask) ^ neg) + base - neg);
    }
    if (fs >= 0) {
      const bool nf = kf.nulls_first;
#pragma unroll
      for (int k = 0; k < N; k++) nulls |= ((((key[k] >> fs) & 1ull) == 0) == nf ? 1u : 0u) << k;
    }
    put_rows<N>(p.out_keys[j], kf.col.type, raw, nulls, pos, live);
  }
  int64_t row[N];   // a carried payload's raw value, or the row index
#pragma unroll
  for (int k = 0; k < N; k++) row[k] = sizeof(V) == 4 ? (int64_t)(int32_t)val[k] : (int64_t)val[k];
  if (!p.carry_rowid) {
    if (p.npay == 1) {
      const ghb_column& c = p.pay[0];
      put_rows<N>(p.out_pay[0], c.type, row, c.null_mode == GHB_NULLS_SENTINEL ? null_bits<N>(c, row, row, live) : 0u,
                  pos, live);
    }
    return;
  }
  if (p.out_rowid) {
#pragma unroll
    for (int k = 0; k < N; k++)
      if (live >> k & 1) p.out_rowid[pos[k]] = (int32_t)row[k];
  }
  for (int j = 0; j < p.npay; j++) {
    const ghb_column& c = p.pay[j];
#pragma unroll
    for (int k = 0; k < N; k++) raw[k] = live >> k & 1 ? ld_raw(c, row[k]) : 0;
    put_rows<N>(p.out_pay[j], c.type, raw, null_bits<N>(c, raw, row, live), pos, live);
  }
}

constexpr int kFinItems = 4;                         // rows a thread works on together
constexpr int kFinTile = 2 * kSortThreads * kFinItems;   // 2048 rows
constexpr int kFinRounds = 2;                        // further rows read to find a run's end:
constexpr int kFinExt = 32 + kFinRounds * kSortThreads;   // 32, then 256 a round
constexpr int kFinNet = 16;                          // longest run one thread sorts
constexpr int kFinField = 28;                        // key bits such a sort compares
constexpr int kFinTieRun = 1024;                     // longest run in which a wide key's columns are compared

__device__ __forceinline__ void word_order(uint32_t& a, uint32_t& b) {
  const uint32_t lo = min(a, b);
  b = max(a, b);
  a = lo;
}

// Sorts the first N words in registers by odd-even merges (Batcher): the
// comparators of distance K of the merges into blocks of 2 P words, then of
// K / 2, then those of 2 P.
template <int N, int P = 1, int K = 1>
__device__ __forceinline__ void sort_words(uint32_t (&w)[kFinNet]) {
#pragma unroll
  for (int e = K % P; e + K < N; e++)
    if ((e - K % P) % (2 * K) < K && e / (2 * P) == (e + K) / (2 * P)) word_order(w[e], w[e + K]);
  if constexpr (K > 1) sort_words<N, P, K / 2>(w);
  else if constexpr (2 * P < N) sort_words<N, 2 * P, 2 * P>(w);
}

// Sorts the places src[0 .. len) by `threads` threads of a warp or a CTA (thread
// t of them, `sync` their barrier): bitonic merges, each beginning with the
// comparison of mirrored places, so that every comparison leaves the earlier row
// (after(x, y): row x goes after row y) in front and places past len take no part.
template <typename AFTER, typename SYNC>
__device__ __forceinline__ void sort_places(uint16_t* src, int len, int t, int threads, const AFTER& after,
                                            const SYNC& sync) {
  for (int size = 2; size / 2 < len; size *= 2)
    for (int stride = size / 2; stride > 0; stride /= 2) {
      const bool mirror = stride == size / 2;
      for (int q = t; 2 * q < len + stride; q += threads) {   // i below len
        const int off = q & (stride - 1), i = 2 * (q - off) + off;
        const int j = mirror ? i + size - 1 - 2 * off : i + stride;
        if (j >= len) continue;
        const uint16_t x = src[i], y = src[j];
        if (after(x, y)) {
          src[i] = y;
          src[j] = x;
        }
      }
      sync();
    }
}

// Order of rows a and b by the whole of their keys (-1, 0, 1), for rows of a wide
// key that its leading 64 bits do not tell apart.  Out of line: rare.
__device__ __noinline__ int row_order(const PassParams& p, int64_t a, int64_t b) {
  for (int j = 0; j < p.K.nkeys; j++) {
    const KeyField& f = p.K.k[j];
    const int64_t x = ld_raw(f.col, a), y = ld_raw(f.col, b);
    const bool nx = raw_is_null(f.col, x, a), ny = raw_is_null(f.col, y, b);
    if (nx != ny) return nx == (bool)f.nulls_first ? -1 : 1;
    if (nx) continue;
    const uint64_t u = key_image(f.col, x), v = key_image(f.col, y);
    if (u != v) return (u < v) != (bool)f.desc ? -1 : 1;
  }
  return 0;
}

// One run of len <= N rows from row a on, put in order by one thread: words
// (field, place in the run) sorted in registers, then, when equal words may be
// of different keys (`partial`), those rows by insertion.
template <int N, typename BELOW>
__device__ __forceinline__ void sort_run(const uint32_t* s_word, uint16_t* s_src, int a, int len, bool partial,
                                         const BELOW& below) {
  uint32_t w[kFinNet];
#pragma unroll
  for (int k = 0; k < N; k++) w[k] = k < len ? s_word[a + k] | k : 0xffffffffu;
  sort_words<N>(w);
  bool tie = false;
#pragma unroll
  for (int k = 0; k < N; k++) {
    if (k < len) s_src[a + k] = (uint16_t)(a + (w[k] & 15u));
    if (partial && k > 0 && k < len) tie |= (w[k] ^ w[k - 1]) < 16u;
  }
  if (tie)
    for (int i = 1; i < len; i++) {
      const uint16_t x = s_src[a + i];
      int j = i;
      for (; j > 0 && below(x, s_src[a + j - 1]); j--) s_src[a + j] = s_src[a + j - 1];
      s_src[a + j] = x;
    }
}

// The rows are sorted by their keys' bits from p.shift up; a tile puts the
// runs that start in it (equal bits from p.shift up) in order by the lower
// bits and writes their rows, in output order.  A run of up to kFinNet rows is
// sorted by one thread in registers; one of up to 32 by a warp, a row a lane
// that counts the rows before it; a longer one by a warp's and past kWarpRun
// rows by the CTA's bitonic merges in shared memory.  A run
// whose end is not found within kFinExt rows of the tile goes to the list of
// long runs.  Bound by instruction issue (205 per 32 rows at six rows to a
// run; DRAM 35 %): 0.56 ms for the 60M-row (d, k) sort, which it spares four
// passes of 0.40 ms.  Other forms measured there: every row counting the rows
// of its run before it 1.04 ms, with 64-bit keys in shared memory 0.96; one
// list of runs found by a thread per row 0.71.  A 1M-row sort of 0.18 ms with
// one unordered run of 500 / 1000 / 2000 rows: 0.19 / 0.20 / 0.23 ms, and 0.29 /
// 0.62 / 1.88 when a warp counted every long run; 4M rows of which 40 % lie in
// runs of 64, 25 % in runs of 100: 0.32 and 0.33 ms (0.32 and 0.35), 0.54 and
// 0.43 with the CTA from 33 rows on.
template <typename V, bool WIDE>
__global__ void __launch_bounds__(kSortThreads, 5) sort_finish_kernel(const __grid_constant__ PassParams p) {
  constexpr int kRows = kFinTile + kFinExt;
  constexpr int kWords = kRows / 32;
  constexpr int kTileWords = kFinTile / 32;
  static_assert(kFinTile == 8 * kSortThreads && kFinTile == 2048 && kFinNet == 16, "a run's list entry");
  // longest run a warp sorts: a longer one keeps a lone warp for too long (a
  // comparison of a wide key's columns is a chain of loads)
  constexpr int kWarpRun = WIDE ? 128 : 256;
  constexpr int kRuns = kFinTile / 2 + 1;        // runs of two rows and more that start in a tile
  __shared__ uint64_t s_key[kRows];
  __shared__ uint32_t s_word[kRows];             // the key's field << 4
  __shared__ uint16_t s_src[kRows];              // row of the tile that goes to each place
  __shared__ uint16_t s_run[kRuns];              // (rows - 1) << 11 | first row: runs of up to 8 rows from the
                                                 // front, of up to kFinNet from the back
  __shared__ uint16_t s_big[kRows / kFinNet];    // first rows of longer runs
  __shared__ uint32_t s_start[kWords + 1];       // bit i: row i starts a run
  __shared__ uint32_t s_n[2];                    // runs in the lists: up to 8 rows | up to kFinNet << 16; longer
  __shared__ uint32_t s_huge;                    // some of the longer runs have more than kWarpRun rows
  if (*(volatile unsigned int*)p.gave_up) return;   // the passes left invalid rows
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t t0 = (int64_t)blockIdx.x * kFinTile;
  const int left = (int)min(p.n - t0, (int64_t)kRows);   // rows from the tile's first to the end
  const unsigned long long* keys_in = (const unsigned long long*)p.keys_in + t0;
  const V* vals_in = (const V*)p.vals_in + t0;
  const uint64_t lead = ~0ull << p.shift;                // 0 < p.shift < 64
  const int fshift = max(0, p.shift - kFinField);
  // equal words may be of keys that differ: below the field, or of a wide key
  // below its leading 64 bits, however few of those the passes left
  const bool partial = WIDE || fshift > 0;
  // row i's key is below row j's (of a wide key: by the bits left out, too)
  auto below = [&](int i, int j) -> bool {
    const uint64_t x = s_key[i], y = s_key[j];
    return x < y || (WIDE && x == y && row_order(p, (int64_t)vals_in[i], (int64_t)vals_in[j]) < 0);
  };
  const uint32_t fmask = (1u << min(p.shift, kFinField)) - 1u;
  if (threadIdx.x < 2) s_n[threadIdx.x] = 0;
  if (threadIdx.x == 0) s_start[kWords] = s_huge = 0;
  // row i of the tile: its key to shared memory, and its start flag
  auto enter = [&](int i, uint64_t key) -> uint32_t {
    uint64_t prev = __shfl_up_sync(0xffffffffu, key, 1);
    if (lane == 0) prev = t0 + i > 0 && i < left ? keys_in[i - 1] : ~key;
    const uint32_t sw = __ballot_sync(0xffffffffu, i >= left || ((prev ^ key) & lead));   // rows past the end
                                                                                          // close the last run
    s_key[i] = key;
    s_word[i] = ((uint32_t)(key >> fshift) & fmask) << 4;
    s_src[i] = (uint16_t)i;
    if (lane == 0) s_start[i >> 5] = sw;
    return sw;
  };
  for (int h = 0; h < kFinTile; h += kSortThreads * kFinItems) {
    uint64_t x[kFinItems];
#pragma unroll
    for (int k = 0; k < kFinItems; k++) {
      const int i = h + k * kSortThreads + threadIdx.x;
      x[k] = i < left ? __ldcs(keys_in + i) : 0;
    }
#pragma unroll
    for (int k = 0; k < kFinItems; k++) enter(h + k * kSortThreads + threadIdx.x, x[k]);
  }
  // the rows after the tile up to the start of a run
  if (warp == 0) enter(kFinTile + lane, kFinTile + lane < left ? keys_in[kFinTile + lane] : 0);
  __syncthreads();
  int rows = kFinTile + 32;                        // rows entered
  bool closed = s_start[kTileWords] != 0;          // the last run's end is among them
  for (int q = 0; q < kFinRounds && !closed; q++) {
    const int i = rows + threadIdx.x;
    closed = __syncthreads_or(enter(i, i < left ? keys_in[i] : 0) != 0);
    rows += kSortThreads;
  }
  // first start after row i, `rows` if there is none
  auto next_start = [&](int i) -> int {
    int w = i >> 5;
    uint32_t m = s_start[w] & (0xfffffffeu << (i & 31));
    while (m == 0 && (w + 1) * 32 < rows) m = s_start[++w];
    return m ? w * 32 + __ffs(m) - 1 : rows;
  };
  // [begin, end): the runs that start in the tile; an open one is a long run
  int begin = kFinTile, end = 0;
  for (int w = 0; w < kTileWords; w++)
    if (s_start[w]) {
      begin = w * 32 + __ffs(s_start[w]) - 1;
      break;
    }
  if (begin >= min(left, kFinTile)) return;        // the whole tile belongs to an earlier tile's run
  if (closed) {
    end = min(left, next_start(kFinTile - 1));
  } else {
    for (int w = kTileWords - 1;; w--)
      if (s_start[w]) {
        end = w * 32 + 31 - __clz(s_start[w]);
        break;
      }
    if (threadIdx.x == 0) p.long_runs[1 + atomicAdd(&p.long_runs[0], 1u)] = (uint32_t)(t0 + end);
  }
  // list the runs of two rows and more: eight rows a thread, from the bits of
  // its rows and the 24 after them
  {
    const int r0 = 8 * threadIdx.x;
    const int w = threadIdx.x >> 2;
    const uint32_t win = __funnelshift_r(s_start[w], s_start[w + 1], 8 * (threadIdx.x & 3));
    uint32_t mine = win & 0xffu;
    if (end - r0 < 8) mine &= end > r0 ? (1u << (end - r0)) - 1u : 0u;
    mine &= ~(win >> 1);                               // not runs of one row
    uint32_t n = 0;                                    // runs of up to 8 rows, of up to kFinNet << 16
    for (uint32_t m = mine; m; m &= m - 1) {
      const int len = __ffs(win >> __ffs(m));
      n += len == 0 || len > kFinNet ? 0u : len <= 8 ? 1u : 1u << 16;
    }
    uint32_t incl = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    uint32_t at = 0;
    if (lane == 31) at = atomicAdd(&s_n[0], incl);
    at = __shfl_sync(0xffffffffu, at, 31) + incl - n;
    for (uint32_t m = mine; m; m &= m - 1) {
      const int j = __ffs(m) - 1, len = __ffs(win >> (j + 1));
      if (len == 0 || len > kFinNet) {
        s_big[atomicAdd(&s_n[1], 1u)] = (uint16_t)(r0 + j);
      } else if (len <= 8) {
        s_run[at & 0xffffu] = (uint16_t)((len - 1) << 11 | (r0 + j));
        at += 1;
      } else {
        s_run[kRuns - 1 - (at >> 16)] = (uint16_t)((len - 1) << 11 | (r0 + j));
        at += 1u << 16;
      }
    }
  }
  __syncthreads();
  const int n8 = s_n[0] & 0xffffu, n16 = s_n[0] >> 16, nbig = s_n[1];
  auto after = [&](int i, int j) -> bool { return below(j, i) || (i > j && !below(i, j)); };
  for (int m = warp; m < nbig; m += kSortThreads / 32) {
    const int a = s_big[m], len = next_start(a) - a;
    if (len > kWarpRun) {
      s_huge = 1;   // the CTA's, below
      continue;
    }
    bool desc = false;
    for (int i = a + 1 + lane; i < a + len; i += 32) desc |= below(i, i - 1);
    if (!__any_sync(0xffffffffu, desc)) continue;   // in order already
    if (len > 32) {
      sort_places(s_src + a, len, lane, 32, after, [] { __syncwarp(); });
    } else if (lane < len) {   // a row a lane: its place is the number of rows before it
      const int i = a + lane;
      const uint64_t mine = s_key[i];
      int at = a;
      for (int j = a; j < a + len; j++) {
        const uint64_t y = s_key[j];
        bool before = y < mine;
        if (y == mine && j != i) before = after(i, j);
        at += before;
      }
      s_src[at] = (uint16_t)i;
    }
  }
  for (int r = threadIdx.x; r < n16; r += kSortThreads) {
    const int e = s_run[kRuns - 1 - r];
    sort_run<16>(s_word, s_src, e & 2047, (e >> 11) + 1, partial, below);
  }
  // the other way round, so that the warps without a run above go first
  for (int r = kSortThreads - 1 - threadIdx.x; r < n8; r += kSortThreads) {
    const int e = s_run[r], a = e & 2047, len = (e >> 11) + 1;
    if (__any_sync(__activemask(), len > 4)) sort_run<8>(s_word, s_src, a, len, partial, below);
    else sort_run<4>(s_word, s_src, a, len, partial, below);
  }
  __syncthreads();
  for (int m = 0; s_huge && m < nbig; m++) {   // the longest runs, the CTA one after another
    const int a = s_big[m], len = next_start(a) - a;
    if (len <= kWarpRun) continue;
    const bool whole = WIDE && len <= kFinTieRun;   // rows of equal leading bits compared by their columns
    bool desc = false;
    for (int i = a + 1 + threadIdx.x; i < a + len; i += kSortThreads)
      desc |= whole ? below(i, i - 1) : s_key[i] < s_key[i - 1];
    if (__syncthreads_or(desc))
      sort_places(s_src + a, len, (int)threadIdx.x, kSortThreads,
                  [&](int i, int j) {
                    const uint64_t x = s_key[i], y = s_key[j];
                    return x != y ? x > y : whole ? after(i, j) : i > j;
                  },
                  [] { __syncthreads(); });
    // else such rows are reported when they are out of order
    for (int i = a + 1 + threadIdx.x; WIDE && !whole && i < a + len; i += kSortThreads) {
      const int x = s_src[i], y = s_src[i - 1];
      if (s_key[x] == s_key[y] && row_order(p, (int64_t)vals_in[x], (int64_t)vals_in[y]) < 0)
        *(volatile unsigned int*)p.ties = 1;
    }
  }
  for (int h = 0; h < kFinTile && h < end; h += kSortThreads * kFinItems) {
    V val[kFinItems];
    uint64_t x[kFinItems];
    uint32_t pos[kFinItems], live = 0;
#pragma unroll
    for (int k = 0; k < kFinItems; k++) {
      const int i = h + k * kSortThreads + threadIdx.x;
      const bool mine = i >= begin && i < end;
      const int src = mine ? s_src[i] : 0;
      val[k] = mine ? vals_in[src] : (V)0;
      x[k] = s_key[src];
      pos[k] = (uint32_t)t0 + (uint32_t)i;
      live |= (mine ? 1u : 0u) << k;
    }
    emit_rows<kFinItems, WIDE>(p, x, val, pos, live);
  }
  for (int i = kFinTile + threadIdx.x; i < end; i += kSortThreads) {   // the last run's rows past the tile
    const uint64_t x[1] = {s_key[s_src[i]]};
    const V v[1] = {vals_in[s_src[i]]};
    const uint32_t at[1] = {(uint32_t)t0 + (uint32_t)i};
    emit_rows<1, WIDE>(p, x, v, at, 1u);
  }
}

// The long runs, one CTA each: rows already in order are written as they are;
// else a stable LSD radix sort of the run by its lower bits, through the other
// ping-pong buffer.
constexpr int kLongThreads = 1024;

template <typename V, bool WIDE>
__global__ void __launch_bounds__(kLongThreads) sort_finish_long_kernel(const __grid_constant__ PassParams p) {
  __shared__ uint32_t s_hist[kBins], s_base[kBins];
  __shared__ uint16_t s_wcnt[kLongThreads / 32][kBins];
  __shared__ int64_t s_end;
  if (*(volatile unsigned int*)p.gave_up) return;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const uint32_t count = *(volatile uint32_t*)p.long_runs;
  for (uint32_t q = blockIdx.x; q < count; q += gridDim.x) {
    const int64_t a = p.long_runs[1 + q];
    uint64_t* kb[2] = {(uint64_t*)p.keys_in, p.keys_out};
    V* vb[2] = {(V*)p.vals_in, (V*)p.vals_out};
    if (threadIdx.x == 0) {   // the run's end: the leading bits ascend
      const uint64_t top = kb[0][a] >> p.shift;
      int64_t lo = a, hi = p.n;   // kb[lo] in the run, hi past it
      while (hi - lo > 1) {
        const int64_t m = lo + (hi - lo) / 2;
        if (kb[0][m] >> p.shift == top) lo = m;
        else hi = m;
      }
      s_end = hi;
    }
    __syncthreads();
    const int64_t b = s_end;
    bool desc = false;
    for (int64_t i = a + 1 + threadIdx.x; i < b; i += kLongThreads) desc |= kb[0][i] < kb[0][i - 1];
    int cur = 0;
    if (__syncthreads_or(desc))
      for (int sh = 0; sh < p.shift; sh += kDigitBits) {
        const uint32_t mask = min(kBins, 1 << min(kDigitBits, p.shift - sh)) - 1;
        for (int i = threadIdx.x; i < kBins; i += kLongThreads) s_hist[i] = 0;
        __syncthreads();
        for (int64_t i = a + threadIdx.x; i < b; i += kLongThreads)
          atomicAdd(&s_hist[(uint32_t)(kb[cur][i] >> sh) & mask], 1u);
        __syncthreads();
        if (warp == 0) {   // exclusive offsets, eight digits a lane
          uint32_t v[kBins / 32], sum = 0;
#pragma unroll
          for (int k = 0; k < kBins / 32; k++) {
            v[k] = s_hist[lane * (kBins / 32) + k];
            sum += v[k];
          }
          uint32_t incl = sum;
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
          }
          uint32_t run = incl - sum;
#pragma unroll
          for (int k = 0; k < kBins / 32; k++) {
            s_base[lane * (kBins / 32) + k] = run;
            run += v[k];
          }
        }
        for (int64_t c = a; c < b; c += kLongThreads) {
          for (int i = threadIdx.x; i < kLongThreads / 32 * kBins; i += kLongThreads) (&s_wcnt[0][0])[i] = 0;
          __syncthreads();
          const int64_t i = c + threadIdx.x;
          const bool live = i < b;
          const uint64_t x = live ? kb[cur][i] : 0;
          const V v = live ? vb[cur][i] : (V)0;
          const uint32_t dk = live ? (uint32_t)(x >> sh) & mask : kBins;
          const unsigned peers = __match_any_sync(0xffffffffu, dk);
          const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
          if (live && rank == 0) s_wcnt[warp][dk] = (uint16_t)__popc(peers);
          __syncthreads();
          if (threadIdx.x < kBins) {
            uint32_t run = s_base[threadIdx.x];
            for (int w = 0; w < kLongThreads / 32; w++) {
              const uint32_t t = s_wcnt[w][threadIdx.x];
              s_wcnt[w][threadIdx.x] = (uint16_t)(run - s_base[threadIdx.x]);
              run += t;
            }
            s_hist[threadIdx.x] = run;
          }
          __syncthreads();
          if (live) {
            const int64_t to = a + s_base[dk] + s_wcnt[warp][dk] + rank;
            kb[cur ^ 1][to] = x;
            vb[cur ^ 1][to] = v;
          }
          __syncthreads();
          if (threadIdx.x < kBins) s_base[threadIdx.x] = s_hist[threadIdx.x];
          __syncthreads();
        }
        cur ^= 1;
      }
    for (int64_t i = a + threadIdx.x; i < b; i += kLongThreads) {
      const uint64_t x[1] = {kb[cur][i]};
      if (WIDE && i > a && kb[cur][i - 1] == x[0] && row_order(p, (int64_t)vb[cur][i], (int64_t)vb[cur][i - 1]) < 0)
        *(volatile unsigned int*)p.ties = 1;
      const V v[1] = {vb[cur][i]};
      const uint32_t at[1] = {(uint32_t)i};
      emit_rows<1, WIDE>(p, x, v, at, 1u);
    }
    __syncthreads();   // s_end and the run's buffers are done with
  }
}

}  // namespace ghb

#include "ghb_sort_small.cuh"

namespace ghb {

// Output in input order (keys all equal): gathers row r to r, or
// row perm[r] to r when a permutation is given.
template <typename V>
__global__ void sort_identity_kernel(PassParams p, const V* perm) {
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < p.n;
       r += (int64_t)gridDim.x * blockDim.x)
    gather_write(p, perm ? (int64_t)perm[r] : r, r);
}

// Words of the analysis: three per key, then the sample's pair counts.
constexpr int kStatWords = 3 * kMaxSortKeys + 9;
// after them: a wide key's long run is out of order below its leading 64 bits; a
// look-back gave up
constexpr int kTieWord = kStatWords, kGaveUpWord = kStatWords + 1;
constexpr size_t kStatBytes = (kStatWords + 2) * 8;

static inline size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// Scratch needed by sort_impl for n rows.
size_t sort_scratch_bytes(int64_t n) {
  int64_t ntiles = (n + kSortTile - 1) / kSortTile;
  size_t b = 0;
  b += 2 * align256((size_t)n * 8);                        // keys ping-pong
  b += 2 * align256((size_t)n * 8);                        // values ping-pong
  b += 2 * align256((size_t)ntiles * kBins * 4);           // look-back words of two passes
  b += align256((size_t)kMaxSeg * kMaxPasses * kBins * 4); // histograms
  b += align256(kStatBytes);                               // min/max, sample, flags
  b += align256(((size_t)n / kFinTile + 2) * 4);           // long runs
  return b + 4096;
}

// The forms of the pass over V values that a sort uses: a 64-bit value is a lone
// payload, carried by a one-segment key, which is always packed and decoded; a
// key of several segments carries the 32-bit row index, reads the columns at
// first and gathers at last.
#define GHB_EACH_PASS(DO)           \
  do {                              \
    DO(kSrcPacked, kDstPacked);     \
    DO(kSrcPacked, kDstDecode);     \
    if constexpr (sizeof(V) == 4) { \
      DO(kSrcPacked, kDstGather);   \
      DO(kSrcCols, kDstPacked);     \
      DO(kSrcCols, kDstGather);     \
      DO(kSrcPerm, kDstPacked);     \
      DO(kSrcPerm, kDstGather);     \
    }                               \
  } while (0)

template <typename V>
static void launch_pass(int src, int dst, int grid, size_t dyn, cudaStream_t s, const PassParams& pp) {
#define GHB_PASS(S, D) \
  if (src == S && dst == D) sort_pass_kernel<V, S, D><<<grid, kSortThreads, dyn, s>>>(pp)
  GHB_EACH_PASS(GHB_PASS);
#undef GHB_PASS
}

template <typename V>
static int32_t set_smem(ghb_ctx* ctx, size_t dyn) {
#define GHB_ATTR(S, D) \
  if (int32_t st = ensure_dyn_smem(ctx, (const void*)sort_pass_kernel<V, S, D>, dyn)) return st
  GHB_EACH_PASS(GHB_ATTR);
#undef GHB_ATTR
  return GHB_OK;
}
#undef GHB_EACH_PASS

// kb / vb: key and value ping-pong buffers; packed: kb[0] / vb[0] already
// hold the packed keys and values of a one-segment key.
template <typename V>
static int32_t run_passes(ghb_ctx* ctx, PassParams& pp, const std::vector<Segment>& segs,
                          const std::vector<std::vector<int>>& run, const uint32_t* d_hist,
                          uint64_t* const kb[2], void* const vbv[2], uint32_t* const words[2], bool packed, int shift0,
                          cudaStream_t stream) {
  int32_t st;
  const bool finish = shift0 > 0;   // the passes leave the lower bits to the finish
  int total = 0;
  for (auto& r : run) total += (int)r.size();
  ctx->sort_passes = total;
  ctx->sort_finish = finish;
  const int64_t n = pp.n;
  V* vb[2] = {(V*)vbv[0], (V*)vbv[1]};
  const bool multi = segs.size() > 1;
  if (total == 0) {
    int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8);
    sort_identity_kernel<V><<<grid, 256, 0, stream>>>(pp, (const V*)nullptr);
    GHB_LAUNCH_CHECK(ctx);
    return GHB_OK;
  }
  // look-back words: each pass zeroes the ones of the pass after it
  GHB_CUDA_TRY(ctx, cudaMemsetAsync(words[0], 0, (size_t)pp.ntiles * kBins * 4, stream));
  const size_t dyn = (size_t)kSortTile * 8;
  if ((st = set_smem<V>(ctx, dyn))) return st;
  int per_sm = 0;
  if ((st = resident_ctas(ctx, (const void*)sort_pass_kernel<V, kSrcPacked, kDstPacked>, kSortThreads, dyn, &per_sm)))
    return st;
  int pgrid = (int)std::min<int64_t>(pp.ntiles, (int64_t)ctx->num_sms * std::max(1, per_sm));
  int done = 0;
  bool have_perm = false;  // a previous pass left the row order in vb[cur]
  int cur = 0;
  for (size_t s = 0; s < segs.size(); s++) {
    pp.seg = segs[s];
    for (size_t i = 0; i < run[s].size(); i++) {
      int q = run[s][i];
      bool last = ++done == total;
      int src = i == 0 ? (have_perm ? kSrcPerm : packed ? kSrcPacked : kSrcCols) : kSrcPacked;
      int dst = last && !finish ? (multi ? kDstGather : kDstDecode) : kDstPacked;
      pp.shift = shift0 + q * kDigitBits;
      pp.hist = d_hist + ((size_t)s * kMaxPasses + q) * kBins;
      pp.keys_in = kb[cur];
      pp.vals_in = vb[cur];
      pp.keys_out = kb[cur ^ 1];
      pp.vals_out = vb[cur ^ 1];
      pp.status = words[done & 1 ? 0 : 1];
      pp.status_next = last ? nullptr : words[done & 1];
      launch_pass<V>(src, dst, pgrid, dyn, stream, pp);
      GHB_LAUNCH_CHECK(ctx);
      cur ^= 1;
      have_perm = true;
    }
  }
  if (finish) {
    pp.keys_in = kb[cur];
    pp.vals_in = vb[cur];
    pp.keys_out = kb[cur ^ 1];
    pp.vals_out = vb[cur ^ 1];
    pp.shift = shift0;
    const int fgrid = (int)((n + kFinTile - 1) / kFinTile);
    const int lgrid = (int)std::min<int64_t>(n / kFinTile + 1, ctx->num_sms);
    if constexpr (sizeof(V) == 4)   // a wide key carries the row index
      if (pp.wide) {
        sort_finish_kernel<V, true><<<fgrid, kSortThreads, 0, stream>>>(pp);
        GHB_LAUNCH_CHECK(ctx);
        sort_finish_long_kernel<V, true><<<lgrid, kLongThreads, 0, stream>>>(pp);
        GHB_LAUNCH_CHECK(ctx);
        return GHB_OK;
      }
    sort_finish_kernel<V, false><<<fgrid, kSortThreads, 0, stream>>>(pp);
    GHB_LAUNCH_CHECK(ctx);
    sort_finish_long_kernel<V, false><<<lgrid, kLongThreads, 0, stream>>>(pp);
    GHB_LAUNCH_CHECK(ctx);
  }
  return GHB_OK;
}

// How many leading digits of a one-segment key of `bits` bits the passes
// sort by, from the sample's pair counts; 0: all of them.  In units of a
// thirtieth of a pass (14 us at 60M rows): the finish costs 38 where a last
// pass that decodes costs 40, and each row has n * pairs / S^2 others in its
// run, cheap while one thread sorts the run in registers (60M rows of about
// six to a run: 0.56 ms) and dear beyond it (1M rows: the finish takes 15 us
// at one or two rows to a run, 40 at 25, a pass 17).  Rows expected in runs of
// more than 32 are never left to the finish.
static int leading_digits(int bits, int64_t n, const unsigned long long* pairs, int S, int first) {
  const int all = (bits + kDigitBits - 1) / kDigitBits;
  int best = 0;
  double cost = 30.0 * all + 10;
  for (int q = first; q * kDigitBits < bits && q <= 8; q++) {
    const double mates = (double)n * (double)pairs[q] / ((double)S * S);
    if (mates > 32) continue;
    const double c = 30.0 * q + 38 + 0.5 * mates + 2.0 * std::max(0.0, mates - 6);
    if (c < cost) {
      cost = c;
      best = q;
    }
  }
  return best;
}

// Digit histograms of one segment's keys (np digits from bit shift0 up); with
// keys_out the packed keys and the carried values are written too.
static int32_t launch_hist(ghb_ctx* ctx, const KeySet& K, const Segment& seg, int64_t n, int np, int shift0,
                           uint32_t* d_hist, uint64_t* keys_out, void* vals_out, bool wide, bool carry_rowid,
                           const ghb_column* payload, int grid, cudaStream_t stream) {
  HistParams hp;
  hp.shift0 = shift0;
  hp.K = K;
  hp.seg = seg;
  hp.n = n;
  hp.npasses = np;
  hp.hist = d_hist;
  for (int i = 0; i < seg.n; i++) {
    const SubField& sf = seg.f[i];
    const KeyField& kf = K.k[sf.key];
    SubPlan& sp = hp.sub[i];
    sp.col = kf.col;
    sp.umin = kf.umin;
    sp.shift = sf.shift;
    sp.is_flag = sf.is_flag;
    sp.desc = (int8_t)kf.desc;
    sp.nulls_first = (int8_t)kf.nulls_first;
    sp.has_null = (int8_t)kf.has_null;
  }
  hp.keys_out = keys_out;
  hp.vals_out = vals_out;
  hp.vals_wide = wide ? 1 : 0;
  hp.carry_rowid = carry_rowid ? 1 : 0;
  hp.pay_src = carry_rowid ? ghb_column{} : payload[0];
  // 16-byte loads and stores when every column read allows them
  auto vec_ok = [](const ghb_column& c) {
    return c.null_mode != GHB_NULLS_BYTEMAP && ((uintptr_t)c.data & 15) == 0;
  };
  hp.vec = 1;
  for (int i = 0; i < seg.n; i++) hp.vec &= vec_ok(hp.sub[i].col) ? 1 : 0;
  if (!carry_rowid) hp.vec &= vec_ok(hp.pay_src) ? 1 : 0;
  if (hp.keys_out && (((uintptr_t)hp.keys_out | (uintptr_t)hp.vals_out) & 15)) hp.vec = 0;
  sort_hist_kernel<<<std::min(grid, ctx->num_sms * 8), 256, 0, stream>>>(hp);
  GHB_LAUNCH_CHECK(ctx);
  return GHB_OK;
}

int32_t sort_impl(ghb_ctx* ctx, const ghb_column* keys, const int32_t* orders,
                  const int32_t* null_orders, int32_t nkeys, const ghb_column* payload,
                  int32_t npayload, ghb_out_column* out_keys, ghb_out_column* out_payload,
                  int32_t* out_rowid, const ghb_sort_cfg* cfg, cudaStream_t stream) {
  (void)cfg;
  if (nkeys < 1 || nkeys > kMaxSortKeys)
    return set_error(ctx, GHB_ERR_INVALID, "nkeys=%d outside [1,%d]", nkeys, kMaxSortKeys);
  if (npayload < 0 || npayload > kMaxSortPay)
    return set_error(ctx, GHB_ERR_INVALID, "npayload=%d outside [0,%d]", npayload, kMaxSortPay);
  int64_t n = 0;
  int32_t st = validate_columns(ctx, keys, nkeys, &n);
  if (st) return st;
  if (npayload) {
    int64_t pn = 0;
    if ((st = validate_columns(ctx, payload, npayload, &pn))) return st;
    if (pn != n) return set_error(ctx, GHB_ERR_INVALID, "payload rows %lld != key rows %lld",
                                  (long long)pn, (long long)n);
  }
  if (n >= (int64_t)INT32_MAX) return set_error(ctx, GHB_ERR_UNSUPPORTED, "sort of 2^31 rows or more");
  if (!out_keys) return set_error(ctx, GHB_ERR_INVALID, "out_keys is NULL");
  for (int j = 0; j < nkeys; j++)
    if (out_keys[j].type != keys[j].type || (!out_keys[j].data && n > 0))
      return set_error(ctx, GHB_ERR_INVALID, "out_keys[%d]: bad type or data", j);
  for (int j = 0; j < npayload; j++)
    if (out_payload[j].type != payload[j].type || (!out_payload[j].data && n > 0))
      return set_error(ctx, GHB_ERR_INVALID, "out_payload[%d]: bad type or data", j);
  if (n == 0) return GHB_OK;

  PassParams pp;
  std::memset(&pp, 0, sizeof(pp));
  KeySet& K = pp.K;
  K.nkeys = nkeys;
  for (int j = 0; j < nkeys; j++) {
    K.k[j].col = keys[j];
    K.k[j].desc = orders && orders[j] == GHB_DESC;
    int no = null_orders ? null_orders[j] : GHB_NULLS_DEFAULT;
    K.k[j].nulls_first = no == GHB_NULLS_FIRST || (no == GHB_NULLS_DEFAULT && !K.k[j].desc);
  }
  if (n <= kSmallRows)
    return sort_small(ctx, K, payload, npayload, out_keys, out_payload, out_rowid, n, stream);
  // one zeroed block: the analysis, the histograms, the count of long runs
  unsigned long long* d_mm = nullptr;
  const size_t stat_bytes = align256(kStatBytes), hist_bytes = (size_t)kMaxSeg * kMaxPasses * kBins * 4;
  if ((st = scratch_alloc(ctx, stat_bytes + hist_bytes + align256(((size_t)n / kFinTile + 2) * 4), (void**)&d_mm,
                          stream)))
    return st;
  uint32_t* d_hist = (uint32_t*)((char*)d_mm + stat_bytes);
  uint32_t* d_long = d_hist + hist_bytes / 4;
  GHB_CUDA_TRY(ctx, cudaMemsetAsync(d_mm, 0, stat_bytes + hist_bytes + 4, stream));
  int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8);
  MinMaxParams mp;
  mp.K = K;
  mp.n = n;
  mp.out = d_mm;
  sort_minmax_kernel<<<grid, 256, 0, stream>>>(mp);
  GHB_LAUNCH_CHECK(ctx);
  // the fewest leading digits whose runs, were the keys spread evenly, would
  // stay at 32 rows; a sample whose one pair stands for few rows
  SampleParams sp;
  sp.first = 1;
  while (sp.first < 4 && (n >> (kDigitBits * sp.first)) > 32) sp.first++;
  sp.S = n > (4 << 20) ? kSampleMax : 1024;
  sp.K = K;
  sp.n = n;
  sp.mm = d_mm;
  sp.pairs = d_mm + 3 * kMaxSortKeys;
  sort_sample_kernel<<<sp.S / kSampleRows, 256, 0, stream>>>(sp);
  GHB_LAUNCH_CHECK(ctx);
  unsigned long long mm[kStatWords];
  GHB_CUDA_TRY(ctx, cudaMemcpyAsync(mm, d_mm, sizeof(mm), cudaMemcpyDeviceToHost, stream));
  GHB_CUDA_TRY(ctx, cudaStreamSynchronize(stream));

  // plan: least significant key first, value bits then its NULL flag above
  std::vector<Segment> segs(1);
  std::memset(&segs[0], 0, sizeof(Segment));
  auto add_sub = [&](int key, int is_flag, int bits) {
    if (bits == 0) return;
    if (segs.back().bits + bits > 64) {
      segs.emplace_back();
      std::memset(&segs.back(), 0, sizeof(Segment));
    }
    Segment& sg = segs.back();
    SubField& sf = sg.f[sg.n++];
    sf.key = (int8_t)key;
    sf.is_flag = (int8_t)is_flag;
    sf.bits = (int8_t)bits;
    sf.shift = (int8_t)sg.bits;
    sg.bits += bits;
  };
  for (int j = nkeys - 1; j >= 0; j--) {
    KeyField& f = K.k[j];
    uint64_t range;
    key_range(mm + 3 * j, &f.umin, &range);
    f.vbits = range == 0 ? 0 : 64 - __builtin_clzll(range);
    f.has_null = mm[3 * j + 2] ? 1 : 0;
    add_sub(j, 0, f.vbits);
    add_sub(j, 1, f.has_null);
  }
  if (segs.size() > (size_t)kMaxSeg) return set_error(ctx, GHB_ERR_UNSUPPORTED, "too many key segments");
  const bool multi = segs.size() > 1;

  // the value: the single payload itself, else the row index
  const bool carry_rowid = multi || out_rowid != nullptr || npayload != 1 ||
                           payload[0].null_mode == GHB_NULLS_BYTEMAP;
  const bool wide = !carry_rowid && type_width(payload[0].type) == 8;
  const size_t vw = wide ? 8 : 4;
  uint64_t* kb[2] = {nullptr, nullptr};
  void* vb[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; i++) {
    if ((st = scratch_alloc(ctx, (size_t)n * 8, (void**)&kb[i], stream))) return st;
    if ((st = scratch_alloc(ctx, (size_t)n * vw, &vb[i], stream))) return st;
  }

  uint32_t* words[2] = {nullptr, nullptr};
  for (int i = 0; i < 2; i++)
    if ((st = scratch_alloc(ctx, (size_t)((n + kSortTile - 1) / kSortTile) * kBins * 4, (void**)&words[i], stream)))
      return st;
  // what every form of the passes shares
  pp.carry_rowid = carry_rowid ? 1 : 0;
  for (int j = 0; j < kMaxSortKeys; j++) {
    pp.dec_vbits[j] = 0;
    pp.dec_vshift[j] = 0;
    pp.dec_fshift[j] = -1;
  }
  if (!carry_rowid) pp.pay_src = payload[0];
  for (int j = 0; j < nkeys; j++) pp.out_keys[j] = out_keys[j];
  pp.npay = npayload;
  for (int j = 0; j < npayload; j++) {
    pp.pay[j] = payload[j];
    pp.out_pay[j] = out_payload[j];
  }
  pp.out_rowid = out_rowid;
  pp.n = n;
  pp.ntiles = (n + kSortTile - 1) / kSortTile;
  pp.counters = ctx->d_counters + 2;
  pp.dev_status = ctx->d_status;
  pp.gave_up = (unsigned int*)(d_mm + kGaveUpWord);
  pp.spin_limit = ctx->spin_limit;
  pp.long_runs = d_long;
  // the leading digits alone, when the finish is to sort the rest
  const unsigned long long* pairs = mm + 3 * kMaxSortKeys;
  int top = leading_digits(multi ? 64 : segs[0].bits, n, pairs, sp.S, sp.first);
  if (multi && top && (double)n * (double)pairs[8] / ((double)sp.S * sp.S) <= 4) {
    // a key wider than 64 bits, few of whose rows share the leading 64: it is
    // sorted as those, the finish comparing the few by their columns, and by
    // every bit after all in the rare case that a long run holds such rows.  An
    // (int32, int64) key of 69 bits, 330k rows with six payloads: nine passes, two
    // of them over unpacked keys, and a gather, 195 us; 95 us now.
    Segment lead;
    std::memset(&lead, 0, sizeof(lead));
    lead.bits = 64;
    int total = 0, off = 0;
    for (int j = 0; j < nkeys; j++) total += K.k[j].vbits + K.k[j].has_null;
    for (int j = nkeys - 1; j >= 0; j--)
      for (int f = 0; f < 2; f++) {
        const int bits = f ? K.k[j].has_null : K.k[j].vbits;
        if (bits > 0 && off + bits > total - 64)
          lead.f[lead.n++] = SubField{(int8_t)j, (int8_t)f, (int8_t)bits, (int8_t)(off - (total - 64))};
        off += bits;
      }
    const int shift0 = 64 - top * kDigitBits;
    if ((st = launch_hist(ctx, K, lead, n, top, shift0, d_hist, kb[0], vb[0], wide, carry_rowid, payload, grid, stream)))
      return st;
    std::vector<std::vector<int>> run(1);
    for (int q = 0; q < top; q++) run[0].push_back(q);
    pp.wide = 1;
    pp.ties = (unsigned int*)(d_mm + kTieWord);
    if ((st = run_passes<uint32_t>(ctx, pp, {lead}, run, d_hist, kb, vb, words, true, shift0, stream))) return st;
    unsigned int ties = 0;
    GHB_CUDA_TRY(ctx, cudaMemcpyAsync(&ties, pp.ties, sizeof(ties), cudaMemcpyDeviceToHost, stream));
    GHB_CUDA_TRY(ctx, cudaStreamSynchronize(stream));
    if (!ties) return GHB_OK;
    pp.wide = 0;
    GHB_CUDA_TRY(ctx, cudaMemsetAsync(d_hist, 0, hist_bytes + 4, stream));   // and the count of long runs
  }
  if (multi) top = 0;
  const int shift0 = top ? segs[0].bits - top * kDigitBits : 0;
  // histograms of every segment, one read each; a one-segment key is packed
  // on the way
  for (size_t s = 0; s < segs.size(); s++) {
    int np = top ? top : (segs[s].bits + kDigitBits - 1) / kDigitBits;
    if (np == 0) continue;
    if ((st = launch_hist(ctx, K, segs[s], n, np, shift0, d_hist + s * kMaxPasses * kBins, multi ? nullptr : kb[0], vb[0],
                          wide, carry_rowid, payload, grid, stream)))
      return st;
  }
  std::vector<std::vector<int>> run(segs.size());
  if (top) {
    for (int q = 0; q < top; q++) run[0].push_back(q);
  } else {
    // every digit is sorted by: the host skips passes whose digit is constant
    std::vector<uint32_t> hist((size_t)segs.size() * kMaxPasses * kBins, 0);
    GHB_CUDA_TRY(ctx, cudaMemcpyAsync(hist.data(), d_hist, hist.size() * 4, cudaMemcpyDeviceToHost, stream));
    GHB_CUDA_TRY(ctx, cudaStreamSynchronize(stream));
    for (size_t s = 0; s < segs.size(); s++) {
      int np = (segs[s].bits + kDigitBits - 1) / kDigitBits;
      for (int q = 0; q < np; q++) {
        bool trivial = false;
        for (int b = 0; b < kBins; b++)
          if (hist[((size_t)s * kMaxPasses + q) * kBins + b] == (uint32_t)n) trivial = true;
        if (!trivial) run[s].push_back(q);
      }
    }
  }

  if (!multi)
    for (int i = 0; i < segs[0].n; i++) {
      const SubField& sf = segs[0].f[i];
      if (sf.is_flag) {
        pp.dec_fshift[sf.key] = sf.shift;
      } else {
        pp.dec_vbits[sf.key] = sf.bits;
        pp.dec_vshift[sf.key] = sf.shift;
      }
    }
  const bool packed = !multi;
  if (wide) return run_passes<uint64_t>(ctx, pp, segs, run, d_hist, kb, vb, words, packed, shift0, stream);
  return run_passes<uint32_t>(ctx, pp, segs, run, d_hist, kb, vb, words, packed, shift0, stream);
}

// ---------------------------------------------------------------- STRING keys
// A STRING sort key compares as Hive's StringExpr.compare (storage-api/src/
// java/org/apache/hadoop/hive/ql/exec/vector/expressions/StringExpr.java:
// 37-47): unsigned bytes, then length.  It is sorted as the tuple
// (chunk 0, ..., chunk m-1, length) of fixed-width keys, chunk i being bytes
// [8i, 8i + 8) big-endian with 0x00 past the end (top bit flipped, so the
// signed order of the int64 is the unsigned order of the bytes): equal
// chunks with a shorter length sort first, as the byte compare does.  A NULL
// string is NULL in every part.
__global__ void __launch_bounds__(256) string_maxlen_kernel(ghb_column c, unsigned long long* out) {
  const int2* aux = (const int2*)c.aux;
  unsigned long long mx = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < c.n; r += (int64_t)gridDim.x * blockDim.x) {
    const int2 ix = aux[r];
    if (ix.x >= 0) mx = max(mx, (unsigned long long)(ix.y - ix.x));
  }
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0 && mx) atomicMax(out, mx);
}

__global__ void __launch_bounds__(256) string_parts_kernel(ghb_column c, int32_t nchunks, int64_t* chunks,
                                                            int32_t* lens, uint8_t* nulls) {
  const int2* aux = (const int2*)c.aux;
  const uint8_t* bytes = (const uint8_t*)c.data;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < c.n; r += (int64_t)gridDim.x * blockDim.x) {
    const int2 ix = aux[r];
    const bool null = ix.x < 0;
    const int len = null ? 0 : ix.y - ix.x;
    nulls[r] = null ? 1 : 0;
    lens[r] = len;
    for (int k = 0; k < nchunks; k++) {
      uint64_t w = 0;
      for (int b = 0; b < 8; b++) {
        const int at = 8 * k + b;
        w = (w << 8) | (at < len ? (uint64_t)bytes[ix.x + at] : 0ull);
      }
      chunks[(int64_t)k * c.n + r] = (int64_t)(w ^ 0x8000000000000000ull);
    }
  }
}

// out[i] = the [start,end) of row rowid[i] of a STRING column (NULL: -1, -1).
__global__ void __launch_bounds__(256) string_gather_kernel(ghb_column c, const int32_t* rowid, int64_t n,
                                                             ghb_out_column out) {
  const int2* aux = (const int2*)c.aux;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int2 ix = aux[rowid[i]];
    ((int2*)out.data)[i] = ix;
    if (out.is_null) out.is_null[i] = ix.x < 0 ? 1 : 0;
  }
}

// ORDER BY with STRING keys: each STRING key becomes its parts; the sort
// runs on the parts with the row ids carried; the STRING outputs are
// gathered from the row ids.
static int32_t sort_with_strings(ghb_ctx* ctx, const ghb_column* keys, const int32_t* orders,
                                 const int32_t* null_orders, int32_t nkeys, const ghb_column* payload,
                                 int32_t npayload, ghb_out_column* out_keys, ghb_out_column* out_payload,
                                 int32_t* out_rowid, const ghb_sort_cfg* cfg, cudaStream_t stream) {
  int64_t n = 0;
  int32_t st = validate_columns(ctx, keys, nkeys, &n, true);
  if (st) return st;
  if (n >= (int64_t)INT32_MAX) return set_error(ctx, GHB_ERR_UNSUPPORTED, "sort of 2^31 rows or more");
  if (!out_keys) return set_error(ctx, GHB_ERR_INVALID, "out_keys is NULL");
  // the longest string of each STRING key (one read, one synchronisation)
  unsigned long long* d_len = nullptr;
  if ((st = scratch_alloc(ctx, 8 * kMaxSortKeys, (void**)&d_len, stream))) return st;
  GHB_CUDA_TRY(ctx, cudaMemsetAsync(d_len, 0, 8 * kMaxSortKeys, stream));
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, (int64_t)ctx->num_sms * 8));
  for (int j = 0; j < nkeys; j++)
    if (keys[j].type == GHB_STRING) {
      string_maxlen_kernel<<<grid, 256, 0, stream>>>(keys[j], d_len + j);
      GHB_LAUNCH_CHECK(ctx);
    }
  unsigned long long len[kMaxSortKeys];
  GHB_CUDA_TRY(ctx, cudaMemcpyAsync(len, d_len, sizeof(len), cudaMemcpyDeviceToHost, stream));
  GHB_CUDA_TRY(ctx, cudaStreamSynchronize(stream));
  std::vector<ghb_column> ek;
  std::vector<int32_t> eo, en;
  std::vector<ghb_out_column> eout;
  for (int j = 0; j < nkeys; j++) {
    const int32_t o = orders ? orders[j] : GHB_ASC, no = null_orders ? null_orders[j] : GHB_NULLS_DEFAULT;
    if (keys[j].type != GHB_STRING) {
      ek.push_back(keys[j]);
      eo.push_back(o);
      en.push_back(no);
      eout.push_back(out_keys[j]);
      continue;
    }
    const int m = (int)((len[j] + 7) / 8);
    if ((int)ek.size() + m + 1 > kMaxSortKeys)
      return set_error(ctx, GHB_ERR_UNSUPPORTED, "STRING sort key %d of up to %llu bytes needs more than %d key "
                       "parts in all", j, len[j], kMaxSortKeys);
    int64_t* chunks = nullptr;
    int32_t* lens = nullptr;
    uint8_t* nulls = nullptr;
    if ((st = scratch_alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 8 * std::max(m, 1), (void**)&chunks, stream)) ||
        (st = scratch_alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 4, (void**)&lens, stream)) ||
        (st = scratch_alloc(ctx, (size_t)std::max<int64_t>(n, 1), (void**)&nulls, stream)))
      return st;
    string_parts_kernel<<<grid, 256, 0, stream>>>(keys[j], m, chunks, lens, nulls);
    GHB_LAUNCH_CHECK(ctx);
    for (int k = 0; k <= m; k++) {
      ghb_column pc{k < m ? GHB_LONG : GHB_INT, GHB_NULLS_BYTEMAP, k < m ? (const void*)(chunks + (int64_t)k * n)
                                                                         : (const void*)lens,
                    nulls, nullptr, n};
      ek.push_back(pc);
      eo.push_back(o);
      en.push_back(no);
      // the parts' sorted values are not kept
      void* od = nullptr;
      if ((st = scratch_alloc(ctx, (size_t)std::max<int64_t>(n, 1) * type_width(pc.type), &od, stream))) return st;
      eout.push_back(ghb_out_column{pc.type, 0, od, nullptr});
    }
  }
  int32_t* rowid = out_rowid;
  if (!rowid && (st = scratch_alloc(ctx, (size_t)std::max<int64_t>(n, 1) * 4, (void**)&rowid, stream))) return st;
  st = sort_impl(ctx, ek.data(), eo.data(), en.data(), (int32_t)ek.size(), payload, npayload, eout.data(),
                 out_payload, rowid, cfg, stream);
  if (st) return st;
  for (int j = 0; j < nkeys; j++)
    if (keys[j].type == GHB_STRING) {
      if (out_keys[j].type != GHB_STRING || (!out_keys[j].data && n > 0))
        return set_error(ctx, GHB_ERR_INVALID, "out_keys[%d]: bad type or data", j);
      string_gather_kernel<<<grid, 256, 0, stream>>>(keys[j], rowid, n, out_keys[j]);
      GHB_LAUNCH_CHECK(ctx);
    }
  return GHB_OK;
}

// Scratch a sort with STRING keys needs beside the sort's own.
static size_t string_sort_scratch_bytes(const ghb_column* keys, int32_t nkeys, int64_t n) {
  size_t b = 4096 + (size_t)n * 4 + 256;
  for (int j = 0; j < nkeys; j++)
    if (keys[j].type == GHB_STRING) b += (size_t)n * (2 * 8 * kMaxSortKeys + 4 + 4 + 1) + 8 * 1024;
  return b;
}

}  // namespace ghb

using namespace ghb;

extern "C" int32_t ghb_sort(ghb_ctx* ctx, const ghb_column* keys, const int32_t* orders,
                            const int32_t* null_orders, int32_t nkeys, const ghb_column* payload,
                            int32_t npayload, ghb_out_column* out_keys, ghb_out_column* out_payload,
                            int32_t* out_rowid, const ghb_sort_cfg* cfg, void* stream) {
  if (!ctx) return GHB_ERR_INVALID;
  CallScope cs(ctx, "sort", (cudaStream_t)stream);
  int64_t n = keys && nkeys > 0 ? keys[0].n : 0;
  cs.rows(n);
  cs.bytes(cols_bytes(keys, nkeys) + cols_bytes(payload, npayload));
  scratch_reset(ctx);
  bool strings = false;
  for (int j = 0; keys && j < nkeys && j < kMaxSortKeys; j++) strings |= keys[j].type == GHB_STRING;
  const size_t extra = strings ? string_sort_scratch_bytes(keys, nkeys, n) : 0;
  int32_t st = scratch_reserve(ctx, sort_scratch_bytes(n) + extra, (cudaStream_t)stream);
  if (st) return cs.done(st);
  ctx->sort_passes = -1;
  if (strings)
    st = sort_with_strings(ctx, keys, orders, null_orders, nkeys, payload, npayload, out_keys, out_payload, out_rowid,
                           cfg, (cudaStream_t)stream);
  else
    st = sort_impl(ctx, keys, orders, null_orders, nkeys, payload, npayload, out_keys, out_payload, out_rowid, cfg,
                   (cudaStream_t)stream);
  cs.passes(ctx->sort_passes, ctx->sort_finish);
  return cs.done(st);
}
