// ghb_sort_small.cuh — ORDER BY of a few thousand rows by one CTA.
//
// The sort of a group-by's result is a few thousand rows: the general path
// spends its time on launches and on the host's waits for the keys' ranges and
// histograms.  Here one CTA finds the ranges, packs the keys, sorts them with
// the same stable 8-bit passes in shared memory (by the leading digits when
// they leave short runs) and writes the output columns: one launch, no scratch,
// no host wait.
#pragma once

namespace ghb {

constexpr int kSmallRows = 8192;      // rows one CTA sorts at most
constexpr int kSmallRow = kBins + 1;  // digit words of a warp, padded: a digit's threads read eight warps' words
constexpr int kSmallLead = 2;         // leading digits the passes sort by when the rest orders short runs
constexpr int kSmallRun = 48;         // longest run of equal leading digits put in order by counting

struct SmallSortParams {
  int32_t nkeys;
  ghb_column key[kMaxSortKeys];
  int8_t desc[kMaxSortKeys];
  int8_t nulls_first[kMaxSortKeys];
  ghb_out_column out_key[kMaxSortKeys];
  int32_t npay;
  ghb_column pay[kMaxSortPay];
  ghb_out_column out_pay[kMaxSortPay];
  int32_t* out_rowid;
  int32_t n;
};

// Shared memory of the kernel for TH threads of IT rows: the packed keys, the
// per-warp digit words, the row indices.
template <int TH, int IT>
constexpr size_t small_sort_smem() {
  return (size_t)TH * IT * 8 + (size_t)(TH / 32) * kSmallRow * 8 + (size_t)TH * IT * 2;
}

// Bit k: raw[k], of row row[k], is NULL (k with bit k of `live`); the NULL
// bytes are loaded together.
template <int N>
__device__ __forceinline__ uint32_t small_nulls(const ghb_column& c, const int64_t* raw, const uint32_t* row,
                                                uint32_t live) {
  uint32_t m = 0;
  if (c.null_mode == GHB_NULLS_NONE) return 0;
  if (c.null_mode == GHB_NULLS_BYTEMAP) {
    uint8_t b[N];
#pragma unroll
    for (int k = 0; k < N; k++) b[k] = live >> k & 1 ? __ldg(c.is_null + row[k]) : 0;
#pragma unroll
    for (int k = 0; k < N; k++) m |= (b[k] ? 1u : 0u) << k;
    return m;
  }
#pragma unroll
  for (int k = 0; k < N; k++) m |= (live >> k & 1 && raw_is_null(c, raw[k], 0) ? 1u : 0u) << k;
  return m;
}

// Writes rows idx[k] (row of position pos0 + 32 k, k with bit k of `live`) of
// column c (all threads of the CTA).
template <int IT>
__device__ __forceinline__ void small_gather(const ghb_column& c, const ghb_out_column& o, const uint32_t (&idx)[IT],
                                             int pos0, uint32_t live) {
  int64_t raw[IT];
  uint32_t pos[IT];
#pragma unroll
  for (int k = 0; k < IT; k++) {
    raw[k] = live >> k & 1 ? ld_raw(c, idx[k]) : 0;
    pos[k] = (uint32_t)(pos0 + 32 * k);
  }
  const uint32_t nulls = small_nulls<IT>(c, raw, idx, live);
  __syncthreads();   // the column is read whole before it is written: a column may be sorted in place
  put_rows<IT>(o, c.type, raw, nulls, pos, live);
}

// One SM's shared-memory path bounds it (about 40 wavefronts per 32 rows and
// pass).  With the host's waits gone a sort of 1000 rows by a 10-bit key with
// six payloads takes 77 us from Python where the general path took 146 (kernel
// 10 us); 7007 rows by two keys, 17 bits, four payloads 45 us; 4000 rows by
// 64-bit keys 24 us, 44 with all eight digits, where the general path's
// kernels and copies take 78 and 60 us beside two waits of the host.
template <int TH, int IT>
__global__ void __launch_bounds__(TH) sort_small_kernel(const __grid_constant__ SmallSortParams p) {
  constexpr int kSmallThreads = TH, kSmallWarps = TH / 32, kParts = TH / kBins;
  static_assert(kSmallWarps == 8 * kParts && kSmallWarps <= 32, "a digit's threads take eight warps each");
  extern __shared__ uint64_t s_dyn_small[];
  uint64_t* s_key = s_dyn_small;
  unsigned long long* s_cnt = (unsigned long long*)(s_key + kSmallThreads * IT);   // [warp][digit]
  uint16_t* s_idx = (uint16_t*)(s_cnt + kSmallWarps * kSmallRow);
  __shared__ long long s_red[2][kSmallWarps];
  __shared__ int s_null[kSmallWarps];
  __shared__ uint32_t s_wsum[kSmallWarps];
  // per key: its least image and where its value and NULL flag bits lie
  __shared__ uint64_t s_umin[kMaxSortKeys];
  __shared__ int8_t s_vseg[kMaxSortKeys], s_vshift[kMaxSortKeys], s_fseg[kMaxSortKeys], s_fshift[kMaxSortKeys];
  __shared__ int s_nseg, s_bits;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int pos0 = warp * (32 * IT) + lane;   // a thread's positions: pos0 + 32 k
  uint32_t live = 0;                          // bit k: the position holds a row
  uint32_t idx[IT];
#pragma unroll
  for (int k = 0; k < IT; k++) {
    live |= (pos0 + 32 * k < p.n ? 1u : 0u) << k;
    idx[k] = min(pos0 + 32 * k, p.n - 1);
  }
  if (threadIdx.x == 0) {
    s_nseg = 0;
    s_bits = 0;
  }
  // ranges, least significant key first; thread 0 places each key's bits
  for (int j = p.nkeys - 1; j >= 0; j--) {
    const ghb_column& c = p.key[j];
    long long mn = INT64_MAX, mx = INT64_MIN;
    int64_t raw[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) raw[k] = ld_raw(c, idx[k]);
    const uint32_t nulls = small_nulls<IT>(c, raw, idx, live);
#pragma unroll
    for (int k = 0; k < IT; k++) {
      if (!((live & ~nulls) >> k & 1)) continue;
      uint64_t u = key_image(c, raw[k]);
      if (p.desc[j]) u = ~u;
      const long long v = (long long)(u ^ 0x8000000000000000ull);   // the images' order as signed values
      mn = min(mn, v);
      mx = max(mx, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      mn = min(mn, __shfl_down_sync(0xffffffffu, mn, o));
      mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
    }
    const bool wnull = __any_sync(0xffffffffu, nulls != 0);
    if (lane == 0) {
      s_red[0][warp] = mn;
      s_red[1][warp] = mx;
      s_null[warp] = wnull;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      bool anynull = false;
      for (int w = 0; w < kSmallWarps; w++) {
        mn = min(mn, s_red[0][w]);
        mx = max(mx, s_red[1][w]);
        anynull |= s_null[w] != 0;
      }
      const bool any = mn <= mx;
      s_umin[j] = any ? (uint64_t)mn ^ 0x8000000000000000ull : 0;
      const uint64_t range = any ? (uint64_t)mx - (uint64_t)mn : 0;
      const int vbits = range == 0 ? 0 : 64 - __clzll((long long)range);
      s_vseg[j] = s_fseg[j] = -1;
      s_vshift[j] = s_fshift[j] = 0;
      for (int f = 0; f < 2; f++) {   // the value's bits, then the NULL flag above them
        const int bits = f ? (anynull ? 1 : 0) : vbits;
        if (bits == 0) continue;
        if (s_bits + bits > 64 || s_nseg == 0) {
          s_nseg++;
          s_bits = 0;
        }
        (f ? s_fseg : s_vseg)[j] = (int8_t)(s_nseg - 1);
        (f ? s_fshift : s_vshift)[j] = (int8_t)s_bits;
        s_bits += bits;
      }
    }
    __syncthreads();
  }
  for (int seg = 0; seg < s_nseg; seg++) {
    // the segment's packed keys, in the order the segments before it left;
    // positions past the end carry the key ~0 and stay where they are
    uint64_t key[IT];
#pragma unroll
    for (int k = 0; k < IT; k++) key[k] = 0;
    for (int j = 0; j < p.nkeys; j++) {
      const bool val = s_vseg[j] == seg, flag = s_fseg[j] == seg;
      if (!val && !flag) continue;
      const ghb_column& c = p.key[j];
      int64_t raw[IT];
#pragma unroll
      for (int k = 0; k < IT; k++) raw[k] = ld_raw(c, idx[k]);
      const uint32_t nulls = small_nulls<IT>(c, raw, idx, live);
#pragma unroll
      for (int k = 0; k < IT; k++) {
        const bool null = nulls >> k & 1;
        uint64_t u = key_image(c, raw[k]);
        if (p.desc[j]) u = ~u;
        if (val && !null) key[k] |= (u - s_umin[j]) << s_vshift[j];
        if (flag && null != (bool)p.nulls_first[j]) key[k] |= 1ull << s_fshift[j];
      }
    }
    // bits that differ between keys (of this position's neighbour or first key)
    const uint64_t first = __shfl_sync(0xffffffffu, key[0], 0);
    uint64_t diff = 0;
#pragma unroll
    for (int k = 0; k < IT; k++) {
      if (live >> k & 1) diff |= key[k] ^ first;
      else key[k] = ~0ull;
    }
    if (lane == 0) s_red[0][warp] = (long long)first;
    const uint32_t dlo = __reduce_or_sync(0xffffffffu, (uint32_t)diff);
    const uint32_t dhi = __reduce_or_sync(0xffffffffu, (uint32_t)(diff >> 32));
    if (lane == 0) s_red[1][warp] = (long long)((uint64_t)dhi << 32 | dlo);
    __syncthreads();
    uint64_t differ = 0;
    for (int w = 0; w < kSmallWarps; w++)
      if (w * 32 * IT < p.n) differ |= (uint64_t)s_red[1][w] | (uint64_t)(s_red[0][w] ^ s_red[0][0]);
    auto pass = [&](int sh) {
      if (((differ >> sh) & (kBins - 1)) == 0) return;   // the digit is constant
      for (int i = threadIdx.x; i < kSmallWarps * kSmallRow; i += kSmallThreads) s_cnt[i] = 0;
      __syncthreads();
      uint32_t rank[IT];
#pragma unroll
      for (int k = 0; k < IT; k++) {
        const uint32_t dk = (uint32_t)(key[k] >> sh) & (kBins - 1);
        volatile unsigned long long* word = &s_cnt[warp * kSmallRow + dk];
        atomicOr((unsigned int*)word, 1u << lane);
        __syncwarp();
        const unsigned long long w = *word;
        const uint32_t peers = (uint32_t)w, before = (uint32_t)(w >> 32);
        __syncwarp();
        if ((peers & lt) == 0) *word = (unsigned long long)(before + __popc(peers)) << 32;
        __syncwarp();
        rank[k] = before + __popc(peers & lt);
      }
      __syncthreads();
      // each digit's kParts threads take eight warps' counts apiece: exclusive
      // over the warps, then over the digits
      const int d = threadIdx.x / kParts, w0 = threadIdx.x % kParts * 8;
      uint32_t excl[8], total = 0;
#pragma unroll
      for (int w = 0; w < 8; w++) {
        excl[w] = total;
        total += (uint32_t)(s_cnt[(w0 + w) * kSmallRow + d] >> 32);
      }
      uint32_t incl = total;   // threads in (digit, part) order: one scan does both
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
      }
      if (lane == 31) s_wsum[warp] = incl;
      __syncthreads();
      uint32_t before = lane < warp ? s_wsum[lane] : 0;
      before = __reduce_add_sync(0xffffffffu, before) + incl - total;
#pragma unroll
      for (int w = 0; w < 8; w++) *(uint32_t*)&s_cnt[(w0 + w) * kSmallRow + d] = before + excl[w];
      __syncthreads();
#pragma unroll
      for (int k = 0; k < IT; k++) {
        const uint32_t dk = (uint32_t)(key[k] >> sh) & (kBins - 1);
        const uint32_t at = *(const uint32_t*)&s_cnt[warp * kSmallRow + dk] + rank[k];
        s_key[at] = key[k];
        s_idx[at] = (uint16_t)idx[k];
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < IT; k++) {
        key[k] = s_key[pos0 + 32 * k];
        idx[k] = s_idx[pos0 + 32 * k];
      }
    };
    // the leading digits first: when they leave short runs only, a row's place
    // in its run is counted and the lower digits are spared
    const int cut = s_bits - kSmallLead * kDigitBits;
    bool all = s_nseg > 1 || cut <= 0;
    if (!all) {
      for (int sh = cut; sh < s_bits; sh += kDigitBits) pass(sh);
#pragma unroll
      for (int k = 0; k < IT; k++) s_key[pos0 + 32 * k] = key[k];
      __syncthreads();
      bool far = false;
#pragma unroll
      for (int k = 0; k < IT; k++) {
        const int i = pos0 + 32 * k + kSmallRun;
        far |= i < p.n && (s_key[i] >> cut) == (key[k] >> cut);
      }
      all = __syncthreads_or(far);
      if (!all) {
#pragma unroll
        for (int k = 0; k < IT; k++) {
          if (!(live >> k & 1)) continue;
          const uint64_t lead = key[k] >> cut;
          int at = pos0 + 32 * k;
          for (int j = at - 1; j >= 0; j--) {
            const uint64_t x = s_key[j];
            if (x >> cut != lead) break;
            at -= x > key[k];
          }
          for (int j = pos0 + 32 * k + 1; j < p.n; j++) {
            const uint64_t x = s_key[j];
            if (x >> cut != lead) break;
            at += x < key[k];
          }
          s_idx[at] = (uint16_t)idx[k];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < IT; k++)
          if (live >> k & 1) idx[k] = s_idx[pos0 + 32 * k];
      }
    }
    if (all)
      for (int sh = 0; sh < 64; sh += kDigitBits) pass(sh);
    __syncthreads();   // s_red is the next segment's
  }
  for (int j = 0; j < p.nkeys; j++) small_gather<IT>(p.key[j], p.out_key[j], idx, pos0, live);
  for (int j = 0; j < p.npay; j++) small_gather<IT>(p.pay[j], p.out_pay[j], idx, pos0, live);
  if (p.out_rowid) {
#pragma unroll
    for (int k = 0; k < IT; k++)
      if (live >> k & 1) p.out_rowid[pos0 + 32 * k] = (int32_t)idx[k];
  }
}

static int32_t sort_small(ghb_ctx* ctx, const KeySet& K, const ghb_column* payload, int32_t npayload,
                          const ghb_out_column* out_keys, const ghb_out_column* out_payload, int32_t* out_rowid,
                          int64_t n, cudaStream_t stream) {
  SmallSortParams p;
  std::memset(&p, 0, sizeof(p));
  p.nkeys = K.nkeys;
  for (int j = 0; j < K.nkeys; j++) {
    p.key[j] = K.k[j].col;
    p.desc[j] = (int8_t)K.k[j].desc;
    p.nulls_first[j] = (int8_t)K.k[j].nulls_first;
    p.out_key[j] = out_keys[j];
  }
  p.npay = npayload;
  for (int j = 0; j < npayload; j++) {
    p.pay[j] = payload[j];
    p.out_pay[j] = out_payload[j];
  }
  p.out_rowid = out_rowid;
  p.n = (int32_t)n;
#define GHB_SMALL(TH, IT)                                                                                \
  do {                                                                                                   \
    constexpr size_t smem = small_sort_smem<TH, IT>();                                                  \
    if (int32_t st = ensure_dyn_smem(ctx, (const void*)sort_small_kernel<TH, IT>, smem)) return st;     \
    sort_small_kernel<TH, IT><<<1, TH, smem, stream>>>(p);                                              \
  } while (0)
  if (n <= 1024) GHB_SMALL(512, 2);
  else if (n <= 4096) GHB_SMALL(1024, 4);
  else GHB_SMALL(1024, 8);
#undef GHB_SMALL
  GHB_LAUNCH_CHECK(ctx);
  return GHB_OK;
}

}  // namespace ghb
