// ghb_range.cuh — the range of a key column's values, read once.
//
// ORDER BY and GROUP BY over several keys pack each key into as many bits as
// its values' range needs; both read the columns once to find it.
#pragma once

#include <type_traits>

#include "ghb_internal.cuh"

namespace ghb {

// Smallest and largest value seen (INT, LONG by value; DOUBLE by its order
// image, sign bit flipped so that it compares as a signed value).
struct RawRange {
  int64_t mn, mx;
  bool null;
};

template <int TYPE>
__device__ __forceinline__ void range_add(RawRange& r, int64_t raw, bool null) {
  r.null |= null;
  if (null) return;
  const int64_t v = TYPE == GHB_DOUBLE ? (int64_t)(flip_f64_bits((uint64_t)raw) ^ 0x8000000000000000ull) : raw;
  r.mn = min(r.mn, v);
  r.mx = max(r.mx, v);
}

// In-band NULL of a value.
template <int TYPE>
__device__ __forceinline__ bool is_sentinel(int64_t raw) {
  if constexpr (TYPE == GHB_INT) return raw == (int64_t)INT32_MAX;
  else if constexpr (TYPE == GHB_LONG) return raw == INT64_MAX;
  else {
    const double d = __longlong_as_double(raw);
    return d != d;
  }
}

// One column by 16-byte loads (a NULL map by one load beside each), U of them
// in flight per thread (the column is read once, evict-first); its rows past
// the last whole vector one at a time.
template <int TYPE, int NULLS>
__device__ __forceinline__ void range_column(const ghb_column& c, int64_t n, int64_t tid, int64_t stride, RawRange& r) {
  constexpr int U = NULLS == GHB_NULLS_BYTEMAP ? 4 : 8;
  using Vec = typename std::conditional<TYPE == GHB_INT, int4, longlong2>::type;
  using Map = typename std::conditional<TYPE == GHB_INT, unsigned int, unsigned short>::type;
  constexpr int W = TYPE == GHB_INT ? 4 : 2;
  const Vec* v = (const Vec*)c.data;
  const Map* m = (const Map*)c.is_null;
  const int64_t nv = n / W;
  auto take = [&](const Vec& x, Map b) {
    if constexpr (TYPE == GHB_INT && NULLS == GHB_NULLS_NONE) {   // 32-bit minima first
      const int lo = min(min(x.x, x.y), min(x.z, x.w)), hi = max(max(x.x, x.y), max(x.z, x.w));
      r.mn = min(r.mn, (int64_t)lo);
      r.mx = max(r.mx, (int64_t)hi);
    } else {
      const int64_t e[4] = {x.x, x.y, TYPE == GHB_INT ? ((const int*)&x)[W == 4 ? 2 : 0] : 0,
                            TYPE == GHB_INT ? ((const int*)&x)[W == 4 ? 3 : 0] : 0};
#pragma unroll
      for (int i = 0; i < W; i++)
        range_add<TYPE>(r, e[i], NULLS == GHB_NULLS_BYTEMAP    ? ((unsigned int)b >> (8 * i) & 0xffu) != 0
                                 : NULLS == GHB_NULLS_SENTINEL ? is_sentinel<TYPE>(e[i])
                                                               : false);
    }
  };
  int64_t b = tid;
  for (; b + (U - 1) * stride < nv; b += U * stride) {
    Vec x[U];
    Map q[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      x[u] = __ldcs(v + b + u * stride);
      q[u] = NULLS == GHB_NULLS_BYTEMAP ? __ldcs(m + b + u * stride) : 0;
    }
#pragma unroll
    for (int u = 0; u < U; u++) take(x[u], q[u]);
  }
  for (; b < nv; b += stride) take(__ldcs(v + b), NULLS == GHB_NULLS_BYTEMAP ? __ldcs(m + b) : 0);
  for (int64_t q = nv * W + tid; q < n; q += stride) {
    const int64_t raw = ld_raw(c, q);
    range_add<TYPE>(r, raw, raw_is_null(c, raw, q));
  }
}

// A column's 16-byte loads are aligned, and its NULL map's loads beside them.
__host__ __device__ inline bool range_vector(const ghb_column& c) {
  return ((uintptr_t)c.data & 15) == 0 &&
         (c.null_mode != GHB_NULLS_BYTEMAP || ((uintptr_t)c.is_null & (c.type == GHB_INT ? 3 : 1)) == 0);
}

// The whole grid (256 threads a CTA) folds column c into out's three words,
// zeroed before: [0] max of ~(order image), [1] max order image, [2] any NULL.
// `desc` complements the images.  Ends with a barrier.
__device__ __forceinline__ void range_to(const ghb_column& c, int64_t n, bool desc, unsigned long long* out) {
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  RawRange r{INT64_MAX, INT64_MIN, false};
#define GHB_RANGE(T)                                                                                        \
  (c.null_mode == GHB_NULLS_NONE       ? range_column<T, GHB_NULLS_NONE>(c, n, tid, stride, r)              \
   : c.null_mode == GHB_NULLS_SENTINEL ? range_column<T, GHB_NULLS_SENTINEL>(c, n, tid, stride, r)          \
                                       : range_column<T, GHB_NULLS_BYTEMAP>(c, n, tid, stride, r))
  if (range_vector(c)) {
    if (c.type == GHB_INT) GHB_RANGE(GHB_INT);
    else if (c.type == GHB_LONG) GHB_RANGE(GHB_LONG);
    else GHB_RANGE(GHB_DOUBLE);
  } else {
    constexpr int U = 4;
    for (int64_t b = tid; b < n; b += U * stride) {
      int64_t raw[U];
#pragma unroll
      for (int u = 0; u < U; u++) raw[u] = b + u * stride < n ? ld_raw(c, b + u * stride) : 0;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int64_t q = b + u * stride;
        if (q >= n) continue;
        const bool null = raw_is_null(c, raw[u], q);
        if (c.type == GHB_DOUBLE) range_add<GHB_DOUBLE>(r, raw[u], null);
        else range_add<GHB_LONG>(r, raw[u], null);
      }
    }
  }
#undef GHB_RANGE
  for (int o = 16; o > 0; o >>= 1) {
    r.mn = min(r.mn, (int64_t)__shfl_down_sync(0xffffffffu, (long long)r.mn, o));
    r.mx = max(r.mx, (int64_t)__shfl_down_sync(0xffffffffu, (long long)r.mx, o));
  }
  const bool wnull = __any_sync(0xffffffffu, r.null);
  // one set of atomics per CTA: every CTA's warps hitting the same three
  // words would serialise at L2
  __shared__ int64_t s_red[2][8];
  __shared__ int s_null[8];
  const int warp = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    s_red[0][warp] = r.mn;
    s_red[1][warp] = r.mx;
    s_null[warp] = wnull;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int64_t mn = r.mn, mx = r.mx;
    bool null = wnull;
    for (int w = 1; w < (int)(blockDim.x >> 5); w++) {
      mn = min(mn, s_red[0][w]);
      mx = max(mx, s_red[1][w]);
      null |= s_null[w] != 0;
    }
    if (mn <= mx) {
      // order images (a value's sign bit flipped); DESC complements them
      uint64_t lo = flip_i64(mn), hi = flip_i64(mx);
      if (desc) {
        const uint64_t t = ~lo;
        lo = ~hi;
        hi = t;
      }
      atomicMax(&out[0], (unsigned long long)~lo);
      atomicMax(&out[1], (unsigned long long)hi);
    }
    if (null) atomicOr(&out[2], 1ull);
  }
  __syncthreads();
}

// Range of a key's order images from its three words; false: no value.
__host__ __device__ __forceinline__ bool key_range(const unsigned long long* mm, uint64_t* umin, uint64_t* range) {
  const uint64_t lo = ~mm[0], hi = mm[1];
  const bool any = lo <= hi;
  *umin = any ? lo : 0;
  *range = any ? hi - lo : 0;
  return any;
}

// Rows r..r+3 (r a multiple of 4) of a column with 16-byte aligned data, as
// raw 64-bit values, by 16-byte loads read once.
__device__ __forceinline__ void load4(const ghb_column& c, int64_t r, int64_t raw[4]) {
  if (c.type == GHB_INT) {
    const int4 x = __ldcs((const int4*)c.data + r / 4);
    raw[0] = x.x;
    raw[1] = x.y;
    raw[2] = x.z;
    raw[3] = x.w;
  } else {
    const longlong2* q = (const longlong2*)c.data + r / 2;
    const longlong2 a = __ldcs(q), b = __ldcs(q + 1);
    raw[0] = a.x;
    raw[1] = a.y;
    raw[2] = b.x;
    raw[3] = b.y;
  }
}

}  // namespace ghb
