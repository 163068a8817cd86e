// ghb_filter.cu — filter with order-preserving stream compaction (F1).
//
// Replaces FilterPredicate::process (gpu_impl/src/Operator/FilterPredicate.cu:
// 434-571: one int32 bitmap per predicate leaf, one thrust::transform per
// AND/OR node) and FilterOperator::clean_data (gpu_impl/src/Operator/
// FilterOperator.cu:36-93: thrust::reduce + thrust::copy_if of row indices,
// D2H of the indices, then a host gather over every column, in place).
//
// One kernel: each CTA claims ranges of rows (whole tiles, about one range
// per resident CTA) in launch order, evaluates the predicate tree a node at a
// time for eight rows per thread, keeps the per-row results as warp ballots in
// shared memory, scans their popcounts across the range, lists the selected
// rows in shared memory, gets the range's global output offset by decoupled
// look-back over earlier ranges, and copies the projected columns of the
// listed rows to their final positions.  No bitmap or index list goes to
// global memory; the output keeps input order (Hive's selected[]).
#include <algorithm>

#include "ghb_ctx.hpp"
#include "ghb_log.hpp"

namespace ghb {

constexpr int kFiltThreads = 256;
constexpr int kFiltItems = 8;   // rows per thread per tile
constexpr int kFiltTile = kFiltThreads * kFiltItems;
constexpr int kFiltWarps = kFiltThreads / 32;
constexpr int kFiltWords = kFiltItems * kFiltWarps;   // ballot words of one tile
constexpr int kFiltMaxTiles = 4;                      // tiles of one claimed range
constexpr int kMaxProj = kMaxCols;
constexpr int kFiltEagerPolls = 2;                    // a smaller look-back bound is not put off
constexpr uint64_t kNotWalked = ~0ull;                // a range whose look-back is still to come

// How a leaf is evaluated.  An integer column against integer literals is a
// test of an interval, in the column's own width; `neg` complements it.
enum LeafKind { kLeafInterval = 0, kLeafDouble = 1, kLeafNotNull = 2, kLeafRow = 3 };

struct LeafPlan {
  int64_t lo, hi;   // kLeafInterval: lo <= x <= hi (an INT column's clamped to 32 bits)
  int32_t kind;
  int32_t neg;
};

struct FilterParams {
  ColSet cols;
  PredProg pred;
  LeafPlan leaf[GHB_MAX_PRED_NODES];
  int32_t nproj;
  int32_t proj[kMaxProj];
  ghb_out_column out[kMaxProj];
  int64_t n;
  int64_t range_rows;            // rows of a claimed range: whole tiles, at most kFiltMaxTiles
  int64_t nranges;
  int64_t cap;
  int64_t* d_out_rows;
  uint64_t* lb;
  uint32_t epoch;
  unsigned long long* counters;  // [0] next range, [1] finished CTAs
  int32_t* status;
  int32_t spin_limit;            // look-back polls before GHB_ERR_TIMEOUT
};

// Bit k: row row0 + k * kFiltThreads (below `end`) passes leaf `node`.  The
// eight rows' values (and NULL bytes) are loaded before any is compared, and
// the leaf's type and mode are decided once for the eight.
__device__ __forceinline__ uint32_t leaf_bits(const FilterParams& p, int node, int64_t row0, int64_t end) {
  const ghb_pred_node& nd = p.pred.nodes[node];
  const LeafPlan& lp = p.leaf[node];
  const ghb_column& c = p.cols.c[nd.col];
  uint32_t bits = 0;
  if (lp.kind == kLeafRow) {   // STRING columns, column against column
#pragma unroll 1
    for (int k = 0; k < kFiltItems; k++) {
      const int64_t row = row0 + k * kFiltThreads;
      if (row < end && eval_leaf(p.pred, nd, p.cols, row)) bits |= 1u << k;
    }
    return bits;
  }
  uint32_t valid = 0;
#pragma unroll
  for (int k = 0; k < kFiltItems; k++) valid |= (row0 + k * kFiltThreads < end ? 1u : 0u) << k;
  uint32_t null = 0;
  if (c.null_mode == GHB_NULLS_BYTEMAP) {
    uint8_t b[kFiltItems];
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) b[k] = valid >> k & 1 ? __ldg(c.is_null + row0 + k * kFiltThreads) : 0;
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) null |= (b[k] ? 1u : 0u) << k;
    if (lp.kind == kLeafNotNull) return valid & ~null;
  }
  const bool sentinel = c.null_mode == GHB_NULLS_SENTINEL;
  if (c.type == GHB_INT && lp.kind != kLeafDouble) {
    int32_t x[kFiltItems];
#pragma unroll
    for (int k = 0; k < kFiltItems; k++)
      x[k] = valid >> k & 1 ? __ldg((const int32_t*)c.data + row0 + k * kFiltThreads) : 0;
    if (sentinel) {
#pragma unroll
      for (int k = 0; k < kFiltItems; k++) null |= (x[k] == INT32_MAX ? 1u : 0u) << k;
    }
    if (lp.kind == kLeafNotNull) return valid & ~null;
    const int32_t lo = (int32_t)lp.lo, hi = (int32_t)lp.hi;
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) bits |= (x[k] >= lo && x[k] <= hi ? 1u : 0u) << k;
    return (lp.neg ? ~bits : bits) & valid & ~null;
  }
  int64_t x[kFiltItems];
  if (c.type == GHB_INT) {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++)
      x[k] = valid >> k & 1 ? __ldg((const int32_t*)c.data + row0 + k * kFiltThreads) : 0;
  } else {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++)
      x[k] = valid >> k & 1 ? __ldg((const long long*)c.data + row0 + k * kFiltThreads) : 0;
  }
  if (sentinel) {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) null |= (raw_is_null(c, x[k], 0) ? 1u : 0u) << k;
  }
  if (lp.kind == kLeafNotNull) return valid & ~null;
  if (lp.kind == kLeafInterval) {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) bits |= (x[k] >= lp.lo && x[k] <= lp.hi ? 1u : 0u) << k;
    return (lp.neg ? ~bits : bits) & valid & ~null;
  }
  const double a = nd.lit_is_double ? nd.lit_d[0] : (double)nd.lit_i[0];
  const double b = nd.lit_is_double ? nd.lit_d[1] : (double)nd.lit_i[1];
#pragma unroll
  for (int k = 0; k < kFiltItems; k++)
    bits |= (cmp_mode<double>(nd.mode, raw_to_f64(c.type, x[k]), a, b) ? 1u : 0u) << k;
  return bits & valid & ~null;
}

// Writes column c's values of kFiltItems listed rows (rows[k] from `base` on,
// k with bit k of `live`) to output rows out0 + i0 + k * kFiltThreads: every
// load is issued before the stores.  A STRING's NULL map is string_nulls'.
template <typename T>
__device__ __forceinline__ void copy_rows(const ghb_column& c, const T* src, const ghb_out_column& o, int64_t base,
                                          const uint32_t (&rows)[kFiltItems], uint32_t live, int64_t at) {
  T* dst = (T*)o.data + at;
  src += base;
  T v[kFiltItems];
  if (live == (1u << kFiltItems) - 1u) {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) v[k] = __ldcs(src + rows[k]);
#pragma unroll
    for (int k = 0; k < kFiltItems; k++) dst[k * kFiltThreads] = v[k];
  } else {
#pragma unroll
    for (int k = 0; k < kFiltItems; k++)
      if (live >> k & 1) v[k] = __ldcs(src + rows[k]);
#pragma unroll
    for (int k = 0; k < kFiltItems; k++)
      if (live >> k & 1) dst[k * kFiltThreads] = v[k];
  }
  if (!o.is_null || c.type == GHB_STRING) return;
  uint8_t b[kFiltItems];
#pragma unroll
  for (int k = 0; k < kFiltItems; k++) {
    b[k] = 0;
    if (!(live >> k & 1) || c.null_mode == GHB_NULLS_NONE) continue;
    if (c.null_mode == GHB_NULLS_BYTEMAP) b[k] = c.is_null[base + rows[k]] != 0;
    else b[k] = raw_is_null(c, (int64_t)v[k], 0);
  }
#pragma unroll
  for (int k = 0; k < kFiltItems; k++)
    if (live >> k & 1) o.is_null[at + k * kFiltThreads] = b[k];
}

// NULL map of `count` listed rows of a STRING column: a row is NULL by its pair
// (start < 0), whatever the column's null mode.  Out of line and apart from
// copy_rows, whose registers spill with that test (two leaves over nullable
// columns of 40M rows: 395 us with it there, 372 apart).
__device__ __noinline__ void string_nulls(const int2* pairs, const uint16_t* list, int count, uint8_t* is_null) {
  for (int i = threadIdx.x; i < count; i += kFiltThreads) is_null[i] = pairs[list[i]].x < 0;
}

// Each CTA claims ranges of rows in launch order.  Per range: the predicate
// tree of every row, kept as warp ballots; one scan of the ballots' counts,
// published for the look-back of later ranges, and the list of the selected
// rows in shared memory.  Then, when the next claimed range has been through
// the same (so that the ranges before it have had time to publish), the
// range's global output offset by look-back (one per range, not per tile) and
// the projected columns of the listed rows.  The parameters stay in the
// constant bank (__grid_constant__): the string leaves' out-of-line compare
// takes references into them, which would otherwise copy the whole parameter
// block to every thread's stack.
//
// Bound by the latency of its loads at three CTAs per SM (78 registers; DRAM
// 42-50 % busy).  One B200, before (a row's whole tree interpreted at a time,
// one range at a time) and now: d < cut on 6M rows, half pass, 71 -> 48 us;
// the same on 40M rows 400 -> 300 us; two leaves over nullable columns, 6 % of
// 40M rows pass, 1076 -> 281 us.  Measured and not kept: four, five or six CTAs
// at 64, 48 or 40 registers (spills: 6M rows 72, 79 and 104 us against 57 in
// one sitting), the predicate columns of a range a round of claims ahead
// prefetched into L2 (308 against 281 us for the two leaves), one range at a
// time with its look-back before its copies (65 us).
__global__ void __launch_bounds__(kFiltThreads, 3) filter_kernel(const __grid_constant__ FilterParams p) {
  constexpr int kWords = kFiltMaxTiles * kFiltWords;
  constexpr int kRangeRows = kFiltMaxTiles * kFiltTile;
  static_assert(kWords == kFiltThreads, "a ballot word per thread");
  static_assert(kRangeRows <= 65536, "a listed row is 16 bits");
  static_assert(kFiltItems == 8, "a node's results of a thread are a byte");
  static_assert(GHB_MAX_PRED_NODES * kFiltThreads <= kRangeRows * 2, "the nodes' results fit a list");
  __shared__ int64_t s_range;
  __shared__ uint32_t s_mask[kWords];       // ballot words in row order: (tile, item, warp)
  __shared__ uint16_t s_list[2][kRangeRows];   // selected rows of two ranges; before a list is made,
                                               // each node's results
  __shared__ uint32_t s_wsum[kFiltWarps];
  __shared__ uint64_t s_excl[2];            // the ranges' output offsets
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;

  // selects: the rows of range r that pass, listed in s_list[buf]; their number
  auto select = [&](int64_t r, int buf) -> uint32_t {
    const int64_t base = r * p.range_rows;
    const int64_t end = min(p.n, base + p.range_rows);
    const int tiles = (int)((end - base + kFiltTile - 1) / kFiltTile);
    uint8_t* node = (uint8_t*)s_list[buf] + threadIdx.x;
    for (int t = 0; t < tiles; t++) {
      const int64_t row0 = base + (int64_t)t * kFiltTile + threadIdx.x;
      uint32_t bits = 0;
      if (p.pred.n_nodes == 0) {
#pragma unroll
        for (int k = 0; k < kFiltItems; k++) bits |= (row0 + k * kFiltThreads < end ? 1u : 0u) << k;
      } else {
        // post-order: AND / OR read their children's results
        for (int q = 0; q < p.pred.n_nodes; q++) {
          const ghb_pred_node& nd = p.pred.nodes[q];
          if (nd.mode == GHB_FILTER_AND) bits = node[nd.child[0] * kFiltThreads] & node[nd.child[1] * kFiltThreads];
          else if (nd.mode == GHB_FILTER_OR) bits = node[nd.child[0] * kFiltThreads] | node[nd.child[1] * kFiltThreads];
          else bits = leaf_bits(p, q, row0, end);
          if (q + 1 < p.pred.n_nodes) node[q * kFiltThreads] = (uint8_t)bits;
        }
      }
#pragma unroll
      for (int k = 0; k < kFiltItems; k++) {
        const unsigned b = __ballot_sync(0xffffffffu, bits >> k & 1u);
        if (lane == 0) s_mask[(t * kFiltItems + k) * kFiltWarps + warp] = b;
      }
    }
    __syncthreads();
    // scan of the words' counts in row order, a word per thread; word w is
    // rows 32 w on
    const uint32_t mask = (int)threadIdx.x < tiles * kFiltWords ? s_mask[threadIdx.x] : 0;
    uint32_t incl = __popc(mask);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_wsum[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kFiltWarps; w++) {
      before += w < warp ? s_wsum[w] : 0;
      total += s_wsum[w];
    }
    if (warp == 0) {
      if (lane == 0) lookback_publish(p.lb, p.epoch, r, total);
      // a bound of one poll is set to run out: it is spent here, where the earlier
      // ranges are still at work, and not after the next range, when they have
      // published (20M rows: 200 of 200 calls run out here, none there)
      uint64_t ex = kNotWalked;
      if (p.spin_limit < kFiltEagerPolls) {
        __syncwarp();
        ex = lookback_walk(p.lb, p.epoch, r, total, p.status, p.spin_limit);
      }
      if (lane == 0) s_excl[buf] = ex;
    }
    // the warp lists the rows of its 32 words, a word at a time
    const uint32_t off = before + incl - __popc(mask);
#pragma unroll 4
    for (int w = 0; w < 32; w++) {
      const uint32_t m = __shfl_sync(0xffffffffu, mask, w), o = __shfl_sync(0xffffffffu, off, w);
      if (m >> lane & 1u)
        s_list[buf][o + __popc(m & ((1u << lane) - 1u))] = (uint16_t)((warp * 32 + w) * 32 + lane);
    }
    return total;
  };

  int64_t pending = -1;     // the range selected last, not written yet
  uint32_t pending_rows = 0;
  int buf = 0;
  while (true) {
    claim_tile(&p.counters[0], &s_range);
    const int64_t r = s_range;
    uint32_t rows = 0;
    if (r < p.nranges) rows = select(r, buf);
    if (pending >= 0) {
      if (warp == 0) {
        uint64_t ex = s_excl[buf ^ 1];
        if (ex == kNotWalked)
          ex = lookback_walk(p.lb, p.epoch, pending, pending_rows, p.status, p.spin_limit);
        if (lane == 0) {
          s_excl[buf ^ 1] = ex;
          if (pending == p.nranges - 1) *p.d_out_rows = (int64_t)(ex + pending_rows);
          if ((int64_t)(ex + pending_rows) > p.cap) raise_status(p.status, kDevCapacity);
        }
      }
      __syncthreads();
      const int64_t out0 = (int64_t)s_excl[buf ^ 1], base = pending * p.range_rows;
      const int count = (int)max((int64_t)0, min((int64_t)pending_rows, p.cap - out0));
      const uint16_t* list = s_list[buf ^ 1];
      for (int i = threadIdx.x; i < count; i += kFiltItems * kFiltThreads) {
        uint32_t row[kFiltItems], live = 0;
#pragma unroll
        for (int k = 0; k < kFiltItems; k++) {
          const bool in = i + k * kFiltThreads < count;
          row[k] = in ? list[i + k * kFiltThreads] : 0;
          live |= (in ? 1u : 0u) << k;
        }
        for (int j = 0; j < p.nproj; j++) {
          const ghb_column& c = p.cols.c[p.proj[j]];
          // LONG, DOUBLE bits, or a STRING row's [start,end) pair into the same bytes
          if (c.type == GHB_INT) copy_rows<int>(c, (const int*)c.data, p.out[j], base, row, live, out0 + i);
          else
            copy_rows<long long>(c, (const long long*)(c.type == GHB_STRING ? c.aux : c.data), p.out[j], base, row,
                                 live, out0 + i);
        }
      }
      for (int j = 0; j < p.nproj; j++)
        if (p.cols.c[p.proj[j]].type == GHB_STRING && p.out[j].is_null)
          string_nulls((const int2*)p.cols.c[p.proj[j]].aux + base, list, count, p.out[j].is_null + out0);
    }
    if (r >= p.nranges) break;
    pending = r;
    pending_rows = rows;
    buf ^= 1;
    __syncthreads();   // the list just written out is the next range's; s_range and s_excl are read
  }
  claim_finish(p.counters);
}

// The leaf's plan: an integer column's comparison with integers as an interval.
static LeafPlan plan_leaf(const ghb_pred_node& nd, const ghb_column* cols) {
  LeafPlan l{0, 0, kLeafRow, 0};
  const int type = cols[nd.col].type;
  if (type == GHB_STRING) return l;
  if (nd.mode == GHB_FILTER_NOT_NULL) {
    l.kind = kLeafNotNull;
    return l;
  }
  if (nd.col2 >= 0) return l;
  if (type == GHB_DOUBLE || nd.lit_is_double) {
    l.kind = kLeafDouble;
    return l;
  }
  l.kind = kLeafInterval;
  const int64_t a = nd.lit_i[0], b = nd.lit_i[1];
  bool empty = false;
  int64_t lo = INT64_MIN, hi = INT64_MAX;
  auto above = [&](int64_t v) { v == INT64_MAX ? (void)(empty = true) : (void)(lo = v + 1); };
  auto below = [&](int64_t v) { v == INT64_MIN ? (void)(empty = true) : (void)(hi = v - 1); };
  switch (nd.mode) {
    case GHB_FILTER_NOT_EQ: l.neg = 1;   // fall through
    case GHB_FILTER_EQ: lo = hi = a; break;
    case GHB_FILTER_LE: hi = a; break;
    case GHB_FILTER_GE: lo = a; break;
    case GHB_FILTER_LT: below(a); break;
    case GHB_FILTER_GT: above(a); break;
    case GHB_FILTER_NOT_EQ_RANGE: l.neg = 1;   // fall through
    case GHB_FILTER_RANGE:
      above(a);
      below(b);
      break;
    case GHB_FILTER_NOT_RANGE: l.neg = 1;   // fall through
    case GHB_FILTER_EQ_RANGE:
      lo = a;
      hi = b;
      break;
    default: l.kind = kLeafRow; return l;
  }
  if (type == GHB_INT) {   // compared in 32 bits
    if (lo > INT32_MAX || hi < INT32_MIN) empty = true;
    lo = std::max<int64_t>(lo, INT32_MIN);
    hi = std::min<int64_t>(hi, INT32_MAX);
  }
  if (empty || lo > hi) {   // no value
    lo = 1;
    hi = 0;
  }
  l.lo = lo;
  l.hi = hi;
  return l;
}

int32_t filter_impl(ghb_ctx* ctx, const ghb_predicate* pred, const ghb_column* cols, int32_t ncols,
                    const int32_t* proj, int32_t nproj, ghb_out_column* out, int64_t out_capacity,
                    int64_t* d_out_rows, cudaStream_t stream) {
  int64_t n = 0;
  int32_t st = validate_columns(ctx, cols, ncols, &n, true);
  if (st) return st;
  if (nproj < 0 || nproj > kMaxProj) return set_error(ctx, GHB_ERR_INVALID, "nproj=%d", nproj);
  if (nproj > 0 && (!proj || !out)) return set_error(ctx, GHB_ERR_INVALID, "proj/out is NULL");
  if (!d_out_rows) return set_error(ctx, GHB_ERR_INVALID, "d_out_rows is NULL");
  if (out_capacity < 0) return set_error(ctx, GHB_ERR_INVALID, "negative out_capacity");
  FilterParams p;
  std::memset(&p, 0, sizeof(p));
  st = build_pred_prog(ctx, pred, cols, ncols, &p.pred);
  if (st) return st;
  for (int j = 0; j < nproj; j++) {
    if (proj[j] < 0 || proj[j] >= ncols)
      return set_error(ctx, GHB_ERR_INVALID, "projection %d: column %d out of range", j, proj[j]);
    if (out[j].type != cols[proj[j]].type)
      return set_error(ctx, GHB_ERR_INVALID, "projection %d: output type %d differs from input %d", j,
                       out[j].type, cols[proj[j]].type);
    if (!out[j].data && out_capacity > 0)
      return set_error(ctx, GHB_ERR_INVALID, "projection %d: output data is NULL", j);
    p.proj[j] = proj[j];
    p.out[j] = out[j];
  }
  for (int k = 0; k < p.pred.n_nodes; k++)
    if (p.pred.nodes[k].mode != GHB_FILTER_AND && p.pred.nodes[k].mode != GHB_FILTER_OR)
      p.leaf[k] = plan_leaf(p.pred.nodes[k], cols);
  for (int i = 0; i < ncols; i++) p.cols.c[i] = cols[i];
  p.cols.n = ncols;
  p.nproj = nproj;
  p.n = n;
  p.cap = out_capacity;
  p.d_out_rows = d_out_rows;
  p.status = ctx->d_status;
  p.counters = ctx->d_counters;
  p.spin_limit = ctx->spin_limit;
  if (n == 0) {
    GHB_CUDA_TRY(ctx, cudaMemsetAsync(d_out_rows, 0, sizeof(int64_t), stream));
    return GHB_OK;
  }
  int per_sm = 0;
  if ((st = resident_ctas(ctx, (const void*)filter_kernel, kFiltThreads, 0, &per_sm))) return st;
  const int64_t slots = (int64_t)ctx->num_sms * std::max(1, per_sm);
  // one range per resident CTA where the rows allow, in whole tiles
  const int64_t ntiles = (n + kFiltTile - 1) / kFiltTile;
  const int64_t per = std::min<int64_t>(kFiltMaxTiles, std::max<int64_t>(1, (ntiles + slots - 1) / slots));
  p.range_rows = per * kFiltTile;
  p.nranges = (ntiles + per - 1) / per;
  st = lookback_prepare(ctx, p.nranges, &p.epoch, stream);
  if (st) return st;
  p.lb = ctx->lb_status;
  int grid = (int)std::min<int64_t>(p.nranges, slots);
  filter_kernel<<<grid, kFiltThreads, 0, stream>>>(p);
  GHB_LAUNCH_CHECK(ctx);
  return GHB_OK;
}

}  // namespace ghb

using namespace ghb;

extern "C" int32_t ghb_filter(ghb_ctx* ctx, const ghb_predicate* pred, const ghb_column* cols,
                              int32_t ncols, const int32_t* proj, int32_t nproj, ghb_out_column* out,
                              int64_t out_capacity, int64_t* d_out_rows, void* stream) {
  if (!ctx) return GHB_ERR_INVALID;
  CallScope cs(ctx, "filter", (cudaStream_t)stream);
  cs.rows(ncols > 0 && cols ? cols[0].n : 0);
  cs.bytes(cols_bytes(cols, ncols));
  scratch_reset(ctx);
  return cs.done(filter_impl(ctx, pred, cols, ncols, proj, nproj, out, out_capacity, d_out_rows,
                             (cudaStream_t)stream));
}
