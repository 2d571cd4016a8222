// GROUP BY with aggregates: one row per distinct key.
//
// The reference plans GROUP BY but ignores the groups: AggregateOperator
// folds every row into one accumulator (include/engine/operators/
// aggregate_operator.hpp:84-104). This follows SQL (DuckDB) semantics instead:
// NULL keys form one group; aggregates skip NULL inputs; SUM/AVG/MIN/MAX over
// no non-NULL input is NULL; COUNT(*) counts rows, COUNT(col) non-NULL values;
// float sums accumulate in FP64.
//
// Sort-based, all on the device:
//   yq_sort_indices   stable LSD radix argsort of the key (NULLs last)
//   k_group_heads     head flag at every sorted position whose key differs
//                     from the one before it (-0.0 equals +0.0, NaNs equal)
//   yq_prefix_sum_mask  -> group index of every sorted position, group count
//   k_group_keys      each group's key into the output
//   k_group_tiles     tiles of 2,048 sorted positions (8 a thread), values
//                     read through the permutation: each thread folds its
//                     positions in order, a segmented scan over the block's
//                     threads (fixed tree) completes every group that starts
//                     and ends in the tile and writes its output row; a group
//                     crossing the tile's edges leaves a partial record
//   k_group_span      each group that crosses tiles, from the tile where it
//                     starts: its tiles' partial records folded in tile order
//                     (fixed tree), output row written
// No floating-point atomics: every sum is added in an order fixed by the
// data's sorted layout, so a query gives the same bits on every run.
//
// Integer keys of few distinct values (up to kFewGroups) skip the sort:
//   k_few_find        the distinct keys, through a hash table per block (a NULL
//                     key or too many keys send the call to the sort), and
//                     their ascending order = the group indices
//   k_few_accumulate  one pass over the input columns into accumulators that
//                     each thread owns in shared memory
//   k_few_finish      each group's partials folded in block order
#include <climits>
#include <cstring>

#include "yq_common.cuh"
#include "yq_sort.cuh"

using namespace yq;

namespace {

constexpr int kGroupThreads = 256;

// Key equality of two rows (canonical floats, NULL == NULL).
__device__ __forceinline__ bool same_key(const yq_column& k, uint32_t a, uint32_t b) {
  if (k.nulls) {
    const bool na = k.nulls[a] != 0, nb = k.nulls[b] != 0;
    if (na || nb) return na == nb;
  }
  switch (k.type) {
    case YQ_INT32: return static_cast<const int32_t*>(k.data)[a] == static_cast<const int32_t*>(k.data)[b];
    case YQ_FLOAT32: {
      const float x = static_cast<const float*>(k.data)[a], y = static_cast<const float*>(k.data)[b];
      return x == y || (x != x && y != y);
    }
    case YQ_FLOAT64: {
      const double x = static_cast<const double*>(k.data)[a], y = static_cast<const double*>(k.data)[b];
      return x == y || (x != x && y != y);
    }
    case YQ_TEXT: {
      const uint32_t* p = reinterpret_cast<const uint32_t*>(static_cast<const char*>(k.data) + (size_t)a * k.width);
      const uint32_t* q = reinterpret_cast<const uint32_t*>(static_cast<const char*>(k.data) + (size_t)b * k.width);
      for (int i = 0; i < k.width / 4; ++i)
        if (p[i] != q[i]) return false;
      return true;
    }
    default: return static_cast<const long long*>(k.data)[a] == static_cast<const long long*>(k.data)[b];
  }
}

__global__ void k_group_heads(const yq_column key, const uint32_t* __restrict__ perm, uint32_t rows,
                              uint8_t* __restrict__ head) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x)
    head[i] = (i == 0 || !same_key(key, perm[i], perm[i - 1])) ? 1 : 0;
}

// First input row of every tile of sorted positions (the tiles run in the
// order of these rows: see yq_group_by).
__global__ void k_tile_first_row(const uint32_t* __restrict__ perm, uint32_t ntiles, uint32_t tile_rows,
                                 uint32_t* __restrict__ first) {
  for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x)
    first[t] = __ldg(perm + (size_t)t * tile_rows);
}

// Head flags from the sorted key words (kw words a row, in sorted order): a
// sequential read instead of two reads through the permutation. Key words
// already equate -0.0 with +0.0 and every NaN, and carry the NULL flag.
__global__ void k_group_heads_words(const uint32_t* __restrict__ words, int kw, uint32_t rows,
                                    uint8_t* __restrict__ head) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
    bool h = i == 0;
    for (int j = 0; j < kw && !h; ++j) h = __ldg(words + (size_t)i * kw + j) != __ldg(words + (size_t)(i - 1) * kw + j);
    head[i] = h ? 1 : 0;
  }
}

__global__ void k_group_keys(const yq_column key, const uint32_t* __restrict__ perm, uint32_t rows,
                             const uint8_t* __restrict__ head, const uint32_t* __restrict__ incl, yq_column out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < rows; i += gridDim.x * blockDim.x) {
    if (!head[i]) continue;
    const uint32_t g = incl[i] - 1, r = perm[i];
    const char* src = static_cast<const char*>(key.data) + (size_t)r * key.width;
    char* dst = static_cast<char*>(out.data) + (size_t)g * key.width;
    for (int b = 0; b < key.width; b += 4) *reinterpret_cast<uint32_t*>(dst + b) = *reinterpret_cast<const uint32_t*>(src + b);
    if (out.nulls) const_cast<uint8_t*>(out.nulls)[g] = key.nulls ? key.nulls[r] : 0;
  }
}

struct GAgg {
  const void* data;      // input column (COUNT_STAR: none)
  const uint8_t* nulls;
  int32_t type;          // input type
  int32_t kind;          // yq_agg_kind
  int32_t width;         // of a cell
};

struct GroupParams {
  GAgg a[YQ_MAX_AGGREGATES];
  int32_t nagg;
  uint32_t rows;
  const uint32_t* perm;
  const uint32_t* incl;  // inclusive scan of the head flags: group = incl - 1
  uint32_t* starts;      // [groups + 1] first sorted position of every group; starts[groups] = rows
  yq_column out[YQ_MAX_AGGREGATES];  // aggregate output columns
  unsigned long long* rec;  // [tiles][2][nagg][2]: head / tail partial (count, value) of every tile
  const uint32_t* tile_order;  // [tiles] the tile block b works on (null: tile b)
  uint32_t* tail_group;     // [tiles] group of the tile's tail record
  uint32_t* tile_flags;     // [tiles] kHeadRec | kTailRec | kTailStarted (set with atomicOr)
  uint32_t* err;
};

constexpr uint32_t kGroupItems = 8;
constexpr uint32_t kGroupTile = kGroupThreads * kGroupItems;  // 2,048 sorted positions
constexpr uint32_t kHeadRec = 1, kTailRec = 2, kTailStarted = 4;

// Order-preserving signed 64-bit key of a double (NaN above +inf, one NaN).
__device__ __forceinline__ long long ordered(double d) {
  unsigned long long u = d != d ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(d);
  u = (u >> 63) ? ~u : (u | (1ull << 63));
  return (long long)(u ^ (1ull << 63));
}
__device__ __forceinline__ double unordered(long long k) {
  unsigned long long u = (unsigned long long)k ^ (1ull << 63);
  u = (u >> 63) ? (u & ~(1ull << 63)) : ~u;
  return __longlong_as_double((long long)u);
}

__device__ __forceinline__ bool is_float(int32_t t) { return t == YQ_FLOAT32 || t == YQ_FLOAT64; }

// Input value r of an aggregate as int64 or double.
__device__ __forceinline__ long long in_int(const GAgg& a, uint32_t r) {
  return a.type == YQ_INT32 ? (long long)static_cast<const int32_t*>(a.data)[r]
                            : static_cast<const long long*>(a.data)[r];
}
__device__ __forceinline__ double in_dbl(const GAgg& a, uint32_t r) {
  return a.type == YQ_FLOAT32 ? (double)static_cast<const float*>(a.data)[r] : static_cast<const double*>(a.data)[r];
}

// One aggregate's partial state: a count and a 64-bit value (int64 sum,
// double sum bits, or the ordered key of MIN / MAX).
struct GPart {
  unsigned long long cnt;
  unsigned long long v;
};

__device__ __forceinline__ GPart part_identity(int kind) {
  return GPart{0ull, kind == YQ_AGG_MIN ? (unsigned long long)LLONG_MAX
                     : kind == YQ_AGG_MAX ? (unsigned long long)LLONG_MIN : 0ull};
}

__device__ __forceinline__ GPart part_combine(int kind, bool flt, GPart a, GPart b) {
  GPart c;
  c.cnt = a.cnt + b.cnt;
  switch (kind) {
    case YQ_AGG_SUM:
    case YQ_AGG_AVG:
      c.v = flt ? (unsigned long long)__double_as_longlong(__longlong_as_double((long long)a.v) +
                                                           __longlong_as_double((long long)b.v))
                : a.v + b.v;
      break;
    case YQ_AGG_MIN: c.v = (long long)a.v < (long long)b.v ? a.v : b.v; break;
    case YQ_AGG_MAX: c.v = (long long)a.v > (long long)b.v ? a.v : b.v; break;
    default: c.v = 0ull; break;
  }
  return c;
}

__device__ __forceinline__ void part_add_row(const GAgg& a, bool flt, GPart& p, uint32_t r) {
  if (a.kind == YQ_AGG_COUNT_STAR) {
    ++p.cnt;
    return;
  }
  if (a.nulls && a.nulls[r]) return;
  ++p.cnt;
  if (a.kind == YQ_AGG_SUM || a.kind == YQ_AGG_AVG) {
    if (flt) p.v = (unsigned long long)__double_as_longlong(__longlong_as_double((long long)p.v) + in_dbl(a, r));
    else p.v += (unsigned long long)in_int(a, r);
  } else if (a.kind == YQ_AGG_MIN || a.kind == YQ_AGG_MAX) {
    const long long k = flt ? ordered(in_dbl(a, r)) : in_int(a, r);
    if (a.kind == YQ_AGG_MIN ? k < (long long)p.v : k > (long long)p.v) p.v = (unsigned long long)k;
  }
}

// Output row g of aggregate a from its complete state.
__device__ __forceinline__ void part_write(const GAgg& a, const yq_column& o, uint32_t g, GPart p) {
  const bool flt = is_float(a.type);
  const bool null = p.cnt == 0 && a.kind != YQ_AGG_COUNT && a.kind != YQ_AGG_COUNT_STAR;
  if (o.nulls) const_cast<uint8_t*>(o.nulls)[g] = null ? 1 : 0;
  switch (a.kind) {
    case YQ_AGG_COUNT:
    case YQ_AGG_COUNT_STAR: static_cast<long long*>(o.data)[g] = (long long)p.cnt; break;
    case YQ_AGG_SUM:
      if (flt) static_cast<double*>(o.data)[g] = null ? 0.0 : __longlong_as_double((long long)p.v);
      else static_cast<long long*>(o.data)[g] = null ? 0 : (long long)p.v;
      break;
    case YQ_AGG_AVG: {
      const double sum = flt ? __longlong_as_double((long long)p.v) : (double)(long long)p.v;
      static_cast<double*>(o.data)[g] = null ? 0.0 : sum / (double)p.cnt;
      break;
    }
    default: {  // MIN / MAX in the input type
      const long long k = (long long)p.v;
      if (a.type == YQ_INT32) static_cast<int32_t*>(o.data)[g] = null ? 0 : (int32_t)k;
      else if (a.type == YQ_FLOAT32) static_cast<float*>(o.data)[g] = null ? 0.0f : (float)unordered(k);
      else if (a.type == YQ_FLOAT64) static_cast<double*>(o.data)[g] = null ? 0.0 : unordered(k);
      else static_cast<long long*>(o.data)[g] = null ? 0 : k;
      break;
    }
  }
}

__device__ __forceinline__ GPart shfl_up_part(GPart p, int d) {
  return GPart{__shfl_up_sync(0xffffffffu, p.cnt, d), __shfl_up_sync(0xffffffffu, p.v, d)};
}

// Inclusive segmented scan over the block's threads in thread order (a
// thread's flag restarts the running state); fixed combine tree. Returns the
// inclusive state and flag; excl / excl_flag = the same up to the thread before.
__device__ __forceinline__ void block_seg_scan(int kind, bool flt, bool flag, GPart x, GPart& incl, bool& incl_flag,
                                               GPart& excl, bool& excl_flag, GPart* s_part, uint32_t* s_flag) {
  constexpr int NW = kGroupThreads / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  GPart v = x;
  bool f = flag;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const GPart u = shfl_up_part(v, d);
    const bool uf = __shfl_up_sync(0xffffffffu, f, d);
    if (lane >= d) {
      if (!f) v = part_combine(kind, flt, u, v);
      f = f || uf;
    }
  }
  if (lane == 31) {
    s_part[warp] = v;
    s_flag[warp] = f;
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // warp prefixes in warp order (exclusive), one thread: fixed order
    GPart run = part_identity(kind);
    bool rf = false;
    for (int w = 0; w < NW; ++w) {
      const GPart wv = s_part[w];
      const bool wf = s_flag[w] != 0u;
      s_part[NW + w] = run;
      s_flag[NW + w] = rf;
      run = wf ? wv : part_combine(kind, flt, run, wv);
      rf = rf || wf;
    }
  }
  __syncthreads();
  const GPart wp = s_part[NW + warp];
  const bool wpf = s_flag[NW + warp] != 0u;
  // lane-level exclusive value within the warp
  GPart le = shfl_up_part(v, 1);
  bool lef = __shfl_up_sync(0xffffffffu, f, 1);
  if (lane == 0) {
    le = part_identity(kind);
    lef = false;
  }
  incl = f ? v : part_combine(kind, flt, wp, v);
  incl_flag = f || wpf;
  excl = lef ? le : (lane == 0 ? wp : part_combine(kind, flt, wp, le));
  excl_flag = lef || wpf;
  __syncthreads();
}

__global__ void __launch_bounds__(kGroupThreads) k_group_tiles(const __grid_constant__ GroupParams P) {
  __shared__ GPart s_part[2 * (kGroupThreads / 32)];
  __shared__ uint32_t s_flag[2 * (kGroupThreads / 32)];
  const uint32_t tile = P.tile_order ? __ldg(P.tile_order + blockIdx.x) : blockIdx.x;
  const uint32_t tile0 = tile * kGroupTile;
  const uint32_t tile_end = min(P.rows, tile0 + kGroupTile);
  const uint32_t p0 = tile0 + threadIdx.x * kGroupItems;
  const uint32_t n = p0 < tile_end ? min(kGroupItems, tile_end - p0) : 0u;  // valid positions of this thread
  // A tile inside one group (with few groups, nearly every tile): every
  // aggregate folds over the whole tile by a fixed-order block reduction,
  // with one barrier instead of a segmented scan per aggregate.
  if (tile0 < tile_end && __ldg(P.incl + tile0) == __ldg(P.incl + tile_end - 1)) {
    __shared__ GPart s_u[YQ_MAX_AGGREGATES][kGroupThreads / 32];
    const uint32_t G = __ldg(P.incl + tile0) - 1u;
    const bool starts = tile0 == 0 || __ldg(P.incl + tile0 - 1) - 1u != G;
    const bool ends = tile_end == P.rows || __ldg(P.incl + tile_end) - 1u != G;
    if (threadIdx.x == 0 && starts) P.starts[G] = tile0;
    uint32_t rr[kGroupItems];
#pragma unroll
    for (int q = 0; q < (int)kGroupItems; ++q) rr[q] = (uint32_t)q < n ? __ldg(P.perm + p0 + q) : 0u;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = 0; j < P.nagg; ++j) {
      const GAgg& a = P.a[j];
      const bool flt = is_float(a.type);
      GPart acc = part_identity(a.kind);
#pragma unroll
      for (int q = 0; q < (int)kGroupItems; ++q)
        if ((uint32_t)q < n) part_add_row(a, flt, acc, rr[q]);
      // fixed tree: lanes pairwise in index order
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const GPart o{__shfl_down_sync(0xffffffffu, acc.cnt, d), __shfl_down_sync(0xffffffffu, acc.v, d)};
        if ((lane & (2 * d - 1)) == 0) acc = part_combine(a.kind, flt, acc, o);
      }
      if (lane == 0) s_u[j][warp] = acc;
    }
    __syncthreads();
    if ((int)threadIdx.x < P.nagg) {  // thread j: aggregate j, warps in order
      const int j = threadIdx.x;
      const GAgg& a = P.a[j];
      const bool flt = is_float(a.type);
      GPart tot = s_u[j][0];
      for (int w = 1; w < kGroupThreads / 32; ++w) tot = part_combine(a.kind, flt, tot, s_u[j][w]);
      unsigned long long* head_rec = P.rec + ((size_t)tile * 2 * P.nagg + j) * 2;
      unsigned long long* tail_rec = P.rec + ((size_t)tile * 2 * P.nagg + P.nagg + j) * 2;
      if (starts && ends) {
        part_write(a, P.out[j], G, tot);
      } else if (ends) {  // the group began before this tile and ends at its last position
        head_rec[0] = tot.cnt;
        head_rec[1] = tot.v;
      } else {  // the group goes on past this tile
        tail_rec[0] = tot.cnt;
        tail_rec[1] = tot.v;
      }
    }
    if (threadIdx.x == 0 && P.nagg > 0 && !(starts && ends)) {
      if (ends) {
        atomicOr(P.tile_flags + tile, kHeadRec);
      } else {
        P.tail_group[tile] = G;
        atomicOr(P.tile_flags + tile, kTailRec | (starts ? kTailStarted : 0u));
      }
    }
    return;
  }
  uint32_t g[kGroupItems], r[kGroupItems];
#pragma unroll
  for (int q = 0; q < (int)kGroupItems; ++q) {
    g[q] = (uint32_t)q < n ? __ldg(P.incl + p0 + q) - 1u : 0u;
    r[q] = (uint32_t)q < n ? __ldg(P.perm + p0 + q) : 0u;
  }
  const uint32_t prev_g = p0 > 0 && n ? __ldg(P.incl + p0 - 1) - 1u : 0xffffffffu;
  const uint32_t last = n ? p0 + n - 1 : 0u;
  const uint32_t next_g = n && last + 1 < P.rows ? __ldg(P.incl + last + 1) - 1u : 0xffffffffu;
  // group starts
#pragma unroll
  for (int q = 0; q < (int)kGroupItems; ++q)
    if ((uint32_t)q < n && (q == 0 ? g[0] != prev_g : g[q] != g[q - 1])) P.starts[g[q]] = p0 + q;
  const bool starts_here = n && g[0] != prev_g;
  bool boundary = false;  // a group starts inside (after the first position)
#pragma unroll
  for (int q = 1; q < (int)kGroupItems; ++q) boundary |= (uint32_t)q < n && g[q] != g[q - 1];
  uint32_t g_last = 0u;
#pragma unroll
  for (int q = 0; q < (int)kGroupItems; ++q)
    if ((uint32_t)q + 1 == n) g_last = g[q];
  const bool ends_here = n && next_g != g_last;
  const bool tile_last = n && last + 1 == tile_end;  // the tile's last valid position is this thread's
  for (int j = 0; j < P.nagg; ++j) {
    const GAgg& a = P.a[j];
    const bool flt = is_float(a.type);
    GPart first = part_identity(a.kind), cur = part_identity(a.kind);
    uint32_t cg = g[0];
    int seg = 0;  // segments closed so far in this thread
#pragma unroll
    for (int q = 0; q < (int)kGroupItems; ++q) {
      if ((uint32_t)q >= n) break;
      if (q > 0 && g[q] != cg) {  // the segment of group cg ends before position q
        if (seg == 0) first = cur;                         // the thread's first segment
        else part_write(a, P.out[j], cg, cur);             // an inner segment: complete here
        if (seg == 0 && starts_here) part_write(a, P.out[j], cg, cur);  // first segment began here too
        ++seg;
        cg = g[q];
        cur = part_identity(a.kind);
      }
      part_add_row(a, flt, cur, r[q]);
    }
    // thread element of the scan: the running state of the thread's last segment
    GPart inc, exc;
    bool inc_f, exc_f;
    block_seg_scan(a.kind, flt, n == 0 || starts_here || boundary, cur, inc, inc_f, exc, exc_f, s_part, s_flag);
    if (n == 0) continue;
    unsigned long long* head_rec = P.rec + ((size_t)tile * 2 * P.nagg + j) * 2;
    unsigned long long* tail_rec = P.rec + ((size_t)tile * 2 * P.nagg + P.nagg + j) * 2;
    if (boundary && !starts_here) {
      // the first segment continues a group from earlier threads and ends here
      const GPart tot = part_combine(a.kind, flt, exc, first);
      if (exc_f) {
        part_write(a, P.out[j], g[0], tot);
      } else {  // the group began before this tile: the tile's head record
        head_rec[0] = tot.cnt;
        head_rec[1] = tot.v;
        if (j == 0) atomicOr(P.tile_flags + tile, kHeadRec);
      }
    }
    // the last segment: its state up to here is the inclusive scan value
    if (ends_here) {
      if (inc_f) {
        part_write(a, P.out[j], g_last, inc);
      } else {
        head_rec[0] = inc.cnt;
        head_rec[1] = inc.v;
        if (j == 0) atomicOr(P.tile_flags + tile, kHeadRec);
      }
    } else if (tile_last) {  // the group goes on past this tile
      tail_rec[0] = inc.cnt;
      tail_rec[1] = inc.v;
      if (j == 0) {
        P.tail_group[tile] = g_last;
        atomicOr(P.tile_flags + tile, kTailRec | (inc_f ? kTailStarted : 0u));
      }
    }
  }
}

// One block per tile: the group that starts in this tile and runs past it.
__global__ void __launch_bounds__(kGroupThreads) k_group_span(const __grid_constant__ GroupParams P, uint32_t ntiles) {
  __shared__ GPart s_red[kGroupThreads / 32];
  const uint32_t t = blockIdx.x;
  const uint32_t fl = P.tile_flags[t];
  if (!(fl & kTailRec) || !(fl & kTailStarted)) return;
  const uint32_t g = P.tail_group[t];
  const uint32_t end = P.starts[g + 1];
  if (end == 0 || end > P.rows) {
    if (threadIdx.x == 0) atomicOr(P.err, 2u);
    return;
  }
  const uint32_t tb = (end - 1) / kGroupTile;
  if (tb <= t || tb >= ntiles || !(P.tile_flags[tb] & kHeadRec)) {
    if (threadIdx.x == 0) atomicOr(P.err, 2u);
    return;
  }
  const uint32_t n = tb - t + 1;  // contributions: tail(t), tail(t+1..tb-1), head(tb)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = 0; j < P.nagg; ++j) {
    const GAgg& a = P.a[j];
    const bool flt = is_float(a.type);
    GPart acc = part_identity(a.kind);
    for (uint32_t k = threadIdx.x; k < n; k += kGroupThreads) {
      const uint32_t tt = t + k;
      const unsigned long long* rec =
          P.rec + ((size_t)tt * 2 * P.nagg + (k + 1 == n ? 0 : P.nagg) + j) * 2;  // head of tb, else tail
      acc = part_combine(a.kind, flt, acc, GPart{rec[0], rec[1]});
    }
    // fixed tree: lanes pairwise in index order, then warps in order
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const GPart o{__shfl_down_sync(0xffffffffu, acc.cnt, d), __shfl_down_sync(0xffffffffu, acc.v, d)};
      if ((lane & (2 * d - 1)) == 0) acc = part_combine(a.kind, flt, acc, o);
    }
    if (lane == 0) s_red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      GPart tot = s_red[0];
      for (int w = 1; w < kGroupThreads / 32; ++w) tot = part_combine(a.kind, flt, tot, s_red[w]);
      part_write(a, P.out[j], g, tot);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------- few distinct keys
// With few groups the sort, its permutation and the reads through it are most
// of the work (32M rows, 11 groups, five aggregates: 1.63 ms of kernels, 0.25 ms
// here, for 384 MB of input). Here the input is read once to find the keys and once to
// accumulate. Each thread owns an accumulator per group and aggregate in
// shared memory (element [group][thread], so a warp's 32 updates hit 32
// banks whatever groups its rows belong to) and adds its rows in row order;
// threads, then blocks, fold in a fixed tree. So sums need no atomics and the
// bits do not depend on scheduling. Latency-bound on the shared-memory
// read-modify-writes; eight rows a thread are loaded ahead.
// The group limit is the accumulators' (few_limit): at 28 bytes a thread and
// group, 50 groups leave one block of 128 threads on an SM and 61 fill it.
constexpr int kFewThreads = 128;
constexpr int kFewItems = 8;
constexpr uint32_t kFewGroups = 96;
constexpr uint32_t kFewSlots = 512;          // hash slots, at most a fifth full
constexpr int kFewFindThreads = 256;
constexpr unsigned long long kNoKey = ~0ull;  // empty slot; the key of that value has a flag of its own

struct FewTable {  // all zero on entry
  unsigned long long keys[kFewSlots];  // ~key (0, an empty slot, would be the key kNoKey's)
  uint32_t count, has_last, overflow, ngroups;
  uint32_t last_gid, ticket, err, pad;
  uint32_t gid[kFewSlots];
  unsigned long long group_key[kFewGroups];
};

__device__ __forceinline__ uint32_t few_hash(unsigned long long k) {  // the top 9 bits of a product
  return (((uint32_t)k ^ ((uint32_t)(k >> 32) * 0x85ebca6bu)) * 0x9e3779b1u) >> 23;
}
static_assert(kFewSlots == 512, "few_hash gives nine bits");

// Puts `value` into the table from slot h on (empty slots hold `empty`, which is
// no value to put in); false when that makes more than `limit` values.
template <typename K>
__device__ __forceinline__ bool few_insert(K* table, uint32_t* count, K value, K empty, uint32_t h, uint32_t limit) {
  for (uint32_t n = 0; n < kFewSlots; ++n, h = (h + 1) & (kFewSlots - 1)) {
    K cur = *reinterpret_cast<volatile K*>(table + h);
    if (cur == value) return true;
    if (cur != empty) continue;
    cur = atomicCAS(table + h, empty, value);
    if (cur == empty) return atomicAdd(count, 1u) < limit;
    if (cur == value) return true;
  }
  return false;
}

// Group index of every key: ascending signed order. The keys are compacted
// first, so that each looks at the others and not at every slot. Run by one
// block, whose stores to T the next kernel reads.
template <int BLOCK>
__device__ __forceinline__ void few_order(FewTable* T, int width, uint32_t limit) {
  __shared__ long long s_val[kFewGroups];
  __shared__ uint32_t s_n;
  const volatile FewTable* V = T;  // other blocks wrote it: not from L1
  const bool has_last = V->has_last != 0u;
  const uint32_t n = V->count + (has_last ? 1u : 0u);
  if (V->overflow || n > limit) {
    if (threadIdx.x == 0) T->overflow = 1u;
    return;
  }
  if (threadIdx.x == 0) s_n = 0u;
  __syncthreads();
  auto value_of = [&](unsigned long long k) { return width == 4 ? (long long)(int32_t)(uint32_t)k : (long long)k; };
  for (uint32_t i = threadIdx.x; i < kFewSlots; i += BLOCK) {
    const unsigned long long k = ~V->keys[i];
    if (k != kNoKey) s_val[atomicAdd(&s_n, 1u)] = value_of(k);
  }
  if (threadIdx.x == 0 && has_last) s_val[atomicAdd(&s_n, 1u)] = -1ll;  // the 8-byte key ~0
  __syncthreads();
  auto rank_of = [&](long long v) {
    uint32_t r = 0;
    for (uint32_t j = 0; j < n; ++j) r += s_val[j] < v ? 1u : 0u;
    return r;
  };
  for (uint32_t i = threadIdx.x; i < kFewSlots; i += BLOCK) {
    const unsigned long long k = ~V->keys[i];
    if (k == kNoKey) continue;
    const uint32_t rank = rank_of(value_of(k));
    T->gid[i] = rank;
    T->group_key[rank] = k;
  }
  if (threadIdx.x == 0) {
    if (has_last) {
      const uint32_t rank = rank_of(-1ll);
      T->last_gid = rank;
      T->group_key[rank] = kNoKey;
    }
    T->ngroups = n;
  }
}

// `head` (mapped host memory): whether the table is of no use, and its groups.
// K: the key's bits. Row 0's key is known to be there, so a block's table is
// filled with it: empty slots need no value outside the key's own, and a probe
// is a product, a load and a compare.
template <typename K>
__global__ void __launch_bounds__(kFewFindThreads) k_few_find(const K* __restrict__ keys,
                                                              const uint8_t* __restrict__ nulls, uint32_t rows,
                                                              uint32_t limit, FewTable* T, uint32_t* head) {
  __shared__ K s_keys[kFewSlots];
  __shared__ uint32_t s_count, s_over, s_last;
  const K first = __ldg(keys);
  for (uint32_t i = threadIdx.x; i < kFewSlots; i += kFewFindThreads) s_keys[i] = first;
  if (threadIdx.x == 0) {
    s_count = 1u;
    s_over = 0u;
  }
  __syncthreads();
  constexpr uint32_t STEP = kFewFindThreads * kFewItems;
  bool ok = true;
  for (uint32_t base = blockIdx.x * STEP; base < rows; base += gridDim.x * STEP) {
    // one thread a block reads the other blocks' flag, along with its keys
    const uint32_t over = threadIdx.x == 0 ? ld_relaxed_u32(&T->overflow) : 0u;
    const uint32_t r0 = base + threadIdx.x;
    K k[kFewItems];
    if (base + STEP <= rows) {
      const K* p = keys + r0;
#pragma unroll
      for (int q = 0; q < kFewItems; ++q) k[q] = __ldg(p + q * kFewFindThreads);
    } else {
#pragma unroll
      for (int q = 0; q < kFewItems; ++q) k[q] = r0 + q * kFewFindThreads < rows ? __ldg(keys + r0 + q * kFewFindThreads) : first;
    }
    if (nulls) {  // a NULL group's key cell is its first row's: the sort finds it
#pragma unroll
      for (int q = 0; q < kFewItems; ++q)
        if (r0 + q * kFewFindThreads < rows && __ldg(nulls + r0 + q * kFewFindThreads)) ok = false;
    }
    // all first probes before any insertion: with few keys nearly every one hits
    uint32_t miss = 0u;
#pragma unroll
    for (int q = 0; q < kFewItems; ++q)
      miss |= (k[q] != first && *reinterpret_cast<volatile K*>(s_keys + few_hash(k[q])) != k[q]) ? 1u << q : 0u;
    for (; miss && ok; miss &= miss - 1) {
      const int m = __ffs(miss) - 1;
      K key = k[0];
#pragma unroll
      for (int q = 1; q < kFewItems; ++q)
        if (q == m) key = k[q];
      ok = few_insert<K>(s_keys, &s_count, key, first, few_hash(key), limit);
    }
    if (!ok || over) s_over = 1u;
    // this block or another one has found too many keys: the table is not used
    if (__any_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t*>(&s_over) != 0u)) break;
  }
  __syncthreads();
  if (s_over) {
    if (threadIdx.x == 0) atomicOr(&T->overflow, 1u);
  } else {
    for (uint32_t i = threadIdx.x; i <= kFewSlots; i += kFewFindThreads) {
      const K key = i < kFewSlots ? s_keys[i] : first;
      if (i < kFewSlots && key == first) continue;
      const unsigned long long k = key;
      if (k == kNoKey) atomicOr(&T->has_last, 1u);
      else if (!few_insert<unsigned long long>(T->keys, &T->count, ~k, 0ull, few_hash(k), limit)) atomicOr(&T->overflow, 1u);
    }
  }
  // the last block to get here has every block's keys before it
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&T->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  few_order<kFewFindThreads>(T, (int)sizeof(K), limit);
  if (threadIdx.x == 0) {  // its own stores, or another block's flag
    head[0] = *reinterpret_cast<volatile uint32_t*>(&T->overflow);
    head[1] = T->ngroups;
    __threadfence_system();
  }
}

// What a thread keeps per group, [group][thread] arrays one after another:
// its rows, per nullable input its non-NULL values, per aggregate its value.
struct FewAcc {
  int32_t cnt_off;  // count array of the aggregate (0: the row counts)
  int32_t val_off;  // value array (-1: a count)
  int32_t val_size;
};
// An input column and the aggregates over it (agg[first, first + count) of
// FewParams::order): its cells are read once for all of them.
struct FewCol {
  const void* data;
  const uint8_t* nulls;
  int32_t type, width;  // width 0: only counted, no cell is read
  int32_t first, count;
  int32_t cnt_off;  // non-NULL counts (with nulls)
};
struct FewParams {
  GroupParams P;
  yq_column key;
  FewAcc acc[YQ_MAX_AGGREGATES];
  FewCol col[YQ_MAX_AGGREGATES];
  int32_t ncol;
  int8_t order[YQ_MAX_AGGREGATES];
  int32_t bytes;      // of all arrays, for one group and thread
  uint32_t ngroups;
  uint32_t rows_per_block;
  const FewTable* T;
  GPart* part;        // [blocks][groups][nagg]
  uint32_t* host_err; // mapped host memory
  yq_column out_key;
};

__device__ __forceinline__ int32_t ordered32(float f) {
  uint32_t u = f != f ? 0x7fc00000u : __float_as_uint(f);
  u = (u >> 31) ? ~u : (u | 0x80000000u);
  return (int32_t)(u ^ 0x80000000u);
}
// ordered32's keys as ordered() gives them for the same value in double.
__device__ __forceinline__ long long widen_ordered32(int32_t k) {
  uint32_t u = (uint32_t)k ^ 0x80000000u;
  u = (u >> 31) ? (u & 0x7fffffffu) : ~u;
  return ordered((double)__uint_as_float(u));
}

// Raw cells of a thread's rows of one input column (4-byte cells zero-extended).
// Rows r0, r0 + kFewThreads, ...; the ones at or past `rows` read the last row.
template <typename T, typename V>
__device__ __forceinline__ void few_cells(const void* data, uint32_t r0, uint32_t rows, V (&v)[kFewItems]) {
  if (r0 + (kFewItems - 1) * kFewThreads < rows) {
    const T* p = static_cast<const T*>(data) + r0;
#pragma unroll
    for (int q = 0; q < kFewItems; ++q) v[q] = __ldg(p + q * kFewThreads);
  } else {
#pragma unroll
    for (int q = 0; q < kFewItems; ++q) v[q] = __ldg(static_cast<const T*>(data) + min(r0 + q * kFewThreads, rows - 1u));
  }
}
__device__ __forceinline__ void few_load(const FewCol& c, uint32_t r0, uint32_t rows,
                                         unsigned long long (&v)[kFewItems]) {
  if (c.width == 4) few_cells<uint32_t>(c.data, r0, rows, v);
  else if (c.width == 8) few_cells<unsigned long long>(c.data, r0, rows, v);
}

// One aggregate over a thread's rows: f folds a cell into the accumulator.
// `e`: each row's element of an accumulator array; `all`: every row of every
// thread of the warp counts (no test a row).
template <typename A, typename F>
__device__ __forceinline__ void few_fold(char* val, const unsigned long long (&v)[kFewItems],
                                         const uint32_t (&e)[kFewItems], uint32_t use, bool all, F f) {
  A* const acc = reinterpret_cast<A*>(val);
  if (all) {
#pragma unroll
    for (int q = 0; q < kFewItems; ++q) acc[e[q]] = f(acc[e[q]], v[q]);
  } else {
#pragma unroll
    for (int q = 0; q < kFewItems; ++q)
      if (use >> q & 1u) acc[e[q]] = f(acc[e[q]], v[q]);
  }
}

// A key's slot and its group index side by side: one load a probe.
template <typename K>
struct FewSlot {
  K key;
  K gid;  // kNoGroup: empty
};
constexpr uint32_t kNoGroup = 0xffffffffu;

template <typename K>
__global__ void __launch_bounds__(kFewThreads, 5) k_few_accumulate(const __grid_constant__ FewParams F) {
  extern __shared__ __align__(16) char s_few[];
  FewSlot<K>* s_slot = reinterpret_cast<FewSlot<K>*>(s_few);
  char* s_acc = s_few + kFewSlots * sizeof(FewSlot<K>);
  const uint32_t G = F.ngroups, tid = threadIdx.x;
  const size_t unit = (size_t)G * kFewThreads;  // elements of one array
  for (uint32_t i = tid; i < kFewSlots; i += kFewThreads) {
    const unsigned long long key = ~F.T->keys[i];
    s_slot[i].key = (K)key;
    s_slot[i].gid = key == kNoKey ? (K)kNoGroup : (K)F.T->gid[i];
  }
  for (size_t i = tid * 4; i < unit * F.bytes; i += kFewThreads * 4) *reinterpret_cast<uint32_t*>(s_acc + i) = 0u;
  __syncthreads();
  for (int j = 0; j < F.P.nagg; ++j) {  // MIN / MAX start at their identity
    const int kind = F.P.a[j].kind;
    if (kind != YQ_AGG_MIN && kind != YQ_AGG_MAX) continue;
    for (uint32_t g = 0; g < G; ++g) {
      char* p = s_acc + unit * F.acc[j].val_off + (size_t)(g * kFewThreads + tid) * F.acc[j].val_size;
      if (F.acc[j].val_size == 4) *reinterpret_cast<int32_t*>(p) = kind == YQ_AGG_MIN ? INT_MAX : INT_MIN;
      else *reinterpret_cast<long long*>(p) = kind == YQ_AGG_MIN ? LLONG_MAX : LLONG_MIN;
    }
  }
  uint32_t* const rows_acc = reinterpret_cast<uint32_t*>(s_acc);
  constexpr uint32_t STEP = kFewThreads * kFewItems;
  const uint32_t rows = F.P.rows;
  const uint32_t r_begin = blockIdx.x * F.rows_per_block;  // a whole number of steps
  const uint32_t r_end = min(rows, r_begin + F.rows_per_block);
  const uint32_t last_gid = F.T->last_gid;
  // The keys of the next step and the next column's cells are always in flight
  // while the current ones are folded.
  K k[kFewItems];
  few_cells<K>(F.key.data, r_begin + tid, rows, k);
  for (uint32_t base = r_begin; base < r_end; base += STEP) {
    const uint32_t r0 = base + tid;
    uint32_t g[kFewItems], in = (1u << kFewItems) - 1u;
    unsigned long long v[kFewItems];
    if (base + STEP > r_end) {
#pragma unroll
      for (int q = 0; q < kFewItems; ++q)
        if (r0 + q * kFewThreads >= r_end) in &= ~(1u << q);
    }
    if (F.ncol) few_load(F.col[0], r0, rows, v);
#pragma unroll
    for (int q = 0; q < kFewItems; ++q) {
      uint32_t h = few_hash(k[q]);
      FewSlot<K> at = s_slot[h];
      if (sizeof(K) == 8 && (unsigned long long)k[q] == kNoKey) {
        at.gid = (K)last_gid;
      } else {
        for (uint32_t n = 0; n < kFewSlots && at.key != k[q]; ++n) {  // a collision (rare)
          h = (h + 1) & (kFewSlots - 1);
          at = s_slot[h];
        }
      }
      g[q] = (uint32_t)at.gid;
    }
#pragma unroll
    for (int q = 0; q < kFewItems; ++q) {
      if (g[q] >= G) {  // cannot be: k_few_find saw every key
        if (in >> q & 1u) atomicOr(F.P.err, kErrBounds);
        in &= ~(1u << q);
        g[q] = 0u;
      }
      g[q] = g[q] * kFewThreads + tid;  // its element from here on
    }
    if (base + STEP < r_end) few_cells<K>(F.key.data, r0 + STEP, rows, k);
#pragma unroll
    for (int q = 0; q < kFewItems; ++q)
      if (in >> q & 1u) ++rows_acc[g[q]];
    for (int c = 0; c < F.ncol; ++c) {
      const FewCol& C = F.col[c];
      unsigned long long next[kFewItems];
      if (c + 1 < F.ncol) few_load(F.col[c + 1], r0, rows, next);
      uint32_t use = in;
      if (C.nulls) {
        uint32_t* cnt = reinterpret_cast<uint32_t*>(s_acc + unit * C.cnt_off);
        uint8_t nul[kFewItems];
#pragma unroll
        for (int q = 0; q < kFewItems; ++q) nul[q] = __ldg(C.nulls + min(r0 + q * kFewThreads, rows - 1u));
#pragma unroll
        for (int q = 0; q < kFewItems; ++q)
          if (use >> q & 1u) {
            if (nul[q]) use &= ~(1u << q);
            else ++cnt[g[q]];
          }
      }
      const bool all = __all_sync(0xffffffffu, use == (1u << kFewItems) - 1u);
      for (int x = C.first; x < C.first + C.count; ++x) {
        const int j = F.order[x];
        if (F.acc[j].val_off < 0) continue;  // a count
        char* const val = s_acc + unit * F.acc[j].val_off;
        const int kind = F.P.a[j].kind;
        if (kind == YQ_AGG_SUM || kind == YQ_AGG_AVG) {
          if (C.type == YQ_FLOAT32)
            few_fold<double>(val, v, g, use, all, [](double s, unsigned long long b) { return s + (double)__uint_as_float((uint32_t)b); });
          else if (C.type == YQ_FLOAT64)
            few_fold<double>(val, v, g, use, all, [](double s, unsigned long long b) { return s + __longlong_as_double((long long)b); });
          else if (C.type == YQ_INT32)
            few_fold<unsigned long long>(val, v, g, use, all, [](unsigned long long s, unsigned long long b) {
              return s + (unsigned long long)(long long)(int32_t)(uint32_t)b;
            });
          else
            few_fold<unsigned long long>(val, v, g, use, all, [](unsigned long long s, unsigned long long b) { return s + b; });
        } else {
          const bool lo = kind == YQ_AGG_MIN;
          if (C.type == YQ_FLOAT32)
            few_fold<int32_t>(val, v, g, use, all, [lo](int32_t s, unsigned long long b) {
              const int32_t o = ordered32(__uint_as_float((uint32_t)b));
              return lo ? min(s, o) : max(s, o);
            });
          else if (C.type == YQ_INT32)
            few_fold<int32_t>(val, v, g, use, all, [lo](int32_t s, unsigned long long b) {
              return lo ? min(s, (int32_t)(uint32_t)b) : max(s, (int32_t)(uint32_t)b);
            });
          else if (C.type == YQ_FLOAT64)
            few_fold<long long>(val, v, g, use, all, [lo](long long s, unsigned long long b) {
              const long long o = ordered(__longlong_as_double((long long)b));
              return lo ? min(s, o) : max(s, o);
            });
          else
            few_fold<long long>(val, v, g, use, all, [lo](long long s, unsigned long long b) {
              return lo ? min(s, (long long)b) : max(s, (long long)b);
            });
        }
      }
#pragma unroll
      for (int q = 0; q < kFewItems; ++q) v[q] = next[q];
    }
  }
  __syncthreads();
  // each (group, aggregate): the block's threads folded by one warp, a lane's
  // threads in order and then the lanes pairwise
  const int lane = tid & 31, warp = tid >> 5;
  for (uint32_t x = warp; x < G * (uint32_t)F.P.nagg; x += kFewThreads / 32) {
    const uint32_t g = x / F.P.nagg;
    const int j = (int)(x % F.P.nagg);
    const GAgg& a = F.P.a[j];
    const FewAcc& A = F.acc[j];
    const bool flt = is_float(a.type);
    GPart acc = part_identity(a.kind);
#pragma unroll
    for (int t = 0; t < kFewThreads / 32; ++t) {
      const size_t e = (size_t)g * kFewThreads + t * 32 + lane;
      GPart p;
      p.cnt = reinterpret_cast<const uint32_t*>(s_acc + unit * A.cnt_off)[e];
      p.v = 0ull;
      if (A.val_off >= 0) {
        const char* val = s_acc + unit * A.val_off;
        if (A.val_size == 8) p.v = reinterpret_cast<const unsigned long long*>(val)[e];
        else {
          const int32_t v = reinterpret_cast<const int32_t*>(val)[e];
          p.v = p.cnt == 0 ? part_identity(a.kind).v
                           : (unsigned long long)(a.type == YQ_FLOAT32 ? widen_ordered32(v) : (long long)v);
        }
      }
      acc = part_combine(a.kind, flt, acc, p);
    }
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const GPart o{__shfl_down_sync(0xffffffffu, acc.cnt, d), __shfl_down_sync(0xffffffffu, acc.v, d)};
      if ((lane & (2 * d - 1)) == 0) acc = part_combine(a.kind, flt, acc, o);
    }
    if (lane == 0) F.part[((size_t)blockIdx.x * G + g) * F.P.nagg + j] = acc;
  }
}

// One block per (group, aggregate): the blocks' partials in a fixed order (a
// thread's in block order, lanes pairwise, then the warps).
constexpr int kFinishThreads = 128;
__global__ void __launch_bounds__(kFinishThreads) k_few_finish(const __grid_constant__ FewParams F, uint32_t nblocks) {
  __shared__ GPart s_part[kFinishThreads / 32];
  const uint32_t g = blockIdx.x;
  const int j = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (j == 0 && threadIdx.x == 0) {
    const unsigned long long k = F.T->group_key[g];
    if (F.out_key.width == 4) static_cast<uint32_t*>(F.out_key.data)[g] = (uint32_t)k;
    else static_cast<unsigned long long*>(F.out_key.data)[g] = k;
    if (F.out_key.nulls) const_cast<uint8_t*>(F.out_key.nulls)[g] = 0;
    if (g == 0) {
      *F.host_err = *F.P.err;
      __threadfence_system();
    }
  }
  if (j >= F.P.nagg) return;
  const GAgg& a = F.P.a[j];
  const bool flt = is_float(a.type);
  GPart acc = part_identity(a.kind);
#pragma unroll 4
  for (uint32_t b = threadIdx.x; b < nblocks; b += kFinishThreads)
    acc = part_combine(a.kind, flt, acc, F.part[((size_t)b * F.ngroups + g) * F.P.nagg + j]);
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const GPart o{__shfl_down_sync(0xffffffffu, acc.cnt, d), __shfl_down_sync(0xffffffffu, acc.v, d)};
    if ((lane & (2 * d - 1)) == 0) acc = part_combine(a.kind, flt, acc, o);
  }
  if (lane == 0) s_part[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    GPart tot = s_part[0];
    for (int w = 1; w < kFinishThreads / 32; ++w) tot = part_combine(a.kind, flt, tot, s_part[w]);
    part_write(a, F.P.out[j], g, tot);
  }
}

int out_type(int32_t kind, int32_t in) {
  switch (kind) {
    case YQ_AGG_COUNT:
    case YQ_AGG_COUNT_STAR: return YQ_INT64;
    case YQ_AGG_SUM: return (in == YQ_FLOAT32 || in == YQ_FLOAT64) ? YQ_FLOAT64 : YQ_INT64;
    case YQ_AGG_AVG: return YQ_FLOAT64;
    default: return in;
  }
}

int type_width(int32_t t) { return (t == YQ_INT32 || t == YQ_FLOAT32) ? 4 : 8; }

unsigned grid_for(uint64_t n, unsigned per_block) {
  const uint64_t g = (n + per_block - 1) / per_block;
  return (unsigned)(g < 1 ? 1 : (g > 65535 ? 65535 : g));
}

// Blocks the accumulation runs at most (its partials are sized for them).
constexpr int kFewBlocksPerSm = 8;

size_t few_workspace_bytes(int32_t nagg) {
  WsSize w;
  w.add<FewTable>(1);
  w.add<GPart>((size_t)sm_count() * kFewBlocksPerSm * kFewGroups * (nagg > 0 ? nagg : 1));
  return w.total();
}

// Rows from which the search for few distinct keys is made. One that fails
// stops within its first steps and costs two launches and a wait, 19 us; where
// it succeeds the call takes 76 us instead of 170 (100K rows, 11 groups, five
// aggregates), and from 130K rows on, where the sort's path also orders its
// tiles, 67 instead of 247.
constexpr uint32_t kFewMinRows = 100000;

// (Above 2^30 rows the sort refuses the call, and 32-bit row arithmetic ends.)
bool few_applies(const yq_column& key, uint32_t rows) {
  return rows >= kFewMinRows && rows < (1u << 30) && (key.type == YQ_INT32 || key.type == YQ_INT64 || key.type == YQ_DATETIME);
}

// The accumulators of a call's aggregates: which arrays a thread keeps per group.
void few_layout(const GroupParams& P, FewParams& F) {
  auto value_size = [&](int j) {
    const GAgg& a = P.a[j];
    if (a.kind == YQ_AGG_COUNT || a.kind == YQ_AGG_COUNT_STAR) return 0;
    return a.kind == YQ_AGG_SUM || a.kind == YQ_AGG_AVG || a.width == 8 ? 8 : 4;
  };
  // An array begins its offset times the elements of one array (a multiple of
  // 128) into the room, so it is aligned whatever its element size.
  int off = 4;  // the row counts
  F.ncol = 0;
  int placed = 0;
  for (int j = 0; j < P.nagg; ++j) F.acc[j] = FewAcc{0, -1, 0};
  for (int j = 0; j < P.nagg; ++j) {
    if (P.a[j].kind == YQ_AGG_COUNT_STAR || (P.a[j].kind == YQ_AGG_COUNT && !P.a[j].nulls)) continue;  // the row count
    bool seen = false;
    for (int i = 0; i < placed; ++i) seen |= F.order[i] == j;
    if (seen) continue;
    FewCol& C = F.col[F.ncol++];
    C = FewCol{P.a[j].data, P.a[j].nulls, P.a[j].type, 0, placed, 0, 0};
    if (C.nulls) {
      C.cnt_off = off;
      off += 4;
    }
    for (int i = j; i < P.nagg; ++i) {
      const GAgg& a = P.a[i];
      if (a.kind == YQ_AGG_COUNT_STAR || a.data != C.data || a.nulls != C.nulls || a.type != C.type) continue;
      F.order[placed++] = (int8_t)i;
      ++C.count;
      if (a.kind != YQ_AGG_COUNT) C.width = a.width;
      F.acc[i].cnt_off = C.cnt_off;
    }
  }
  for (int j = 0; j < P.nagg; ++j) {
    if (value_size(j) == 0) continue;
    F.acc[j].val_off = off;
    F.acc[j].val_size = value_size(j);
    off += value_size(j);
  }
  F.bytes = off;
}

size_t few_smem(int key_width, uint32_t groups, int bytes) {
  return (size_t)kFewSlots * 2 * key_width + (size_t)groups * kFewThreads * bytes;
}

// Groups whose accumulators a block has room for. The search for the keys stops
// at it: a key of more values is known after its first rows instead of after
// the whole column.
constexpr size_t kFewSmem = 220 * 1024;
uint32_t few_limit(int key_width, int bytes) {
  const size_t n = (kFewSmem - few_smem(key_width, 0, 0)) / ((size_t)kFewThreads * bytes);
  return n < kFewGroups ? (uint32_t)n : kFewGroups;
}

// The sort-free path. *done = false: the keys are too many (or one is NULL)
// and nothing was written.
int group_by_few(const GroupParams& P, const yq_column& key, const yq_column& out_key, uint32_t capacity,
                 uint32_t* groups, void* few_ws, size_t few_bytes, cudaStream_t s, bool* done) {
  *done = false;
  FewParams F;
  F.P = P;
  few_layout(P, F);
  const uint32_t limit = few_limit(key.width, F.bytes);
  if (limit == 0) return YQ_OK;
  Workspace ws;
  YQ_TRY(ws.acquire(few_ws, few_bytes, few_workspace_bytes(P.nagg), s));
  FewTable* T = ws.take<FewTable>(1);
  GPart* part = ws.take<GPart>((size_t)sm_count() * kFewBlocksPerSm * kFewGroups * (P.nagg > 0 ? P.nagg : 1));
  // one memset, and each kernel leaves the host's words itself: a search that
  // fails costs two launches and a wait
  MappedWords m;
  YQ_TRY(m.acquire());
  YQ_TRY_CUDA(cudaMemsetAsync(T, 0, sizeof(FewTable), s));
  const unsigned step = kFewFindThreads * kFewItems;
  unsigned grid = grid_for(P.rows, step);
  const void* find = key.width == 4 ? (const void*)k_few_find<uint32_t> : (const void*)k_few_find<unsigned long long>;
  const unsigned resident = (unsigned)(sm_count() * kernel_blocks_per_sm(find, kFewFindThreads, 0));
  if (grid > resident) grid = resident;
  {
    ProfScope ps("group_few_find", s, (double)P.rows * key.width);
    if (key.width == 4)
      k_few_find<uint32_t><<<grid, kFewFindThreads, 0, s>>>(static_cast<const uint32_t*>(key.data), key.nulls, P.rows,
                                                            limit, T, m.device);
    else
      k_few_find<unsigned long long><<<grid, kFewFindThreads, 0, s>>>(static_cast<const unsigned long long*>(key.data),
                                                                      key.nulls, P.rows, limit, T, m.device);
    YQ_CHECK_LAUNCH();
  }
  YQ_TRY_CUDA(cudaStreamSynchronize(s));
  const uint32_t G = m.host[1];
  if (m.host[0] || G == 0) return YQ_OK;
  F.P.err = &T->err;
  F.key = key;
  F.out_key = out_key;
  F.ngroups = G;
  F.T = T;
  F.part = part;
  F.host_err = m.device + 2;
  if (G > capacity) {
    *groups = G;
    *done = true;
    return YQ_ERR_CAPACITY;
  }
  const size_t smem = few_smem(key.width, G, F.bytes);
  void (*const accumulate)(FewParams) =
      key.width == 4 ? k_few_accumulate<uint32_t> : k_few_accumulate<unsigned long long>;
  YQ_TRY(kernel_allow_smem((const void*)accumulate, smem));
  int per_sm = kernel_blocks_per_sm((const void*)accumulate, kFewThreads, smem);
  if (per_sm > kFewBlocksPerSm) per_sm = kFewBlocksPerSm;
  unsigned blocks = grid_for(P.rows, kFewThreads * kFewItems);
  if (blocks > (unsigned)(sm_count() * per_sm)) blocks = (unsigned)(sm_count() * per_sm);
  F.rows_per_block = (uint32_t)align_up(((size_t)P.rows + blocks - 1) / blocks, kFewThreads * kFewItems);
  blocks = (P.rows + F.rows_per_block - 1) / F.rows_per_block;
  double in_bytes = (double)P.rows * key.width;
  for (int j = 0; j < P.nagg; ++j)
    if (P.a[j].data) in_bytes += (double)P.rows * (type_width(P.a[j].type) + (P.a[j].nulls ? 1 : 0));
  {
    ProfScope ps("group_few_accumulate", s, in_bytes);
    accumulate<<<blocks, kFewThreads, smem, s>>>(F);
    YQ_CHECK_LAUNCH();
  }
  k_few_finish<<<dim3(G, (unsigned)(P.nagg > 0 ? P.nagg : 1)), kFinishThreads, 0, s>>>(F, blocks);
  YQ_CHECK_LAUNCH();
  YQ_TRY_CUDA(cudaStreamSynchronize(s));
  *groups = G;
  *done = true;
  return m.host[2] ? YQ_ERR_INVALID_ARG : YQ_OK;
}

}  // namespace

extern "C" {

// Sort workspace for ordering `ntiles` tiles by their first row (4-byte keys).
// Sizing reads no column data: the placeholder pointer only has to be non-null.
static size_t tile_order_sort_bytes(uint32_t ntiles) {
  const yq_column c{reinterpret_cast<void*>(static_cast<uintptr_t>(256)), nullptr, YQ_INT32, 4};
  return yq_sort_workspace_size(&c, ntiles);
}

size_t yq_group_by_workspace_size(const yq_column* key, uint32_t rows, int32_t nagg, uint32_t capacity) {
  if (!key) return 0;
  const size_t tiles = ((size_t)rows + kGroupTile - 1) / kGroupTile + 1;
  WsSize w;
  w.add<uint8_t>(yq_sort_workspace_size(key, rows));
  w.add<uint32_t>((size_t)rows + 1);          // permutation
  const int kwm = sort_key_words_max(*key);
  w.add<uint32_t>((size_t)rows * (kwm > 0 ? kwm : 1) + 16);  // sorted key words
  w.add<uint8_t>((size_t)rows + 16);          // head flags
  w.add<uint32_t>((size_t)rows + 1);          // group of every sorted position
  w.add<uint8_t>(yq_prefix_sum_workspace_size(rows));
  w.add<uint32_t>((size_t)capacity + 2);      // group starts
  w.add<unsigned long long>(tiles * 4 * (size_t)(nagg > 0 ? nagg : 1));  // tile head / tail records
  w.add<uint32_t>(tiles);                     // tail group of every tile
  w.add<uint32_t>(2 * tiles);                 // first row of every tile, tile order
  w.add<uint8_t>(tile_order_sort_bytes((uint32_t)tiles));
  w.add<uint32_t>(tiles);                     // tile flags
  w.add<uint32_t>(4);                         // error word
  if (few_applies(*key, rows)) w.add<char>(few_workspace_bytes(nagg));
  return w.total();
}

int yq_group_by(const yq_batch* batch, int32_t key_col, const yq_group_agg* aggs, int32_t nagg, yq_column* out,
                uint32_t capacity, uint32_t* groups, void* workspace, size_t workspace_bytes, void* stream) {
  if (!batch || !groups || !out || nagg < 0 || nagg > YQ_MAX_AGGREGATES || key_col < 0 ||
      key_col >= batch->ncols || (nagg && !aggs))
    return YQ_ERR_INVALID_ARG;
  *groups = 0;
  const yq_column key = batch->columns[key_col];
  const uint32_t rows = batch->rows;
  if (!(key.type == YQ_INT32 || key.type == YQ_INT64 || key.type == YQ_DATETIME || key.type == YQ_FLOAT32 ||
        key.type == YQ_FLOAT64 || key.type == YQ_TEXT))
    return YQ_ERR_UNSUPPORTED;
  if (out[0].type != key.type || out[0].width != key.width || (rows && !out[0].data)) return YQ_ERR_INVALID_ARG;
  GroupParams P;
  memset(&P, 0, sizeof(P));
  P.nagg = nagg;
  P.rows = rows;
  for (int j = 0; j < nagg; ++j) {
    const yq_group_agg& g = aggs[j];
    const bool star = g.kind == YQ_AGG_COUNT_STAR;
    if (g.kind < YQ_AGG_COUNT_STAR || g.kind > YQ_AGG_MAX) return YQ_ERR_INVALID_ARG;
    if (!star && (g.column < 0 || g.column >= batch->ncols)) return YQ_ERR_INVALID_ARG;
    const yq_column in = star ? yq_column{nullptr, nullptr, YQ_INT64, 8} : batch->columns[g.column];
    const int it = in.type;
    const bool numeric = it == YQ_INT32 || it == YQ_INT64 || it == YQ_FLOAT32 || it == YQ_FLOAT64;
    if (!star && g.kind != YQ_AGG_COUNT && !(numeric || (it == YQ_DATETIME && (g.kind == YQ_AGG_MIN ||
                                                                              g.kind == YQ_AGG_MAX))))
      return YQ_ERR_UNSUPPORTED;
    const int ot = out_type(g.kind, it);
    const yq_column& o = out[1 + j];
    if (o.type != ot || o.width != type_width(ot) || (rows && !o.data)) return YQ_ERR_INVALID_ARG;
    if (!o.nulls && g.kind != YQ_AGG_COUNT && g.kind != YQ_AGG_COUNT_STAR && rows) return YQ_ERR_INVALID_ARG;
    P.a[j] = GAgg{in.data, in.nulls, it, g.kind, in.width};
    P.out[j] = o;
  }
  if (rows == 0) return YQ_OK;
  cudaStream_t s = as_stream(stream);
  Workspace ws;
  YQ_TRY(ws.acquire(workspace, workspace_bytes, yq_group_by_workspace_size(&key, rows, nagg, capacity), s));
  const uint32_t ntiles = (uint32_t)(((size_t)rows + kGroupTile - 1) / kGroupTile);
  const size_t sort_ws = yq_sort_workspace_size(&key, rows);
  void* d_sort = ws.take<uint8_t>(sort_ws);
  uint32_t* perm = ws.take<uint32_t>((size_t)rows + 1);
  const int kwm = sort_key_words_max(key);
  uint32_t* words = ws.take<uint32_t>((size_t)rows * (kwm > 0 ? kwm : 1) + 16);
  uint8_t* head = ws.take<uint8_t>((size_t)rows + 16);
  uint32_t* incl = ws.take<uint32_t>((size_t)rows + 1);
  void* scan_ws = ws.take<uint8_t>(yq_prefix_sum_workspace_size(rows));
  uint32_t* starts = ws.take<uint32_t>((size_t)capacity + 2);
  unsigned long long* rec = ws.take<unsigned long long>(((size_t)ntiles + 1) * 4 * (size_t)(nagg > 0 ? nagg : 1));
  uint32_t* tail_group = ws.take<uint32_t>((size_t)ntiles + 1);
  uint32_t* first_row = ws.take<uint32_t>((size_t)ntiles + 1);
  uint32_t* tile_order = ws.take<uint32_t>((size_t)ntiles + 1);
  const size_t order_ws_bytes = tile_order_sort_bytes(ntiles + 1);
  void* order_ws = ws.take<uint8_t>(order_ws_bytes);
  uint32_t* tile_flags = ws.take<uint32_t>((size_t)ntiles + 1);
  uint32_t* d_err = ws.take<uint32_t>(4);
  if (few_applies(key, rows)) {
    const size_t few_bytes = few_workspace_bytes(nagg);
    char* few_ws = ws.take<char>(few_bytes);
    bool done = false;
    const int st = group_by_few(P, key, out[0], capacity, groups, few_ws, few_bytes, s, &done);
    if (done || st != YQ_OK) return st;
  }
  // The sort skips the passes whose digit every key shares (a key of few
  // distinct values sorts in one or two passes) and hands over its key words
  // in sorted order; a text key too long for one pass's words sorts without
  // them, and its heads compare the rows through the permutation.
  KeyJob job{key, 0, 0};
  const uint32_t offs[2] = {0, rows};
  int kw = 0;
  int st = sort_segments_impl(&job, 1, rows, offs, 1, perm, nullptr, d_sort, sort_ws, s, nullptr, words, &kw);
  const bool have_words = st == YQ_OK;
  if (st == YQ_ERR_UNSUPPORTED)
    st = sort_segments_impl(&job, 1, rows, offs, 1, perm, nullptr, d_sort, sort_ws, s, nullptr);
  YQ_TRY(st);
  if (have_words) {
    ProfScope ps("group_heads", s, (double)rows * 4.0 * (kw > 0 ? kw : 1));
    k_group_heads_words<<<grid_for(rows, kGroupThreads), kGroupThreads, 0, s>>>(words, kw, rows, head);
    YQ_CHECK_LAUNCH();
  } else {
    ProfScope ps("group_heads", s, (double)rows * (key.width + 4));
    k_group_heads<<<grid_for(rows, kGroupThreads), kGroupThreads, 0, s>>>(key, perm, rows, head);
    YQ_CHECK_LAUNCH();
  }
  YQ_TRY(yq_prefix_sum_mask(head, incl, rows, scan_ws, yq_prefix_sum_workspace_size(rows), stream));
  uint32_t G = 0;
  YQ_TRY(d2h_sync(&G, incl + rows - 1, sizeof(G), s));
  *groups = G;
  if (G > capacity) return YQ_ERR_CAPACITY;
  P.perm = perm;
  P.incl = incl;
  P.starts = starts;
  P.rec = rec;
  P.tail_group = tail_group;
  P.tile_flags = tile_flags;
  P.err = d_err;
  k_group_keys<<<grid_for(rows, kGroupThreads), kGroupThreads, 0, s>>>(key, perm, rows, head, incl, out[0]);
  YQ_CHECK_LAUNCH();
  if (nagg) {
    const uint32_t end_word[1] = {rows};
    YQ_TRY(h2d_async(starts + G, end_word, sizeof(uint32_t), s));  // starts[G] = rows
    YQ_TRY_CUDA(cudaMemsetAsync(tile_flags, 0, ((size_t)ntiles + 1) * sizeof(uint32_t), s));
    YQ_TRY_CUDA(cudaMemsetAsync(d_err, 0, 4 * sizeof(uint32_t), s));
    double in_bytes = 8.0 * rows;  // group index + permutation
    for (int j = 0; j < nagg; ++j)
      if (P.a[j].data) in_bytes += (double)rows * (type_width(P.a[j].type) + (P.a[j].nulls ? 1 : 0));
    // Tiles run in the order of their first input row. The rows of one group
    // ascend through its sorted positions, so the tiles resident together
    // (one stretch of every group) read values from one stretch of rows,
    // which L2 then holds for all of them; in position order they would be
    // one group's tiles reading rows spread over the whole table. The
    // results do not depend on the order: each tile writes its own records.
    if (ntiles >= 64) {
      k_tile_first_row<<<grid_for(ntiles, kGroupThreads), kGroupThreads, 0, s>>>(perm, ntiles, kGroupTile, first_row);
      YQ_CHECK_LAUNCH();
      const yq_column fc{first_row, nullptr, YQ_INT32, 4};
      KeyJob oj{fc, 0, 0};
      const uint32_t oo[2] = {0, ntiles};
      YQ_TRY(sort_segments_impl(&oj, 1, ntiles, oo, 1, tile_order, nullptr, order_ws, order_ws_bytes, s, nullptr));
      P.tile_order = tile_order;
    }
    {
      ProfScope ps("group_accumulate", s, in_bytes);
      k_group_tiles<<<ntiles, kGroupThreads, 0, s>>>(P);
      YQ_CHECK_LAUNCH();
      k_group_span<<<ntiles, kGroupThreads, 0, s>>>(P, ntiles);
      YQ_CHECK_LAUNCH();
    }
    uint32_t err = 0;
    YQ_TRY(d2h_sync(&err, d_err, sizeof(err), s));
    if (err) return YQ_ERR_INVALID_ARG;
  }
  return YQ_OK;
}

}  // extern "C"
