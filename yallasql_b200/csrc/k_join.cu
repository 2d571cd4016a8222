// Inner join (nested-loop semantics), cross product and the fused star-join
// aggregate for sm_100a.
//
// Replaces ComparisonJoinExpression / ConjunctionJoinExpression with
// outer_join_batches (one thread per (l, r) pair, one global atomic per match)
// and and_join_batches (P1 x P2 intersection of pair lists), move_rows_join
// per output column, and CrossProductOperator's per-column replication
// (include/engine/operators/filters/comparison_join.hpp:70-236,
//  src/kernels/comparison_operators_kernel.cu:6-54,136-167,
//  src/kernels/move_rows_kernel.cu:8-30, include/engine/operators/join_operator.hpp:36-265,
//  include/engine/operators/cross_product_operator.hpp:87-125, src/kernels/cross_product_kernel.cu:8-27).
//
// All conditions are evaluated in one kernel and pairs come out in a fixed
// order (left row ascending, then right row ascending):
//  - equality path: the right side's equality key is bucketed once into a
//    stably ordered hash table that every block copies into shared memory;
//    each left row probes its bucket, checks the remaining conditions, counts,
//    and after a decoupled look-back over tiles writes its pairs;
//    A longer right side is sorted by its key and probed through a hash table
//    of its distinct keys in global memory;
//  - nested-loop path: a warp per left row sweeps the right rows 32 at a time,
//    ballots the matches and appends them with popc offsets (coalesced);
//  - no condition: the cross product is written directly, left-major.
#include <limits.h>
#include <string.h>
#include <type_traits>
#include <vector>
#include "vm_host.cuh"
#include "row_kernels.cuh"
#include "yq_jit.cuh"
#include "yq_sort.cuh"

namespace yq {

constexpr int kJoinBlock = 256;
constexpr int kJoinItems = 4;
constexpr uint32_t kJoinTile = kJoinBlock * kJoinItems;
constexpr uint32_t kHashMaxRows = 8192;  // right rows that fit the shared-memory table
constexpr int kMaxConds = 8;
constexpr int kMaxJoinOut = YQ_MAX_PROJECTIONS;

struct JCond {
  JCol l, r;
  int32_t cmp;
};

struct JOut {
  const char* src;
  const uint8_t* src_nulls;
  char* dst;
  uint8_t* dst_nulls;
  int32_t width;
  int32_t side;  // 0 = left, 1 = right
};

struct JoinParams {
  JCond cond[kMaxConds];
  int32_t ncond;
  // OR of ANDs: condition i belongs to disjunct group[i]; a pair matches when
  // every condition of at least one group holds. ngroups <= 1: one conjunction.
  int8_t group[kMaxConds];
  int32_t ngroups;
  int32_t eq;  // index of the equality condition used for hashing (-1: nested loop)
  JOut out[kMaxJoinOut];
  int32_t nout;          // 0: write pairs
  uint32_t* out_left;    // pair output (nout == 0)
  uint32_t* out_right;
  unsigned long long capacity;
  uint32_t L, R;
  // hash table (equality path)
  const uint32_t* bstart;  // nbuckets + 1
  const unsigned long long* hkeys;
  const uint32_t* hrows;
  uint32_t nbuckets, hrows_n;
  unsigned long long* status;
  uint32_t* tile_counter;
  unsigned long long* total;
  uint32_t* err;
  const uint32_t* counts;  // typed nested loop: matches per left row, counted up front (null: count in the kernel)
  char* vdst[2];           // typed nested loop writing values from registers: left / right output (or null)
  const char* vsrc;        // and the left output's column
};


__device__ __forceinline__ bool cmp_holds(int s, int op) {
  switch (op) {
    case YQ_LT: return s < 0;
    case YQ_LE: return s <= 0;
    case YQ_GT: return s > 0;
    case YQ_GE: return s >= 0;
    case YQ_EQ: return s == 0;
    default: return s != 0;
  }
}

// Three-way compare of left row l and right row r for one condition; false
// when either side is NULL (an SQL comparison with NULL is not TRUE).
__device__ __forceinline__ bool cond_holds(const JCond& c, uint32_t l, uint32_t r) {
  if (cell_null(c.l, l) || cell_null(c.r, r)) return false;
  int s;
  if (c.l.type == YQ_TEXT) {
    const uint32_t* p = reinterpret_cast<const uint32_t*>(c.l.data + (size_t)l * c.l.width);
    const uint32_t* q = reinterpret_cast<const uint32_t*>(c.r.data + (size_t)r * c.r.width);
    const int pw = c.l.width >> 2, qw = c.r.width >> 2, n = pw > qw ? pw : qw;
    s = 0;
    for (int i = 0; i < n && s == 0; ++i) {
      const uint32_t a = i < pw ? __byte_perm(__ldg(p + i), 0, 0x0123) : 0u;
      const uint32_t b = i < qw ? __byte_perm(__ldg(q + i), 0, 0x0123) : 0u;
      s = (a > b) - (a < b);
    }
  } else {
    const uint64_t a = cell_u64(c.l, l), b = cell_u64(c.r, r);
    switch (c.l.type) {
      case YQ_FLOAT32: {
        const float x = __uint_as_float((uint32_t)a), y = __uint_as_float((uint32_t)b);
        s = (x > y) - (x < y);
        break;
      }
      case YQ_FLOAT64: {
        const double x = __longlong_as_double((long long)a), y = __longlong_as_double((long long)b);
        s = (x > y) - (x < y);
        break;
      }
      default: {
        const int64_t x = (int64_t)a, y = (int64_t)b;
        s = (x > y) - (x < y);
      }
    }
    if (c.l.type == YQ_FLOAT32 || c.l.type == YQ_FLOAT64) {
      // NaN never satisfies a comparison
      const bool nan_a = c.l.type == YQ_FLOAT32 ? isnan(__uint_as_float((uint32_t)a))
                                                : isnan(__longlong_as_double((long long)a));
      const bool nan_b = c.l.type == YQ_FLOAT32 ? isnan(__uint_as_float((uint32_t)b))
                                                : isnan(__longlong_as_double((long long)b));
      if (nan_a || nan_b) return c.cmp == YQ_NE;
    }
  }
  return cmp_holds(s, c.cmp);
}

// A disjunction of conjunctions: a group fails at its first condition that
// does not hold (a comparison with a NULL side does not hold), later
// conditions of a failed group are skipped, and the pair matches while some
// group has not failed. Only TRUE selects a pair, so this two-valued
// evaluation gives the rows SQL's three-valued OR/AND selects.
__device__ __forceinline__ bool any_group(const JoinParams& J, uint32_t l, uint32_t r) {
  const uint32_t all = (1u << J.ngroups) - 1u;
  uint32_t failed = 0u;
  for (int i = 0; i < J.ncond; ++i) {
    const uint32_t bit = 1u << J.group[i];
    if (!(failed & bit) && !cond_holds(J.cond[i], l, r)) {
      failed |= bit;
      if (failed == all) return false;
    }
  }
  return true;
}

__device__ __forceinline__ bool all_conds(const JoinParams& J, uint32_t l, uint32_t r, int skip) {
  if (J.ngroups > 1) return any_group(J, l, r);
  for (int i = 0; i < J.ncond; ++i)
    if (i != skip && !cond_holds(J.cond[i], l, r)) return false;
  return true;
}

__device__ __forceinline__ void copy_cell_j(char* dst, const char* src, int width) {
  if (width == 4) *reinterpret_cast<uint32_t*>(dst) = __ldg(reinterpret_cast<const uint32_t*>(src));
  else if (width == 8)
    *reinterpret_cast<unsigned long long*>(dst) = __ldg(reinterpret_cast<const unsigned long long*>(src));
  else if (width == 1) *dst = *src;
  else
    for (int i = 0; i < width; i += 4)
      *reinterpret_cast<uint32_t*>(dst + i) = __ldg(reinterpret_cast<const uint32_t*>(src + i));
}

__device__ __forceinline__ void emit_pair(const JoinParams& J, unsigned long long pos, uint32_t l, uint32_t r) {
  if (pos >= J.capacity) return;
  if (J.nout == 0) {
    J.out_left[pos] = l;
    J.out_right[pos] = r;
    return;
  }
  for (int o = 0; o < J.nout; ++o) {
    const JOut& w = J.out[o];
    const uint32_t row = w.side ? r : l;
    copy_cell_j(w.dst + (size_t)pos * w.width, w.src + (size_t)row * w.width, w.width);
    if (w.dst_nulls) w.dst_nulls[pos] = w.src_nulls ? w.src_nulls[row] : 0;
  }
}

// ------------------------------------------------------------ hash build
// One block buckets the right rows (optionally only those passing a
// predicate) by hash of the equality key; within a bucket rows stay in
// ascending row order, so probing yields right rows in ascending order.
struct BuildParams {
  VmProgram P;        // predicate over the right batch (pred_len == 0: all rows)
  int32_t pred_len;
  JCol key;
  uint32_t R;
  uint32_t nbuckets;
  uint32_t* bstart;   // [nbuckets + 1]
  unsigned long long* hkeys;
  uint32_t* hrows;
  uint32_t* counts;   // [0] rows kept, [1] duplicate keys seen, [2..3] least and [4..5] greatest key (signed)
};


constexpr int kBuildBlock = 1024;

__global__ void __launch_bounds__(kBuildBlock) k_hash_build(const __grid_constant__ BuildParams B) {
  extern __shared__ uint32_t sb[];
  uint32_t* s_cnt = sb;                        // [nbuckets] counts, then cursors
  uint32_t* s_rows = s_cnt + B.nbuckets;       // [R] kept rows in order
  uint32_t* s_warp = s_rows + kHashMaxRows;    // [33]
  __shared__ uint32_t s_kept;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < B.nbuckets; i += kBuildBlock) s_cnt[i] = 0;
  if (threadIdx.x == 0) s_kept = 0;
  __syncthreads();
  // 1. stable compaction of the rows passing the predicate
  for (uint32_t base = 0; base < B.R; base += kBuildBlock * ITEMS) {
    const uint32_t row0 = base + threadIdx.x * ITEMS;
    uint32_t inr = 0;
    if (row0 < B.R) inr = (B.R - row0 >= (uint32_t)ITEMS) ? 0xfu : ((1u << (B.R - row0)) - 1u);
    SelEmit E;
    E.sel = inr;
    if (B.pred_len > 0) {
      Ctx X;
      X.tile0 = base;
      X.lr = threadIdx.x * ITEMS;
      X.inr = inr;
      X.stage = 0;
      X.vec_ok = (base & 15u) == 0u;
      Stack S;
      run_vm<false>(B.P, 0, B.pred_len, X, S, E);
    }
    // key NULLs never join
    for (int k = 0; k < ITEMS; ++k)
      if ((E.sel >> k & 1u) && cell_null(B.key, row0 + k)) E.sel &= ~(1u << k);
    uint32_t total;
    const uint32_t excl = block_exclusive_sum<kBuildBlock>(__popc(E.sel), s_warp, total);
    uint32_t pos = s_kept + excl;
    for (int k = 0; k < ITEMS; ++k)
      if (E.sel >> k & 1u) {
        if (pos < kHashMaxRows) s_rows[pos] = row0 + k;
        ++pos;
      }
    __syncthreads();
    if (threadIdx.x == 0) s_kept += total;
    __syncthreads();
  }
  const uint32_t kept = min(s_kept, kHashMaxRows);
  // 2. bucket counts and starts, key range
  __shared__ long long s_min, s_max;
  if (threadIdx.x == 0) {
    s_min = LLONG_MAX;
    s_max = LLONG_MIN;
  }
  __syncthreads();
  {
    long long lo = LLONG_MAX, hi = LLONG_MIN;
    for (uint32_t i = threadIdx.x; i < kept; i += kBuildBlock) {
      const long long k = (long long)hash_key(B.key, s_rows[i]);
      atomicAdd(&s_cnt[hash_bucket((uint64_t)k, B.nbuckets)], 1u);
      lo = min(lo, k);
      hi = max(hi, k);
    }
    if (lo <= hi) {
      atomicMin(&s_min, lo);
      atomicMax(&s_max, hi);
    }
  }
  __syncthreads();
  uint32_t run = 0;
  for (uint32_t b0 = 0; b0 < B.nbuckets; b0 += kBuildBlock) {
    const uint32_t b = b0 + threadIdx.x;
    uint32_t total;
    const uint32_t at = run + block_exclusive_sum<kBuildBlock>(b < B.nbuckets ? s_cnt[b] : 0u, s_warp, total);
    if (b < B.nbuckets) {
      B.bstart[b] = at;
      s_cnt[b] = at;  // becomes the insertion cursor
    }
    run += total;
  }
  if (threadIdx.x == 0) {
    B.bstart[B.nbuckets] = run;
    B.counts[0] = s_kept;
    *reinterpret_cast<long long*>(B.counts + 2) = s_min;
    *reinterpret_cast<long long*>(B.counts + 4) = s_max;
  }
  __syncthreads();
  // 3. stable scatter: rows in ascending order, one warp at a time
  for (uint32_t base = 0; base < kept; base += kBuildBlock) {
    const uint32_t i = base + threadIdx.x;
    const bool valid = i < kept;
    const uint32_t row = valid ? s_rows[i] : 0u;
    const uint64_t key = valid ? hash_key(B.key, row) : 0ull;
    const uint32_t b = valid ? hash_bucket(key, B.nbuckets) : 0xffffffffu;
    const uint32_t peers = __match_any_sync(0xffffffffu, b) & __ballot_sync(0xffffffffu, valid);
    const uint32_t rank = __popc(peers & lanemask_lt());
    for (int w = 0; w < kBuildBlock / 32; ++w) {
      if (warp == w && valid) {
        const uint32_t slot = s_cnt[b] + rank;
        B.hkeys[slot] = key;
        B.hrows[slot] = row;
        __syncwarp(peers);
        if (rank == 0) s_cnt[b] += __popc(peers);
      }
      __syncthreads();
    }
  }
  __syncthreads();
  // 4. duplicate keys (the fused aggregate needs unique dimension keys)
  for (uint32_t b = threadIdx.x; b < B.nbuckets; b += kBuildBlock) {
    const uint32_t s0 = B.bstart[b], s1 = B.bstart[b + 1];
    for (uint32_t x = s0; x < s1; ++x)
      for (uint32_t y = x + 1; y < s1; ++y)
        if (B.hkeys[x] == B.hkeys[y]) atomicAdd(&B.counts[1], 1u);
  }
  (void)lane;
}

// ------------------------------------------------------ equality probing
struct ProbeSmem {
  uint32_t* bstart;
  unsigned long long* keys;
  uint32_t* rows;
};

__device__ __forceinline__ ProbeSmem load_table(const JoinParams& J, uint32_t* sm) {
  ProbeSmem t;
  t.bstart = sm;
  t.keys = reinterpret_cast<unsigned long long*>(sm + ((J.nbuckets + 2) & ~1u));
  t.rows = reinterpret_cast<uint32_t*>(t.keys + J.hrows_n);
  for (uint32_t i = threadIdx.x; i <= J.nbuckets; i += blockDim.x) t.bstart[i] = __ldg(J.bstart + i);
  for (uint32_t i = threadIdx.x; i < J.hrows_n; i += blockDim.x) {
    t.keys[i] = __ldg(J.hkeys + i);
    t.rows[i] = __ldg(J.hrows + i);
  }
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(kJoinBlock) k_join_hash(const __grid_constant__ JoinParams J) {
  extern __shared__ uint32_t sm[];
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[kJoinBlock / 32 + 1];
  __shared__ unsigned long long s_prefix;
  if (threadIdx.x == 0) s_tile = atomicAdd(J.tile_counter, 1u);
  const ProbeSmem T = load_table(J, sm);
  const uint32_t tile = s_tile;
  const uint32_t l0 = tile * kJoinTile + threadIdx.x * kJoinItems;
  const JCond& ec = J.cond[J.eq];
  // pass 1: count
  uint32_t cnt = 0;
  for (int k = 0; k < kJoinItems; ++k) {
    const uint32_t l = l0 + k;
    if (l >= J.L || cell_null(ec.l, l)) continue;
    const uint64_t key = hash_key(ec.l, l);
    const uint32_t b = hash_bucket(key, J.nbuckets);
    for (uint32_t x = T.bstart[b]; x < T.bstart[b + 1]; ++x)
      if (T.keys[x] == key && all_conds(J, l, T.rows[x], J.eq)) ++cnt;
  }
  uint32_t total;
  const uint32_t excl = block_exclusive_sum<kJoinBlock>(cnt, s_warp, total);
  if (threadIdx.x < 32) {
    const unsigned long long p = tile_lookback(J.status, tile, total, J.err);
    if (threadIdx.x == 0) s_prefix = p;
  }
  __syncthreads();
  unsigned long long pos = s_prefix + excl;
  // pass 2: write
  if (cnt) {
    for (int k = 0; k < kJoinItems; ++k) {
      const uint32_t l = l0 + k;
      if (l >= J.L || cell_null(ec.l, l)) continue;
      const uint64_t key = hash_key(ec.l, l);
      const uint32_t b = hash_bucket(key, J.nbuckets);
      for (uint32_t x = T.bstart[b]; x < T.bstart[b + 1]; ++x)
        if (T.keys[x] == key && all_conds(J, l, T.rows[x], J.eq)) emit_pair(J, pos++, l, T.rows[x]);
    }
  }
  if (tile == gridDim.x - 1 && threadIdx.x == 0) *J.total = s_prefix + total;
}

// --------------------------------------- equality probing, long right sides
// A right side too long for a shared-memory table is sorted once by its key
// (the stable radix sort, so rows of one key are contiguous and ascending) and
// a hash table in global memory maps each distinct key to its run. A slot holds
// key, run and, for a key that does not repeat, the right row itself, so such a
// probe is one 16-byte read (2M rows to 300K: 122 us with separate arrays of
// slots, keys and rows, 104 so). A key's repeats
// are a contiguous run, so the outputs of a tile are written position by
// position by all its threads (coalesced, and one left row with many matches
// does not serialise a thread). The nested loop this replaces compares every
// pair: 2M x 300K INT32 rows took 303 ms.
struct SortedJoin {
  const uint32_t* perm;  // right rows in key order
  uint4* slots;          // {key, first sorted position (kNoSlot: empty), run}
  uint32_t nslots;       // power of two, >= 1.5 R
  uint32_t rows;         // R
  uint32_t tile_rows;    // left rows a block takes, at most kJoinTile
};
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint32_t kOneRow = 0x80000000u;  // run field: the key's only row (row ids are below 2^30)
constexpr uint32_t kSortedMinRows = 1024;  // right rows from which a sorted table may be chosen, and from
constexpr uint32_t kTableRows = 4096;      // which it always is

__device__ __forceinline__ bool key_joins(const JCol& c, uint32_t row) {
  if (cell_null(c, row)) return false;
  if (c.type == YQ_FLOAT32) return !isnan(__uint_as_float((uint32_t)cell_u64(c, row)));
  if (c.type == YQ_FLOAT64) return !isnan(__longlong_as_double((long long)cell_u64(c, row)));
  return true;
}

__global__ void __launch_bounds__(256) k_join_sorted_build(const __grid_constant__ SortedJoin S, const JCol key,
                                                           uint32_t R, const uint32_t* sort_err, uint32_t* err) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && *sort_err) atomicOr(err, *sort_err);
  auto row_at = [&](uint32_t i) {
    const uint32_t row = __ldg(S.perm + i);
    if (row >= R) atomicOr(err, kErrBounds);  // a failed sort left no permutation
    return min(row, R - 1u);
  };
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x) {
    const uint32_t row = row_at(i);
    if (!key_joins(key, row)) continue;
    const uint64_t k = hash_key(key, row);
    auto same = [&](uint32_t j) {
      const uint32_t r = row_at(j);
      return key_joins(key, r) && hash_key(key, r) == k;
    };
    if (i > 0 && same(i - 1)) continue;
    uint32_t step = 1;  // run end: doubling steps, then a binary search inside the last one
    while (step < R - i && same(i + step)) step <<= 1;
    uint32_t lo = i + (step >> 1), hi = step < R - i ? i + step : R;  // key at lo matches; hi is past the run
    while (lo + 1 < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (same(mid)) lo = mid;
      else hi = mid;
    }
    const uint32_t run = lo + 1u - i;
    uint32_t h = hash_bucket(k, S.nslots);  // keys are distinct here: the first empty slot is this key's
    for (uint32_t n = 0; n < S.nslots; ++n, h = (h + 1u) & (S.nslots - 1u)) {
      uint32_t* slot = reinterpret_cast<uint32_t*>(S.slots + h);
      if (atomicCAS(slot + 2, kNoSlot, i) != kNoSlot) continue;
      slot[0] = (uint32_t)k;
      slot[1] = (uint32_t)(k >> 32);
      slot[3] = run == 1u ? kOneRow | row : run;
      break;
    }
  }
}

// Matches of a thread's ITEMS consecutive left rows: the number of rows of
// each one's key, and where they are (a sorted position, or kOneRow and the
// row). The first probe of every row goes out before any is looked at.
template <int ITEMS>
__device__ __forceinline__ void sorted_matches(const SortedJoin& S, const JCol& key, uint32_t l0, uint32_t L,
                                               uint32_t (&where)[ITEMS], uint32_t (&run)[ITEMS]) {
  uint64_t k[ITEMS];
  uint32_t h[ITEMS], joins = 0u;
  uint4 at[ITEMS];
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    const uint32_t l = l0 + i < L ? l0 + i : L - 1u;
    if (l0 + i < L && key_joins(key, l)) joins |= 1u << i;
    k[i] = hash_key(key, l);
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    h[i] = hash_bucket(k[i], S.nslots);
    at[i] = __ldg(S.slots + h[i]);
  }
#pragma unroll
  for (int i = 0; i < ITEMS; ++i) {
    where[i] = run[i] = 0u;
    if (!(joins >> i & 1u)) continue;
    auto mine = [&](const uint4& e) { return e.x == (uint32_t)k[i] && e.y == (uint32_t)(k[i] >> 32); };
    for (uint32_t n = 1; n < S.nslots && at[i].z != kNoSlot && !mine(at[i]); ++n) {
      h[i] = (h[i] + 1u) & (S.nslots - 1u);
      at[i] = __ldg(S.slots + h[i]);
    }
    if (at[i].z == kNoSlot || !mine(at[i])) continue;
    run[i] = (at[i].w & kOneRow) ? 1u : at[i].w;
    where[i] = (at[i].w & kOneRow) ? at[i].w : at[i].z;
  }
}

// Right row of match x of a key at `where` (a failed sort, which the error word
// reports, must not send the reads out of range).
__device__ __forceinline__ uint32_t match_row(const SortedJoin& S, uint32_t where, uint32_t x) {
  return (where & kOneRow) ? where & ~kOneRow : min(__ldg(S.perm + where + x), S.rows - 1u);
}

// (16 bytes at a time where they are aligned; in emit_pair that took the general
// nested loop's comparisons their registers: 505 us became 562, 40K x 1,025 rows)
__device__ __forceinline__ void write_col(const JOut& w, unsigned long long pos, uint32_t row) {
  char* const dst = w.dst + (size_t)pos * w.width;
  const char* const src = w.src + (size_t)row * w.width;
  if (w.width >= 16 && ((w.width | reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0)
    for (int i = 0; i < w.width; i += 16) *reinterpret_cast<uint4*>(dst + i) = ldg_nc_v4(src + i);
  else copy_cell_j(dst, src, w.width);
  if (w.dst_nulls) w.dst_nulls[pos] = w.src_nulls ? w.src_nulls[row] : 0;
}

constexpr uint32_t kSortedChunk = 2048;  // outputs resolved to (left, right) rows at a time

// The equality is the only condition: a left row's matches are its key's run.
__global__ void __launch_bounds__(kJoinBlock) k_join_sorted(const __grid_constant__ JoinParams J,
                                                            const __grid_constant__ SortedJoin S) {
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_warp[kJoinBlock / 32 + 1];
  __shared__ unsigned long long s_prefix;
  __shared__ uint32_t s_off[kJoinTile + 1];
  __shared__ uint32_t s_first[kJoinTile];
  __shared__ __align__(8) uint32_t s_l[kSortedChunk];
  __shared__ uint32_t s_r[kSortedChunk];
  if (threadIdx.x == 0) s_tile = atomicAdd(J.tile_counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t base = tile * S.tile_rows, end = min(J.L, base + S.tile_rows);
  uint32_t first[kJoinItems], run[kJoinItems], sum = 0;
  sorted_matches<kJoinItems>(S, J.cond[J.eq].l, base + threadIdx.x * kJoinItems, end, first, run);
  unsigned long long wide = 0;  // the tile's pairs may exceed 32 bits (a hot key on both sides)
#pragma unroll
  for (int k = 0; k < kJoinItems; ++k) {
    wide += run[k];
    sum += run[k];
  }
  const int huge = __syncthreads_or(wide > 0xfffffu);  // 256 sums below 2^20 fit a 32-bit scan
  unsigned long long total;
  unsigned long long excl;
  if (!huge) {
    uint32_t t32;
    excl = block_exclusive_sum<kJoinBlock>(sum, s_warp, t32);
    total = t32;
  } else {
    __shared__ unsigned long long s_wide[2 * (kJoinBlock / 32 + 1)];
    unsigned long long a = wide, b = 0, tb;
    block_exclusive_sum2<kJoinBlock>(a, b, s_wide, total, tb);
    excl = a;
  }
  if (threadIdx.x < 32) {
    const unsigned long long p = tile_lookback(J.status, tile, total, J.err);
    if (threadIdx.x == 0) s_prefix = p;
  }
  __syncthreads();
  const unsigned long long prefix = s_prefix;
  if (tile == gridDim.x - 1 && threadIdx.x == 0) *J.total = prefix + total;
  if (prefix >= J.capacity || total == 0) return;  // nothing of this tile is stored
  if (!huge) {
    uint32_t at = (uint32_t)excl;
#pragma unroll
    for (int k = 0; k < kJoinItems; ++k) {
      s_off[threadIdx.x * kJoinItems + k] = at;
      s_first[threadIdx.x * kJoinItems + k] = first[k];
      at += run[k];
    }
    if (threadIdx.x == 0) s_off[kJoinTile] = (uint32_t)total;
    const unsigned long long room = J.capacity - prefix;
    const uint32_t n_out = total < room ? (uint32_t)total : (uint32_t)room;
    for (uint32_t c0 = 0; c0 < n_out; c0 += kSortedChunk) {
      const uint32_t n = min(kSortedChunk, n_out - c0);
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < n; i += kJoinBlock) {
        uint32_t lo = 0, hi = S.tile_rows;  // the left row whose outputs hold position c0 + i
        while (lo + 1 < hi) {
          const uint32_t mid = (lo + hi) >> 1;
          if (s_off[mid] <= c0 + i) lo = mid;
          else hi = mid;
        }
        s_l[i] = base + lo;
        s_r[i] = match_row(S, s_first[lo], c0 + i - s_off[lo]);
      }
      __syncthreads();
      const unsigned long long p0 = prefix + c0;
      if (J.nout == 0) {
        for (uint32_t i = threadIdx.x; i < n; i += kJoinBlock) {
          J.out_left[p0 + i] = s_l[i];
          J.out_right[p0 + i] = s_r[i];
        }
      } else {
        for (int o = 0; o < J.nout; ++o) {
          const JOut& w = J.out[o];
          const uint32_t* rows = w.side ? s_r : s_l;
          for (uint32_t i = threadIdx.x; i < n; i += kJoinBlock) write_col(w, p0 + i, rows[i]);
        }
      }
    }
    return;
  }
  // A tile of more pairs than 32 bits count: the same by 64-bit offsets, pair by
  // pair (one row with 3M matches, two columns written: 12 ms; 92 when a warp
  // wrote each such row).
  static_assert(kJoinTile * 8 <= sizeof(s_l), "64-bit offsets in the place of the chunk's left rows");
  unsigned long long* const s_wide_off = reinterpret_cast<unsigned long long*>(s_l);
  unsigned long long at = excl;
#pragma unroll
  for (int k = 0; k < kJoinItems; ++k) {
    s_wide_off[threadIdx.x * kJoinItems + k] = at;
    s_first[threadIdx.x * kJoinItems + k] = first[k];
    at += run[k];
  }
  __syncthreads();
  const unsigned long long n_out = min(total, J.capacity - prefix);
  for (unsigned long long i = threadIdx.x; i < n_out; i += kJoinBlock) {
    uint32_t lo = 0, hi = S.tile_rows;
    while (lo + 1 < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (s_wide_off[mid] <= i) lo = mid;
      else hi = mid;
    }
    emit_pair(J, prefix + i, base + lo, match_row(S, s_first[lo], (uint32_t)(i - s_wide_off[lo])));
  }
}

// Right rows up to which all of them are candidates of every left row (below), and
// the same with very many left rows. The general comparison costs more than the
// typed one from there on: 200,000 x 66 rows, the condition's columns, 215 us
// against 157; 1M x 66, pairs, 488 against 1,008; 1M x 250, 1,432 against 890.
constexpr uint32_t kSmallRight = 40, kSmallRightMany = 72, kManyLeft = 500000;

// With further conditions the rows of a key's run are candidates. A block's
// candidates form one sequence (left row by left row, right rows ascending, the
// order of the output), cut into eight equal parts for its warps, so that a key
// with many rows on both sides is shared by all of them: 3,000 left rows to
// 20,000 right ones of one key and two more conditions took 246 ms with a warp
// going through the long runs of its 128 left rows one after the other, 9.4 in
// the nested loop.
// ALL: no equality and a right side of a few rows, every one of which is a
// candidate of every left row. (A block of the typed nested loop takes 16 left
// rows, and its counter, look-back and waits are most of its work then: 1M left
// rows to 5 right ones under <, pairs, 980 us there and 112 here.) Which of them
// match is kept as bits for the second sweep (1M x 24 rows: 246 us, 320 without).
template <bool ALL>
__global__ void __launch_bounds__(kJoinBlock) k_join_candidates(const __grid_constant__ JoinParams J,
                                                                const __grid_constant__ SortedJoin S) {
  constexpr int NW = kJoinBlock / 32;
  __shared__ uint32_t s_tile;
  __shared__ unsigned long long s_off[kJoinBlock + 1];  // first candidate of every left row
  __shared__ uint32_t s_where[kJoinBlock];
  __shared__ unsigned long long s_scan[2 * (NW + 1)];
  __shared__ unsigned long long s_cnt[NW];
  __shared__ unsigned long long s_prefix;
  __shared__ uint32_t s_bits[ALL ? kJoinBlock * kSmallRightMany / 32 : 1];  // which candidates match
  if (threadIdx.x == 0) s_tile = atomicAdd(J.tile_counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint32_t base = tile * S.tile_rows, end = min(J.L, base + S.tile_rows);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long candidates;
  if constexpr (ALL) {
    candidates = (unsigned long long)(end - base) * J.R;
  } else {
    uint32_t where[1], run[1];
    sorted_matches<1>(S, J.cond[J.eq].l, base + threadIdx.x, end, where, run);
    unsigned long long first = run[0], zero = 0, tz;
    block_exclusive_sum2<kJoinBlock>(first, zero, s_scan, candidates, tz);
    s_off[threadIdx.x] = first;
    s_where[threadIdx.x] = where[0];
    if (threadIdx.x == 0) s_off[kJoinBlock] = candidates;
  }
  __syncthreads();
  const unsigned long long part = ((candidates + NW - 1) / NW + 31) & ~31ull;
  const unsigned long long x0 = min(candidates, part * warp), x1 = min(candidates, x0 + part);
  // The last row whose first candidate is at or before x (it has candidates: x is one), from row `lo` on.
  auto row_of = [&](unsigned long long x, uint32_t lo) {
    uint32_t hi = S.tile_rows;
    while (lo + 1 < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (s_off[mid] <= x) lo = mid;
      else hi = mid;
    }
    return lo;
  };
  // f(candidates, left row, right row, whether this lane has one), 32 at a time in order
  auto sweep = [&](auto f) {
    if constexpr (ALL) {
      uint32_t at = ((uint32_t)x0 + lane) / J.R, r = (uint32_t)x0 + lane - at * J.R;
      for (uint32_t x = (uint32_t)x0; x < (uint32_t)x1; x += 32) {
        f(x, base + at, r, x + lane < (uint32_t)x1);
        if (J.R >= 32u) {
          r += 32u;
          if (r >= J.R) {
            r -= J.R;
            ++at;
          }
        } else {
          at = (x + 32u + lane) / J.R;
          r = x + 32u + lane - at * J.R;
        }
      }
    } else {
      if (x0 >= x1) return;
      uint32_t row = row_of(x0, 0u);
      for (unsigned long long x = x0; x < x1; x += 32) {
        const unsigned long long mine = min(x + lane, x1 - 1), last = min(x + 31, x1 - 1);
        const uint32_t at = last < s_off[row + 1] ? row : row_of(mine, row);
        f(0u, base + at, match_row(S, s_where[at], (uint32_t)(mine - s_off[at])), x + lane < x1);
        row = __shfl_sync(0xffffffffu, at, 31);
      }
    }
  };
  unsigned long long count = 0;
  sweep([&](uint32_t x, uint32_t l, uint32_t r, bool in) {
    const uint32_t bal = __ballot_sync(0xffffffffu, in && all_conds(J, l, r, J.eq));
    if (ALL && lane == 0) s_bits[x >> 5] = bal;  // kept for the second sweep
    count += __popc(bal);
  });
  if (lane == 0) s_cnt[warp] = count;
  __syncthreads();
  unsigned long long total = 0, before = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    before += w < warp ? s_cnt[w] : 0ull;
    total += s_cnt[w];
  }
  if (threadIdx.x < 32) {
    const unsigned long long p = tile_lookback(J.status, tile, total, J.err);
    if (threadIdx.x == 0) s_prefix = p;
  }
  __syncthreads();
  if (tile == gridDim.x - 1 && threadIdx.x == 0) *J.total = s_prefix + total;
  unsigned long long pos = s_prefix + before;
  if (count == 0 || pos >= J.capacity) return;  // nothing of this warp is stored
  const uint32_t lt = lanemask_lt();
  sweep([&](uint32_t x, uint32_t l, uint32_t r, bool in) {
    const uint32_t bal = ALL ? s_bits[x >> 5] : __ballot_sync(0xffffffffu, in && all_conds(J, l, r, J.eq));
    if (bal >> lane & 1u) emit_pair(J, pos + __popc(bal & lt), l, r);
    pos += __popc(bal);
  });
}


// Left rows a block of the sorted join takes: few enough that four blocks an SM
// have some, as one row may have any number of matches.
static uint32_t sorted_tile_rows(uint32_t L, bool eq_only) {
  const uint32_t most = eq_only ? kJoinTile : kJoinBlock, rows = ceil_div<uint32_t>(L, (uint32_t)sm_count() * 4u);
  return rows < 1u ? 1u : (rows < most ? rows : most);
}

// ------------------------------------------------------------ nested loop
constexpr int kNlRowsPerWarp = 4;
constexpr uint32_t kNlTile = (kJoinBlock / 32) * kNlRowsPerWarp;  // left rows per block

__global__ void __launch_bounds__(kJoinBlock) k_join_nested(const __grid_constant__ JoinParams J) {
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_cnt[kNlTile];
  __shared__ uint32_t s_warp[kJoinBlock / 32 + 1];
  __shared__ unsigned long long s_prefix;
  if (threadIdx.x == 0) s_tile = atomicAdd(J.tile_counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = lanemask_lt();
  // pass 1: per left row, count the matching right rows (warp ballots)
  for (int i = 0; i < kNlRowsPerWarp; ++i) {
    const uint32_t slot = warp * kNlRowsPerWarp + i;
    const uint32_t l = tile * kNlTile + slot;
    uint32_t c = 0;
    if (l < J.L)
      for (uint32_t r0 = 0; r0 < J.R; r0 += 32) {
        const uint32_t r = r0 + lane;
        const bool m = r < J.R && all_conds(J, l, r, -1);
        c += __popc(__ballot_sync(0xffffffffu, m));
      }
    if (lane == 0) s_cnt[slot] = c;
  }
  __syncthreads();
  const uint32_t mine = threadIdx.x < kNlTile ? s_cnt[threadIdx.x] : 0u;
  uint32_t total;
  const uint32_t excl = block_exclusive_sum<kJoinBlock>(mine, s_warp, total);
  if (threadIdx.x < kNlTile) s_cnt[threadIdx.x] = excl;  // row offset within the tile
  if (threadIdx.x < 32) {
    const unsigned long long p = tile_lookback(J.status, tile, total, J.err);
    if (threadIdx.x == 0) s_prefix = p;
  }
  __syncthreads();
  // pass 2: write matches, 32 right rows per ballot, consecutive positions
  for (int i = 0; i < kNlRowsPerWarp; ++i) {
    const uint32_t slot = warp * kNlRowsPerWarp + i;
    const uint32_t l = tile * kNlTile + slot;
    if (l >= J.L) continue;
    unsigned long long pos = s_prefix + s_cnt[slot];
    for (uint32_t r0 = 0; r0 < J.R; r0 += 32) {
      const uint32_t r = r0 + lane;
      const bool m = r < J.R && all_conds(J, l, r, -1);
      const uint32_t bal = __ballot_sync(0xffffffffu, m);
      if (m) emit_pair(J, pos + __popc(bal & lt), l, r);
      pos += __popc(bal);
    }
  }
  if (tile == gridDim.x - 1 && threadIdx.x == 0) *J.total = s_prefix + total;
}

template <typename T, int OP>
__device__ __forceinline__ bool nl_cmp(T a, T b) {
  if constexpr (OP == YQ_LT) return a < b;
  else if constexpr (OP == YQ_LE) return a <= b;
  else if constexpr (OP == YQ_GT) return a > b;
  else if constexpr (OP == YQ_GE) return a >= b;
  else return a != b;
}

// Matches per left row of one typed comparison, from the right column sorted
// ascending with its NaNs (float columns) at the end, `nvalid` values before
// them: two binary searches per left row instead of a pass over the right
// side. A NaN compares false except under <>, as in nl_cmp.
template <typename T>
__device__ __forceinline__ bool nan_of(T v) {
  return v != v;
}

template <typename T>
__global__ void k_join_count_valid(const T* __restrict__ sorted, uint32_t R, uint32_t* nvalid) {
  uint32_t nan = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < R; i += gridDim.x * blockDim.x)
    nan += nan_of(__ldg(sorted + i)) ? 1u : 0u;
  for (int d = 16; d > 0; d >>= 1) nan += __shfl_xor_sync(0xffffffffu, nan, d);
  if ((threadIdx.x & 31) == 0 && nan) atomicSub(nvalid, nan);
}

template <typename T, int OP>
__global__ void k_join_count_sorted(const T* __restrict__ lcol, uint32_t L, const T* __restrict__ sorted,
                                    const uint32_t* __restrict__ nvalid_p, uint32_t R, uint32_t* __restrict__ counts) {
  const uint32_t nvalid = *nvalid_p;
  for (uint32_t l = blockIdx.x * blockDim.x + threadIdx.x; l < L; l += gridDim.x * blockDim.x) {
    const T v = __ldg(lcol + l);
    uint32_t c;
    if (nan_of(v)) {
      c = OP == YQ_NE ? R : 0u;
    } else {
      uint32_t lo = 0, hi = nvalid;  // first position holding a value >= v
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(sorted + mid) < v) lo = mid + 1;
        else hi = mid;
      }
      const uint32_t lb = lo;
      hi = nvalid;  // first position holding a value > v
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (!(v < __ldg(sorted + mid))) lo = mid + 1;
        else hi = mid;
      }
      const uint32_t ub = lo;
      if constexpr (OP == YQ_LT) c = nvalid - ub;
      else if constexpr (OP == YQ_LE) c = nvalid - lb;
      else if constexpr (OP == YQ_GT) c = lb;
      else if constexpr (OP == YQ_GE) c = ub;
      else c = R - (ub - lb);
    }
    counts[l] = c;
  }
}

// Nested loop for one comparison of two columns of the same fixed-width
// numeric type without nulls (the common inequality join). Each warp holds
// kNtRows left values in registers and compares every right value a lane loads
// with all of them, so a comparison costs a compare, a ballot and a popc. IEEE
// comparisons give the SQL results for NaN (only <> holds) and for -0.0 = +0.0.
// Same tiles, look-back and output order (left row major, right rows
// ascending) as k_join_nested.
//
// Each left row's matches are compacted into a shared-memory ring of two runs
// (512 bytes of values, 256 row ids), whose entries sit where their output
// positions lie in a 16-byte word; a full run of values leaves 16 bytes a lane. Storing each match as it is found
// (64 unaligned bytes a store for a comparison that half the pairs pass) held
// the kernel to 2.3 TB/s of output: 20K x 20K INT32 rows under <, 199M pairs,
// 677 us for the writing alone. A row's ring is looked at once for kNtUnroll
// right values a lane (they cross at most one run), which keeps the run writer
// out of the unrolled comparisons: with a look after every value the kernel
// waited for its instructions. The right column is read through L1 (80 KB at
// 20K rows) rather than staged, so warps never wait for one another; blocks of
// four warps keep the last wave short (1,250 blocks at 20K left rows).
constexpr int kNtBlock = 128;
constexpr int kNtRows = 4;
constexpr uint32_t kNtTile = (kNtBlock / 32) * kNtRows;  // left rows per block
constexpr int kNtCountUnroll = 16;  // right values a lane loads ahead while counting,
constexpr int kNtUnroll = 4;        // and while it writes

// Cells [pb, pb + cells) of one output of left row l, moved in pieces of V
// (`pieces` a cell): a lane has four loads in flight before its first store.
// Bound by the latency of these loads where few left rows meet a long right
// side (a warp holds four left rows): 500 x 40,000 INT32 rows under <, two other
// 4-byte columns written, 0.74 ms; one load and store at a time, by runs of 128,
// 2.30; every match stored as it is found 1.27. 20-byte texts 1.60, 2.5 and 2.0.
template <typename V>
__device__ __forceinline__ void write_cells(const char* src_, char* dst_, bool right, uint32_t pieces, uint32_t l,
                                            unsigned long long pb, uint32_t cells, const uint32_t* rows) {
  constexpr int K = 4;
  const V* const src = reinterpret_cast<const V*>(src_);
  V* const dst = reinterpret_cast<V*>(dst_) + pb * pieces;
  const uint32_t lane = threadIdx.x & 31;
  V v[K];
  if (pieces == 1) {
    if (!right) {  // one value for all of them
      const V mine = __ldg(src + l);
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = mine;
    }
    for (uint32_t x0 = lane; x0 < cells; x0 += 32 * K) {
      if (right)
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (x0 + 32 * k < cells) v[k] = __ldg(src + rows[x0 + 32 * k]);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (x0 + 32 * k < cells) dst[x0 + 32 * k] = v[k];
    }
    return;
  }
  if constexpr (sizeof(V) == 4 || sizeof(V) == 16) {
    // piece x of the run is piece x % pieces of cell x / pieces, kept by steps of 32
    if (cells == 0) return;
    const uint32_t n = cells * pieces, qs = 32u / pieces, rs = 32u - qs * pieces, width = pieces * sizeof(V);
    uint32_t c = lane / pieces, r = lane - c * pieces;
    auto pass = [&](uint32_t x0, auto full) {
      constexpr bool FULL = decltype(full)::value;
      uint32_t row[K], piece[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        row[k] = right ? rows[FULL || x0 + 32 * k < n ? c : 0u] : l;  // past the end: the first cell again
        piece[k] = r;
        c += qs;
        r += rs;
        const bool carry = r >= pieces;
        r -= carry ? pieces : 0u;
        c += carry ? 1u : 0u;
      }
#pragma unroll
      for (int k = 0; k < K; ++k)
        v[k] = __ldg(reinterpret_cast<const V*>(src_ + (unsigned long long)row[k] * width) + piece[k]);
#pragma unroll
      for (int k = 0; k < K; ++k)
        if (FULL || x0 + 32 * k < n) dst[x0 + 32 * k] = v[k];
    };
    uint32_t x0 = 0;
    for (; x0 + 32 * K <= n; x0 += 32 * K) pass(x0 + lane, std::true_type{});
    if (x0 < n) pass(x0 + lane, std::false_type{});
  }
}

// Outputs [pb, pb + n) of left row l: right rows rows[0 .. n).
__device__ __forceinline__ void write_rows(const JoinParams& J, uint32_t l, unsigned long long pb, uint32_t n,
                                           const uint32_t* rows) {
  const uint32_t lane = threadIdx.x & 31;
  if (pb >= J.capacity) return;
  if (pb + n > J.capacity) n = (uint32_t)(J.capacity - pb);
  if (J.nout == 0) {
    for (uint32_t i = lane; i < n; i += 32) {
      J.out_left[pb + i] = l;
      J.out_right[pb + i] = rows[i];
    }
    return;
  }
#pragma unroll 1
  for (int o = 0; o < J.nout; ++o) {
    const JOut& w = J.out[o];
    const bool right = w.side != 0;
    if (w.width == 4) write_cells<uint32_t>(w.src, w.dst, right, 1u, l, pb, n, rows);
    else if (w.width == 8) write_cells<unsigned long long>(w.src, w.dst, right, 1u, l, pb, n, rows);
    else if (w.width == 1) write_cells<uint8_t>(w.src, w.dst, right, 1u, l, pb, n, rows);
    else if (((w.width | reinterpret_cast<uintptr_t>(w.dst) | reinterpret_cast<uintptr_t>(w.src)) & 15) == 0)
      write_cells<uint4>(w.src, w.dst, right, (uint32_t)w.width / 16u, l, pb, n, rows);
    else write_cells<uint32_t>(w.src, w.dst, right, (uint32_t)w.width / 4u, l, pb, n, rows);
    if (!w.dst_nulls) continue;
    if (w.src_nulls)
      write_cells<uint8_t>(reinterpret_cast<const char*>(w.src_nulls), reinterpret_cast<char*>(w.dst_nulls), right, 1u,
                           l, pb, n, rows);
    else
      for (uint32_t i = lane; i < n; i += 32) w.dst_nulls[pb + i] = 0;
  }
}

// VALUES: the outputs are the condition's right column and a left column as wide
// (SELECT a.x, b.y ... WHERE a.x < b.y, a.x or another column of a), or one of
// them, written from registers; otherwise the runs hold row ids. Their writer
// stands once, behind the comparisons: called out of line from each row's place
// it cost the kernel 128 registers a thread, 16 warps an SM.
template <typename T, int OP, bool VALUES>
__global__ void __launch_bounds__(kNtBlock) k_join_nested_typed(const __grid_constant__ JoinParams J) {
  using B = typename std::conditional<VALUES, T, uint32_t>::type;
  constexpr uint32_t VEC = 16 / sizeof(B);
  constexpr uint32_t RUN = VALUES ? 32 * VEC : 256;  // row ids: what an output's set-up costs, over more cells
  constexpr uint32_t RING = RUN * (RUN < 32u * kNtUnroll ? 4 : 2);  // a batch of matches crosses less than half of it
  static_assert(RING >= RUN + 32 * kNtUnroll, "a batch must not overtake the run being written");
  __shared__ __align__(16) B s_buf[kNtBlock / 32][kNtRows][RING];
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_cnt[kNtTile];
  __shared__ uint32_t s_warp[kNtBlock / 32 + 1];
  __shared__ unsigned long long s_prefix;
  if (threadIdx.x == 0) s_tile = atomicAdd(J.tile_counter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = lanemask_lt();
  const T* lcol = reinterpret_cast<const T*>(J.cond[0].l.data);
  const T* rcol = reinterpret_cast<const T*>(J.cond[0].r.data);
  const uint32_t l0 = tile * kNtTile + warp * kNtRows;
  T lv[kNtRows];
  T lw[kNtRows];  // VALUES: the left output's cells
  bool lok[kNtRows];
#pragma unroll
  for (int i = 0; i < kNtRows; ++i) {
    lok[i] = l0 + i < J.L;
    lv[i] = lok[i] ? __ldg(lcol + l0 + i) : T(0);
    lw[i] = T(0);
    if constexpr (VALUES)
      if (J.vdst[0] && lok[i]) lw[i] = __ldg(reinterpret_cast<const T*>(J.vsrc) + l0 + i);
  }
  // pass 1: matches per left row (counted up front from the sorted right
  // side when J.counts is given, else here over the whole right side)
  if (J.counts) {
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < kNtRows; ++i) s_cnt[warp * kNtRows + i] = lok[i] ? __ldg(J.counts + l0 + i) : 0u;
  } else {
    uint32_t cnt[kNtRows];
#pragma unroll
    for (int i = 0; i < kNtRows; ++i) cnt[i] = 0;
    // per-lane counts (a compare and an add a comparison), summed over the warp below
    constexpr uint32_t STEP = 32 * kNtCountUnroll;
    const uint32_t whole = J.R / STEP * STEP;
    for (uint32_t r0 = lane; r0 < whole; r0 += STEP) {
      T rv[kNtCountUnroll];
#pragma unroll
      for (int u = 0; u < kNtCountUnroll; ++u) rv[u] = __ldg(rcol + r0 + u * 32);
#pragma unroll
      for (int u = 0; u < kNtCountUnroll; ++u)
#pragma unroll
        for (int i = 0; i < kNtRows; ++i) cnt[i] += nl_cmp<T, OP>(lv[i], rv[u]) ? 1u : 0u;
    }
    for (uint32_t r0 = whole + lane; r0 < J.R; r0 += 32 * kNtUnroll) {
      T rv[kNtUnroll];
#pragma unroll
      for (int u = 0; u < kNtUnroll; ++u) rv[u] = r0 + u * 32 < J.R ? __ldg(rcol + r0 + u * 32) : T(0);
#pragma unroll
      for (int u = 0; u < kNtUnroll; ++u)
#pragma unroll
        for (int i = 0; i < kNtRows; ++i) cnt[i] += r0 + u * 32 < J.R && nl_cmp<T, OP>(lv[i], rv[u]) ? 1u : 0u;
    }
#pragma unroll
    for (int i = 0; i < kNtRows; ++i)
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) cnt[i] += __shfl_xor_sync(0xffffffffu, cnt[i], d);
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < kNtRows; ++i) s_cnt[warp * kNtRows + i] = lok[i] ? cnt[i] : 0u;
  }
  __syncthreads();
  const uint32_t mine = threadIdx.x < kNtTile ? s_cnt[threadIdx.x] : 0u;
  uint32_t total32;
  unsigned long long excl, total;
  if (J.R < (1u << 27)) {  // kNtTile rows of up to R matches: the sum fits 32 bits
    excl = block_exclusive_sum<kNtBlock>(mine, s_warp, total32);
    total = total32;
  } else {
    __shared__ unsigned long long s_wide[2 * (kNtBlock / 32 + 1)];
    unsigned long long zero = 0, tz;
    excl = mine;
    block_exclusive_sum2<kNtBlock>(excl, zero, s_wide, total, tz);
  }
  __shared__ unsigned long long s_off[kNtTile];
  if (threadIdx.x < kNtTile) s_off[threadIdx.x] = excl;  // row offset within the tile
  if (threadIdx.x < 32) {
    const unsigned long long p = tile_lookback(J.status, tile, total, J.err);
    if (threadIdx.x == 0) s_prefix = p;
  }
  __syncthreads();
  const unsigned long long prefix = s_prefix;
  if (tile == gridDim.x - 1 && threadIdx.x == 0) *J.total = prefix + total;
  if (prefix >= J.capacity) return;  // nothing of this tile is stored
  // pass 2: write the matches, consecutive positions per left row
  T* const vl = reinterpret_cast<T*>(J.vdst[0]);
  T* const vr = reinterpret_cast<T*>(J.vdst[1]);
  // every pair of this tile fits and the outputs take 16-byte stores
  const bool whole = prefix + total <= J.capacity &&
                     ((reinterpret_cast<uintptr_t>(vl) | reinterpret_cast<uintptr_t>(vr)) & 15) == 0;
  unsigned long long p0[kNtRows];  // output position of ring entry 0 (a whole 16-byte word)
  uint32_t head[kNtRows];          // first entry of the run that is not yet written
  uint32_t fill[kNtRows];          // entries so far, the head's empty ones included
  bool any = false;
#pragma unroll
  for (int i = 0; i < kNtRows; ++i) {
    const unsigned long long p = prefix + s_off[warp * kNtRows + i];
    head[i] = fill[i] = (uint32_t)(p & (VEC - 1));
    p0[i] = p - head[i];
    lok[i] = lok[i] && s_cnt[warp * kNtRows + i] > 0 && p < J.capacity;
    any |= lok[i];
  }
  if (!any) return;
  // VALUES: entries [head, n) of row i, all within one run
  auto flush = [&](int i, uint32_t n) {
    __syncwarp();
    const uint32_t r0 = head[i] & ~(RUN - 1u);  // the run's first entry
    const B* buf = s_buf[warp][i] + (r0 & (RING - 1u));
    const unsigned long long pos = p0[i] + r0;
    if constexpr (VALUES) {
      if (whole && head[i] == r0 && n == r0 + RUN) {
        if (vl) {
          T x[VEC];
#pragma unroll
          for (uint32_t v = 0; v < VEC; ++v) x[v] = lw[i];
          *reinterpret_cast<uint4*>(vl + pos + lane * VEC) = *reinterpret_cast<const uint4*>(x);
        }
        if (vr) *reinterpret_cast<uint4*>(vr + pos + lane * VEC) = *reinterpret_cast<const uint4*>(buf + lane * VEC);
      } else {
        for (uint32_t x = head[i] - r0 + lane; x < n - r0; x += 32)
          if (pos + x < J.capacity) {
            if (vl) vl[pos + x] = lw[i];
            if (vr) vr[pos + x] = buf[x];
          }
      }
    }
    __syncwarp();
    head[i] = n;
  };
  // Row ids: the runs that are full, and on the last batch all that is left.
  auto flush_rows = [&](bool last) {
    __syncwarp();
    for (;;) {
      uint32_t h = 0u, n = 0u;
      unsigned long long p = 0ull;
      int row = -1;
#pragma unroll
      for (int i = kNtRows - 1; i >= 0; --i) {
        const uint32_t end = (head[i] | (RUN - 1u)) + 1u;
        if (fill[i] >= end || (last && fill[i] > head[i])) {
          row = i;
          h = head[i];
          n = min(fill[i], end);
          p = p0[i];
        }
      }
      if (row < 0) break;
      write_rows(J, l0 + row, p + h, n - h, reinterpret_cast<const uint32_t*>(s_buf[warp][row]) + (h & (RING - 1u)));
#pragma unroll
      for (int i = 0; i < kNtRows; ++i)
        if (i == row) head[i] = n;
    }
    __syncwarp();
  };
  // kNtUnroll right values a lane against every row; FULL: all of them exist
  auto batch = [&](uint32_t r0, auto full) {
    constexpr bool FULL = decltype(full)::value;
    T rv[kNtUnroll];
#pragma unroll
    for (int u = 0; u < kNtUnroll; ++u) rv[u] = FULL || r0 + u * 32 < J.R ? __ldg(rcol + r0 + u * 32) : T(0);
#pragma unroll
    for (int i = 0; i < kNtRows; ++i) {
      const uint32_t before = fill[i];
#pragma unroll
      for (int u = 0; u < kNtUnroll; ++u) {
        const bool m = (FULL || r0 + u * 32 < J.R) && lok[i] && nl_cmp<T, OP>(lv[i], rv[u]);
        const uint32_t bal = __ballot_sync(0xffffffffu, m);
        if (m) {
          const uint32_t at = (fill[i] + __popc(bal & lt)) & (RING - 1u);
          if constexpr (VALUES) s_buf[warp][i][at] = rv[u];
          else s_buf[warp][i][at] = r0 + u * 32;
        }
        fill[i] += __popc(bal);
      }
      if constexpr (VALUES)
        for (uint32_t run = (before | (RUN - 1u)) + 1u; run <= fill[i]; run += RUN) flush(i, run);
    }
  };
  uint32_t r0 = lane;
  for (; r0 - lane + 32 * kNtUnroll <= J.R; r0 += 32 * kNtUnroll) {
    batch(r0, std::true_type{});
    if constexpr (!VALUES) {
      bool due = false;
#pragma unroll
      for (int i = 0; i < kNtRows; ++i) due |= fill[i] > (head[i] | (RUN - 1u));
      if (due) flush_rows(false);
    }
  }
  if (r0 - lane < J.R) batch(r0, std::false_type{});
  if constexpr (VALUES) {
#pragma unroll
    for (int i = 0; i < kNtRows; ++i)
      if (lok[i] && fill[i] > head[i]) flush(i, fill[i]);
  } else {
    flush_rows(true);
  }
}

template <typename T, bool VALUES>
static int launch_nested_typed_op(int op, unsigned grid, const JoinParams& J, cudaStream_t s) {
  switch (op) {
    case YQ_LT: k_join_nested_typed<T, YQ_LT, VALUES><<<grid, kNtBlock, 0, s>>>(J); break;
    case YQ_LE: k_join_nested_typed<T, YQ_LE, VALUES><<<grid, kNtBlock, 0, s>>>(J); break;
    case YQ_GT: k_join_nested_typed<T, YQ_GT, VALUES><<<grid, kNtBlock, 0, s>>>(J); break;
    case YQ_GE: k_join_nested_typed<T, YQ_GE, VALUES><<<grid, kNtBlock, 0, s>>>(J); break;
    case YQ_NE: k_join_nested_typed<T, YQ_NE, VALUES><<<grid, kNtBlock, 0, s>>>(J); break;
    default: return YQ_ERR_UNSUPPORTED;  // equalities take a table or the general loop
  }
  return YQ_OK;
}

template <typename T>
static int launch_nested_typed(int op, unsigned grid, JoinParams J, cudaStream_t s) {
  // a left column of the condition's width and the condition's right column, each at most once
  bool values = J.nout >= 1 && J.nout <= 2;
  J.vdst[0] = J.vdst[1] = nullptr;
  for (int o = 0; o < J.nout && values; ++o) {
    const JOut& w = J.out[o];
    values = w.width == (int)sizeof(T) && !w.dst_nulls && !J.vdst[w.side != 0] && (!w.side || w.src == J.cond[0].r.data);
    if (!values) break;
    J.vdst[w.side != 0] = w.dst;
    if (!w.side) J.vsrc = w.src;
  }
  return values ? launch_nested_typed_op<T, true>(op, grid, J, s) : launch_nested_typed_op<T, false>(op, grid, J, s);
}

// ------------------------------------------------------- cross product
// Every (l, r), left-major: output row l*R + r.
__global__ void __launch_bounds__(256) k_cross_fill(const __grid_constant__ JoinParams J) {
  const unsigned long long n = (unsigned long long)J.L * J.R;
  const unsigned long long lim = n < J.capacity ? n : J.capacity;
  for (unsigned long long p = blockIdx.x * 256ull + threadIdx.x; p < lim; p += (unsigned long long)gridDim.x * 256ull) {
    const uint32_t l = (uint32_t)(p / J.R), r = (uint32_t)(p % J.R);
    emit_pair(J, p, l, r);
  }
}

template <bool STAGED>
__global__ void __launch_bounds__(kRowBlock, 2) k_join_aggregate(const __grid_constant__ JAParams F, uint32_t n,
                                                                 Acc* __restrict__ partials, uint32_t* ticket,
                                                                 Acc* state) {
  join_aggregate_body<STAGED, InterpRunner>(F, n, partials, ticket, state);
}

// ---------------------------------------------------------------- host
static bool join_col_ok(const yq_column& c) {
  if (!c.data) return false;
  return ProgramBuilder::valid_column(c);
}

static JCol jcol(const yq_column& c) {
  JCol j;
  j.data = static_cast<const char*>(c.data);
  j.nulls = c.nulls;
  j.type = c.type;
  j.width = c.width;
  return j;
}

static bool hashable(int t) {
  return t == YQ_INT32 || t == YQ_INT64 || t == YQ_DATETIME || t == YQ_FLOAT32 || t == YQ_FLOAT64 || t == YQ_BOOL;
}

// (2^31, the greatest there is, for more: sizes are asked for any row count)
static uint32_t pow2_at_least(uint32_t x) {
  uint32_t p = 16;
  while (p < x && p < (1u << 31)) p <<= 1;
  return p;
}

static size_t table_smem(uint32_t nbuckets, uint32_t nrows, bool with_rows) {
  return sizeof(uint32_t) * ((nbuckets + 2) & ~1u) + sizeof(unsigned long long) * nrows +
         (with_rows ? sizeof(uint32_t) * nrows : 0);
}

static int build_table(const yq_batch* right, const yq_program* pred, const yq_constants* consts, int key_col,
                       uint32_t nbuckets, uint32_t* bstart, unsigned long long* hkeys, uint32_t* hrows,
                       uint32_t* counts, cudaStream_t s) {
  BuildParams B;
  memset(&B, 0, sizeof(B));
  ProgramBuilder PB;
  YQ_TRY(PB.set_columns(right->columns, right->ncols));
  YQ_TRY(PB.set_constants(consts));
  if (pred && pred->len > 0) {
    int t = -1;
    YQ_TRY(PB.append(pred, t));
    if (t != YQ_BOOL) return YQ_ERR_INVALID_ARG;
    YQ_TRY(PB.emit(OP_EMIT_PRED, 0, 0, YQ_BOOL));
  }
  YQ_TRY(PB.finalize());
  memcpy(&B.P, &PB.P, sizeof(VmProgram));
  B.pred_len = PB.len;
  B.key = jcol(right->columns[key_col]);
  B.R = right->rows;
  B.nbuckets = nbuckets;
  B.bstart = bstart;
  B.hkeys = hkeys;
  B.hrows = hrows;
  B.counts = counts;
  const size_t smem = sizeof(uint32_t) * (nbuckets + kHashMaxRows + 40);
  YQ_TRY(kernel_allow_smem((const void*)k_hash_build, smem));
  ProfScope ps("join_hash_build", s, (double)right->rows * right->columns[key_col].width);
  k_hash_build<<<1, kBuildBlock, smem, s>>>(B);
  YQ_CHECK_LAUNCH();
  return YQ_OK;
}

// The typed nested loop counts each left row's matches up front from this many
// pairs on (and a right side worth sorting): one sort of the right key and two
// binary searches per left row, instead of a comparison pass over L x R.
constexpr uint32_t kCountFirstRows = 4096;
constexpr unsigned long long kCountFirstPairs = 1ull << 31;
static bool counts_first(uint32_t L, uint32_t R) {
  return R >= kCountFirstRows && (unsigned long long)L * R >= kCountFirstPairs;
}

// Sort workspace for a right side of R rows (an 8-byte key, nullable or not,
// bounds the 4-byte ones). Sizing reads no column data: the placeholder
// pointers only have to be non-null.
static size_t join_sort_bytes(uint32_t R, bool nullable) {
  const uintptr_t some = 256;
  yq_column dummy{reinterpret_cast<void*>(some), nullable ? reinterpret_cast<const uint8_t*>(some) : nullptr, YQ_INT64, 8};
  KeyJob j{dummy, 0, 0};
  uint32_t offs[2] = {0, R};
  size_t sb = 0;
  if (sort_segments_impl(&j, 1, R, offs, 1, nullptr, nullptr, nullptr, 0, nullptr, &sb) != YQ_OK) return 0;
  return sb;
}

struct CountWs {
  char* sort_ws;
  size_t sort_bytes;
  uint32_t* perm;     // [R]
  char* sorted;       // [R] values of the right key, ascending
  uint32_t* nvalid;   // [1] values before the NaNs
  uint32_t* counts;   // [L]
};

static void count_ws_layout(uint32_t L, uint32_t R, size_t sort_bytes, WsSize& w) {
  w.add<char>(sort_bytes);
  w.add<uint32_t>(R ? R : 1);
  w.add<unsigned long long>(R ? R : 1);
  w.add<uint32_t>(4);
  w.add<uint32_t>(L ? L : 1);
}

// Slots of the sorted join's table: a load of 0.33 to 0.67.
static uint32_t sorted_slots(uint32_t R) { return pow2_at_least(R + R / 2); }

static void sorted_ws_layout(uint32_t R, size_t sort_bytes, WsSize& w) {
  w.add<char>(sort_bytes);
  w.add<uint32_t>(R);
  w.add<uint4>(sorted_slots(R));
}

template <typename T>
static int count_matches_typed(const JoinParams& J, const CountWs& c, cudaStream_t s) {
  const JCond& c0 = J.cond[0];
  const yq_column rc{const_cast<char*>(c0.r.data), nullptr, c0.r.type, c0.r.width};
  KeyJob j{rc, 0, 0};
  uint32_t offs[2] = {0, J.R};
  YQ_TRY(sort_segments_impl(&j, 1, J.R, offs, 1, c.perm, nullptr, c.sort_ws, c.sort_bytes, s, nullptr));
  const yq_column sc{c.sorted, nullptr, rc.type, rc.width};
  YQ_TRY(gather_impl(&rc, 1, c.perm, J.R, &sc, nullptr, s));
  const uint32_t R = J.R;
  YQ_TRY(h2d_async(c.nvalid, &R, sizeof(R), s));
  const int grid = sm_count() * 4;
  const T* sorted = reinterpret_cast<const T*>(c.sorted);
  const T* lcol = reinterpret_cast<const T*>(c0.l.data);
  k_join_count_valid<T><<<grid, 256, 0, s>>>(sorted, J.R, c.nvalid);
  YQ_CHECK_LAUNCH();
  switch (c0.cmp) {
    case YQ_LT: k_join_count_sorted<T, YQ_LT><<<grid, 256, 0, s>>>(lcol, J.L, sorted, c.nvalid, R, c.counts); break;
    case YQ_LE: k_join_count_sorted<T, YQ_LE><<<grid, 256, 0, s>>>(lcol, J.L, sorted, c.nvalid, R, c.counts); break;
    case YQ_GT: k_join_count_sorted<T, YQ_GT><<<grid, 256, 0, s>>>(lcol, J.L, sorted, c.nvalid, R, c.counts); break;
    case YQ_GE: k_join_count_sorted<T, YQ_GE><<<grid, 256, 0, s>>>(lcol, J.L, sorted, c.nvalid, R, c.counts); break;
    default: k_join_count_sorted<T, YQ_NE><<<grid, 256, 0, s>>>(lcol, J.L, sorted, c.nvalid, R, c.counts); break;
  }
  YQ_CHECK_LAUNCH();
  return YQ_OK;
}

// Shared by yq_join_pairs / yq_join_project.
static int join_impl(const yq_batch* left, const yq_batch* right, const yq_join_cond* conds, const int32_t* disjunct,
                     int32_t ncond, const yq_join_output* outputs, int32_t nout, yq_column* out, uint32_t* out_left,
                     uint32_t* out_right, uint64_t capacity, uint64_t* count_host, void* workspace,
                     size_t workspace_bytes, cudaStream_t s) {
  if (!left || !right || ncond < 0 || ncond > kMaxConds || (ncond > 0 && !conds) || nout < 0 || nout > kMaxJoinOut ||
      (nout > 0 && (!outputs || !out)))
    return YQ_ERR_INVALID_ARG;
  JoinParams J;
  memset(&J, 0, sizeof(J));
  J.L = left->rows;
  J.R = right->rows;
  J.ncond = ncond;
  J.eq = -1;
  J.ngroups = 1;
  if (disjunct && ncond > 0) {  // groups numbered 0..G-1, each used by some condition
    int g = 0;
    uint32_t used = 0u;
    for (int i = 0; i < ncond; ++i) {
      if (disjunct[i] < 0 || disjunct[i] >= kMaxConds) return YQ_ERR_INVALID_ARG;
      J.group[i] = (int8_t)disjunct[i];
      used |= 1u << disjunct[i];
      g = disjunct[i] + 1 > g ? disjunct[i] + 1 : g;
    }
    if (used != (1u << g) - 1u) return YQ_ERR_INVALID_ARG;
    J.ngroups = g;
  }
  for (int i = 0; i < ncond; ++i) {
    const yq_join_cond& c = conds[i];
    if (c.left_col < 0 || c.left_col >= left->ncols || c.right_col < 0 || c.right_col >= right->ncols ||
        c.cmp < YQ_LT || c.cmp > YQ_NE)
      return YQ_ERR_INVALID_ARG;
    const yq_column& a = left->columns[c.left_col];
    const yq_column& b = right->columns[c.right_col];
    if (!join_col_ok(a) || !join_col_ok(b) || a.type != b.type) return YQ_ERR_INVALID_ARG;
    J.cond[i].l = jcol(a);
    J.cond[i].r = jcol(b);
    J.cond[i].cmp = c.cmp;
    if (J.eq < 0 && J.ngroups == 1 && c.cmp == YQ_EQ && hashable(a.type)) J.eq = i;
  }
  for (int o = 0; o < nout; ++o) {
    const yq_join_output& w = outputs[o];
    const yq_batch* side = w.side ? right : left;
    if (w.column < 0 || w.column >= side->ncols) return YQ_ERR_INVALID_ARG;
    const yq_column& c = side->columns[w.column];
    if (!join_col_ok(c) || out[o].type != c.type || out[o].width != c.width || !out[o].data) return YQ_ERR_INVALID_ARG;
    J.out[o].src = static_cast<const char*>(c.data);
    J.out[o].src_nulls = c.nulls;
    J.out[o].dst = static_cast<char*>(out[o].data);
    J.out[o].dst_nulls = const_cast<uint8_t*>(out[o].nulls);
    J.out[o].width = c.width;
    J.out[o].side = w.side;
  }
  J.nout = nout;
  if (nout == 0 && capacity > 0 && (!out_left || !out_right)) return YQ_ERR_INVALID_ARG;
  J.out_left = out_left;
  J.out_right = out_right;
  J.capacity = capacity;

  if (J.L == 0 || J.R == 0) {
    if (count_host) *count_host = 0;
    return YQ_OK;
  }
  if (ncond == 0) {  // cross product: size known up front
    const unsigned long long n = (unsigned long long)J.L * J.R;
    double row_bytes = nout == 0 ? 8.0 : 0.0;
    for (int o = 0; o < nout; ++o) row_bytes += J.out[o].width + (J.out[o].dst_nulls ? 1 : 0);
    ProfScope ps("cross_product", s, (double)(n < capacity ? n : capacity) * row_bytes);
    const unsigned long long lim = n < capacity ? n : capacity;
    int grid = (int)((lim + 255) / 256);
    const int cap = sm_count() * 16;
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    k_cross_fill<<<grid, 256, 0, s>>>(J);
    YQ_CHECK_LAUNCH();
    if (count_host) *count_host = n;
    return n > capacity ? YQ_ERR_CAPACITY : YQ_OK;
  }

  // The sorted table holds any length the sort takes; the shared-memory table is
  // built by one block and copied by every block of the probe. Its build is the
  // longer one from about 4,096 rows on (20K left rows to 8,000 right ones:
  // 0.30 ms against 0.16), its copies cost more than the sort's launches from
  // about 2^32 pairs on (2M to 4,000: 0.36 ms against 0.23; 2M to 2,000: 0.23
  // both; 20K to 2,000: 0.15 against 0.18). BOOL keys stay with the other paths
  // (the sort orders every non-zero byte as one value, a join compares the
  // bytes), and float keys as long as the shared-memory table holds them (it
  // joins equal NaN bit patterns).
  const bool eq_float = J.eq >= 0 && (J.cond[J.eq].r.type == YQ_FLOAT32 || J.cond[J.eq].r.type == YQ_FLOAT64);
  const uint32_t table_rows =
      eq_float ? kHashMaxRows : ((unsigned long long)J.L * J.R > (1ull << 32) ? kSortedMinRows : kTableRows);
  const size_t eq_sort_bytes = J.eq >= 0 && J.R > table_rows && J.cond[J.eq].r.type != YQ_BOOL
                                   ? join_sort_bytes(J.R, J.cond[J.eq].r.nulls != nullptr) : 0;
  const JCond& t0 = J.cond[0];
  bool use_sorted = eq_sort_bytes != 0, use_hash, typed, small, count_first;
  uint32_t nbuckets, ntiles;
  size_t count_bytes;
  Workspace ws;
  for (;;) {
    use_hash = J.eq >= 0 && !use_sorted && J.R <= kHashMaxRows;
    nbuckets = use_hash ? pow2_at_least(J.R) : 0u;
    typed = !use_hash && !use_sorted && J.ncond == 1 && J.ngroups == 1 && t0.l.type == t0.r.type && !t0.l.nulls &&
                       !t0.r.nulls && t0.l.width == t0.r.width && t0.cmp != YQ_EQ &&
                       (t0.l.type == YQ_INT32 || t0.l.type == YQ_FLOAT32 || t0.l.type == YQ_INT64 ||
                        t0.l.type == YQ_DATETIME || t0.l.type == YQ_FLOAT64);
    small = typed && J.R <= (J.L >= kManyLeft ? kSmallRightMany : kSmallRight);
    const uint32_t tile_rows = use_sorted ? sorted_tile_rows(J.L, J.ncond == 1)
                               : use_hash ? kJoinTile
                               : small    ? sorted_tile_rows(J.L, false)
                               : typed    ? kNtTile : kNlTile;
    ntiles = ceil_div<uint32_t>(J.L, tile_rows);
    count_bytes = typed && counts_first(J.L, J.R) ? join_sort_bytes(J.R, false) : 0;
    count_first = count_bytes != 0;  // else (a right side too long to sort) the kernel counts
    WsSize w;
    w.add<uint32_t>(nbuckets + 1);
    w.add<unsigned long long>(use_hash ? J.R : 1);
    w.add<uint32_t>(use_hash ? J.R : 1);
    w.add<unsigned long long>((size_t)ntiles + 3);
    w.add<uint32_t>(8);
    if (count_first) count_ws_layout(J.L, J.R, count_bytes, w);
    if (use_sorted) sorted_ws_layout(J.R, eq_sort_bytes, w);
    const int st = ws.acquire(workspace, workspace_bytes, w.total(), s);
    if (st == YQ_OK) break;
    // no room for the sorted table (up to 70 bytes a right row): the forms that
    // need a few words a tile give the same pairs
    if (!use_sorted || !(workspace ? workspace_bytes < w.total() : st == YQ_ERR_ALLOC)) return st;
    use_sorted = false;
  }
  uint32_t* d_bstart = ws.take<uint32_t>(nbuckets + 1);
  unsigned long long* d_hkeys = ws.take<unsigned long long>(use_hash ? J.R : 1);
  uint32_t* d_hrows = ws.take<uint32_t>(use_hash ? J.R : 1);
  J.status = ws.take<unsigned long long>((size_t)ntiles + 3);  // then [total][tile counter, err]
  uint32_t* d_build = ws.take<uint32_t>(8);                    // [0..1] build counts
  J.total = J.status + ntiles + 1;
  J.tile_counter = reinterpret_cast<uint32_t*>(J.total + 1);
  J.err = J.tile_counter + 1;
  CountWs cw{};
  if (count_first) {
    cw.sort_ws = ws.take<char>(count_bytes);
    cw.sort_bytes = count_bytes;
    cw.perm = ws.take<uint32_t>(J.R ? J.R : 1);
    cw.sorted = reinterpret_cast<char*>(ws.take<unsigned long long>(J.R ? J.R : 1));
    cw.nvalid = ws.take<uint32_t>(4);
    cw.counts = ws.take<uint32_t>(J.L ? J.L : 1);
  }
  YQ_TRY_CUDA(cudaMemsetAsync(J.status, 0, ((size_t)ntiles + 3) * sizeof(unsigned long long), s));
  double out_row_bytes = nout == 0 ? 8.0 : 0.0;
  for (int o = 0; o < nout; ++o) out_row_bytes += J.out[o].width + (J.out[o].dst_nulls ? 1 : 0);
  if (use_hash) {
    YQ_TRY_CUDA(cudaMemsetAsync(d_build, 0, 8 * sizeof(uint32_t), s));
    YQ_TRY(build_table(right, nullptr, nullptr, conds[J.eq].right_col, nbuckets, d_bstart, d_hkeys, d_hrows, d_build,
                       s));
    J.bstart = d_bstart;
    J.hkeys = d_hkeys;
    J.hrows = d_hrows;
    J.nbuckets = nbuckets;
    J.hrows_n = J.R;
    const size_t smem = table_smem(nbuckets, J.R, true);
    YQ_TRY(kernel_allow_smem((const void*)k_join_hash, smem));
    ProfScope ps("join_hash_probe", s, (double)J.L * left->columns[conds[J.eq].left_col].width);
    k_join_hash<<<ntiles, kJoinBlock, smem, s>>>(J);
    YQ_CHECK_LAUNCH();
  } else if (use_sorted) {
    const JCond& ec = J.cond[J.eq];
    char* sort_ws = ws.take<char>(eq_sort_bytes);
    uint32_t* perm = ws.take<uint32_t>(J.R);
    SortedJoin S;
    S.perm = perm;
    S.rows = J.R;
    S.nslots = sorted_slots(J.R);
    S.tile_rows = sorted_tile_rows(J.L, J.ncond == 1);
    S.slots = ws.take<uint4>(S.nslots);
    const yq_column rc{const_cast<char*>(ec.r.data), ec.r.nulls, ec.r.type, ec.r.width};
    KeyJob j{rc, 0, 0};
    uint32_t offs[2] = {0, J.R};
    uint32_t* sort_err = nullptr;
    // A 4-byte key keeps all four passes rather than wait for the host to learn
    // which of them change nothing (13 us a pass against some 20 for the wait).
    const yq_sort_config keep{0, 0, 0, 1};
    const bool no_wait = ec.r.width == 4 && !ec.r.nulls;
    YQ_TRY(sort_segments_impl(&j, 1, J.R, offs, 1, perm, no_wait ? &keep : nullptr, sort_ws, eq_sort_bytes, s, nullptr,
                              nullptr, nullptr, true, &sort_err));
    YQ_TRY_CUDA(cudaMemsetAsync(S.slots, 0xff, (size_t)S.nslots * sizeof(uint4), s));
    int grid = (int)ceil_div<uint32_t>(J.R, 256);
    if (grid > sm_count() * 8) grid = sm_count() * 8;
    {
      ProfScope ps("join_sorted_build", s, (double)J.R * ec.r.width);
      k_join_sorted_build<<<grid, 256, 0, s>>>(S, ec.r, J.R, sort_err, J.err);
      YQ_CHECK_LAUNCH();
    }
    ProfScope ps("join_sorted_probe", s, (double)J.L * ec.l.width);
    if (J.ncond == 1) k_join_sorted<<<ntiles, kJoinBlock, 0, s>>>(J, S);
    else k_join_candidates<false><<<ntiles, kJoinBlock, 0, s>>>(J, S);
    YQ_CHECK_LAUNCH();
  } else {
    ProfScope ps("join_nested_loop", s, (double)J.L * J.R * 0.0);
    const JCond& c0 = J.cond[0];
    if (small) {
      SortedJoin S{};
      S.rows = J.R;
      S.tile_rows = sorted_tile_rows(J.L, false);
      k_join_candidates<true><<<ntiles, kJoinBlock, 0, s>>>(J, S);
    } else if (typed) {
      if (count_first) {
        switch (c0.l.type) {
          case YQ_INT32: YQ_TRY(count_matches_typed<int32_t>(J, cw, s)); break;
          case YQ_FLOAT32: YQ_TRY(count_matches_typed<float>(J, cw, s)); break;
          case YQ_FLOAT64: YQ_TRY(count_matches_typed<double>(J, cw, s)); break;
          default: YQ_TRY(count_matches_typed<long long>(J, cw, s)); break;  // INT64, DATETIME
        }
        J.counts = cw.counts;
      }
      switch (c0.l.type) {
        case YQ_INT32: YQ_TRY(launch_nested_typed<int32_t>(c0.cmp, ntiles, J, s)); break;
        case YQ_FLOAT32: YQ_TRY(launch_nested_typed<float>(c0.cmp, ntiles, J, s)); break;
        case YQ_FLOAT64: YQ_TRY(launch_nested_typed<double>(c0.cmp, ntiles, J, s)); break;
        default: YQ_TRY(launch_nested_typed<long long>(c0.cmp, ntiles, J, s)); break;  // INT64, DATETIME
      }
    } else {
      k_join_nested<<<ntiles, kJoinBlock, 0, s>>>(J);
    }
    YQ_CHECK_LAUNCH();
  }
  struct {
    unsigned long long total;
    uint32_t counter, err;
  } h{};
  YQ_TRY(d2h_sync(&h, J.total, sizeof(h), s));
  const unsigned long long h_total = h.total;
  const uint32_t h_err = h.err;
  if (count_host) *count_host = h_total;
  if (h_err & kErrTimeout) return YQ_ERR_TIMEOUT;
  if (h_err & kErrBounds) return YQ_ERR_INVALID_ARG;
  return h_total > capacity ? YQ_ERR_CAPACITY : YQ_OK;
}

}  // namespace yq

using namespace yq;

extern "C" {

size_t yq_join_workspace_size(uint32_t left_rows, uint32_t right_rows) {
  const uint32_t nb = pow2_at_least(right_rows);
  uint32_t ntiles = ceil_div<uint32_t>(left_rows, kNtTile < kNlTile ? kNtTile : kNlTile);
  for (const bool eq_only : {false, true}) {
    const uint32_t sorted = ceil_div<uint32_t>(left_rows, sorted_tile_rows(left_rows, eq_only));
    if (sorted > ntiles) ntiles = sorted;
  }
  WsSize w;
  w.add<uint32_t>(nb + 1);
  w.add<unsigned long long>(right_rows ? right_rows : 1);
  w.add<uint32_t>(right_rows ? right_rows : 1);
  w.add<unsigned long long>((size_t)ntiles + 3);
  w.add<uint32_t>(8);
  WsSize sorted = w;
  if (counts_first(left_rows, right_rows)) count_ws_layout(left_rows, right_rows, join_sort_bytes(right_rows, false), w);
  const size_t eq_sort_bytes = right_rows > kSortedMinRows ? join_sort_bytes(right_rows, true) : 0;
  if (eq_sort_bytes) sorted_ws_layout(right_rows, eq_sort_bytes, sorted);  // (0: more rows than the sort takes)
  return w.total() > sorted.total() ? w.total() : sorted.total();
}

int yq_join_pairs(const yq_batch* left, const yq_batch* right, const yq_join_cond* conds, int32_t ncond,
                  uint32_t* out_left, uint32_t* out_right, uint64_t capacity, uint64_t* count_host, void* workspace,
                  size_t workspace_bytes, void* stream) {
  return join_impl(left, right, conds, nullptr, ncond, nullptr, 0, nullptr, out_left, out_right, capacity,
                   count_host, workspace, workspace_bytes, as_stream(stream));
}

int yq_join_project(const yq_batch* left, const yq_batch* right, const yq_join_cond* conds, int32_t ncond,
                    const yq_join_output* outputs, int32_t nout, yq_column* out, uint64_t capacity,
                    uint64_t* count_host, void* workspace, size_t workspace_bytes, void* stream) {
  if (nout <= 0) return YQ_ERR_INVALID_ARG;
  return join_impl(left, right, conds, nullptr, ncond, outputs, nout, out, nullptr, nullptr, capacity, count_host,
                   workspace, workspace_bytes, as_stream(stream));
}

int yq_join_pairs_or(const yq_batch* left, const yq_batch* right, const yq_join_cond* conds, const int32_t* disjunct,
                     int32_t ncond, uint32_t* out_left, uint32_t* out_right, uint64_t capacity, uint64_t* count_host,
                     void* workspace, size_t workspace_bytes, void* stream) {
  if (ncond <= 0 || !disjunct) return YQ_ERR_INVALID_ARG;
  return join_impl(left, right, conds, disjunct, ncond, nullptr, 0, nullptr, out_left, out_right, capacity,
                   count_host, workspace, workspace_bytes, as_stream(stream));
}

int yq_join_project_or(const yq_batch* left, const yq_batch* right, const yq_join_cond* conds,
                       const int32_t* disjunct, int32_t ncond, const yq_join_output* outputs, int32_t nout,
                       yq_column* out, uint64_t capacity, uint64_t* count_host, void* workspace,
                       size_t workspace_bytes, void* stream) {
  if (nout <= 0 || ncond <= 0 || !disjunct) return YQ_ERR_INVALID_ARG;
  return join_impl(left, right, conds, disjunct, ncond, outputs, nout, out, nullptr, nullptr, capacity, count_host,
                   workspace, workspace_bytes, as_stream(stream));
}

size_t yq_join_aggregate_workspace_size(uint32_t fact_rows, uint32_t dim_rows, int32_t nagg) {
  (void)fact_rows;
  (void)nagg;
  const uint32_t nb = pow2_at_least(dim_rows);
  WsSize w;
  w.add<uint32_t>(nb + 1);
  w.add<unsigned long long>(dim_rows ? dim_rows : 1);
  w.add<uint32_t>(dim_rows ? dim_rows : 1);
  w.add<uint32_t>(8);
  w.add<Acc>((size_t)sm_count() * 8 * YQ_MAX_AGGREGATES);
  return w.total();
}

}  // extern "C"

// The fact side of a star-join aggregate: predicate and aggregate inputs as
// one program over the fact columns.
static int join_agg_params(const yq_batch* fact, const yq_program* fact_predicate, int32_t fact_key,
                           const yq_constants* constants, const yq_agg_spec* aggs, int32_t nagg, JAParams& F) {
  memset(&F, 0, sizeof(F));
  {
    ProgramBuilder B;
    YQ_TRY(B.set_columns(fact->columns, fact->ncols));
    YQ_TRY(B.set_constants(constants));
    if (fact_predicate && fact_predicate->len > 0) {
      int t = -1;
      YQ_TRY(B.append(fact_predicate, t));
      if (t != YQ_BOOL) return YQ_ERR_INVALID_ARG;
      YQ_TRY(B.emit(OP_EMIT_PRED, 0, 0, YQ_BOOL));
    }
    const int pred_end = B.len;
    for (int a = 0; a < nagg; ++a) {
      const yq_agg_spec& g = aggs[a];
      if (g.kind < YQ_AGG_COUNT_STAR || g.kind > YQ_AGG_MAX) return YQ_ERR_INVALID_ARG;
      const bool flt = (g.input_type == YQ_FLOAT32 || g.input_type == YQ_FLOAT64);
      uint8_t upd;
      switch (g.kind) {
        case YQ_AGG_COUNT_STAR: upd = UPD_COUNT_STAR; break;
        case YQ_AGG_COUNT: upd = UPD_COUNT; break;
        case YQ_AGG_SUM:
        case YQ_AGG_AVG: upd = flt ? UPD_SUM_F : UPD_SUM_I; break;
        case YQ_AGG_MIN: upd = flt ? UPD_MIN_F : UPD_MIN_I; break;
        default: upd = flt ? UPD_MAX_F : UPD_MAX_I; break;
      }
      F.A.upd[a] = upd;
      if (g.kind == YQ_AGG_COUNT_STAR) continue;
      int t = -1;
      YQ_TRY(B.append(&g.input, t));
      if (g.kind != YQ_AGG_COUNT && t != g.input_type) return YQ_ERR_INVALID_ARG;
      YQ_TRY(B.emit(OP_EMIT_AGG, (uint8_t)a, upd, (uint8_t)t));
    }
    YQ_TRY(B.finalize());
    F.fkey_col = fact_key;
    if (!plan_stages(B.P, B.used_cols | (1u << fact_key), F.SP)) F.SP.nstages = 0;
    memcpy(&F.P, &B.P, sizeof(VmProgram));
    F.pred_end = B.remap[pred_end];
    F.pc_end = B.len;
    F.A.nagg = nagg;
  }
  return YQ_OK;
}

// Probe launch over a built dimension table (nbuckets buckets, `kept` rows).
static int join_agg_launch(JAParams& F, const yq_batch* fact, int32_t fact_key, uint32_t nbuckets, uint32_t kept,
                           uint32_t* d_bstart, unsigned long long* d_hkeys, const uint32_t* d_counts, Acc* partials,
                           uint32_t* d_misc, void* state, cudaStream_t s) {
  const yq_column& fk = fact->columns[fact_key];
  const int grid_cap = sm_count() * 8;
  const uint32_t counts[1] = {kept};
  F.fkey = jcol(fk);
  F.nbuckets = nbuckets;
  F.hrows_n = counts[0];
  F.bstart = d_bstart;
  F.hkeys = d_hkeys;
  F.krange = reinterpret_cast<const long long*>(d_counts + 2);
  const size_t table = table_smem(nbuckets, counts[0], false);
  // The ring leaves room for the table; with too few stages left the kernel
  // reads the fact columns from global memory.
  const size_t budget = kStageBudget + 8 * 1024;
  if (F.SP.nstages && stage_smem_bytes(F.SP) + table > budget) {
    const int fit = (int)((budget > table ? budget - table : 0) / (F.SP.stage_bytes + 8));
    F.SP.nstages = fit >= 2 ? (fit > kStageMax ? kStageMax : fit) : 0;
  }
  const bool staged = F.SP.nstages > 0;
  F.table_off = (uint32_t)align_up(stage_smem_bytes(F.SP), 16);
  F.table_words = (uint32_t)(table / 4);
  const size_t smem = F.table_off + table;
  const void* kern = staged ? (const void*)k_join_aggregate<true> : (const void*)k_join_aggregate<false>;
  YQ_TRY(kernel_allow_smem(kern, smem));
  int per_sm = kernel_blocks_per_sm(kern, kRowBlock, smem);
  if (per_sm > 8) per_sm = 8;
  const uint32_t tiles = ceil_div<uint32_t>(fact->rows, kStepRows);
  int grid = sm_count() * per_sm;
  if ((uint32_t)grid > tiles) grid = (int)tiles;
  const double row_bytes = row_bytes_of(F.P, program_columns(F.P, F.pc_end, 1u << fact_key));
  const void* jk = jit_kernel(JIT_JOIN_AGG, staged, F.P, F.pred_end, F.pc_end);
  ProfScope ps("join_aggregate", s, (double)fact->rows * row_bytes);
  if (jk) {
    size_t jsmem = smem;
    if (staged) {  // ring depth for the specialised kernel's occupancy, table after it
      F.SP.nstages = jit_stages(jk, F.SP.stage_bytes, F.SP.nstages, table);
      F.table_off = (uint32_t)align_up(stage_smem_bytes(F.SP), 16);
      jsmem = F.table_off + table;
    }
    uint32_t n = fact->rows;
    Acc* st = static_cast<Acc*>(state);
    void* args[] = {&F, &n, &partials, &d_misc, &st};
    return jit_launch(jk, grid_cap, tiles, jsmem, args, s);
  }
  if (staged)
    k_join_aggregate<true><<<grid, kRowBlock, smem, s>>>(F, fact->rows, partials, d_misc, static_cast<Acc*>(state));
  else
    k_join_aggregate<false><<<grid, kRowBlock, smem, s>>>(F, fact->rows, partials, d_misc, static_cast<Acc*>(state));
  YQ_CHECK_LAUNCH();
  return YQ_OK;
}


extern "C" {

int yq_join_aggregate(const yq_batch* fact, const yq_program* fact_predicate, int32_t fact_key, const yq_batch* dim,
                      const yq_program* dim_predicate, int32_t dim_key, const yq_constants* constants,
                      const yq_agg_spec* aggs, int32_t nagg, void* state, void* workspace, size_t workspace_bytes,
                      void* stream) {
  if (!fact || !dim || !state || fact_key < 0 || fact_key >= fact->ncols || dim_key < 0 || dim_key >= dim->ncols ||
      nagg < 0 || nagg > YQ_MAX_AGGREGATES || (nagg > 0 && !aggs))
    return YQ_ERR_INVALID_ARG;
  const yq_column& fk = fact->columns[fact_key];
  const yq_column& dk = dim->columns[dim_key];
  if (!join_col_ok(fk) || !join_col_ok(dk) || fk.type != dk.type || !hashable(fk.type)) return YQ_ERR_INVALID_ARG;
  if (dim->rows > kHashMaxRows) return YQ_ERR_UNSUPPORTED;
  cudaStream_t s = as_stream(stream);
  JAParams F;
  YQ_TRY(join_agg_params(fact, fact_predicate, fact_key, constants, aggs, nagg, F));
  if (fact->rows == 0 || nagg == 0) return YQ_OK;
  const uint32_t nbuckets = pow2_at_least(dim->rows ? dim->rows : 1);
  Workspace ws;
  YQ_TRY(ws.acquire(workspace, workspace_bytes, yq_join_aggregate_workspace_size(fact->rows, dim->rows, nagg), s));
  uint32_t* d_bstart = ws.take<uint32_t>(nbuckets + 1);
  unsigned long long* d_hkeys = ws.take<unsigned long long>(dim->rows ? dim->rows : 1);
  uint32_t* d_hrows = ws.take<uint32_t>(dim->rows ? dim->rows : 1);
  uint32_t* d_misc = ws.take<uint32_t>(8);  // [0] ticket [2] kept rows [3] duplicate keys
  const int grid_cap = sm_count() * 8;
  Acc* partials = ws.take<Acc>((size_t)grid_cap * YQ_MAX_AGGREGATES);
  YQ_TRY_CUDA(cudaMemsetAsync(d_misc, 0, 8 * sizeof(uint32_t), s));
  YQ_TRY(build_table(dim, dim_predicate, constants, dim_key, nbuckets, d_bstart, d_hkeys, d_hrows, d_misc + 2, s));
  uint32_t counts[2] = {0, 0};
  YQ_TRY(d2h_sync(counts, d_misc + 2, sizeof(counts), s));
  if (counts[1] != 0) return YQ_ERR_UNSUPPORTED;  // dimension keys repeat: use yq_join_pairs + an aggregate
  return join_agg_launch(F, fact, fact_key, nbuckets, counts[0], d_bstart, d_hkeys, d_misc + 2, partials, d_misc, state,
                         s);
}

// ------------------------------------------------ prepared dimension table
// Table layout: [8 counters][bucket starts nb+1][keys dim_rows][rows dim_rows].
static size_t dim_table_layout(uint32_t dim_rows, WsSize& w) {
  const uint32_t nb = pow2_at_least(dim_rows ? dim_rows : 1);
  w.add<uint32_t>(8);
  w.add<uint32_t>(nb + 1);
  w.add<unsigned long long>(dim_rows ? dim_rows : 1);
  w.add<uint32_t>(dim_rows ? dim_rows : 1);
  return w.total();
}

size_t yq_join_dim_table_size(uint32_t dim_rows) {
  WsSize w;
  return dim_table_layout(dim_rows, w);
}

int yq_join_dim_table_build(const yq_batch* dim, const yq_program* dim_predicate, int32_t dim_key,
                            const yq_constants* constants, void* table, size_t table_bytes, uint32_t* kept,
                            void* stream) {
  if (!dim || !table || !kept || dim_key < 0 || dim_key >= dim->ncols) return YQ_ERR_INVALID_ARG;
  const yq_column& dk = dim->columns[dim_key];
  if (!join_col_ok(dk) || !hashable(dk.type)) return YQ_ERR_INVALID_ARG;
  if (dim->rows > kHashMaxRows) return YQ_ERR_UNSUPPORTED;
  if (table_bytes < yq_join_dim_table_size(dim->rows)) return YQ_ERR_CAPACITY;
  cudaStream_t s = as_stream(stream);
  const uint32_t nbuckets = pow2_at_least(dim->rows ? dim->rows : 1);
  Workspace ws;
  YQ_TRY(ws.acquire(table, table_bytes, yq_join_dim_table_size(dim->rows), s));
  uint32_t* d_misc = ws.take<uint32_t>(8);
  uint32_t* d_bstart = ws.take<uint32_t>(nbuckets + 1);
  unsigned long long* d_hkeys = ws.take<unsigned long long>(dim->rows ? dim->rows : 1);
  uint32_t* d_hrows = ws.take<uint32_t>(dim->rows ? dim->rows : 1);
  YQ_TRY_CUDA(cudaMemsetAsync(d_misc, 0, 8 * sizeof(uint32_t), s));
  YQ_TRY(build_table(dim, dim_predicate, constants, dim_key, nbuckets, d_bstart, d_hkeys, d_hrows, d_misc + 2, s));
  uint32_t counts[2] = {0, 0};
  YQ_TRY(d2h_sync(counts, d_misc + 2, sizeof(counts), s));
  if (counts[1] != 0) return YQ_ERR_UNSUPPORTED;
  *kept = counts[0];
  return YQ_OK;
}

size_t yq_join_aggregate_prepared_workspace_size(int32_t nagg) {
  (void)nagg;
  WsSize w;
  w.add<uint32_t>(8);
  w.add<Acc>((size_t)sm_count() * 8 * YQ_MAX_AGGREGATES);
  return w.total();
}

int yq_join_aggregate_prepared(const yq_batch* fact, const yq_program* fact_predicate, int32_t fact_key,
                               const void* table, uint32_t dim_rows, uint32_t kept, int32_t key_type,
                               const yq_constants* constants, const yq_agg_spec* aggs, int32_t nagg, void* state,
                               void* workspace, size_t workspace_bytes, void* stream) {
  if (!fact || !table || !state || fact_key < 0 || fact_key >= fact->ncols || nagg < 0 ||
      nagg > YQ_MAX_AGGREGATES || (nagg > 0 && !aggs) || kept > dim_rows || dim_rows > kHashMaxRows)
    return YQ_ERR_INVALID_ARG;
  const yq_column& fk = fact->columns[fact_key];
  if (!join_col_ok(fk) || fk.type != key_type || !hashable(fk.type)) return YQ_ERR_INVALID_ARG;
  cudaStream_t s = as_stream(stream);
  JAParams F;
  YQ_TRY(join_agg_params(fact, fact_predicate, fact_key, constants, aggs, nagg, F));
  if (fact->rows == 0 || nagg == 0) return YQ_OK;
  const uint32_t nbuckets = pow2_at_least(dim_rows ? dim_rows : 1);
  const size_t tbytes = yq_join_dim_table_size(dim_rows);
  Workspace tw;  // the caller's table, carved as yq_join_dim_table_build laid it out
  YQ_TRY(tw.acquire(const_cast<void*>(table), tbytes, tbytes, s));
  uint32_t* d_counts = tw.take<uint32_t>(8) + 2;
  uint32_t* d_bstart = tw.take<uint32_t>(nbuckets + 1);
  unsigned long long* d_hkeys = tw.take<unsigned long long>(dim_rows ? dim_rows : 1);
  Workspace ws;
  YQ_TRY(ws.acquire(workspace, workspace_bytes, yq_join_aggregate_prepared_workspace_size(nagg), s));
  uint32_t* d_misc = ws.take<uint32_t>(8);
  Acc* partials = ws.take<Acc>((size_t)sm_count() * 8 * YQ_MAX_AGGREGATES);
  YQ_TRY_CUDA(cudaMemsetAsync(d_misc, 0, 8 * sizeof(uint32_t), s));
  return join_agg_launch(F, fact, fact_key, nbuckets, kept, d_bstart, d_hkeys, d_counts, partials, d_misc, state, s);
}

}  // extern "C"
