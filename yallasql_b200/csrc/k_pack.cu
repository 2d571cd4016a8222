// Gather of many narrow columns through packed rows (sm_100a).
//
// A column-by-column gather reads a 4- to 16-byte cell from a random row for
// every column, and each read costs a 32-byte L2 sector and, on a table beyond
// L2, a 64-byte DRAM burst of its own. Here the columns are first packed side
// by side into one record per row (a streaming pass), the records are gathered
// (one random read of adjacent sectors per row, whatever the column count) and
// unpacked through shared memory, so the outputs leave in coalesced stores.
// Replaces the per-column moves of move_rows_kernel on the reference's ORDER BY
// path (src/kernels/move_rows_kernel.cu:8-30, include/kernels/move_rows_kernel.hpp:51-83).
//
// Both kernels are bound by the bytes in flight: a thread issues eight 16-byte
// record reads (gather) or four cells of a column (pack) before it stores any.
// Records lie an odd number of 16-byte units apart in shared memory, which keeps
// 16-byte accesses free of bank conflicts, 8-byte ones two-way and 4-byte ones
// four-way (at an even number, four pieces, 4-byte cells were 16-way).
#include <string.h>
#include "yq_sort.cuh"

namespace yq {

constexpr int kPackBlock = 256;
constexpr int kPackRows = 4;                                // rows a thread packs
constexpr uint32_t kPackTile = kPackBlock * kPackRows;
constexpr int kMaxPieces = 8;                               // records of up to 128 bytes
constexpr int kMaxCellWidth = 32;                           // wider cells fill their sectors alone

template <int P>
constexpr int kRecStride = (P | 1) * 16;

struct PackField {
  const char* src;
  char* dst;
  int32_t off;    // within the record
  int32_t width;  // 1, 4, 8, 16, or a multiple of 4 up to kMaxCellWidth
};
struct PackParams {
  PackField f[2 * YQ_MAX_BATCH_COLUMNS];
  int32_t nf;
  uint32_t rows;
  char* rec;
};

template <typename V>
__device__ __forceinline__ void pack_cells(const PackField& f, uint32_t r0, uint32_t n, char* s, int stride) {
  V v[kPackRows];
#pragma unroll
  for (int k = 0; k < kPackRows; ++k) {
    const uint32_t i = threadIdx.x + k * kPackBlock;
    if (i < n) v[k] = f.src ? __ldg(reinterpret_cast<const V*>(f.src) + r0 + i) : V{};
  }
#pragma unroll
  for (int k = 0; k < kPackRows; ++k) {
    const uint32_t i = threadIdx.x + k * kPackBlock;
    if (i < n) *reinterpret_cast<V*>(s + i * stride + f.off) = v[k];
  }
}

template <int P>
__global__ void __launch_bounds__(kPackBlock) k_pack_rows(const __grid_constant__ PackParams G) {
  extern __shared__ __align__(16) char s_rec[];
  constexpr int stride = kRecStride<P>;
  for (uint32_t tile = blockIdx.x; tile * (unsigned long long)kPackTile < G.rows; tile += gridDim.x) {
    const uint32_t r0 = tile * kPackTile;
    const uint32_t n = min(kPackTile, G.rows - r0);
    for (int c = 0; c < G.nf; ++c) {
      const PackField& f = G.f[c];
      switch (f.width) {
        case 1: pack_cells<uint8_t>(f, r0, n, s_rec, stride); break;
        case 4: pack_cells<uint32_t>(f, r0, n, s_rec, stride); break;
        case 8: pack_cells<uint2>(f, r0, n, s_rec, stride); break;
        case 16: pack_cells<uint4>(f, r0, n, s_rec, stride); break;
        default:
          for (uint32_t i = threadIdx.x; i < n; i += kPackBlock)
            for (int b = 0; b < f.width; b += 4)
              *reinterpret_cast<uint32_t*>(s_rec + i * stride + f.off + b) =
                  __ldg(reinterpret_cast<const uint32_t*>(f.src + (size_t)(r0 + i) * f.width + b));
      }
    }
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(G.rec) + (size_t)r0 * P;
    for (uint32_t q = threadIdx.x; q < n * P; q += kPackBlock)
      out[q] = *reinterpret_cast<const uint4*>(s_rec + (q / P) * stride + (q % P) * 16);
    __syncthreads();
  }
}

// Each thread reads whole records: kGatherRows of them in flight, 16 bytes a
// load. A record then passes through a shared-memory slot of the thread's own,
// from which its cells are read at their (run-time) offsets and stored, 32
// consecutive rows of a column a store. No thread waits for another.
template <int P>
constexpr int kGatherRows = P <= 2 ? 4 : (P <= 4 ? 2 : 1);

// Two adjacent 16-byte pieces of a record in one 32-byte load (32-byte
// aligned): one L1 lookup a row instead of two.
__device__ __forceinline__ void ldg_nc_v8(const uint4* p, uint4& a, uint4& b) {
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w)
      : "l"(p));
}

template <typename V>
__device__ __forceinline__ void store_cell(const PackField& f, uint32_t i, const char* slot) {
  reinterpret_cast<V*>(f.dst)[i] = *reinterpret_cast<const V*>(slot + f.off);
}

template <int P>
__global__ void __launch_bounds__(kPackBlock) k_gather_rows(const __grid_constant__ PackParams G,
                                                            const uint32_t* __restrict__ perm) {
  constexpr int ROWS = kGatherRows<P>;
  constexpr uint32_t TILE = kPackBlock * ROWS;
  __shared__ __align__(16) char s_slot[kPackBlock][kRecStride<P>];
  char* const slot = s_slot[threadIdx.x];
  for (unsigned long long i0 = (unsigned long long)blockIdx.x * TILE; i0 < G.rows;
       i0 += (unsigned long long)gridDim.x * TILE) {
    uint32_t r[ROWS];
    uint4 v[ROWS][P];
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const unsigned long long i = i0 + k * kPackBlock + threadIdx.x;
      r[k] = i < G.rows ? __ldg(perm + i) : 0xffffffffu;
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      const uint4* rec = reinterpret_cast<const uint4*>(G.rec) + (size_t)min(r[k], G.rows - 1u) * P;
      if (P % 2 == 0) {
#pragma unroll
        for (int p = 0; p < P; p += 2) ldg_nc_v8(rec + p, v[k][p], v[k][p + 1 < P ? p + 1 : p]);
      } else {
#pragma unroll
        for (int p = 0; p < P; ++p) v[k][p] = __ldg(rec + p);
      }
    }
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
      if (r[k] >= G.rows) continue;  // past the end, or perm is no permutation: nothing is written
      const uint32_t i = (uint32_t)(i0 + k * kPackBlock + threadIdx.x);
#pragma unroll
      for (int p = 0; p < P; ++p) reinterpret_cast<uint4*>(slot)[p] = v[k][p];
      for (int c = 0; c < G.nf; ++c) {
        const PackField& f = G.f[c];
        switch (f.width) {
          case 1: store_cell<uint8_t>(f, i, slot); break;
          case 4: store_cell<uint32_t>(f, i, slot); break;
          case 8: store_cell<uint2>(f, i, slot); break;
          case 16: store_cell<uint4>(f, i, slot); break;
          default:
            for (int b = 0; b < f.width; b += 4)
              *reinterpret_cast<uint32_t*>(f.dst + (size_t)i * f.width + b) =
                  *reinterpret_cast<const uint32_t*>(slot + f.off + b);
        }
      }
    }
  }
}

template <int P>
static int launch_packed(const PackParams& G, const uint32_t* perm, double cell_bytes, cudaStream_t s) {
  constexpr size_t pack_smem = (size_t)kPackTile * kRecStride<P>;
  constexpr uint32_t tile = kPackBlock * kGatherRows<P>;
  static_assert(pack_smem <= 227 * 1024, "a pack tile must fit shared memory");
  const void* pk = (const void*)k_pack_rows<P>;
  const void* gk = (const void*)k_gather_rows<P>;
  YQ_TRY(kernel_allow_smem(pk, pack_smem));
  uint32_t grid = (uint32_t)(kernel_blocks_per_sm(pk, kPackBlock, pack_smem) * sm_count());
  uint32_t tiles = ceil_div<uint32_t>(G.rows, kPackTile);
  {
    ProfScope ps("pack_rows", s, (double)G.rows * (cell_bytes + 16.0 * P));
    k_pack_rows<P><<<tiles < grid ? tiles : grid, kPackBlock, pack_smem, s>>>(G);
    YQ_CHECK_LAUNCH();
  }
  grid = (uint32_t)(kernel_blocks_per_sm(gk, kPackBlock, 0) * sm_count());
  tiles = ceil_div<uint32_t>(G.rows, tile);
  ProfScope ps("gather_rows", s, (double)G.rows * (4.0 + 16.0 * P + cell_bytes));
  k_gather_rows<P><<<tiles < grid ? tiles : grid, kPackBlock, 0, s>>>(G, perm);
  YQ_CHECK_LAUNCH();
  return YQ_OK;
}

static bool packable(const yq_column& a, const yq_column& b) {
  const int w = a.width;
  if (w > kMaxCellWidth || (w != 1 && w % 4 != 0)) return false;
  const uintptr_t align = w == 1 ? 1 : (w == 8 || w == 16 ? (uintptr_t)w : 4);
  return ((reinterpret_cast<uintptr_t>(a.data) | reinterpret_cast<uintptr_t>(b.data)) & (align - 1)) == 0;
}

// Fields of the packed columns, widest alignment first (16-byte cells at
// 16-byte offsets and so on down), the null bytes last.
static uint32_t plan_fields(const yq_column* in, int32_t ncols, const yq_column* out, const uint32_t* const* only_if,
                            PackParams& G, int& pieces, double& cell_bytes) {
  uint32_t packed = 0;
  int off = 0, cells = 0;
  G.nf = 0;
  cell_bytes = 0;
  for (const int align : {16, 8, 4, 1}) {
    for (int c = 0; c < ncols; ++c) {
      const int w = in[c].width;
      const int a = w == 16 ? 16 : (w == 8 ? 8 : (w == 1 ? 1 : 4));
      if ((only_if && only_if[c]) || !packable(in[c], out[c])) continue;
      if (a == align) {
        if (off + w + ncols > kMaxPieces * 16) continue;  // leaves room for null bytes: this column moves by itself
        G.f[G.nf++] = PackField{static_cast<const char*>(in[c].data), static_cast<char*>(out[c].data), off, w};
        packed |= 1u << c;
        off += w;
        cell_bytes += w;
        ++cells;
      }
    }
  }
  for (int c = 0; c < ncols; ++c)
    if ((packed >> c & 1u) && out[c].nulls) {
      G.f[G.nf++] = PackField{reinterpret_cast<const char*>(in[c].nulls),
                              reinterpret_cast<char*>(const_cast<uint8_t*>(out[c].nulls)), off, 1};
      off += 1;
      cell_bytes += 1;
      ++cells;
    }
  pieces = (off + 15) / 16;
  return cells >= 2 ? packed : 0u;
}

// From this many packed bytes on the cells no longer stay in L2 between the
// reads of neighbouring columns, and a random cell costs a DRAM burst.
constexpr double kPackedGatherBytes = 64.0 * 1024 * 1024;

size_t packed_gather_bytes(const yq_column* in, int32_t ncols, const yq_column* out, const uint32_t* const* only_if,
                           uint32_t rows) {
  static_assert(YQ_MAX_BATCH_COLUMNS <= 32, "a column mask is one word");
  PackParams G;
  int pieces = 0;
  double cell_bytes = 0;
  if (!plan_fields(in, ncols, out, only_if, G, pieces, cell_bytes)) return 0;
  if (cell_bytes * rows < kPackedGatherBytes) return 0;
  return (size_t)rows * pieces * 16;
}

int packed_gather(const yq_column* in, int32_t ncols, const yq_column* out, const uint32_t* const* only_if,
                  const uint32_t* perm, uint32_t rows, void* records, cudaStream_t s, uint32_t* moved) {
  PackParams G;
  int pieces = 0;
  double cell_bytes = 0;
  *moved = plan_fields(in, ncols, out, only_if, G, pieces, cell_bytes);
  G.rows = rows;
  G.rec = static_cast<char*>(records);
  switch (pieces) {
    case 1: return launch_packed<1>(G, perm, cell_bytes, s);
    case 2: return launch_packed<2>(G, perm, cell_bytes, s);
    case 3: return launch_packed<3>(G, perm, cell_bytes, s);
    case 4: return launch_packed<4>(G, perm, cell_bytes, s);
    case 5: return launch_packed<5>(G, perm, cell_bytes, s);
    case 6: return launch_packed<6>(G, perm, cell_bytes, s);
    case 7: return launch_packed<7>(G, perm, cell_bytes, s);
    case 8: return launch_packed<8>(G, perm, cell_bytes, s);
    default: return YQ_ERR_UNSUPPORTED;
  }
}

}  // namespace yq
