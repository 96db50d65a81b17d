// Batched exit-depth propagation inside one LAST_EXITED pool.
//
// When a token leaves the recurrence at plane e, every deeper plane must hold a copy of
// plane e's K/V row so that later tokens attending at those depths read the last computed
// state. The reference does this per token with basic-index copies
// (KVCacheManager.finalize_token, vllm_rlt/core/kv_cache_manager.py:1053-1076) or with a
// Triton kernel over (row, target plane, channel tile) plus a second launch for the scales
// (finalize_kernel, vllm_rlt/kernels/routing.py:147-179; ModelRunner.finalize_many,
// vllm_rlt/worker/model_runner.py:1349-1395). Here one launch covers K, V and both scale
// tensors: each row of every selected layer is loaded once and stored to every deeper plane.
//
// Work decomposition. kGroupRows consecutive rows of the batch form a group; they are usually consecutive tokens of one
// request, so that the copies of one layer on one plane are neighbours in one block. A thread takes one vector of the group's
// (selected layer, row, vector of the row) for one of its tensors, looks its row and its blocks up itself (the threads of a warp
// mostly the same ones, so the lookups hit L1) and stores the vector to every deeper plane. The grid holds one CTA per 8 KiB
// in that order: HBM is fastest while the SMs work close together (block_moves.cu has the measurements), and a decode step of
// a few rows still reaches every SM. Nothing is shared inside a CTA: lists of rows and blocks in shared memory, with two
// barriers before the first load, cost 8.5 us where this takes 6.2 (64 rows of four planes), 277 where it takes 274 (4,000 rows).
// Measured before that, with persistent CTAs that scanned all rows' costs first: 13.8 and 322 us.
//
// HBM roofline: each selected (layer, tensor) row is read once and written once per deeper plane.

#include <algorithm>

#include "common.cuh"

namespace rlt {
namespace {

struct FinalizeRegion {
  char* key;
  char* value;
  long long block_bytes, layer_bytes, token_bytes;
  int vec_bytes;
  int row_vecs;        // token_bytes / vec_bytes
  unsigned row_magic;  // div_magic(row_vecs), 0 for one-vector rows
  int parts;           // CTAs per (group, tensor)
};

struct FinalizeParams {
  FinalizeRegion region[2];
  int parts;  // CTAs per group
  int planes, block_size, num_blocks, num_layers;
  unsigned long long layer_mask;  // bit l set: layer l is copied (the recurrent layers)
  int layers;                     // bits set in layer_mask
  int plane_chunk;                // planes one CTA stores to
  int dense_layers;               // the selected layers are 0 .. layers - 1
  const int* tables;              // [requests, planes, table_width]
  int table_width, num_requests;
  const int* rows;                // [n][3]: request index, exit plane, token position
  int n;
  int first_row;                  // of this launch in the caller's list
  int* status;
};

constexpr int kGroupRows = 16;
// Deeper planes whose blocks are looked up together with the source's, before the source is read: rows -> blocks -> payload are three dependent
// accesses then, not four and one more per plane. us at none / 2, launches one behind another in a graph: one row 1.88 / 1.81, 64 rows of four planes
// 6.35 / 6.28, 8, 64 and 1,200 rows of 32 planes with geometric exits 6.78 / 6.54, 24.8 / 24.5 and 403 / 395, 300 rows of eight planes of 1 KiB 12.8 /
// 12.6, 4,000 rows of four planes 273.0 / 273.1. (3 no longer fits the registers of eight CTAs per SM: 4,000 rows 2 % slower.)
constexpr int kAhead = 2;
constexpr long long kMostRows = 1ll << 28;  // of one launch: three times a row's index stays in 32 bits

// Vectors per thread: one of 32 or 16 bytes, more of the narrow ones.
template <typename T>
__host__ __device__ constexpr int vectors_of() {
  return sizeof(T) >= 16 ? 1 : sizeof(T) == 4 ? 4 : 8;
}

// Position of the k-th (0-based) set bit.
__device__ __forceinline__ int nth_set_bit(unsigned long long mask, int k) {
  const unsigned lo = static_cast<unsigned>(mask), hi = static_cast<unsigned>(mask >> 32);
  const int in_lo = __popc(lo);
  return k < in_lo ? static_cast<int>(__fns(lo, 0, k + 1)) : 32 + static_cast<int>(__fns(hi, 0, k - in_lo + 1));
}

// Vector `k` of the part that begins at vector `first` of the group, to every deeper plane. `say`: this CTA reports invalid rows.
template <typename T, bool kChunked>
__device__ __forceinline__ void fill_deeper(const FinalizeParams& p, const FinalizeRegion& rg, int group, int kv, int first, int k, bool say) {
  if (first + k >= p.layers * kGroupRows * rg.row_vecs) return;
  const int row0 = first / rg.row_vecs;
  const unsigned j = static_cast<unsigned>(first - row0 * rg.row_vecs + k);
  const int q = rg.row_magic ? static_cast<int>(__umulhi(j, rg.row_magic)) : static_cast<int>(j);
  const int slot = (row0 + q) / kGroupRows;
  const int row = group * kGroupRows + (row0 + q) % kGroupRows;
  if (row >= p.n) return;
  const int request = p.rows[3 * row], e = p.rows[3 * row + 1], position = p.rows[3 * row + 2];
  if (request < 0 || request >= p.num_requests || e < 0 || e >= p.planes || position < 0 || position >= p.table_width * p.block_size) {
    if (say && slot == 0) report(p.status, RLT_STATUS_BAD_PLANE, p.first_row + row, position, e);
    return;
  }
  // the deeper planes of this CTA's chunk (all of them, unless the launch is small)
  const int from = kChunked ? max(e + 1, static_cast<int>(blockIdx.y) * p.plane_chunk) : e + 1;
  const int to = kChunked ? min(p.planes, (static_cast<int>(blockIdx.y) + 1) * p.plane_chunk) : p.planes;
  if (from >= to) return;
  const int page = position / p.block_size;
  const int* table = p.tables + static_cast<long long>(request) * p.planes * p.table_width + page;
  const int source = table[static_cast<long long>(e) * p.table_width];
  int block[kAhead];
#pragma unroll
  for (int i = 0; i < kAhead; ++i) block[i] = from + i < to ? table[static_cast<long long>(from + i) * p.table_width] : 0;
  const int layer = p.dense_layers ? slot : nth_set_bit(p.layer_mask, slot);
  char* at = (kv ? rg.value : rg.key) + layer * rg.layer_bytes + (position - page * p.block_size) * rg.token_bytes +
             (static_cast<int>(j) - q * rg.row_vecs) * static_cast<int>(sizeof(T));
  const auto outside = [&](int id) { return static_cast<unsigned>(id) >= static_cast<unsigned>(p.num_blocks); };
  int wrong = outside(source) ? source : 0;  // the first id that is no block's
  if (wrong == 0) {
    const T v = ld_stream(reinterpret_cast<const T*>(at + source * rg.block_bytes));
    const auto store = [&](int id) {
      if (outside(id)) {
        if (wrong == 0) wrong = id;
      } else {
        st_stream(reinterpret_cast<T*>(at + id * rg.block_bytes), v);
      }
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
      if (from + i < to) store(block[i]);
    }
    for (int t = from + kAhead; t < to; ++t) store(table[static_cast<long long>(t) * p.table_width]);
  }
  // (the row is read again for what the report says: registers are short)
  if (wrong != 0) report(p.status, RLT_STATUS_BAD_BLOCK, p.rows[3 * row], p.rows[3 * row + 2] / p.block_size, wrong);
}

template <typename T, bool kChunked>
__device__ __forceinline__ void copy_part(const FinalizeParams& p, const FinalizeRegion& rg, int group, int kv, int part, bool say) {
  constexpr int kPer = kThreads * vectors_of<T>();
  if constexpr (vectors_of<T>() == 1) {
    fill_deeper<T, kChunked>(p, rg, group, kv, part * kPer, static_cast<int>(threadIdx.x), say);
  } else {
#pragma unroll 1
    for (int k = static_cast<int>(threadIdx.x); k < kPer; k += kThreads) fill_deeper<T, kChunked>(p, rg, group, kv, part * kPer, k, say);
  }
}

// kWide: every row is a multiple of 32 bytes. The loops of the narrow types would cost this kernel a fifth of its CTAs.
template <bool kWide, bool kChunked>
__global__ void __launch_bounds__(kThreads, kWide ? 8 : 6) finalize_kernel(const __grid_constant__ FinalizeParams p) {
  const int group = static_cast<int>(blockIdx.x / p.parts);
  int at = static_cast<int>(blockIdx.x) - group * p.parts;
  const int g = at >= 2 * p.region[0].parts;
  const FinalizeRegion& rg = p.region[g];
  if (g) at -= 2 * p.region[0].parts;
  const int kv = at >= rg.parts;
  const int part = at - kv * rg.parts;
  const bool say = g == 0 && kv == 0 && blockIdx.y == 0;
  follow_stream();
  if (kWide || rg.vec_bytes == 32) {
    copy_part<Vec32, kChunked>(p, rg, group, kv, part, say);
  } else if (rg.vec_bytes == 16) {
    copy_part<uint4, kChunked>(p, rg, group, kv, part, say);
  } else if (rg.vec_bytes == 4) {
    copy_part<uint32_t, kChunked>(p, rg, group, kv, part, say);
  } else {
    copy_part<uint8_t, kChunked>(p, rg, group, kv, part, say);
  }
}

}  // namespace
}  // namespace rlt

extern "C" {

int rlt_kv_finalize(const RltPool* pool, const int32_t* tables, int32_t num_requests, int32_t table_width,
                    const int32_t* rows, int32_t count, uint64_t layer_mask, int32_t* status, rlt_stream_t stream) {
  const rlt::NvtxRange range("rlt.kv_finalize");
  if (count == 0) return RLT_OK;
  if (pool == nullptr || tables == nullptr || rows == nullptr || count < 0 || num_requests < 1 || table_width < 1)
    return RLT_E_INVALID;
  if (pool->codes.key == nullptr || pool->codes.value == nullptr) return RLT_E_INVALID;
  if (pool->num_layers < 1 || pool->num_layers > 64 || pool->block_size < 1 || pool->num_planes < 1 ||
      pool->num_blocks < 1)
    return RLT_E_LIMIT;
  if (pool->num_planes == 1) return RLT_OK;  // a SHARED pool has nothing deeper to fill
  rlt::FinalizeParams p{};
  const int regions = pool->scales.key != nullptr ? 2 : 1;
  if (regions == 2 && pool->scales.value == nullptr) return RLT_E_INVALID;
  const uint64_t all = pool->num_layers == 64 ? ~0ull : ((1ull << pool->num_layers) - 1ull);
  p.layer_mask = layer_mask == 0 ? all : (layer_mask & all);
  p.layers = __builtin_popcountll(p.layer_mask);
  if (p.layers == 0) return RLT_OK;
  p.dense_layers = (p.layer_mask & (p.layer_mask + 1)) == 0;
  for (int g = 0; g < regions; ++g) {
    const RltRegion& r = g == 0 ? pool->codes : pool->scales;
    if (r.token_bytes <= 0 || r.layer_bytes != r.token_bytes * pool->block_size ||
        r.block_bytes != r.layer_bytes * pool->num_layers)
      return RLT_E_GEOMETRY;
    rlt::FinalizeRegion& out = p.region[g];
    out.key = static_cast<char*>(r.key);
    out.value = static_cast<char*>(r.value);
    out.block_bytes = r.block_bytes;
    out.layer_bytes = r.layer_bytes;
    out.token_bytes = r.token_bytes;
    const uintptr_t bits = reinterpret_cast<uintptr_t>(r.key) | reinterpret_cast<uintptr_t>(r.value) |
                           static_cast<uintptr_t>(r.token_bytes);
    out.vec_bytes = (bits & 31u) == 0 ? 32 : (bits & 15u) == 0 ? 16 : (bits & 3u) == 0 ? 4 : 1;
    const long long row_vecs = r.token_bytes / out.vec_bytes;
    // (row_vecs + vectors of a part) * row_vecs must stay below 2^32 for the multiplier split, and so must a group's
    // vectors for 32-bit counts
    if ((row_vecs + 65536) * row_vecs >= (1ll << 32) || row_vecs * rlt::kGroupRows * p.layers >= (1ll << 31)) return RLT_E_LIMIT;
    out.row_vecs = static_cast<int>(row_vecs);
    out.row_magic = row_vecs == 1 ? 0u : rlt::div_magic(static_cast<uint32_t>(row_vecs));
  }
  p.planes = pool->num_planes;
  p.block_size = pool->block_size;
  p.num_blocks = pool->num_blocks;
  p.num_layers = pool->num_layers;
  p.tables = tables;
  p.table_width = table_width;
  p.num_requests = num_requests;
  p.status = status;
  for (int g = 0; g < regions; ++g) {
    rlt::FinalizeRegion& rg = p.region[g];
    const int per = rlt::kThreads * (rg.vec_bytes == 32 ? rlt::vectors_of<rlt::Vec32>() : rg.vec_bytes == 16 ? rlt::vectors_of<uint4>()
                                     : rg.vec_bytes == 4 ? rlt::vectors_of<uint32_t>() : rlt::vectors_of<uint8_t>());
    const long long vectors = static_cast<long long>(p.layers) * rlt::kGroupRows * rg.row_vecs;
    rg.parts = static_cast<int>((vectors + per - 1) / per);
    p.parts += 2 * rg.parts;
  }
  int sms = 0;
  const int rc = rlt::sm_count(&sms);
  if (rc != RLT_OK) return rc;
  const bool wide = p.region[0].vec_bytes == 32 && (regions == 1 || p.region[1].vec_bytes == 32);
  // One launch, unless the rows need more CTAs than a grid holds (89 million rows of 24 layers with 4 KiB each).
  const long long most = std::min(0x7fffffffll / p.parts * rlt::kGroupRows, rlt::kMostRows);
  for (long long first = 0; first < count; first += most) {
    p.rows = rows + 3 * first;
    p.first_row = static_cast<int>(first);
    p.n = static_cast<int>(std::min<long long>(most, count - first));
    const long long grid = static_cast<long long>((p.n + rlt::kGroupRows - 1) / rlt::kGroupRows) * p.parts;
    // A launch too small to fill the GPU is short of stores in flight where each thread has many planes to fill: the planes
    // are then dealt to several CTAs, each of which reads the source rows (from L2, after the first) for itself. 8 rows of 32
    // planes: 13.3 -> 10.0 us.
    p.plane_chunk = grid < 8ll * sms && p.planes > 8 ? 8 : p.planes;
    const dim3 ctas(static_cast<unsigned>(grid), static_cast<unsigned>((p.planes + p.plane_chunk - 1) / p.plane_chunk));
    auto* kernel = ctas.y > 1 ? (wide ? rlt::finalize_kernel<true, true> : rlt::finalize_kernel<false, true>)
                              : (wide ? rlt::finalize_kernel<true, false> : rlt::finalize_kernel<false, false>);
    RLT_CUDA_TRY(rlt::launch_following(kernel, ctas, rlt::kThreads, reinterpret_cast<cudaStream_t>(stream), p));
    rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  }
  return RLT_OK;
}

}  // extern "C"
