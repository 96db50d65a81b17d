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
// request, so that the copies of one layer on one plane are neighbours in one block. The CTAs of a group share out
// the vectors (selected layer, row, vector of the row) of one of its tensors in equal parts, rows that need no copy left
// out. The grid holds one short CTA per part, in order of the groups: bound by HBM, the kernel is fastest while the
// SMs work close together (block_moves.cu has the measurements), and a decode step of a few rows still reaches every SM.
// A CTA's own preparation is two rounds of lookups: the rows, then the blocks of their planes.
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
  const int* tables;              // [requests, planes, table_width]
  int table_width, num_requests;
  const int* rows;                // [n][3]: request index, exit plane, token position
  int n;
  int* status;
};

constexpr int kGroupRows = 16;
constexpr int kPlaneChunk = 64;  // planes whose blocks are looked up together

struct GroupShared {
  int layer_of[64];                               // the selected layers, in order
  int carried;                                    // rows of the group with something to copy; the lists below hold those
  int request[kGroupRows], page[kGroupRows], exit_plane[kGroupRows], token[kGroupRows];
  long long src[kGroupRows];                      // byte offset of the exit plane's block, -1 if its id is bad
  long long dst[kGroupRows][kPlaneChunk];         // the same for the planes of the chunk; -1 also where nothing is due
};

// The rows of the group that need copies, compacted by warp 0. An invalid row is reported by the group's first CTA.
__device__ __forceinline__ void list_rows(const FinalizeParams& p, int group, bool say, GroupShared& s) {
  const int tid = static_cast<int>(threadIdx.x);
  if (tid < 64 && ((p.layer_mask >> tid) & 1ull)) s.layer_of[__popcll(p.layer_mask & ((1ull << tid) - 1ull))] = tid;
  if (tid >= 32) return;
  const long long row = static_cast<long long>(group) * kGroupRows + tid;
  int request = -1, e = 0, position = 0;
  bool carry = false;
  if (tid < kGroupRows && row < p.n) {
    request = p.rows[3 * row];
    e = p.rows[3 * row + 1];
    position = p.rows[3 * row + 2];
    const bool valid = request >= 0 && request < p.num_requests && e >= 0 && e < p.planes && position >= 0 &&
                       position < p.table_width * p.block_size;
    if (!valid && say) report(p.status, RLT_STATUS_BAD_PLANE, static_cast<int>(row), position, e);
    carry = valid && e + 1 < p.planes;
  }
  const unsigned keep = __ballot_sync(0xffffffffu, carry);
  if (carry) {
    const int slot = __popc(keep & ((1u << tid) - 1u));
    s.request[slot] = request;
    s.exit_plane[slot] = e;
    s.page[slot] = position / p.block_size;
    s.token[slot] = position % p.block_size;
  }
  if (tid == 0) s.carried = __popc(keep);
}

// The share of a group's vectors that one CTA copies: vectors [first, first + count) in the order layer, listed row,
// vector of the row; the first lies `rem` vectors into line `line`, a line being one row of one layer.
struct Share {
  int first, count, line, rem, lines;
};
__device__ __forceinline__ Share share_of(const FinalizeParams& p, const FinalizeRegion& rg, int part, int carried) {
  const long long all = static_cast<long long>(p.layers) * carried * rg.row_vecs;
  Share h;
  h.first = static_cast<int>(all * part / rg.parts);
  h.count = static_cast<int>(all * (part + 1) / rg.parts) - h.first;
  h.line = h.first / rg.row_vecs;
  h.rem = h.first - h.line * rg.row_vecs;
  h.lines = (h.rem + h.count + rg.row_vecs - 1) / rg.row_vecs;
  return h;
}

// Blocks of planes [chunk, chunk + kPlaneChunk) of the listed rows that the share touches, and of their exit planes.
__device__ __forceinline__ void look_up_blocks(const FinalizeParams& p, const FinalizeRegion& rg, const Share& h, int chunk,
                                               GroupShared& s) {
  const int width = min(kPlaneChunk, p.planes - chunk) + 1;  // the last column is the exit plane
  const int n = s.carried, touched = min(h.lines, n), from = h.line % n;
  for (int i = static_cast<int>(threadIdx.x); i < touched * width; i += kThreads) {
    const int i_row = i / width, column = i - i_row * width;
    const int r = from + i_row < n ? from + i_row : from + i_row - n;
    const bool source = column == width - 1;
    const int e = s.exit_plane[r], plane = source ? e : chunk + column;
    long long at = -1;
    if (source || plane > e) {
      const int block = p.tables[(static_cast<long long>(s.request[r]) * p.planes + plane) * p.table_width + s.page[r]];
      if (static_cast<unsigned>(block) < static_cast<unsigned>(p.num_blocks)) {
        at = block * rg.block_bytes;
      } else {
        report(p.status, RLT_STATUS_BAD_BLOCK, s.request[r], s.page[r], block);
      }
    }
    if (source) {
      s.src[r] = at;
    } else {
      s.dst[r][column] = at;
    }
  }
}

template <typename T>
__device__ __forceinline__ void copy_share(const FinalizeParams& p, const FinalizeRegion& rg, char* pool, const Share& h, int chunk,
                                           const GroupShared& s) {
  const int n = s.carried;
  const unsigned n_magic = n == 1 ? 0u : static_cast<unsigned>((1ull << 32) / static_cast<unsigned>(n)) + 1u;
  const int chunk_planes = min(kPlaneChunk, p.planes - chunk);
  for (int k = static_cast<int>(threadIdx.x); k < h.count; k += kThreads) {
    const unsigned j = static_cast<unsigned>(h.rem + k);
    const int q = rg.row_magic ? static_cast<int>(__umulhi(j, rg.row_magic)) : static_cast<int>(j);
    const int line = h.line + q;
    const int layer = n_magic ? static_cast<int>(__umulhi(static_cast<unsigned>(line), n_magic)) : line;
    const int row = line - layer * n;
    const long long src = s.src[row];
    if (src < 0) continue;
    char* at = pool + s.layer_of[layer] * rg.layer_bytes + s.token[row] * rg.token_bytes +
               (static_cast<int>(j) - q * rg.row_vecs) * static_cast<int>(sizeof(T));
    const T v = ld_stream(reinterpret_cast<const T*>(at + src));
    for (int c = max(s.exit_plane[row] + 1 - chunk, 0); c < chunk_planes; ++c) {
      const long long to = s.dst[row][c];
      if (to >= 0) st_stream(reinterpret_cast<T*>(at + to), v);
    }
  }
}

__global__ void __launch_bounds__(kThreads, 5) finalize_kernel(const __grid_constant__ FinalizeParams p) {
  __shared__ GroupShared s;
  const int group = static_cast<int>(blockIdx.x / p.parts);
  int at = static_cast<int>(blockIdx.x) - group * p.parts;
  follow_stream();
  list_rows(p, group, at == 0, s);
  const int g = at >= 2 * p.region[0].parts;
  const FinalizeRegion& rg = p.region[g];
  if (g) at -= 2 * p.region[0].parts;
  const int kv = at >= rg.parts;
  char* pool = kv ? rg.value : rg.key;
  const int part = at - kv * rg.parts;
  __syncthreads();
  if (s.carried == 0) return;
  const Share h = share_of(p, rg, part, s.carried);
  for (int chunk = 0; chunk < p.planes; chunk += kPlaneChunk) {
    look_up_blocks(p, rg, h, chunk, s);
    __syncthreads();
    if (rg.vec_bytes == 32) {
      copy_share<Vec32>(p, rg, pool, h, chunk, s);
    } else if (rg.vec_bytes == 16) {
      copy_share<uint4>(p, rg, pool, h, chunk, s);
    } else if (rg.vec_bytes == 4) {
      copy_share<uint32_t>(p, rg, pool, h, chunk, s);
    } else {
      copy_share<uint8_t>(p, rg, pool, h, chunk, s);
    }
    if (chunk + kPlaneChunk < p.planes) __syncthreads();
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
  p.rows = rows;
  p.n = count;
  p.status = status;
  int sms = 0;
  const int rc = rlt::sm_count(&sms);
  if (rc != RLT_OK) return rc;
  const long long groups = (static_cast<long long>(count) + rlt::kGroupRows - 1) / rlt::kGroupRows;
  // Vectors per thread of a CTA's share: enough stores behind the two rounds of lookups, whatever the number of planes.
  // 4,000 rows of four planes (Ouro-1.4B): 485 us at 1, 282 at 4, 277 at 6, 278 at 8; 483 rows of 32 planes (Huginn): 318 us at 1,
  // 337 at 2. (The persistent kernel this one replaced: 324 and 369 us; 64 rows of a decode step 12.6 -> 8.5 us.)
  const int rounds = std::clamp(24 / p.planes, 1, 8);
  for (int g = 0; g < regions; ++g) {
    rlt::FinalizeRegion& rg = p.region[g];
    const long long per = static_cast<long long>(rlt::kThreads) * rounds * (rg.vec_bytes == 32 ? 1 : rg.vec_bytes == 16 ? 2 : rg.vec_bytes == 4 ? 4 : 8);
    const long long vectors = static_cast<long long>(p.layers) * rlt::kGroupRows * rg.row_vecs;
    rg.parts = static_cast<int>((vectors + per - 1) / per);
    p.parts += 2 * rg.parts;
  }
  const long long grid = groups * p.parts;
  if (grid > 0x7fffffffll) return RLT_E_LIMIT;
  RLT_CUDA_TRY(rlt::launch_following(rlt::finalize_kernel, static_cast<unsigned>(grid), rlt::kThreads,
                                     reinterpret_cast<cudaStream_t>(stream), p));
  rlt::g_launches.fetch_add(1, std::memory_order_relaxed);
  return RLT_OK;
}

}  // extern "C"
