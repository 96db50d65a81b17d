// What the table-driven launches are told: the walk's parameters, worked out on the host from the pools, the batch
// and the options by table_params(), which is also where every argument error of those entry points is found.
#pragma once

#include "common.cuh"

namespace rlt {

struct RegionParams {
  const char* src_key;
  const char* src_value;
  char* dst_key;
  char* dst_value;
  long long block_bytes;
  long long layer_bytes;
  long long token_bytes;
  int vec_bytes;        // 16, 4 or 1
  int row_vecs;         // token_bytes / vec_bytes
  unsigned row_magic;   // div_magic(row_vecs)
  int wide_ok;          // rows and bases are 32-byte multiples: 32-byte accesses may be used
  int layers_per_unit;  // layers one unit covers
  int chunks;           // ceil(layers in slice / layers_per_unit)
};

struct TableCopyParams {
  RegionParams region[2];
  int num_regions;
  int num_requests;
  int table_width;
  int src_planes;
  int dst_planes;   // destination planes, or wire planes for pack
  int plane_begin;  // planes iterated by this launch: [plane_begin, plane_begin + plane_count)
  int plane_count;
  int block_size;
  int src_blocks;
  int dst_blocks;
  const int* src_tables;
  const int* dst_tables;
  const int* tok_begin;
  const int* tok_end;
  const int* exit_planes;
  const long long* exit_offsets;
  long long exit_count;  // entries in exit_planes
  int plane_bias;   // 0: source plane = min(p, exit); src_planes: source plane = exit
  int layer_begin;
  int layer_end;
  int src_packed;   // source is the packed image (scatter)
  int dst_packed;   // destination is the packed image (pack)
  long long packed_token_bytes;  // 2 * layers in slice * (codes row + scales row)
  long long packed_bytes;        // size of the packed image; rows past it are skipped
  unsigned long long deep_layer_mask;  // layers carried for planes >= 1; 0 = all
  int dedup_wire;                // the packed image holds, per token, only planes up to its exit plane
  const int* dedup_prefix;       // [planes * total blocks] wire tokens before each (request, plane, block)
  int fan;                       // pool-to-pool dedup that reads each row once and stores it to every plane it fills
  int* status;
};

enum Direction { kDirect, kPack, kScatter };

// Checks the arguments of a handoff / pack / scatter and fills `p` (everything but dedup_prefix); RLT_OK or the code
// the entry point returns. Only the null-ness of the batch's arrays is looked at.
int table_params(Direction dir, const RltPool* src, const RltPool* dst, const RltBatch* batch, const RltOptions* opt,
                 void* packed, long long packed_bytes, TableCopyParams& p);

long long dedup_workspace_bytes(long long requests, long long width, long long planes);

}  // namespace rlt
