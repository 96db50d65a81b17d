// Handoff, pack and scatter of a batch whose tables the HOST holds: the host writes one record per (request, page)
// and the kernels of block_moves.cu look nothing up but that record. Internal to the library and its Python module.
#pragma once

#include <stdint.h>

#include "rlt_kv_handoff.h"

// A record is `words` int32 long:
//   [0] request   [1] logical page
//   [2] first token of the page in range | one past the last << 8; -1: the request's range is bad, [3] / [4] hold it
//   [3] tokens of the request's range before this page   [4] tokens of the batch before the request
//   [5] tokens of the request's range
//   [6 ...] source block of every source plane, destination block of every destination plane, and, if the batch has
//   exit planes, one exit plane per token of the page (only those in range are read).
constexpr int kRecordHeader = 6;
constexpr int kRecordBad = -1;

// Pools of more planes are served by the table-driven kernels.
constexpr int kMaxRecordPlanes = 64;

// Records up to this many words travel as kernel parameters: no staging slot, no copy, no event. (The launch takes the smallest of
// three parameter blocks that holds them.)
constexpr int kInlineWords = 7680;
constexpr int kInlineMediumWords = 1920;
constexpr int kInlineSmallWords = 896;

struct RltBlockMoves {
  const int32_t* host_records;    // always given
  const int32_t* device_records;  // the same, staged; may be NULL while the records fit the kernel parameters
  int32_t blocks;                 // records
  int32_t words;                  // int32 per record
  int32_t src_planes, dst_planes; // 0: that side has no tables
  int32_t block_size;
  int32_t has_exit;
  int32_t num_requests, table_width;  // of the batch the records were made from
  // A dedup wire image (pack / scatter in RLT_MODE_DEDUP) also needs, per record and plane, the (token, plane) pairs
  // that lie before it on the wire, and their total.
  const int32_t* host_wire;    // [blocks][planes] or NULL
  const int32_t* device_wire;  // the same, staged, or NULL
  int64_t wire_tokens;
};

#ifdef __cplusplus
extern "C" {
#endif

// Whether this launch can be made from records; if not, the entry points of rlt_kv_handoff.h serve it.
enum { RLT_MOVE_DIRECT = 0, RLT_MOVE_PACK = 1, RLT_MOVE_SCATTER = 2 };
#define RLT_MOVE_UNSUITED 1

// RLT_OK, an error code with the conditions of rlt_kv_handoff / rlt_kv_pack / rlt_kv_scatter, or RLT_MOVE_UNSUITED
// (nothing launched): options that steer the table-driven kernels, more than 64 planes, very long rows.
RLT_API int rlt_move_blocks(int direction, const RltPool* src, const RltPool* dst, const RltBlockMoves* moves,
                            const RltOptions* options, void* packed, int64_t packed_bytes, rlt_stream_t stream);

// The same for a direct handoff whose records are not staged: records that do not fit the kernel parameters go through a
// slot of rlt_kv_handoff_host's staging ring, RLT_MOVE_UNSUITED if they do not fit that either.
RLT_API int rlt_handoff_staged(const RltPool* src, const RltPool* dst, const RltBlockMoves* moves, const RltOptions* options,
                               rlt_stream_t stream);

#ifdef __cplusplus
}
#endif
