// Host-side interface of the JSONPath query kernels (internal).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "indexer.cuh"
#include "ir.cuh"

namespace gpjb {

// Status bit a query raises when a record had more results than its slots:
// a "[*]" array or open slice longer than the wildcard limit, or more
// "..name" matches.
// Only IR with extension opcodes can raise it.  Kept clear of the indexer's
// error bits (1, 2, 4), with which it shares the batch's error word.
constexpr unsigned int kQueryStatusOverflow = 0x100u;

// Queries over every record of one partition, run by one launch (up to
// kMaxLaunchQueries, their IR packed in the IrBlob).
constexpr int kMaxLaunchQueries = 8;
struct QueryOne {
  int ir_off = 0;
  int ir_len = 0;
  int num_results = 0;           // result slots per record
  int base_level = 0;            // bitmap level of query level 0 (1: elements
                                 // of a top-level array are the records)
  void *out = nullptr;           // [num_lines][num_results][2] int32 or int64
  bool ext = false;              // extension opcodes (query_launch sets it)
};
struct QueryLaunch {
  const uint8_t *in = nullptr;   // partition bytes
  int64_t n = 0;
  const int64_t *NL = nullptr;   // newline index
  int64_t num_lines = 0;
  const uint64_t *S = nullptr;   // string mask [W]
  const uint64_t *LB = nullptr;  // leveled bitmaps [L*W]
  int64_t W = 0;
  int num_levels = 0;            // levels present in LB; deeper reads see 0
  bool wide = false;             // 64-bit offsets in `out`
  int num_queries = 1;
  QueryOne queries[kMaxLaunchQueries];
  unsigned int *status = nullptr;  // kQueryStatusOverflow is OR-ed here (optional)
};

// The IR travels in the kernel parameters (4 KiB, copied into shared memory
// by every CTA), so concurrent launches never share an IR buffer.
struct IrBlob {
  uint8_t bytes[kMaxQueryIrBytes];
};

// One launch, or two where queries with "..name" (a warp per record) go apart.
cudaError_t query_launch(QueryLaunch q, const IrBlob &ir, cudaStream_t stream);

// Batched query over every record of every file of a multi-file index build:
// record r belongs to the file whose record range holds it (file_info from
// index_finalize_files); the file's query group selects the IR (packed in the
// IrBlob), slot count and record level.  The record count is read on the
// device, so the launch needs no host round trip.
constexpr int kMaxBatchGroups = 8;
struct BatchQueryGroup {
  int ir_off = 0;
  int ir_len = 0;
  int num_results = 0;
  int base_level = 0;
  bool ext = false;  // extension opcodes (batch_query_launch sets it)
};
struct BatchQueryLaunch {
  const uint8_t *in = nullptr;
  const uint64_t *S = nullptr;
  const uint64_t *LB = nullptr;
  const int64_t *NL = nullptr;
  const IndexFile *files = nullptr;
  uint32_t num_files = 0;
  const uint64_t *file_info = nullptr;  // kFileInfoWords per file
  const uint64_t *totals = nullptr;
  int32_t *out = nullptr;
  unsigned int *status = nullptr;  // kQueryStatusOverflow is OR-ed here (optional)
  unsigned int *file_status = nullptr;  // or into one word per file (optional, first)
  // records are handed to warps from this counter, which the launch zeroes
  // first unless the kernels before it did (optional; without it each warp
  // strides)
  unsigned long long *record_counter = nullptr;
  bool counter_cleared = false;
  // about the number of records (0: unknown, many) and their bytes: choose the
  // lanes per record, the number bounds the grid; the results do not depend on
  // them
  uint64_t expected_records = 0, expected_bytes = 0;
  int num_groups = 0;
  BatchQueryGroup groups[kMaxBatchGroups];
  uint32_t used_groups = ~0u;  // bit g: some file is of group g
  // groups whose files' records a launch of some of them runs (batch_query_launch
  // sets it)
  uint32_t group_mask = 0;
};

// Blocks that batch_query_launch starts of the `grid` it may (in its first launch
// where it makes two).
int batch_query_grid(BatchQueryLaunch q, const IrBlob &ir, int grid, int block);

// One launch, or two where files with a "..name" query (a warp per record) go
// apart: each passes over the other's files.
cudaError_t batch_query_launch(BatchQueryLaunch q, const IrBlob &ir, int grid, int block,
                               cudaStream_t stream);

}  // namespace gpjb
