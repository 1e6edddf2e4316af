// Many small copies between device and pinned host memory in one launch
// (internal).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace gpjb {

struct CopyItem {
  const void *src = nullptr;  // null: zeroes are written
  void *dst = nullptr;
  uint64_t bytes = 0;
};

// Enqueues the copies on `stream`, one kernel per 64 of them, in no order among
// each other.  Every address must be accessible to the device (device memory,
// or pinned host memory that host_range_mapped confirmed or cudaMallocHost
// returned).
cudaError_t copy_many(const CopyItem *items, int count, cudaStream_t stream);

// True when [p, p + bytes) lies inside one page-locked host allocation or
// registration that kernels can read at the same address.
bool host_range_mapped(const void *p, uint64_t bytes);

// Up to this size a host input is read by copy_many instead of the copy
// engine: a copy of its own takes the engine 5-6 us beside the bytes' time at
// 55 GB/s, a kernel reads them together (21 files, 4 MiB in all: 80 us for 190;
// a burst of 40 requests 1,414 -> 1,171 us with the results moved likewise; a
// burst from buffers never read before 1,320 us, 1,515 with the engine for the
// inputs).
constexpr uint64_t kCopyManyMaxInput = 1u << 20;
// The same for results, which are mostly a few KiB.
constexpr uint64_t kCopyManyMaxResult = 256u << 10;

}  // namespace gpjb
