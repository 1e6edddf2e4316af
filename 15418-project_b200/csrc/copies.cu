// Many small copies in one launch.  A request of the server moves a small file
// to the device and a few KiB of results and status words back; as copies of
// their own these took 6-9 us each, one after another on their stream, and two
// to three microseconds each of the scheduler thread.  PCIe bounds what is
// left: the kernel only has to keep enough 16-byte loads in flight.
#include "copies.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

namespace gpjb {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxItems = 64;
constexpr uint32_t kChunk = 16384;  // bytes per block: four 16-byte loads a thread

struct CopyTable {
  CopyItem item[kMaxItems];
  uint32_t first[kMaxItems + 1];  // first block of each item
  int count;
};

// Copies (or zeroes) `bytes` bytes of elements of type T by the whole block.
template <typename T>
__device__ __forceinline__ void copy_elements(uint8_t *dst, const uint8_t *src, uint32_t bytes) {
  T *d = reinterpret_cast<T *>(dst);
  const T *s = reinterpret_cast<const T *>(src);
  const uint32_t n = bytes / uint32_t(sizeof(T));
  for (uint32_t i = threadIdx.x; i < n; i += 4u * kThreads) {
    T v[4] = {};
    if (s != nullptr) {
#pragma unroll
      for (uint32_t k = 0; k < 4u; ++k)
        if (i + k * kThreads < n) v[k] = s[i + k * kThreads];
    }
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
      if (i + k * kThreads < n) d[i + k * kThreads] = v[k];
  }
}

__global__ void __launch_bounds__(kThreads) copy_kernel(const __grid_constant__ CopyTable t) {
  int i = 0;
  while (i + 1 < t.count && t.first[i + 1] <= blockIdx.x) ++i;
  const uint64_t off = uint64_t(blockIdx.x - t.first[i]) * kChunk;
  const uint64_t left = t.item[i].bytes - off;
  const uint32_t bytes = left < kChunk ? uint32_t(left) : kChunk;
  uint8_t *dst = static_cast<uint8_t *>(t.item[i].dst) + off;
  const uint8_t *src =
      t.item[i].src != nullptr ? static_cast<const uint8_t *>(t.item[i].src) + off : nullptr;
  const uintptr_t both = reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src);
  uint32_t done = 0;
  if ((both & 15u) == 0) {
    copy_elements<uint4>(dst, src, bytes);
    done = bytes & ~15u;
  } else if ((both & 3u) == 0) {
    copy_elements<uint32_t>(dst, src, bytes);
    done = bytes & ~3u;
  }
  copy_elements<uint8_t>(dst + done, src != nullptr ? src + done : nullptr, bytes - done);
}

}  // namespace

cudaError_t copy_many(const CopyItem *items, int count, cudaStream_t stream) {
  for (int at = 0; at < count;) {
    CopyTable t;
    t.count = 0;
    uint64_t blocks = 0;
    for (; at < count && t.count < kMaxItems; ++at) {
      if (items[at].bytes == 0) continue;
      const uint64_t mine = (items[at].bytes + kChunk - 1) / kChunk;
      if (blocks + mine > 0x7FFFFFFFull) {
        if (t.count == 0) return cudaErrorInvalidValue;
        break;
      }
      t.item[t.count] = items[at];
      t.first[t.count++] = uint32_t(blocks);
      blocks += mine;
    }
    if (t.count == 0) continue;
    copy_kernel<<<uint32_t(blocks), kThreads, 0, stream>>>(t);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

bool host_range_mapped(const void *p, uint64_t bytes) {
  static const auto get = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuPointerGetAttributes", &fn, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fn = nullptr;
    (void)cudaGetLastError();
    return reinterpret_cast<PFN_cuPointerGetAttributes_v7000>(fn);
  }();
  if (get == nullptr || p == nullptr || bytes == 0) return false;
  unsigned int type = 0;
  CUdeviceptr device = 0, start = 0;
  size_t size = 0;
  CUpointer_attribute what[] = {
      CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_DEVICE_POINTER,
      CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, CU_POINTER_ATTRIBUTE_RANGE_SIZE};
  void *into[] = {&type, &device, &start, &size};
  const auto at = reinterpret_cast<CUdeviceptr>(p);
  if (get(4, what, into, at) != CUDA_SUCCESS) return false;
  return type == CU_MEMORYTYPE_HOST && device == at && start <= at && size >= bytes &&
         at - start <= size - bytes;
}

}  // namespace gpjb
