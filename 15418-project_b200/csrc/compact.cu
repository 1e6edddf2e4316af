// Device-side materialisation of query results: the int32 result array
// [lines][slots][2] of one query (partition-local offsets, -1 = no match)
// becomes a dense list of matches in (line, slot) order with global offsets,
// and the bytes of each match are gathered into one contiguous arena.  The
// reference does this on the host for every line and slot, building one
// std::string per match from the host copy of the partition
// (src/gpjson/query/kernels/orig/query_executor_host.cu:80-119); here only
// the matches and their bytes cross PCIe.
//
// Two launches, deterministic order: the first counts every block's matches
// and bytes, and its last block to finish scans those counts; in the second
// every block writes its matches at its scanned offsets.  The matches of a
// block are listed in shared memory, so that their records leave as one
// stream of words and each text is copied by several lanes: 111,000 posts with
// eight slots each (890,000 pairs, 7.1 MB; 440,000 matches, 18 MB of records)
// take 36 us; 83 us when each thread wrote its own matches and copied their
// bytes one by one (67 us in that kernel alone, a dependent load and store per
// byte).  What is left is bound by instructions (27 a match) and by the texts'
// scattered sectors (35 MB read for 5 MB of text).
#include "compact.cuh"
#include "overlap.cuh"

namespace gpjb {
namespace {

// A block of the writing kernel: small, so that the last wave is nearly full
// and a block's matches take 20 KB of shared memory.
constexpr int kThreads = 128;
constexpr int kItemsPerThread = 4;
constexpr uint32_t kItemsPerBlock = kThreads * kItemsPerThread;
// A block of the counting kernel counts for four of them; its size is what the
// scan over all counts takes a step.
constexpr int kCountThreads = 512;
constexpr uint32_t kCountBlocks = kCountThreads / kThreads;

// A block's counts in scratch: before the scan {bytes, matches | invalid <<
// 32}, after it the bytes and matches before the block.
struct BlockCounts {
  unsigned long long bytes, matches;
};

// One (line, slot) pair: -1 on either side is "no match", as in the
// reference; a pair with start > end or end beyond the partition is an
// invalid range (the reference raises an execution error for it).
struct Item {
  uint32_t start, len;
  bool match, invalid;
};

__device__ __forceinline__ Item classify(int32_t a, int32_t b, uint64_t n) {
  Item it;
  const bool some = a >= 0 && b >= 0;
  it.invalid = some && (a > b || uint64_t(b) > n);
  it.match = some && !it.invalid;
  it.start = uint32_t(a);
  it.len = it.match ? uint32_t(b - a) : 0u;
  return it;
}

// The thread's four consecutive pairs, as 16-byte loads where the array is
// aligned for them.
__device__ __forceinline__ void load_items(const int32_t *res, uint64_t first, uint64_t items,
                                           uint64_t n, Item (&out)[kItemsPerThread]) {
  static_assert(kItemsPerThread == 4, "two 16-byte loads");
  int32_t v[8];
  if (first + 4 <= items && (reinterpret_cast<uintptr_t>(res) & 15u) == 0) {
    const int4 *p = reinterpret_cast<const int4 *>(res + 2 * first);
    const int4 x = p[0], y = p[1];
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
    v[4] = y.x, v[5] = y.y, v[6] = y.z, v[7] = y.w;
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = first + k / 2 < items ? res[2 * first + k] : -1;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) out[k] = classify(v[2 * k], v[2 * k + 1], n);
}

// Block-wide exclusive scan of a 64-bit and a 32-bit counter, with totals.
template <int kBlock>
__device__ __forceinline__ void block_scan(uint64_t &b, uint32_t &m, uint64_t &total_b,
                                           uint32_t &total_m) {
  constexpr int kWarps = kBlock / 32;
  __shared__ unsigned long long s_b[kWarps];
  __shared__ uint32_t s_m[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t ib = b;
  uint32_t im = m;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint64_t xb = __shfl_up_sync(0xFFFFFFFFu, ib, off);
    const uint32_t xm = __shfl_up_sync(0xFFFFFFFFu, im, off);
    if (lane >= off) {
      ib += xb;
      im += xm;
    }
  }
  if (lane == 31) {
    s_b[warp] = ib;
    s_m[warp] = im;
  }
  __syncthreads();
  uint64_t wb = 0;
  uint32_t wm = 0;
  total_b = 0;
  total_m = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) {
      wb += s_b[w];
      wm += s_m[w];
    }
    total_b += s_b[w];
    total_m += s_m[w];
  }
  b = wb + ib - b;
  m = wm + im - m;
  __syncthreads();
}

// `ticket` counts finished blocks (zero on entry; it wraps to zero with the
// last one); the last block scans the counts of all writing blocks in place and
// writes the totals.
__global__ void __launch_bounds__(kCountThreads)
    count_kernel(const int32_t *res, uint64_t items, uint64_t n, BlockCounts *blocks,
                 uint32_t num_blocks, unsigned int *ticket, unsigned long long *counts) {
  __shared__ unsigned long long s_b[kCountThreads / 32];
  __shared__ uint32_t s_m[kCountThreads / 32];
  __shared__ bool s_last;
  // the writing kernel may start: it waits for this grid before it reads the
  // counts
  asm volatile("griddepcontrol.launch_dependents;");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Item it[kItemsPerThread];
  load_items(res, (uint64_t(blockIdx.x) * kCountThreads + threadIdx.x) * kItemsPerThread, items, n,
             it);
  uint64_t b = 0;
  uint32_t m = 0;  // matches | invalid << 16: at most 512 of each
#pragma unroll
  for (int k = 0; k < kItemsPerThread; ++k) {
    b += it[k].len;
    m += uint32_t(it[k].match) | uint32_t(it[k].invalid) << 16;
  }
  m = __reduce_add_sync(0xFFFFFFFFu, m);
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) b += __shfl_down_sync(0xFFFFFFFFu, b, off);
  if (lane == 0) {
    s_b[warp] = b;
    s_m[warp] = m;
  }
  __syncthreads();
  const uint32_t mine = blockIdx.x * kCountBlocks + threadIdx.x;
  if (threadIdx.x < kCountBlocks && mine < num_blocks) {
    constexpr int kEach = kThreads / 32;
    b = 0;
    m = 0;
#pragma unroll
    for (int w = 0; w < kEach; ++w) {
      b += s_b[threadIdx.x * kEach + w];
      m += s_m[threadIdx.x * kEach + w];
    }
    blocks[mine] = {b, uint64_t(m & 0xFFFFu) | uint64_t(m >> 16) << 32};
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // four consecutive counts per thread and step
  uint64_t carry_b = 0, carry_m = 0, invalid = 0, total_b;
  uint32_t total_m;
  for (uint32_t first = 0; first < num_blocks; first += 4u * kCountThreads) {
    const uint32_t i = first + 4u * threadIdx.x;
    ulonglong2 c[4];
    uint64_t eb = 0;
    uint32_t em = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k)
      c[k] = i + k < num_blocks ? __ldcg(reinterpret_cast<const ulonglong2 *>(&blocks[i + k]))
                                : make_ulonglong2(0, 0);
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
      eb += c[k].x;
      em += uint32_t(c[k].y);
      invalid += c[k].y >> 32;
    }
    block_scan<kCountThreads>(eb, em, total_b, total_m);
    uint64_t at_b = carry_b + eb, at_m = carry_m + em;
#pragma unroll
    for (uint32_t k = 0; k < 4u; ++k) {
      if (i + k < num_blocks) blocks[i + k] = {at_b, at_m};
      at_b += c[k].x;
      at_m += uint32_t(c[k].y);
    }
    carry_b += total_b;
    carry_m += total_m;
  }
  uint32_t none = 0;
  block_scan<kCountThreads>(invalid, none, total_b, total_m);
  if (threadIdx.x == 0) {
    counts[0] = carry_m;
    counts[1] = carry_b;
    counts[2] = total_b;
  }
}

// Copies len bytes by `width` threads (this is thread `rank` of them), four
// bytes in flight per thread.
__device__ __forceinline__ void copy_text(uint8_t *__restrict__ dst,
                                          const uint8_t *__restrict__ src, uint32_t len,
                                          uint32_t rank, uint32_t width) {
  uint64_t x = rank;
  for (; x + 3u * width < len; x += 4u * width) {
    const uint8_t a = src[x], b = src[x + width], c = src[x + 2u * width],
                  d = src[x + 3u * width];
    dst[x] = a;
    dst[x + width] = b;
    dst[x + 2u * width] = c;
    dst[x + 3u * width] = d;
  }
  for (; x < len; x += width) dst[x] = src[x];
}

// Texts up to these lengths are copied by 8 lanes and by a warp, longer ones by
// the whole block.
constexpr uint32_t kShortText = 256, kLongText = 16384;

// A match record as it leaves: gpj_match as five words.
struct Record {
  unsigned long long line, slot_len, start, end, text;
};
static_assert(sizeof(Record) == sizeof(gpj_match) && sizeof(Record) == 40, "five words");

__global__ void __launch_bounds__(kThreads, 10)
    write_kernel(const int32_t *res, uint64_t items, uint32_t slots, const uint8_t *in, uint64_t n,
                 int64_t base_offset, const BlockCounts *blocks, unsigned int *ticket,
                 gpj_match *matches, uint64_t match_cap, uint8_t *arena, uint64_t arena_cap) {
  __shared__ Record s_match[kItemsPerBlock];
  __shared__ uint32_t s_longer;  // bit 0: texts for a warp, bit 1: for the block
  const uint64_t first_item = uint64_t(blockIdx.x) * kItemsPerBlock;
  const uint32_t mine = threadIdx.x * kItemsPerThread;
  Item it[kItemsPerThread];
  load_items(res, first_item + mine, items, n, it);
  if (threadIdx.x == 0) s_longer = 0;
  uint64_t b = 0, total_b;
  uint32_t m = 0, count;
#pragma unroll
  for (int k = 0; k < kItemsPerThread; ++k) {
    b += it[k].len;
    m += it[k].match ? 1u : 0u;
  }
  block_scan<kThreads>(b, m, total_b, count);  // its barriers order s_longer as well
  // launched while the counting kernel runs; from here on its counts are there
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // The next call starts from zero whatever happened to the ticket: the last
  // of several overlapping calls to get here follows all their counting.
  if (blockIdx.x == 0 && threadIdx.x == 0) *ticket = 0;
  const BlockCounts before = blocks[blockIdx.x];
  // line and slot of the thread's first pair; the first line is the block's
  uint64_t line = first_item / slots;
  const uint64_t pair = first_item % slots + mine;
  const uint32_t lines_on =
      pair <= 0xFFFFFFFFull ? uint32_t(pair) / slots : uint32_t(pair / slots);
  line += lines_on;
  uint32_t slot = uint32_t(pair - uint64_t(lines_on) * slots);
  uint32_t longer = 0;
#pragma unroll
  for (int k = 0; k < kItemsPerThread; ++k) {
    if (it[k].match) {
      Record r;
      r.line = line;
      r.slot_len = uint64_t(slot) | uint64_t(it[k].len) << 32;
      r.start = uint64_t(base_offset) + it[k].start;
      r.end = r.start + it[k].len;
      r.text = before.bytes + b;
      s_match[m] = r;
      longer |= it[k].len > kLongText ? 2u : (it[k].len > kShortText ? 1u : 0u);
      ++m;
      b += it[k].len;
    }
    if (++slot == slots) {
      slot = 0;
      ++line;
    }
  }
  if (longer != 0) atomicOr(&s_longer, longer);
  __syncthreads();

  // the match records leave as one stream of words
  if (before.matches < match_cap) {
    const uint64_t room = match_cap - before.matches;
    const uint32_t words = 5u * (room < count ? uint32_t(room) : count);
    const auto *from = reinterpret_cast<const unsigned long long *>(s_match);
    auto *to = reinterpret_cast<unsigned long long *>(matches + before.matches);
    for (uint32_t w = threadIdx.x; w < words; w += kThreads) to[w] = from[w];
  }
  if (arena == nullptr || in == nullptr) return;

  const bool all_fit = before.bytes + total_b <= arena_cap;
  auto length = [&](uint32_t j) {  // 0 where the arena ends before the text does
    const uint32_t len = uint32_t(s_match[j].slot_len >> 32);
    return all_fit || s_match[j].text + len <= arena_cap ? len : 0u;
  };
  auto source = [&](uint32_t j) {
    return in + uint32_t(uint32_t(s_match[j].start) - uint32_t(base_offset));
  };
  // Short texts: 8 lanes each, the first 16 bytes of four texts in flight per
  // group (a text is some ten bytes in a sector of its own: the reads wait on
  // memory one by one otherwise).
  constexpr uint32_t kGroups = kThreads / 8u;
  const uint32_t rank = threadIdx.x % 8u;
  for (uint32_t j0 = threadIdx.x / 8u; j0 < count; j0 += 4u * kGroups) {
    uint8_t lo[4], hi[4];
    uint32_t len[4];
    uint32_t longest = 0;
#pragma unroll
    for (uint32_t u = 0; u < 4u; ++u) {
      const uint32_t j = j0 + u * kGroups;
      len[u] = j < count ? length(j) : 0u;
      if (len[u] > kShortText) len[u] = 0;
      longest = len[u] > longest ? len[u] : longest;
      if (rank < len[u]) {
        const uint8_t *src = source(j) + rank;
        lo[u] = src[0];
        if (rank + 8u < len[u]) hi[u] = src[8];
      }
    }
#pragma unroll
    for (uint32_t u = 0; u < 4u; ++u) {
      if (rank < len[u]) {
        uint8_t *dst = arena + s_match[j0 + u * kGroups].text + rank;
        dst[0] = lo[u];
        if (rank + 8u < len[u]) dst[8] = hi[u];
      }
    }
    if (longest > 16u) {
#pragma unroll
      for (uint32_t u = 0; u < 4u; ++u) {
        const uint32_t j = j0 + u * kGroups;
        if (len[u] > 16u)
          copy_text(arena + s_match[j].text + 16u, source(j) + 16u, len[u] - 16u, rank, 8u);
      }
    }
  }
  if (s_longer & 1u) {
    for (uint32_t j = threadIdx.x / 32u; j < count; j += kThreads / 32) {
      const uint32_t len = length(j);
      if (len > kShortText && len <= kLongText)
        copy_text(arena + s_match[j].text, source(j), len, threadIdx.x % 32u, 32u);
    }
  }
  if (s_longer & 2u) {
    for (uint32_t j = 0; j < count; ++j) {
      const uint32_t len = length(j);
      if (len > kLongText)
        copy_text(arena + s_match[j].text, source(j), len, threadIdx.x, kThreads);
    }
  }
}

}  // namespace

uint64_t compact_scratch_bytes(uint64_t lines, uint32_t slots) {
  const uint64_t items = lines * uint64_t(slots);
  const uint64_t blocks = (items + kItemsPerBlock - 1) / kItemsPerBlock;
  return kCompactHeaderBytes + blocks * sizeof(BlockCounts);
}

cudaError_t compact_launch(const int32_t *d_results, uint64_t lines, uint32_t slots,
                           const uint8_t *d_input, uint64_t n, int64_t base_offset,
                           gpj_match *d_matches, uint64_t match_cap, uint8_t *d_arena,
                           uint64_t arena_cap, unsigned long long *d_counts, void *scratch,
                           cudaStream_t stream) {
  const uint64_t items = lines * uint64_t(slots);
  if (items == 0) return cudaMemsetAsync(d_counts, 0, 3 * sizeof(unsigned long long), stream);
  const uint64_t blocks = (items + kItemsPerBlock - 1) / kItemsPerBlock;
  if (blocks > 0x7FFFFFFFull) return cudaErrorInvalidValue;
  auto *ticket = static_cast<unsigned int *>(scratch);
  auto *bc = reinterpret_cast<BlockCounts *>(static_cast<uint8_t *>(scratch) + kCompactHeaderBytes);
  count_kernel<<<uint32_t((blocks + kCountBlocks - 1) / kCountBlocks), kCountThreads, 0, stream>>>(
      d_results, items, n, bc, uint32_t(blocks), ticket, d_counts);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_overlapped(write_kernel, uint32_t(blocks), kThreads, 0, stream, d_results, items,
                           slots, d_input, n, base_offset, bc, ticket, d_matches, match_cap,
                           d_arena, arena_cap);
}

}  // namespace gpjb
