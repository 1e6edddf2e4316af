// JSONPath query kernel: a group of 1 to 32 lanes per record interprets the
// byte IR over the leveled bitmaps and the string mask and writes (start, end)
// byte offsets per result slot.  Semantics follow
// src/gpjson/query/kernels/orig/query.cu:144-454 of the reference; the IR is
// passed in the kernel parameters and staged in shared memory instead of a
// process-global __constant__ array (query.cu:11), so launches on different
// streams do not race.  Positions are 32-bit for partitions below 2 GiB (every
// value equals the reference's int arithmetic) and 64-bit beyond.
#include "query.cuh"

#include <algorithm>
#include <type_traits>

namespace gpjb {
namespace {

constexpr unsigned kAll = 0xFFFFFFFFu;
constexpr int kIrPad = 16;  // zero bytes after an IR in shared memory

// The G lanes that run one record; a warp runs 32 / G records in lockstep.
// The IR has no jumps, so every record of a warp is at the same opcode and
// the same level, and all 32 lanes take part in every vote; a record that
// failed a step (or a lane without a record) is carried along inactive.
template <int G>
struct Group {
  static_assert(G >= 1 && G <= 32 && (G & (G - 1)) == 0, "lanes per record");
  int lane, shift;
  __device__ __forceinline__ Group() {
    const int l = int(threadIdx.x & 31u);
    lane = l & (G - 1);
    shift = l - lane;
  }
  // bit i = predicate of the group's lane i
  __device__ __forceinline__ unsigned ballot(bool p) const {
    if constexpr (G == 1) return p ? 1u : 0u;
    const unsigned b = __ballot_sync(kAll, p);
    return G == 32 ? b : (b >> shift) & ((1u << (G & 31)) - 1u);
  }
  __device__ __forceinline__ int32_t shfl(int32_t v, int src) const {
    return G == 1 ? v : __shfl_sync(kAll, v, src, G);
  }
  __device__ __forceinline__ int64_t shfl(int64_t v, int src) const {
    return G == 1 ? v : __shfl_sync(kAll, static_cast<long long>(v), src, G);
  }
  // sum over the group's lanes before this one, and over all of them
  __device__ __forceinline__ int sum_before(int v, int &total) const {
    int inc = v;
#pragma unroll
    for (int off = 1; off < G; off <<= 1) {
      const int o = __shfl_up_sync(kAll, inc, off, G);
      if (lane >= off) inc += o;
    }
    total = shfl(inc, G - 1);
    return inc - v;
  }
};

// Counts the steps of a search loop.
template <typename Pos>
using Steps = std::make_unsigned_t<Pos>;

template <typename Pos>
struct Rec {
  const uint8_t *in;
  Pos n;
  const uint64_t *S;
  const uint64_t *LB;
  Pos W;
  int levels;  // levels present in LB
  unsigned int *status;  // kQueryStatusOverflow is OR-ed here (may be null)
};

// The query a warp runs, the same for all its records.
struct Query {
  const uint8_t *ir;  // shared memory
  int ir_len;
  int num_results;
  int base;  // bitmap level of query level 0
  int nlev, marks;  // levels and open marks there are slots for
  bool ext;  // its own IR holds extension opcodes (others of the launch may, too)
};

// The reference reads file[] unguarded; well-formed JSON never leaves the
// partition.  Out-of-range reads return 0 here.
template <typename Pos>
__device__ __forceinline__ uint8_t at(const Rec<Pos> &c, Pos i) {
  return (i >= 0 && i < c.n) ? c.in[i] : uint8_t(0);
}
__device__ __forceinline__ uint8_t ir_at(const Query &q, int i) {
  return (i >= 0 && i < q.ir_len) ? q.ir[i] : uint8_t(0);
}
// Eight IR bytes from i on, as two little-endian words (0 <= i <= ir_len + 1:
// the shared copy ends in kIrPad zero bytes).
__device__ __forceinline__ uint2 ir_window(const Query &q, int i) {
  const uint32_t *w = reinterpret_cast<const uint32_t *>(q.ir) + (i >> 2);
  const uint32_t shift = uint32_t(i & 3) * 8u;
  const uint32_t a = w[0], b = w[1], c = w[2];
  return make_uint2(__funnelshift_r(a, b, shift), __funnelshift_r(b, c, shift));
}

__device__ __forceinline__ uint64_t mask_through_bit(int b) {
  return b == 63 ? ~0ull : ((1ull << (b + 1)) - 1ull);
}

// One lane.  Last set bit of `bm` in [min_index, index], -1 if there is none
// (query.cu:39-77); min_index >= 0 and index < 64 * words.
template <typename Pos>
__device__ Pos prev_bit(const uint64_t *bm, Pos min_index, Pos index) {
  if (index < min_index) return -1;
  const Pos wmin = min_index >> 6;
  uint64_t keep = mask_through_bit(int(index & 63));
  for (Pos w = index >> 6; w >= wmin; --w) {
    uint64_t cand = bm[w] & keep;
    if (w == wmin) cand &= ~0ull << (min_index & 63);
    if (cand != 0) return w * 64 + 63 - __clzll(static_cast<long long>(cand));
    keep = ~0ull;
  }
  return -1;
}

// Leveled-bitmap words of a bitmap level, or null for a level the index does
// not hold (it has no structural characters).
template <typename Pos>
__device__ __forceinline__ const uint64_t *level_words(const Rec<Pos> &c, int l) {
  return (l < 0 || l >= c.levels) ? nullptr : c.LB + uint64_t(c.W) * uint64_t(l);
}

// The structural characters of word w in [from, level_end]; words outside the
// bitmap are empty.
template <typename Pos>
__device__ __forceinline__ uint64_t struct_word(const Rec<Pos> &c, const uint64_t *lvl, Pos w,
                                                Pos from, Pos level_end) {
  if (w < 0 || w >= c.W || w > (level_end >> 6)) return 0ull;
  uint64_t cand = lvl[w];
  if (w == (from >> 6)) cand &= ~0ull << (from & 63);
  if (w == (level_end >> 6)) cand &= mask_through_bit(int(level_end & 63));
  return cand;
}

// One lane: first structural character in [line_index, level_end], level_end
// if there is none (query.cu:79-115).
template <typename Pos>
__device__ Pos next_struct_lane(const Rec<Pos> &c, Pos level_end, Pos line_index,
                                const uint64_t *lvl) {
  if (line_index >= level_end || lvl == nullptr) return level_end;
  const Pos last = level_end >> 6;
  for (Pos w = line_index >> 6; w <= last && w < c.W; ++w) {
    const uint64_t cand = struct_word(c, lvl, w, line_index, level_end);
    if (cand != 0) return w * 64 + __ffsll(static_cast<long long>(cand)) - 1;
  }
  return level_end;
}

// One lane's walk over the structural characters of a level, in order from
// `from` on: the words come two at a time with one 16-byte load where the row
// allows it, so a long gap (a string value, a skipped member) costs half the
// round trips.  The two words are taken from without a branch: lanes refill at
// different times, and each path that only some of them take costs all of
// them its instructions (5 % on small inputs against one word at a time).
template <typename Pos>
struct Walk {
  const uint64_t *lvl;
  Pos W, last;  // words of the row, last word to look at
  Pos w, wnext;
  uint64_t cand, after;  // characters left in word w, and in word w + 1
  __device__ __forceinline__ Walk(const Rec<Pos> &c, const uint64_t *row, Pos from, Pos level_end)
      : lvl(row), W(c.W), last(min(Pos(level_end >> 6), Pos(c.W - 1))), w(from >> 6),
        wnext(w), cand(0), after(0) {
    load();
    cand &= ~0ull << (from & 63);
  }
  __device__ __forceinline__ void load() {  // words wnext (and wnext + 1)
    w = wnext;
    if (w > last) return;
    const uint64_t *p = lvl + w;
    if ((reinterpret_cast<uintptr_t>(p) & 15u) == 0 && w + 1 < W) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(p);
      cand = v.x;
      after = v.y;
      wnext = w + 2;
    } else {
      cand = *p;
      wnext = w + 1;
    }
  }
  // The next character, -1 after the last one; positions beyond level_end come
  // out too, up to the end of the last words read.
  __device__ __forceinline__ Pos next() {
    while ((cand | after) == 0) {
      if (wnext > last) return -1;
      load();
    }
    const bool second = cand == 0;
    uint64_t x = second ? after : cand;
    const Pos p = (w + (second ? 1 : 0)) * 64 + __ffsll(static_cast<long long>(x)) - 1;
    x &= x - 1;
    if (second) after = x;
    else cand = x;
    return p;
  }
};

// The same search for every active record of the warp: G words (64 * G bytes)
// a round.
template <typename Pos, int G>
__device__ __forceinline__ Pos next_struct(const Rec<Pos> &c, const Group<G> &g, bool active,
                                           Pos level_end, Pos line_index, const uint64_t *lvl) {
  if constexpr (G == 1) {
    if (!active || lvl == nullptr || line_index >= level_end) return level_end;
    Walk<Pos> walk(c, lvl, line_index, level_end);
    const Pos p = walk.next();
    return p < 0 || p > level_end ? level_end : p;
  } else {
    Pos w0 = line_index >> 6, found = level_end;
    const Pos last = min(Pos(level_end >> 6), Pos(c.W - 1));
    bool need = active && lvl != nullptr && line_index < level_end && w0 <= last;
    while (__any_sync(kAll, need)) {
      const Pos w = w0 + g.lane;
      const uint64_t cand = need ? struct_word(c, lvl, w, line_index, level_end) : 0ull;
      const unsigned hit = g.ballot(cand != 0);
      const Pos p = g.shfl(Pos(w * 64 + __ffsll(static_cast<long long>(cand)) - 1),
                           __ffs(int(hit)) - 1);
      if (need) {
        if (hit != 0) found = p;
        w0 += G;
        need = hit == 0 && w0 <= last;
      }
    }
    return found;
  }
}

// Last structural character at or before line_index, 0 if there is none
// (query.cu:117-128 with level_start = 0).
template <typename Pos, int G>
__device__ __forceinline__ Pos prev_struct(const Rec<Pos> &c, const Group<G> &g, bool active,
                                           Pos line_index, const uint64_t *lvl) {
  Pos w0 = line_index >> 6, found = 0;
  bool need = active && lvl != nullptr && line_index > 0;
  while (__any_sync(kAll, need)) {
    const Pos w = w0 - g.lane;
    uint64_t cand = (need && w >= 0 && w < c.W) ? lvl[w] : 0ull;
    if (w == (line_index >> 6)) cand &= mask_through_bit(int(line_index & 63));
    const unsigned hit = g.ballot(cand != 0);
    const Pos p = g.shfl(Pos(w * 64 + 63 - __clzll(static_cast<long long>(cand))),
                         __ffs(int(hit)) - 1);
    if (need) {
      if (hit != 0) found = p;
      w0 -= G;
      need = hit == 0 && w0 >= 0;
    }
  }
  return found;
}

// The same for one array index after another: the character mostly stands in
// the first word looked at, from which every lane of the group takes it without
// a vote's round trip (element 400 from the end, 8 K records: 327 us, 287 so).
template <typename Pos, int G>
__device__ __forceinline__ Pos next_struct_near(const Rec<Pos> &c, const Group<G> &g, bool active,
                                                Pos level_end, Pos line_index,
                                                const uint64_t *lvl) {
  if constexpr (G == 1) return next_struct(c, g, active, level_end, line_index, lvl);
  uint64_t here = 0;
  if (active && lvl != nullptr && line_index < level_end)
    here = struct_word(c, lvl, Pos(line_index >> 6), line_index, level_end);
  Pos p = (line_index & ~Pos(63)) + __ffsll(static_cast<long long>(here)) - 1;
  const bool far = active && here == 0;
  if (__any_sync(kAll, far)) {
    const Pos q = next_struct(c, g, far, level_end, line_index, lvl);
    if (far) p = q;
  }
  return p;
}
template <typename Pos, int G>
__device__ __forceinline__ Pos prev_struct_near(const Rec<Pos> &c, const Group<G> &g, bool active,
                                                Pos line_index, const uint64_t *lvl) {
  if constexpr (G == 1) return prev_struct(c, g, active, line_index, lvl);
  uint64_t here = 0;
  if (active && lvl != nullptr && line_index > 0)
    here = lvl[line_index >> 6] & mask_through_bit(int(line_index & 63));
  Pos p = (line_index & ~Pos(63)) + 63 - __clzll(static_cast<long long>(here));
  const bool far = active && here == 0;
  if (__any_sync(kAll, far)) {
    const Pos q = prev_struct(c, g, far, line_index, lvl);
    if (far) p = q;
  }
  return p;
}

// One lane.  Steps forward over commas while the index is below the target and
// the next character is there (MOVE_TO_INDEX, query.cu:304-346); returns false
// at a character that is none.  The loop of all lanes takes over from where
// this ends.  (Element 700, 30 K records: 756 us, 923 with a search from the
// start of its word for every step.)
template <typename Pos>
__device__ bool step_forward(const Rec<Pos> &c, Steps<Pos> max_steps, Pos level_end,
                             const uint64_t *lvl, int32_t target, Pos &line_index, int32_t &index,
                             Steps<Pos> &steps) {
  if (lvl == nullptr || line_index >= level_end) return true;
  Walk<Pos> walk(c, lvl, Pos(line_index + 1), level_end);
  while (index < target && steps < max_steps) {
    const Pos p = walk.next();
    if (p < 0 || p > level_end) break;
    ++steps;
    line_index = p;
    ++index;
    if (at(c, p) != ',') return false;
  }
  return true;
}
// The same backward (MOVE_TO_INDEX_REVERSE, query.cu:348-392): element 400 from the end, 30 K
// records: 422 us, 538 with a search for every step.
template <typename Pos>
__device__ bool step_backward(const Rec<Pos> &c, Steps<Pos> max_steps, const uint64_t *lvl,
                              int32_t target, Pos &line_index, int32_t &index, Steps<Pos> &steps) {
  if (lvl == nullptr || line_index <= 1) return true;
  Pos w = (line_index - 1) >> 6;
  uint64_t cand = lvl[w] & mask_through_bit(int((line_index - 1) & 63));
  while (index < target && steps < max_steps) {
    while (cand == 0 && w > 0) cand = lvl[--w];
    if (cand == 0) break;
    const int b = 63 - __clzll(static_cast<long long>(cand));
    cand &= ~(1ull << b);
    ++steps;
    line_index = w * 64 + b;
    ++index;
    if (at(c, line_index) != ',' && index != target) return false;
  }
  return true;
}

// The operand at pos; `first` is its first byte, nearly always the only one.
__device__ __noinline__ int2 read_long_varint(const uint8_t *ir, int ir_len, int pos) {
  const IrOperand o = ir_varint(ir, ir_len, pos);
  return make_int2(o.value, o.next);
}
__device__ __forceinline__ int read_varint(const Query &q, int &pos, uint32_t first) {
  if (first < 0x80u) {
    ++pos;
    return int(first);
  }
  const int2 v = read_long_varint(q.ir, q.ir_len, pos);
  pos = v.y;
  return v.x;
}

// ---- Extensions of this build (the reference's compiler rejects them) ----
//
// Exact decimal comparison of two JSON numbers (no floating point): a number
// is 0.d1d2d3... x 10^E with d1 != 0, or zero; exponents saturate at
// +-10^15.  Bytes come from a getter so the same code reads the partition
// (bounds-checked) and the IR.
struct DecNum {
  bool neg, zero;
  int64_t E, nd, first, int_len, int_pos, frac_pos;
};

constexpr int64_t kExpLimit = 1000000000000000ll;

__device__ __forceinline__ bool is_digit(uint8_t c) { return c >= '0' && c <= '9'; }

template <class Get>
__device__ __forceinline__ uint8_t dec_digit(const Get &get, const DecNum &x, int64_t k) {
  return get(k < x.int_len ? x.int_pos + k : x.frac_pos + (k - x.int_len));
}

// Parses bytes [0, len) of the getter as one JSON number (RFC 8259).
template <class Get>
__device__ bool dec_parse(const Get &get, int64_t len, DecNum &o) {
  int64_t i = 0;
  o.neg = false;
  if (i < len && get(i) == '-') {
    o.neg = true;
    ++i;
  }
  if (i >= len) return false;
  o.int_pos = i;
  const uint8_t c0 = get(i);
  if (c0 == '0') {
    ++i;
  } else if (c0 >= '1' && c0 <= '9') {
    while (i < len && is_digit(get(i))) ++i;
  } else {
    return false;
  }
  o.int_len = i - o.int_pos;
  int64_t frac_len = 0;
  o.frac_pos = i;
  if (i < len && get(i) == '.') {
    ++i;
    o.frac_pos = i;
    while (i < len && is_digit(get(i))) ++i;
    frac_len = i - o.frac_pos;
    if (frac_len == 0) return false;
  }
  int64_t ex = 0;
  if (i < len && (get(i) == 'e' || get(i) == 'E')) {
    ++i;
    bool eneg = false;
    if (i < len && (get(i) == '+' || get(i) == '-')) {
      eneg = get(i) == '-';
      ++i;
    }
    const int64_t es = i;
    while (i < len && is_digit(get(i))) {
      if (ex < kExpLimit) ex = ex * 10 + (get(i) - '0');
      ++i;
    }
    if (i == es) return false;
    if (ex > kExpLimit) ex = kExpLimit;
    if (eneg) ex = -ex;
  }
  if (i != len) return false;
  const int64_t total = o.int_len + frac_len;
  int64_t z = 0;
  while (z < total && dec_digit(get, o, z) == '0') ++z;
  o.zero = z == total;
  o.first = z;
  o.nd = total - z;
  o.E = o.int_len - z + ex;
  return true;
}

template <class GetA, class GetB>
__device__ int dec_cmp(const GetA &ga, const DecNum &a, const GetB &gb, const DecNum &b) {
  const int sa = a.zero ? 0 : (a.neg ? -1 : 1);
  const int sb = b.zero ? 0 : (b.neg ? -1 : 1);
  if (sa != sb) return sa < sb ? -1 : 1;
  if (sa == 0) return 0;
  int mag = 0;
  if (a.E != b.E) {
    mag = a.E > b.E ? 1 : -1;
  } else {
    const int64_t n = a.nd > b.nd ? a.nd : b.nd;
    for (int64_t k = 0; k < n && mag == 0; ++k) {
      const uint8_t da = k < a.nd ? dec_digit(ga, a, a.first + k) : uint8_t('0');
      const uint8_t db = k < b.nd ? dec_digit(gb, b, b.first + k) : uint8_t('0');
      if (da != db) mag = da > db ? 1 : -1;
    }
  }
  return sa > 0 ? mag : -mag;
}

__device__ __forceinline__ bool cmp_holds(int op, int r) {
  switch (op) {
  case 0: return r == 0;
  case 1: return r != 0;
  case 2: return r < 0;
  case 3: return r <= 0;
  case 4: return r > 0;
  case 5: return r >= 0;
  default: return false;
  }
}

template <typename Pos>
__device__ __forceinline__ void raise_status(const Rec<Pos> &c, unsigned int bits) {
  if (c.status != nullptr) atomicOr(c.status, bits);
}

// A key to look for: where it stands in the IR, and its opening quote and
// first three bytes as one little-endian word under a mask.
struct Key {
  int pos, len;
  uint32_t head, mask;
  __device__ __forceinline__ Key(const Query &q, int key_pos, int key_len)
      : pos(key_pos), len(key_len) {
    const uint32_t first = key_pos <= q.ir_len ? ir_window(q, key_pos).x : 0u;
    mask = key_len >= 3 ? 0xFFFFFFFFu : (0x100u << (8 * key_len)) - 1u;
    head = ((first << 8) | uint32_t('"')) & mask;
  }
};

// One lane.  Does the string before the ':' at `colon` equal the key (the
// test of MOVE_TO_KEY, query.cu:254-302)?  `s_word` is the string-mask word of
// the byte before the colon.  Most keys differ in length or in their first
// bytes: the quote and three bytes are compared as one word, first as far as
// the aligned word that holds the quote goes, then with the next one.
template <typename Pos>
__device__ __forceinline__ bool key_at_colon(const Rec<Pos> &c, const Query &q, Pos line_start,
                                             Pos colon, uint64_t s_word, const Key &key) {
  const Pos before = colon - 1;
  // last in-string byte before the colon: nearly always in its own word
  const uint64_t in_string = s_word << (63 - int(before & 63));
  Pos string_end = before - __clzll(static_cast<long long>(in_string));
  if (in_string == 0 || string_end <= line_start)
    string_end = prev_bit(c.S, Pos(line_start + 1), before);
  const Pos string_start = string_end - key.len;
  if (string_start < line_start) return false;
  const uintptr_t addr = reinterpret_cast<uintptr_t>(c.in + string_start);
  const uint32_t *word = reinterpret_cast<const uint32_t *>(addr & ~uintptr_t(3));
  const uint32_t shift = uint32_t(addr & 3u) * 8u;
  uint32_t head = word[0] >> shift;
  if (((head ^ key.head) & key.mask & (0xFFFFFFFFu >> shift)) != 0) return false;
  // bytes up to the string's end only: the second word holds one of them
  if (shift != 0 && (key.mask >> (32 - shift)) != 0) head |= word[1] << (32 - shift);
  if (((head ^ key.head) & key.mask) != 0) return false;
  for (int i = 3; i < key.len; ++i)
    if (ir_at(q, key.pos + i) != c.in[string_start + i + 1]) return false;
  return true;
}

template <typename Pos>
__device__ __forceinline__ uint64_t string_word_before(const Rec<Pos> &c, Pos p) {
  return p > 0 ? c.S[(p - 1) >> 6] : 0ull;
}

// find_key (below) by one lane for its own record: one pair of characters a
// step, their bytes loaded together; several keys end in one string-mask word,
// which is kept (1 M records of 512 bytes, 24 keys each, none the one looked
// for: 256 us with the word loaded for every key, 237 so, 211 with the two-step
// comparison of key_at_colon; posts, 131 K: 88, 84 and 82).
template <typename Pos>
__device__ __forceinline__ bool find_key_lane(const Rec<Pos> &c, const Query &q, Pos line_start,
                                              Pos level_end, const uint64_t *lvl, const Key &key,
                                              Pos &line_index, Pos &next, bool &open) {
  const Pos from = line_index + 1;
  Walk<Pos> walk(c, lvl, from, level_end);
  Pos s_at = -1;
  uint64_t s_word = 0;
  for (;;) {
    const Pos p1 = walk.next();
    if (p1 < 0 || p1 > level_end) return false;
    Pos p2 = walk.next();
    if (p2 > level_end) p2 = -1;
    const uint8_t b1 = c.in[p1];
    const uint8_t b2 = p2 >= 0 ? c.in[p2] : uint8_t(0);
    if (((p1 - 1) >> 6) != s_at) {
      s_at = (p1 - 1) >> 6;
      s_word = c.S[s_at];
    }
    if (b1 != ':' || key_at_colon(c, q, line_start, p1, s_word, key)) {
      line_index = p1;
      next = p2;
      open = false;
      return true;
    }
    if (p2 < 0) {
      // the second of the pair is level_end itself
      if (at(c, level_end) == '}') open = false;
      return false;
    }
    if (b2 == '}') {
      open = false;
      return false;
    }
  }
}

// Structural characters a group looks at in one round, at most (a word has at
// most 64).
template <int G>
constexpr int kListed = G == 32 ? 256 : 64;

// One lane.  Writes the positions of a word's set bits, plus `first`.
__device__ __forceinline__ void list_bits(uint16_t *list, uint64_t word, int first) {
  for (uint32_t m = uint32_t(word); m != 0; m &= m - 1)
    *list++ = uint16_t(first + __ffs(int(m)) - 1);
  for (uint32_t m = uint32_t(word >> 32); m != 0; m &= m - 1)
    *list++ = uint16_t(first + 31 + __ffs(int(m)));
}

// The key search of MOVE_TO_KEY (query.cu:254-302) for every active record of
// the warp.  The structural characters after line_index, up to level_end, come
// in pairs: one that should be a ':' and the one after its value.  Returns
// true with line_index on the first of a pair that is not a ':' or whose key
// matches; false when the second of a pair is a '}' first (or the search would
// never end, on malformed input).  `next`: the structural character after
// line_index, -1 where the search did not come across it.
//
// A round takes up to G bitmap words of the record, one per lane; the lanes
// list the positions of their structural characters in shared memory, and
// each lane then tests one pair of the list.  All keys of 64 * G bytes cost
// one chain of dependent loads (bitmap and string-mask word, byte, quote, key
// bytes) instead of one chain each, and no lane loops over its own word while
// the others wait.
template <typename Pos, int G>
__device__ bool find_key(const Rec<Pos> &c, const Query &q, const Group<G> &g, bool active,
                         Pos line_start, Steps<Pos> max_steps, Pos level_end, const uint64_t *lvl,
                         const Key &key, Pos &line_index, Pos &next, uint16_t *list) {
  next = -1;
  bool found = false;
  // A reverse index on malformed input can leave the record: more characters
  // may then follow than the step bound allows, and they are taken one pair
  // at a time.
  bool stray = active && lvl != nullptr && line_index < line_start;
  if (__any_sync(kAll, stray)) {
    if (stray) {
      for (Steps<Pos> steps = 1; steps <= max_steps; ++steps) {
        const Pos p1 = next_struct_lane(c, level_end, Pos(line_index + 1), lvl);
        line_index = p1;
        if (at(c, p1) != ':' ||
            key_at_colon(c, q, line_start, p1, string_word_before(c, p1), key)) {
          found = true;
          break;
        }
        line_index = next_struct_lane(c, level_end, Pos(p1 + 1), lvl);
        if (at(c, line_index) == '}') break;
      }
      active = false;
    }
    __syncwarp();
  }
  const Pos from = line_index + 1;
  const Pos last = min(Pos(level_end >> 6), Pos(c.W - 1));
  int second = 0;      // 1: the next character is the second of its pair
  bool open = active;  // no end found yet
  Pos w0 = from >> 6;
  bool need = active && lvl != nullptr && from < level_end && w0 <= last;
  if constexpr (G == 1) {
    if (need)
      found = find_key_lane(c, q, line_start, level_end, lvl, key, line_index, next, open);
    need = false;
  }
  while (G > 1 && __any_sync(kAll, need)) {
    const Pos w = w0 + g.lane;
    const bool have = need && w <= last;
    uint64_t cand = have ? lvl[w] : 0ull;
    const uint64_t s_word = have ? c.S[w] : 0ull;
    if (w == (from >> 6)) cand &= ~0ull << (from & 63);
    if (w == (level_end >> 6)) cand &= mask_through_bit(int(level_end & 63));
    const int mine = __popcll(cand);
    int total;
    int at_slot = g.sum_before(mine, total);
    int words = G;
    if (__any_sync(kAll, total > kListed<G>)) {  // more than a round's: fewer words
      words = __popc(g.ballot(g.lane == 0 || at_slot + mine <= kListed<G>));
      total = g.shfl(at_slot + mine, words - 1);
    }
    if (g.lane < words) list_bits(list + at_slot, cand, g.lane * 64);
    __syncwarp();
    const Pos base = w0 * 64;
    const uint8_t *text = c.in + base;
    bool look = need;
    int e = 2 * g.lane - second;  // this lane's pair: list[e], list[e + 1]
    while (__any_sync(kAll, look)) {
      const bool has1 = look && e >= 0 && e < total;
      const bool has2 = look && e + 1 < total;
      const int o1 = has1 ? int(list[e]) : 0;
      const int o2 = has2 ? int(list[e + 1]) : 0;
      const uint8_t b1 = has1 ? text[o1] : uint8_t(0);
      const uint8_t b2 = has2 ? text[o2] : uint8_t(0);
      uint64_t s = __shfl_sync(kAll, (unsigned long long)s_word, (o1 - 1) >> 6, G);
      if (has1 && o1 == 0) s = string_word_before(c, base);
      // 1: the search ends at the first of the pair, 2: there is no such key
      unsigned event = b2 == '}' ? 2u : 0u;
      if (has1 &&
          (b1 != ':' || key_at_colon(c, q, line_start, Pos(base + o1), s, key)))
        event = 1u;
      __syncwarp();
      const unsigned hit = g.ballot(event != 0);
      // event, and both positions within the round (o2 = 0: not seen)
      const unsigned what =
          unsigned(g.shfl(int32_t(event | unsigned(o1) << 2 | unsigned(o2) << 16),
                          __ffs(int(hit)) - 1));
      e += 2 * G;
      if (look) {
        look = hit == 0 && e - 2 * g.lane < total;
        if (hit != 0) {
          open = false;
          found = (what & 3u) == 1u;
          line_index = base + Pos((what >> 2) & 0x3FFFu);
          if ((what >> 16) != 0) next = base + Pos(what >> 16);
        }
      }
    }
    if (need) {
      second = (second + total) & 1;
      w0 += words;
      need = open && w0 <= last;
    }
  }
  // No more structural characters: every further step lands on level_end.
  if (open && active) {
    found = !(second != 0 && at(c, level_end) == '}') &&
            (at(c, level_end) != ':' ||
             key_at_colon(c, q, line_start, level_end, string_word_before(c, level_end), key));
    line_index = level_end;
  }
  __syncwarp();
  return found;
}

// One lane.  Stores the member whose ':' is at p, `level` or a level above it.
template <typename Pos, typename OutT>
__device__ __forceinline__ void store_member(const Rec<Pos> &c, const Query &q, Pos level_end,
                                             int level, Pos p, int slot, OutT *out) {
  if (slot >= q.num_results) {
    raise_status(c, kQueryStatusOverflow);
    return;
  }
  int l = level;
  while (l < c.levels && (level_words(c, l) == nullptr ||
                          ((level_words(c, l)[p >> 6] >> (p & 63)) & 1ull) == 0ull))
    ++l;
  const Pos vend = next_struct_lane(c, level_end, Pos(p + 1), level_words(c, l));
  Pos vs = p + 1;
  while (at(c, vs) == ' ' && vs < vend) ++vs;
  Pos ve = vend;
  while (ve > vs && at(c, ve - 1) == ' ') --ve;
  out[2 * slot] = OutT(vs);
  out[2 * slot + 1] = OutT(ve);
}

// The structural characters of word w at any level from `lowest` up, in
// [line_index, level_end).
template <typename Pos>
__device__ __forceinline__ uint64_t any_level_word(const Rec<Pos> &c, int lowest, Pos w,
                                                   Pos line_index, Pos level_end) {
  uint64_t cand = 0;
  const uint64_t *row = c.LB + uint64_t(c.W) * uint64_t(lowest) + w;
#pragma unroll 4
  for (int l = lowest; l < c.levels; ++l, row += c.W) cand |= *row;
  if (w == (line_index >> 6)) cand &= ~0ull << (line_index & 63);
  if (w == (level_end >> 6)) cand &= (1ull << (level_end & 63)) - 1ull;
  return cand;
}

// "..name": every member named key inside (line_index, level_end), at any level
// from `level` up, in document order (by the position of its ':'), for every
// active record of the warp.  The lanes of a group list the structural
// characters of all those levels in their words, test one each for the key, and
// collect the few that match; those are then resolved one per lane.  (Each lane
// testing the characters of its own word left two thirds of the lanes idle:
// 41 K posts 231 us, so 200.)  One lane tests them one after another.  Returns
// `stored` plus the record's matches.
template <typename Pos, typename OutT, int G>
__device__ int descend(const Rec<Pos> &c, const Query &q, const Group<G> &g, bool active,
                       Pos line_start, Pos line_index, Pos level_end, int level, const Key &key,
                       int stored, OutT *out, uint16_t *list, Pos *matches) {
  const int lowest = level > 0 ? level : 0;
  const Pos last = min(Pos((level_end - 1) >> 6), Pos(c.W - 1));
  Pos w0 = line_index >> 6;
  if constexpr (G == 1) {
    if (active) {
      for (Pos w = max(w0, Pos(0)); w <= last; ++w) {
        uint64_t cand = any_level_word(c, lowest, w, line_index, level_end);
        const uint64_t s_word = cand != 0 ? c.S[w] : 0ull;
        for (; cand != 0; cand &= cand - 1) {
          const Pos p = w * 64 + __ffsll(static_cast<long long>(cand)) - 1;
          if (c.in[p] == ':' &&
              key_at_colon(c, q, line_start, p, (p & 63) != 0 ? s_word : string_word_before(c, p),
                           key))
            store_member(c, q, level_end, level, p, stored++, out);
        }
      }
    }
    __syncwarp();
    return stored;
  } else {
    int waiting = 0;  // collected matches
    auto resolve = [&] {
      __syncwarp();
      if (g.lane < waiting)
        store_member(c, q, level_end, level, matches[g.lane], stored + g.lane, out);
      stored += waiting;
      waiting = 0;
      __syncwarp();
    };
    bool need = active && w0 <= last;
    while (__any_sync(kAll, need)) {
      const Pos w = w0 + g.lane;
      const bool have = need && w >= 0 && w <= last;
      const uint64_t cand = have ? any_level_word(c, lowest, w, line_index, level_end) : 0ull;
      const uint64_t s_word = have ? c.S[w] : 0ull;
      const int mine = __popcll(cand);
      int total;
      const int at_slot = g.sum_before(mine, total);
      int words = G;
      if (__any_sync(kAll, total > kListed<G>)) {
        words = __popc(g.ballot(g.lane == 0 || at_slot + mine <= kListed<G>));
        total = g.shfl(at_slot + mine, words - 1);
      }
      if (g.lane < words) list_bits(list + at_slot, cand, g.lane * 64);
      __syncwarp();
      const Pos base = w0 * 64;
      const uint8_t *text = c.in + base;
      for (int e0 = 0; __any_sync(kAll, e0 < total); e0 += G) {
        const bool has = e0 + g.lane < total;
        const int o = has ? int(list[e0 + g.lane]) : 0;
        const uint8_t b = has ? text[o] : uint8_t(0);
        uint64_t s = __shfl_sync(kAll, (unsigned long long)s_word, (o - 1) >> 6, G);
        if (has && o == 0) s = string_word_before(c, base);
        const bool match = b == ':' && key_at_colon(c, q, line_start, Pos(base + o), s, key);
        __syncwarp();
        const unsigned hits = g.ballot(match);
        const int found = __popc(hits);
        if (!__any_sync(kAll, found != 0)) continue;
        if (__any_sync(kAll, waiting + found > G)) resolve();
        if (match) matches[waiting + __popc(hits & ((1u << g.lane) - 1u))] = base + o;
        waiting += found;
      }
      if (need) {
        w0 += words;
        need = w0 <= last;
      }
      __syncwarp();
    }
    resolve();
    return stored;
  }
}

// One lane.  Commas among the structural characters after line_index, up to
// the first that is none or `limit` of them.
template <typename Pos>
__device__ int count_commas(const Rec<Pos> &c, Steps<Pos> max_steps, Pos level_end,
                            const uint64_t *lvl, Pos line_index, int limit) {
  int commas = 0;
  Pos p = line_index;
  for (Steps<Pos> steps = 1; commas < limit && steps <= max_steps; ++steps) {
    p = next_struct_lane(c, level_end, Pos(p + 1), lvl);
    if (at(c, p) != ',') break;
    ++commas;
  }
  return commas;
}

// Opcodes an instance of the kernels runs: the reference's; with the numeric
// filters and the element checks of "[*]" and the open slices; with "..name"
// too.
enum : int { kReference = 0, kExtensions = 1, kDescends = 2 };

// Runs the query over the warp's records (one per group of G lanes; `alive`:
// the group has one).  `ends` and `marks` are the thread's slots of per-level
// and per-mark positions in shared memory ([level * stride]).
template <typename Pos, typename OutT, int kOps, int G>
__device__ void run_records(const Rec<Pos> &c, const Query &q, const Group<G> &g, bool alive,
                            Pos line_start, Pos line_end, OutT *out, Pos *ends, Pos *marks,
                            int stride, uint16_t *list, Pos *matches) {
  constexpr bool kExt = kOps >= kExtensions;
  // every lane keeps its own copy of its record's state, so no lane reads
  // what another wrote, except the result slots
  if (alive)
    for (int i = g.lane; i < 2 * q.num_results; i += G) out[i] = OutT(-1);
  alive = alive && line_start >= 0 && line_start < c.n && line_end >= 0;
  if (line_end >= c.n) line_end = c.n - 1;
  // the record's braces: last '}' back from line_end, first '{' from
  // line_start, G bytes a round
  if constexpr (G == 1) {
    if (alive) {
      while (line_end > line_start && at(c, line_end) != '}') --line_end;
      while (line_start < line_end && at(c, line_start) != '{') ++line_start;
    }
    __syncwarp();
  } else {
    for (bool need = alive; __any_sync(kAll, need);) {
      const Pos p = line_end - g.lane;
      const unsigned hit = g.ballot(need && (p <= line_start || at(c, p) == '}'));
      if (need) {
        line_end -= hit != 0 ? __ffs(int(hit)) - 1 : G;
        need = hit == 0;
      }
    }
    for (bool need = alive; __any_sync(kAll, need);) {
      const bool past = line_end - line_start <= g.lane;
      const unsigned hit = g.ballot(need && (past || at(c, Pos(line_start + g.lane)) == '{'));
      if (need) {
        line_start += hit != 0 ? __ffs(int(hit)) - 1 : G;
        need = hit == 0;
      }
    }
  }
  alive = alive && line_start < line_end;

  Pos line_index = line_start;
  int level = 0;
  int qp = 0;
  // Step bound of one search loop.  On well-formed JSON every step lands on a
  // new structural character of the record, so the bound is never reached;
  // on malformed input the reference's loops can revisit the same character
  // forever, and the record is abandoned instead.
  // (Unsigned: a record of 2^31 - 1 bytes has as many steps and two more.)
  const Steps<Pos> max_steps = Steps<Pos>(line_end - line_start) + 2u;
  ends[0] = line_end;
  for (int i = 1; i < q.nlev; ++i) ends[i * stride] = -1;
  // A record still alive after an index step stands on that index, so the
  // current index of a level is the same for all of them: lane l holds level
  // l's.  Marked levels are the same for all as well (a byte each).
  int32_t level_index = -1;
  uint64_t mark_levels[2] = {0, 0};
  int marked = -1;
  int stored = 0;
  // structural character after the key that the last opcode found, on level
  // next_level (-1: the last opcode was no key search)
  Pos next = -1;
  int next_level = -1;

#define LEVEL_OK(l) ((l) >= 0 && (l) < q.nlev)
  for (;;) {
    if (!__any_sync(kAll, alive)) return;
    const uint2 window = ir_window(q, qp);
    const uint32_t op = window.x & 0xFFu, operand = (window.x >> 8) & 0xFFu;
    ++qp;
    if (op != OP_MOVE_DOWN) next_level = -1;
    switch (op) {
    case OP_END:
      return;
    case OP_STORE_RESULT: {
      if (!LEVEL_OK(level)) return;
      if (alive) {
        const Pos lend = ends[level * stride];
        Pos end_str = lend;
        while (at(c, line_index) == ' ' && line_index < lend) ++line_index;
        while (end_str > line_index && at(c, end_str - 1) == ' ') --end_str;
        if (stored < q.num_results) {
          // the lanes that cleared the slot
          if ((2 * stored) % G == g.lane) out[2 * stored] = OutT(line_index);
          if ((2 * stored + 1) % G == g.lane) out[2 * stored + 1] = OutT(end_str);
        } else if constexpr (kExt) {
          // (reference syntax may be given fewer slots than it stores)
          if (q.ext && g.lane == 0) raise_status(c, kQueryStatusOverflow);
        }
      }
      ++stored;
      break;
    }
    case OP_MOVE_UP:
      if (!LEVEL_OK(level)) return;
      line_index = ends[level * stride];
      ends[level * stride] = -1;
      --level;
      break;
    case OP_MOVE_DOWN: {
      ++level;
      if (!LEVEL_OK(level) || level < 1) return;
      const bool fresh = alive && ends[level * stride] == -1;
      // right after a key search the end of the value is often known already
      const bool known = next_level == level - 1 && next > line_index;
      // (an empty object's key search ends one beyond its '}', and nothing
      // follows that, nor might line_index + 1 be a position)
      const Pos lend = ends[(level - 1) * stride];
      Pos p = next_struct(c, g, fresh && !known && line_index < lend, lend,
                          Pos(Steps<Pos>(line_index) + 1u), level_words(c, q.base + level - 1));
      if (known) p = next;
      if (fresh) {
        ends[level * stride] = p;
        while (at(c, line_index) == ' ') ++line_index;
      }
      break;
    }
    case OP_MOVE_TO_KEY: {
      const int key_len = read_varint(q, qp, operand);
      const int key_pos = qp;
      if (key_len < 0 || !LEVEL_OK(level)) return;
      qp = ir_skip(q.ir_len, qp, key_len);
      alive = alive && at(c, line_index) == '{';
      alive = find_key(c, q, g, alive, line_start, max_steps, ends[level * stride],
                       level_words(c, q.base + level), Key(q, key_pos, key_len), line_index, next,
                       list);
      ++line_index;
      next_level = level;
      break;
    }
    case OP_MOVE_TO_INDEX: {
      const int target = read_varint(q, qp, operand);
      if (!LEVEL_OK(level)) return;
      const int32_t current = __shfl_sync(kAll, level_index, level);
      const uint8_t ch = alive ? at(c, line_index) : uint8_t(0);
      alive = alive && (ch == '[' || ch == ',' || ch == ']');
      int32_t ci = ch == '[' ? 0 : current + 1;
      const Pos lend = ends[level * stride];
      const uint64_t *lvl = level_words(c, q.base + level);
      Steps<Pos> steps = 0;
      bool walked = false;  // this lane stands on the target already
      if constexpr (G == 1) {  // (a single step is the loop's: eight slots, 372 -> 368 us)
        if (alive && target > 1 && ci < target - 1) {
          alive = step_forward(c, max_steps, lend, lvl, target, line_index, ci, steps);
          walked = ci == target;
          if (walked) alive = alive && steps < max_steps;
        }
        __syncwarp();
      }
      for (bool run = alive && !walked; __any_sync(kAll, run);) {
        bool forward = false, back = false;
        if (run) {
          alive = ++steps <= max_steps;
          forward = alive && ci < target;
          back = alive && ci > target;
        }
        if (__any_sync(kAll, forward)) {
          const Pos p = next_struct_near(c, g, forward, lend, Pos(line_index + 1), lvl);
          if (forward) {
            line_index = p;
            ++ci;
            alive = at(c, p) == ',';
          }
        }
        if (__any_sync(kAll, back)) {
          const Pos p = prev_struct_near(c, g, back, Pos(line_index - 1), lvl);
          if (back) {
            line_index = p;
            --ci;
          }
        }
        run = alive && (forward || back);
      }
      if (int(threadIdx.x & 31u) == level) level_index = target;
      alive = alive && at(c, line_index) != ']';
      ++line_index;
      break;
    }
    case OP_MOVE_TO_INDEX_REVERSE: {
      const int target = read_varint(q, qp, operand);
      if (!LEVEL_OK(level)) return;
      const int32_t current = __shfl_sync(kAll, level_index, level);
      const Pos lend = ends[level * stride];
      line_index = lend - 1;
      if (alive)
        while (at(c, line_index) == ' ') --line_index;
      const uint8_t ch = alive ? at(c, line_index) : uint8_t(0);
      alive = alive && (ch == ']' || ch == ',' || ch == '[');
      int32_t ci = ch == ']' ? 0 : current + 1;
      const uint64_t *lvl = level_words(c, q.base + level);
      Steps<Pos> steps = 0;
      bool walked = false;  // this lane stands on the target already
      if constexpr (G == 1) {  // (a single step is the loop's: eight slots, 372 -> 368 us)
        if (alive && target > 1 && ci < target - 1) {
          alive = step_backward(c, max_steps, lvl, target, line_index, ci, steps);
          walked = ci == target;
          if (walked) alive = alive && steps < max_steps;
        }
        __syncwarp();
      }
      for (bool run = alive && !walked; __any_sync(kAll, run);) {
        bool forward = false, back = false;
        if (run) {
          alive = ++steps <= max_steps;
          back = alive && ci < target;
          forward = alive && ci > target;
        }
        if (__any_sync(kAll, back)) {
          const Pos p = prev_struct_near(c, g, back, Pos(line_index - 1), lvl);
          if (back) {
            line_index = p;
            alive = at(c, p) == ',' || ci + 1 == target;
            ++ci;
          }
        }
        if (__any_sync(kAll, forward)) {
          const Pos p = next_struct_near(c, g, forward, lend, Pos(line_index + 1), lvl);
          if (forward) {
            line_index = p;
            --ci;
          }
        }
        run = alive && (forward || back);
      }
      if (int(threadIdx.x & 31u) == level) level_index = target;
      ++line_index;
      break;
    }
    case OP_MARK_POSITION:
      if (marked + 1 >= q.marks) return;
      ++marked;
      marks[marked * stride] = line_index;
      mark_levels[marked >> 3] &= ~(0xFFull << (8 * (marked & 7)));
      mark_levels[marked >> 3] |= uint64_t(uint8_t(level)) << (8 * (marked & 7));
      break;
    case OP_RESET_POSITION:
      if (marked < 0) return;
      line_index = marks[marked * stride];
      level = int(int8_t(uint8_t(mark_levels[marked >> 3] >> (8 * (marked & 7)))));
      --marked;
      for (int i = level + 1; i < q.nlev; ++i) {
        if (i < 0) continue;
        if (ends[i * stride] == -1) break;
        ends[i * stride] = -1;
      }
      break;
    case OP_EXPRESSION_STRING_EQUALS: {
      const int key_len = read_varint(q, qp, operand);
      const int key_pos = qp;
      if (key_len < 0 || !LEVEL_OK(level)) return;
      qp = ir_skip(q.ir_len, qp, key_len);
      if (alive) {
        const Pos lend = ends[level * stride];
        while (at(c, line_index) == ' ' && line_index < lend) ++line_index;
        Pos string_end = lend - 1;
        while (line_index < string_end && at(c, string_end) == ' ') --string_end;
        alive = string_end - line_index + 1 == key_len;
        for (int i = 0; alive && i < key_len; ++i)
          alive = ir_at(q, key_pos + i) == at(c, Pos(line_index + i));
      }
      break;
    }
    case OP_NUMBER_COMPARE: {
      if constexpr (!kExt) return;
      const int cmp = int(operand);
      ++qp;
      const int lit_len = read_varint(q, qp, (window.x >> 16) & 0xFFu);
      const int lit_pos = qp;
      if (lit_len < 0 || lit_len > q.ir_len - lit_pos || !LEVEL_OK(level)) return;
      qp += lit_len;
      if (alive) {
        const Pos lend = ends[level * stride];
        while (at(c, line_index) == ' ' && line_index < lend) ++line_index;
        Pos value_end = lend - 1;
        while (line_index < value_end && at(c, value_end) == ' ') --value_end;
        alive = line_index >= 0 && value_end < c.n && value_end >= line_index;
        if (alive) {
          const Pos v0 = line_index;
          auto gv = [&](int64_t i) { return at(c, Pos(v0 + i)); };
          auto gl = [&](int64_t i) { return ir_at(q, int(lit_pos + i)); };
          DecNum v, lit;
          alive = dec_parse(gv, int64_t(value_end - line_index) + 1, v) &&
                  dec_parse(gl, int64_t(lit_len), lit) &&
                  cmp_holds(cmp, dec_cmp(gv, v, gl, lit));
        }
      }
      break;
    }
    case OP_DESCEND_KEY: {
      if constexpr (kOps < kDescends) {
        return;
      } else {
        const int key_len = read_varint(q, qp, operand);
        const int key_pos = qp;
        if (key_len < 0 || !LEVEL_OK(level)) return;
        qp = ir_skip(q.ir_len, qp, key_len);
        stored = descend(c, q, g, alive, line_start, line_index, ends[level * stride],
                         q.base + level, Key(q, key_pos, key_len), stored, out, list, matches);
        break;
      }
    }
    case OP_EXPECT_AT_MOST: {
      if constexpr (!kExt) return;
      const int limit = read_varint(q, qp, operand);
      if (limit < 0 || !LEVEL_OK(level)) return;
      if (limit == 0) break;
      // K commas at this level before the closing bracket: K+1 elements
      if (alive && g.lane == 0 && at(c, line_index) == '[' &&
          count_commas(c, max_steps, ends[level * stride], level_words(c, q.base + level),
                       line_index, limit) >= limit)
        raise_status(c, kQueryStatusOverflow);
      break;
    }
    case OP_EXPECT_FOLLOWING: {
      if constexpr (!kExt) return;
      const int need = read_varint(q, qp, operand);
      if (need < 0 || !LEVEL_OK(level)) return;
      // The element must exist (an empty array has no element 0) and be
      // followed by `need` commas at this level before the closing bracket;
      // otherwise it is among the last `need` (and so is every later one):
      // the record is done.
      if (alive) {
        const Pos lend = ends[level * stride];
        Pos p = line_index;
        while (p < lend && at(c, p) == ' ') ++p;
        alive = at(c, p) != ']' &&
                count_commas(c, max_steps, lend, level_words(c, q.base + level),
                             Pos(line_index - 1), need) >= need;
      }
      break;
    }
    default:
      break;
    }
    __syncwarp();
    if (qp > q.ir_len + 1) return;
  }
#undef LEVEL_OK
}

// kOps: the opcodes of the IR of the launch's queries.
// kBlocks: 256-thread blocks per SM that the registers are held to.
template <typename Pos, typename OutT, int kOps, int G, int kBlocks>
__global__ void __launch_bounds__(256, kBlocks)
    query_kernel(const __grid_constant__ QueryLaunch q, const __grid_constant__ IrBlob ir,
                 int nlev, int max_marks) {
  __shared__ __align__(16) uint8_t s_ir[kMaxQueryIrBytes + kIrPad];
  __shared__ uint16_t s_list[G > 1 ? 256 / G : 1][kListed<G>];
  __shared__ Pos s_match[kOps == kDescends && G > 1 ? 256 / G : 1][G];
  extern __shared__ __align__(8) uint8_t s_state[];  // Pos[nlev + marks][bdim]
  const QueryOne &one = q.queries[blockIdx.y];
  for (int i = threadIdx.x; i < one.ir_len + kIrPad; i += blockDim.x)
    s_ir[i] = i < one.ir_len ? ir.bytes[one.ir_off + i] : uint8_t(0);
  __syncthreads();
  const Group<G> g;
  const Rec<Pos> c{q.in, Pos(q.n), q.S, q.LB, Pos(q.W), q.num_levels, q.status};
  const Query query{s_ir, one.ir_len, one.num_results, one.base_level, nlev, max_marks, one.ext};
  OutT *const out = static_cast<OutT *>(one.out);
  Pos *ends = reinterpret_cast<Pos *>(s_state) + threadIdx.x;
  Pos *marks = ends + nlev * blockDim.x;
  const int64_t warps = int64_t(blockDim.x / 32u) * gridDim.x;
  const int64_t warp = int64_t(blockIdx.x) * (blockDim.x / 32u) + threadIdx.x / 32u;
  for (int64_t base = warp * (32 / G); base < q.num_lines; base += warps * (32 / G)) {
    const int64_t r = base + g.shift / G;
    const bool alive = r < q.num_lines;
    const int64_t start = alive ? q.NL[r] : 0;
    const int64_t end = alive && r + 1 < q.num_lines ? q.NL[r + 1] : q.n - 1;
    run_records<Pos, OutT, kOps, G>(c, query, g, alive, Pos(start), Pos(end),
                                    out + r * int64_t(one.num_results) * 2, ends, marks,
                                    int(blockDim.x), s_list[G > 1 ? threadIdx.x / G : 0],
                                    s_match[kOps == kDescends && G > 1 ? threadIdx.x / G : 0]);
    __syncwarp();
  }
}

// File of record r (the same for the whole warp): the last whose first record
// is not beyond it.  32 probes a round.
__device__ uint32_t file_of_record(const BatchQueryLaunch &q, uint64_t r) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lo = 0, hi = q.num_files;  // file_info[lo].rec_off <= r
  while (hi - lo > 1) {
    const uint32_t probe = lo + 1u + uint32_t(uint64_t(hi - lo - 1u) * lane / 32u);
    const int k = __popc(__ballot_sync(
        kAll, q.file_info[uint64_t(probe) * kFileInfoWords + kFiRecOff] <= r));
    const uint32_t below = __shfl_sync(kAll, probe, k > 0 ? k - 1 : 0);
    const uint32_t above = __shfl_sync(kAll, probe, k < 32 ? k : 31);
    if (k > 0) lo = below;
    if (k < 32) hi = above;
  }
  return lo;
}

__device__ __forceinline__ uint32_t group_of(const BatchQueryLaunch &q, const uint64_t *row) {
  return row[kFiQuery] < uint64_t(q.num_groups) ? uint32_t(row[kFiQuery]) : 0u;
}

// kPart: the launch runs the records of some groups' files only (group_mask).
template <int kOps, int G, int kBlocks, bool kPart>
__global__ void __launch_bounds__(256, kBlocks)
    batch_query_kernel(const BatchQueryLaunch q, const __grid_constant__ IrBlob ir, int nlev,
                       int max_marks) {
  // every group's IR starts on a word and ends in kIrPad zero bytes
  __shared__ __align__(16) uint8_t s_ir[kMaxQueryIrBytes + kMaxBatchGroups * (kIrPad + 4)];
  __shared__ int s_ir_off[kMaxBatchGroups];
  extern __shared__ __align__(8) uint8_t s_state[];  // int32[nlev + marks][bdim]
  for (int k = 0, off = 0; k < q.num_groups; ++k) {
    const int len = q.groups[k].ir_len;
    for (int i = threadIdx.x; i < len + kIrPad; i += blockDim.x)
      s_ir[off + i] = i < len ? ir.bytes[q.groups[k].ir_off + i] : uint8_t(0);
    if (threadIdx.x == 0) s_ir_off[k] = off;
    off += (len + kIrPad + 3) & ~3;
  }
  __syncthreads();
  __shared__ uint16_t s_list[G > 1 ? 256 / G : 1][kListed<G>];
  __shared__ int32_t s_match[kOps == kDescends && G > 1 ? 256 / G : 1][G];
  const Group<G> g;
  int32_t *ends = reinterpret_cast<int32_t *>(s_state) + threadIdx.x;
  int32_t *marks = ends + nlev * blockDim.x;
  constexpr uint32_t kRecords = 32 / G;  // a warp runs at once
  const uint64_t records = q.totals[kTotRecords];
  // Every warp starts with its own run of records and takes further runs from
  // a counter, so a warp whose records were quick takes more; without a
  // counter it strides.  A run is at most 32 records, less where the launch
  // has warps for a finer split.
  const uint64_t warps = uint64_t(blockDim.x / 32u) * gridDim.x;
  const uint64_t share = records / (warps * 4u) / kRecords * kRecords;
  const uint32_t chunk = uint32_t(share < kRecords ? kRecords : (share > 32u ? 32u : share));
  uint64_t base = (uint64_t(threadIdx.x / 32u) * gridDim.x + blockIdx.x) * chunk;
  while (base < records) {
    uint32_t f = file_of_record(q, base);
    for (uint32_t k = 0; k < chunk && base + k < records; k += kRecords) {
      if constexpr (kPart) {  // to the next record of the launch's groups, if the run has one
        const uint64_t end = base + chunk < records ? base + chunk : records;
        uint64_t at = base + k;
        for (f = __shfl_sync(kAll, f, 0); at < end; ++f) {
          const uint64_t *row = q.file_info + uint64_t(f) * kFileInfoWords;
          const uint64_t next = row[kFiRecOff] + row[kFiLines];
          if (at >= next) continue;
          if ((q.group_mask >> group_of(q, row)) & 1u) break;
          at = next;
        }
        if (at >= end) break;
        k = uint32_t(at - base);
      }
      const uint64_t r = base + k + uint32_t(g.shift / G);
      bool pending = r < records;
      if constexpr (kPart) pending = pending && r < base + chunk;
      uint64_t rec_off = 0, lines = 0;
      if (pending) {
        for (;; ++f) {  // the warp's later records may be in later files
          rec_off = q.file_info[uint64_t(f) * kFileInfoWords + kFiRecOff];
          lines = q.file_info[uint64_t(f) * kFileInfoWords + kFiLines];
          if (r < rec_off + lines) break;
        }
      }
      const uint64_t *row = q.file_info + uint64_t(f) * kFileInfoWords;
      const IndexFile F = q.files[f];
      const uint32_t qid = group_of(q, row);
      if constexpr (kPart) pending = pending && ((q.group_mask >> qid) & 1u) != 0;
      const uint64_t i = r - rec_off;
      const int64_t *nl = q.NL + row[kFiNlOff];
      // batch files are below 2 GiB (int32 results): 32-bit positions
      const bool text = pending && F.n != 0;
      const int32_t start = text ? int32_t(nl[i]) : -1;
      const int32_t end = text && i + 1 < lines ? int32_t(nl[i + 1]) : int32_t(F.n) - 1;
      const Rec<int32_t> c{q.in + F.in_off, int32_t(F.n), q.S + F.s_off, q.LB + F.lb_off,
                           int32_t((F.n + 63u) / 64u), F.levels,
                           q.file_status ? q.file_status + f : q.status};
      // one pass per query among the warp's records (usually one file, one query)
      for (;;) {
        const unsigned left = __ballot_sync(kAll, pending);
        if (left == 0) break;
        const uint32_t now = __shfl_sync(kAll, qid, __ffs(int(left)) - 1);
        const bool mine = pending && qid == now;
        const BatchQueryGroup grp = q.groups[now];
        const Query query{s_ir + s_ir_off[now], grp.ir_len, grp.num_results, grp.base_level, nlev,
                          max_marks, grp.ext};
        run_records<int32_t, int32_t, kOps, G>(
            c, query, g, mine, start, end,
            q.out + row[kFiOutOff] + i * uint64_t(grp.num_results) * 2u, ends, marks,
            int(blockDim.x), s_list[G > 1 ? threadIdx.x / G : 0],
            s_match[kOps == kDescends && G > 1 ? threadIdx.x / G : 0]);
        __syncwarp();
        pending = pending && !mine;
      }
    }
    if (q.record_counter != nullptr) {
      unsigned long long next = 0;
      if ((threadIdx.x & 31u) == 0) next = atomicAdd(q.record_counter, (unsigned long long)chunk);
      base = warps * chunk + __shfl_sync(kAll, next, 0);
    } else {
      base += warps * chunk;
    }
  }
}

}  // namespace

namespace {

uint64_t resident_threads() {
  static int sms_per_device[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148u * 1024u;
  if (sms_per_device[dev] == 0) {
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        sms <= 0)
      sms = 148;
    sms_per_device[dev] = sms;
  }
  return uint64_t(sms_per_device[dev]) * 1024u;
}

// Lanes per record.  More lanes shorten a record's chain of dependent loads
// and instructions but execute more instructions per record in total (a
// round of the group's search costs about the same for 8 lanes as for 32).
// The launch takes the most lanes with which all records are resident at once
// (four 256-thread blocks per SM), and one lane beyond.  Measured (us, one / 8
// / 16 / 32 lanes, one thread per record before this split in brackets) for
// $.user.lang on posts: 437 records 38 / 20.5 / 14 / 11 (53), 3.5 K 40 / 22.6 /
// 16.4 / 12.9 (55), 7 K 39.4 / 23.1 / 17.4 / 20.6 (56), 14 K 41 / 24.6 / 26 / 33
// (55), 28 K 50 / 44 / 48 / 66 (67), 56 K 67 / 75 / 90 / 125 (85); for
// eight-slot arrays 14 K records 90 / 83 / 127 / 163 (110), 28 K 115 / 165 / 218
// / 293 (140).  Where one lane begins to win depends on the IR, at which the
// rule does not look: its line (19 K records) lies between the short IR's, which
// loses 6 us at 28 K by it, and the eight-slot one's, which gains 50 there.
// Records of one bitmap word on average skip 16 and 8 lanes: there is nothing to
// share (15 K records of 32 bytes with a numeric filter: 13 us, 16.6 with 8).
//
// "..name" reads every level's words of the whole record, which only a wide
// group reads in whole sectors: 41 K posts of 2,400 bytes 897 us with one lane,
// 293 with 8, 231 with 32 (200 with the search of descend).  Shorter records
// leave its lanes idle (us, 32 / 8 / one lane, one thread per record before this
// split in brackets): 2 M of 8 bytes 2,061 / 516 / 89 (92), of 128 bytes 2,455 /
// 667 / 237 (249); 300 K of 512 bytes, all alike, 419 / 138 / 95 (112), 256 K of
// 422 bytes, mixed, 632 / 485 / 589 (700); 15 K of 1,024 bytes 26 / 15 / 30 (40),
// 60 K 84 / 41 / 49 (59).  From 2 KiB on mixed records, as posts are, win more
// by 32 lanes (240 K of 2.4 KB 746 / 860 / 2,997 (2,967)) than records all alike
// lose (200 K 476 (434)).
int lanes_per_record(uint64_t records, uint64_t bytes, bool descends) {
  if (records == 0) return descends ? 32 : 1;
  const uint64_t threads = resident_threads();
  const uint64_t mean = bytes / records;
  if (records * 32u <= threads) return 32;
  if (descends) {
    if (mean <= 1024u) return records * 8u <= threads ? 8 : 1;
    return mean <= 2048u ? 8 : 32;
  }
  if (mean <= 64u) return 1;
  for (int g : {16, 8})
    if (records * uint64_t(g) <= threads) return g;
  return 1;
}

// Do queries with "..name" go in a launch of their own?  They make the launch a
// warp per record for all its queries, which costs the others several times
// their instructions where one lane each would do (2.3 M records of which one
// small file asks "..id": query stage 5,696 us together, 1,318 apart).  Up to
// there a launch of each after the other takes longer (1.5 K records: 35 and 54
// us; 14 K runs in a host call: 290 and 327).
bool descending_apart(uint64_t records, uint64_t bytes) {
  return lanes_per_record(records, bytes, false) == 1;
}

// What the queries of a launch need together.
struct QueryNeeds : IrNeeds {
  void add(const IrNeeds &one) {
    levels = std::max(levels, one.levels);
    marks = std::max(marks, one.marks);
    ext = ext || one.ext;
    descends = descends || one.descends;
  }
};

// Dynamic shared memory of a block: a position per thread, level and mark.  Up
// to 32 KiB fit beside a kernel's own arrays (10 KiB at most) in the 48 KiB a
// launch may take unasked: all of 32-bit positions (256 threads, 16 levels, 16
// marks), 64-bit ones up to 16 levels and marks together.
template <typename Pos, typename Kernel>
cudaError_t state_bytes(Kernel kernel, const QueryNeeds &needs, int block, size_t &bytes) {
  bytes = size_t(needs.levels + needs.marks) * size_t(block) * sizeof(Pos);
  if (bytes <= (32u << 10)) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(2 * kMaxQueryLevels * 256 * sizeof(Pos)));
}

// "..name" runs with 32, 8 or 1 lanes (lanes_per_record), the last without a
// choice of blocks per SM.
template <int G, int kBlocks>
constexpr bool descending_instance() {
  return G == 32 || G == 8 || (G == 1 && kBlocks <= 4);
}

template <int G, int kBlocks, bool kPart = false>
cudaError_t batch_query_start(const BatchQueryLaunch &q, const IrBlob &ir, const QueryNeeds &needs,
                              int grid, int block, cudaStream_t stream) {
  // A plain launch: blocks that start beside the indexer's last CTAs keep the
  // SM split for those (200 KB of shared memory, little L1) for as long as they
  // run (1,500 MiB of files: 1,371 us a replay instead of 1,213).
  auto kernel = needs.ext ? batch_query_kernel<kExtensions, G, kBlocks, kPart>
                          : batch_query_kernel<kReference, G, kBlocks, kPart>;
  if constexpr (descending_instance<G, kBlocks>())
    if (needs.descends) kernel = batch_query_kernel<kDescends, G, kBlocks, kPart>;
  size_t smem = 0;
  const cudaError_t e = state_bytes<int32_t>(kernel, needs, block, smem);
  if (e != cudaSuccess) return e;
  kernel<<<grid, block, smem, stream>>>(q, ir, needs.levels, needs.marks);
  return cudaGetLastError();
}

template <typename Pos, typename OutT, int G, int kBlocks>
cudaError_t query_start(const QueryLaunch &q, const IrBlob &ir, const QueryNeeds &needs, int block,
                        cudaStream_t stream) {
  const int64_t per_block = block / G;
  const dim3 grid(
      unsigned(std::min<int64_t>((q.num_lines + per_block - 1) / per_block, 0x7FFFFFFF)),
      unsigned(q.num_queries));
  auto kernel = needs.ext ? query_kernel<Pos, OutT, kExtensions, G, kBlocks>
                          : query_kernel<Pos, OutT, kReference, G, kBlocks>;
  if constexpr (descending_instance<G, kBlocks>())
    if (needs.descends) kernel = query_kernel<Pos, OutT, kDescends, G, kBlocks>;
  size_t smem = 0;
  const cudaError_t e = state_bytes<Pos>(kernel, needs, block, smem);
  if (e != cudaSuccess) return e;
  kernel<<<grid, block, smem, stream>>>(q, ir, needs.levels, needs.marks);
  return cudaGetLastError();
}

// Blocks per SM of the one-lane kernel.  Its blocks start together and take
// about as long as each other, so a launch runs in waves, and a wave takes time
// about in proportion to the blocks of it per SM from four on: the fewest waves
// times blocks win, fewer blocks where two are equal.  153 K array elements:
// 87, 71 and 78 us with four, five and six; 208 K: 111, 124 and 102; 236 K:
// 113, 128 and 160; 349 K: 165, 145 and 182.  (Full waves of $.user.lang on
// posts take 76, 98 and 126 us, a little more than 4 : 5 : 6.  By those weights
// 606 to 682 K records would take four blocks instead of six, which array
// elements want, 265 us for 290, and posts do not, 366 for 338.)  Many waves
// overlap, and from twenty blocks per SM on five are the better of four and
// five: 1 M records of 512 bytes 221 us, 229 with four; 3 M of 32 bytes 113 and
// 120; 850 K posts 416 and 429, array elements 321 and 318.
int blocks_per_sm(uint64_t records) {
  const uint64_t per_block = resident_threads() / 4u;  // one block on every SM
  if (records > 20u * per_block) return 5;
  int best = 4;
  uint64_t best_cost = ~uint64_t(0);
  for (int b : {4, 5, 6}) {
    const uint64_t wave = per_block * uint64_t(b);
    const uint64_t cost = (records + wave - 1) / wave * uint64_t(b);
    if (cost < best_cost) {
      best = b;
      best_cost = cost;
    }
  }
  return best;
}

template <typename OutT>
cudaError_t query_start_narrow(const QueryLaunch &q, const IrBlob &ir, const QueryNeeds &needs,
                               int lanes, uint64_t runs, int block, cudaStream_t stream) {
  if (lanes == 32) return query_start<int32_t, OutT, 32, 4>(q, ir, needs, block, stream);
  if (lanes == 16) return query_start<int32_t, OutT, 16, 4>(q, ir, needs, block, stream);
  if (lanes == 8) return query_start<int32_t, OutT, 8, 4>(q, ir, needs, block, stream);
  switch (needs.descends ? 4 : blocks_per_sm(runs)) {
  case 5: return query_start<int32_t, OutT, 1, 5>(q, ir, needs, block, stream);
  case 6: return query_start<int32_t, OutT, 1, 6>(q, ir, needs, block, stream);
  default: return query_start<int32_t, OutT, 1, 4>(q, ir, needs, block, stream);
  }
}

// Lanes per record, blocks and blocks per SM of a batch's query launch that may
// take up to `grid` blocks.
struct BatchShape {
  int lanes, grid;
  bool five = false;
};
BatchShape batch_shape(const BatchQueryLaunch &q, const QueryNeeds &needs, int grid, int block) {
  BatchShape s{lanes_per_record(q.expected_records, q.expected_bytes, needs.descends), grid};
  if (q.expected_records > 0) {
    const uint64_t blocks = (q.expected_records * uint64_t(s.lanes) + uint64_t(block) - 1) / block;
    s.grid = int(std::min<uint64_t>(uint64_t(grid), blocks));
  }
  if (s.lanes > 1) return s;
  // Five blocks per SM where they hold all the records and four do not
  // (157 K records: 125 us, 160 with four; 184 K: 134 and 170).  More records
  // share out through the counter, and four are better (192 K: 155 us, 167
  // with six; 216 K: 162 and 179; 588 K: 316 and 327 with five; 3.8 M: 1.62 ms
  // and 1.94 with six).
  const uint64_t one_each = resident_threads() / 4u;  // records of a block on every SM
  s.five = !needs.descends && q.expected_records > 4u * one_each && q.expected_records <= 5u * one_each;
  // Runs taken from the counter want no blocks beyond the resident ones: a
  // later block's first run is its own and waits for it (192 K records: 169 us
  // with eight blocks per SM in the grid, 155 with four; 274 K: 193 and 181).
  if (q.record_counter != nullptr)
    s.grid = int(std::min<uint64_t>(uint64_t(s.grid),
                                    one_each * (s.five ? 5u : 4u) / uint64_t(block)));
  return s;
}

template <bool kPart>
cudaError_t batch_query_part(const BatchQueryLaunch &q, const IrBlob &ir, const QueryNeeds &needs,
                             int grid, int block, cudaStream_t stream) {
  const BatchShape s = batch_shape(q, needs, grid, block);
  if (q.record_counter != nullptr && !q.counter_cleared) {
    const cudaError_t e = cudaMemsetAsync(q.record_counter, 0, sizeof(unsigned long long), stream);
    if (e != cudaSuccess) return e;
  }
  if (s.lanes == 32) return batch_query_start<32, 4, kPart>(q, ir, needs, s.grid, block, stream);
  if constexpr (!kPart)  // (a part has 32 lanes, 8 or one: descending_apart)
    if (s.lanes == 16) return batch_query_start<16, 4>(q, ir, needs, s.grid, block, stream);
  if (s.lanes == 8) return batch_query_start<8, 4, kPart>(q, ir, needs, s.grid, block, stream);
  return s.five ? batch_query_start<1, 5, kPart>(q, ir, needs, s.grid, block, stream)
                : batch_query_start<1, 4, kPart>(q, ir, needs, s.grid, block, stream);
}

cudaError_t query_part(const QueryLaunch &q, const IrBlob &ir, const QueryNeeds &needs,
                       cudaStream_t stream) {
  constexpr int kBlock = 256;
  // the queries of a launch are resident side by side
  const uint64_t runs = uint64_t(q.num_lines) * uint64_t(q.num_queries);
  const int lanes = lanes_per_record(runs, uint64_t(q.n) * uint64_t(q.num_queries), needs.descends);
  // partitions below 2 GiB take 32-bit positions whatever the result width
  // (700 MiB of posts, eight int64 slots: 427 us, 513 us before)
  if (!q.wide) return query_start_narrow<int32_t>(q, ir, needs, lanes, runs, kBlock, stream);
  if (q.n <= 0x7FFFFFFF)
    return query_start_narrow<int64_t>(q, ir, needs, lanes, runs, kBlock, stream);
  if (lanes == 32 || (lanes > 1 && needs.descends))
    return query_start<int64_t, int64_t, 32, 3>(q, ir, needs, kBlock, stream);
  // (four blocks per SM, 60 registers: 2.3 GiB of posts, one path 515 us, 588 with
  // the 69 registers of three; eight slots 1,229 and 1,330)
  return query_start<int64_t, int64_t, 1, 4>(q, ir, needs, kBlock, stream);
}

// A batch's groups by launch: those that do not descend and those that do where
// they go apart (`split`), else all of them in the first.  Marks the groups with
// extension opcodes.
struct BatchParts {
  QueryNeeds needs[2];
  uint32_t masks[2] = {0, 0};
  bool split;
  BatchParts(BatchQueryLaunch &q, const IrBlob &ir) {
    for (int g = 0; g < q.num_groups; ++g) {
      const IrNeeds one = ir_needs(ir.bytes + q.groups[g].ir_off, q.groups[g].ir_len);
      q.groups[g].ext = one.ext;
      if (((q.used_groups >> g) & 1u) == 0) continue;
      needs[one.descends].add(one);
      masks[one.descends] |= 1u << g;
    }
    split = masks[0] != 0 && masks[1] != 0 && descending_apart(q.expected_records, q.expected_bytes);
    if (!split) needs[0].add(needs[1]);
  }
};

}  // namespace

int batch_query_grid(BatchQueryLaunch q, const IrBlob &ir, int grid, int block) {
  const BatchParts parts(q, ir);
  return batch_shape(q, parts.needs[0], grid, block).grid;
}

cudaError_t batch_query_launch(BatchQueryLaunch q, const IrBlob &ir, int grid, int block,
                               cudaStream_t stream) {
  const BatchParts parts(q, ir);
  if (!parts.split) return batch_query_part<false>(q, ir, parts.needs[0], grid, block, stream);
  for (int d = 0; d < 2; ++d) {
    q.group_mask = parts.masks[d];
    const cudaError_t e = batch_query_part<true>(q, ir, parts.needs[d], grid, block, stream);
    if (e != cudaSuccess) return e;
    q.counter_cleared = false;
  }
  return cudaSuccess;
}

cudaError_t query_launch(QueryLaunch q, const IrBlob &ir, cudaStream_t stream) {
  if (q.num_lines <= 0 || q.n <= 0 || q.num_queries <= 0) return cudaSuccess;
  QueryLaunch parts[2] = {q, q};  // the queries that do not descend, those that do
  QueryNeeds needs[2];
  parts[0].num_queries = parts[1].num_queries = 0;
  for (int i = 0; i < q.num_queries; ++i) {
    const IrNeeds one = ir_needs(ir.bytes + q.queries[i].ir_off, q.queries[i].ir_len);
    q.queries[i].ext = one.ext;
    QueryLaunch &part = parts[one.descends];
    part.queries[part.num_queries++] = q.queries[i];
    needs[one.descends].add(one);
  }
  const bool split = parts[0].num_queries > 0 && parts[1].num_queries > 0 &&
                     descending_apart(uint64_t(q.num_lines) * uint64_t(q.num_queries),
                                      uint64_t(q.n) * uint64_t(q.num_queries));
  if (!split) {
    needs[0].add(needs[1]);
    return query_part(q, ir, needs[0], stream);
  }
  const cudaError_t e = query_part(parts[0], ir, needs[0], stream);
  return e != cudaSuccess ? e : query_part(parts[1], ir, needs[1], stream);
}

}  // namespace gpjb
