// Host check of the IR reader: whatever the bytes, an operand's position stays
// within [0, len + 2], and text that ends inside the IR is passed exactly.
#include "ir.cuh"

#include <climits>
#include <cstdio>
#include <initializer_list>

using namespace gpjb;

static unsigned long long state = 88172645463325252ull;
static uint64_t rnd() {
  state ^= state << 13;
  state ^= state >> 7;
  state ^= state << 17;
  return state;
}

int main() {
  int bad = 0;
  // lengths up to the largest int at every place of a small IR
  for (int len = 0; len <= 12; ++len) {
    for (int pos = 0; pos <= len + 6; ++pos) {
      for (int n : {0, 1, 2, len, len + 1, 4096, INT_MAX - 7, INT_MAX - 1, INT_MAX}) {
        const long long end = (long long)pos + n;
        const int got = ir_skip(len, pos, n);
        if (got != (end <= len ? int(end) : len + 2)) ++bad;
      }
    }
  }
  // five bytes decode to any int, a fifth with the high bit to -1
  const uint8_t huge[] = {0xFF, 0xFF, 0xFF, 0xFF, 0x07}, over[] = {0xFF, 0xFF, 0xFF, 0xFF, 0xFF, 1};
  if (ir_varint(huge, 5, 0).value != INT_MAX || ir_varint(huge, 5, 0).next != 5) ++bad;
  if (ir_varint(over, 6, 0).value != -1 || ir_varint(over, 6, 0).next != 5) ++bad;
  if (ir_varint(huge, 3, 0).next != 4) ++bad;  // cut off: reads as zero bytes from there on
  for (int t = 0; t < 200000; ++t) {
    uint8_t ir[24];
    const int len = int(rnd() % 24);
    for (int i = 0; i < len; ++i) ir[i] = rnd() % 3 ? 0xFF : uint8_t(rnd());
    for (int pos = 0; pos <= len + 1;) {
      const IrOperand o = ir_varint(ir, len, pos);
      if (o.next <= pos || o.next > pos + 5) ++bad;
      const int next = o.value < 0 ? o.next : ir_skip(len, o.next, o.value);
      if (next <= pos || next > len + 6) ++bad;
      pos = next;
    }
  }
  std::printf("%s %d\n", bad ? "MISMATCH" : "OK", bad);
  return bad ? 1 : 0;
}
