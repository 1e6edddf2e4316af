// Host check of what a launch provides for an IR: open marks, not mark bytes;
// opcodes, not operand bytes.
#include "ir.cuh"

#include <cstdio>
#include <string>

using namespace gpjb;

static int bad = 0;
static void check(const std::string &ir, int levels, int marks, bool ext, bool descends) {
  const IrNeeds n = ir_needs(reinterpret_cast<const uint8_t *>(ir.data()), int(ir.size()));
  if (n.levels != levels || n.marks != marks || n.ext != ext || n.descends != descends) {
    std::printf("levels %d marks %d ext %d descends %d:", n.levels, n.marks, n.ext, n.descends);
    for (char c : ir) std::printf(" %02x", uint8_t(c));
    std::printf("\n");
    ++bad;
  }
}
static std::string times(const std::string &s, int n) {
  std::string out;
  while (n-- > 0) out += s;
  return out;
}
static std::string key(const std::string &name) {
  return std::string("\x04") + char(name.size()) + name + "\x03";
}

int main() {
  const std::string mark = "\x07", reset = "\x08", up = "\x02", store = "\x01", end(1, '\0');
  check("", 1, 0, false, false);
  check(store + end, 1, 0, false, false);
  // seven-letter keys, element 7, a key of mark bytes
  check(times(key("country") + "\x05\x07\x03" + up + store + up, 16) + end, 3, 0, false, false);
  check(key(std::string(11, '\x07')) + store + end, 2, 0, false, false);
  // one filter after another, and nested ones
  check(times(mark + key("user") + "\x09\x03\"a\"" + reset, 9) + store + end, 2, 1, false, false);
  check(mark + key("a") + mark + key("b") + mark + reset + reset + mark + reset + reset, 3, 3,
        false, false);
  check(times(mark, 16) + times(reset, 16) + times(key("a"), 15), 16, 16, false, false);
  // a 17th open mark and a reset without one end the record
  check(times(mark, 17) + key("a") + "\x0B\x01k", 1, 16, false, false);
  check(reset + key("a"), 1, 0, false, false);
  // the marked level comes back
  check(key("a") + mark + key("b") + key("c") + reset + key("d"), 4, 1, false, false);
  check(times("\x03", 20), 16, 0, false, false);
  // extensions, and operands that only look like them
  check("\x0B\x01k" + end, 1, 0, true, true);
  check(key("screen_name") + store + end, 2, 0, false, false);
  check(std::string("\x0A\x04\x02") + "10" + store + end, 1, 0, true, false);
  check("\x0C\x0B" + store + end, 1, 0, true, false);
  check("\x05\x0B" + store + end, 1, 0, false, false);
  check(end + "\x0B\x01k", 1, 0, false, false);
  // text that leaves the IR ends it, wherever the length points
  check("\x04\xff\xff\xff\xff\x07\x0B\x01k", 1, 0, false, false);
  check("\x04\xff\xff\xff\xff\x0f\x0B\x01k", 1, 0, false, false);
  check("\x04\x05k", 1, 0, false, false);
  check("\x0B\xff\xff\xff\xff\x07" + mark, 1, 0, true, true);
  // an over-long operand takes five bytes
  check("\x05\xff\xff\xff\xff\xff" + mark + "\x03" + end, 2, 1, false, false);
  std::printf("%s %d\n", bad ? "MISMATCH" : "OK", bad);
  return bad ? 1 : 0;
}
