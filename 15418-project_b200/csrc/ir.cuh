// The byte IR of a compiled query: opcodes, operands, and what a launch has to
// provide for it.  IR comes from callers and may be anything: no operand moves
// the reader outside [0, len + 2].
//
// Host and device: the CPU unit test walks malformed IR with these functions.
#pragma once

#include <cstdint>

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace gpjb {

constexpr int kMaxQueryLevels = 16;     // orig.hpp:10 kMaxQueryLevels
constexpr int kMaxQueryIrBytes = 4096;  // orig.hpp:11 kMaxQueryIrBytes

enum : uint8_t {
  OP_END = 0x00,
  OP_STORE_RESULT = 0x01,
  OP_MOVE_UP = 0x02,
  OP_MOVE_DOWN = 0x03,
  OP_MOVE_TO_KEY = 0x04,
  OP_MOVE_TO_INDEX = 0x05,
  OP_MOVE_TO_INDEX_REVERSE = 0x06,
  OP_MARK_POSITION = 0x07,
  OP_RESET_POSITION = 0x08,
  OP_EXPRESSION_STRING_EQUALS = 0x09,
  // Extensions of this build (never emitted for the reference's syntax):
  OP_NUMBER_COMPARE = 0x0A,  // numeric filter: cmp byte, varint length, number text
  OP_DESCEND_KEY = 0x0B,     // "..name" as the last step: varint length, key bytes
  OP_EXPECT_AT_MOST = 0x0C,  // "[*]" element-count check: varint limit
  OP_EXPECT_FOLLOWING = 0x0D,  // "[a:-b]": varint count of elements that must follow
};

// An operand and the position after it.
struct IrOperand {
  int value, next;
};

// query.cu:130-140 of the reference (LEB128).  Unsigned arithmetic
// reinterpreted as int, as the reference's int result wraps; an operand longer
// than five bytes (never produced by the compiler) reads as -1.  Bytes past the
// end read as zero.
__host__ __device__ __forceinline__ IrOperand ir_varint(const uint8_t *ir, int len, int pos) {
  uint32_t value = 0, byte = 0;
  int shift = 0;
  for (;;) {
    byte = pos < len ? ir[pos] : 0u;
    ++pos;
    if ((byte & 0x80u) == 0) break;
    value |= (byte & 0x7Fu) << shift;
    shift += 7;
    if (shift > 28) return IrOperand{-1, pos};
  }
  return IrOperand{int(value | (byte << shift)), pos};
}

// The position after `bytes` (>= 0) bytes of text at `pos`.  Text that does not
// end inside the IR ends the program (len + 2 is where the interpreter stops):
// a length is a caller's number of up to 2^31 - 1, and pos + bytes may not be
// an int.
__host__ __device__ __forceinline__ int ir_skip(int len, int pos, int bytes) {
  return bytes <= len - pos ? pos + bytes : len + 2;
}

// What running an IR takes.
struct IrNeeds {
  int levels = 1;         // query levels it can reach, at most kMaxQueryLevels
  int marks = 0;          // marks open at once, at most kMaxQueryLevels
  bool ext = false;       // it comes across an extension opcode
  bool descends = false;  // it comes across DESCEND_KEY
};

// Follows the IR as the interpreter does (it has no jumps; reset returns to the
// level of the last mark), up to where the interpreter leaves every record.
inline IrNeeds ir_needs(const uint8_t *ir, int len) {
  IrNeeds needs;
  int level = 0, open = 0;
  int marked[kMaxQueryLevels] = {};
  for (int p = 0; p <= len + 1;) {
    const uint8_t op = p < len ? ir[p] : uint8_t(OP_END);
    ++p;
    switch (op) {
    case OP_END: return needs;
    case OP_MOVE_UP: --level; break;
    case OP_MOVE_DOWN:
      ++level;
      if (level + 1 > needs.levels && level < kMaxQueryLevels) needs.levels = level + 1;
      break;
    case OP_MARK_POSITION:
      if (open == kMaxQueryLevels) return needs;
      marked[open++] = level;
      if (open > needs.marks) needs.marks = open;
      break;
    case OP_RESET_POSITION:
      if (open == 0) return needs;
      level = marked[--open];
      break;
    case OP_NUMBER_COMPARE: ++p; [[fallthrough]];  // comparator
    case OP_DESCEND_KEY:
    case OP_MOVE_TO_KEY:
    case OP_EXPRESSION_STRING_EQUALS: {
      if (op == OP_NUMBER_COMPARE || op == OP_DESCEND_KEY) needs.ext = true;
      if (op == OP_DESCEND_KEY) needs.descends = true;
      const IrOperand text = ir_varint(ir, len, p);
      if (text.value < 0) return needs;
      p = ir_skip(len, text.next, text.value);
      break;
    }
    case OP_EXPECT_AT_MOST:
    case OP_EXPECT_FOLLOWING: needs.ext = true; [[fallthrough]];
    case OP_MOVE_TO_INDEX:
    case OP_MOVE_TO_INDEX_REVERSE: p = ir_varint(ir, len, p).next; break;
    default: break;
    }
  }
  return needs;
}

}  // namespace gpjb
