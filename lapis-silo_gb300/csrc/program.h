// Device filter program: the postorder lowering of a compiled operator tree.
//
// Every filter operator of the reference is chunk-local (AND/OR/ANDNOT per roaring key, complement
// within each chunk's rows, NOf per row; reference: src/rhydb/query_engine/copy_on_write_bitmap.cpp:145-298,
// src/rhydb/storage/column/row_layout.cpp:18-23, src/rhydb/query_engine/filter/operators/threshold.cpp:64-138),
// so a program is evaluated independently for every tile of rows: one CTA runs the instruction
// list over a stack of dense bit tiles held in shared memory.
#pragma once

#include <cstdint>

namespace rhygpu {

enum OpCode : uint8_t {
   OP_PUSH_EMPTY = 0,
   OP_PUSH_FULL = 1,     // all rows of the tile that exist in the chunk
   OP_PUSH_SCAN = 2,     // col = sequence column, a = position, b = symbol mask: OR of the containers
                         // (c = ordinal among the program's PUSH_SCAN / PUSH_DICT leaves, from 1)
   OP_PUSH_NULLS = 3,    // col = sequence column: rows whose sequence is null
   OP_PUSH_DICT = 4,     // col = dictionary column, a = value id: inverted-index rows (c as for PUSH_SCAN)
   OP_PUSH_COVERED = 5,  // col = sequence column, a = position, flags&1: not covered instead of covered
                         // (c = ordinal among the program's PUSH_COVERED leaves, from 1)
   OP_PUSH_DATE = 6,     // col = date column; rows with lo <= date <= hi (a = lo, b = hi as int32),
                         // flags&2 = inverted (outside the range), flags&1 = null dates match
   OP_AND = 7,           // pop y, pop x, push x & y
   OP_ANDNOT = 8,        // pop y, pop x, push x & ~y
   OP_OR = 9,            // pop y, pop x, push x | y
   OP_NOT = 10,          // pop x, push valid & ~x
   OP_THR_BEGIN = 11,    // a = planes: push `a` zero counter planes
   OP_THR_ADD = 12,      // a = planes, flags&1 = negated child: pop x, count += x (or ~x). The top plane is
                         // sticky: once a count reaches 2^(a-1) it stays above n, whatever is added
   OP_THR_END = 13,      // a = planes, b = n, flags&1 = exactly: pop planes, push count >= n (== n)
   OP_JZ = 14,           // a = target: jump if the top tile is all zero
   OP_JFULL = 15,        // a = target: jump if the top tile holds every valid row
   OP_GROUP = 17,        // the next a instructions are row-list leaves applied together (see group_leaves):
                         // b = first container leaf | their number << 16, c = first coverage leaf |
                         // their number << 16 (the container leaves come first); flags: GroupFlags
   OP_PUSH_AUX = 16,     // a = index of a row set computed (a MutationProfile) or uploaded (a caller's row
                         // set, flags & AUX_LITERAL) before the program runs
};

constexpr uint16_t AUX_LITERAL = 1;  // PUSH_AUX of a caller's row set

constexpr bool is_leaf(uint8_t op) { return op <= OP_PUSH_DATE || op == OP_PUSH_AUX; }

// A leaf whose value the next instruction consumes at once is one instruction: bits 8..10 of the
// leaf's flags name the operator applied to the top of the stack (AND, ANDNOT, OR) or to the counter
// planes on top of it (THR_ADD, with the leaf's complement for FUSE_THR_ADD_NOT), bits 11..15 the
// number of planes. See fuse_leaves.
enum FuseOp : uint32_t {
   FUSE_NONE = 0,
   FUSE_AND = 1,
   FUSE_ANDNOT = 2,
   FUSE_OR = 3,
   FUSE_THR_ADD = 4,
   FUSE_THR_ADD_NOT = 5,
};
constexpr uint32_t leaf_fused(uint16_t flags) { return (flags >> 8) & 7u; }
constexpr uint32_t leaf_planes(uint16_t flags) { return (flags >> 11) & 31u; }
constexpr uint16_t fuse_flags(FuseOp op, uint32_t planes) { return static_cast<uint16_t>((op << 8) | (planes << 11)); }

// Comparators of the date predicate (reference: src/rhydb/query_engine/filter/operators/selection.h:40-72).
enum CmpCode : uint32_t { CMP_EQ = 0, CMP_NE = 1, CMP_LT = 2, CMP_LE = 3, CMP_GT = 4, CMP_GE = 5 };

struct alignas(16) Instr {  // the kernels read it as one 16-byte load
   uint8_t op;
   uint8_t col;
   uint16_t flags;
   uint32_t a;
   uint32_t b;
   uint32_t c;
};
static_assert(sizeof(Instr) == 16 && alignof(Instr) == 16, "instruction layout");

// How a leaf's rows reach their target: set in the top tile, removed from it, or counted in the planes.
enum RowOp : int { A_OR = 0, A_ANDNOT = 1, A_ADD = 2 };
// OP_GROUP flags: bits 0..1 the RowOp, bit 2: a new tile first (empty for A_OR, every valid row for
// A_ANDNOT), bits 11..15 the planes of A_ADD (as in a leaf's flags).
constexpr uint16_t GROUP_PUSH = 4;

// A MutationProfile that differs from the local reference at up to this many positions, held by few enough rows
// (profile_by_differences), is counted from the differences (profile_delta_kernel), any other from the whole
// row index (see profile.cu): 50 us for
// 1,344 positions at 2M rows, against 133 us for the row index; a row's sum in the kernel has 16 bits.
constexpr uint32_t PROFILE_DELTA_MAX = 2048;

constexpr uint32_t MAX_PROGRAM = 4096;   // instructions per program
// A single query's program of up to this many instructions travels in the filter kernel's parameters (2 KiB
// of their 4), a longer one is copied to device memory first: the copy is an operation of its own on the
// stream, which the kernel waits for. Generated trees have 5 to 60 instructions.
constexpr uint32_t INLINE_CODE = 128;
struct InlineCode {
   Instr code[INLINE_CODE];
};
constexpr uint32_t MAX_THR_PLANES = 16;  // counter planes (NOf up to 65,534 children)

}  // namespace rhygpu
