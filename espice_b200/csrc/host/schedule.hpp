// Compiles the lead lane's pivot tape (a factored SparseLu) into the warp
// programs the kernels run. One value space per lane: the tape values (U
// entries, the diagonal, L entries, one discard slot, as the reference's
// refactor tape lays them out, sparse_lu.zig buildTape :1041-1082) followed
// by the n entries of the permuted right-hand side y.
//
// Program A is the refactor with the forward substitution through unit L
// merged in (a column's forward updates run as soon as its L entries and
// y entry are final, overlapping later columns' refactor); program B is the
// back substitution through U. Each is list-scheduled into rows of tasks
// (common.h: up to three updates of one value and its division), one task
// per thread of the lane's warp or CTA; and, for the interpreted lane LU,
// into rows of 32 single ops, each row of divisions only or
// multiply-subtracts only.
#pragma once

#include <cstdint>
#include <vector>

#include "sparse.hpp"

namespace esl {

struct Op {
  uint32_t w0, w1;  // see common.h OpKind
};

// The same with full 32-bit value indices (any tape size): w0 = dst | (kind
// << 28), then the two sources.
struct Op4 {
  uint32_t w0, a, b, pad;
};

struct Programs {
  uint32_t nu = 0, nl = 0, ntv = 0, n = 0;
  uint32_t nv = 0;                 // value space: ntv + n (y) + 0.0, 1.0, sink
  std::vector<uint32_t> amap;      // pattern slot -> tape value
  std::vector<uint32_t> fill;      // tape values no pattern slot writes
  std::vector<Op> a_ops;           // rows x 32: refactor + forward solve (pack_op_rows)
  std::vector<Op> b_ops;           // rows x 32: back solve
  std::vector<Op> a_list, b_list;  // the ops in the replay's sequential order (column by column), 16-bit indices
  std::vector<Op4> a_seq, b_seq;   // the same, with 32-bit indices (any value space)
  uint32_t a_rows = 0, b_rows = 0, a_levels = 0, b_levels = 0;  // levels: longest chain
  uint32_t a_nops = 0, b_nops = 0; // real ops (no padding)
  std::vector<uint8_t> l_scaled;   // per L entry: its column took the row-scaled pivot
  uint64_t flops = 0;              // refactor multiply-subtracts (the census F)
  bool has_void = false;
};

// A block-lane program as each warp's stream of chunks, a chunk the 32 tasks
// (common.h) its lanes run between two barriers: warp w's chunks are
// off[w] .. off[w + 1] (in chunks of 32 * task_words words), the last
// kTaskRing of them only read ahead.
constexpr uint32_t kTaskWarps = 16;  // a block lane's CTA has at most this many
struct TaskStream {
  std::vector<uint32_t> words;
  uint32_t off[kTaskWarps + 1] = {};
  uint32_t rows = 0;  // steps between barriers (a warp's or the CTA's)
};

// The programs of a block lane: A (refactor + forward solve), B (back
// solve) and F, the forward substitution alone (the mixed form's refinement
// solves on finished factors).
struct BlockPrograms {
  TaskStream a, b, f;
  uint32_t a_levels = 0;
  bool compact = true;
};

// Every op reads final operands and every value's updates keep their
// sequential order, so the programs are bitwise the column replay and the
// sparse triangular solves.
Programs compile_tape(const SparseLu& lu);
// The rows of 32 single ops (a_ops, b_ops and their counts; value spaces
// below 65,536), which the interpreted lane LU and esl_compile_tape take.
void pack_op_rows(Programs& P);

// The warp lanes' programs A and B as one warp's compact task stream each
// (value spaces below 65,536).
void compile_warp(const Programs& P, TaskStream& a, TaskStream& b);

// The block lanes' task streams for a CTA of `warps` warps (at most kTaskWarps).
BlockPrograms compile_block(const Programs& P, uint32_t warps);

constexpr uint32_t kRow = 32;

}  // namespace esl
