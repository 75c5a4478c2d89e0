// See schedule.hpp.
#include "schedule.hpp"

#include <algorithm>

#include "../common.h"

namespace esl {

namespace {

struct SeqOp {
  uint32_t kind, dst, a, b;  // a, b: value sources (kNone when unused)
};

Op encode(uint32_t kind, uint32_t dst, uint32_t a, uint32_t b) {
  Op o;
  o.w0 = dst | (kind << 28);
  o.w1 = (a == kNone ? 0 : a) | ((b == kNone ? 0 : b) << 16);
  return o;
}

bool is_div(uint32_t kind) { return kind == kOpDivGrowth || kind == kOpDivScaled || kind == kOpDivY; }

// Dependences: an op follows the last write of each value it reads, the
// last write of its destination (a value's updates keep their sequential
// order, so every sum rounds as in the column replay), and every read of its
// destination since that write (no value is overwritten before it is read).
// The ops are then list-scheduled into rows of kRow ops (one per thread),
// each row one class, the divisions or the multiply-subtracts (the kernel's
// two warp-uniform paths; the checks inside a path are per op): row by row,
// the class of the ready op with the longest path to the end of the program,
// then up to kRow ready ops of that class, longest paths first. An op's
// successors become ready only for a later row. `n_levels` is the longest
// dependence chain, the least number of rows any packing can have.
// Padding ops write the sink slot (space - 1) from the constants 1.0
// (space - 2) and 0.0 (space - 3): 1.0 / 1.0 in a division row, a
// zero-skipped 1.0 * 0.0 in a multiply-subtract row.
template <class Enc, class OpT>
void pack_rows(const std::vector<SeqOp>& seq, uint32_t space, uint32_t width, Enc enc, const OpT& pad_div,
               const OpT& pad_flop, std::vector<OpT>& rows, uint32_t& n_rows, uint32_t& n_levels) {
  const size_t n = seq.size();
  std::vector<int32_t> last_write(space, -1);
  std::vector<std::vector<uint32_t>> readers(space);
  std::vector<uint32_t> succ_ptr(n + 1, 0), n_pred(n, 0);
  std::vector<std::pair<uint32_t, uint32_t>> edges;  // (pred, succ)
  std::vector<uint32_t> preds;
  for (size_t i = 0; i < n; ++i) {
    const SeqOp& s = seq[i];
    preds.clear();
    for (uint32_t src : {s.a, s.b})
      if (src != kNone && last_write[src] >= 0) preds.push_back(uint32_t(last_write[src]));
    if (last_write[s.dst] >= 0) preds.push_back(uint32_t(last_write[s.dst]));
    for (uint32_t r : readers[s.dst])
      if (r != i) preds.push_back(r);
    std::sort(preds.begin(), preds.end());
    preds.erase(std::unique(preds.begin(), preds.end()), preds.end());
    for (uint32_t p : preds) edges.push_back({p, uint32_t(i)});
    n_pred[i] = uint32_t(preds.size());
    last_write[s.dst] = int32_t(i);
    readers[s.dst].clear();
    for (uint32_t src : {s.a, s.b})
      if (src != kNone) readers[src].push_back(uint32_t(i));
  }
  for (const auto& e : edges) ++succ_ptr[e.first + 1];
  for (size_t i = 0; i < n; ++i) succ_ptr[i + 1] += succ_ptr[i];
  std::vector<uint32_t> succ(edges.size()), fill(succ_ptr.begin(), succ_ptr.end() - 1);
  for (const auto& e : edges) succ[fill[e.first]++] = e.second;
  // height: ops on the longest path from this op to the end, inclusive
  std::vector<uint32_t> height(n, 1);
  uint32_t top = 0;
  for (size_t i = n; i-- > 0;) {
    for (uint32_t e = succ_ptr[i]; e < succ_ptr[i + 1]; ++e) height[i] = std::max(height[i], height[succ[e]] + 1);
    top = std::max(top, height[i]);
  }
  n_levels = top;
  // ready queues per class, longest path first, then sequence order
  auto later = [&](uint32_t x, uint32_t y) { return height[x] != height[y] ? height[x] < height[y] : x > y; };
  std::vector<uint32_t> ready[2];
  for (size_t i = 0; i < n; ++i)
    if (n_pred[i] == 0) ready[is_div(seq[i].kind)].push_back(uint32_t(i));
  for (auto& q : ready) std::make_heap(q.begin(), q.end(), later);
  rows.clear();
  n_rows = 0;
  std::vector<uint32_t> row;
  while (!ready[0].empty() || !ready[1].empty()) {
    int c;
    if (ready[0].empty()) c = 1;
    else if (ready[1].empty()) c = 0;
    else c = later(ready[0].front(), ready[1].front()) ? 1 : 0;
    auto& q = ready[c];
    row.clear();
    while (!q.empty() && row.size() < width) {
      std::pop_heap(q.begin(), q.end(), later);
      row.push_back(q.back());
      q.pop_back();
    }
    for (uint32_t t = 0; t < width; ++t) {
      if (t < row.size()) rows.push_back(enc(seq[row[t]]));
      else rows.push_back(c ? pad_div : pad_flop);
    }
    ++n_rows;
    for (uint32_t i : row)
      for (uint32_t e = succ_ptr[i]; e < succ_ptr[i + 1]; ++e) {
        const uint32_t j = succ[e];
        if (--n_pred[j] == 0) {
          auto& qj = ready[is_div(seq[j].kind)];
          qj.push_back(j);
          std::push_heap(qj.begin(), qj.end(), later);
        }
      }
  }
}

void pack(const std::vector<SeqOp>& seq, uint32_t space, std::vector<Op>& rows, uint32_t& n_rows,
          uint32_t& n_levels) {
  auto enc = [](const SeqOp& s) { return encode(s.kind, s.dst, s.a, s.b); };
  pack_rows(seq, space, kRow, enc, encode(kOpDivY, space - 1, space - 2, space - 2),
            encode(kOpSubNz, space - 1, space - 2, space - 3), rows, n_rows, n_levels);
}

}  // namespace

namespace {

// Ops on the longest dependence chain (each op after the last write of the
// values it reads and of its destination).
uint32_t longest_chain(const std::vector<Op4>& seq, uint32_t nv) {
  std::vector<uint32_t> level(nv, 0);
  uint32_t top = 0;
  for (const Op4& o : seq) {
    const uint32_t v = o.w0 & 0x0fffffffu;
    level[v] = std::max({level[v], level[o.a], level[o.b]}) + 1;
    top = std::max(top, level[v]);
  }
  return top;
}

}  // namespace

Programs compile_tape(const SparseLu& lu) {
  Programs P;
  const Csc& A = *lu.a;
  const uint32_t n = A.n;
  P.n = n;
  P.nu = uint32_t(lu.ui.size());
  P.nl = uint32_t(lu.li.size());
  const uint32_t lx0 = P.nu + n;
  const uint32_t discard = lx0 + P.nl;
  P.ntv = discard + 1;
  const uint32_t y0 = P.ntv;  // y[k] lives at y0 + k
  for (auto v : lu.void_col) P.has_void |= v != 0;

  // buildTape's slot map: per column k, its U rows, the diagonal, its L rows.
  std::vector<uint32_t> pos(n, kNone);
  P.amap.assign(A.nnz(), discard);
  std::vector<SeqOp> a;
  for (uint32_t k = 0; k < n; ++k) {
    const bool void_k = lu.void_col[k] != 0;
    for (uint32_t p = lu.up[k]; p < lu.up[k + 1]; ++p) pos[lu.ui[p]] = p;
    pos[k] = P.nu + k;
    for (uint32_t q = lu.lp[k]; q < lu.lp[k + 1]; ++q) pos[lu.li[q]] = lx0 + q;
    for (uint32_t p = lu.up[k]; p < lu.up[k + 1]; ++p) {
      const uint32_t i = lu.ui[p];
      for (uint32_t q = lu.lp[i]; q < lu.lp[i + 1]; ++q) {
        const uint32_t r = lu.li[q];
        a.push_back({kOpFlop, (void_k && r > k) ? discard : pos[r], lx0 + q, p});
        ++P.flops;
      }
    }
    const uint32_t c = lu.q[k];
    for (uint32_t e = A.col_ptr[c]; e < A.col_ptr[c + 1]; ++e) {
      const uint32_t r = lu.prow[e];
      P.amap[e] = (void_k && r > k) ? discard : pos[r];
    }
    const uint32_t div = lu.scaled[k] ? kOpDivScaled : kOpDivGrowth;
    for (uint32_t q = lu.lp[k]; q < lu.lp[k + 1]; ++q) a.push_back({div, lx0 + q, P.nu + k, lx0 + q});
    // Forward substitution of column k (sparse_lu.zig solve): y[li] -= l * y[k].
    for (uint32_t q = lu.lp[k]; q < lu.lp[k + 1]; ++q) a.push_back({kOpSubNz, y0 + lu.li[q], lx0 + q, y0 + k});
  }
  P.nv = P.ntv + n + 3;
  P.a_seq.reserve(a.size());
  for (const SeqOp& s : a) {
    if (P.nv < 65536) P.a_list.push_back(encode(s.kind, s.dst, s.a, s.b));
    P.a_seq.push_back(Op4{s.dst | (s.kind << 28), s.a, s.b, 0u});
  }
  if (P.nv < 65536) P.a_levels = longest_chain(P.a_seq, P.nv);
  P.a_nops = uint32_t(a.size());

  std::vector<uint8_t> written(P.ntv, 0);
  for (uint32_t e = 0; e < A.nnz(); ++e) written[P.amap[e]] = 1;
  for (uint32_t s = 0; s < P.ntv; ++s)
    if (!written[s]) P.fill.push_back(s);

  P.l_scaled.assign(P.nl, 0);
  for (uint32_t k = 0; k < n; ++k)
    for (uint32_t q = lu.lp[k]; q < lu.lp[k + 1]; ++q) P.l_scaled[q] = lu.scaled[k];

  // Back substitution through U: the diagonal division first in each column.
  std::vector<SeqOp> b;
  for (uint32_t k = n; k-- > 0;) {
    b.push_back({kOpDivY, y0 + k, P.nu + k, y0 + k});
    for (uint32_t p = lu.up[k]; p < lu.up[k + 1]; ++p) b.push_back({kOpSubNz, y0 + lu.ui[p], p, y0 + k});
  }
  for (const SeqOp& s : b) {
    if (P.nv < 65536) P.b_list.push_back(encode(s.kind, s.dst, s.a, s.b));
    P.b_seq.push_back(Op4{s.dst | (s.kind << 28), s.a, s.b, 0u});
  }
  if (P.nv < 65536) P.b_levels = longest_chain(P.b_seq, P.nv);
  P.b_nops = uint32_t(b.size());
  return P;
}

}  // namespace esl

namespace esl {

namespace {

std::vector<SeqOp> unpack(const std::vector<Op4>& ops) {
  std::vector<SeqOp> out;
  out.reserve(ops.size());
  for (const Op4& o : ops) {
    const uint32_t kind = o.w0 >> 28;
    // a multiply-subtract reads a and b; a division reads a (divisor) and b
    out.push_back(SeqOp{kind, o.w0 & 0x0fffffffu, o.a, o.b});
  }
  return out;
}

// Estimated cycles of a task's parts, for the longest-path priorities: an
// update, a division, and the step from one row to the next.
constexpr int kCostOp = 12, kCostDiv = 115, kCostRow = 75;
// A task far from the critical path (its longest path kSlack cycles shorter
// than the longest in the ready list) waits until kTaskOps updates, or its
// last ones, can run at once.
constexpr int kSlack = 300;

// Packs a sequential program into task rows. Every value's updates are one
// list in sequential order; a value is read by other values only once its
// list has run (the column replay and the triangular solves read finished
// entries only), so a task, the next updates of one value, may run as soon
// as their operands are finished in earlier rows. Row by row, the ready
// tasks of the longest remaining paths run, up to one per thread of the
// CTA; tasks with a division, then by updates, then by value (a column's
// entries side by side: their multiplier is one broadcast, their other
// operands neighbours) share a warp. A row of at most 32 tasks is warp 0's
// alone, and between two such rows no CTA barrier is needed.
// Against rows of single ops (434 rows for the 498-unknown analog block's
// refactor, 233 for its back solve) a task keeps its value in a register
// over its updates and its division: 176 and 107 rows, and 3 loads an update
// in place of 4 accesses.
// Where the rows are bound by their number and not by the paths through them
// (a full row's tasks for all the ops make up the longest path), tasks that
// are full go first and then the columns in their order, whatever their
// paths: a row's tasks are neighbours in a column, at the same updates, and
// 32 threads' operands fall into few sectors. Working sets of that size lie
// in global memory (20,001-unknown digital block, eight warps: 86.0M sectors
// of loads by longest paths, 25.9M so, in 49,426 and 50,576 rows; 256 lanes,
// 30 ps: FP64 7,575 -> 2,010 ms, mixed 5,484 -> 1,866; rows of four single ops
// a thread 5,272 and 3,864). With paths a little longer than the rows the
// longest ones stay the better order (1,001-unknown mesh, sixteen warps, 162
// full rows of 319: 0.78 ms against 0.81).
TaskStream pack_tasks(const std::vector<Op4>& seq, uint32_t nv, uint32_t warps, bool compact) {
  const uint32_t sink = nv - 1, one = nv - 2, zero = nv - 3;
  const size_t n = seq.size();
  struct Pair {
    uint32_t a, b;
  };
  auto dst_of = [](const Op4& o) { return o.w0 & 0x0fffffffu; };
  // ops[vptr[v] .. vptr[v + 1]): the operands of value v's ops; kind[v]: its last op's
  std::vector<uint32_t> vptr(nv + 1, 0);
  std::vector<Pair> ops(n);
  std::vector<uint8_t> kind(nv, kOpNop);
  for (const Op4& o : seq) ++vptr[dst_of(o) + 1];
  for (uint32_t v = 0; v < nv; ++v) vptr[v + 1] += vptr[v];
  std::vector<uint32_t> pos(vptr.begin(), vptr.end() - 1);
  for (const Op4& o : seq) {
    const uint32_t v = dst_of(o);
    ops[pos[v]++] = {o.a, o.b};
    kind[v] = uint8_t(o.w0 >> 28);
  }
  auto divides = [&](uint32_t v) { return is_div(kind[v]); };
  // cycles of value v's last `left` ops
  auto rest = [&](uint32_t v, uint32_t left) {
    const bool d = divides(v);
    return int(left - (d ? 1u : 0u)) * kCostOp + (d ? kCostDiv : 0);
  };
  // tail[v]: the longest path from v's end to the program's
  std::vector<int> tail(nv, 0);
  {
    std::vector<uint32_t> left(nv, 0);
    for (size_t i = n; i-- > 0;) {
      const Op4& o = seq[i];
      const uint32_t v = dst_of(o);
      const int path = kCostRow + rest(v, ++left[v]) + tail[v];
      for (uint32_t s : {o.a, o.b})
        if (s != v) tail[s] = std::max(tail[s], path);
    }
  }
  std::copy(vptr.begin(), vptr.end() - 1, pos.begin());  // a value's next op
  std::vector<uint32_t> ready(pos);                      // its ops before ready[v] can run
  std::vector<uint8_t> done(nv, 0);
  for (uint32_t v = 0; v < nv; ++v) done[v] = vptr[v] == vptr[v + 1];
  // the values that wait for value s: head[s], next[head[s]], ..
  std::vector<uint32_t> head(nv, kNone), next(nv, kNone);
  auto advance = [&](uint32_t v) {
    for (; ready[v] < vptr[v + 1]; ++ready[v]) {
      const Pair o = ops[ready[v]];
      for (uint32_t s : {o.a, o.b})
        if (s != v && !done[s]) {
          next[v] = head[s];
          head[s] = v;
          return;
        }
    }
  };
  int longest = 0;
  for (uint32_t v = 0; v < nv; ++v)
    if (vptr[v] < vptr[v + 1]) longest = std::max(longest, rest(v, vptr[v + 1] - vptr[v]) + tail[v]);
  const bool near = warps > 1 && n * (kCostRow + kTaskOps * kCostOp) >= size_t(longest) * kTaskOps * 32 * warps;
  // the values by their first ops' places in the sequence (column by column)
  std::vector<uint32_t> by_place, place(near ? nv : 0, kNone);
  for (size_t i = 0; near && i < n; ++i) {
    const uint32_t v = dst_of(seq[i]);
    if (place[v] != kNone) continue;
    place[v] = uint32_t(by_place.size());
    by_place.push_back(v);
  }
  // a task's worth of updates, or all that are left
  auto full = [&](uint32_t v) { return ready[v] == vptr[v + 1] || ready[v] - pos[v] >= kTaskOps; };
  // The ready tasks, the longest path on top (near: the full ones, the first
  // column), and those that wait to be full. key[v] is value v's place among
  // them, 0 when it has none; an entry that does not agree with it is stale.
  std::vector<uint64_t> key(nv, 0), queue, parked;
  std::vector<uint8_t> is_parked(nv, 0);
  auto push = [](std::vector<uint64_t>& q, uint64_t k) {
    q.push_back(k);
    std::push_heap(q.begin(), q.end());
  };
  auto pop = [](std::vector<uint64_t>& q) {
    std::pop_heap(q.begin(), q.end());
    const uint64_t k = q.back();
    q.pop_back();
    return k;
  };
  auto path_of = [](uint64_t k) { return int(k >> 32); };
  auto value_of = [&](uint64_t k) { return near ? by_place[~uint32_t(k)] : uint32_t(k); };
  auto offer = [&](uint32_t v) {
    if (ready[v] == pos[v]) return;
    if (near) {
      const uint64_t k = uint64_t(full(v)) << 32 | ~place[v];
      if (key[v] != k) push(queue, k);
      key[v] = k;
      return;
    }
    if (key[v] && !(is_parked[v] && full(v))) return;
    key[v] = uint64_t(uint32_t(rest(v, vptr[v + 1] - pos[v]) + tail[v])) << 32 | v;
    is_parked[v] = 0;
    push(queue, key[v]);
  };
  for (uint32_t v = 0; v < nv; ++v)
    if (!done[v]) {
      advance(v);
      offer(v);
    }
  struct Task {
    uint32_t v, lo, ops;  // ops updates from vop[lo], then the division when div
    bool div;
  };
  auto take = [&](uint32_t v) {
    const uint32_t run = ready[v] - pos[v];
    const bool last = ready[v] == vptr[v + 1] && divides(v);
    Task t{v, pos[v], std::min(run - (last ? 1u : 0u), kTaskOps), false};
    t.div = last && t.ops + 1 == run && t.ops < kTaskOps;
    return t;
  };
  std::vector<uint32_t> out[kTaskWarps];
  uint32_t idle[kTaskWarps] = {};
  struct Words {
    uint32_t dst, flags, pair[kTaskOps][2];
  };
  Words lanes[32];
  auto put = [&](uint32_t w) {
    std::vector<uint32_t>& o = out[w];
    if (compact) {
      for (const Words& x : lanes) {
        o.push_back(x.dst | (x.flags << 16));
        for (const auto& p : x.pair) o.push_back(p[0] | (p[1] << 16));
      }
      return;
    }
    for (const Words& x : lanes) o.insert(o.end(), {x.dst, x.flags, x.pair[0][0], x.pair[0][1]});
    for (const Words& x : lanes) o.insert(o.end(), {x.pair[1][0], x.pair[1][1], x.pair[2][0], x.pair[2][1]});
  };
  auto put_idle = [&](uint32_t w, uint32_t barriers) {
    do {  // the count takes the first update's words
      const uint32_t k = std::min(barriers, 0xffffu);
      for (Words& x : lanes) x = Words{0, kTaskIdle, {{k, 0}, {0, 0}, {0, 0}}};
      put(w);
      barriers -= k;
    } while (barriers);
  };
  auto flush = [&](uint32_t w) {
    if (idle[w]) put_idle(w, idle[w]);
    idle[w] = 0;
  };
  TaskStream S;
  // One row's tasks onto the warps; `cta`: a CTA barrier follows.
  auto emit = [&](const std::vector<Task>& row, bool cta) {
    for (uint32_t w = 0; w < warps; ++w) {
      if (32 * w >= row.size()) {
        idle[w] += cta;
        continue;
      }
      flush(w);
      const size_t t0 = 32 * size_t(w), nt = std::min<size_t>(32, row.size() - t0);
      uint32_t most = 0;
      bool any_div = false;
      for (size_t l = 0; l < nt; ++l) {
        most = std::max(most, row[t0 + l].ops);
        any_div |= row[t0 + l].div;
      }
      const uint32_t common =
          (most > 1 ? kTaskMore : 0u) | (any_div ? kTaskDivAny : 0u) | (cta ? kTaskCta : 0u);
      for (uint32_t l = 0; l < 32; ++l) {
        Words& x = lanes[l];
        x = Words{sink, common, {{zero, one}, {zero, one}, {zero, one}}};
        if (l >= nt) continue;
        const Task& t = row[t0 + l];
        x.dst = t.v;
        for (uint32_t j = 0; j < t.ops; ++j) {
          x.pair[j][0] = ops[t.lo + j].a;
          x.pair[j][1] = ops[t.lo + j].b;
        }
        // a value's updates are of one kind: the solves' before a y entry's
        // division, the refactor's before an L entry's
        const uint32_t k = kind[t.v];
        if (k == kOpSubNz || k == kOpDivY) x.flags |= kTaskNz;
        if (t.div) {
          x.flags |= kTaskDiv | (k == kOpDivGrowth ? kTaskGrowth : 0u) | (k == kOpDivScaled ? kTaskScaled : 0u);
          x.pair[kTaskOps - 1][0] = ops[t.lo + t.ops].a;
          x.pair[kTaskOps - 1][1] = one;
        }
      }
      put(w);
    }
    ++S.rows;
  };
  std::vector<Task> row, prev;
  std::vector<uint32_t> finished;
  size_t left = n;
  while (left) {
    row.clear();
    uint64_t top = queue.empty() ? 0 : queue.front();
    if (!parked.empty()) top = std::max(top, parked.front());
    const int bar = path_of(top) - kSlack;
    while (!parked.empty() && path_of(parked.front()) >= bar) {
      const uint64_t k = pop(parked);
      const uint32_t v = value_of(k);
      if (key[v] != k || !is_parked[v]) continue;
      is_parked[v] = 0;
      push(queue, k);
    }
    while (!queue.empty() && row.size() < 32 * warps) {
      const uint64_t k = pop(queue);
      const uint32_t v = value_of(k);
      if (key[v] != k || is_parked[v]) continue;
      if (!near && path_of(k) < bar && !full(v)) {
        is_parked[v] = 1;
        push(parked, k);
        continue;
      }
      key[v] = 0;
      row.push_back(take(v));
    }
    std::sort(row.begin(), row.end(), [&](const Task& x, const Task& y) {
      if (row.size() > 32) {
        if (x.div != y.div) return x.div;
        if ((x.ops > 1) != (y.ops > 1)) return x.ops > 1;
      }
      return x.v < y.v;
    });
    // the row before goes out once it is known whether this one is warp 0's
    if (!prev.empty()) emit(prev, prev.size() > 32 || row.size() > 32);
    finished.clear();
    for (const Task& t : row) {
      const uint32_t k = t.ops + (t.div ? 1u : 0u);
      pos[t.v] += k;
      left -= k;
      if (pos[t.v] == vptr[t.v + 1]) finished.push_back(t.v);
    }
    for (uint32_t v : finished) done[v] = 1;
    for (uint32_t v : finished) {
      for (uint32_t x = head[v]; x != kNone;) {
        const uint32_t after = next[x];
        advance(x);
        offer(x);
        x = after;
      }
    }
    for (const Task& t : row) offer(t.v);
    prev.swap(row);
  }
  if (!prev.empty()) emit(prev, true);
  size_t total = 0;
  for (uint32_t w = 0; w < warps; ++w) {
    flush(w);
    const size_t chunk = 32 * task_words(compact);
    for (uint32_t c = 0; c < kTaskRing; ++c) put_idle(w, 0u);
    total += out[w].size();
    S.off[w + 1] = uint32_t(total / chunk);
  }
  S.words.reserve(total);
  for (auto& o : out) {
    S.words.insert(S.words.end(), o.begin(), o.end());
    std::vector<uint32_t>().swap(o);
  }
  return S;
}

}  // namespace

void pack_op_rows(Programs& P) {
  if (P.nv >= 65536 || !P.a_ops.empty() || !P.b_ops.empty()) return;
  uint32_t levels = 0;
  pack(unpack(P.a_seq), P.nv, P.a_ops, P.a_rows, levels);
  pack(unpack(P.b_seq), P.nv, P.b_ops, P.b_rows, levels);
}

void compile_warp(const Programs& P, TaskStream& a, TaskStream& b) {
  a = pack_tasks(P.a_seq, P.nv, 1, true);
  b = pack_tasks(P.b_seq, P.nv, 1, true);
}

BlockPrograms compile_block(const Programs& P, uint32_t warps) {
  BlockPrograms B;
  B.compact = P.nv < 65536;
  B.a = pack_tasks(P.a_seq, P.nv, warps, B.compact);
  B.b = pack_tasks(P.b_seq, P.nv, warps, B.compact);
  // the forward substitution alone (program A's solve ops), for the mixed
  // form's refinement corrections on the finished factors
  std::vector<Op4> f;
  for (const Op4& s : P.a_seq)
    if ((s.w0 >> 28) == kOpSubNz) f.push_back(s);
  B.f = pack_tasks(f, P.nv, warps, B.compact);
  B.a_levels = longest_chain(P.a_seq, P.nv);
  return B;
}

}  // namespace esl
