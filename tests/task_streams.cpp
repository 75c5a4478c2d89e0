// Test helper: packs a matrix's tape into the block lanes' task streams
// (host/schedule.cpp compile_block) and runs them as the kernels do, a row of
// every warp between two barriers at a time. Input file: n, col_ptr, row_idx,
// lead values, then a lane's values and right-hand side. For each number of
// warps prints: rows, sectors of program A's loads per update, and a verdict.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "common.h"
#include "host/schedule.hpp"

using namespace esl;

static void fail(const char* what) {
  std::printf("FAIL %s\n", what);
  std::exit(0);
}

// Distinct sectors of 32 bytes (four values) among a warp's 32 operands.
static size_t sectors_of(uint32_t* x, size_t n) {
  for (size_t k = 0; k < n; ++k) x[k] /= 4;
  std::sort(x, x + n);
  return size_t(std::unique(x, x + n) - x);
}

struct Task {
  uint32_t dst, flags, idle, a[3], b[3];
};

static Task decode(const TaskStream& S, bool compact, uint32_t chunk, int lane) {
  const uint32_t* p = &S.words[size_t(chunk) * 32 * task_words(compact)];
  Task t{};
  if (compact) {
    const uint32_t* q = p + 4 * lane;
    t = {q[0] & 0xffffu, q[0] >> 16, q[1], {q[1] & 0xffffu, q[2] & 0xffffu, q[3] & 0xffffu},
         {q[1] >> 16, q[2] >> 16, q[3] >> 16}};
  } else {
    const uint32_t *q = p + 4 * lane, *e = p + 128 + 4 * lane;
    t = {q[0], q[1], q[2], {q[2], e[0], e[2]}, {q[3], e[1], e[3]}};
  }
  return t;
}

// Runs one program; returns the sectors its loads touch (FP64) and counts its
// updates.
static double run(const TaskStream& S, bool compact, uint32_t warps, std::vector<double>& v, size_t& updates) {
  const uint32_t nv = uint32_t(v.size()), sink = nv - 1, zero = nv - 3;
  std::vector<uint32_t> at(warps), idle(warps, 0);
  for (uint32_t w = 0; w < warps; ++w) at[w] = S.off[w];
  double sectors = 0;
  // the barrier interval and warp that last wrote a value
  std::vector<uint32_t> when(nv, 0), who(nv, 0);
  std::vector<std::pair<uint32_t, uint32_t>> read;  // value, warp
  for (uint32_t interval = 1;; ++interval) {
    // every warp up to its next barrier; who wrote or read what in between
    read.clear();
    uint32_t at_barrier = 0, ended = 0;
    for (uint32_t w = 0; w < warps; ++w) {
      for (;;) {
        if (idle[w]) {
          --idle[w];
          ++at_barrier;
          break;
        }
        if (at[w] + kTaskRing == S.off[w + 1]) {
          ++ended;
          break;
        }
        const uint32_t c = at[w]++;
        const Task first = decode(S, compact, c, 0);
        if (first.flags & kTaskIdle) {
          idle[w] = first.idle;
          continue;
        }
        double out[32];
        Task ts[32];
        uint32_t touched[7][32], dsts[32];
        size_t n_touched[7] = {}, n_dsts = 0;
        for (int l = 0; l < 32; ++l) {
          const Task t = decode(S, compact, c, l);
          if ((t.flags ^ first.flags) & (kTaskMore | kTaskDivAny | kTaskCta | kTaskIdle)) fail("flags differ in a warp");
          if (t.dst != sink) dsts[n_dsts++] = t.dst;
          double d = v[t.dst];
          const bool div = t.flags & kTaskDiv;
          touched[0][n_touched[0]++] = t.dst;
          for (int j = 0; j < 3; ++j) {
            if (j && !(t.flags & kTaskMore) && !(j == 2 && div)) continue;
            touched[1 + 2 * j][n_touched[1 + 2 * j]++] = t.a[j];
            touched[2 + 2 * j][n_touched[2 + 2 * j]++] = t.b[j];
            read.push_back({t.a[j], w});
            read.push_back({t.b[j], w});
            if (j == 2 && div) continue;
            if (t.a[j] != zero) ++updates;
            if (v[t.b[j]] != 0.0 || !(t.flags & kTaskNz)) d = d - v[t.a[j]] * v[t.b[j]];
          }
          if (div && !(t.flags & kTaskDivAny)) fail("a division in a warp without the flag");
          if (div) d = d / v[t.a[2]];
          out[l] = d;
          ts[l] = t;
        }
        std::sort(dsts, dsts + n_dsts);
        if (std::adjacent_find(dsts, dsts + n_dsts) != dsts + n_dsts) fail("two tasks of a row on one value");
        for (int k = 0; k < 7; ++k) sectors += double(sectors_of(touched[k], n_touched[k]));
        for (const Task& t : ts) {
          v[t.dst] = out[&t - ts];
          if (t.dst == sink) continue;
          if (when[t.dst] == interval && who[t.dst] != w) fail("two warps write one value between barriers");
          when[t.dst] = interval;
          who[t.dst] = w;
        }
        if (first.flags & kTaskCta) {
          ++at_barrier;
          break;
        }
      }
    }
    for (const auto& x : read)
      if (when[x.first] == interval && who[x.first] != x.second)
        fail("a warp reads what another writes between barriers");
    if (at_barrier + ended != warps || (at_barrier && ended)) fail("warps meet different numbers of barriers");
    if (ended == warps) return sectors;
  }
}

int main(int argc, char** argv) {
  FILE* f = argc > 1 ? std::fopen(argv[1], "rb") : nullptr;
  Csc pat;
  if (!f || std::fread(&pat.n, 4, 1, f) != 1) return 1;
  pat.col_ptr.resize(pat.n + 1);
  if (std::fread(pat.col_ptr.data(), 4, pat.n + 1, f) != pat.n + 1) return 1;
  const size_t nnz = pat.col_ptr[pat.n];
  pat.row_idx.resize(nnz);
  std::vector<double> lead(nnz), vals(nnz), rhs(pat.n);
  if (std::fread(pat.row_idx.data(), 4, nnz, f) != nnz || std::fread(lead.data(), 8, nnz, f) != nnz ||
      std::fread(vals.data(), 8, nnz, f) != nnz || std::fread(rhs.data(), 8, pat.n, f) != pat.n)
    return 1;
  SparseLu lu;
  lu.init(&pat, order_columns(pat));
  lu.fill_cap = kRepivotFillCap;
  lu.keep_min = kGrowthLimit;
  if (!lu.factor(lead.data(), kPivotTol)) return 1;
  const Programs P = compile_tape(lu);
  std::vector<double> start(P.nv, 0.0);
  start[P.nv - 2] = 1.0;
  for (size_t e = 0; e < nnz; ++e) start[P.amap[e]] = vals[e];
  for (uint32_t i = 0; i < P.n; ++i) start[P.ntv + lu.pinv[i]] = -rhs[i];
  // the sequential replay
  std::vector<double> ref = start;
  for (const auto* seq : {&P.a_seq, &P.b_seq})
    for (const Op4& o : *seq) {
      const uint32_t kind = o.w0 >> 28, d = o.w0 & 0x0fffffffu;
      if (kind == kOpFlop || kind == kOpSubNz) {
        if (kind == kOpFlop || ref[o.b] != 0.0) ref[d] = ref[d] - ref[o.a] * ref[o.b];
      } else {
        ref[d] = ref[o.b] / ref[o.a];
      }
    }
  for (uint32_t warps : {4u, 8u, 16u}) {
    const BlockPrograms B = compile_block(P, warps);
    std::vector<double> v = start;
    size_t updates = 0, more = 0;
    const double sectors = run(B.a, B.compact, warps, v, updates);
    run(B.b, B.compact, warps, v, more);
    if (updates + more + P.nl + P.n != P.a_seq.size() + P.b_seq.size()) fail("ops lost or doubled");
    if (std::memcmp(v.data(), ref.data(), 8 * size_t(P.nv - 3)) != 0) fail("not the replay's values");
    std::printf("ok %u %u %.4f\n", warps, B.a.rows, updates ? sectors / double(updates) : 0.0);
  }
  return 0;
}
