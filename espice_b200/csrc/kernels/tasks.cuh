// The task programs (host/schedule.cpp pack_tasks) over a lane's value
// space: every lane of a warp takes one task a chunk, up to kTaskOps updates
// of one value and its division; a block lane's CTA steps from row to row by
// barriers, a warp lane is one warp and its rows follow each other.
//
// What bounds it is the chain of rows, not the arithmetic: a row costs a
// warp's in-order pass through one chunk and the barrier. So a row does as
// much as it can: a value stays in a register over its updates and its
// division, every operand of a chunk is loaded before the first is used, and
// selects stand in place of branches. The words stream from L2 through a
// ring of four chunks a warp by cp.async: loads into registers, three chunks
// ahead, share the warp's few scoreboards with the operands' loads, which
// then wait for L2 as well (analog block, mixed, two CTAs an SM: 210k cycles a
// refactor; one chunk ahead 260k; through the ring 142k).
//
// A division tests its pivot as the CPU replay does (growth, or a finite
// quotient in a row-scaled column), and in a column without row scaling
// also the L entry it makes against the wide-multiplier bound.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "../common.h"

namespace esl {

namespace {

__device__ __forceinline__ bool task_zero(double x) { return ((__double2hiint(x) << 1) | __double2loint(x)) == 0; }
__device__ __forceinline__ bool task_finite(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }
__device__ __forceinline__ bool task_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) != 0x7f800000u; }
// d / a rounded to nearest. The FP64 division's fast path leaves a zero
// dividend to its slow path, and whole warps meet one (padding, zero
// right-hand sides), so a zero divides as 2^-200 and the quotient's sign and
// special cases come back with the product.
__device__ __forceinline__ double task_div(double d, double a) {
  const bool z = task_zero(d);
  const double q = __ddiv_rn(z ? 0x1p-200 : d, a);
  return z ? __dmul_rn(d, q) : q;
}
__device__ __forceinline__ float task_div(float d, float a) { return __fdiv_rn(d, a); }
__device__ __forceinline__ double task_msub(double d, double a, double b) { return __dsub_rn(d, __dmul_rn(a, b)); }
__device__ __forceinline__ float task_msub(float d, float a, float b) { return __fsub_rn(d, __fmul_rn(a, b)); }
__device__ __forceinline__ double task_growth(double) { return 1e-12; }
__device__ __forceinline__ float task_growth(float) { return 1e-12f; }

// The value space, in the CTA's shared memory or its slab of global memory.
template <typename V, bool kShared>
struct TaskMem;
template <>
struct TaskMem<double, true> {
  uint32_t at;
  __device__ explicit TaskMem(double* v) : at(static_cast<uint32_t>(__cvta_generic_to_shared(v))) {}
  __device__ __forceinline__ double ld(uint32_t i) const {
    double r;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(r) : "r"(at + 8 * i));
    return r;
  }
  __device__ __forceinline__ void st(uint32_t i, double x) const {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(at + 8 * i), "d"(x) : "memory");
  }
};
template <>
struct TaskMem<float, true> {
  uint32_t at;
  __device__ explicit TaskMem(float* v) : at(static_cast<uint32_t>(__cvta_generic_to_shared(v))) {}
  __device__ __forceinline__ float ld(uint32_t i) const {
    float r;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r) : "r"(at + 4 * i));
    return r;
  }
  __device__ __forceinline__ void st(uint32_t i, float x) const {
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 4 * i), "f"(x) : "memory");
  }
};
template <>
struct TaskMem<double, false> {
  double* at;
  __device__ explicit TaskMem(double* v) : at(v) {}
  __device__ __forceinline__ double ld(uint32_t i) const {
    double r;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(r) : "l"(at + i));
    return r;
  }
  __device__ __forceinline__ void st(uint32_t i, double x) const {
    asm volatile("st.global.f64 [%0], %1;" ::"l"(at + i), "d"(x) : "memory");
  }
};
template <>
struct TaskMem<float, false> {
  float* at;
  __device__ explicit TaskMem(float* v) : at(v) {}
  __device__ __forceinline__ float ld(uint32_t i) const {
    float r;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(r) : "l"(at + i));
    return r;
  }
  __device__ __forceinline__ void st(uint32_t i, float x) const {
    asm volatile("st.global.f32 [%0], %1;" ::"l"(at + i), "f"(x) : "memory");
  }
};

__device__ __forceinline__ uint4 task_lds(uint32_t at) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(at));
  return r;
}
__device__ __forceinline__ void task_copy(uint32_t to, const uint4* from) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
__device__ __forceinline__ void task_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void task_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// One lane's task words (common.h), from a ring slot.
template <bool kCompact>
struct TaskLane;
template <>
struct TaskLane<true> {
  static constexpr uint32_t kBytes = 512;  // a chunk
  uint4 c;
  __device__ __forceinline__ void load(uint32_t at) { c = task_lds(at); }
  static __device__ __forceinline__ void copy(uint32_t to, const uint4* from) { task_copy(to, from); }
  __device__ __forceinline__ uint32_t flags() const { return c.x >> 16; }
  __device__ __forceinline__ uint32_t dst() const { return c.x & 0xffffu; }
  __device__ __forceinline__ uint32_t idle() const { return c.y; }
  __device__ __forceinline__ uint32_t a(int j) const { return (j == 0 ? c.y : j == 1 ? c.z : c.w) & 0xffffu; }
  __device__ __forceinline__ uint32_t b(int j) const { return (j == 0 ? c.y : j == 1 ? c.z : c.w) >> 16; }
};
template <>
struct TaskLane<false> {
  static constexpr uint32_t kBytes = 1024;
  uint4 c, e;
  __device__ __forceinline__ void load(uint32_t at) {
    c = task_lds(at);
    e = task_lds(at + 512);
  }
  static __device__ __forceinline__ void copy(uint32_t to, const uint4* from) {
    task_copy(to, from);
    task_copy(to + 512, from + 32);
  }
  __device__ __forceinline__ uint32_t flags() const { return c.y; }
  __device__ __forceinline__ uint32_t dst() const { return c.x; }
  __device__ __forceinline__ uint32_t idle() const { return c.z; }
  __device__ __forceinline__ uint32_t a(int j) const { return j == 0 ? c.z : j == 1 ? e.x : e.z; }
  __device__ __forceinline__ uint32_t b(int j) const { return j == 0 ? c.w : j == 1 ? e.y : e.w; }
};

// The barrier between two rows of a CTA's program. Its warps come to it from
// different places of run_task, a warp without tasks in a row from its idle
// chunk: the PTX barrier counts warps wherever they arrive, __syncthreads()
// in such code is defined for a CTA of one mind only.
__device__ __forceinline__ void task_barrier() {
  asm volatile("bar.sync 0;" ::: "memory");
}

// kCta: the program of a CTA's warps (idle chunks, CTA barriers), else of
// one warp.
template <typename V, bool kShared, bool kCompact, bool kCta>
__device__ __forceinline__ void run_task(const TaskLane<kCompact>& c, const TaskMem<V, kShared>& v, uint32_t& bad) {
  const uint32_t f = c.flags();
  if constexpr (kCta) {
    if (f & kTaskIdle) {
      for (uint32_t k = c.idle(); k; --k) task_barrier();
      return;
    }
  }
  const uint32_t dst = c.dst();
  const bool all = !(f & kTaskNz), div = f & kTaskDiv;
  V d = v.ld(dst);
  const V a0 = v.ld(c.a(0)), b0 = v.ld(c.b(0)), a2 = v.ld(c.a(2));
  if (f & kTaskMore) {
    const V a1 = v.ld(c.a(1)), b1 = v.ld(c.b(1)), b2 = v.ld(c.b(2));
    const bool r0 = b0 != V(0) || all, r1 = b1 != V(0) || all, r2 = (b2 != V(0) || all) && !div;
    V t = task_msub(d, a0, b0);
    d = r0 ? t : d;
    t = task_msub(d, a1, b1);
    d = r1 ? t : d;
    t = task_msub(d, a2, b2);
    d = r2 ? t : d;
  } else {
    const bool r0 = b0 != V(0) || all;
    const V t = task_msub(d, a0, b0);
    d = r0 ? t : d;
  }
  if (f & kTaskDivAny) {
    // a lane that does not divide takes 1.0: its other operand may be zero,
    // and one such lane sends the warp down the division's slow path (the
    // ring's two programs: 31k cycles, against 25k)
    const V piv = div ? a2 : V(1);
    const V q = task_div(d, piv);
    const bool shrunk = !(fabs(piv) >= task_growth(piv) * fabs(d) && fabs(q) <= V(1e3)), wild = !task_finite(q);
    bad |= (uint32_t(shrunk) & (f / kTaskGrowth)) | (uint32_t(wild) & (f / kTaskScaled));
    d = div ? q : d;
  }
  v.st(dst, d);
  if (kCta && (f & kTaskCta)) task_barrier();
  else __syncwarp();
}

// Runs a warp's `chunks` from `first` of a program's words, streamed through
// the warp's part of the ring (shared address): while a chunk runs, the next
// one's words are on their way into registers and the two after that into
// the ring. Returns bit 0 set when a division of this thread failed its
// pivot test.
template <typename V, bool kShared, bool kCompact, bool kCta = true>
__device__ __noinline__ uint32_t run_tasks(const uint32_t* words, uint32_t first, uint32_t chunks, uint32_t ring,
                                           V* values) {
  using Lane = TaskLane<kCompact>;
  constexpr uint32_t kBytes = Lane::kBytes, kStep = kBytes / 16, kSpan = kTaskRing * kBytes;
  const uint32_t lane = threadIdx.x & 31;
  const uint4* s = reinterpret_cast<const uint4*>(words) + size_t(first) * kStep + lane;
  const uint32_t base = ring + (threadIdx.x >> 5) * kSpan + 16 * lane;
  const TaskMem<V, kShared> v(values);
#pragma unroll
  for (uint32_t k = 0; k + 1 < kTaskRing; ++k) {
    Lane::copy(base + k * kBytes, s);
    task_commit();
    s += kStep;
  }
  uint32_t bad = 0, read = 0, fill = (kTaskRing - 1) * kBytes;
  Lane c, next;
  task_wait<kTaskRing - 2>();
  c.load(base);
  for (uint32_t k = 0; k < chunks; ++k) {
    Lane::copy(base + fill, s);
    task_commit();
    s += kStep;
    read = (read + kBytes) & (kSpan - 1);
    fill = (fill + kBytes) & (kSpan - 1);
    task_wait<kTaskRing - 2>();
    next.load(base + read);
    run_task<V, kShared, kCompact, kCta>(c, v, bad);
    c = next;
  }
  task_wait<0>();
  return bad & 1u;
}

// Runs one warp's program of `chunks` whose words lie in shared memory
// (`words`, a shared address), the next chunk's read while this one runs.
__device__ __noinline__ uint32_t run_warp_tasks(uint32_t words, uint32_t chunks, double* values) {
  uint32_t at = words + 16 * (threadIdx.x & 31), bad = 0;
  const TaskMem<double, true> v(values);
  TaskLane<true> c, next;
  c.load(at);
  for (uint32_t k = 0; k < chunks; ++k) {
    at += TaskLane<true>::kBytes;
    next.load(at);
    run_task<double, true, true, false>(c, v, bad);
    c = next;
  }
  return bad & 1u;
}

// The same with the words in global memory and no ring: a warp whose lane
// takes all of its CTA's shared memory.
__device__ __noinline__ uint32_t run_far_tasks(const uint32_t* words, uint32_t first, uint32_t chunks, double* values) {
  const uint4* s = reinterpret_cast<const uint4*>(words) + size_t(first) * 32 + (threadIdx.x & 31);
  const TaskMem<double, true> v(values);
  uint32_t bad = 0;
  TaskLane<true> c, next;
  c.c = __ldg(s);
  for (uint32_t k = 0; k < chunks; ++k) {
    s += 32;
    next.c = __ldg(s);
    run_task<double, true, true, false>(c, v, bad);
    c = next;
  }
  return bad & 1u;
}

}  // namespace

}  // namespace esl
