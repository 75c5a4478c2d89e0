// The block lanes' task programs (host/schedule.cpp pack_tasks) over a
// lane's value space: every lane of a warp takes one task a chunk, up to
// kTaskOps updates of one value and its division, and the CTA steps from
// row to row by barriers.
//
// What bounds it is the chain of rows, not the arithmetic: a row costs a
// warp's in-order pass through one chunk (about 340 cycles with three
// updates, 165 more with a division; B200, all eight warps in step) and the
// barrier (50). So a row does as much as it can: a value stays in a register
// over its updates and its division, every operand of a chunk is loaded
// before the first is used, selects stand in place of branches, and the next
// chunks' words are already in registers (read kTaskUnroll ahead, straight
// from L2: a ring in shared memory is 5% faster alone, but its 24 KB cost
// the second CTA of an SM).
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

// One lane's task of a chunk (common.h), read past L1: a CTA reads each once.
struct TaskChunk {
  uint4 h, u;
  __device__ __forceinline__ void load(const uint4* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(h.x), "=r"(h.y), "=r"(h.z), "=r"(h.w)
                 : "l"(p));
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w)
                 : "l"(p + 32));
  }
};

template <typename V, bool kShared>
__device__ __forceinline__ void run_task(const TaskChunk& c, const TaskMem<V, kShared>& v, uint32_t& bad) {
  const uint32_t w0 = c.h.x, w1 = c.h.y, dst = w0 & kTaskIndex;
  if (dst == kTaskIdle) {
    for (uint32_t k = w1; k; --k) __syncthreads();
    return;
  }
  const bool all = !(w0 & kTaskNz);
  V d = v.ld(dst);
  const V a0 = v.ld(c.h.z), b0 = v.ld(c.h.w), piv = v.ld(w1 & kTaskIndex);
  if (w0 & kTaskMore) {
    const V a1 = v.ld(c.u.x), b1 = v.ld(c.u.y), a2 = v.ld(c.u.z), b2 = v.ld(c.u.w);
    const bool r0 = b0 != V(0) || all, r1 = b1 != V(0) || all, r2 = b2 != V(0) || all;
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
  if (w1 & kTaskDivAny) {
    const V q = task_div(d, piv);
    const bool shrunk = !(fabs(piv) >= task_growth(piv) * fabs(d)), wild = !task_finite(q);
    bad |= (uint32_t(shrunk) & (w1 / kTaskGrowth)) | (uint32_t(wild) & (w1 / kTaskScaled));
    d = (w0 & kTaskDiv) ? q : d;
  }
  v.st(dst, d);
  if (w0 & kTaskCta) __syncthreads();
  else __syncwarp();
}

// Runs a warp's `chunks` (a multiple of kTaskUnroll) from `first` of a
// program's words. Returns bit 0 set when a division of this thread failed
// its pivot test.
template <typename V, bool kShared>
__device__ __noinline__ uint32_t run_tasks(const uint32_t* words, uint32_t first, uint32_t chunks, V* values) {
  constexpr uint32_t kStep = 8 * kTaskWords;  // uint4 a chunk
  const uint4* s = reinterpret_cast<const uint4*>(words) + size_t(first) * kStep + (threadIdx.x & 31);
  const TaskMem<V, kShared> v(values);
  static_assert(kTaskUnroll == 3, "three chunks in registers");
  TaskChunk c0, c1, c2;
  c0.load(s);
  c1.load(s + kStep);
  c2.load(s + 2 * kStep);
  uint32_t bad = 0;
  for (uint32_t k = 0; k < chunks; k += kTaskUnroll) {
    s += kTaskUnroll * kStep;
    run_task(c0, v, bad);
    c0.load(s);
    run_task(c1, v, bad);
    c1.load(s + kStep);
    run_task(c2, v, bad);
    c2.load(s + 2 * kStep);
  }
  return bad & 1u;
}

}  // namespace

}  // namespace esl
