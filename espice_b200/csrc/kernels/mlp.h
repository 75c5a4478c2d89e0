// Launchers of the learned warm start's tensor-core kernels (mlp.cu).
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace esl {

// C = A (M x K) . B (N x K)^T, BF16 in, FP32 accumulate; K, N multiples of
// 16; epilogue: + bias[n], FP32 store to c, tanh (act 1) or identity as BF16
// to h. err receives 1 when a tensor-core completion wait ran out (after
// wait_rounds try_wait rounds; 0: the kernel's default bound; ~0u: no
// round at all, the wait runs out at once), and then nothing is stored.
cudaError_t launch_gemm_bf16(const __nv_bfloat16* a, int lda, const __nv_bfloat16* b, int ldb, int M, int N, int K,
                             const float* bias, float* c, int ldc, __nv_bfloat16* h, int ldh, int act, int* err,
                             cudaStream_t s, uint32_t wait_rounds = 0);
// A layer's dZ (rows x cols) from dH: through tanh's slope at zpre into dz
// (zpre null: dh is dZ already), as BF16 (dzb) and transposed (dzt).
cudaError_t launch_layer_grad(const float* dh, const float* zpre, int rows, int cols, float* dz, __nv_bfloat16* dzb,
                              __nv_bfloat16* dzt, cudaStream_t s);
cudaError_t launch_transpose_bf16(const __nv_bfloat16* in, int rows, int cols, int ldi, __nv_bfloat16* out, int ldo,
                                  cudaStream_t s);
cudaError_t launch_bias_grad(const float* dz, int rows, int cols, int ld, float* db, cudaStream_t s);
cudaError_t launch_mse_grad(const float* y, const float* t, int rows, int outs, int ld, float* d, cudaStream_t s);
cudaError_t launch_mse_loss(const float* y, const float* t, int rows, int outs, int ld, float* loss, cudaStream_t s);

// One Adam step of several tensors, w rows x cols each; wb, wt: BF16 copies
// (row-major, transposed) to refresh, or null. rates[*step]: the learning
// rate and the bias corrections 1 - beta^t.
constexpr float kAdamB1 = 0.9f, kAdamB2 = 0.999f;
struct AdamRate {
  float lr, c1, c2;
};
struct AdamTensor {
  float *w, *g, *m, *v;
  __nv_bfloat16 *wb, *wt;
  int rows, cols;
  uint32_t first;  // its first block (launch_adam sets it)
};
constexpr int kAdamMax = 16;
struct AdamTensors {
  int n;
  AdamTensor t[kAdamMax];
};
cudaError_t launch_adam(AdamTensors T, const AdamRate* rates, uint32_t* step, cudaStream_t s);
// wb, wt: w (rows x cols) as BF16 and its transpose.
cudaError_t launch_weight_copies(const float* w, int rows, int cols, __nv_bfloat16* wb, __nv_bfloat16* wt,
                                 cudaStream_t s);
cudaError_t launch_next_step(uint32_t* step, cudaStream_t s);

}  // namespace esl
