// Test helper: the device models' quotients by one divisor (models.cuh
// Divisor) beside the division, n of each from device arrays a, b.
#include <cuda_runtime.h>

#include "kernels/models.cuh"

namespace esl {

__global__ void divide(const double* a, const double* b, double* one, double* three, double* div, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const Divisor by(b[i]);
  one[i] = by.quot(a[i]);
  // a's neighbours with it, so that the three of a call are of all kinds
  double x = a[i], y = a[(i + 1) % n], z = a[(i + 7) % n];
  by.quot3(x, y, z);
  three[i] = x;
  three[n + i] = y;
  three[2 * n + i] = z;
  div[i] = __ddiv_rn(a[i], b[i]);
  div[n + i] = __ddiv_rn(a[(i + 1) % n], b[i]);
  div[2 * n + i] = __ddiv_rn(a[(i + 7) % n], b[i]);
}

}  // namespace esl

extern "C" int probe(const double* a, const double* b, double* one, double* three, double* div, int n) {
  esl::divide<<<(n + 255) / 256, 256>>>(a, b, one, three, div, n);
  const cudaError_t e = cudaGetLastError();
  return int(e == cudaSuccess ? cudaDeviceSynchronize() : e);
}
