// sepx_blas.h -- launchers of the BLAS-1 kernels (sepx_blas.cu).
#pragma once
#include <cuda_runtime.h>

namespace sepx {

// FP64 dot product of two float vectors (b == nullptr: sum of a), written to
// *out (device or mapped host memory); `scratch`: vec_dot_scratch_doubles()
// doubles, zero before the first call and used by one stream at a time.
cudaError_t vec_dot(const float *a, const float *b, long long n, double *scratch, double *out,
                    cudaStream_t st);
int vec_dot_scratch_doubles();
// n zeroed doubles on the device; *p is set only once the clear is queued (a
// buffer whose clear was refused must not be found by the next call: the dot
// product's counter would never come round, and its result never be written)
inline cudaError_t alloc_zeroed(double **p, size_t n, cudaStream_t st) {
  double *q = nullptr;
  cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&q), n * sizeof(double));
  if (e != cudaSuccess) return e;
  e = cudaMemsetAsync(q, 0, n * sizeof(double), st);
  if (e != cudaSuccess) {
    cudaFree(q);
    return e;
  }
  *p = q;
  return cudaSuccess;
}
cudaError_t vec_fill(float *x, long long n, float v, cudaStream_t st);
cudaError_t vec_scale(float *y, long long n, double a, cudaStream_t st);
cudaError_t vec_scale_add(float *y, const float *x, long long n, double a, double b, cudaStream_t st);
cudaError_t vec_scale_add2(float *y, const float *x1, const float *x2, long long n, double a,
                           double b, cudaStream_t st);
cudaError_t vec_add(float *y, const float *x, long long n, cudaStream_t st);
cudaError_t vec_mult(float *y, const float *x, long long n, cudaStream_t st);
cudaError_t vec_random(float *y, long long n, unsigned long long seed, cudaStream_t st);

}  // namespace sepx
