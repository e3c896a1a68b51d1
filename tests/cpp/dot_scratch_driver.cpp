// alloc_zeroed (csrc/sepx_blas.h) over stand-ins of the three CUDA calls it
// makes: a refused allocation or clear leaves the caller's pointer unset and
// nothing allocated, so that the next call allocates and clears again.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "sepx_blas.h"

static int g_live = 0, g_clears = 0;
static cudaError_t g_malloc = cudaSuccess, g_clear = cudaSuccess;

extern "C" {
cudaError_t CUDARTAPI cudaMalloc(void **p, size_t n) {
  if (g_malloc != cudaSuccess) return g_malloc;
  *p = std::malloc(n);
  std::memset(*p, 0xff, n);
  g_live++;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaFree(void *p) {
  if (p) g_live--;
  std::free(p);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
  if (g_clear != cudaSuccess) return g_clear;
  g_clears++;
  std::memset(p, v, n);
  return cudaSuccess;
}
}

#define CHECK(c)                                   \
  if (!(c)) {                                      \
    std::printf("line %d: %s\n", __LINE__, #c);    \
    return 1;                                      \
  }

int main() {
  double *p = nullptr;
  g_clear = cudaErrorLaunchFailure;
  CHECK(sepx::alloc_zeroed(&p, 5, nullptr) == cudaErrorLaunchFailure);
  CHECK(p == nullptr && g_live == 0);
  g_clear = cudaSuccess;
  g_malloc = cudaErrorMemoryAllocation;
  CHECK(sepx::alloc_zeroed(&p, 5, nullptr) == cudaErrorMemoryAllocation);
  CHECK(p == nullptr && g_live == 0);
  g_malloc = cudaSuccess;
  CHECK(sepx::alloc_zeroed(&p, 5, nullptr) == cudaSuccess);
  CHECK(p != nullptr && g_live == 1 && g_clears == 1);
  for (int i = 0; i < 5; i++) CHECK(p[i] == 0.0);
  cudaFree(p);
  return 0;
}
