// sepx_blas.cu -- BLAS-1 on device-resident float vectors for the operator
// and solver layer (my_vector / hypercube_float, Born/hypercube_float.cpp:
// 123-223): products accumulated in FP64 like the reference's dot / sum, the
// rest in FP32 with the reference's double scale factors.
//
// Reductions are deterministic: a fixed grid writes one FP64 partial per block
// into scratch and a single block sums the partials in a fixed order.
#include <cuda_runtime.h>
#include <stdint.h>

#include "sepx_blas.h"

namespace sepx {

// What bounds these kernels is the FP64 pipe (2 operations per clock and SM),
// which also runs the conversions between float and double: with them a dot
// product of 65.5 M elements took 364 us and y = a x1 + b x2 626 us, 1.4 and
// 1.3 TB/s.  Conversions are therefore done on the integer units (the same
// values; a group with anything but normal numbers and zeros takes the
// conversion instructions), and rows are read and written 16 bytes at a time:
// one FP64 operation per element is left in the dot product (127 us), two in
// the scaled sums (265 us).

// subnormal, infinite or NaN
__device__ __forceinline__ bool f2d_odd(float x) {
  const uint32_t m = __float_as_uint(x) & 0x7fffffffu;
  return m - 0x00800000u >= 0x7f000000u && m != 0u;
}
// a normal number or a zero as a double
__device__ __forceinline__ double f2d_int(float x) {
  const uint32_t u = __float_as_uint(x), m = u & 0x7fffffffu;
  const uint32_t hi = m ? (m >> 3) + 0x38000000u : 0u;   // exponent bias 127 -> 1023
  return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)(u << 29));
}
// N floats as doubles: the conversion instructions only where one of them needs
// them, in one real branch (a predicated conversion occupies the pipe all the
// same; volatile: nothing is hoisted)
template <int N>
__device__ __forceinline__ void f2d(const float (&x)[N], double (&d)[N]) {
  bool odd = false;
#pragma unroll
  for (int i = 0; i < N; i++) odd |= f2d_odd(x[i]);
  if (__any_sync(__activemask(), odd)) {
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("cvt.f64.f32 %0, %1;" : "=d"(d[i]) : "f"(x[i]));
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) d[i] = f2d_int(x[i]);
  }
}

// results outside the normal range of float (or at its upper end, where
// rounding may leave it), zeros apart
__device__ __forceinline__ bool d2f_odd(double d) {
  const uint32_t m = (uint32_t)__double2hiint(d) & 0x7fffffffu;
  return m - 0x38100000u >= 0x0fd00000u && (m | (uint32_t)__double2loint(d)) != 0u;
}
// the others, rounded to the nearest float, ties to even: 29 bits go, half of
// the last kept bit is added (less one where that bit is even)
__device__ __forceinline__ float d2f_int(double d) {
  const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d), m = hi & 0x7fffffffu;
  const uint64_t r = (((uint64_t)(m - 0x38000000u) << 32) | lo) + 0x0fffffffu + ((lo >> 29) & 1u);
  return __uint_as_float(((m | lo) ? (uint32_t)(r >> 29) : 0u) | (hi & 0x80000000u));
}
template <int N>
__device__ __forceinline__ void d2f(const double (&d)[N], float (&x)[N]) {
  bool odd = false;
#pragma unroll
  for (int i = 0; i < N; i++) odd |= d2f_odd(d[i]);
  if (__any_sync(__activemask(), odd)) {
#pragma unroll
    for (int i = 0; i < N; i++) asm volatile("cvt.rn.f32.f64 %0, %1;" : "=f"(x[i]) : "d"(d[i]));
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = d2f_int(d[i]);
  }
}

constexpr int kDotBlocks = 4 * 152;   // 4 CTAs per SM on a 152-SM GB300
constexpr int kDotThreads = 256;

__device__ __forceinline__ double block_sum(double v) {
  __shared__ double red[kDotThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) red[w] = v;
  __syncthreads();
  v = 0.0;
  if (w == 0) {
    v = (l < kDotThreads / 32) ? red[l] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;
}

// partials[b] = sum over the grid-stride elements of block b of a[i]*b[i]
// (b == nullptr: sum of a[i]); the block that finishes last adds the partials
// in block order (a fixed order: repeatable bits) and writes *out, which may
// be mapped host memory.  done: a counter that is 0 before and after.
// VEC: both pointers 16-byte aligned, four elements per load.
template <bool VEC>
__global__ void __launch_bounds__(kDotThreads)
    dot_kernel(const float *__restrict__ a, const float *__restrict__ b, long long n, double *partials,
               unsigned int *done, double *out) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  long long i0 = t;
  if (VEC) {
    const float4 *a4 = reinterpret_cast<const float4 *>(a), *b4 = reinterpret_cast<const float4 *>(b);
    const long long n4 = n >> 2;
    for (long long i = t; i < n4; i += stride) {
      const float4 x = __ldg(a4 + i);
      if (b) {
        const float4 y = __ldg(b4 + i);
        const float v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        double d[8];
        f2d(v, d);
#pragma unroll
        for (int e = 0; e < 4; e++) acc[e] += d[e] * d[4 + e];
      } else {
        const float v[4] = {x.x, x.y, x.z, x.w};
        double d[4];
        f2d(v, d);
#pragma unroll
        for (int e = 0; e < 4; e++) acc[e] += d[e];
      }
    }
    i0 = (n4 << 2) + t;
  }
  for (long long i = i0; i < n; i += stride) acc[0] += (double)a[i] * (b ? (double)b[i] : 1.0);
  double v = block_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
  __shared__ bool last;
  if (threadIdx.x == 0) {
    partials[blockIdx.x] = v;
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;   // uniform for the block
  __threadfence();
  v = 0.0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) v += __ldcg(partials + i);
  __syncthreads();     // block_sum's shared array again
  v = block_sum(v);
  if (threadIdx.x == 0) {
    *out = v;
    *done = 0u;
  }
}

// ---- elementwise operations on N elements at a time, y = op(y, x1, x2) ----
struct OpFill {
  float v;
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&)[N], const float (&)[N]) const {
#pragma unroll
    for (int i = 0; i < N; i++) y[i] = v;
  }
};
// y = y*a (hypercube_float::scale)
struct OpScale {
  double a;
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&)[N], const float (&)[N]) const {
    double d[N];
    f2d(y, d);
#pragma unroll
    for (int i = 0; i < N; i++) d[i] *= a;
    d2f(d, y);
  }
};
// y = y*a + x*b  (hypercube_float::scale_add(a, x, b): vals = vals*a + b*x,
// Born/hypercube_float.cpp:437-443; evaluated in double as the reference does)
struct OpScaleAdd {
  double a, b;
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&x)[N], const float (&)[N]) const {
    double d[N], e[N];
    f2d(y, d);
    f2d(x, e);
#pragma unroll
    for (int i = 0; i < N; i++) d[i] = d[i] * a + b * e[i];
    d2f(d, y);
  }
};
// y = x1*a + x2*b  (the four-argument scale_add, :368-378)
struct OpScaleAdd2 {
  double a, b;
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&x1)[N], const float (&x2)[N]) const {
    double d[N], e[N];
    f2d(x1, d);
    f2d(x2, e);
#pragma unroll
    for (int i = 0; i < N; i++) d[i] = d[i] * a + e[i] * b;
    d2f(d, y);
  }
};
struct OpAdd {
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&x)[N], const float (&)[N]) const {
#pragma unroll
    for (int i = 0; i < N; i++) y[i] = y[i] + x[i];
  }
};
struct OpMult {
  template <int N>
  __device__ void operator()(float (&y)[N], const float (&x)[N], const float (&)[N]) const {
#pragma unroll
    for (int i = 0; i < N; i++) y[i] = y[i] * x[i];
  }
};

// A thread takes U * W elements a step, W neighbours per access (4: every
// pointer 16-byte aligned), U accesses a grid's width apart; then W at a time,
// then, past the last four, one.
template <int W, int U, bool Y, bool X1, bool X2, class OP>
__global__ void __launch_bounds__(256) map_kernel(float *y, const float *x1, const float *x2, long long n, OP op) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x, stride = (long long)gridDim.x * blockDim.x;
  const long long nu = n / W;
  auto load = [](const float *p, long long k, float *v) {
    if constexpr (W == 4) {
      const float4 q = reinterpret_cast<const float4 *>(p)[k];
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
      v[0] = p[k];
    }
  };
  auto store = [](float *p, long long k, const float *v) {
    if constexpr (W == 4)
      reinterpret_cast<float4 *>(p)[k] = make_float4(v[0], v[1], v[2], v[3]);
    else
      p[k] = v[0];
  };
  long long i = t;
  if constexpr (U > 1) {
    for (; i + (U - 1) * stride < nu; i += U * stride) {
      float v[U * W] = {}, p[U * W] = {}, q[U * W] = {};
#pragma unroll
      for (int h = 0; h < U; h++) {
        if (Y) load(y, i + h * stride, v + W * h);
        if (X1) load(x1, i + h * stride, p + W * h);
        if (X2) load(x2, i + h * stride, q + W * h);
      }
      op(v, p, q);
#pragma unroll
      for (int h = 0; h < U; h++) store(y, i + h * stride, v + W * h);
    }
  }
  for (; i < nu; i += stride) {
    float v[W] = {}, p[W] = {}, q[W] = {};
    if (Y) load(y, i, v);
    if (X1) load(x1, i, p);
    if (X2) load(x2, i, q);
    op(v, p, q);
    store(y, i, v);
  }
  if constexpr (W > 1) {
    for (long long k = nu * W + t; k < n; k += stride) {
      float v[1] = {Y ? y[k] : 0.f};
      const float p[1] = {X1 ? x1[k] : 0.f}, q[1] = {X2 ? x2[k] : 0.f};
      op(v, p, q);
      y[k] = v[0];
    }
  }
}

// uniform(-0.5, 0.5) from a counter hash (splitmix64) of (seed, index)
__global__ void random_kernel(float *y, long long n, unsigned long long seed) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    y[i] = (float)((double)(z >> 11) * (1.0 / 9007199254740992.0) - 0.5);
  }
}

static bool al16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static int grid_for(long long n) {
  long long g = (n + 255) / 256;
  return (int)(g < 2048 ? (g < 1 ? 1 : g) : 2048);
}

// Eight elements a thread and step keep the conversions' slow path a real
// branch and the loads of a step in flight, 16 bytes at a time where the
// pointers allow; shorter vectors take one element a thread, as eight would
// leave most SMs, and their FP64 pipes, idle.  Measured (one -> eight, us; y =
// a x1 + b x2): 5000 elements 3.3 -> 6.1, 180 000 4.1 -> 6.1, 262 144 6.1 ->
// 5.1, 3 M 26.7 -> 16.4, 60 M 472 -> 252; not 16-byte aligned 400 000 6.1 ->
// 8.2, 600 000 8.2 -> 8.2, 3 M 26.7 -> 18.5, 60 M 471 -> 252.  (Unaligned
// vectors in the eights' kernel one element at a time: y += x of 60 M 336 us,
// half the warps of a kernel of its own, 166; 128 so.)
template <bool Y, bool X1, bool X2, class OP>
static cudaError_t map(float *y, const float *x1, const float *x2, long long n, OP op, cudaStream_t st) {
  const bool al = al16(y) && (!X1 || al16(x1)) && (!X2 || al16(x2));
  const bool eights = n >= (al ? 1LL << 18 : 1LL << 19);
  const int grid = grid_for(eights ? (n + 7) / 8 : n);
  if (!eights)
    map_kernel<1, 1, Y, X1, X2><<<grid, 256, 0, st>>>(y, x1, x2, n, op);
  else if (al)
    map_kernel<4, 2, Y, X1, X2><<<grid, 256, 0, st>>>(y, x1, x2, n, op);
  else
    map_kernel<1, 8, Y, X1, X2><<<grid, 256, 0, st>>>(y, x1, x2, n, op);
  return cudaGetLastError();
}

// scratch: vec_dot_scratch_doubles() doubles (partials, then the counter,
// which must be zero before the first call)
cudaError_t vec_dot(const float *a, const float *b, long long n, double *scratch, double *out, cudaStream_t st) {
  unsigned int *done = reinterpret_cast<unsigned int *>(scratch + kDotBlocks);
  // at least eight elements per thread: few blocks for short vectors, whose
  // partials the last block waits for
  const long long want = (n + 8 * kDotThreads - 1) / (8 * kDotThreads);
  const int blocks = (int)(want < 1 ? 1 : (want > kDotBlocks ? kDotBlocks : want));
  if (al16(a) && al16(b))
    dot_kernel<true><<<blocks, kDotThreads, 0, st>>>(a, b, n, scratch, done, out);
  else
    dot_kernel<false><<<blocks, kDotThreads, 0, st>>>(a, b, n, scratch, done, out);
  return cudaGetLastError();
}

int vec_dot_scratch_doubles() { return kDotBlocks + 1; }

cudaError_t vec_fill(float *x, long long n, float v, cudaStream_t st) {
  return map<false, false, false>(x, nullptr, nullptr, n, OpFill{v}, st);
}
cudaError_t vec_scale(float *y, long long n, double a, cudaStream_t st) {
  return map<true, false, false>(y, nullptr, nullptr, n, OpScale{a}, st);
}
cudaError_t vec_scale_add(float *y, const float *x, long long n, double a, double b, cudaStream_t st) {
  return map<true, true, false>(y, x, nullptr, n, OpScaleAdd{a, b}, st);
}
cudaError_t vec_scale_add2(float *y, const float *x1, const float *x2, long long n, double a, double b,
                           cudaStream_t st) {
  return map<false, true, true>(y, x1, x2, n, OpScaleAdd2{a, b}, st);
}
cudaError_t vec_add(float *y, const float *x, long long n, cudaStream_t st) {
  return map<true, true, false>(y, x, nullptr, n, OpAdd{}, st);
}
cudaError_t vec_mult(float *y, const float *x, long long n, cudaStream_t st) {
  return map<true, true, false>(y, x, nullptr, n, OpMult{}, st);
}
cudaError_t vec_random(float *y, long long n, unsigned long long seed, cudaStream_t st) {
  random_kernel<<<grid_for(n), 256, 0, st>>>(y, n, seed);
  return cudaGetLastError();
}

}  // namespace sepx
