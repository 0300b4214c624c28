// GELU (tanh form) of the transformer block's MLP with its tangent, and its primal backward.
//
//   u(x) = sqrt(2 / pi) (x + 0.044715 x^3),  h = tanh u                     gelu(x)  = 0.5 x (1 + h)
//                                                                           gelu'(x) = 0.5 (1 + h) + 0.5 x (1 - h^2) u'
//   y = gelu(x)        ty = gelu'(x) tx        dx = gelu'(x) dy
//
// The arithmetic is pinned operation by operation (which products are fused into sums): every 16-bit result is the library's
// bit for bit, so a model gives the same outputs whichever of the two runs, limits and overflows included.  (The logistic
// form x / (1 + exp(-2 u)) is shorter, 10 us on y alone and 6 us on the backward below, but rounds differently, and its
// derivative is NaN where x^3 overflows and gelu' is 0 or 1.)
// What bounds it: HBM, and for y alone tanhf.  The tensors are the widest of the model (4 C per token).  Each thread has
// kGeluVecs 16-byte loads of each tensor in flight and ends: a grid-stride loop over 4 to 8 blocks per SM is 10 to 15 %
// slower.  8192 x 4608 bf16 with L2 flushed (75 MB a tensor), of the measured copy rate: y alone 39 us (0.59), y and ty
// 53 us (0.87), backward 47 us (0.74); the library's kernels take 43, 43 + 53 and 53 us.
#pragma once

#include <stdint.h>

#include "vec8.cuh"

namespace dmf {

struct GeluParams {
  const void* x;
  const void* t;   // tangent (forward) / dy (backward); nullptr: plain forward
  void* y;         // y (forward) / nullptr (backward)
  void* ty;        // ty (forward) / dx (backward)
  int64_t n8;      // whole 8-element vectors
  int tail;        // elements after them
};

constexpr int kGeluThreads = 256;
constexpr int kGeluVecs = 4;

constexpr float kGeluC = 0.7978845608028654f;  // sqrt(2 / pi)
constexpr float kGeluK = 0.044715f;

// tanh u(x)
__device__ __forceinline__ float gelu_tanh(float x) {
  const float cube = __fmul_rn(__fmul_rn(x, x), x);
  return tanhf(__fmul_rn(kGeluC, fmaf(kGeluK, cube, x)));
}
// h = tanh u(x)
__device__ __forceinline__ float gelu_value(float x, float h) { return __fmul_rn(__fmul_rn(0.5f, x), __fadd_rn(1.f, h)); }
__device__ __forceinline__ float gelu_grad(float x, float h) {
  const float du = __fmul_rn(kGeluC, fmaf(3.f * kGeluK, __fmul_rn(x, x), 1.f));
  const float right = __fmul_rn(__fmul_rn(0.5f, x), fmaf(-h, h, 1.f));
  return fmaf(right, du, __fmul_rn(0.5f, __fadd_rn(1.f, h)));
}

// kY: writes gelu(x); kT: writes gelu'(x) t
template <typename T, bool kY, bool kT>
__global__ void __launch_bounds__(kGeluThreads) gelu_kernel(const GeluParams p) {
  const uint4* x = reinterpret_cast<const uint4*>(p.x);
  const uint4* t = reinterpret_cast<const uint4*>(p.t);
  const int64_t i0 = static_cast<int64_t>(blockIdx.x) * (kGeluThreads * kGeluVecs) + threadIdx.x;
  uint4 xv[kGeluVecs], tv[kGeluVecs];
#pragma unroll
  for (int u = 0; u < kGeluVecs; ++u) {
    const int64_t i = i0 + u * kGeluThreads;
    if (i >= p.n8) continue;
    xv[u] = x[i];  // plain loads: the outputs may be the inputs
    if constexpr (kT) tv[u] = t[i];
  }
#pragma unroll
  for (int u = 0; u < kGeluVecs; ++u) {
    const int64_t i = i0 + u * kGeluThreads;
    if (i >= p.n8) continue;
    float a[8], b[8];
    unpack8<T>(xv[u], a);
    if constexpr (kT) unpack8<T>(tv[u], b);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float h = gelu_tanh(a[j]);
      if constexpr (kT) b[j] *= gelu_grad(a[j], h);
      if constexpr (kY) a[j] = gelu_value(a[j], h);
    }
    if constexpr (kY) store8(reinterpret_cast<T*>(p.y) + 8 * i, a);
    if constexpr (kT) store8(reinterpret_cast<T*>(p.ty) + 8 * i, b);
  }
  if (blockIdx.x == 0 && threadIdx.x < p.tail) {
    const int64_t i = 8 * p.n8 + threadIdx.x;
    const float a = static_cast<float>(reinterpret_cast<const T*>(p.x)[i]);
    const float h = gelu_tanh(a);
    float b = 0.f;
    if constexpr (kT) b = gelu_grad(a, h) * static_cast<float>(reinterpret_cast<const T*>(p.t)[i]);
    if constexpr (kY) reinterpret_cast<T*>(p.y)[i] = static_cast<T>(gelu_value(a, h));
    if constexpr (kT) reinterpret_cast<T*>(p.ty)[i] = static_cast<T>(b);
  }
}

}  // namespace dmf
