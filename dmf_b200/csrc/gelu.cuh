// GELU (tanh form) of the transformer block's MLP with its tangent, and its primal backward.
//
//   s(x) = 1 / (1 + exp(-2 u)),  u = sqrt(2 / pi) (x + 0.044715 x^3)        gelu(x)  = x s
//                                                                            gelu'(x) = s + 2 x u' s (1 - s)
//   y = gelu(x)        ty = gelu'(x) tx        dx = gelu'(x) dy
//
// (0.5 (1 + tanh u) = s: the logistic form has no cancellation for negative x and takes one exponential and one reciprocal.)
// What bounds it: HBM.  The tensors are the widest of the model (4 C per token) and nothing is computed between them.  Each
// thread has kGeluVecs 16-byte loads of each tensor in flight and ends: a grid-stride loop over 4 to 8 blocks per SM is 10 to
// 15 % slower.  8192 x 4608 bf16 with L2 flushed (75 MB a tensor), of the measured copy rate: y alone 29 us (0.79), y and ty
// 53 us (0.87), backward 41 us (0.84); the library's kernels take 39, 39 + 50 and 50 us.
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

__device__ __forceinline__ float gelu_s(float x) {
  const float z = x * fmaf(x * x, -2.f * 0.7978845608028654f * 0.044715f, -2.f * 0.7978845608028654f);  // -2 u
  return __fdividef(1.f, 1.f + __expf(z));
}
__device__ __forceinline__ float gelu_grad(float x, float s) {
  const float du2 = fmaf(x * x, 6.f * 0.7978845608028654f * 0.044715f, 2.f * 0.7978845608028654f);  // 2 u'
  return fmaf(x * du2, s * (1.f - s), s);
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
      const float s = gelu_s(a[j]);
      if constexpr (kT) b[j] *= gelu_grad(a[j], s);
      a[j] *= s;
    }
    if constexpr (kY) store8(reinterpret_cast<T*>(p.y) + 8 * i, a);
    if constexpr (kT) store8(reinterpret_cast<T*>(p.ty) + 8 * i, b);
  }
  if (blockIdx.x == 0 && threadIdx.x < p.tail) {
    const int64_t i = 8 * p.n8 + threadIdx.x;
    const float a = static_cast<float>(reinterpret_cast<const T*>(p.x)[i]);
    const float s = gelu_s(a);
    float b = 0.f;
    if constexpr (kT) b = gelu_grad(a, s) * static_cast<float>(reinterpret_cast<const T*>(p.t)[i]);
    if constexpr (kY) reinterpret_cast<T*>(p.y)[i] = static_cast<T>(a * s);
    if constexpr (kT) reinterpret_cast<T*>(p.ty)[i] = static_cast<T>(b);
  }
}

}  // namespace dmf
