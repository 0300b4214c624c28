// Eight 16-bit elements (16 bytes) at a time: loads, conversion to fp32 and back.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "sm100_ptx.cuh"

namespace dmf {

__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {  // read-once data: no L1 allocation
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

template <typename T>
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = unpack2<T>(u[i]);
    f[2 * i] = a.x;
    f[2 * i + 1] = a.y;
  }
}

template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&f)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(Pack2<T>::pack(f[0], f[1]), Pack2<T>::pack(f[2], f[3]),
                                            Pack2<T>::pack(f[4], f[5]), Pack2<T>::pack(f[6], f[7]));
}

}  // namespace dmf
