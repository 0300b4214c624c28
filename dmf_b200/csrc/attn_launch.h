// Launchers of the attention kernels that live in translation units of their own (dmf_attn.cu picks between them).
#pragma once

#include <cuda_runtime.h>

#include "dmf_attn.h"

namespace dmf {

struct FwdParams;

// Opts a kernel into `bytes` of dynamic shared memory, once per device instead of once per launch.
template <typename Kernel>
inline bool allow_smem(Kernel kernel, int bytes, bool (&done)[64]) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
  if (__atomic_load_n(&done[dev], __ATOMIC_ACQUIRE)) return true;  // (threads that race here all set the same attribute)
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  __atomic_store_n(&done[dev], true, __ATOMIC_RELEASE);
  return true;
}

// attn_fwd_duo.cu: plain forward, two query tiles per CTA
int launch_fwd_duo(const FwdParams& p, int tail, int dtype, int grid, cudaStream_t stream);

}  // namespace dmf
