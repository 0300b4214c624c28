// Launches of attn_fwd_duo_kernel (attn_fwd_duo.cuh).
#include "attn_fwd_duo.cuh"

#include "attn_launch.h"

namespace dmf {
namespace {

template <typename T, int TAIL, bool kCubics>
int launch_inst(const FwdParams& p, int grid, cudaStream_t stream) {
  static bool done[64];
  auto kernel = attn_fwd_duo_kernel<T, TAIL, kCubics>;
  if (!allow_smem(kernel, DuoTraits<TAIL>::kSmemBytes, done)) return DMF_ATTN_ERR_LAUNCH;
  kernel<<<grid, kDuoThreads, DuoTraits<TAIL>::kSmemBytes, stream>>>(p);
  return cudaGetLastError() == cudaSuccess ? DMF_ATTN_OK : DMF_ATTN_ERR_LAUNCH;
}

template <typename T, int TAIL>
int launch(const FwdParams& p, int grid, cudaStream_t stream) {
  if constexpr (duo_cubics(TAIL, 2)) {
    if (duo_cubics(TAIL, p.num_q_tiles)) return launch_inst<T, TAIL, true>(p, grid, stream);
  }
  return launch_inst<T, TAIL, false>(p, grid, stream);
}

template <typename T>
int launch_tail(const FwdParams& p, int tail, int grid, cudaStream_t stream) {
  switch (tail) {
    case 0: return launch<T, 0>(p, grid, stream);
    case 16: return launch<T, 16>(p, grid, stream);
    case 32: return launch<T, 32>(p, grid, stream);
    case 64: return launch<T, 64>(p, grid, stream);
    default: return DMF_ATTN_ERR_HEAD_DIM;
  }
}

}  // namespace

int launch_fwd_duo(const FwdParams& p, int tail, int dtype, int grid, cudaStream_t stream) {
  return dtype == DMF_ATTN_BF16 ? launch_tail<__nv_bfloat16>(p, tail, grid, stream)
                                : launch_tail<__half>(p, tail, grid, stream);
}

}  // namespace dmf
