// lmm_bf16.cu -- tiled MIN / MAX kernels for bf16 storage (local_minmax_kernels.cuh).
#include "local_minmax_kernels.cuh"

namespace hgb {
template int launch_minmax_k<__nv_bfloat16>(const MinMaxKernelParams &, int, cudaStream_t);
}  // namespace hgb
