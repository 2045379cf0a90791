// lmm_u8.cu -- tiled MIN / MAX kernels for u8 storage (local_minmax_kernels.cuh).
#include "local_minmax_kernels.cuh"

namespace hgb {
template int launch_minmax_k<uint8_t>(const MinMaxKernelParams &, int, cudaStream_t);
}  // namespace hgb
