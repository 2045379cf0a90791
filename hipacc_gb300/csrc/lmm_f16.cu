// lmm_f16.cu -- tiled MIN / MAX kernels for f16 storage (local_minmax_kernels.cuh).
#include "local_minmax_kernels.cuh"

namespace hgb {
template int launch_minmax_k<__half>(const MinMaxKernelParams &, int, cudaStream_t);
}  // namespace hgb
