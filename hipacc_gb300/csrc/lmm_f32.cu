// lmm_f32.cu -- tiled MIN / MAX kernels for f32 storage (local_minmax_kernels.cuh).
#include "local_minmax_kernels.cuh"

namespace hgb {
template int launch_minmax_k<float>(const MinMaxKernelParams &, int, cudaStream_t);
}  // namespace hgb
