// line_k3_9.cu -- tiled line adjoint kernels for K = 3, 5, 7, 9 (line_adjoint_kernels.cuh).
#include "line_adjoint_kernels.cuh"

namespace hgb {
template LineKernel line_kernel_k<3>(LineForm, bool, int);
template LineKernel line_kernel_k<5>(LineForm, bool, int);
template LineKernel line_kernel_k<7>(LineForm, bool, int);
template LineKernel line_kernel_k<9>(LineForm, bool, int);
}  // namespace hgb
