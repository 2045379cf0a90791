// line_k11_15.cu -- tiled line adjoint kernels for K = 11, 13, 15 (line_adjoint_kernels.cuh).
#include "line_adjoint_kernels.cuh"

namespace hgb {
template LineKernel line_kernel_k<11>(LineForm, bool, int);
template LineKernel line_kernel_k<13>(LineForm, bool, int);
template LineKernel line_kernel_k<15>(LineForm, bool, int);
}  // namespace hgb
