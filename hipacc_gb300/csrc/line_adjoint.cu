// line_adjoint.cu -- dispatch of the tiled line adjoints (line_adjoint_kernels.cuh)
// and the FP64 combine of their tap gradients.
#include <algorithm>
#include <cstring>

#include "line_adjoint.h"

namespace hgb {
namespace {

// one CTA per tap: the partials in FP64, strided over the threads, then a fixed tree
__global__ void __launch_bounds__(256) line_combine_kernel(const __grid_constant__ LineCombine c) {
  __shared__ double sh[256];
  int o = blockIdx.x, a = 0;
  if (o >= c.taps[0]) {
    o -= c.taps[0];
    a = 1;
  }
  double s = 0.0;
  for (int k = threadIdx.x; k < c.nparts[a]; k += 256) s += __ldcg(c.part[a] + (size_t)o * c.nparts[a] + k);
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int d = 128; d > 0; d >>= 1) {
    if (threadIdx.x < d) sh[threadIdx.x] += sh[threadIdx.x + d];
    __syncthreads();
  }
  if (threadIdx.x == 0) c.out[a][o] = (float)sh[0];
}

LineKernel line_kernel(LineForm f, int k, bool dev, int py) {
  switch (k) {
    case 3: return line_kernel_k<3>(f, dev, py);
    case 5: return line_kernel_k<5>(f, dev, py);
    case 7: return line_kernel_k<7>(f, dev, py);
    case 9: return line_kernel_k<9>(f, dev, py);
    case 11: return line_kernel_k<11>(f, dev, py);
    case 13: return line_kernel_k<13>(f, dev, py);
    case 15: return line_kernel_k<15>(f, dev, py);
  }
  return nullptr;
}

}  // namespace

bool line_adjoint_size(int k) { return k >= 3 && k <= 15 && (k & 1); }

// rows per thread: 4, or 1 where 32-row tiles would leave an SM fewer than four
// CTAs (two 139 x 274 images, K = 7, forward and adjoint as one graph: 27 -> 19 us)
static int line_rows(int w, int h, int batch) {
  return (int64_t)cdiv(w, LN_TW) * cdiv(h, 32) * batch >= 4 * num_sms() ? 4 : 1;
}

int line_adjoint_grid(LineForm form, int k, bool mask_dev, int w, int h, int batch) {
  const int py = line_rows(w, h, batch);
  const int64_t tiles = (int64_t)cdiv(w, LN_TW) * cdiv(h, 8 * py) * batch;
  const int wave = num_sms() * resident_ctas((const void *)line_kernel(form, k, mask_dev, py), LN_NT, 0);
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, wave));
}

int run_line_adjoint(LineForm form, int k, LineAdjParams *p, int grid, cudaStream_t st) {
  const int py = line_rows(p->w, p->h, p->batch);
  p->tiles_x = cdiv(p->w, LN_TW);
  p->tiles_y = cdiv(p->h, 8 * py);
  const int64_t tiles = (int64_t)p->tiles_x * p->tiles_y * p->batch;
  HGB_REQUIRE(tiles < 0x7fffffff, "line adjoint: too many tiles");
  p->ntiles = (int)tiles;
  line_kernel(form, k, p->mask_dev != nullptr, py)<<<grid, LN_NT, 0, st>>>(*p);
  return HGB_OK;
}

int run_line_combine(const LineCombine &c, cudaStream_t st) {
  line_combine_kernel<<<c.taps[0] + c.taps[1], 256, 0, st>>>(c);
  return HGB_OK;
}

}  // namespace hgb
