// line_adjoint.h -- adjoint of a 1 x K or K x 1 SUM operator on tiles (line_adjoint.cu).
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

struct LineAdjParams {
  const float *in, *gout;                            // in may be null without part
  float *gin;                                        // may be null
  int64_t in_p, in_b, gout_p, gout_b, gin_p, gin_b;  // bytes
  int w, h, batch, bmode;
  int tiles_x, tiles_y, ntiles;
  const float *mask_dev;                             // taps on the device, or null
  float mask[15];
  float cval;
  float row[15];                                     // row taps that recompute t (column form of the separable filter)
  double *part;                                      // [taps][CTAs] partials of the tap gradient, or null
};

enum LineForm { kLineRow = 0, kLineCol = 1, kLineColOfRows = 2 };

bool line_adjoint_size(int k);  // K has a tiled kernel
// CTAs of a launch (the partials per tap)
int line_adjoint_grid(LineForm form, int k, bool mask_dev, int w, int h, int batch);
int run_line_adjoint(LineForm form, int k, LineAdjParams *p, int grid, cudaStream_t st);

constexpr int LN_NT = 128, LN_TW = 64;  // threads, tile width
using LineKernel = void (*)(LineAdjParams);
template <int K>
LineKernel line_kernel_k(LineForm f, bool dev, int py);  // line_k*.cu; py rows per thread, 4 or 1

struct LineCombine {  // up to two tap gradients, summed in FP64 in a fixed order
  const double *part[2];
  float *out[2];
  int taps[2], nparts[2];
};
int run_line_combine(const LineCombine &c, cudaStream_t st);

}  // namespace hgb
