// conv_adjoint.h -- adjoint of the SUM local operator with a 3 x 3, 5 x 5 or 7 x 7
// mask on tiles (conv_adjoint.cu).
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

struct ConvAdjParams {
  const float *in, *gout;                            // in may be null without part
  float *gin;                                        // may be null
  int64_t in_p, in_b, gout_p, gout_b, gin_p, gin_b;  // bytes
  int w, h, batch, bmode;
  int tiles_x, tiles_y, ntiles;
  const float *mask_dev;                             // K x K taps on the device, or null
  float mask[49];
  double *part;                                      // [taps][CTAs] partials of the mask gradient, or null
};

bool conv_adjoint_size(int k);  // 3, 5 or 7
int conv_adjoint_grid(int k, int w, int h, int batch);  // CTAs of a launch (the partials per tap)
int run_conv_adjoint(int k, ConvAdjParams *p, int grid, cudaStream_t st);

}  // namespace hgb
