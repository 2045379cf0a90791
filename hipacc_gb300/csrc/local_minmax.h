// local_minmax.h -- tiled MIN / MAX over a Domain (local_minmax.cu).
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

// Row structure of a Domain of up to 7 x 7 cells whose every row is empty or
// one run centred on the window: sel[h] has bit y set when row y of the K x K
// window is the run of half-width h.  Returns false for other domains.
struct MinMaxDomain {
  int k;               // 3, 5 or 7
  uint32_t sel[4];     // rows (bits) of half-width 0 .. 3
  uint32_t rows[7];    // the cells of each row (bit x), for the ordered fold
};
bool minmax_domain(const uint8_t *domain, int mw, int mh, MinMaxDomain *out);

// out(is) = MIN / MAX over the domain; in and out of one storage type
int run_minmax_domain(const hgb_view &in, const hgb_window &acc, const hgb_view &out, const hgb_window &is,
                      const MinMaxDomain &d, int reduce, int boundary, float cval, cudaStream_t st);

struct MinMaxKernelParams {
  const char *in;
  int64_t in_pitch, in_bstride;
  char *out;
  int64_t out_pitch, out_bstride;
  int ax, ay, aw, ah;  // accessor window
  int ix, iy, iw, ih;  // iteration space
  int bmode, vec_out;
  float cval;
  int excess;          // how far the iteration space exceeds the accessor window
  uint32_t flip;       // 0x80000000 for MAX: values and result change sign
  MinMaxDomain d;
};
template <typename TI>
int launch_minmax_k(const MinMaxKernelParams &p, int batch, cudaStream_t st);  // lmm_*.cu

}  // namespace hgb
