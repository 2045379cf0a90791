// local_minmax.cu -- dispatch of the tiled MIN / MAX over a Domain
// (local_minmax_kernels.cuh).
#include <algorithm>
#include <cstring>

#include "local_minmax.h"

namespace hgb {

bool minmax_domain(const uint8_t *domain, int mw, int mh, MinMaxDomain *out) {
  int k = mw > mh ? mw : mh;
  if (k % 2 == 0) ++k;
  if (k < 3) k = 3;
  if (k > 7 || !domain) return false;
  memset(out, 0, sizeof(*out));
  out->k = k;
  // cell (x, y) of the given window sits at offset (x - mw/2, y - mh/2)
  const int r = k / 2, dx = r - mw / 2, dy = r - mh / 2;
  for (int y = 0; y < mh; ++y)
    for (int x = 0; x < mw; ++x)
      if (domain[y * mw + x]) out->rows[y + dy] |= 1u << (x + dx);
  for (int y = 0; y < k; ++y) {
    const uint32_t bits = out->rows[y];
    if (!bits) continue;
    int h = 0;
    while (h <= r && bits != (((1u << (2 * h + 1)) - 1u) << (r - h))) ++h;
    if (h > r) return false;
    out->sel[h] |= 1u << y;
  }
  return true;
}

int run_minmax_domain(const hgb_view &in, const hgb_window &acc, const hgb_view &out, const hgb_window &is,
                      const MinMaxDomain &d, int reduce, int boundary, float cval, cudaStream_t st) {
  MinMaxKernelParams p;
  memset(&p, 0, sizeof(p));
  const int es = dtype_size(out.dtype);
  p.in = (const char *)in.data;
  p.in_pitch = in.pitch;
  p.in_bstride = in.batch_stride;
  p.out = (char *)out.data;
  p.out_pitch = out.pitch;
  p.out_bstride = out.batch_stride;
  p.ax = acc.offset_x;
  p.ay = acc.offset_y;
  p.aw = acc.width;
  p.ah = acc.height;
  p.ix = is.offset_x;
  p.iy = is.offset_y;
  p.iw = is.width;
  p.ih = is.height;
  p.bmode = boundary;
  p.cval = cval;
  p.excess = std::max(0, std::max(is.width - acc.width, is.height - acc.height));
  p.flip = reduce == HGB_REDUCE_MAX ? 0x80000000u : 0u;
  p.d = d;
  const int64_t four = 4 * es;  // bytes of a thread's four outputs
  p.vec_out = ((uintptr_t)out.data + (uintptr_t)is.offset_x * es) % four == 0 && out.pitch % four == 0 &&
              (out.batch == 1 || out.batch_stride % four == 0);
  switch (in.dtype) {
    case HGB_F32: return launch_minmax_k<float>(p, in.batch, st);
    case HGB_BF16: return launch_minmax_k<__nv_bfloat16>(p, in.batch, st);
    case HGB_F16: return launch_minmax_k<__half>(p, in.batch, st);
    case HGB_U8: return launch_minmax_k<uint8_t>(p, in.batch, st);
  }
  return set_error(HGB_ERR_UNSUPPORTED, "local_op: storage type");
}

}  // namespace hgb
