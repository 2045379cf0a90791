// band.cuh -- edge bands and boundary pre-images for the adjoint kernels.
//
// A tile path that takes groups of four horizontally adjacent pixels whose
// taps stay inside the image leaves out a band of radius R along the edges:
// rows [0, R) and [H-R, H) whole, then, for the rows in between, columns
// [0, L) and [W-wr, W) with L = R rounded up to 4 and wr = W - 4 floor((W -
// R) / 4) (the image must be wide enough that the two do not meet).  Those pixels go
// through the boundary's pre-images one pixel per thread, from a flat list of
// the batch's band pixels that every CTA takes an equal contiguous share of.
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

__host__ __device__ __forceinline__ int band_left(int R) { return (R + 3) / 4 * 4; }
__host__ __device__ __forceinline__ int band_right(int W, int R) { return W - 4 * ((W - R) / 4); }
__host__ __device__ __forceinline__ int band_size(int W, int H, int R) {
  return 2 * R * W + (H - 2 * R) * (band_left(R) + band_right(W, R));
}
__device__ __forceinline__ void band_pos(int k, int W, int H, int R, int &y, int &x) {
  if (k < 2 * R * W) {
    const int yy = k / W;
    x = k - yy * W;
    y = yy < R ? yy : H - 2 * R + yy;
    return;
  }
  k -= 2 * R * W;
  const int L = band_left(R), mid = (H - 2 * R) * L;
  if (k < mid) {
    y = R + k / L;
    x = k - (y - R) * L;
    return;
  }
  k -= mid;
  const int wr = band_right(W, R);
  const int yy = k / wr;
  y = R + yy;
  x = W - wr + (k - yy * wr);
}

// the contiguous share of n band entries that this CTA takes
__device__ __forceinline__ void cta_share(int64_t n, int64_t &k0, int64_t &k1) {
  k0 = n * blockIdx.x / gridDim.x;
  k1 = n * (blockIdx.x + 1) / gridDim.x;
}

// per-axis pre-images of index j under the remap, among virtual positions
// within `rad` of the image: at most 1 + rad entries
__device__ __forceinline__ int preimages(int mode, int j, int n, int rad, int *out) {
  int k = 0;
  out[k++] = j;
  if (mode == HGB_BOUNDARY_CONSTANT || (j >= rad && j < n - rad)) return k;
  for (int v = -rad; v < 0; ++v)
    if (remap(mode, v, 0, n) == j) out[k++] = v;
  for (int v = n; v < n + rad; ++v)
    if (remap(mode, v, 0, n) == j) out[k++] = v;
  return k;
}

// The same pre-images, besides j itself, as bits: bit t < R stands for the
// virtual position t - R, bit t >= R for n + t - R (no tap reaches farther).
template <int R>
__device__ __forceinline__ unsigned preimage_bits(int mode, int j, int n) {
  if (mode == HGB_BOUNDARY_CONSTANT || (j >= R && j < n - R)) return 0;
  unsigned m = 0;
  if (n >= R) {  // no position is remapped twice
    if (mode == HGB_BOUNDARY_MIRROR) {  // -1 - j, 2n - 1 - j
      if (j < R) m = 1u << (R - 1 - j);
      if (n - 1 - j < R) m |= 1u << (R + n - 1 - j);
    } else if (mode == HGB_BOUNDARY_REPEAT) {  // j - n, j + n
      if (n - j <= R) m = 1u << (R + j - n);
      if (j < R) m |= 1u << (R + j);
    } else {
      if (j == 0) m = (1u << R) - 1u;
      if (j == n - 1) m |= ((1u << R) - 1u) << R;
    }
    return m;
  }
#pragma unroll 1
  for (int t = 0; t < R; ++t) {
    if (remap(mode, t - R, 0, n) == j) m |= 1u << t;
    if (remap(mode, n + t, 0, n) == j) m |= 1u << (R + t);
  }
  return m;
}
template <int R>
__device__ __forceinline__ int preimage_pos(int t, int n) { return t < R ? t - R : n + t - R; }

// Band pixels (within R of an edge of the image) of a tw x th tile at (i0, j0),
// for a CTA to take one per thread.
struct TileBand {
  int tw, th, top, bottom, left, right, count;
};
template <int R>
__device__ __forceinline__ TileBand tile_band(int i0, int j0, int tw, int th, int W, int H, bool rows, bool cols) {
  TileBand b;
  b.tw = min(tw, W - i0);
  b.th = min(th, H - j0);
  b.top = rows ? min(b.th, max(0, R - j0)) : 0;
  b.bottom = rows ? min(b.th - b.top, max(0, j0 + b.th - (H - R))) : 0;
  b.left = cols ? min(b.tw, max(0, R - i0)) : 0;
  b.right = cols ? min(b.tw - b.left, max(0, i0 + b.tw - (W - R))) : 0;
  b.count = (b.top + b.bottom) * b.tw + (b.th - b.top - b.bottom) * (b.left + b.right);
  return b;
}
__device__ __forceinline__ void tile_band_pos(const TileBand &b, int k, int &x, int &y) {  // tile-relative
  const int full = (b.top + b.bottom) * b.tw;
  if (k < full) {
    y = k / b.tw;
    x = k - y * b.tw;
    if (y >= b.top) y += b.th - b.top - b.bottom;
    return;
  }
  const int n = b.left + b.right, d = k - full;
  y = d / n;
  x = d - y * n;
  y += b.top;
  if (x >= b.left) x += b.tw - n;
}

}  // namespace hgb
