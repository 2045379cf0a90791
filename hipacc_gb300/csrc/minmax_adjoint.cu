// minmax_adjoint.cu -- hgb_local_op_minmax_adjoint: the adjoint of the MIN /
// MAX local operator, Kernel::reduce(Domain, Reduce::MIN/MAX) and
// Kernel::convolve(mask, Reduce::MIN/MAX) (dsl/kernel.hpp:241-315;
// lib/AST/Convolution.cpp:43-100: acc starts at FLT_MAX / FLT_MIN and takes
// acc = acc < v ? acc : v (MIN) or acc > v ? acc : v (MAX) per tap in
// row-major order, v = m * x for convolve, x for a Domain).
//
// Each output's value came from one tap: the last one whose update replaced
// the running value (on a tie the later tap replaces, as the forward's
// expression does).  Its gradient goes to the pixel that tap read, times the
// mask weight for convolve.  Nothing flows when the initial value was never
// replaced, or when the winning tap read the CONSTANT value outside the image.
//
// Two kernels, deterministic, for any window (minmax_select_kernel,
// minmax_gather_kernel) and on tiles for Domains of up to 7 x 7 cells
// (minmax_select_tile_kernel, minmax_gather_tile_kernel):
//   1. select: per output, the winning tap (0 .. taps-1) or 0xFF,
//      into a byte per output in the library workspace;
//   2. gather: per input pixel, the sum over every (virtual
//      position that the boundary remap sends to it, tap) of the gradients of
//      the outputs whose winner is that tap, in a fixed order: rows and
//      columns of the pre-images ascending, then taps in row-major order.
#include <algorithm>
#include <cfloat>
#include <cstring>

#include "band.cuh"
#include "stage_groups.cuh"

namespace hgb {
namespace {

constexpr int MM_MAX = 15, MM_T = 256, MM_NONE = 0xFF;

struct MinMaxParams {
  const float *in, *gout;
  float *gin;
  uint8_t *sel;
  int64_t in_p, in_b, gout_p, gout_b, gin_p, gin_b;  // floats
  int w, h, batch;
  int mw, mh, red, bmode;
  float cval;
  int has_mask;
  float mask[MM_MAX * MM_MAX];
  uint8_t dom[MM_MAX * MM_MAX];
};

__global__ void __launch_bounds__(MM_T) minmax_select_kernel(const __grid_constant__ MinMaxParams p) {
  const int64_t n = (int64_t)p.w * p.h;
  const int64_t idx = (int64_t)blockIdx.x * MM_T + threadIdx.x;
  const int b = blockIdx.y;
  if (idx >= n) return;
  const int y = (int)(idx / p.w), x = (int)(idx - (int64_t)y * p.w);
  const int rx = p.mw / 2, ry = p.mh / 2;
  const float *in = p.in + (int64_t)b * p.in_b;
  const bool is_max = p.red == HGB_REDUCE_MAX;
  float acc = is_max ? FLT_MIN : FLT_MAX;
  int win = MM_NONE;
  for (int my = 0; my < p.mh; ++my)
    for (int mx = 0; mx < p.mw; ++mx) {
      const int k = my * p.mw + mx;
      if (!p.dom[k]) continue;
      const int ax = remap(p.bmode, x + mx - rx, 0, p.w), ay = remap(p.bmode, y + my - ry, 0, p.h);
      const bool outside = ax == (int)0x80000000 || ay == (int)0x80000000;
      const float xv = outside ? p.cval : __ldg(in + (int64_t)ay * p.in_p + ax);
      const float v = p.has_mask ? __fmul_rn(p.mask[k], xv) : xv;
      const bool keep = is_max ? acc > v : acc < v;
      if (!keep) {
        acc = v;
        win = outside ? MM_NONE : k;  // a CONSTANT tap outside carries no gradient
      }
    }
  p.sel[(int64_t)b * n + idx] = (uint8_t)win;
}

// virtual positions v in [-reach, n + reach) that the remap sends to i (i itself first)
__device__ __forceinline__ int mm_pre(int mode, int i, int n, int reach, int *out) {
  int k = 0;
  out[k++] = i;
  if (mode == HGB_BOUNDARY_CONSTANT) return k;
  for (int v = -reach; v < 0; ++v)
    if (remap(mode, v, 0, n) == i && k < 2 * MM_MAX + 1) out[k++] = v;
  for (int v = n; v < n + reach; ++v)
    if (remap(mode, v, 0, n) == i && k < 2 * MM_MAX + 1) out[k++] = v;
  return k;
}

__global__ void __launch_bounds__(MM_T) minmax_gather_kernel(const __grid_constant__ MinMaxParams p) {
  const int64_t n = (int64_t)p.w * p.h;
  const int64_t idx = (int64_t)blockIdx.x * MM_T + threadIdx.x;
  const int b = blockIdx.y;
  if (idx >= n) return;
  const int iy = (int)(idx / p.w), ix = (int)(idx - (int64_t)iy * p.w);
  const int rxl = p.mw / 2, ryl = p.mh / 2, rxh = p.mw - 1 - rxl, ryh = p.mh - 1 - ryl;
  const uint8_t *sel = p.sel + (int64_t)b * n;
  const float *gout = p.gout + (int64_t)b * p.gout_b;
  int prx[2 * MM_MAX + 1], pry[2 * MM_MAX + 1];
  const int rx = max(rxl, rxh), ry = max(ryl, ryh);
  const bool inner = ix >= rx && ix < p.w - rx && iy >= ry && iy < p.h - ry;
  int nx = 1, ny = 1;
  prx[0] = ix;
  pry[0] = iy;
  if (!inner) {  // near a border: every virtual position the remap sends here
    nx = mm_pre(p.bmode, ix, p.w, rx + 1, prx);
    ny = mm_pre(p.bmode, iy, p.h, ry + 1, pry);
  }
  float acc = 0.0f;
  for (int a = 0; a < ny; ++a)
    for (int c = 0; c < nx; ++c)
      for (int my = 0; my < p.mh; ++my)
        for (int mx = 0; mx < p.mw; ++mx) {
          const int k = my * p.mw + mx;
          // output j read virtual position v = j + o through tap o
          const int jy = pry[a] - (my - ryl), jx = prx[c] - (mx - rxl);
          if (jx < 0 || jx >= p.w || jy < 0 || jy >= p.h) continue;
          const int64_t j = (int64_t)jy * p.w + jx;
          if (sel[j] != k) continue;
          const float g = __ldg(gout + (int64_t)jy * p.gout_p + jx);
          acc = p.has_mask ? __fmaf_rn(p.mask[k], g, acc) : __fadd_rn(acc, g);
        }
  p.gin[(int64_t)b * p.gin_b + (int64_t)iy * p.gin_p + ix] = acc;
}

// ---------------------------------------------------------------- tiles
// 64 x 8 PY pixels per CTA, a thread per 4 x PY (PY = 4, fewer on small
// batches).  The general kernels above spend
// a remap and a global load on every tap of every pixel; here the tile and its
// halo are staged once and a row's taps come from a register window.  Select is
// bound by the ALU pipe (a compare and two selects per tap: 85 % busy on 8 images of
// 1024 x 1024), gather by its loads (first stall long_scoreboard, issue slots 64 %
// busy, ALU pipe 40 %).  Forward and adjoint of the 5 x 5 disc on 8
// images of 509 x 381: 176 -> 38 us; of the 7 x 7 disc on
// 2309 x 2207: 779 -> 142 us.
constexpr int MT_BX = 16, MT_NT = 128, MT_PAD = 3, MT_TW = 64, MT_SW = MT_TW + 8, MT_G = MT_SW / 4;

struct MinMaxTileParams {
  const float *in, *gout;
  float *gin;
  uint8_t *sel;
  int64_t in_p, in_b, gout_p, gout_b, gin_p, gin_b;  // bytes
  int64_t sel_p, sel_b;
  int w, h, bmode;
  float cval;
  uint32_t flip;     // MAX runs as MIN of the negated values: every comparison has the same outcome
  // cells of the K x K window, a bit per column: row my at [my + MT_PAD], with
  // empty rows on either side, so that a staged row finds its window row for
  // each of a thread's outputs without a test
  uint32_t rows[7 + 2 * MT_PAD];
};

__device__ __forceinline__ void window12(const float *row, float (&w)[12]) {
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    const float4 t = reinterpret_cast<const float4 *>(row)[v];
    w[4 * v] = t.x;
    w[4 * v + 1] = t.y;
    w[4 * v + 2] = t.z;
    w[4 * v + 3] = t.w;
  }
}

template <int K, int PY>
__global__ void __launch_bounds__(MT_NT) minmax_select_tile_kernel(const __grid_constant__ MinMaxTileParams p) {
  constexpr int R = K / 2, MT_TH = 8 * PY, SH = MT_TH + 2 * R;
  __shared__ __align__(16) float tile[SH * MT_SW];
  const int b = blockIdx.z, i0 = blockIdx.x * MT_TW, j0 = blockIdx.y * MT_TH;
  stage_groups<float, MT_SW, SH, MT_NT>(tile, (const char *)p.in + b * p.in_b, p.in_p, i0 - 4, j0 - R, 0, p.w, 0, p.h,
                                        p.bmode, p.cval, R);
  stage_wait();
  __syncthreads();
  const int tx = threadIdx.x % MT_BX, ty = threadIdx.x / MT_BX;
  const float first = p.flip ? -FLT_MIN : FLT_MAX;
  float acc[PY][4];
  int win[PY][4];
#pragma unroll
  for (int oy = 0; oy < PY; ++oy)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc[oy][q] = first;
      win[oy][q] = MM_NONE;
    }
  // rolled over the staged rows: the loop unrolled is 20 to 30 KB of code, and a
  // CTA runs through it once, at the pace of instruction cache misses
#pragma unroll 1
  for (int r = 0; r < PY + K - 1; ++r) {
    float w[12];
    window12(&tile[(ty * PY + r) * MT_SW + tx * 4], w);
#pragma unroll
    for (int i = 0; i < 12; ++i) w[i] = __uint_as_float(__float_as_uint(w[i]) ^ p.flip);
#pragma unroll
    for (int oy = 0; oy < PY; ++oy) {
      const uint32_t bits = p.rows[r - oy + MT_PAD];  // window row r - oy, ascending in r: row-major per output
      if (!bits) continue;
      const int k0 = (r - oy) * K;
#pragma unroll
      for (int mx = 0; mx < K; ++mx) {
        if (!(bits >> mx & 1u)) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float v = w[4 - R + mx + q];
          const bool keep = acc[oy][q] < v;
          acc[oy][q] = keep ? acc[oy][q] : v;
          win[oy][q] = keep ? win[oy][q] : k0 + mx;
        }
      }
    }
  }
  const int x = i0 + 4 * tx;
  if (x >= p.w) return;
#pragma unroll
  for (int oy = 0; oy < PY; ++oy) {
    const int y = j0 + ty * PY + oy;
    if (y >= p.h) break;
    if (p.bmode == HGB_BOUNDARY_CONSTANT && (x < R || x + 4 > p.w - R || y < R || y >= p.h - R)) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {  // a CONSTANT tap outside carries no gradient
        const int my = win[oy][q] / K, ay = y + my - R, ax = x + q + (win[oy][q] - my * K) - R;
        if (ay < 0 || ay >= p.h || ax < 0 || ax >= p.w) win[oy][q] = MM_NONE;
      }
    }
    // rows of the byte plane start on words and are padded to whole words
    *reinterpret_cast<uint32_t *>(p.sel + b * p.sel_b + y * p.sel_p + x) =
        (uint32_t)win[oy][0] | (uint32_t)win[oy][1] << 8 | (uint32_t)win[oy][2] << 16 | (uint32_t)win[oy][3] << 24;
  }
}

// The band pixels of a gather tile.  S = float: added to the pixel's own sum in
// grad_in; S = double: the whole sum, own taps included.
template <int K, int SH, typename S>
__device__ __forceinline__ void minmax_band(const MinMaxTileParams &p, const TileBand &band, int b, int i0, int j0,
                                            const int *sel, const float *g, const uint8_t *selb, const char *gout) {
  constexpr int R = K / 2;
  constexpr bool whole = sizeof(S) == 8;
  const int part = threadIdx.x % 4;  // a quarter of the window's rows each
#pragma unroll 1
  for (int k0 = 0; k0 < 4 * band.count; k0 += MT_NT) {
    const int k = (k0 + (int)threadIdx.x) / 4;
    int bx = 0, by = 0;
    unsigned px = 0, py = 0;
    if (k < band.count) {
      tile_band_pos(band, k, bx, by);
      px = preimage_bits<R>(p.bmode, i0 + bx, p.w);
      py = preimage_bits<R>(p.bmode, j0 + by, p.h);
    }
    const int ix = i0 + bx, iy = j0 + by;
    float *dst = reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + iy * p.gin_p) + ix;
    S s = S(0);
    if (px | py) {
      if (!whole && part == 0) s = (S)*dst;
      for (unsigned ym = py << 1 | 1u; ym; ym &= ym - 1u) {  // bit 0: the row itself
        const int vy = ym & 1u ? iy : preimage_pos<R>(__ffs((int)ym) - 2, p.h), lo = max(0, vy + R - p.h + 1);
        const unsigned xs = (ym & 1u) && !whole ? px << 1 : px << 1 | 1u;
#pragma unroll 1
        for (int my = lo + ((part - lo) & 3); my <= min(K - 1, vy + R); my += 4) {
          const int jy = vy - (my - R), ry = jy - (j0 - R);
          for (unsigned xm = xs; xm; xm &= xm - 1u) {
            const int vx = xm & 1u ? ix : preimage_pos<R>(__ffs((int)xm) - 2, p.w);
            const int m1 = min(K - 1, vx + R);  // columns of taps inside the image
#pragma unroll 2
            for (int mx = max(0, vx + R - p.w + 1); mx <= m1; ++mx) {
              const int jx = vx - (mx - R), rx = jx - (i0 - 4);
              if (ry >= 0 && ry < SH && rx >= 0 && rx < MT_SW) {
                if (sel[ry * MT_SW + rx] == my * K + mx) s += (S)g[ry * MT_SW + rx];
              } else if (__ldcg(selb + jy * p.sel_p + jx) == my * K + mx) {
                s += (S)__ldg(reinterpret_cast<const float *>(gout + jy * p.gout_p) + jx);
              }
            }
          }
        }
      }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((px | py) && part == 0) *dst = (float)s;
  }
}

template <int K, int PY>
__global__ void __launch_bounds__(MT_NT, 6) minmax_gather_tile_kernel(const __grid_constant__ MinMaxTileParams p) {
  constexpr int R = K / 2, MT_TH = 8 * PY, SH = MT_TH + 2 * R;
  __shared__ __align__(16) float g[SH * MT_SW];
  __shared__ __align__(16) int sel[SH * MT_SW];
  const int b = blockIdx.z, i0 = blockIdx.x * MT_TW, j0 = blockIdx.y * MT_TH;
  const char *gout = (const char *)p.gout + b * p.gout_b;
  const uint8_t *selb = p.sel + b * p.sel_b;
#pragma unroll 2
  for (int c = threadIdx.x; c < SH * MT_G; c += MT_NT) {
    const int r = c / MT_G, k = c - r * MT_G, x = i0 - 4 + 4 * k, y = j0 - R + r;
    uint32_t s = 0xffffffffu;
    if (y >= 0 && y < p.h && x >= 0 && x < p.w) s = __ldcg(reinterpret_cast<const uint32_t *>(selb + y * p.sel_p + x));
    int4 v;
    v.x = s & 0xffu;
    v.y = x + 1 < p.w ? (int)(s >> 8 & 0xffu) : MM_NONE;
    v.z = x + 2 < p.w ? (int)(s >> 16 & 0xffu) : MM_NONE;
    v.w = x + 3 < p.w ? (int)(s >> 24) : MM_NONE;
    reinterpret_cast<int4 *>(sel)[c] = v;
    reinterpret_cast<float4 *>(g)[c] =
        load_group<float>(gout, p.gout_p, x, y, 0, p.w, 0, p.h, HGB_BOUNDARY_CONSTANT, 0.0f, 0);
  }
  __syncthreads();
  const int tx = threadIdx.x % MT_BX, ty = threadIdx.x / MT_BX;
  const int x = i0 + 4 * tx;
  float acc[PY][4];
#pragma unroll
  for (int oy = 0; oy < PY; ++oy)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[oy][q] = 0.0f;
#pragma unroll 1
  for (int r = PY + K - 2; r >= 0; --r) {  // tap rows ascending: output rows descending
    float gw[12];
    int sw[12];
    window12(&g[(ty * PY + r) * MT_SW + tx * 4], gw);
    const int4 *srow = reinterpret_cast<const int4 *>(&sel[(ty * PY + r) * MT_SW + tx * 4]);
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const int4 t = srow[v];
      sw[4 * v] = t.x;
      sw[4 * v + 1] = t.y;
      sw[4 * v + 2] = t.z;
      sw[4 * v + 3] = t.w;
    }
#pragma unroll
    for (int oy = 0; oy < PY; ++oy) {
      const int my = oy + 2 * R - r;
      const uint32_t bits = p.rows[my + MT_PAD];
      if (!bits) continue;
      const int k0 = my * K;
#pragma unroll
      for (int mx = 0; mx < K; ++mx) {
        if (!(bits >> mx & 1u)) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q)  // output column x + q - (mx - R)
          if (sw[4 + R - mx + q] == k0 + mx) acc[oy][q] = __fadd_rn(acc[oy][q], gw[4 + R - mx + q]);
      }
    }
  }
#pragma unroll
  for (int oy = 0; oy < PY; ++oy) {
    const int y = j0 + ty * PY + oy;
    if (x >= p.w || y >= p.h) break;
    float *dst = reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + y * p.gin_p) + x;
    if (x + 4 <= p.w && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
      *reinterpret_cast<float4 *>(dst) = make_float4(acc[oy][0], acc[oy][1], acc[oy][2], acc[oy][3]);
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (x + q < p.w) dst[q] = acc[oy][q];
    }
  }
  // ---- near a border: the virtual positions that the remap sends to a pixel
  // add to its own sum, only the taps that reach back into the image, from the
  // staged tile where it holds the output (REPEAT reaches the other side).
  // Four lanes share a band pixel.  Walking every tap of every position in the
  // lane that owns the pixel made the border tiles the slowest: 87 us against
  // 51 us for 8 images of 509 x 381, forward included.  On images hardly wider
  // than the window hundreds of terms meet in one pixel and cancel: there the
  // whole sum is taken again, in FP64.
  if (p.bmode == HGB_BOUNDARY_CONSTANT) return;
  const TileBand band = tile_band<R>(i0, j0, MT_TW, MT_TH, p.w, p.h, true, true);
  if (band.count == 0) return;
  __syncthreads();  // the sums without the other pre-images are written
  if (p.w < 2 * K || p.h < 2 * K)
    minmax_band<K, SH, double>(p, band, b, i0, j0, sel, g, selb, gout);
  else
    minmax_band<K, SH, float>(p, band, b, i0, j0, sel, g, selb, gout);
}

// The tiled form of a Domain of at most 7 x 7 cells: its window embedded in an
// odd K x K one (tap numbers are private to the two kernels).  Tiles are lower
// where 32 rows would leave an SM fewer than eight CTAs: a thread runs through
// a few thousand dependent instructions whatever the image, so a small image is
// done sooner with fewer pixels per thread (140 x 131, three
// calls as one graph: 37 -> 18 us).
template <int K, int PY>
void launch_minmax_tiles(const MinMaxTileParams &p, int batch, cudaStream_t st) {
  const dim3 grid(cdiv(p.w, MT_TW), cdiv(p.h, 8 * PY), batch);
  minmax_select_tile_kernel<K, PY><<<grid, MT_NT, 0, st>>>(p);
  minmax_gather_tile_kernel<K, PY><<<grid, MT_NT, 0, st>>>(p);
}
template <int K>
void launch_minmax_tiles(const MinMaxTileParams &p, int batch, cudaStream_t st) {
  const int64_t cols = (int64_t)cdiv(p.w, MT_TW) * batch, want = 8 * num_sms();
  if (cols * cdiv(p.h, 32) >= want)
    launch_minmax_tiles<K, 4>(p, batch, st);
  else if (cols * cdiv(p.h, 16) >= want)
    launch_minmax_tiles<K, 2>(p, batch, st);
  else
    launch_minmax_tiles<K, 1>(p, batch, st);
}

}  // namespace
}  // namespace hgb

using namespace hgb;

extern "C" int hgb_local_op_minmax_adjoint(const hgb_view *in, const hgb_view *grad_out, const hgb_view *grad_in,
                                           const float *mask, const uint8_t *domain, int mask_w, int mask_h,
                                           int reduce, int boundary, float const_val, void *stream) {
  int rc = check_view(in, "in");
  if (rc) return rc;
  rc = check_view(grad_out, "grad_out");
  if (rc) return rc;
  rc = check_view(grad_in, "grad_in");
  if (rc) return rc;
  HGB_REQUIRE(in->dtype == HGB_F32 && grad_out->dtype == HGB_F32 && grad_in->dtype == HGB_F32,
              "hgb_local_op_minmax_adjoint: f32 storage expected");
  HGB_REQUIRE(in->width == grad_out->width && in->height == grad_out->height && in->batch == grad_out->batch &&
                  grad_in->width == in->width && grad_in->height == in->height && grad_in->batch == in->batch,
              "hgb_local_op_minmax_adjoint: size mismatch");
  HGB_REQUIRE(mask_w >= 1 && mask_h >= 1 && mask_w <= MM_MAX && mask_h <= MM_MAX,
              "hgb_local_op_minmax_adjoint: mask size must be 1..15");
  HGB_REQUIRE(reduce == HGB_REDUCE_MIN || reduce == HGB_REDUCE_MAX, "hgb_local_op_minmax_adjoint: MIN or MAX");
  HGB_REQUIRE(boundary >= 0 && boundary <= 4, "hgb_local_op_minmax_adjoint: bad boundary");
  HGB_REQUIRE(in->batch <= 65535, "hgb_local_op_minmax_adjoint: at most 65535 images per call");
  MinMaxParams p;
  memset(&p, 0, sizeof(p));
  p.in = (const float *)in->data;
  p.gout = (const float *)grad_out->data;
  p.gin = (float *)grad_in->data;
  HGB_REQUIRE(in->pitch % 4 == 0 && grad_out->pitch % 4 == 0 && grad_in->pitch % 4 == 0 &&
                  in->batch_stride % 4 == 0 && grad_out->batch_stride % 4 == 0 && grad_in->batch_stride % 4 == 0,
              "hgb_local_op_minmax_adjoint: pitches must be whole floats");
  p.in_p = in->pitch / 4;
  p.in_b = in->batch_stride / 4;
  p.gout_p = grad_out->pitch / 4;
  p.gout_b = grad_out->batch_stride / 4;
  p.gin_p = grad_in->pitch / 4;
  p.gin_b = grad_in->batch_stride / 4;
  p.w = in->width;
  p.h = in->height;
  p.batch = in->batch;
  p.mw = mask_w;
  p.mh = mask_h;
  p.red = reduce;
  p.bmode = boundary;
  p.cval = const_val;
  p.has_mask = mask != nullptr;
  for (int k = 0; k < mask_w * mask_h; ++k) {
    p.mask[k] = mask ? mask[k] : 1.0f;
    p.dom[k] = domain ? (domain[k] != 0) : 1;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t npx = (int64_t)p.w * p.h;
  const int span = std::max(std::max(mask_w, mask_h), 3), K = span | 1;
  if (!mask && K <= 7 && cdiv(p.h, 8) <= 65535) {
    MinMaxTileParams t;
    memset(&t, 0, sizeof(t));
    t.in = p.in;
    t.gout = p.gout;
    t.gin = p.gin;
    t.in_p = in->pitch;
    t.in_b = in->batch_stride;
    t.gout_p = grad_out->pitch;
    t.gout_b = grad_out->batch_stride;
    t.gin_p = grad_in->pitch;
    t.gin_b = grad_in->batch_stride;
    t.w = p.w;
    t.h = p.h;
    t.bmode = boundary;
    t.cval = const_val;
    t.flip = reduce == HGB_REDUCE_MAX ? 0x80000000u : 0u;
    const int dx = K / 2 - mask_w / 2, dy = K / 2 - mask_h / 2;
    for (int y = 0; y < mask_h; ++y)
      for (int x = 0; x < mask_w; ++x)
        if (p.dom[y * mask_w + x]) t.rows[y + dy + MT_PAD] |= 1u << (x + dx);
    t.sel_p = ((int64_t)p.w + 3) / 4 * 4;
    t.sel_b = t.sel_p * p.h;
    Workspace ws;
    rc = workspace_get((size_t)t.sel_b * p.batch + 64, &ws);
    if (rc) return rc;
    t.sel = (uint8_t *)ws.base;
    cudaEvent_t ev = before_launch(st);
    if (K == 3)
      launch_minmax_tiles<3>(t, p.batch, st);
    else if (K == 5)
      launch_minmax_tiles<5>(t, p.batch, st);
    else
      launch_minmax_tiles<7>(t, p.batch, st);
    return after_launch("minmax_gather_tile_kernel", st, ev);
  }
  const int64_t nblk = (npx + MM_T - 1) / MM_T;
  HGB_REQUIRE(nblk < (int64_t)0x7fffffff, "hgb_local_op_minmax_adjoint: image too large");
  Workspace ws;
  rc = workspace_get((size_t)npx * p.batch + 64, &ws);
  if (rc) return rc;
  p.sel = (uint8_t *)ws.base;
  const dim3 grid((unsigned)nblk, (unsigned)p.batch);
  cudaEvent_t ev = before_launch(st);
  minmax_select_kernel<<<grid, MM_T, 0, st>>>(p);
  minmax_gather_kernel<<<grid, MM_T, 0, st>>>(p);
  return after_launch("minmax_gather_kernel", st, ev);
}
