// pipelines.cu -- two multi-kernel sample programs of the reference as hand-fused
// kernel chains, with their plain per-kernel launch structure for comparison.
//
// Harris corner (samples-public/3_Preprocessing/Harris_Corner/src/main.cpp:56-166,
// 258-307, the 3x3 configuration): nine kernels in the reference --
//   dx = (short)(sum over Domain(mx) in * mx / 6), dy likewise with my
//        (mx = [-1 0 1] in every row, my = its transpose; short sums, C
//        division truncating toward zero)
//   sx = dx^2, sy = dy^2, sxy = dx * dy                     (short)
//   Gx = (short)(sum over the 3x3 mask [1 2 1; 2 4 2; 1 2 1] of sx * m / 16),
//        Gy, Gxy likewise (int sums)
//   R  = (float)(Gx Gy - Gxy^2) - (k (float)(Gx + Gy)) (float)(Gx + Gy),
//        every float operation rounded separately;  out = R > threshold ? 1 : 0
// Every local operator reads through the boundary remap (CONSTANT taps read
// 0; the Gaussian reads the products at their remapped positions).  Fused form:
// one kernel stages the u8 input with a 2-pixel halo, keeps the products in
// registers and writes the 0/1 image: 1 byte in and 1 byte out per pixel instead of the nine launches' short intermediates.
//
// Unsharp (samples-public/1_Local_Operators/Unsharp/src/main.cpp:53-149,203-247,
// 3x3): five kernels in the reference --
//   gray  = 0.2126f * powf(R, c) + 0.7152 * powf(G, c) + 0.0722 * powf(B, c),
//           c = 1.0f / 2.2f; the two last literals are double, so the sum is
//           evaluated in double and rounded to float
//   blur  = 3x3 convolution of gray (products and sums rounded separately)
//   sharp = 2 gray - blur;  ratio = sharp / max(gray, 0.01f)
//   out   = (R ratio, G ratio, B ratio, A), each channel the float product
//           converted to uchar as the CPU back end does (truncated to an int,
//           low byte kept)
// The luminance depends on the bytes only: the powf terms come from 256-entry
// tables computed on the host with the host's powf (the CPU back end's own
// function) and the double products split into float pairs.  The double sum
// is reproduced by an exact float-float sum; a pixel whose sum lies within a
// tiny margin of a float rounding midpoint (about 1 in 10^5) is recomputed in
// FP64, so the result equals the double evaluation bit for bit.  Fused form:
// one kernel reads and writes 8 bytes per pixel instead of the five launches'
// float intermediates.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

#include "band.cuh"
#include "stage_groups.cuh"

namespace hgb {
namespace {

// ------------------------------------------------------------------ Harris

struct HarrisParams {
  const uint8_t *in;
  int64_t in_p, in_b;
  uint8_t *out;
  int64_t out_p, out_b;
  int w, h, bmode;
  float k, threshold;
  // plain launch structure: short intermediates [image][h][w]
  int16_t *dx, *dy, *sx, *sy, *sxy, *dxy;
};

__device__ __forceinline__ int hc_in(const HarrisParams &p, const uint8_t *img, int vx, int vy) {
  const int rx = remap(p.bmode, vx, 0, p.w), ry = remap(p.bmode, vy, 0, p.h);
  if (rx == (int)0x80000000 || ry == (int)0x80000000) return 0;
  return img[(int64_t)ry * p.in_p + rx];
}

// the two derivative sums at a pixel from a 3x3 neighbourhood v[row][col]
__device__ __forceinline__ void hc_deriv(const int v[3][3], int16_t &dx, int16_t &dy) {
  // Domain order, row-major; the short accumulator of the sample
  int16_t ax = 0, ay = 0;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    ax = (int16_t)(ax + (int16_t)(-v[r][0]));
    ax = (int16_t)(ax + (int16_t)v[r][2]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) ay = (int16_t)(ay + (int16_t)(-v[0][c]));
#pragma unroll
  for (int c = 0; c < 3; ++c) ay = (int16_t)(ay + (int16_t)v[2][c]);
  dx = (int16_t)(ax / 6);
  dy = (int16_t)(ay / 6);
}

__device__ __forceinline__ uint8_t hc_response(const HarrisParams &p, int gx, int gy, int gxy) {
  const float det = __int2float_rn(gx * gy - gxy * gxy);
  const float tr = __int2float_rn(gx + gy);
  const float R = __fsub_rn(det, __fmul_rn(__fmul_rn(p.k, tr), tr));
  return R > p.threshold ? 1 : 0;
}

// Fused form.  Pixels at least two from every edge need no boundary: their
// whole 5 x 5 neighbourhood lies in the image.  A warp walks 128 columns of
// TR rows of a staged byte tile, a lane four columns: per row the derivative
// sums on six columns, their quotients, products, the Gaussian's row sums, and
// from three of those the response of the row two above.  Everything up to the
// sixteenths is an integer below 2^24, held exactly in FP32 and computed two
// columns per packed f32x2 operation; the sixteenths truncate by rounding a
// value moved to the middle of its step (x / 16 - 15/32, toward zero for either
// sign).  The two-pixel frame takes four lanes per pixel and the
// boundary rule at every read, in the grid's first CTAs.
//
// Bound by instructions at 20 warps per SM (89 registers): issue slots 57 % busy, the
// FMA pipe, which a packed operation holds for two cycles, 55 %.  One pixel per thread
// with 27 shared 4-byte reads and int products took 89 us for 4032 x 3024; this takes
// 43 us (HBM floor 3.6 us).
constexpr int HT_W = 128, HT_NT = 128, HT_SW = HT_W + 8;  // tile and staged bytes per row

__device__ __forceinline__ f2 f2_both(float v) { return f2_pack(v, v); }

// x / 6 truncated toward zero, |x| <= 765 (each lane): 1 / 6 rounds up in FP32,
// so a multiple of six does not fall below its quotient, and the next quotient is
// at least 1 / 6 away.  The truncation runs on the conversion unit, which is idle
// otherwise.
__device__ __forceinline__ f2 hc_sixth(f2 x) {
  const f2 t = f2_mul(x, f2_both(0.166666672f));
  return f2_pack(truncf(f2_lo(t)), truncf(f2_hi(t)));
}

// 1 where the response of the sixteen-fold Gaussian sums exceeds the threshold;
// u = sum / 16 + 1.5 * 2^23 (the integer sits in the low mantissa bits), tr = gx + gy
__device__ __forceinline__ uint32_t hc_corner(float k, float threshold, float uxf, float uyf, float uxyf, float tr) {
  const int gx = __float_as_int(uxf) - 0x4B400000, gy = __float_as_int(uyf) - 0x4B400000,
            gxy = __float_as_int(uxyf) - 0x4B400000;
  const float det = __int2float_rn(gx * gy - gxy * gxy);
  return __fsub_rn(det, __fmul_rn(__fmul_rn(k, tr), tr)) > threshold ? 1u : 0u;
}

// the response at a pixel with the boundary rule at every read, by four lanes (a
// row of products each): the Gaussian reads the products at their remapped
// positions (CONSTANT: 0, as products of pixels that read 0).  The rows and columns
// are remapped first, so that a lane's 27 loads are in flight together (one product
// after the other took the smallest images from 4.9 to 6.4 us with CONSTANT).
__device__ __forceinline__ uint8_t hc_frame_pixel(const HarrisParams &p, const uint8_t *img, int x, int y, int part) {
  int a = 0, bb = 0, cc = 0;
  const int uy = part < 3 ? remap(p.bmode, y - 1 + part, 0, p.h) : (int)0x80000000;
  int row[3], col[3][3];  // negative: reads 0
#pragma unroll
  for (int r = 0; r < 3; ++r) row[r] = uy < 0 ? uy : remap(p.bmode, uy - 1 + r, 0, p.h);
#pragma unroll
  for (int dj = 0; dj < 3; ++dj) {
    const int ux = remap(p.bmode, x - 1 + dj, 0, p.w);
#pragma unroll
    for (int c = 0; c < 3; ++c) col[dj][c] = ux < 0 ? ux : remap(p.bmode, ux - 1 + c, 0, p.w);
  }
  int v[3][3][3];
#pragma unroll
  for (int dj = 0; dj < 3; ++dj)
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        v[dj][r][c] = (row[r] | col[dj][c]) < 0 ? 0 : __ldg(img + (int64_t)row[r] * p.in_p + col[dj][c]);
#pragma unroll
  for (int dj = 0; dj < 3; ++dj) {
    int16_t dx, dy;
    hc_deriv(v[dj], dx, dy);
    const int m = (part == 1 ? 2 : 1) * (dj == 1 ? 2 : 1);
    a += (int16_t)(dx * dx) * m;
    bb += (int16_t)(dy * dy) * m;
    cc += (int16_t)(dx * dy) * m;
  }
#pragma unroll
  for (int d = 1; d < 4; d <<= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, d);
    bb += __shfl_xor_sync(0xffffffffu, bb, d);
    cc += __shfl_xor_sync(0xffffffffu, cc, d);
  }
  return hc_response(p, (int16_t)(a / 16), (int16_t)(bb / 16), (int16_t)(cc / 16));
}

template <int TR>
__global__ void __launch_bounds__(HT_NT) harris_fused_kernel(const __grid_constant__ HarrisParams p, int tiles_x,
                                                             int nframe) {
  constexpr int TH = 4 * TR, SH = TH + 4, G = HT_SW / 4;
  __shared__ __align__(16) uint32_t tile[SH * G];
  const int b = blockIdx.z;
  const uint8_t *img = p.in + (int64_t)b * p.in_b;
  uint8_t *out = p.out + (int64_t)b * p.out_b;
  if ((int)blockIdx.x < nframe) {  // the frame, first: its threads take longest
    const TileBand f = tile_band<2>(0, 0, p.w, p.h, p.w, p.h, true, true);
    const int k = (blockIdx.x * HT_NT + threadIdx.x) / 4, part = threadIdx.x % 4;
    int x = 0, y = 0;
    if (k < f.count) tile_band_pos(f, k, x, y);
    const uint8_t v = hc_frame_pixel(p, img, x, y, part);
    if (k < f.count && part == 0) out[(int64_t)y * p.out_p + x] = v;
    return;
  }
  const int t = (int)blockIdx.x - nframe, X0 = (t % tiles_x) * HT_W, Y0 = (t / tiles_x) * TH;
  // bytes outside the image reach no pixel stored below
  stage_words<G, SH, HT_NT>(tile, img, p.in_p, X0 - 4, Y0 - 2, p.w, p.h);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = X0 + 4 * lane, y0 = Y0 + warp * TR;
  // rolling state of the last two rows: input (columns x - 2 .. x + 5 as biased
  // floats 2^23 + byte; only differences are taken), column differences, and the
  // Gaussian's row sums of the three products
  f2 in[2][4], E[2][3], H[2][3][2];
#pragma unroll
  for (int l = 0; l < 2; ++l) {
#pragma unroll
    for (int i = 0; i < 4; ++i) in[l][i] = 0ull;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      E[l][i] = 0ull;
      H[l][i][0] = H[l][i][1] = 0ull;
    }
  }
  const uint32_t *src = &tile[warp * TR * G + lane];
  auto row = [&](int r, int l) {  // l: parity of r, the slot of the row two above
    const uint32_t w0 = src[r * G], w1 = src[r * G + 1], w2 = src[r * G + 2];
    auto byte = [](uint32_t w, int q) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 + q)); };
    const f2 v[4] = {f2_pack(byte(w0, 2), byte(w0, 3)), f2_pack(byte(w1, 0), byte(w1, 1)),
                     f2_pack(byte(w1, 2), byte(w1, 3)), f2_pack(byte(w2, 0), byte(w2, 1))};
    f2 e[3], P[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i) e[i] = f2_sub(v[i + 1], v[i]);
    f2 d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) d[i] = f2_sub(v[i], in[l][i]);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const f2 dx = hc_sixth(f2_add(f2_add(E[l][i], E[l ^ 1][i]), e[i]));
      const f2 mid = f2_pack(f2_hi(d[i]), f2_lo(d[i + 1]));
      const f2 dy = hc_sixth(f2_add(f2_add(d[i], mid), d[i + 1]));
      P[0][i] = f2_mul(dx, dx);
      P[1][i] = f2_mul(dy, dy);
      P[2][i] = f2_mul(dx, dy);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) in[l][i] = v[i];
#pragma unroll
    for (int i = 0; i < 3; ++i) E[l][i] = e[i];
    f2 u[3][2];
    const f2 two = f2_both(2.0f), sixteenth = f2_both(0.0625f), m = f2_both(12582912.0f);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const f2 mid = f2_pack(f2_hi(P[a][i]), f2_lo(P[a][i + 1]));
        const f2 h = f2_fma(two, mid, f2_add(P[a][i], P[a][i + 1]));
        const f2 s = f2_fma(two, H[l ^ 1][a][i], f2_add(H[l][a][i], h));
        H[l][a][i] = h;
        f2 half;
        if (a < 2) {  // sums of squares: not negative
          half = f2_both(-0.46875f);
        } else {
          const uint32_t n = 0xBEF00000u;  // -0.46875f
          half = f2_pack(__uint_as_float((__float_as_uint(f2_lo(s)) & 0x80000000u) ^ n),
                         __uint_as_float((__float_as_uint(f2_hi(s)) & 0x80000000u) ^ n));
        }
        u[a][i] = f2_add(f2_fma(s, sixteenth, half), m);
      }
    const int y = y0 + r - 4;
    if (r < 4 || y < 2 || y >= p.h - 2) return;
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const f2 tr = f2_add(f2_sub(u[0][i], m), f2_sub(u[1][i], m));
      o |= hc_corner(p.k, p.threshold, f2_lo(u[0][i]), f2_lo(u[1][i]), f2_lo(u[2][i]), f2_lo(tr)) << (16 * i);
      o |= hc_corner(p.k, p.threshold, f2_hi(u[0][i]), f2_hi(u[1][i]), f2_hi(u[2][i]), f2_hi(tr)) << (16 * i + 8);
    }
    uint8_t *dst = out + (int64_t)y * p.out_p + x;
    if (x >= 2 && x + 4 <= p.w - 2 && (reinterpret_cast<uintptr_t>(dst) & 3u) == 0) {
      *reinterpret_cast<uint32_t *>(dst) = o;
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (x + q >= 2 && x + q < p.w - 2) dst[q] = (uint8_t)(o >> (8 * q));
    }
  };
#pragma unroll 1
  for (int r = 0; r < TR + 4; r += 2) {
    row(r, 0);
    row(r + 1, 1);
  }
}

// ---- the reference's nine launches (one pixel per thread, short intermediates)
__device__ __forceinline__ bool hc_pixel(const HarrisParams &p, int &x, int &y, int &b) {
  x = blockIdx.x * 32 + (threadIdx.x & 31);
  y = blockIdx.y * 8 + (threadIdx.x >> 5);
  b = blockIdx.z;
  return x < p.w && y < p.h;
}
__device__ __forceinline__ int64_t hc_at(const HarrisParams &p, int b, int x, int y) {
  return ((int64_t)b * p.h + y) * p.w + x;
}

__global__ void __launch_bounds__(256) harris_deriv_kernel(const __grid_constant__ HarrisParams p, int which) {
  int x, y, b;
  if (!hc_pixel(p, x, y, b)) return;
  const uint8_t *img = p.in + (int64_t)b * p.in_b;
  int v[3][3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) v[i][j] = hc_in(p, img, x - 1 + j, y - 1 + i);
  int16_t dx, dy;
  hc_deriv(v, dx, dy);
  (which ? p.dy : p.dx)[hc_at(p, b, x, y)] = which ? dy : dx;
}

__global__ void __launch_bounds__(256) harris_square_kernel(const __grid_constant__ HarrisParams p, int which) {
  int x, y, b;
  if (!hc_pixel(p, x, y, b)) return;
  const int64_t o = hc_at(p, b, x, y);
  const int16_t a = which == 1 ? p.dy[o] : p.dx[o], c = which == 0 ? p.dx[o] : p.dy[o];
  (which == 0 ? p.sx : which == 1 ? p.sy : p.sxy)[o] = (int16_t)(a * c);
}

__global__ void __launch_bounds__(256) harris_gauss_kernel(const __grid_constant__ HarrisParams p, const int16_t *src,
                                                           int16_t *dst) {
  int x, y, b;
  if (!hc_pixel(p, x, y, b)) return;
  int s = 0;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int rx = remap(p.bmode, x - 1 + j, 0, p.w), ry = remap(p.bmode, y - 1 + i, 0, p.h);
      const int v = (rx == (int)0x80000000 || ry == (int)0x80000000) ? 0 : src[hc_at(p, b, rx, ry)];
      s += v * ((i == 1 ? 2 : 1) * (j == 1 ? 2 : 1));
    }
  dst[hc_at(p, b, x, y)] = (int16_t)(s / 16);
}

__global__ void __launch_bounds__(256) harris_response_kernel(const __grid_constant__ HarrisParams p) {
  int x, y, b;
  if (!hc_pixel(p, x, y, b)) return;
  const int64_t o = hc_at(p, b, x, y);
  // the sample's Gaussians of sx and sy land in the dx and dy images
  p.out[(int64_t)b * p.out_b + (int64_t)y * p.out_p + x] = hc_response(p, p.dx[o], p.dy[o], p.dxy[o]);
}

// ------------------------------------------------------------------ Unsharp
// luminance terms per byte value (host-computed, see the header comment)
struct UnsTables {
  float p[256];           // powf(v, c)
  float t0[256];          // 0.2126f * powf(v, c)
  float b1h[256], b1l[256];  // 0.7152 * powf(v, c) as a float pair
  float b2h[256], b2l[256];  // 0.0722 * powf(v, c) as a float pair
  double b1[256], b2[256];   // the double products, for the FP64 recomputation
};

struct UnsharpParams {
  const uchar4 *in;
  int64_t in_p, in_b;  // uchar4 elements
  uchar4 *out;
  int64_t out_p, out_b;
  int w, h, bmode;
  int batch;
  f2 nz;  // kNegativeZeros (f2_mul_rounded)
  const UnsTables *tab;  // device copy
  // plain launch structure: float intermediates [image][h][w]
  float *gray, *blur, *sharp, *ratio;
};

__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (float)(((double)t0 + b1) + b2) for the bytes (r, g, bl)
__device__ __forceinline__ float uns_gray(const UnsTables &T, const float *t0, const float *b1h, const float *b1l,
                                          const float *b2h, const float *b2l, int r, int g, int bl) {
  const float a = t0[r];
  float s, e1, e2;
  two_sum(a, b1h[g], s, e1);
  two_sum(s, b2h[bl], s, e2);
  const float e = __fadd_rn(__fadd_rn(e1, e2), __fadd_rn(b1l[g], b2l[bl]));
  const float y = __fadd_rn(s, e);
  if (y == 0.0f) return y;
  // distance of the exact sum from the rounding midpoints around y
  const float rho = __fadd_rn(__fsub_rn(s, y), e);
  const float ulp = __int_as_float(__float_as_int(y) & 0x7f800000) * 1.1920928955078125e-7f;  // 2^-23
  const bool pow2 = (__float_as_int(y) & 0x007fffff) == 0;
  const float below = pow2 ? 0.25f * ulp : 0.5f * ulp;
  const float margin = y * 9.094947017729282e-13f;  // 2^-40: far above every error of the float-float sum
  if (fabsf(rho - 0.5f * ulp) > margin && fabsf(rho + below) > margin) return y;
  return (float)__dadd_rn(__dadd_rn((double)a, T.b1[g]), T.b2[bl]);
}

__device__ __forceinline__ uchar4 uns_scale(uchar4 v, float r) {
  // (uchar)(v * r): truncated to an int, low byte kept
  v.x = (unsigned char)(__float2int_rz(__fmul_rn((float)v.x, r)) & 0xff);
  v.y = (unsigned char)(__float2int_rz(__fmul_rn((float)v.y, r)) & 0xff);
  v.z = (unsigned char)(__float2int_rz(__fmul_rn((float)v.z, r)) & 0xff);
  return v;
}

__device__ __forceinline__ float uns_blur(const float *g, int stride) {
  const float m0 = 0.057118f, m1 = 0.124758f, m2 = 0.272496f;
  const float m[9] = {m0, m1, m0, m1, m2, m1, m0, m1, m0};
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) s = __fadd_rn(s, __fmul_rn(m[i * 3 + j], g[i * stride + j]));
  return s;
}

__device__ __forceinline__ float uns_ratio(float g, float blur) {
  const float sharp = __fsub_rn(__fmul_rn(2.0f, g), blur);
  return __fdiv_rn(sharp, fmaxf(g, 0.01f));
}

// Fused form.  A warp walks down a strip of 120 or 60 columns, a lane four or two
// (the outer two lanes only supply the strip's halo), and keeps everything but
// the power table in registers: the gray of a row is formed once, its products
// with the mask's three weights once, and each output row adds the nine products
// in the reference's order as its three rows pass (two partial sums roll along).
// Additions and products run on two pixels per packed f32x2 operation.
//
// The power table is a copy per lane, entry v of lane l at word 32 v + l, so the
// three lookups of a pixel hit 32 banks whatever the bytes; the products 0.7152 p
// and 0.0722 p come from p as exact float pairs instead of four more tables.
// unsharp_shape() shares out the rows.
//
// Bound by instruction issue (72 % of the slots busy).  One pixel per thread over
// 32 x 16 tiles took 120 us for 4032 x 3024; this takes 54 us (HBM floor 14.4 us).
constexpr int UF_NT = 256;
constexpr int uf_cols(int np) { return 30 * 2 * np; }  // columns of a strip with np pairs per lane

// (float)(((double)(0.2126f p_r) + 0.7152 p_g) + 0.0722 p_b) of two pixels w0, w1
__device__ __forceinline__ f2 uns_gray2(const float *tab, const UnsTables *T, f2 nz, uint32_t w0, uint32_t w1) {
  // tab: the lane's column of the table
  auto look = [tab](uint32_t w0, uint32_t w1, int k) {
    return f2_pack(tab[((w0 >> (8 * k)) & 255u) * 32], tab[((w1 >> (8 * k)) & 255u) * 32]);
  };
  auto both = [](float v) { return f2_pack(v, v); };
  constexpr float g_hi = (float)0.7152, g_lo = (float)(0.7152 - (double)(float)0.7152);
  constexpr float b_hi = (float)0.0722, b_lo = (float)(0.0722 - (double)(float)0.0722);
  const f2 pr = look(w0, w1, 0), pg = look(w0, w1, 1), pb = look(w0, w1, 2);
  const f2 a = f2_mul_rounded(both(0.2126f), pr, nz);
  // c p as a pair: hi = fl(c_hi p), lo = (c_hi p - hi) + c_lo p
  const f2 gh = f2_mul_rounded(both(g_hi), pg, nz), bh = f2_mul_rounded(both(b_hi), pb, nz);
  const f2 gl = f2_sub(f2_mul(both(g_lo), pg), f2_fma(both(-g_hi), pg, gh));
  const f2 bl = f2_sub(f2_mul(both(b_lo), pb), f2_fma(both(-b_hi), pb, bh));
  auto two_sum2 = [](f2 x, f2 y, f2 &s, f2 &e) {
    s = f2_add(x, y);
    const f2 yy = f2_sub(s, x);
    e = f2_add(f2_sub(x, f2_sub(s, yy)), f2_sub(y, yy));
  };
  f2 s1, e1, s, e2;
  two_sum2(a, gh, s1, e1);
  two_sum2(s1, bh, s, e2);
  const f2 e = f2_add(f2_add(e1, e2), f2_add(gl, bl));
  f2 y2 = f2_add(s, e);
  const f2 rho2 = f2_add(f2_sub(s, y2), e);  // what the rounding to y took away
  float y[2] = {f2_lo(y2), f2_hi(y2)};
  const float rho[2] = {f2_lo(rho2), f2_hi(rho2)};
  bool redo[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    // within 2^-40 of a rounding midpoint, or at a power of two (whose lower
    // midpoint is nearer): evaluate in double
    const uint32_t u = __float_as_uint(y[i]);
    const float half = __uint_as_float(u & 0x7f800000u) * 5.9604644775390625e-8f;  // half an ulp
    redo[i] = (__fmaf_rn(y[i], 9.094947017729282e-13f, fabsf(rho[i])) >= half || (u & 0x007fffffu) == 0) && y[i] != 0.0f;
  }
  if (redo[0] || redo[1]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const uint32_t w = i ? w1 : w0;
      if (redo[i])
        y[i] = (float)__dadd_rn(__dadd_rn((double)__ldg(&T->t0[w & 255u]), __ldg(&T->b1[w >> 8 & 255u])),
                                __ldg(&T->b2[w >> 16 & 255u]));
    }
    y2 = f2_pack(y[0], y[1]);
  }
  return y2;
}

__device__ __forceinline__ uint32_t uns_scale_word(uint32_t v, float r) {
  // (uchar)(channel * r): truncated to an int, low byte kept; alpha copied
  uint32_t o = v;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float c = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 + k)) - 8388608.0f;
    const uint32_t t = (uint32_t)__float2int_rz(__fmul_rn(c, r));
    o = __byte_perm(o, t, k == 0 ? 0x3214 : (k == 1 ? 0x3240 : 0x3410));
  }
  return o;
}

template <int NP>
__global__ void __launch_bounds__(UF_NT) unsharp_fused_kernel(const __grid_constant__ UnsharpParams p, int strips,
                                                              int rows_per, int segments) {
  constexpr int CPL = 2 * NP;  // columns per lane
  __shared__ __align__(16) float tab[256 * 32];
  const int lane = threadIdx.x & 31;
  const float *tl = tab + lane;
  const int64_t job = (int64_t)blockIdx.x * (UF_NT / 32) + (threadIdx.x >> 5);
  const int64_t per = (int64_t)strips * segments;
  // (a 64-bit division takes several times a 32-bit one)
  const int b = (int)((job | per) >> 32 ? job / per : (int64_t)((unsigned)job / (unsigned)per)), jr = (int)(job - b * per);
  const bool idle = b >= p.batch;
  const int seg = jr / strips, x = (jr - seg * strips) * uf_cols(NP) - CPL + CPL * lane;  // this lane's columns
  const int y0 = seg * rows_per, y1 = min(y0 + rows_per, p.h);
  const uint32_t *img = reinterpret_cast<const uint32_t *>(p.in) + (int64_t)b * p.in_b;
  uint32_t *out = reinterpret_cast<uint32_t *>(p.out) + (int64_t)b * p.out_b;
  const bool whole = x >= 0 && x + CPL <= p.w;
  const bool stores = lane > 0 && lane < 31 && x < p.w;
  bool in_col[CPL];  // false: a CONSTANT column, gray 0
  int cx[CPL];
#pragma unroll
  for (int q = 0; q < CPL; ++q) {
    in_col[q] = true;
    cx[q] = x + q;
  }
  if (!whole) {
#pragma unroll
    for (int q = 0; q < CPL; ++q) {
      // columns past the halo serve no pixel: any valid address will do
      const int rx = x + q > p.w ? p.w - 1 : (x + q < -1 ? 0 : remap(p.bmode, x + q, 0, p.w));
      in_col[q] = rx != (int)0x80000000;
      cx[q] = in_col[q] ? rx : 0;
    }
  }
  auto load = [&](int ry, uint32_t (&w)[CPL]) {
    const uint32_t *row = img + (int64_t)ry * p.in_p;
    if (whole && (reinterpret_cast<uintptr_t>(row + x) & (4 * CPL - 1)) == 0) {
      if constexpr (NP == 2) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(row + x));
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
      } else {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(row + x));
        w[0] = v.x;
        w[1] = v.y;
      }
    } else {
#pragma unroll
      for (int q = 0; q < CPL; ++q) w[q] = __ldg(row + cx[q]);
    }
  };
  const float m0 = 0.057118f, m1 = 0.124758f, m2 = 0.272496f;
  auto both = [](float v) { return f2_pack(v, v); };
  f2 one[NP], two[NP];  // partial sums after one and two rows of their windows
  f2 gp[NP];            // gray of the row above
  uint32_t wp[CPL], wn[CPL];
#pragma unroll
  for (int i = 0; i < NP; ++i) one[i] = two[i] = gp[i] = 0ull;
#pragma unroll
  for (int q = 0; q < CPL; ++q) wp[q] = wn[q] = 0;
  if (!idle) {  // the first row's loads are in flight while the table is copied
    const int r0 = remap(p.bmode, y0 - 1, 0, p.h);
    load(r0 == (int)0x80000000 ? 0 : r0, wn);
  }
#pragma unroll
  for (int i = threadIdx.x; i < 256 * 8; i += UF_NT) {
    const float v = __ldg(&p.tab->p[i >> 3]);
    reinterpret_cast<float4 *>(tab)[i] = make_float4(v, v, v, v);
  }
  __syncthreads();
  if (idle) return;
#pragma unroll 1
  for (int y = y0 - 1; y <= y1; ++y) {
    uint32_t w[CPL];
#pragma unroll
    for (int q = 0; q < CPL; ++q) w[q] = wn[q];
    const bool row_in = (y >= 0 && y < p.h) || p.bmode != HGB_BOUNDARY_CONSTANT;
    if (y < y1) {  // the next row's loads are in flight while this one computes
      const int rn = remap(p.bmode, y + 1, 0, p.h);
      load(rn == (int)0x80000000 ? 0 : rn, wn);
    }
    f2 g[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) g[i] = uns_gray2(tl, p.tab, p.nz, w[2 * i], w[2 * i + 1]);
    if (p.bmode == HGB_BOUNDARY_CONSTANT && (!row_in || !whole)) {
#pragma unroll
      for (int i = 0; i < NP; ++i)
        g[i] = f2_pack(row_in && in_col[2 * i] ? f2_lo(g[i]) : 0.0f, row_in && in_col[2 * i + 1] ? f2_hi(g[i]) : 0.0f);
    }
    const float left = __shfl_up_sync(0xffffffffu, f2_hi(g[NP - 1]), 1);
    const float right = __shfl_down_sync(0xffffffffu, f2_lo(g[0]), 1);
    f2 go[NP + 1];  // columns (-1, 0), (1, 2), .. relative to x
#pragma unroll
    for (int i = 0; i <= NP; ++i)
      go[i] = f2_pack(i == 0 ? left : f2_hi(g[i > 0 ? i - 1 : 0]), i == NP ? right : f2_lo(g[i < NP ? i : 0]));
    f2 a0[NP + 1], a1[NP + 1], c1[NP], c2[NP];
#pragma unroll
    for (int i = 0; i <= NP; ++i) {
      a0[i] = f2_mul_rounded(both(m0), go[i], p.nz);
      a1[i] = f2_mul_rounded(both(m1), go[i], p.nz);
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      c1[i] = f2_mul_rounded(both(m1), g[i], p.nz);
      c2[i] = f2_mul_rounded(both(m2), g[i], p.nz);
    }
    f2 blur[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      // this row as the last of the window above, the middle of the next, the first of the one below
      blur[i] = f2_add(f2_add(f2_add(two[i], a0[i]), c1[i]), a0[i + 1]);
      two[i] = f2_add(f2_add(f2_add(one[i], a1[i]), c2[i]), a1[i + 1]);
      one[i] = f2_add(f2_add(f2_add(0ull, a0[i]), c1[i]), a0[i + 1]);
    }
    if (y > y0 && stores) {  // the window centred on row y - 1 is complete
      uint32_t o[CPL];
#pragma unroll
      for (int q = 0; q < CPL; ++q) {
        const f2 G = gp[q / 2], B = blur[q / 2];
        o[q] = uns_scale_word(wp[q], q & 1 ? uns_ratio(f2_hi(G), f2_hi(B)) : uns_ratio(f2_lo(G), f2_lo(B)));
      }
      uint32_t *dst = out + (int64_t)(y - 1) * p.out_p + x;
      if (x + CPL <= p.w && (reinterpret_cast<uintptr_t>(dst) & (4 * CPL - 1)) == 0) {
        if constexpr (NP == 2)
          *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
        else
          *reinterpret_cast<uint2 *>(dst) = make_uint2(o[0], o[1]);
      } else {
#pragma unroll
        for (int q = 0; q < CPL; ++q)
          if (x + q < p.w) dst[q] = o[q];
      }
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) gp[i] = g[i];
#pragma unroll
    for (int q = 0; q < CPL; ++q) wp[q] = w[q];
  }
}

// ---- the reference's five launches (one pixel per thread, float intermediates)
__device__ __forceinline__ bool us_pixel(const UnsharpParams &p, int &x, int &y, int &b) {
  x = blockIdx.x * 32 + (threadIdx.x & 31);
  y = blockIdx.y * 8 + (threadIdx.x >> 5);
  b = blockIdx.z;
  return x < p.w && y < p.h;
}
__device__ __forceinline__ int64_t us_at(const UnsharpParams &p, int b, int x, int y) {
  return ((int64_t)b * p.h + y) * p.w + x;
}

using UnsharpKernel = void (*)(UnsharpParams, int, int, int);
UnsharpKernel unsharp_kernel(int np) { return np == 2 ? unsharp_fused_kernel<2> : unsharp_fused_kernel<1>; }

// Pairs per lane and rows per warp.  A warp's rows (two more than it stores) run one
// after another, in 0.30 us + 0.47 us (two pairs) or 0.26 us (one pair) per CTA on the
// SM, measured on 64 x 64 to 4032 x 3024; the least sum over the CTAs per SM wins.  One
// pair also leaves less of a strip empty on narrow images.  4032 x 3024 54 us (60 us
// with one pair), 1920 x 1080 13.7 us (15.0 us in one full wave of two pairs), 1280 x 720
// 9.3 us (10.3), 640 x 480 6.0 us (6.4), 64 x 64 3.5 us (5.1).
struct UnsharpShape {
  int np, strips, rows, segments;
  int64_t ctas;
};
UnsharpShape unsharp_shape(int w, int h, int batch) {
  constexpr int kWarps = UF_NT / 32;
  UnsharpShape best = {};
  int64_t least = -1;
  for (int np = 2; np >= 1; --np) {
    const int strips = cdiv(w, uf_cols(np)), fit = resident_ctas((const void *)unsharp_kernel(np), UF_NT, 0);
    const int64_t columns = (int64_t)strips * batch, sms = num_sms();
    for (int c = 1; c <= fit; ++c) {
      const int64_t most = std::max<int64_t>(1, c * sms * kWarps / columns);  // segments
      const int rows = (int)((h + most - 1) / most), segments = cdiv(h, rows);
      const int64_t ctas = (columns * segments + kWarps - 1) / kWarps;
      const int64_t cost = (rows + 2) * (30 + (np == 2 ? 47 : 26) * ((ctas + sms - 1) / sms));
      if (least < 0 || cost < least) {
        least = cost;
        best = {np, strips, rows, segments, ctas};
      }
    }
  }
  return best;
}

__global__ void __launch_bounds__(256) unsharp_gray_kernel(const __grid_constant__ UnsharpParams p) {
  int x, y, b;
  if (!us_pixel(p, x, y, b)) return;
  const UnsTables &T = *p.tab;
  const uchar4 v = p.in[(int64_t)b * p.in_b + (int64_t)y * p.in_p + x];
  p.gray[us_at(p, b, x, y)] = uns_gray(T, T.t0, T.b1h, T.b1l, T.b2h, T.b2l, v.x, v.y, v.z);
}

__global__ void __launch_bounds__(256) unsharp_blur_kernel(const __grid_constant__ UnsharpParams p) {
  int x, y, b;
  if (!us_pixel(p, x, y, b)) return;
  float g[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int rx = remap(p.bmode, x - 1 + j, 0, p.w), ry = remap(p.bmode, y - 1 + i, 0, p.h);
      g[i * 3 + j] = (rx == (int)0x80000000 || ry == (int)0x80000000) ? 0.0f : p.gray[us_at(p, b, rx, ry)];
    }
  p.blur[us_at(p, b, x, y)] = uns_blur(g, 3);
}

__global__ void __launch_bounds__(256) unsharp_sharp_kernel(const __grid_constant__ UnsharpParams p) {
  int x, y, b;
  if (!us_pixel(p, x, y, b)) return;
  const int64_t o = us_at(p, b, x, y);
  p.sharp[o] = __fsub_rn(__fmul_rn(2.0f, p.gray[o]), p.blur[o]);
}

__global__ void __launch_bounds__(256) unsharp_ratio_kernel(const __grid_constant__ UnsharpParams p) {
  int x, y, b;
  if (!us_pixel(p, x, y, b)) return;
  const int64_t o = us_at(p, b, x, y);
  p.ratio[o] = __fdiv_rn(p.sharp[o], fmaxf(p.gray[o], 0.01f));
}

__global__ void __launch_bounds__(256) unsharp_scale_kernel(const __grid_constant__ UnsharpParams p) {
  int x, y, b;
  if (!us_pixel(p, x, y, b)) return;
  p.out[(int64_t)b * p.out_b + (int64_t)y * p.out_p + x] =
      uns_scale(p.in[(int64_t)b * p.in_b + (int64_t)y * p.in_p + x], p.ratio[us_at(p, b, x, y)]);
}

// host tables, built once per process with the host's powf; device copies per device
std::mutex g_uns_mu;
bool g_uns_host_ready = false;
UnsTables g_uns_host;
constexpr int kMaxDev = 64;
UnsTables *g_uns_dev[kMaxDev] = {};

int unsharp_tables(const UnsTables **out) {
  int dev = 0;
  HGB_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDev) return set_error(HGB_ERR_LIMIT, "hgb_unsharp: device index too large");
  std::lock_guard<std::mutex> lk(g_uns_mu);
  if (!g_uns_host_ready) {
    const float c = 1.0f / 2.2f;
    for (int v = 0; v < 256; ++v) {
      const float pv = powf((float)v, c);
      g_uns_host.p[v] = pv;
      g_uns_host.t0[v] = 0.2126f * pv;
      const double d1 = 0.7152 * (double)pv, d2 = 0.0722 * (double)pv;
      g_uns_host.b1[v] = d1;
      g_uns_host.b2[v] = d2;
      g_uns_host.b1h[v] = (float)d1;
      g_uns_host.b1l[v] = (float)(d1 - (double)g_uns_host.b1h[v]);
      g_uns_host.b2h[v] = (float)d2;
      g_uns_host.b2l[v] = (float)(d2 - (double)g_uns_host.b2h[v]);
    }
    g_uns_host_ready = true;
  }
  if (!g_uns_dev[dev]) {
    UnsTables *d = nullptr;
    HGB_CHECK_CUDA(cudaMalloc((void **)&d, sizeof(UnsTables)));
    const cudaError_t e = cudaMemcpy(d, &g_uns_host, sizeof(UnsTables), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
      cudaFree(d);
      return cuda_error(e, "hgb_unsharp: table upload");
    }
    g_uns_dev[dev] = d;
  }
  *out = g_uns_dev[dev];
  return HGB_OK;
}

}  // namespace
}  // namespace hgb

using namespace hgb;

extern "C" int hgb_harris_corner(const hgb_view *in, const hgb_view *out, float k, float threshold, int boundary,
                                 int mode, void *stream) {
  int rc = check_view(in, "in");
  if (rc) return rc;
  rc = check_view(out, "out");
  if (rc) return rc;
  HGB_REQUIRE(in->dtype == HGB_U8 && out->dtype == HGB_U8, "hgb_harris_corner: u8 images expected");
  HGB_REQUIRE(in->width == out->width && in->height == out->height && in->batch == out->batch,
              "hgb_harris_corner: size mismatch");
  HGB_REQUIRE(boundary >= 0 && boundary <= 4, "hgb_harris_corner: bad boundary");
  HGB_REQUIRE(mode == 0 || mode == 1, "hgb_harris_corner: mode must be 0 (fused) or 1 (nine launches)");
  HarrisParams p;
  memset(&p, 0, sizeof(p));
  p.in = (const uint8_t *)in->data;
  p.in_p = in->pitch;
  p.in_b = in->batch_stride;
  p.out = (uint8_t *)out->data;
  p.out_p = out->pitch;
  p.out_b = out->batch_stride;
  p.w = in->width;
  p.h = in->height;
  p.bmode = boundary;
  p.k = k;
  p.threshold = threshold;
  cudaStream_t st = (cudaStream_t)stream;
  if (mode == 0) {
    const int tiles_x = cdiv(p.w, HT_W);
    const int64_t edge = 4 * ((int64_t)p.w + p.h);  // at least the frame's pixels
    const int frame = (int)((4 * std::min<int64_t>(edge, (int64_t)p.w * p.h) + HT_NT - 1) / HT_NT);
    // 64-row tiles (16 rows per warp, 4 more to start from) where they give every
    // SM four CTAs, else 16-row ones, or 8-row ones where five quarters of the SMs have
    // one (the time of a small image is the chain of rows that a warp walks: 640 x 480
    // 5.95 us with 16 rows, 5.4 with 8; 800 x 600 5.97 and 6.4); 128-row tiles are slower
    // (one wave of uneven CTAs, 60 us against 51 us for 4032 x 3024, with the frame before)
    const int64_t per_row = (int64_t)tiles_x * in->batch;
    const int rows = per_row * cdiv(p.h, 64) >= 4 * num_sms() ? 64 : 4 * per_row * cdiv(p.h, 16) > 5 * num_sms() ? 16 : 8;
    const int64_t ntiles = (int64_t)tiles_x * cdiv(p.h, rows);
    HGB_REQUIRE(ntiles + frame < 0x7fffffff, "hgb_harris_corner: image too large");
    const dim3 grid((unsigned)(ntiles + frame), 1, in->batch);
    cudaEvent_t ev = before_launch(st);
    if (rows == 64)
      harris_fused_kernel<16><<<grid, HT_NT, 0, st>>>(p, tiles_x, frame);
    else if (rows == 16)
      harris_fused_kernel<4><<<grid, HT_NT, 0, st>>>(p, tiles_x, frame);
    else
      harris_fused_kernel<2><<<grid, HT_NT, 0, st>>>(p, tiles_x, frame);
    return after_launch("harris_fused_kernel", st, ev);
  }
  const size_t px = (size_t)p.w * p.h * in->batch;
  Workspace ws;
  rc = workspace_get(px * 2 * 6, &ws);
  if (rc) return rc;
  int16_t *base = (int16_t *)ws.base;
  p.dx = base;
  p.dy = base + px;
  p.sx = base + 2 * px;
  p.sy = base + 3 * px;
  p.sxy = base + 4 * px;
  p.dxy = base + 5 * px;
  const dim3 g(cdiv(p.w, 32), cdiv(p.h, 8), in->batch);
  cudaEvent_t ev = before_launch(st);
  harris_deriv_kernel<<<g, 256, 0, st>>>(p, 0);
  harris_deriv_kernel<<<g, 256, 0, st>>>(p, 1);
  harris_square_kernel<<<g, 256, 0, st>>>(p, 0);
  harris_square_kernel<<<g, 256, 0, st>>>(p, 1);
  harris_square_kernel<<<g, 256, 0, st>>>(p, 2);
  // as the sample: the Gaussians of sx and sy overwrite dx and dy
  harris_gauss_kernel<<<g, 256, 0, st>>>(p, p.sx, p.dx);
  harris_gauss_kernel<<<g, 256, 0, st>>>(p, p.sy, p.dy);
  harris_gauss_kernel<<<g, 256, 0, st>>>(p, p.sxy, p.dxy);
  harris_response_kernel<<<g, 256, 0, st>>>(p);
  return after_launch("harris nine launches", st, ev);
}

extern "C" int hgb_unsharp(const hgb_view *in, const hgb_view *out, int boundary, int mode, void *stream) {
  int rc = check_view(in, "in");
  if (rc) return rc;
  rc = check_view(out, "out");
  if (rc) return rc;
  HGB_REQUIRE(in->dtype == HGB_U8X4 && out->dtype == HGB_U8X4, "hgb_unsharp: uchar4 images expected");
  HGB_REQUIRE(in->width == out->width && in->height == out->height && in->batch == out->batch,
              "hgb_unsharp: size mismatch");
  HGB_REQUIRE(in->data != out->data, "hgb_unsharp: in and out must differ");
  HGB_REQUIRE(in->pitch % 4 == 0 && out->pitch % 4 == 0 && in->batch_stride % 4 == 0 && out->batch_stride % 4 == 0 &&
                  (uintptr_t)in->data % 4 == 0 && (uintptr_t)out->data % 4 == 0,
              "hgb_unsharp: uchar4 rows must be 4-byte aligned");
  HGB_REQUIRE(boundary >= 0 && boundary <= 4, "hgb_unsharp: bad boundary");
  HGB_REQUIRE(mode == 0 || mode == 1, "hgb_unsharp: mode must be 0 (fused) or 1 (five launches)");
  UnsharpParams p;
  memset(&p, 0, sizeof(p));
  p.in = (const uchar4 *)in->data;
  p.in_p = in->pitch / 4;
  p.in_b = in->batch_stride / 4;
  p.out = (uchar4 *)out->data;
  p.out_p = out->pitch / 4;
  p.out_b = out->batch_stride / 4;
  p.w = in->width;
  p.h = in->height;
  p.bmode = boundary;
  p.batch = in->batch;
  p.nz = kNegativeZeros;
  rc = unsharp_tables(&p.tab);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  if (mode == 0) {
    const UnsharpShape u = unsharp_shape(p.w, p.h, in->batch);
    HGB_REQUIRE(u.ctas < 0x7fffffff, "hgb_unsharp: image too large");
    cudaEvent_t ev = before_launch(st);
    unsharp_kernel(u.np)<<<(unsigned)u.ctas, UF_NT, 0, st>>>(p, u.strips, u.rows, u.segments);
    return after_launch("unsharp_fused_kernel", st, ev);
  }
  const size_t px = (size_t)p.w * p.h * in->batch;
  Workspace ws;
  rc = workspace_get(px * 4 * 4, &ws);
  if (rc) return rc;
  float *base = (float *)ws.base;
  p.gray = base;
  p.blur = base + px;
  p.sharp = base + 2 * px;
  p.ratio = base + 3 * px;
  const dim3 g(cdiv(p.w, 32), cdiv(p.h, 8), in->batch);
  cudaEvent_t ev = before_launch(st);
  unsharp_gray_kernel<<<g, 256, 0, st>>>(p);
  unsharp_blur_kernel<<<g, 256, 0, st>>>(p);
  unsharp_sharp_kernel<<<g, 256, 0, st>>>(p);
  unsharp_ratio_kernel<<<g, 256, 0, st>>>(p);
  unsharp_scale_kernel<<<g, 256, 0, st>>>(p);
  return after_launch("unsharp five launches", st, ev);
}
