// local_minmax_kernels.cuh -- MIN / MAX over a Domain (erosion, dilation) on tiles.
//
// Semantics: Kernel::reduce(Domain, Reduce::MIN / MAX) (dsl/kernel.hpp:270-296;
// lib/AST/Convolution.cpp:43-100): acc starts at FLT_MAX (MIN) or FLT_MIN
// (MAX) and takes acc = acc < v ? acc : v (acc > v ? acc : v) over the cells in
// row-major order.
//
// Without NaNs and negative zeros that fold does not depend on the order, so
// the tile is reduced by rows: for one staged row, the minima H_h of the runs
// of half-width h follow from each other, H_h(x) = min(H_{h-1}(x), v(x - h),
// v(x + h)) (one three-input minimum), and each output takes one more minimum
// per row of the Domain.  MAX runs as MIN of the negated values (exact).  A CTA
// whose staged tile holds a NaN or a negative zero folds its outputs cell by
// cell in the stated order instead.
//
// Included by the per-storage-type units lmm_{f32,bf16,f16,u8}.cu.
#pragma once

#include <cfloat>

#include "local_minmax.h"
#include "stage_groups.cuh"

namespace hgb {

constexpr int MM_BX = 16, MM_BY = 8, MM_NT = MM_BX * MM_BY, MM_PX = 4;

// Row profiles known at compile time, four bits per row: 0 for an empty row,
// else the run's half-width + 1.  Every half-width of the two commonest
// structuring elements, the square and the disc, is then a constant; other
// profiles (kAnyProfile) test sel[] per row.  The tests and their predicated
// minima kept the ALU pipe 70 % busy and the instruction cache missing: 64 u8
// images of 1024 x 1024 through the 5 x 5 disc took 202 us that way (1091 us
// in the general kernel, one pixel per thread over 16 x 16 tiles), 143 us
// with the profile compiled in and 82 us with the staging as it is now (ALU pipe
// 69 %, issue slots 66 % busy).
constexpr uint32_t kAnyProfile = 0;
__host__ __device__ constexpr uint32_t square_profile(int k) {
  uint32_t v = 0;
  for (int y = 0; y < k; ++y) v |= (uint32_t)(k / 2 + 1) << (4 * y);
  return v;
}
__host__ __device__ constexpr uint32_t disc_profile(int k) {  // x^2 + y^2 <= (k / 2)^2 about the centre
  uint32_t v = 0;
  for (int y = 0; y < k; ++y) {
    const int dy = y - k / 2;
    int h = 0;
    while (h < k / 2 && 4 * ((h + 1) * (h + 1) + dy * dy) <= k * k) ++h;
    v |= (uint32_t)(h + 1) << (4 * y);
  }
  return v;
}

template <typename TI, int K, int PY, uint32_t PROFILE>
__global__ void __launch_bounds__(MM_NT) minmax_kernel(const __grid_constant__ MinMaxKernelParams p) {
  constexpr int R = K / 2, HL = 4, TW = MM_BX * MM_PX, TH = MM_BY * PY, SW = TW + 2 * HL, SH = TH + 2 * R;
  __shared__ __align__(16) float tile[SH * SW];
  const int b = blockIdx.z, i0 = blockIdx.x * TW, j0 = blockIdx.y * TH;
  const char *in = p.in + (int64_t)b * p.in_bstride;
  const uint32_t flip = p.flip;
  // ---- stage, with the sign of MAX; note NaNs and negative zeros
  int odd = 0;
  auto put = [&](int c, float4 v) {
    const uint32_t u[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
    if constexpr (sizeof(TI) > 1) {
#pragma unroll
      for (int q = 0; q < 4; ++q) odd |= (u[q] == 0x80000000u) | ((u[q] & 0x7fffffffu) > 0x7f800000u);
    }
    reinterpret_cast<uint4 *>(tile)[c] = make_uint4(u[0] ^ flip, u[1] ^ flip, u[2] ^ flip, u[3] ^ flip);
  };
  stage_groups_each<TI, SW, SH, MM_NT>(in, p.in_pitch, p.ax + i0 - HL, p.ay + j0 - R, p.ax, p.ax + p.aw, p.ay,
                                       p.ay + p.ah, p.bmode, p.cval, R + p.excess, put);
  if constexpr (sizeof(TI) == 1) {  // bytes are neither; the constant may be
    const uint32_t u = __float_as_uint(p.cval);
    odd = u == 0x80000000u || (u & 0x7fffffffu) > 0x7f800000u;
    __syncthreads();
  } else {
    odd = __syncthreads_or(odd);
  }
  const int tx = threadIdx.x % MM_BX, ty = threadIdx.x / MM_BX;
  float acc[PY][MM_PX];
  const float first = flip ? -FLT_MIN : FLT_MAX;
#pragma unroll
  for (int oy = 0; oy < PY; ++oy)
#pragma unroll
    for (int q = 0; q < MM_PX; ++q) acc[oy][q] = first;
  if (!odd) {
    // two staged rows at a time: an output that both reach takes one three-input minimum
    static_assert((PY + K - 1) % 2 == 0, "row pairs");
#pragma unroll
    for (int r = 0; r < PY + K - 1; r += 2) {
      float H[2][R + 1][MM_PX];  // the run minima of both rows
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        float w[12];
        const float4 *row = reinterpret_cast<const float4 *>(&tile[(ty * PY + r + l) * SW + tx * MM_PX]);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const float4 t = row[v];
          w[4 * v] = t.x;
          w[4 * v + 1] = t.y;
          w[4 * v + 2] = t.z;
          w[4 * v + 3] = t.w;
        }
#pragma unroll
        for (int h = 0; h <= R; ++h)
#pragma unroll
          for (int q = 0; q < MM_PX; ++q)
            H[l][h][q] = h == 0 ? w[HL + q] : fminf(fminf(H[l][h > 0 ? h - 1 : 0][q], w[HL + q - h]), w[HL + q + h]);
      }
      if constexpr (PROFILE != kAnyProfile) {
#pragma unroll
        for (int oy = 0; oy < PY; ++oy) {
          const int m0 = r - oy, m1 = r + 1 - oy;
          const int h0 = m0 >= 0 && m0 < K ? (int)(PROFILE >> (4 * m0) & 15u) - 1 : -1;
          const int h1 = m1 >= 0 && m1 < K ? (int)(PROFILE >> (4 * m1) & 15u) - 1 : -1;
#pragma unroll
          for (int q = 0; q < MM_PX; ++q) {
            if (h0 >= 0 && h1 >= 0)
              acc[oy][q] = fminf(fminf(acc[oy][q], H[0][h0 < 0 ? 0 : h0][q]), H[1][h1 < 0 ? 0 : h1][q]);
            else if (h0 >= 0)
              acc[oy][q] = fminf(acc[oy][q], H[0][h0 < 0 ? 0 : h0][q]);
            else if (h1 >= 0)
              acc[oy][q] = fminf(acc[oy][q], H[1][h1 < 0 ? 0 : h1][q]);
          }
        }
      } else {
#pragma unroll
        for (int l = 0; l < 2; ++l)
#pragma unroll
          for (int h = 0; h <= R; ++h)
#pragma unroll
            for (int oy = 0; oy < PY; ++oy) {
              const int my = r + l - oy;
              if (my < 0 || my >= K) continue;
              if (p.d.sel[h] >> my & 1u) {
#pragma unroll
                for (int q = 0; q < MM_PX; ++q) acc[oy][q] = fminf(acc[oy][q], H[l][h][q]);
              }
            }
      }
    }
  } else {
#pragma unroll
    for (int oy = 0; oy < PY; ++oy)
#pragma unroll 1
      for (int my = 0; my < K; ++my)
#pragma unroll 1
        for (int mx = 0; mx < K; ++mx) {
          if (!(p.d.rows[my] >> mx & 1u)) continue;
#pragma unroll
          for (int q = 0; q < MM_PX; ++q) {
            const float v = tile[(ty * PY + oy + my) * SW + tx * MM_PX + q + HL - R + mx];
            acc[oy][q] = acc[oy][q] < v ? acc[oy][q] : v;
          }
        }
  }
  // ---- store
  const int i = i0 + tx * MM_PX;
  char *out = p.out + (int64_t)b * p.out_bstride;
#pragma unroll
  for (int oy = 0; oy < PY; ++oy) {
    const int j = j0 + ty * PY + oy;
    if (j >= p.ih || i >= p.iw) continue;
    float v[MM_PX];
#pragma unroll
    for (int q = 0; q < MM_PX; ++q) v[q] = __uint_as_float(__float_as_uint(acc[oy][q]) ^ flip);
    TI *dst = reinterpret_cast<TI *>(out + (int64_t)(p.iy + j) * p.out_pitch) + p.ix + i;
    if (p.vec_out && i + MM_PX <= p.iw) {
      TI t4[4] = {Storage<TI>::from_f(v[0]), Storage<TI>::from_f(v[1]), Storage<TI>::from_f(v[2]),
                  Storage<TI>::from_f(v[3])};
      if constexpr (sizeof(TI) == 4)
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
      else if constexpr (sizeof(TI) == 2)
        *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(t4);
      else
        *reinterpret_cast<uint32_t *>(dst) = (uint32_t)t4[0] | (uint32_t)t4[1] << 8 | (uint32_t)t4[2] << 16 |
                                             (uint32_t)t4[3] << 24;
    } else {
#pragma unroll
      for (int q = 0; q < MM_PX; ++q)
        if (i + q < p.iw) dst[q] = Storage<TI>::from_f(v[q]);
    }
  }
}

template <typename TI, int K, uint32_t PROFILE>
int launch_minmax(const MinMaxKernelParams &p, int batch, cudaStream_t st) {
  // 64 x 64 tiles; lower ones where those would not give every SM four CTAs
  const int64_t cols = (int64_t)cdiv(p.iw, 64) * batch, want = 4 * num_sms();
  cudaEvent_t ev = before_launch(st);
  if (cols * cdiv(p.ih, 64) >= want)
    minmax_kernel<TI, K, 8, PROFILE><<<dim3(cdiv(p.iw, 64), cdiv(p.ih, 64), batch), MM_NT, 0, st>>>(p);
  else if (cols * cdiv(p.ih, 32) >= want)
    minmax_kernel<TI, K, 4, PROFILE><<<dim3(cdiv(p.iw, 64), cdiv(p.ih, 32), batch), MM_NT, 0, st>>>(p);
  else
    minmax_kernel<TI, K, 2, PROFILE><<<dim3(cdiv(p.iw, 64), cdiv(p.ih, 16), batch), MM_NT, 0, st>>>(p);
  return after_launch("minmax_kernel", st, ev);
}

template <typename TI, int K>
int launch_minmax_profile(const MinMaxKernelParams &p, int batch, cudaStream_t st) {
  uint32_t v = 0;
  for (int h = 0; h <= K / 2; ++h)
    for (int y = 0; y < K; ++y)
      if (p.d.sel[h] >> y & 1u) v |= (uint32_t)(h + 1) << (4 * y);
  if (v == square_profile(K)) return launch_minmax<TI, K, square_profile(K)>(p, batch, st);
  if constexpr (disc_profile(K) != square_profile(K))
    if (v == disc_profile(K)) return launch_minmax<TI, K, disc_profile(K)>(p, batch, st);
  return launch_minmax<TI, K, kAnyProfile>(p, batch, st);
}

template <typename TI>
int launch_minmax_k(const MinMaxKernelParams &p, int batch, cudaStream_t st) {
  switch (p.d.k) {
    case 3: return launch_minmax_profile<TI, 3>(p, batch, st);
    case 5: return launch_minmax_profile<TI, 5>(p, batch, st);
    default: return launch_minmax_profile<TI, 7>(p, batch, st);
  }
}

}  // namespace hgb
