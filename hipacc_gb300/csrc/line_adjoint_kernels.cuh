// line_adjoint_kernels.cuh -- adjoint of the SUM local operator with a 1 x K or K x 1
// mask (K odd, 3..15), and of the column pass of a separable filter.
//
// out(j) = sum_k m_k in(r(j + k - R)) along one axis (r = boundary remap,
// lib/AST/BorderHandling.cpp:41-120), so
//   grad_in(i) = sum over the virtual positions v that r sends to i (i itself
//                first) of sum_k m_k grad_out(v - (k - R)),
//   grad_m(k)  = sum_j grad_out(j) in(r(j + k - R)),
// CONSTANT taps outside carrying no gradient and reading 0 in grad_m.
//
// One pass: a CTA walks 64 x 32 tiles (64 x 8 on small batches), stages grad_out (zero outside the image)
// and in (through the boundary) with the halo of one axis, and a thread keeps
// 4 x 4 (4 x 1) pixels: grad_in from register windows, the tap gradient in one packed
// f32x2 accumulator per tap, which joins the warp's compensated sums after each tile
// (tap_fold.cuh).  The general
// kernels (local_adjoint.cu) read every tap from global memory and walk the
// images once per tap.  In the column form of a separable filter the row pass
// t = rows(in) is recomputed in shared memory (the forward's operations and
// order) instead of written to memory and read back.
// Bound by the wait for each tile's loads and by latencies at 6 to 9 CTAs per SM (issue
// slots 49 to 53 % busy, first stall long_scoreboard): a tile is staged, then computed.
// Forward and adjoint of the separable filter: K = 9 on 4 images of 1920 x 1080
// 485 -> 87 us, K = 5 on 4096 x 2048 689 -> 90 us.
//
// Included by line_k3_9.cu and line_k11_15.cu, which compile in parallel.
#pragma once

#include "band.cuh"
#include "line_adjoint.h"
#include "stage_groups.cuh"
#include "tap_fold.cuh"

namespace hgb {

template <int K, int FORM, int LN_PY>
struct LnShape {
  static constexpr int LN_TH = 8 * LN_PY;
  static constexpr int R = K / 2, HL = round_up(R, 4);
  static constexpr bool kRow = FORM == kLineRow;
  static constexpr int SWG = kRow ? LN_TW + 2 * HL : LN_TW;  // staged columns of grad_out
  static constexpr int SWI = FORM == kLineCol ? LN_TW : LN_TW + 2 * HL;
  static constexpr int SH = kRow ? LN_TH : LN_TH + 2 * R;
};

// four consecutive f32 at p (16-byte aligned) into w[i .. i + 3]
__device__ __forceinline__ void put4(float *w, const float *p) {
  const float4 t = *reinterpret_cast<const float4 *>(p);
  w[0] = t.x;
  w[1] = t.y;
  w[2] = t.z;
  w[3] = t.w;
}

template <int K, int FORM, bool DEV, int LN_PY>
__global__ void __launch_bounds__(LN_NT) line_adjoint_kernel(const __grid_constant__ LineAdjParams p) {
  using S = LnShape<K, FORM, LN_PY>;
  constexpr int LN_TH = S::LN_TH, R = S::R, HL = S::HL, SWG = S::SWG, SWI = S::SWI, SH = S::SH;
  constexpr bool kRow = S::kRow, kT = FORM == kLineColOfRows;
  constexpr int SWX = kRow ? SWI : LN_TW;  // row pitch of what the tap gradient reads
  __shared__ __align__(16) float sg[SH * SWG];
  __shared__ __align__(16) float si[SH * SWI];
  __shared__ __align__(16) float st[kT ? SH * LN_TW : 4];
  __shared__ float sm[DEV ? K : 1];
  __shared__ TapSum sum[LN_NT / 32][K];  // tap gradient of each warp's pixels
  if (DEV) {
    if (threadIdx.x < K) sm[threadIdx.x] = __ldg(p.mask_dev + threadIdx.x);
    __syncthreads();
  }
  auto tap = [&](int k) { return DEV ? sm[k] : p.mask[k]; };
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  if (threadIdx.x < LN_NT / 32 * K) (&sum[0][0])[threadIdx.x] = TapSum{0.0f, 0.0f};
  for (int t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
    const int per = p.tiles_x * p.tiles_y, b = t / per, rt = t - b * per, by = rt / p.tiles_x;
    const int i0 = (rt - by * p.tiles_x) * LN_TW, j0 = by * LN_TH;
    const char *gout = (const char *)p.gout + b * p.gout_b;
    const int gx = kRow ? i0 - HL : i0, gy = kRow ? j0 : j0 - R;
    stage_groups<float, SWG, SH, LN_NT>(sg, gout, p.gout_p, gx, gy, 0, p.w, 0, p.h, HGB_BOUNDARY_CONSTANT, 0.0f, 0);
    if (p.part)
      stage_groups<float, SWI, SH, LN_NT>(si, (const char *)p.in + b * p.in_b, p.in_p, kT ? i0 - HL : gx, gy, 0, p.w, 0,
                                          p.h, p.bmode, kT ? p.cval : 0.0f, R);
    stage_wait();
    __syncthreads();
    if (kT && p.part) {  // t = rows(in) on the staged rows
      for (int c = threadIdx.x; c < SH * (LN_TW / 4); c += LN_NT) {
        const int r = c / (LN_TW / 4), k4 = c - r * (LN_TW / 4);
        float w[4 + 2 * HL];
#pragma unroll
        for (int v = 0; v < (4 + 2 * HL) / 4; ++v) put4(w + 4 * v, &si[r * SWI + 4 * k4 + 4 * v]);
        f2 a0 = 0ull, a1 = 0ull;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const f2 m = f2_pack(p.row[k], p.row[k]);
          a0 = f2_fma(m, f2_pack(w[HL - R + k], w[HL - R + k + 1]), a0);
          a1 = f2_fma(m, f2_pack(w[HL - R + k + 2], w[HL - R + k + 3]), a1);
        }
        // CONSTANT rows outside the image read 0 in the tap gradient
        const bool out = p.bmode == HGB_BOUNDARY_CONSTANT && (gy + r < 0 || gy + r >= p.h);
        reinterpret_cast<float4 *>(st)[c] = out ? make_float4(0.0f, 0.0f, 0.0f, 0.0f)
                                                : make_float4(f2_lo(a0), f2_hi(a0), f2_lo(a1), f2_hi(a1));
      }
      __syncthreads();
    }
    const float *sx = kT ? st : si;
    const int x = i0 + 4 * tx, y0 = j0 + ty * LN_PY;
    if (x < p.w && y0 < p.h) {
      // ---- grad_in
      f2 G[LN_PY][2];
      if (p.gin) {
#pragma unroll
        for (int oy = 0; oy < LN_PY; ++oy) G[oy][0] = G[oy][1] = 0ull;
        if constexpr (kRow) {
#pragma unroll
          for (int oy = 0; oy < LN_PY; ++oy) {
            float w[4 + 2 * HL];
#pragma unroll
            for (int v = 0; v < (4 + 2 * HL) / 4; ++v) put4(w + 4 * v, &sg[(ty * LN_PY + oy) * SWG + 4 * tx + 4 * v]);
#pragma unroll
            for (int k = 0; k < K; ++k) {  // column x - (k - R)
              const float mv = tap(k);
              const f2 m = f2_pack(mv, mv);
              G[oy][0] = f2_fma(m, f2_pack(w[HL + R - k], w[HL + R - k + 1]), G[oy][0]);
              G[oy][1] = f2_fma(m, f2_pack(w[HL + R - k + 2], w[HL + R - k + 3]), G[oy][1]);
            }
          }
        } else {
#pragma unroll
          for (int r = LN_PY + K - 2; r >= 0; --r) {  // rows descending: taps ascending per output
            const float4 v = *reinterpret_cast<const float4 *>(&sg[(ty * LN_PY + r) * SWG + 4 * tx]);
            const f2 v0 = f2_pack(v.x, v.y), v1 = f2_pack(v.z, v.w);
#pragma unroll
            for (int oy = 0; oy < LN_PY; ++oy) {
              const int k = oy + 2 * R - r;
              if (k < 0 || k >= K) continue;
              const float mv = tap(k);
              const f2 m = f2_pack(mv, mv);
              G[oy][0] = f2_fma(m, v0, G[oy][0]);
              G[oy][1] = f2_fma(m, v1, G[oy][1]);
            }
          }
        }
#pragma unroll
        for (int oy = 0; oy < LN_PY; ++oy) {
          const int y = y0 + oy;
          if (y >= p.h) break;
          const float o[4] = {f2_lo(G[oy][0]), f2_hi(G[oy][0]), f2_lo(G[oy][1]), f2_hi(G[oy][1])};
          float *dst = reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + (int64_t)y * p.gin_p) + x;
          if (x + 4 <= p.w && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
            *reinterpret_cast<float4 *>(dst) = make_float4(o[0], o[1], o[2], o[3]);
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (x + q < p.w) dst[q] = o[q];
          }
        }
      }
    }
    // ---- tap gradient
    if (p.part) {
      f2 gm[K];  // even and odd pixels of the pairs
#pragma unroll
      for (int k = 0; k < K; ++k) gm[k] = 0ull;
      if (x < p.w && y0 < p.h) {
        if (x + 4 <= p.w && y0 + LN_PY <= p.h) {
          f2 g0[LN_PY], g1[LN_PY];
#pragma unroll
          for (int oy = 0; oy < LN_PY; ++oy) {
            const float4 v = *reinterpret_cast<const float4 *>(
                &sg[(ty * LN_PY + oy + (kRow ? 0 : R)) * SWG + 4 * tx + (kRow ? HL : 0)]);
            g0[oy] = f2_pack(v.x, v.y);
            g1[oy] = f2_pack(v.z, v.w);
          }
          if constexpr (kRow) {
#pragma unroll
            for (int oy = 0; oy < LN_PY; ++oy) {
              float w[4 + 2 * HL];
#pragma unroll
              for (int v = 0; v < (4 + 2 * HL) / 4; ++v)
                put4(w + 4 * v, &sx[(ty * LN_PY + oy) * SWX + 4 * tx + 4 * v]);
#pragma unroll
              for (int k = 0; k < K; ++k) {
                gm[k] = f2_fma(g0[oy], f2_pack(w[HL - R + k], w[HL - R + k + 1]), gm[k]);
                gm[k] = f2_fma(g1[oy], f2_pack(w[HL - R + k + 2], w[HL - R + k + 3]), gm[k]);
              }
            }
          } else {
#pragma unroll
            for (int r = 0; r < LN_PY + K - 1; ++r) {
              const float4 v = *reinterpret_cast<const float4 *>(&sx[(ty * LN_PY + r) * SWX + 4 * tx]);
              const f2 v0 = f2_pack(v.x, v.y), v1 = f2_pack(v.z, v.w);
#pragma unroll
              for (int oy = 0; oy < LN_PY; ++oy) {
                const int k = r - oy;
                if (k < 0 || k >= K) continue;
                gm[k] = f2_fma(g0[oy], v0, gm[k]);
                gm[k] = f2_fma(g1[oy], v1, gm[k]);
              }
            }
          }
        } else {  // groups that leave the image: only the pixels inside
#pragma unroll 1
          for (int oy = 0; oy < LN_PY && y0 + oy < p.h; ++oy)
#pragma unroll 1
            for (int q = 0; q < 4 && x + q < p.w; ++q) {
              const int r = ty * LN_PY + oy;
              const float g = sg[(r + (kRow ? 0 : R)) * SWG + 4 * tx + q + (kRow ? HL : 0)];
#pragma unroll
              for (int k = 0; k < K; ++k)
                gm[k] = f2_fma(f2_pack(g, 0.0f),
                               f2_pack(kRow ? sx[r * SWX + 4 * tx + q + HL - R + k] : sx[(r + k) * SWX + 4 * tx + q], 0.0f),
                               gm[k]);
            }
        }
      }
      float v[K];
#pragma unroll
      for (int k = 0; k < K; ++k) v[k] = f2_lo(gm[k]) + f2_hi(gm[k]);
      fold_taps(v, sum[threadIdx.x >> 5], 0, K);
    }
    // ---- near a border: a pixel with other pre-images sums over all of them, a
    // band pixel per thread, only the taps that reach back into the image.  On
    // images of a few pixels hundreds of terms meet in one and cancel, so the
    // few band sums run in FP64
    if (p.gin && p.bmode != HGB_BOUNDARY_CONSTANT) {
      const TileBand band = tile_band<R>(i0, j0, LN_TW, LN_TH, p.w, p.h, !kRow, kRow);
      if (band.count > 0) {
        __syncthreads();  // the sums without the other pre-images are written
#pragma unroll 1
        for (int c = threadIdx.x; c < band.count; c += LN_NT) {
          int bx, by2;
          tile_band_pos(band, c, bx, by2);
          const int ix = i0 + bx, iy = j0 + by2, n = kRow ? p.w : p.h;
          const unsigned pre = preimage_bits<R>(p.bmode, kRow ? ix : iy, n);
          if (!pre) continue;
          float *dst = reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + (int64_t)iy * p.gin_p) + ix;
          double o = 0.0;
#pragma unroll 1
          for (int a = -1; a < 2 * R; ++a) {
            if (a >= 0 && !(pre >> a & 1u)) continue;
            const int v = a < 0 ? (kRow ? ix : iy) : preimage_pos<R>(a, n), m1 = min(K - 1, v + R);
#pragma unroll 2
            for (int k = max(0, v + R - n + 1); k <= m1; ++k) {
              const int j = v - (k - R);
              const int rx = kRow ? j - (i0 - HL) : bx, ry = kRow ? by2 : j - (j0 - R);
              float g;
              if (rx >= 0 && rx < SWG && ry >= 0 && ry < SH)
                g = sg[ry * SWG + rx];
              else  // REPEAT reaches the other side of the image
                g = __ldg(reinterpret_cast<const float *>(gout + (int64_t)(kRow ? iy : j) * p.gout_p) + (kRow ? j : ix));
              o = fma((double)tap(k), (double)g, o);
            }
          }
          *dst = (float)o;
        }
      }
    }
    __syncthreads();  // the tile is read before the next one is staged
  }
  if (!p.part) return;
  // the tiles end with a barrier
  if (threadIdx.x < K) p.part[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = tap_total(sum, threadIdx.x);
}

template <int K, int PY>
LineKernel line_kernel_py(LineForm f, bool dev) {
  if (f == kLineColOfRows) return line_adjoint_kernel<K, kLineColOfRows, false, PY>;
  if (f == kLineRow) return dev ? line_adjoint_kernel<K, kLineRow, true, PY> : line_adjoint_kernel<K, kLineRow, false, PY>;
  return dev ? line_adjoint_kernel<K, kLineCol, true, PY> : line_adjoint_kernel<K, kLineCol, false, PY>;
}
template <int K>
LineKernel line_kernel_k(LineForm f, bool dev, int py) {
  return py == 4 ? line_kernel_py<K, 4>(f, dev) : line_kernel_py<K, 1>(f, dev);
}

}  // namespace hgb
