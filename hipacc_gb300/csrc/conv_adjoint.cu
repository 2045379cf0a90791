// conv_adjoint.cu -- adjoint of the SUM local operator with a square mask,
//   out(j) = sum_o m_o in(r(j + o)),  o = (mx - R, my - R)
// (r = boundary remap, lib/AST/BorderHandling.cpp:41-120):
//   grad_in(i) = sum over the virtual positions v that r sends to i (i itself
//                first) of sum_o m_o grad_out(v - o),
//   grad_m(o)  = sum_j grad_out(j) in(r(j + o)),
// CONSTANT taps outside carrying no gradient and reading 0 in grad_m.
//
// A CTA walks 64 x 32 tiles (64 x 8 on small batches), stages grad_out (zero
// outside the image) and in (through the boundary) with the mask's halo, and a
// thread keeps 4 x 4 (4 x 1) pixels.  grad_in: each staged row is read once and
// serves all the thread's rows, two pixels per packed f32x2 operation.  grad_m: a
// row of in, the same way, against the thread's grad_out, two taps per packed
// operation; a tile's sums join the warp's compensated ones (tap_fold.cuh).  The next tile is
// staged (asynchronous copies) while this one computes.  Any row alignment.
//
// Bound by instruction fetch (the unrolled passes) and latencies at 16 to 24 warps per SM
// (the mask gradient's registers): 7 x 7 keeps 42 % of the issue slots and of the FMA pipe
// busy, its first stall is no_instruction.  Its 2 K^2 lane operations per pixel are 24 us of
// the 88 us that 8.4 Mpx take.  Two kernels without a register block over rows took the
// layouts and forms that come here before: 7 x 7 on 2 images of 2049 x 2051 224 us, now 96 us.
#include <algorithm>
#include <cstring>

#include "band.cuh"
#include "conv_adjoint.h"
#include "stage_groups.cuh"
#include "tap_fold.cuh"

namespace hgb {
namespace {

constexpr int CA_NT = 128, CA_TW = 64, CA_SW = CA_TW + 8;

__device__ __forceinline__ void ca_window(const float *row, f2 (&E)[6], f2 (&O)[5]) {
  float w[12];
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    const float4 t = reinterpret_cast<const float4 *>(row)[v];
    w[4 * v] = t.x;
    w[4 * v + 1] = t.y;
    w[4 * v + 2] = t.z;
    w[4 * v + 3] = t.w;
  }
#pragma unroll
  for (int j = 0; j < 6; ++j) E[j] = f2_pack(w[2 * j], w[2 * j + 1]);
#pragma unroll
  for (int j = 0; j < 5; ++j) O[j] = f2_pack(w[2 * j + 1], w[2 * j + 2]);
}

// The pixels that the boundary sends other positions to (within R of an edge): the
// whole sum over their pre-images, only the taps that reach back into the image,
// by four lanes (a quarter of the mask's rows each).  Every CTA takes an equal share
// while its first tile lands; the tiles leave these pixels out.  Done by the tiles
// after their own pixels, a border tile took twice an inner one's time and the CTAs
// that drew two of them set the launch's (60 -> 54 us for 7 x 7 on 2048 x 2048).  S = double on images hardly wider than the mask, where
// hundreds of terms meet in one pixel and cancel.
template <int K, typename S>
__device__ __forceinline__ void ca_frame(const ConvAdjParams &p, const float *msk) {
  constexpr int R = K / 2;
  const TileBand f = tile_band<R>(0, 0, p.w, p.h, p.w, p.h, true, true);
  const int64_t n = (int64_t)f.count * p.batch;
  const int64_t k0 = n * blockIdx.x / gridDim.x, k1 = n * (blockIdx.x + 1) / gridDim.x;
#pragma unroll 1
  for (int64_t kb = k0; kb < k1; kb += CA_NT / 4) {
    const int64_t k = kb + threadIdx.x / 4;
    const int part = threadIdx.x % 4;
    // (a 64-bit division takes several times a 32-bit one)
    const int b = k >= k1 ? p.batch : (n < 0x7fffffff ? (int)((unsigned)k / (unsigned)f.count) : (int)(k / f.count));
    int ix = 0, iy = 0;
    unsigned px = 0, py = 0;
    if (b < p.batch) {
      tile_band_pos(f, (int)(k - (int64_t)b * f.count), ix, iy);
      px = preimage_bits<R>(p.bmode, ix, p.w);
      py = preimage_bits<R>(p.bmode, iy, p.h);
    }
    S s = S(0);
    if (px | py) {
      const char *gout = (const char *)p.gout + b * p.gout_b;
      for (unsigned ym = py << 1 | 1u; ym; ym &= ym - 1u) {  // bit 0: the row itself
        const int vy = ym & 1u ? iy : preimage_pos<R>(__ffs((int)ym) - 2, p.h), lo = max(0, vy + R - p.h + 1);
#pragma unroll 1
        for (int my = lo + ((part - lo) & 3); my <= min(K - 1, vy + R); my += 4) {
          const float *grow = reinterpret_cast<const float *>(gout + (int64_t)(vy - (my - R)) * p.gout_p);
          for (unsigned xm = px << 1 | 1u; xm; xm &= xm - 1u) {
            const int vx = xm & 1u ? ix : preimage_pos<R>(__ffs((int)xm) - 2, p.w);
#pragma unroll
            for (int mx = 0; mx < K; ++mx) {  // a row's loads in flight together
              const int jx = vx - (mx - R);
              if (jx >= 0 && jx < p.w) s += (S)msk[my * K + mx] * (S)__ldg(grow + jx);
            }
          }
        }
      }
    }
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if ((px | py) && part == 0)
      reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + (int64_t)iy * p.gin_p)[ix] = (float)s;
  }
}

// CTAs per SM: the mask gradient's registers (8, 30 and 56 of them) leave room for six, five and four
template <int K, int PY>
__global__ void __launch_bounds__(CA_NT, K == 3 ? 6 : (K == 5 ? 5 : 4)) conv_adjoint_kernel(const __grid_constant__ ConvAdjParams p) {
  constexpr int R = K / 2, TH = 8 * PY, SH = TH + 2 * R, NP = (K + 1) / 2;
  static_assert(R <= 3, "twelve-value windows cover radius 3");
  extern __shared__ __align__(16) float ca_stage[];  // two buffers of [grad_out][in]: the next tile lands meanwhile
  __shared__ __align__(16) f2 m2[K][2 * NP];  // mask pairs (m, m), an even count per row
  __shared__ float msk[K * K];
  __shared__ TapSum sum[CA_NT / 32][K * K];  // mask gradient of each warp's pixels
  for (int i = threadIdx.x; i < K * 2 * NP; i += CA_NT) {
    const int y = i / (2 * NP), x = i - y * (2 * NP);
    const float m = x < K ? (p.mask_dev ? __ldg(p.mask_dev + y * K + x) : p.mask[y * K + x]) : 0.0f;
    m2[y][x] = f2_pack(m, m);
    if (x < K) msk[y * K + x] = m;
  }
  for (int i = threadIdx.x; i < CA_NT / 32 * K * K; i += CA_NT) (&sum[0][0])[i] = TapSum{0.0f, 0.0f};
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  auto origin = [&](int t, int &b, int &i0, int &j0) {
    const int per = p.tiles_x * p.tiles_y;
    b = t / per;
    const int rt = t - b * per, by = rt / p.tiles_x;
    i0 = (rt - by * p.tiles_x) * CA_TW;
    j0 = by * TH;
  };
  auto stage = [&](int t, int s) {
    int b, i0, j0;
    origin(t, b, i0, j0);
    float *buf = ca_stage + s * 2 * SH * CA_SW;
    stage_groups<float, CA_SW, SH, CA_NT>(buf, (const char *)p.gout + b * p.gout_b, p.gout_p, i0 - 4, j0 - R, 0, p.w, 0,
                                          p.h, HGB_BOUNDARY_CONSTANT, 0.0f, 0);
    if (p.part)
      stage_groups<float, CA_SW, SH, CA_NT>(buf + SH * CA_SW, (const char *)p.in + b * p.in_b, p.in_p, i0 - 4, j0 - R,
                                            0, p.w, 0, p.h, p.bmode, 0.0f, R);
  };
  stage(blockIdx.x, 0);
  stage_commit();
  __syncthreads();  // the mask is there
  if (p.gin && p.bmode != HGB_BOUNDARY_CONSTANT) {
    if (p.w < 2 * K || p.h < 2 * K)
      ca_frame<K, double>(p, msk);
    else
      ca_frame<K, float>(p, msk);
  }
#pragma unroll 1
  for (int t = blockIdx.x, it = 0; t < p.ntiles; t += gridDim.x, ++it) {
    const int s = it & 1;
    if (t + (int)gridDim.x < p.ntiles) stage(t + gridDim.x, s ^ 1);
    stage_commit();
    stage_wait_but_newest();
    __syncthreads();
    int b, i0, j0;
    origin(t, b, i0, j0);
    const float *sg = ca_stage + s * 2 * SH * CA_SW, *sx = sg + SH * CA_SW;
    const int x = i0 + 4 * tx, y0 = j0 + ty * PY;
    if (p.gin && x < p.w && y0 < p.h) {
      f2 G[PY][2];
#pragma unroll
      for (int oy = 0; oy < PY; ++oy) G[oy][0] = G[oy][1] = 0ull;
#pragma unroll
      for (int r = PY + K - 2; r >= 0; --r) {  // rows descending: taps ascending per output
        f2 E[6], O[5];
        ca_window(&sg[(ty * PY + r) * CA_SW + 4 * tx], E, O);
#pragma unroll
        for (int oy = 0; oy < PY; ++oy) {
          const int my = oy + 2 * R - r;
          if (my < 0 || my >= K) continue;
#pragma unroll
          for (int o2 = 0; o2 < NP; ++o2) {
            const ulonglong2 mm = reinterpret_cast<const ulonglong2 *>(&m2[my][0])[o2];
#pragma unroll
            for (int l = 0; l < 2; ++l) {
              const int mx = 2 * o2 + l, s = 4 + R - mx;  // column x - (mx - R)
              if (mx >= K) continue;
              const f2 M = l ? mm.y : mm.x;
              G[oy][0] = f2_fma(M, (s & 1) ? O[s >> 1] : E[s >> 1], G[oy][0]);
              G[oy][1] = f2_fma(M, (s & 1) ? O[(s >> 1) + 1] : E[(s >> 1) + 1], G[oy][1]);
            }
          }
        }
      }
#pragma unroll
      for (int oy = 0; oy < PY; ++oy) {
        const int y = y0 + oy;
        if (y >= p.h) break;
        float *dst = reinterpret_cast<float *>((char *)p.gin + b * p.gin_b + (int64_t)y * p.gin_p) + x;
        const float o[4] = {f2_lo(G[oy][0]), f2_hi(G[oy][0]), f2_lo(G[oy][1]), f2_hi(G[oy][1])};
        if (p.bmode != HGB_BOUNDARY_CONSTANT && (x < R || x + 4 > p.w - R || y < R || y >= p.h - R)) {
          const unsigned py = preimage_bits<R>(p.bmode, y, p.h);  // pixels with other pre-images are the frame's
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (x + q < p.w && !(py | preimage_bits<R>(p.bmode, x + q, p.w))) dst[q] = o[q];
        } else if (x + 4 <= p.w && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
          *reinterpret_cast<float4 *>(dst) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (x + q < p.w) dst[q] = o[q];
        }
      }
    }
    if (p.part) {
      f2 DM[K][NP];  // mask gradient per pair of taps (my, 2 op), (my, 2 op + 1)
#pragma unroll
      for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = 0; j < NP; ++j) DM[i][j] = 0ull;
      if (x + 4 <= p.w && y0 + PY <= p.h) {
        f2 GG[PY][4];
#pragma unroll
        for (int oy = 0; oy < PY; ++oy) {
          const float4 g = *reinterpret_cast<const float4 *>(&sg[(ty * PY + oy + R) * CA_SW + 4 * tx + 4]);
          GG[oy][0] = f2_pack(g.x, g.x);
          GG[oy][1] = f2_pack(g.y, g.y);
          GG[oy][2] = f2_pack(g.z, g.z);
          GG[oy][3] = f2_pack(g.w, g.w);
        }
#pragma unroll
        for (int r = 0; r < PY + K - 1; ++r) {
          f2 E[6], O[5];
          ca_window(&sx[(ty * PY + r) * CA_SW + 4 * tx], E, O);
#pragma unroll
          for (int oy = 0; oy < PY; ++oy) {
            const int my = r - oy;
            if (my < 0 || my >= K) continue;
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
              for (int op = 0; op < NP; ++op) {
                const int s = 4 - R + q + 2 * op;  // column x + q + 2 op - R
                DM[my][op] = f2_fma(GG[oy][q], (s & 1) ? O[s >> 1] : E[s >> 1], DM[my][op]);
              }
          }
        }
      } else if (x < p.w) {  // groups that leave the image: only the pixels inside
#pragma unroll 1
        for (int oy = 0; oy < PY && y0 + oy < p.h; ++oy)
#pragma unroll 1
          for (int q = 0; q < 4 && x + q < p.w; ++q) {
            const int r = ty * PY + oy;
            const float g = sg[(r + R) * CA_SW + 4 * tx + 4 + q];
            const f2 gg = f2_pack(g, g);
            const float *src = &sx[r * CA_SW + 4 * tx + 4 + q - R];
#pragma unroll
            for (int my = 0; my < K; ++my)
#pragma unroll
              for (int op = 0; op < NP; ++op)
                DM[my][op] = f2_fma(gg, f2_pack(src[my * CA_SW + 2 * op], 2 * op + 1 < K ? src[my * CA_SW + 2 * op + 1] : 0.0f),
                                    DM[my][op]);
          }
      }
      float dm[K * K];
#pragma unroll
      for (int o = 0; o < K * K; ++o) {
        const f2 v = DM[o / K][o % K >> 1];
        dm[o] = (o % K & 1) ? f2_hi(v) : f2_lo(v);
      }
      fold_taps(dm, sum[threadIdx.x >> 5], 0, K * K);
    }
    __syncthreads();  // this buffer is read before the tile after the next is staged into it
  }
  if (!p.part) return;
  __syncthreads();
  for (int o = threadIdx.x; o < K * K; o += CA_NT) p.part[(size_t)o * gridDim.x + blockIdx.x] = tap_total(sum, o);
}

using ConvAdjKernel = void (*)(ConvAdjParams);
// rows per thread: 4, or 1 where 32-row tiles would leave an SM fewer than four CTAs
int ca_rows(int w, int h, int batch) {
  return (int64_t)cdiv(w, CA_TW) * cdiv(h, 32) * batch >= 4 * num_sms() ? 4 : 1;
}
size_t ca_smem(int k, int py) { return (size_t)4 * (8 * py + k - 1) * CA_SW * sizeof(float); }
ConvAdjKernel ca_kernel(int k, int py) {
  if (k == 3) return py == 4 ? conv_adjoint_kernel<3, 4> : conv_adjoint_kernel<3, 1>;
  if (k == 5) return py == 4 ? conv_adjoint_kernel<5, 4> : conv_adjoint_kernel<5, 1>;
  return py == 4 ? conv_adjoint_kernel<7, 4> : conv_adjoint_kernel<7, 1>;
}

}  // namespace

bool conv_adjoint_size(int k) { return k == 3 || k == 5 || k == 7; }

int conv_adjoint_grid(int k, int w, int h, int batch) {
  const int py = ca_rows(w, h, batch);
  const int64_t tiles = (int64_t)cdiv(w, CA_TW) * cdiv(h, 8 * py) * batch;
  const int wave = num_sms() * resident_ctas((const void *)ca_kernel(k, py), CA_NT, ca_smem(k, py));
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, wave));
}

int run_conv_adjoint(int k, ConvAdjParams *p, int grid, cudaStream_t st) {
  const int py = ca_rows(p->w, p->h, p->batch);
  p->tiles_x = cdiv(p->w, CA_TW);
  p->tiles_y = cdiv(p->h, 8 * py);
  const int64_t tiles = (int64_t)p->tiles_x * p->tiles_y * p->batch;
  HGB_REQUIRE(tiles < 0x7fffffff, "conv adjoint: too many tiles");
  p->ntiles = (int)tiles;
  const size_t smem = ca_smem(k, py);
  const int rc = ensure_dynamic_smem((const void *)ca_kernel(k, py), smem);
  if (rc) return rc;
  ca_kernel(k, py)<<<grid, CA_NT, smem, st>>>(*p);
  return HGB_OK;
}

}  // namespace hgb
