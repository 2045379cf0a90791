// bilateral.cu -- hgb_bilateral: the bilateral filter of
// samples-public/3_Preprocessing/Bilateral_Filter/src/main.cpp:63-77:
//   c_r = 0.5 / sigma_r^2, centre = in(),
//   for every Domain(mask) cell: diff = in(dom) - centre,
//     s = exp(-c_r * diff^2) * mask(dom);  d += s;  p += s * in(dom)
//   out = p / d
// with a float range sigma and a float result.
//
// The filter is bound by arithmetic (one exponential and four FP32 lane
// operations per tap and pixel), not by HBM.  The weight is one base-2
// exponential with the spatial weight folded into the exponent; the staged
// tile is pre-scaled by q = sqrt(c_r * log2(e)), so that the exponent of a
// tap is a single fused multiply-add of the scaled difference d':
//   s = exp2(-(d'^2 + nl)),  nl = -log2(mask)
// (mask cells of 0 give nl = +inf, i.e. s = 0, which is the Domain's skip),
// and out = (sum s * v') / (sum s) / q.  The FP32 path evaluates the
// differences and the two sums for two pixels per packed f32x2 operation and
// the exponential with ex2.approx (32 per clock and SM on this part).
// For BF16 / F16 storage the fast path (flags bit 0) evaluates two taps'
// weights per instruction with packed half precision (h2exp2) and keeps every
// accumulation in FP32; its error against FP64 is stated by the tests.
#include <cmath>

#include "stage.cuh"
#include "stage_groups.cuh"

namespace hgb {
namespace {

constexpr int kBilMax = 13;

struct BilParams {
  const char *in;
  int64_t in_pitch, in_bstride;
  char *out;
  int64_t out_pitch, out_bstride;
  int w, h;
  int bmode;
  float cval;
  int vec_in, vec_out;
  float k2;                         // -c_r * log2(e)
  float q, inv_q;                   // sqrt(-k2) and 1 / q: the FP32 path's tile scale
  float lmask[kBilMax * kBilMax];   // log2(mask), -inf for zero cells
};

constexpr int BL_BX = 16, BL_BY = 16, BL_PX = 4;
constexpr int BL_TW = BL_BX * BL_PX, BL_TH = BL_BY;

template <typename T, int S>
struct BilShape {
  static constexpr int R = S / 2;
  static constexpr int VI = Vec16<T>::N;
  static constexpr int HL = round_up(R, VI);
  static constexpr int SW = HL + BL_TW + round_up(R, VI);
  static constexpr int SH = BL_TH + S - 1;
};

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}


// Half-precision weights (flags bit 0).
template <typename T, int S>
__global__ void __launch_bounds__(BL_BX *BL_BY) bilateral_half_kernel(const __grid_constant__ BilParams p) {
  using SH_ = BilShape<T, S>;
  constexpr int R = SH_::R, HL = SH_::HL, SW = SH_::SW, SH = SH_::SH;
  __shared__ __align__(16) float tile[SH * SW];
  const int b = blockIdx.z;
  const int i0 = blockIdx.x * BL_TW, j0 = blockIdx.y * BL_TH;
  stage_tile<T, SW, SH, BL_BX * BL_BY>(tile, p.in + (int64_t)b * p.in_bstride, p.in_pitch, i0 - HL, j0 - R, 0, p.w,
                                        0, p.h, p.bmode, p.cval, p.vec_in);
  __syncthreads();
  const int tx = threadIdx.x % BL_BX, ty = threadIdx.x / BL_BX;
  constexpr int OFF = (HL - R) % 4;
  constexpr int NV = cdiv(OFF + BL_PX + S - 1, 4);
  const int cb = HL - R - OFF + tx * BL_PX;
  float ctr[BL_PX], d[BL_PX], pp[BL_PX];
#pragma unroll
  for (int px = 0; px < BL_PX; ++px) {
    ctr[px] = tile[(ty + R) * SW + HL + tx * BL_PX + px];
    d[px] = 0.0f;
    pp[px] = 0.0f;
  }
#pragma unroll 1
  for (int my = 0; my < S; ++my) {
    float win[NV * 4];
    const float *row = &tile[(ty + my) * SW + cb];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float4 t = *reinterpret_cast<const float4 *>(row + 4 * v);
      win[4 * v] = t.x;
      win[4 * v + 1] = t.y;
      win[4 * v + 2] = t.z;
      win[4 * v + 3] = t.w;
    }
    // two outputs per half2: lanes (px, px+1)
    const __half2 k2h = __float2half2_rn(p.k2);
    __half2 c01 = __floats2half2_rn(ctr[0], ctr[1]), c23 = __floats2half2_rn(ctr[2], ctr[3]);
#pragma unroll
    for (int mx = 0; mx < S; ++mx) {
      const __half2 lm = __float2half2_rn(p.lmask[my * S + mx]);
      const __half2 v01 = __floats2half2_rn(win[OFF + mx], win[OFF + mx + 1]);
      const __half2 v23 = __floats2half2_rn(win[OFF + mx + 2], win[OFF + mx + 3]);
      const __half2 df01 = __hsub2(v01, c01), df23 = __hsub2(v23, c23);
      const float2 s01 = __half22float2(h2exp2(__hfma2(__hmul2(k2h, df01), df01, lm)));
      const float2 s23 = __half22float2(h2exp2(__hfma2(__hmul2(k2h, df23), df23, lm)));
      d[0] += s01.x;
      d[1] += s01.y;
      d[2] += s23.x;
      d[3] += s23.y;
      pp[0] = __fmaf_rn(s01.x, win[OFF + mx], pp[0]);
      pp[1] = __fmaf_rn(s01.y, win[OFF + mx + 1], pp[1]);
      pp[2] = __fmaf_rn(s23.x, win[OFF + mx + 2], pp[2]);
      pp[3] = __fmaf_rn(s23.y, win[OFF + mx + 3], pp[3]);
    }
  }
  float res[BL_PX];
#pragma unroll
  for (int px = 0; px < BL_PX; ++px) res[px] = __fdiv_rn(pp[px], d[px]);
  const int i = i0 + tx * BL_PX, j = j0 + ty;
  if (j < p.h && i < p.w)
    store_row<T, BL_PX>(reinterpret_cast<T *>(p.out + (int64_t)b * p.out_bstride + (int64_t)j * p.out_pitch) + i, res, i,
                        p.w, p.vec_out);
}


// FP32 weights.  A thread owns four (two on small images) columns of two rows, each pixel pair (rows y
// and y + 1 of a column) one f32x2 lane pair.  The tile is kept as pairs too, cell
// (r, x) = (v[r][x], v[r + 1][x]), so that a tap's operand for a pixel pair is one
// aligned register pair straight from a 16-byte load: of horizontal pairs every
// second one has to be assembled from two.  Row-major tap order per pixel.
// 13 x 13, f32 4096 x 4096: 469 us before, 425 us now, the FMA pipe and
// the exponential unit both 72 % busy.  The values are scaled as the pairs form, so
// that f32 tiles are staged by asynchronous copies (3 x 3, 4096 x 4096: 53 us, 61 us with
// values scaled on their way through registers).
constexpr int BP_NT = 256, BP_TW = 64;
// rows of a tile with CPT columns per thread
constexpr int bp_rows(int cpt) { return 2 * BP_NT / (BP_TW / cpt); }

template <typename T, int S, int CPT>
__global__ void __launch_bounds__(BP_NT) bilateral_kernel(const __grid_constant__ BilParams p) {
  constexpr int R = S / 2, HL = round_up(R, 4), SW = BP_TW + 2 * HL, TH = bp_rows(CPT), SH = TH + S - 1, S2 = (S + 1) / 2 * 2;
  constexpr int OFF = (HL - R) % 2, NC = (OFF + CPT + S - 1 + 1) / 2 * 2;  // cells of a row's window
  extern __shared__ __align__(16) float bil_smem[];
  f2 *cell = reinterpret_cast<f2 *>(bil_smem);             // (SH - 1) x SW pairs
  float *tile = bil_smem + 2 * (SH - 1) * SW;              // SH x SW values
  __shared__ __align__(16) f2 nl[S][S2];                   // -log2(mask) as pairs
  const int b = blockIdx.z, i0 = blockIdx.x * BP_TW, j0 = blockIdx.y * TH;
  for (int k = threadIdx.x; k < S * S2; k += BP_NT) {
    const int y = k / S2, x = k - y * S2;
    const float v = x < S ? -p.lmask[y * S + x] : 0.0f;
    nl[y][x] = f2_pack(v, v);
  }
  stage_groups<T, SW, SH, BP_NT>(tile, p.in + (int64_t)b * p.in_bstride, p.in_pitch, i0 - HL, j0 - R, 0, p.w, 0, p.h,
                                 p.bmode, p.cval, R);
  stage_wait();
  __syncthreads();
  const float q = p.q;  // the FP32 path works on values scaled by q
#pragma unroll 2
  for (int c = threadIdx.x; c < (SH - 1) * (SW / 2); c += BP_NT) {
    const float2 lo = reinterpret_cast<const float2 *>(tile)[c], hi = reinterpret_cast<const float2 *>(tile)[c + SW / 2];
    reinterpret_cast<float4 *>(cell)[c] =
        make_float4(__fmul_rn(lo.x, q), __fmul_rn(hi.x, q), __fmul_rn(lo.y, q), __fmul_rn(hi.y, q));
  }
  __syncthreads();
  const int tx = threadIdx.x % (BP_TW / CPT), ty = threadIdx.x / (BP_TW / CPT);
  f2 C[CPT], D[CPT], P[CPT];
#pragma unroll
  for (int k = 0; k < CPT; ++k) {
    C[k] = cell[(2 * ty + R) * SW + HL + CPT * tx + k];
    D[k] = P[k] = 0ull;
  }
  const f2 *row = cell + 2 * ty * SW + HL - R - OFF + CPT * tx;
#pragma unroll 1
  for (int my = 0; my < S; ++my, row += SW) {
    f2 W[NC];
#pragma unroll
    for (int v = 0; v < NC / 2; ++v) {
      const ulonglong2 t = reinterpret_cast<const ulonglong2 *>(row)[v];
      W[2 * v] = t.x;
      W[2 * v + 1] = t.y;
    }
#pragma unroll
    for (int m2 = 0; m2 < S2 / 2; ++m2) {
      const ulonglong2 n2 = reinterpret_cast<const ulonglong2 *>(&nl[my][0])[m2];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const int mx = 2 * m2 + l;
        if (mx >= S) continue;
        const f2 NL = l ? n2.y : n2.x;
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
          const f2 V = W[OFF + mx + k];
          const f2 df = f2_sub(V, C[k]);
          const f2 t = f2_fma(df, df, NL);  // d'^2 - lm
          const f2 sw = f2_pack(fast_exp2(-f2_lo(t)), fast_exp2(-f2_hi(t)));
          D[k] = f2_add(D[k], sw);
          P[k] = f2_fma(sw, V, P[k]);
        }
      }
    }
  }
  const int i = i0 + CPT * tx;
  if (i >= p.w) return;
#pragma unroll
  for (int l = 0; l < 2; ++l) {
    const int j = j0 + 2 * ty + l;
    if (j >= p.h) break;
    float res[CPT];
#pragma unroll
    for (int k = 0; k < CPT; ++k)
      res[k] = __fmul_rn(l ? __fdiv_rn(f2_hi(P[k]), f2_hi(D[k])) : __fdiv_rn(f2_lo(P[k]), f2_lo(D[k])), p.inv_q);
    T *dst = reinterpret_cast<T *>(p.out + (int64_t)b * p.out_bstride + (int64_t)j * p.out_pitch) + i;
    if constexpr (CPT == 4) {
      store_row<T, 4>(dst, res, i, p.w, p.vec_out);
    } else {
#pragma unroll
      for (int k = 0; k < CPT; ++k)
        if (i + k < p.w) dst[k] = Storage<T>::from_f(res[k]);
    }
  }
}

template <int S, int CPT>
constexpr size_t bil_smem_bytes() {
  constexpr int SW = BP_TW + 2 * round_up(S / 2, 4), SH = bp_rows(CPT) + S - 1;
  return sizeof(float) * (size_t)SW * (2 * (SH - 1) + SH);
}

template <typename T, int S, int CPT>
int launch_bil_pairs(const BilParams &p, int batch, cudaStream_t st) {
  constexpr size_t smem = bil_smem_bytes<S, CPT>();
  const int rc = ensure_dynamic_smem((const void *)bilateral_kernel<T, S, CPT>, smem);
  if (rc) return rc;
  const dim3 grid(cdiv(p.w, BP_TW), cdiv(p.h, bp_rows(CPT)), batch);
  cudaEvent_t ev = before_launch(st);
  bilateral_kernel<T, S, CPT><<<grid, BP_NT, smem, st>>>(p);
  return after_launch("bilateral_kernel", st, ev);
}

template <typename T, int S, bool FAST>
int launch_bil_s(const BilParams &p, int batch, cudaStream_t st) {
  if constexpr (FAST) {
    const dim3 grid(cdiv(p.w, BL_TW), cdiv(p.h, BL_TH), batch);
    cudaEvent_t ev = before_launch(st);
    bilateral_half_kernel<T, S><<<grid, BL_BX * BL_BY, 0, st>>>(p);
    return after_launch("bilateral_half_kernel", st, ev);
  } else {
    // four columns per thread (64 x 32 tiles), or two (64 x 16) where those would
    // not give every SM four CTAs: a small image's time is one thread's taps, and up
    // to a few tiles per SM the last wave counts.  f32, four / two, 9 x 9 and 13 x 13:
    // 320 x 256 7.9 / 5.5 and 12.9 / 8.3 us, 1024 x 1024 19.8 / 18.1 and 36.2 / 32.5, 4 of
    // 640 x 480 20.6 / 20.6 and 37.1 / 36.2; 1920 x 1080 31.6 / 32.6 and 59.6 / 59.6, 4096 x
    // 4096 215.6 / 229.1 and 426 / 434
    if ((int64_t)cdiv(p.w, BP_TW) * cdiv(p.h, bp_rows(4)) * batch >= 4 * num_sms())
      return launch_bil_pairs<T, S, 4>(p, batch, st);
    return launch_bil_pairs<T, S, 2>(p, batch, st);
  }
}

template <typename T, bool FAST>
int launch_bil(const BilParams &p, int size, int batch, cudaStream_t st) {
  switch (size) {
    case 3: return launch_bil_s<T, 3, FAST>(p, batch, st);
    case 5: return launch_bil_s<T, 5, FAST>(p, batch, st);
    case 7: return launch_bil_s<T, 7, FAST>(p, batch, st);
    case 9: return launch_bil_s<T, 9, FAST>(p, batch, st);
    case 11: return launch_bil_s<T, 11, FAST>(p, batch, st);
    case 13: return launch_bil_s<T, 13, FAST>(p, batch, st);
  }
  return set_error(HGB_ERR_UNSUPPORTED, "hgb_bilateral: size must be odd, 3..13");
}

}  // namespace
}  // namespace hgb

using namespace hgb;

extern "C" int hgb_bilateral(const hgb_view *in, const hgb_view *out, const float *smask, int size, float sigma_r,
                             int boundary, float const_val, int flags, void *stream) {
  int rc = check_view(in, "in");
  if (rc) return rc;
  rc = check_view(out, "out");
  if (rc) return rc;
  HGB_REQUIRE(in->dtype == out->dtype && is_float_storage(in->dtype), "hgb_bilateral: same float storage expected");
  HGB_REQUIRE(in->width == out->width && in->height == out->height && in->batch == out->batch,
              "hgb_bilateral: size mismatch");
  HGB_REQUIRE(smask, "hgb_bilateral: null mask");
  HGB_REQUIRE(size >= 3 && size <= kBilMax && (size & 1), "hgb_bilateral: size must be odd, 3..13");
  HGB_REQUIRE(sigma_r > 0.0f, "hgb_bilateral: sigma_r must be positive");
  HGB_REQUIRE(boundary >= 0 && boundary <= 4, "hgb_bilateral: bad boundary");
  const bool fast = (flags & 1) != 0;
  HGB_REQUIRE(!fast || in->dtype != HGB_F32, "hgb_bilateral: packed half weights need bf16 / f16 storage");
  BilParams p;
  memset(&p, 0, sizeof(p));
  p.in = (const char *)in->data;
  p.in_pitch = in->pitch;
  p.in_bstride = in->batch_stride;
  p.out = (char *)out->data;
  p.out_pitch = out->pitch;
  p.out_bstride = out->batch_stride;
  p.w = in->width;
  p.h = in->height;
  p.bmode = boundary;
  p.cval = const_val;
  p.vec_in = ((uintptr_t)in->data % 16 == 0) && in->pitch % 16 == 0 && (in->batch == 1 || in->batch_stride % 16 == 0);
  const int64_t four = 4 * dtype_size(out->dtype);  // a thread stores four pixels of a row
  p.vec_out = (uintptr_t)out->data % four == 0 && out->pitch % four == 0 &&
              (out->batch == 1 || out->batch_stride % four == 0);
  const double c_r = 0.5 / ((double)sigma_r * (double)sigma_r);
  p.k2 = (float)(-c_r * 1.4426950408889634);  // log2(e)
  p.q = (float)std::sqrt(c_r * 1.4426950408889634);
  p.inv_q = (float)(1.0 / std::sqrt(c_r * 1.4426950408889634));
  for (int i = 0; i < size * size; ++i)
    p.lmask[i] = smask[i] > 0.0f ? (float)std::log2((double)smask[i]) : -INFINITY;
  for (int i = 0; i < size * size; ++i)
    HGB_REQUIRE(smask[i] >= 0.0f, "hgb_bilateral: spatial weights must be non-negative");
  cudaStream_t st = (cudaStream_t)stream;
  switch (in->dtype) {
    case HGB_F32: return launch_bil<float, false>(p, size, in->batch, st);
    case HGB_BF16:
      return fast ? launch_bil<__nv_bfloat16, true>(p, size, in->batch, st)
                  : launch_bil<__nv_bfloat16, false>(p, size, in->batch, st);
    default:
      return fast ? launch_bil<__half, true>(p, size, in->batch, st) : launch_bil<__half, false>(p, size, in->batch, st);
  }
}
