// tap_fold.cuh -- tap gradients of a tile, from a warp's lanes into running sums.
//
// Every lane of a warp holds an FP32 partial sum of each of N taps.  Five exchanges
// add them up: in each, a lane keeps half of its taps and gives the other half to its
// partner, so a tap takes about one shuffle instead of five (51 for the 49 taps of a
// 7 x 7 mask).  The last two additions and the sum over tiles keep what FP32 rounds
// away beside them, so the error of a tap gradient does not grow with the image: a
// product is rounded in its thread's chain of one tile and in three additions after
// it.  One FP32 chain through all tiles of a CTA erred 4.9 times as much on 6001 x 6003
// (7 x 7, RMS against FP64), 3.5 times on 64 images of 1024 x 1024 (1 x 9).
//
// Mask gradient alone, one chain against a fold per tile: 7 x 7 on 6001 x 6003 201.5 /
// 196 us (202 us with the sums in FP64 in place of pairs), 3 x 3 on 2 x 2049 x 2051 32.5 /
// 34.1 us, 1 x 9 on 4 x 1920 x 1080 25.0 / 27.1 us, 1 x 15 on 4096 x 4096 76.6 / 50.2 us
// (the accumulators' registers are free between tiles).  Folding a tile's sums while
// the next one lands instead of at its end: 216, 34.1, 27.1 and 79 us.
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

struct TapSum {  // s + c
  float s, c;
};

// the exact sum of two FP32 values (Knuth's two-sum)
__device__ __forceinline__ TapSum tap_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ TapSum tap_add(TapSum a, TapSum b) {
  const TapSum t = tap_two_sum(a.s, b.s);
  return {t.s, __fadd_rn(t.c, __fadd_rn(a.c, b.c))};
}

// one exchange: own value and the partner's
template <int D>
__device__ __forceinline__ float tap_exchange(float keep, float give) {
  return keep + __shfl_xor_sync(0xffffffffu, give, D);
}
template <int D>
__device__ __forceinline__ TapSum tap_exchange(TapSum keep, TapSum give) {
  return tap_add(keep, {__shfl_xor_sync(0xffffffffu, give.s, D), __shfl_xor_sync(0xffffffffu, give.c, D)});
}

// v[i], i < count: this lane's share of tap base + i.  Adds the warp's sum of every
// tap to sum[tap]; each tap has the same lane on every call.  All lanes take part.
template <int D = 16, int N, typename T>
__device__ __forceinline__ void fold_taps(const T (&v)[N], TapSum *sum, int base, int count) {
  if constexpr (D == 0) {
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (i < count) sum[base + i] = tap_add(sum[base + i], v[i]);
  } else {
    constexpr int H = (N + 1) / 2;
    const bool up = threadIdx.x & D;
    T w[H];
    TapSum pair[H];
#pragma unroll
    for (int i = 0; i < H; ++i) {
      const T hi = H + i < N ? v[H + i < N ? H + i : 0] : T{};
      const T give = up ? v[i] : hi, keep = up ? hi : v[i];
      if constexpr (D == 2)
        pair[i] = tap_two_sum(keep, __shfl_xor_sync(0xffffffffu, give, D));
      else
        w[i] = tap_exchange<D>(keep, give);
    }
    base += up ? H : 0;
    count = up ? count - H : min(count, H);
    if constexpr (D == 2)
      fold_taps<1>(pair, sum, base, count);
    else
      fold_taps<D / 2>(w, sum, base, count);
  }
}

// sum of a tap over the CTA's warps (FP64 only at the end: its additions take long)
template <int W, int N>
__device__ __forceinline__ double tap_total(const TapSum (&sum)[W][N], int tap) {
  TapSum v = sum[0][tap];
#pragma unroll
  for (int w = 1; w < W; ++w) v = tap_add(v, sum[w][tap]);
  return (double)v.s + (double)v.c;
}

}  // namespace hgb
