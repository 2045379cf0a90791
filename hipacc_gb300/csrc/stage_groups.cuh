// stage_groups.cuh -- staging of a halo tile into shared memory as FP32 for any
// row alignment and any boundary, four columns at a time.
//
// Rows [Y0, Y0 + SH) x columns [X0, X0 + SW) of an accessor window are copied
// into `tile` (row pitch SW floats).  In a tile inside the window every group of
// four columns is loaded whole: one vector load where the rows' alignment allows
// it, else the aligned words around it, shifted into place (u8 and 16-bit rows of
// odd length start at any byte).  A border tile evaluates the boundary remap
// (lib/AST/BorderHandling.cpp:41-120) once per row and column and loads every
// group element by element through those tables.
//
// Why: the per-element staging this replaces spent a remap (two compares and
// often a branch per axis) and one byte load on every staged cell, ~21 cells
// per thread and tile, also in tiles far from any border.
#pragma once

#include "hgb_internal.cuh"

namespace hgb {

// four bytes of a word as floats: a byte in the mantissa of 2^23 is 2^23 + b
__device__ __forceinline__ float4 bytes_to_f4(uint32_t w) {
  const f2 k23 = f2_pack(8388608.0f, 8388608.0f);
  const f2 lo = f2_sub(f2_pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440)),
                               __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7441))), k23);
  const f2 hi = f2_sub(f2_pack(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7442)),
                               __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7443))), k23);
  return make_float4(f2_lo(lo), f2_hi(lo), f2_lo(hi), f2_hi(hi));
}

// Four consecutive elements at `p`, which have at least four more elements of
// the same row on either side unless `p` is aligned for a vector load.
template <typename T> struct Load4;
template <> struct Load4<uint8_t> {
  static constexpr int kAlign = 4;
  static __device__ __forceinline__ float4 staged(const uint8_t *p) {  // from shared memory
    return bytes_to_f4(*reinterpret_cast<const uint32_t *>(p));
  }
  static __device__ __forceinline__ float4 whole(const uint8_t *p) {
    return bytes_to_f4(__ldg(reinterpret_cast<const uint32_t *>(p)));
  }
  static __device__ __forceinline__ float4 shifted(const uint8_t *p) {
    const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(p) & 3u);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(p - s);
    return bytes_to_f4(__funnelshift_r(__ldg(w), __ldg(w + 1), 8 * s));
  }
};
template <> struct Load4<float> {
  static constexpr int kAlign = 16;
  static __device__ __forceinline__ float4 whole(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
  // two aligned vectors and nine selects: four 4-byte loads 16 bytes apart across
  // the lanes take twice the cycles of the load unit
  static __device__ __forceinline__ float4 shifted(const float *p) {
    const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(p) & 15u);
    const float4 *q = reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(p) - s);
    const float4 a = __ldg(q), b = __ldg(q + 1);
    const bool two = s & 8u, one = s & 4u;
    const float t0 = two ? a.z : a.x, t1 = two ? a.w : a.y, t2 = two ? b.x : a.z, t3 = two ? b.y : a.w,
                t4 = two ? b.z : b.x;
    return make_float4(one ? t1 : t0, one ? t2 : t1, one ? t3 : t2, one ? t4 : t3);
  }
};
template <typename T> struct Load4Half {
  static constexpr int kAlign = 8;
  static __device__ __forceinline__ float4 widen(uint32_t a, uint32_t b) {
    T h[4];
    const uint2 v = make_uint2(a, b);
    __builtin_memcpy(h, &v, 8);
    return make_float4(Storage<T>::to_f(h[0]), Storage<T>::to_f(h[1]), Storage<T>::to_f(h[2]), Storage<T>::to_f(h[3]));
  }
  static __device__ __forceinline__ float4 staged(const T *p) {  // from shared memory
    const uint2 v = *reinterpret_cast<const uint2 *>(p);
    return widen(v.x, v.y);
  }
  static __device__ __forceinline__ float4 whole(const T *p) {
    const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
    return widen(v.x, v.y);
  }
  static __device__ __forceinline__ float4 shifted(const T *p) {
    const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(p) & 2u);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(p) - s);
    const uint32_t a = __ldg(w), b = __ldg(w + 1), c = s ? __ldg(w + 2) : 0u;
    return widen(__funnelshift_r(a, b, 8 * s), __funnelshift_r(b, c, 8 * s));
  }
};
template <> struct Load4<__nv_bfloat16> : Load4Half<__nv_bfloat16> {};
template <> struct Load4<__half> : Load4Half<__half> {};

// The group of columns [x, x + 4) of row y of the window.  Cells farther than
// `reach` outside the window serve no output and read the constant (a tile that
// overhangs a small image would spend most of its staging on them).
template <typename TI>
__device__ __forceinline__ float4 load_group(const char *in, int64_t pitch, int x, int y, int ax_lo, int ax_hi,
                                             int ay_lo, int ay_hi, int bmode, float cval, int reach) {
  if (y >= ay_lo && y < ay_hi && x >= ax_lo && x + 4 <= ax_hi) {
    const TI *p = reinterpret_cast<const TI *>(in + (int64_t)y * pitch) + x;
    if ((reinterpret_cast<uintptr_t>(p) & (Load4<TI>::kAlign - 1)) == 0) return Load4<TI>::whole(p);
    if (x >= ax_lo + 4 && x + 8 <= ax_hi) return Load4<TI>::shifted(p);
  }
  if (x + 3 < ax_lo - reach || x >= ax_hi + reach || y < ay_lo - reach || y >= ay_hi + reach)
    return make_float4(cval, cval, cval, cval);
  const int ry = remap(bmode, y, ay_lo, ay_hi);
  const TI *row = reinterpret_cast<const TI *>(in + (int64_t)(ry == (int)0x80000000 ? ay_lo : ry) * pitch);
  float f[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int rx = x + q >= ax_hi + reach ? (int)0x80000000 : remap(bmode, x + q, ax_lo, ax_hi);
    f[q] = (rx == (int)0x80000000 || ry == (int)0x80000000) ? cval : Storage<TI>::load(row + rx);
  }
  return make_float4(f[0], f[1], f[2], f[3]);
}

// Every group of the tile to put(c, values), c = row * (SW / 4) + group, NT
// threads.  A tile that lies inside the window with four columns to spare takes
// its addresses by adding to one pointer and tests nothing per group: the tests,
// the division and the 64-bit products of the general loop are about 30
// instructions a group, several per pixel.
template <typename TI, int SW, int SH, int NT, typename F>
__device__ __forceinline__ void stage_groups_each(const char *in, int64_t pitch, int X0, int Y0, int ax_lo, int ax_hi,
                                                  int ay_lo, int ay_hi, int bmode, float cval, int reach, F put) {
  static_assert(SW % 4 == 0, "whole groups");
  constexpr int G = SW / 4, ES = (int)sizeof(TI);
  int r = threadIdx.x / G, k = threadIdx.x - r * G;
  if (X0 - 4 >= ax_lo && X0 + SW + 4 <= ax_hi && Y0 >= ay_lo && Y0 + SH <= ay_hi) {
    const char *p = in + (int64_t)(Y0 + r) * pitch + (int64_t)(X0 + 4 * k) * ES;
    const int64_t step = (int64_t)(NT / G) * pitch + (NT % G) * 4 * ES, wrap = pitch - G * 4 * ES;
    const uint64_t bits = reinterpret_cast<uint64_t>(in) | (uint64_t)pitch | (uint64_t)((int64_t)X0 * ES);
    auto run = [&](auto load) {
#pragma unroll 4
      for (int c = threadIdx.x; c < SH * G; c += NT) {
        put(c, load(reinterpret_cast<const TI *>(p)));
        k += NT % G;
        p += step;
        if (k >= G) {
          k -= G;
          p += wrap;
        }
      }
    };
    if ((bits & (uint64_t)(Load4<TI>::kAlign - 1)) == 0)
      run([](const TI *q) { return Load4<TI>::whole(q); });
    else
      run([](const TI *q) { return Load4<TI>::shifted(q); });
    return;
  }
  // Border tiles: the remapped columns and rows are tabled once, then every group
  // loads four elements through the tables.  (Letting the groups inside the window
  // take their vector loads and the others a remapping branch made each step of a
  // warp two dependent loads: 4 images of 1241 x 872, 5 x 5 bf16, 13 -> 17 us.)
  // Cells farther than `reach` outside the window serve no output.
  __shared__ __align__(16) int cmap[SW];
  __shared__ int rmap[SH];
  __syncthreads();  // an earlier call's reads of the tables are done
  for (int i = threadIdx.x; i < SW + SH; i += NT) {
    const bool col = i < SW;
    const int v = col ? X0 + i : Y0 + i - SW, lo = col ? ax_lo : ay_lo, hi = col ? ax_hi : ay_hi;
    int m = v < lo - reach || v >= hi + reach ? (int)0x80000000 : remap(bmode, v, lo, hi);
    m = m == (int)0x80000000 ? -1 : m;
    if (col)
      cmap[i] = m;
    else
      rmap[i - SW] = m;
  }
  __syncthreads();
#pragma unroll 4
  for (int c = threadIdx.x; c < SH * G; c += NT) {
    const int4 x = reinterpret_cast<const int4 *>(cmap)[k];
    const int y = rmap[r];
    const TI *row = reinterpret_cast<const TI *>(in + (int64_t)max(y, 0) * pitch);
    float4 v;
    v.x = (x.x | y) < 0 ? cval : Storage<TI>::load(row + x.x);
    v.y = (x.y | y) < 0 ? cval : Storage<TI>::load(row + x.y);
    v.z = (x.z | y) < 0 ? cval : Storage<TI>::load(row + x.z);
    v.w = (x.w | y) < 0 ? cval : Storage<TI>::load(row + x.w);
    put(c, v);
    k += NT % G;
    r += NT / G;
    if (k >= G) {
      k -= G;
      ++r;
    }
  }
}

__device__ __forceinline__ void copy_async16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async4(float *dst, const float *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// The tile into shared memory; complete for every thread after stage_wait() and
// a CTA barrier.  f32 tiles inside the window are copied without passing through
// registers: 16 bytes at a time where the rows allow it, else a row per warp, 4
// bytes per lane (coalesced, two instructions a copy).
template <typename TI, int SW, int SH, int NT>
__device__ __forceinline__ void stage_groups(float *tile, const char *in, int64_t pitch, int X0, int Y0, int ax_lo,
                                             int ax_hi, int ay_lo, int ay_hi, int bmode, float cval, int reach) {
  if constexpr (sizeof(TI) == 4) {
    constexpr int G = SW / 4;
    if (X0 >= ax_lo && X0 + SW <= ax_hi && Y0 >= ay_lo && Y0 + SH <= ay_hi) {
      const uint64_t bits = reinterpret_cast<uint64_t>(in) | (uint64_t)pitch | (uint64_t)((int64_t)X0 * 4);
      if ((bits & 15u) == 0) {
        int k = threadIdx.x % G;
        const char *p = in + (int64_t)(Y0 + (int)threadIdx.x / G) * pitch + (int64_t)(X0 + 4 * k) * 4;
        const int64_t step = (int64_t)(NT / G) * pitch + (NT % G) * 16, wrap = pitch - G * 16;
#pragma unroll 4
        for (int c = threadIdx.x; c < SH * G; c += NT) {
          copy_async16(tile + 4 * c, reinterpret_cast<const float *>(p));
          k += NT % G;
          p += step;
          if (k >= G) {
            k -= G;
            p += wrap;
          }
        }
      } else {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const char *p = in + (int64_t)(Y0 + warp) * pitch + (int64_t)(X0 + lane) * 4;
        float *q = tile + warp * SW + lane;
#pragma unroll 2
        for (int r = warp; r < SH; r += NT / 32) {
          const float *row = reinterpret_cast<const float *>(p);
#pragma unroll
          for (int i = 0; i < SW; i += 32)
            if (i + 32 <= SW || i + lane < SW) copy_async4(q + i, row + i);
          p += (int64_t)(NT / 32) * pitch;
          q += NT / 32 * SW;
        }
      }
      return;
    }
  }
  stage_groups_each<TI, SW, SH, NT>(in, pitch, X0, Y0, ax_lo, ax_hi, ay_lo, ay_hi, bmode, cval, reach,
                                    [tile](int c, float4 v) { reinterpret_cast<float4 *>(tile)[c] = v; });
}
__device__ __forceinline__ void stage_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// tiles staged ahead: commit after staging one, then wait for all but the newest
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void stage_wait_but_newest() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The same for a byte tile kept as words; bytes outside the image read 0.
template <int G, int SH, int NT>
__device__ __forceinline__ void stage_words(uint32_t *tile, const uint8_t *img, int64_t pitch, int X0, int Y0, int w,
                                            int h) {
  int r = threadIdx.x / G, k = threadIdx.x - r * G;
  if (X0 - 4 >= 0 && X0 + 4 * G + 4 <= w && Y0 >= 0 && Y0 + SH <= h) {
    const uint8_t *p = img + (int64_t)(Y0 + r) * pitch + X0 + 4 * k;
    const int64_t step = (int64_t)(NT / G) * pitch + (NT % G) * 4, wrap = pitch - G * 4;
    const uint64_t bits = reinterpret_cast<uint64_t>(img) | (uint64_t)pitch | (uint64_t)(int64_t)X0;
    auto run = [&](auto load) {
#pragma unroll 4
      for (int c = threadIdx.x; c < SH * G; c += NT) {
        tile[c] = load(p);
        k += NT % G;
        p += step;
        if (k >= G) {
          k -= G;
          p += wrap;
        }
      }
    };
    if ((bits & 3u) == 0)
      run([](const uint8_t *q) { return __ldg(reinterpret_cast<const uint32_t *>(q)); });
    else
      run([](const uint8_t *q) {
        const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(q) & 3u);
        const uint32_t *u = reinterpret_cast<const uint32_t *>(q - s);
        return __funnelshift_r(__ldg(u), __ldg(u + 1), 8 * s);
      });
    return;
  }
  // Border tiles: first the words with four columns to spare and those outside, with
  // the loads of eight words in flight, then the few words at the left and right
  // edges byte by byte.  (One loop with both kinds kept two words in flight: 250 x 250
  // Sobel 6.6 us.)
#pragma unroll 8
  for (int c = threadIdx.x; c < SH * G; c += NT) {
    const int x = X0 + 4 * k, y = Y0 + r;
    const bool row = y >= 0 && y < h, spare = row && x >= 4 && x + 8 <= w;
    uint32_t v = 0;
    if (spare) {
      const uint8_t *q = img + (int64_t)y * pitch + x;
      const unsigned s = (unsigned)(reinterpret_cast<uintptr_t>(q) & 3u);
      const uint32_t *u = reinterpret_cast<const uint32_t *>(q - s);
      v = __funnelshift_r(__ldg(u), __ldg(u + 1), 8 * s);
    }
    if (spare || !row || x + 3 < 0 || x >= w) tile[c] = v;
    k += NT % G;
    r += NT / G;
    if (k >= G) {
      k -= G;
      ++r;
    }
  }
  // words of each row that hold an edge: the one at column 0 and the last two, from x
  // > w - 8 on (X0 is a multiple of 4)
  const int kl = -X0 / 4, kr = (max(w - 7, 0) + 3) / 4 - X0 / 4;
#pragma unroll 2
  for (int c = threadIdx.x; c < 3 * SH; c += NT) {
    const int e = c / SH, rr = c - e * SH, kk = e == 0 ? kl : kr + e - 1;
    const int x = X0 + 4 * kk, y = Y0 + rr;
    if (kk < 0 || kk >= G || y < 0 || y >= h || x >= w || (x >= 4 && x + 8 <= w)) continue;
    const uint8_t *q = img + (int64_t)y * pitch + x;
    uint32_t v = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (x + i < w) v |= (uint32_t)__ldg(q + i) << (8 * i);
    tile[rr * G + kk] = v;
  }
}

}  // namespace hgb
