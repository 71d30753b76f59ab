// composite.cuh -- one tile of the composite, by one CTA, shared by the
// single-mosaic kernel (k_composite.cu) and the batch kernel (k_batch.cu):
// main.rs:583-592 copies the adjusted tile into the output;
// color_adjustment.rs:53-87 adjust_pixel on each pixel.
//
// The brightness/contrast step of adjust_pixel is a function of one byte, so
// the CTA tabulates it for the tile's adjustment (256 entries) and each pixel
// looks its three channels up; the HSV part stays per pixel, as adjust_words
// for adjustments in adjustment_new's ranges (every adjustment the composite
// computes) and adjust_unit otherwise (mg_math.h: adjust_from_bc rearranged
// for channels in [0, 1] without changing a result).
// With tile widths a multiple of 4, four pixels of a tile row are 12 bytes,
// 4-byte aligned in the thumbnail and in the output, and move as three 32-bit
// words.
#pragma once
#include "mg_internal.h"
#include "roots.cuh"

namespace mg {

__device__ __forceinline__ uint32_t byte_of(uint32_t w, int i) { return (w >> (8 * i)) & 0xFFu; }

// v/255 - 0.5 for every byte v, once per CTA.
__device__ __forceinline__ void tile_unit_table(float* s_unit) {
  for (int v = threadIdx.x; v < 256; v += blockDim.x) s_unit[v] = __fsub_rn(u8_unit((uint32_t)v), 0.5f);
}
// brightness_contrast (color_adjustment.rs:91-96) of v/255 for every byte v, from
// tile_unit_table (written by the same threads).
__device__ __forceinline__ void tile_bc_table(float* s_bc, const float* s_unit, const Adjust& a) {
  for (int v = threadIdx.x; v < 256; v += blockDim.x)
    s_bc[v] = rclamp(__fadd_rn(rclamp(__fadd_rn(__fmul_rn(s_unit[v], a.contrast), 0.5f), 0.0f, 1.0f), a.brightness), 0.0f, 1.0f);
}

// The sector permutations of adjust_words in shared memory (threads 0..7).
__device__ __forceinline__ void sector_perm_table(uint32_t* s_perm) {
  if (threadIdx.x < 8) s_perm[threadIdx.x] = sector_perm(threadIdx.x);
}

// Per-pixel arithmetic of a tile: 0 a copy, 1 adjust_unit, 2 adjust_words.
enum TileMode { kTileCopy = 0, kTileUnit = 1, kTileWord = 2 };

// adjust_word (mg_math.h) of two pixels (component x, component y of the
// channels) for channels that brightness_contrast made, each output as one word (r | g << 8 | b << 16; byte 3 is not part of it).
// `perm` holds sector_perm(i) at index i (0..7; shared memory).  Rearranged
// without changing a result, in packed FP32x2 where both pixels do the same:
//  - the largest and smallest channel by maxima and minima; which of them the
//    hue is counted from by the two comparisons of rgb_to_hsv;
//  - a grey pixel (d = 0) gets saturation 0 and then, whatever its hue, the
//    value in every channel, so its hue need not be 0, only finite: the
//    divisors are kept from 0;
//  - the divisions sep / d and d / mx by Markstein's theorem (P. Markstein,
//    "Computation of elementary functions on the IBM RISC System/6000
//    processor", 1990): from the correctly rounded reciprocal y and q = a y, the
//    fused q + (a - q b) y is the correctly rounded quotient.  Channels differ by
//    0 or at least 2^-51 (both steps of brightness_contrast end in a sum whose
//    terms are multiples of that), so nothing underflows;
//  - the shifted hue lies in [-240, 480], so fmod_360 and the wrap below zero are
//    x + 360 below zero and then x - 360 (exact) from 360 up;
//  - pos / 60 by a multiply and an FMA correction at every pos: below 2^-120
//    both quotients are below 2^-126, and a quotient that small reaches the
//    output only through sector 0 and t = |h - 1| = 1;
//  - floor(h) and 2 floor(h / 2) read from h + 2^21, rounded toward zero;
//  - c <= v <= 1 and x <= c, so c + m and x + m with m = v - c round to 1 at
//    most and need no clamp: each output channel is one of c + m, x + m and m,
//    each converted once (times 255, plus 2^23 rounded toward zero), and the
//    sector's byte permutation picks them.
// What bounds it: instructions issued, 95 a pixel with the tile's share (78% of
// the issue slots; comparisons, selects and byte moves take the ALU pipe two
// cycles each, 60% of it).  Measured, GB300, before (pixel by pixel, calls of the
// IEEE division, 156 instructions) -> now: 24.6 M pixels in tiles of 32 x 32 0.123
// -> 0.079 ms, 64 mosaics (314 M pixels) 1.57 -> 1.16.  Not kept: operations with
// a constant in scalar form (87.7 M warp instructions for 83.1), 40 to 64 registers.
__device__ __forceinline__ uint2 adjust_words(const Adjust& a, float2 c0, float2 c1, float2 c2, const uint32_t* perm) {
  auto pair = [](float v) { return make_float2(v, v); };
  auto neg = [](float2 v) { return make_float2(-v.x, -v.y); };
  // A product that is then added to is scalar: of a packed product and a packed
  // sum the assembler makes one FMA, which rounds once.
  auto mul = [](float2 u, float2 v) { return make_float2(__fmul_rn(u.x, v.x), __fmul_rn(u.y, v.y)); };
  float2 mx, mn, p, q, coeff;
  auto order = [](float r, float g, float b, float& mx, float& mn, float& p, float& q, float& coeff) {
    const bool rg = r > g;
    const float m = fmaxf(r, g);
    const bool blue = b > m;
    mx = fmaxf(m, b);
    mn = fminf(fminf(r, g), b);
    p = blue ? r : rg ? g : b;
    q = blue ? g : rg ? b : r;
    coeff = blue ? 4.0f : rg ? 0.0f : 2.0f;
  };
  order(c0.x, c1.x, c2.x, mx.x, mn.x, p.x, q.x, coeff.x);
  order(c0.y, c1.y, c2.y, mx.y, mn.y, p.y, q.y, coeff.y);
  const float2 sep = __fadd2_rn(p, neg(q)), d = __fadd2_rn(mx, neg(mn));
  // (the divisors are at most 1)
  const float2 yd = rcp2_in_range(make_float2(fmaxf(d.x, 1e-20f), fmaxf(d.y, 1e-20f)));
  const float2 ym = rcp2_in_range(make_float2(fmaxf(mx.x, 1e-20f), fmaxf(mx.y, 1e-20f)));
  float2 hd = __fmul2_rn(sep, yd), s = __fmul2_rn(d, ym);
  hd = __ffma2_rn(__ffma2_rn(neg(hd), d, sep), yd, hd);
  s = __ffma2_rn(__ffma2_rn(neg(s), mx, d), ym, s);
  float2 pos = __fadd2_rn(mul(__fadd2_rn(hd, coeff), pair(60.0f)), pair(a.hue_shift));
  auto wrap = [](float x) {
    if (x < 0.0f) x = __fadd_rn(x, 360.0f);
    if (x >= 360.0f) x = __fadd_rn(x, -360.0f);
    return x;
  };
  pos.x = wrap(pos.x);
  pos.y = wrap(pos.y);
  const float2 h0 = __fmul2_rn(pos, pair(1.0f / 60.0f));
  const float2 h = __ffma2_rn(__ffma2_rn(neg(h0), pair(60.0f), pos), pair(1.0f / 60.0f), h0);
  const float2 hz = __fadd2_rz(h, pair(2097152.0f));  // 2^21 + floor(4 h) / 4
  const uint32_t qx = __float_as_uint(hz.x), qy = __float_as_uint(hz.y);
  const float2 even = make_float2(__uint_as_float(qx & ~7u), __uint_as_float(qy & ~7u));
  const float2 t = __fadd2_rn(__fadd2_rn(h, neg(__fadd2_rn(even, pair(-2097152.0f)))), pair(-1.0f));
  const float2 f = make_float2(__fsub_rn(1.0f, fabsf(t.x)), __fsub_rn(1.0f, fabsf(t.y)));
  float2 sat = __fmul2_rn(s, pair(a.saturation));
  sat = make_float2(fminf(sat.x, 1.0f), fminf(sat.y, 1.0f));
  const float2 c = mul(mx, sat);
  const float2 x = mul(c, f);
  const float2 m = __fadd2_rn(mx, neg(c));
  const float2 top = pair(8388608.0f), full = pair(255.0f);
  const float2 wc = __fadd2_rz(mul(__fadd2_rn(c, m), full), top);
  const float2 wx = __fadd2_rz(mul(__fadd2_rn(x, m), full), top);
  const float2 wz = __fadd2_rz(mul(m, full), top);
  auto pick = [&](uint32_t hq, float wc, float wx, float wz) {
    const uint32_t sel = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(perm) + (hq & 0x1Cu));
    return __byte_perm(__byte_perm(__float_as_uint(wc), __float_as_uint(wx), 0x40u), __float_as_uint(wz), sel);
  };
  return make_uint2(pick(qx, wc.x, wx.x, wz.x), pick(qy, wc.y, wx.y, wz.y));
}

// One pixel (channels b0, b1, b2) as r | g << 8 | b << 16 (byte 3 not used).
template <int kMode>
__device__ __forceinline__ uint32_t tile_pixel(uint32_t b0, uint32_t b1, uint32_t b2, const Adjust& a,
                                               const float* s_bc, const uint32_t* s_perm) {
  if (kMode == kTileCopy) return b0 | b1 << 8 | b2 << 16;
  if (kMode == kTileWord) {
    const float c0 = s_bc[b0], c1 = s_bc[b1], c2 = s_bc[b2];
    return adjust_words(a, make_float2(c0, c0), make_float2(c1, c1), make_float2(c2, c2), s_perm).x;
  }
  uint8_t o0, o1, o2;
  adjust_unit(a, s_bc[b0], s_bc[b1], s_bc[b2], o0, o1, o2);
  return (uint32_t)o0 | (uint32_t)o1 << 8 | (uint32_t)o2 << 16;
}

// A thread's place in a tile of `per_row` items a row: its first item and the
// step to its next one; the same for every tile, so the divisions are made once.
// (A tile may hold more than 2^31 bytes: its bytes are walked by pointer.)
struct TileLane {
  int per_row, row, col, drow, dcol;
};
__device__ __forceinline__ TileLane tile_lane(int tw) {
  TileLane t;
  t.per_row = (tw & 3) == 0 ? tw >> 2 : (tw + 1) >> 1;  // groups of four pixels, or pairs
  t.row = (int)threadIdx.x / t.per_row;
  t.col = (int)threadIdx.x - t.row * t.per_row;
  t.drow = (int)blockDim.x / t.per_row;
  t.dcol = (int)blockDim.x - t.drow * t.per_row;
  return t;
}

// Two pixels.
template <int kMode>
__device__ __forceinline__ uint2 tile_pixels2(uint32_t l0, uint32_t l1, uint32_t l2, uint32_t r0, uint32_t r1,
                                              uint32_t r2, const Adjust& a, const float* s_bc, const uint32_t* s_perm) {
  if (kMode == kTileWord)
    return adjust_words(a, make_float2(s_bc[l0], s_bc[r0]), make_float2(s_bc[l1], s_bc[r1]),
                        make_float2(s_bc[l2], s_bc[r2]), s_perm);
  return make_uint2(tile_pixel<kMode>(l0, l1, l2, a, s_bc, s_perm), tile_pixel<kMode>(r0, r1, r2, a, s_bc, s_perm));
}

template <int kMode>
__device__ __forceinline__ void tile_pixels(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int tw,
                                            int th, size_t pitch, const TileLane& lane, const Adjust& a,
                                            const float* s_bc, const uint32_t* s_perm) {
  int row = lane.row, col = lane.col;
  auto step = [&] {
    row += lane.drow;
    col += lane.dcol;
    if (col >= lane.per_row) {
      col -= lane.per_row;
      ++row;
    }
  };
  if ((tw & 3) == 0) {
    // a tile's groups are contiguous: a thread's next one is blockDim.x of them on
    for (const uint8_t* group = src + 12 * threadIdx.x; row < th; step(), group += 12 * blockDim.x) {
      uint32_t* d = reinterpret_cast<uint32_t*>(dst + row * pitch + 12 * col);
      const uint32_t* s = reinterpret_cast<const uint32_t*>(group);
      const uint32_t w0 = __ldg(s), w1 = __ldg(s + 1), w2 = __ldg(s + 2);
      if (kMode == kTileCopy) {
        d[0] = w0;
        d[1] = w1;
        d[2] = w2;
        continue;
      }
      // pixel k: bytes 3k .. 3k + 2 of w0:w1:w2; results packed back as bytes 0-2 of each
      const uint2 p01 = tile_pixels2<kMode>(byte_of(w0, 0), byte_of(w0, 1), byte_of(w0, 2), byte_of(w0, 3),
                                            byte_of(w1, 0), byte_of(w1, 1), a, s_bc, s_perm);
      const uint2 p23 = tile_pixels2<kMode>(byte_of(w1, 2), byte_of(w1, 3), byte_of(w2, 0), byte_of(w2, 1),
                                            byte_of(w2, 2), byte_of(w2, 3), a, s_bc, s_perm);
      const uint32_t p0 = p01.x, p1 = p01.y, p2 = p23.x, p3 = p23.y;
      d[0] = __byte_perm(p0, p1, 0x4210);
      d[1] = __byte_perm(p1, p2, 0x5421);
      d[2] = __byte_perm(p2, p3, 0x6542);
    }
    return;
  }
  if (kMode == kTileCopy) {
    for (int q = threadIdx.x; q < tw * th; q += blockDim.x) {
      const int row = q / tw, x = q - row * tw;
      uint8_t* d = dst + row * pitch + (size_t)x * 3;
      const uint8_t* s = src + (size_t)q * 3;
      d[0] = s[0];
      d[1] = s[1];
      d[2] = s[2];
    }
    return;
  }
  // pairs; a row of odd width ends in a pixel of its own, three bytes short of a pair
  const int lost = 3 * (tw & 1);
  const uint8_t* s = src + 6 * threadIdx.x - lost * row;
  for (int from = row; row < th; from = row, step(), s += 6 * (int)blockDim.x - lost * (row - from)) {
    const int x = 2 * col;
    uint8_t* d = dst + row * pitch + 3 * x;
    const bool two = x + 1 < tw;
    const uint32_t l0 = s[0], l1 = s[1], l2 = s[2];
    const uint2 p = tile_pixels2<kMode>(l0, l1, l2, two ? s[3] : l0, two ? s[4] : l1, two ? s[5] : l2, a, s_bc, s_perm);
    d[0] = (uint8_t)p.x;
    d[1] = (uint8_t)(p.x >> 8);
    d[2] = (uint8_t)(p.x >> 16);
    if (two) {
      d[3] = (uint8_t)p.y;
      d[4] = (uint8_t)(p.y >> 8);
      d[5] = (uint8_t)(p.y >> 16);
    }
  }
}

// The tile of thumbnail `src` (tw x th RGB8; nullptr: an empty cell, black)
// into `dst` (row pitch `pitch` bytes), adjusted when `adjust` (s_bc from
// tile_bc_table for `a`, s_perm from sector_perm_table).  `adjust` and `a` are
// uniform over the CTA.
__device__ __forceinline__ void composite_tile(const uint8_t* __restrict__ src, uint8_t* __restrict__ dst, int tw,
                                               int th, size_t pitch, const TileLane& lane, bool adjust,
                                               const Adjust& a, const float* s_bc, const uint32_t* s_perm) {
  if (!src) {
    const int per_row = (tw & 3) == 0 ? 3 * tw / 4 : 3 * tw;  // 32-bit words, else bytes
    for (int q = threadIdx.x; q < per_row * th; q += blockDim.x) {
      const int row = q / per_row, k = q - row * per_row;
      if ((tw & 3) == 0) reinterpret_cast<uint32_t*>(dst + row * pitch)[k] = 0u;
      else dst[row * pitch + k] = 0;
    }
    return;
  }
  if (!adjust) tile_pixels<kTileCopy>(src, dst, tw, th, pitch, lane, a, s_bc, s_perm);
  else if (adjust_word_applies(a)) tile_pixels<kTileWord>(src, dst, tw, th, pitch, lane, a, s_bc, s_perm);
  else tile_pixels<kTileUnit>(src, dst, tw, th, pitch, lane, a, s_bc, s_perm);
}

// Threads per CTA for tiles of tw x th: the fewest passes over the tile's
// pixel groups at up to 256 threads, in whole warps.
inline int tile_threads(int tw, int th) {
  const int groups = (tw & 3) == 0 ? (tw >> 2) * th : tw * th;
  const int passes = (groups + 255) / 256;
  const int per = (groups + passes - 1) / passes;
  return ((per + 31) / 32) * 32;
}

}  // namespace mg
