// cc_resample.cuh - the colour converter's resample kernel: every conversion
// whose content is not the source rectangle pixel for pixel.
//
// A thread takes four pixels across and one row (two rows into 4:2:0 formats,
// whose rows share chroma). What bounded the kernel was instruction issue
// (ncu: 76-78 % of the slots when a thread took one pixel, 306 instructions per
// pixel bilinear and 700 for a 3x3 area footprint, a third of them integer),
// and with fewer instructions it is the latency of the source's loads, so that
//   - pixels run in pairs, two lanes per instruction, and a sample's
//     conversion to float is part of its weighting: with B = 2^23 + c the
//     float whose low bits are the code c, fma(B, w, -2^23 w) is c w rounded
//     once, as the definition's product is;
//   - taps of weight zero are not skipped but added: c x 0 is +0 and changes no
//     sum; so all taps of a pair (area: of four source columns) load at once;
//   - the alpha of formats that store none, 255 at every tap, is not carried
//     along: its weighted mean is 255 within 0.2 and stores as 255 (up to
//     kConstAlphaTaps taps; larger footprints carry it, resample_alpha);
//   - area footprints of whole pixels (kScale) are sums of integers, formed
//     four bytes at a time (sum_whole).
// Measured as a replayed graph of one call each, before -> after: 1920x1080 NV12
// into 1280x720 RGBA8, bilinear, 10.5 -> 6.6 us; into RGB8, area (1.5 columns),
// 14.2 -> 8.5; 3840x2160 NV12 into 1280x720 RGB8, area of 3x3, 22.5 -> 6.5;
// 1280x720 RGBA8 into 1920x1080, bilinear, 18.1 -> 10.6.
#pragma once

#include <type_traits>

#include "cc_kernels.cuh"

namespace cc_b200 {

constexpr int kResampleThreadsY = 4;
constexpr float kConstAlphaTaps = 4096.0F;

// Whether a conversion of this plan carries alpha through its weights.
inline bool resample_alpha(const Plan& p) {
  if (p.dst.format != CC_RGBA8 && p.dst.format != CC_BGRA8) return false;
  if (p.src.format == CC_RGBA8 || p.src.format == CC_BGRA8) return true;
  return p.mode == CC_AREA && (p.scale_x + 2.0F) * (p.scale_y + 2.0F) > kConstAlphaTaps;
}

template <int kF>
__host__ __device__ constexpr bool is_wide() { return kF == CC_MONO16 || kF == CC_RGB16; }
template <int kF>
__host__ __device__ constexpr bool is_gray() { return kF == CC_MONO8 || kF == CC_MONO16; }

__device__ __forceinline__ int clamp_to(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// 2^23 + byte k of w, as a float.
__device__ __forceinline__ float biased(uint32_t w, int k) {
  return __uint_as_float(__byte_perm(w, kTwo23Bits, 0x7650U | static_cast<uint32_t>(k)));
}

// A source row: where it starts in each plane. kFast: planes below 4 GB, so
// that offsets are 32 bits and a load's address is the plane's uniform base
// plus one register, and chroma pairs or packed words aligned to be read
// whole; else 64-bit offsets and byte loads (fast_source).
template <bool kFast>
struct SourceRow {
  using Offset = std::conditional_t<kFast, uint32_t, size_t>;
  Offset at[3];
};

template <int kF, bool kFast>
__device__ __forceinline__ SourceRow<kFast> source_row(const Image& img, int y) {
  using Offset = typename SourceRow<kFast>::Offset;
  constexpr FormatInfo fi = info_of(kF);
  SourceRow<kFast> r{};
#pragma unroll
  for (int k = 0; k < fi.planes; ++k) {
    r.at[k] = static_cast<Offset>(k > 0 ? (y >> fi.shift_y) : y) * static_cast<Offset>(img.pitch[k]);
  }
  return r;
}

// The samples of column x of a source row (kernel_math.hpp:112-161): 2^23 +
// code for 8-bit formats, the value itself for 16-bit ones; gray formats fill
// c0 only.
template <int kF, bool kAlpha, bool kFast>
__device__ __forceinline__ Px load_biased(const Image& img, const SourceRow<kFast>& row, int x) {
  using Offset = typename SourceRow<kFast>::Offset;
  const auto byte_at = [&](int plane, int i) -> uint32_t {
    return __ldg(img.data[plane] + (row.at[plane] + static_cast<Offset>(i)));
  };
  const auto word_sample_at = [&](int i) {  // 16-bit little-endian, of any alignment
    return div257(byte_at(0, i) | (byte_at(0, i + 1) << 8));
  };
  const float opaque = __uint_as_float(kTwo23Bits | 255U);
  if constexpr (kF == CC_MONO16) {
    return {word_sample_at(2 * x), 0.0F, 0.0F, 255.0F};
  } else if constexpr (kF == CC_RGB16) {
    return {word_sample_at(6 * x), word_sample_at(6 * x + 2), word_sample_at(6 * x + 4), 255.0F};
  } else if constexpr (kF == CC_MONO8) {
    return {biased(byte_at(0, x), 0), 0.0F, 0.0F, opaque};
  } else if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    const Offset at = row.at[1] + static_cast<Offset>(x & ~1);
    const uint32_t w = kFast ? __ldg(reinterpret_cast<const uint16_t*>(img.data[1] + at))
                             : byte_at(1, x & ~1) | (byte_at(1, x | 1) << 8);
    return {biased(byte_at(0, x), 0), biased(w, 0), biased(w, 1), opaque};
  } else if constexpr (kF == CC_I420) {
    return {biased(byte_at(0, x), 0), biased(byte_at(1, x >> 1), 0), biased(byte_at(2, x >> 1), 0), opaque};
  } else if constexpr (kF == CC_RGB8 || kF == CC_BGR8) {
    const float a = biased(byte_at(0, 3 * x), 0), b = biased(byte_at(0, 3 * x + 1), 0), c = biased(byte_at(0, 3 * x + 2), 0);
    return kF == CC_RGB8 ? Px{a, b, c, opaque} : Px{c, b, a, opaque};
  } else {
    // Four bytes: a pixel (RGBA8, BGRA8) or a pixel pair (YUYV, UYVY).
    constexpr bool kPair = kF == CC_YUYV || kF == CC_UYVY;
    const int i = kPair ? 2 * (x & ~1) : 4 * x;
    const uint32_t w = kFast ? ldw(img.data[0] + (row.at[0] + static_cast<Offset>(i)))
                             : byte_at(0, i) | (byte_at(0, i + 1) << 8) | (byte_at(0, i + 2) << 16) | (byte_at(0, i + 3) << 24);
    if constexpr (kF == CC_YUYV) return {biased((x & 1) ? w >> 16 : w, 0), biased(w, 1), biased(w, 3), opaque};
    if constexpr (kF == CC_UYVY) return {biased((x & 1) ? w >> 16 : w, 1), biased(w, 0), biased(w, 2), opaque};
    const float al = kAlpha ? biased(w, 3) : opaque;
    return kF == CC_RGBA8 ? Px{biased(w, 0), biased(w, 1), biased(w, 2), al}
                          : Px{biased(w, 2), biased(w, 1), biased(w, 0), al};
  }
}

// Two pixels' samples, one per lane, and their weighted sums.
struct Pair {
  float2 c[4];
};

template <int kF, bool kAlpha, bool kFast>
__device__ __forceinline__ Pair load_pair(const Image& img, const SourceRow<kFast>& row, int xa, int xb) {
  const Px a = load_biased<kF, kAlpha>(img, row, xa), b = load_biased<kF, kAlpha>(img, row, xb);
  return {{make_float2(a.c0, b.c0), make_float2(a.c1, b.c1), make_float2(a.c2, b.c2), make_float2(a.a, b.a)}};
}

// sum += sample x w per lane, product then sum, each rounded (:163-165); kFirst:
// the sum is the product (0 + product).
template <int kF, bool kAlpha, bool kFirst>
__device__ __forceinline__ void weigh(Pair& sum, const Pair& s, float2 w) {
  const float2 bias = isp_b200::mul2(w, isp_b200::bc2(-kTwo23));
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if ((k == 1 || k == 2) && is_gray<kF>()) continue;
    if (k == 3 && !kAlpha) continue;
    const float2 product = is_wide<kF>() ? isp_b200::mul2(s.c[k], w) : isp_b200::exact_scale_add2(s.c[k], w, bias);
    sum.c[k] = kFirst ? product : isp_b200::psum2(product, sum.c[k]);
  }
}

// The plain samples behind load_pair's.
template <int kF>
__device__ __forceinline__ void unbias(Pair& s) {
  if constexpr (!is_wide<kF>()) {
#pragma unroll
    for (int k = 0; k < 4; ++k) s.c[k] = isp_b200::sub2(s.c[k], isp_b200::bc2(kTwo23));
  }
  if constexpr (is_gray<kF>()) s.c[1] = s.c[2] = isp_b200::bc2(0.0F);
}

// Weights of source pixels [ia, ia + 1) and [ib, ib + 1) in the footprints
// [lo, hi) of two pixels (:168-172): the overlap, 0 outside.
__device__ __forceinline__ float covered(int i, float lo, float hi) {
  const float a = fmaxf(static_cast<float>(i), lo);
  const float b = fminf(static_cast<float>(i + 1), hi);
  return fmaxf(__fsub_rn(b, a), 0.0F);
}
__device__ __forceinline__ float2 covered2(int ia, int ib, float2 lo, float2 hi) {
  return make_float2(covered(ia, lo.x, hi.x), covered(ib, lo.y, hi.y));
}

// s / d per lane, correctly rounded, from r = RN(1 / d): two of Markstein's
// correction steps (IBM Journal of Research and Development 34, 1990) on
// q = RN(s r). q is within 1.5 units in the last place, the first step leaves
// it within one, and from there the second gives the rounded quotient (the
// residuals are exact: no s here is near the subnormals).
__device__ __forceinline__ float2 divide2(float2 s, float2 d, float2 r) {
  using isp_b200::exact_scale_add2;
  const float2 minus_d = make_float2(-d.x, -d.y);
  const float2 q0 = isp_b200::mul2(s, r);
  const float2 q1 = exact_scale_add2(exact_scale_add2(q0, minus_d, s), r, q0);
  return exact_scale_add2(exact_scale_add2(q1, minus_d, s), r, q1);
}

// One axis of a destination pixel at `r` from the content's edge: where it
// samples the source (:175-233).
struct Axis {
  int a, b;       // nearest: a; bilinear: the two taps; area: the first pixel and one past the last
  float wa, wb;   // bilinear: the taps' weights; area: the footprint [wa, wb)
};

template <int kMode>
__device__ __forceinline__ Axis axis_at(int r, float first, float scale, int lo, int hi) {
  const float rf = static_cast<float>(r);
  Axis t{};
  if constexpr (kMode == CC_NEAREST) {
    t.a = clamp_to(static_cast<int>(floorf(__fadd_rn(first, __fmul_rn(__fadd_rn(rf, 0.5F), scale)))), lo, hi);
  } else if constexpr (kMode == CC_BILINEAR) {
    const float f = __fsub_rn(__fadd_rn(first, __fmul_rn(__fadd_rn(rf, 0.5F), scale)), 0.5F);
    const float base = floorf(f);
    const int i = static_cast<int>(base);
    t.wb = __fsub_rn(f, base);
    t.wa = __fsub_rn(1.0F, t.wb);
    t.a = clamp_to(i, lo, hi);
    t.b = clamp_to(i + 1, lo, hi);
  } else {
    // The footprint [l, h), inside the source rectangle.
    const float l = __fadd_rn(first, __fmul_rn(rf, scale));
    const float end = static_cast<float>(hi + 1);
    const float ls = __fadd_rn(l, scale);
    t.wa = l;
    t.wb = ls < end ? ls : end;
    t.a = clamp_to(static_cast<int>(floorf(l)), lo, hi);
    // The pixels i from a on with i <= hi and float(i) < h.
    t.b = clamp_to(static_cast<int>(ceilf(t.wb)), t.a, hi + 1);
  }
  return t;
}

// Area sums of four pixels over their footprints, kTaps columns of every row
// (0: any number, two at a time): past a pixel's own footprint the weight is 0
// and the tap any pixel of the source.
template <int kF, bool kAlpha, bool kFast, int kTaps>
__device__ __forceinline__ void sum_area(const Plan& p, const Axis (&x)[kGroupX], const Axis& y, int taps, Pair (&s)[2],
                                         float2 (&total)[2]) {
  using isp_b200::bc2;
  using isp_b200::mul2;
  using isp_b200::psum2;
  constexpr int kAtOnce = kTaps > 0 ? kTaps : 2;
  float2 wx[2][kAtOnce];
  const auto weights = [&](int t0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const Axis &a = x[2 * h], &b = x[2 * h + 1];
#pragma unroll
      for (int t = 0; t < kAtOnce; ++t) {
        wx[h][t] = covered2(a.a + t0 + t, b.a + t0 + t, make_float2(a.wa, b.wa), make_float2(a.wb, b.wb));
      }
    }
  };
  if constexpr (kTaps > 0) weights(0);
  for (int j = y.a; j < y.b; ++j) {
    const float2 wy = bc2(covered(j, y.wa, y.wb));
    const SourceRow<kFast> row = source_row<kF, kFast>(p.src, j);
    for (int t0 = 0; t0 < (kTaps > 0 ? 1 : taps); t0 += kAtOnce) {
      if constexpr (kTaps == 0) weights(t0);
      Pair tap[2][kAtOnce];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int t = 0; t < kAtOnce; ++t) {
          tap[h][t] = load_pair<kF, kAlpha>(p.src, row, min(x[2 * h].a + t0 + t, p.sx1), min(x[2 * h + 1].a + t0 + t, p.sx1));
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int t = 0; t < kAtOnce; ++t) {
          const float2 w = mul2(wx[h][t], wy);
          weigh<kF, kAlpha, false>(s[h], tap[h][t], w);
          total[h] = psum2(w, total[h]);
        }
      }
    }
  }
}

// The source sampled for four pixels of a row.
template <int kF, int kMode, bool kAlpha, bool kFast>
__device__ __forceinline__ void sample_group(const Plan& p, const Axis (&x)[kGroupX], const Axis& y, Px (&v)[kGroupX]) {
  using isp_b200::bc2;
  using isp_b200::mul2;
  Pair s[2];
  const SourceRow<kFast> first = source_row<kF, kFast>(p.src, y.a);
  if constexpr (kMode == CC_NEAREST) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      s[h] = load_pair<kF, kAlpha>(p.src, first, x[2 * h].a, x[2 * h + 1].a);
      unbias<kF>(s[h]);
    }
  } else if constexpr (kMode == CC_BILINEAR) {
    const SourceRow<kFast> second = source_row<kF, kFast>(p.src, y.b);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const Axis &a = x[2 * h], &b = x[2 * h + 1];
      const float2 wa = make_float2(a.wa, b.wa), wb = make_float2(a.wb, b.wb);
      const Pair t00 = load_pair<kF, kAlpha>(p.src, first, a.a, b.a);
      const Pair t10 = load_pair<kF, kAlpha>(p.src, first, a.b, b.b);
      const Pair t01 = load_pair<kF, kAlpha>(p.src, second, a.a, b.a);
      const Pair t11 = load_pair<kF, kAlpha>(p.src, second, a.b, b.b);
      weigh<kF, kAlpha, true>(s[h], t00, mul2(wa, bc2(y.wa)));
      weigh<kF, kAlpha, false>(s[h], t10, mul2(wb, bc2(y.wa)));
      weigh<kF, kAlpha, false>(s[h], t01, mul2(wa, bc2(y.wb)));
      weigh<kF, kAlpha, false>(s[h], t11, mul2(wb, bc2(y.wb)));
    }
  } else {
    s[0] = s[1] = Pair{};
    float2 total[2] = {bc2(0.0F), bc2(0.0F)};
    const int taps = max(max(x[0].b - x[0].a, x[1].b - x[1].a), max(x[2].b - x[2].a, x[3].b - x[3].a));
    switch (taps) {
      case 1:
      case 2: sum_area<kF, kAlpha, kFast, 2>(p, x, y, taps, s, total); break;
      case 3: sum_area<kF, kAlpha, kFast, 3>(p, x, y, taps, s, total); break;
      default: sum_area<kF, kAlpha, kFast, 0>(p, x, y, taps, s, total); break;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (total[h].x > 0.0F && total[h].y > 0.0F) {
        const float2 r = make_float2(__frcp_rn(total[h].x), __frcp_rn(total[h].y));
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if ((k == 1 || k == 2) && is_gray<kF>()) continue;
          if (k == 3 && !kAlpha) continue;
          s[h].c[k] = divide2(s[h].c[k], total[h], r);
        }
      } else {
        // A footprint of no weight takes its first pixel.
        Pair edge = load_pair<kF, kAlpha>(p.src, first, x[2 * h].a, x[2 * h + 1].a);
        unbias<kF>(edge);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          s[h].c[k].x = total[h].x > 0.0F ? __fdiv_rn(s[h].c[k].x, total[h].x) : edge.c[k].x;
          s[h].c[k].y = total[h].y > 0.0F ? __fdiv_rn(s[h].c[k].y, total[h].y) : edge.c[k].y;
        }
      }
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if constexpr (is_gray<kF>()) s[h].c[1] = s[h].c[2] = bc2(0.0F);
    if constexpr (!kAlpha) s[h].c[3] = bc2(255.0F);
    v[2 * h] = Px{s[h].c[0].x, s[h].c[1].x, s[h].c[2].x, s[h].c[3].x};
    v[2 * h + 1] = Px{s[h].c[0].y, s[h].c[1].y, s[h].c[2].y, s[h].c[3].y};
  }
}

// Stores rows y0 .. of a block of four pixels across (n of them inside the
// image) and their chroma. Whole blocks of 4-byte aligned rows go out as the
// direct path's; others pixel by pixel.
template <int kDst, int kRows>
__device__ __forceinline__ void store_block(const Plan& p, int x, int y0, int n, int rows, const Px (&v)[kRows][kGroupX]) {
  constexpr FormatInfo fi = info_of(kDst);
  constexpr bool kYuvDst = fi.model == kYuv;
  constexpr int kBlockRows = kYuvDst ? (1 << fi.shift_y) : 1;  // rows that share chroma
#pragma unroll
  for (int top = 0; top + kBlockRows <= kRows; top += kBlockRows) {
    if (top >= rows) break;
    const int down = rows - top < kBlockRows ? 1 : kBlockRows;  // rows of this block inside the image
    float cbs[2] = {0.0F, 0.0F}, crs[2] = {0.0F, 0.0F};
    bool whole = n == kGroupX;
#pragma unroll
    for (int r = top; r < top + kBlockRows; ++r) {
      if (r >= rows) break;
      whole = whole && aligned4(row_of(p.dst, 0, y0 + r));
      if constexpr (kYuvDst) {
#pragma unroll
        for (int i = 0; i < kGroupX; ++i) {
          if (i < n) {
            cbs[i >> 1] = __fadd_rn(cbs[i >> 1], v[r][i].c1);
            crs[i >> 1] = __fadd_rn(crs[i >> 1], v[r][i].c2);
          }
        }
      }
    }
    // Chroma means: a block holds 1, 2 or 4 pixels, so dividing by the count
    // is exactly the product by its reciprocal.
    if constexpr (kYuvDst) {
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const int count = (n - 2 * b >= 2 ? 2 : 1) * down;
        const float inv = count == 4 ? 0.25F : (count == 2 ? 0.5F : 1.0F);
        cbs[b] = __fmul_rn(cbs[b], inv);
        crs[b] = __fmul_rn(crs[b], inv);
      }
    }
    const uint32_t cb[2] = {code8_bits(cbs[0]), code8_bits(cbs[1])}, cr[2] = {code8_bits(crs[0]), code8_bits(crs[1])};
#pragma unroll
    for (int r = top; r < top + kBlockRows; ++r) {
      if (r >= rows) break;
      if (whole) {
        store_full4<kDst>(p.dst, x, y0 + r, v[r], cb, cr);
      } else {
#pragma unroll
        for (int i = 0; i < kGroupX; ++i) {
          if (i < n) store_px<kDst>(p.dst, x + i, y0 + r, v[r][i]);
        }
      }
    }
    if constexpr (kYuvDst) {
      constexpr bool kPacked = kDst == CC_YUYV || kDst == CC_UYVY;  // in the rows' own words
      if (!(kPacked && whole)) {
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if (2 * b < n) store_chroma<kDst>(p.dst, (x >> 1) + b, (y0 + top) >> fi.shift_y, cbs[b], crs[b]);
        }
      }
    }
  }
}

// ---- Area footprints of whole pixels --------------------------------------
//
// With the source rectangle exactly kScale times the content across and a whole
// number of times down, every weight is 1 and every sum an integer below 2^24:
// the definition's float sums are exact, so integer sums in any order give the
// same value, and only the division by the pixel count rounds. Four pixels'
// sources are then 4 kScale columns, whole 32-bit words of each plane, and
// __dp4a adds the bytes of a sample with constant 0 / 1 / 2 weights.

// How often byte `b` of plane `plane` of a row of 4 kScale columns counts for
// sample `c` of pixel `i`.
template <int kF>
__host__ __device__ constexpr uint32_t byte_weight(int scale, int plane, int b, int i, int c) {
  uint32_t n = 0;
  for (int x = i * scale; x < (i + 1) * scale; ++x) {
    int at = -1;  // the byte of sample c of column x in this plane
    if (kF == CC_NV12 || kF == CC_NV16) {
      at = plane == 0 ? (c == 0 ? x : -1) : (c == 1 || c == 2 ? 2 * (x >> 1) + c - 1 : -1);
    } else if (kF == CC_I420) {
      at = plane == c ? (c == 0 ? x : (x >> 1)) : -1;
    } else if (kF == CC_YUYV) {
      at = c == 0 ? 2 * x : c < 3 ? 4 * (x >> 1) + 2 * c - 1 : -1;
    } else if (kF == CC_UYVY) {
      at = c == 0 ? 2 * x + 1 : c < 3 ? 4 * (x >> 1) + 2 * c - 2 : -1;
    } else if (kF == CC_RGB8 || kF == CC_BGR8) {
      at = c < 3 ? 3 * x + (kF == CC_BGR8 ? 2 - c : c) : -1;
    } else if (kF == CC_RGBA8 || kF == CC_BGRA8) {
      at = 4 * x + (c < 3 && kF == CC_BGRA8 ? 2 - c : c);
    } else {
      at = c == 0 ? x : -1;
    }
    if (at == b) ++n;
  }
  return n;
}

// Words of a row of 4 kScale columns in each plane.
template <int kF>
__host__ __device__ constexpr int row_words(int scale, int plane) {
  return kF == CC_I420 ? (plane == 0 ? scale : scale / 2)
         : kF == CC_YUYV || kF == CC_UYVY ? 2 * scale
         : kF == CC_RGB8 || kF == CC_BGR8 ? 3 * scale
         : kF == CC_RGBA8 || kF == CC_BGRA8 ? 4 * scale
                                            : scale;
}

template <int kF, int kScale, int kWord>
struct WordWeights {
  template <int kPlane, int kPx, int kC>
  static constexpr uint32_t value = byte_weight<kF>(kScale, kPlane, 4 * kWord, kPx, kC) |
                                    byte_weight<kF>(kScale, kPlane, 4 * kWord + 1, kPx, kC) << 8 |
                                    byte_weight<kF>(kScale, kPlane, 4 * kWord + 2, kPx, kC) << 16 |
                                    byte_weight<kF>(kScale, kPlane, 4 * kWord + 3, kPx, kC) << 24;
};

template <int kF, int kScale, int kPlane, int kWord, int kPx, int kC>
__device__ __forceinline__ void add_word(uint32_t w, uint32_t (&sum)[kGroupX][4]) {
  constexpr uint32_t kWeights = WordWeights<kF, kScale, kWord>::template value<kPlane, kPx, kC>;
  if constexpr (kWeights != 0U) sum[kPx][kC] = __dp4a(w, kWeights, sum[kPx][kC]);
  if constexpr (kC + 1 < 4) {
    add_word<kF, kScale, kPlane, kWord, kPx, kC + 1>(w, sum);
  } else if constexpr (kPx + 1 < kGroupX) {
    add_word<kF, kScale, kPlane, kWord, kPx + 1, 0>(w, sum);
  }
}

template <int kF, int kScale, int kPlane, int kWord = 0>
__device__ __forceinline__ void add_words(const uint32_t (&w)[row_words<kF>(kScale, kPlane)], uint32_t (&sum)[kGroupX][4]) {
  if constexpr (kWord < row_words<kF>(kScale, kPlane)) {
    add_word<kF, kScale, kPlane, kWord, 0, 0>(w[kWord], sum);
    add_words<kF, kScale, kPlane, kWord + 1>(w, sum);
  }
}

// Adds row sy of plane kPlane and those after it; sx: the group's first source column.
template <int kF, int kScale, int kPlane>
__device__ __forceinline__ void add_row(const Image& img, int sx, int sy, uint32_t (&sum)[kGroupX][4]) {
  constexpr int kN = row_words<kF>(kScale, kPlane);
  constexpr int kShift = kPlane > 0 && (kF == CC_NV12 || kF == CC_I420) ? 1 : 0;
  // Bytes before column sx: as many as the words of sx columns.
  const uint8_t* at = row_of(img, kPlane, sy >> kShift) + 4 * kN * (sx / (4 * kScale)) ;
  uint32_t w[kN];
#pragma unroll
  for (int k = 0; k < kN; ++k) w[k] = ldw(at + 4 * k);
  add_words<kF, kScale, kPlane>(w, sum);
  if constexpr (kPlane + 1 < info_of(kF).planes) add_row<kF, kScale, kPlane + 1>(img, sx, sy, sum);
}

// Whether a plan's area footprints are whole pixels that sum_whole takes, and
// the factor across (0: no). Every group of four content pixels must start at
// a multiple of four in the destination, and its source on whole words.
inline int whole_scale(const Plan& p) {
  if (p.mode != CC_AREA || p.src.format == CC_MONO16 || p.src.format == CC_RGB16) return 0;
  const int sw = p.sx1 - p.sx0 + 1, sh = p.sy1 - p.sy0 + 1, cw = p.cx1 - p.cx0, ch = p.cy1 - p.cy0;
  const int scale = sw / cw;
  if (scale < 2 || scale > 4 || sw != scale * cw || sh % ch != 0 || sh / ch > 4096) return 0;
  if (p.sx1 >= (1 << 22) || p.sy1 >= (1 << 22) || p.cx0 % kGroupX != 0) return 0;  // exact coordinates
  const bool thirds = p.src.format == CC_I420;  // chroma words: 2 kScale columns a byte pair
  if (p.sx0 != 0 || (thirds && scale % 2 != 0)) return 0;
  for (int k = 0; k < info_of(p.src.format).planes; ++k) {
    if (((reinterpret_cast<uintptr_t>(p.src.data[k]) | p.src.pitch[k]) & 3U) != 0U) return 0;
  }
  return scale;
}

// Four pixels whose footprints are kScale columns by `high` rows from (sx, sy).
template <int kF, int kScale>
__device__ __forceinline__ void sum_whole(const Plan& p, int sx, int sy, int high, Px (&v)[kGroupX]) {
  uint32_t sum[kGroupX][4] = {};
#pragma unroll 2
  for (int j = 0; j < high; ++j) add_row<kF, kScale, 0>(p.src, sx, sy + j, sum);
  const float count = static_cast<float>(kScale * high);
  const float2 d = make_float2(count, count);
  const float2 r = isp_b200::bc2(__frcp_rn(count));
  constexpr bool kAlpha = kF == CC_RGBA8 || kF == CC_BGRA8;
#pragma unroll
  for (int i = 0; i < kGroupX; i += 2) {
    float2 c[4] = {isp_b200::bc2(0.0F), isp_b200::bc2(0.0F), isp_b200::bc2(0.0F), isp_b200::bc2(255.0F)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if ((k == 1 || k == 2) && is_gray<kF>()) continue;
      if (k == 3 && !kAlpha) continue;
      c[k] = divide2(make_float2(static_cast<float>(sum[i][k]), static_cast<float>(sum[i + 1][k])), d, r);
    }
    v[i] = Px{c[0].x, c[1].x, c[2].x, c[3].x};
    v[i + 1] = Px{c[0].y, c[1].y, c[2].y, c[3].y};
  }
}

// Whether a plan's source suits SourceRow's fast form.
inline bool fast_source(const Plan& p) {
  const FormatInfo fi = info_of(p.src.format);
  const bool words = p.src.format == CC_YUYV || p.src.format == CC_UYVY || p.src.format == CC_RGBA8 || p.src.format == CC_BGRA8;
  for (int k = 0; k < fi.planes; ++k) {
    if (p.src.pitch[k] > 0xFFFFFFFFU / static_cast<size_t>(p.src.height)) return false;
    if (((reinterpret_cast<uintptr_t>(p.src.data[k]) | p.src.pitch[k]) & (words ? 3U : fi.planes == 2 && k == 1 ? 1U : 0U)) != 0U) {
      return false;
    }
  }
  return true;
}

// CTAs per SM asked of the compiler.
__host__ __device__ constexpr int resample_blocks(int mode, int rows, int scale) {
  return rows == 2 ? 4 : scale > 0 ? 6 : 5;
}

// kRows: rows per thread, 2 for 4:2:0 destinations and 1 for others. kScale:
// the factor of whole area footprints (whole_scale), or 0.
template <int kF, int kMode, bool kAlpha, int kRows, int kScale, bool kFast>
__global__ void __launch_bounds__(kThreadsX* kResampleThreadsY, resample_blocks(kMode, kRows, kScale)) cc_resample_kernel(const __grid_constant__ Plan p, int across,
                                                                                   int down) {
  // A programmatic dependent (launch_dependent): no memory before the wait.
  isp_b200::griddep_launch_dependents();
  isp_b200::griddep_wait();
  const int gx = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
  if (gx >= across) return;
  const int x = gx * kGroupX;
  const int n = min(p.dst.width - x, kGroupX);
  const bool inside = x >= p.cx0 && x + kGroupX <= p.cx1;
  // Pixels outside the content sample its edge (every tap is clamped to the
  // source) and then take the fill.
  Axis ax[kGroupX];
  if (kScale == 0 || !inside) {
#pragma unroll
    for (int i = 0; i < kGroupX; ++i) {
      ax[i] = axis_at<kMode>(clamp_to(x + i, p.cx0, p.cx1 - 1) - p.cx0, static_cast<float>(p.sx0), p.scale_x, p.sx0, p.sx1);
    }
  }
  // One pass unless the image has more block rows than a grid may have.
  for (int gy = static_cast<int>(blockIdx.y * blockDim.y + threadIdx.y); gy < down; gy += static_cast<int>(gridDim.y * blockDim.y)) {
    const int y0 = gy * kRows;
    const int rows = min(p.dst.height - y0, kRows);
    Px v[kRows][kGroupX];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const int y = clamp_to(y0 + r, p.cy0, p.cy1 - 1);
      if (kScale > 0 && inside) {
        const int high = static_cast<int>(p.scale_y);
        sum_whole<kF, (kScale > 0 ? kScale : 2)>(p, (x - p.cx0) * kScale, p.sy0 + (y - p.cy0) * high, high, v[r]);
      } else {
        const Axis ay = axis_at<kMode>(y - p.cy0, static_cast<float>(p.sy0), p.scale_y, p.sy0, p.sy1);
        sample_group<kF, kMode, kAlpha, kFast>(p, ax, ay, v[r]);
      }
      if (!p.identity) {
        affine_pair(p, v[r][0], v[r][1]);
        affine_pair(p, v[r][2], v[r][3]);
      }
      if (!inside || y != y0 + r) {
#pragma unroll
        for (int i = 0; i < kGroupX; ++i) {
          if (y != y0 + r || x + i < p.cx0 || x + i >= p.cx1) v[r][i] = Px{p.fill[0], p.fill[1], p.fill[2], p.fill[3]};
        }
      }
    }
    if constexpr (kRows == 2) {
      if (p.dst.format == CC_NV12) {
        store_block<CC_NV12>(p, x, y0, n, rows, v);
      } else {
        store_block<CC_I420>(p, x, y0, n, rows, v);
      }
    } else {
      switch (p.dst.format) {
        case CC_NV16: store_block<CC_NV16>(p, x, y0, n, rows, v); break;
        case CC_YUYV: store_block<CC_YUYV>(p, x, y0, n, rows, v); break;
        case CC_UYVY: store_block<CC_UYVY>(p, x, y0, n, rows, v); break;
        case CC_RGB8: store_block<CC_RGB8>(p, x, y0, n, rows, v); break;
        case CC_BGR8: store_block<CC_BGR8>(p, x, y0, n, rows, v); break;
        case CC_RGBA8: store_block<CC_RGBA8>(p, x, y0, n, rows, v); break;
        case CC_BGRA8: store_block<CC_BGRA8>(p, x, y0, n, rows, v); break;
        case CC_MONO8: store_block<CC_MONO8>(p, x, y0, n, rows, v); break;
        case CC_MONO16: store_block<CC_MONO16>(p, x, y0, n, rows, v); break;
        default: store_block<CC_RGB16>(p, x, y0, n, rows, v); break;
      }
    }
  }
}

// Rows a thread takes for a destination format.
inline int resample_rows(int dst) { return dst == CC_NV12 || dst == CC_I420 ? 2 : 1; }

// What picks an instance besides the source format and the mode.
struct ResampleKey {
  int dst;
  bool alpha;
  int scale;  // whole_scale
  bool fast;  // fast_source
};

template <int kSrc, int kMode, bool kAlpha, int kRows>
const void* resample_scaled(const ResampleKey& key) {
  if (!key.fast) return reinterpret_cast<const void*>(&cc_resample_kernel<kSrc, kMode, kAlpha, kRows, 0, false>);
  if constexpr (kMode == CC_AREA && !is_wide<kSrc>()) {
    if (key.scale == 2) return reinterpret_cast<const void*>(&cc_resample_kernel<kSrc, kMode, kAlpha, kRows, 2, true>);
    if constexpr (kSrc != CC_I420) {
      if (key.scale == 3) return reinterpret_cast<const void*>(&cc_resample_kernel<kSrc, kMode, kAlpha, kRows, 3, true>);
    }
    if (key.scale == 4) return reinterpret_cast<const void*>(&cc_resample_kernel<kSrc, kMode, kAlpha, kRows, 4, true>);
  }
  return reinterpret_cast<const void*>(&cc_resample_kernel<kSrc, kMode, kAlpha, kRows, 0, true>);
}

template <int kSrc, int kMode>
const void* resample_mode(const ResampleKey& key) {
  if (resample_rows(key.dst) == 2) return resample_scaled<kSrc, kMode, false, 2>(key);  // no alpha in 4:2:0
  if constexpr (kSrc == CC_RGBA8 || kSrc == CC_BGRA8 || kMode == CC_AREA) {
    if (key.alpha) return resample_scaled<kSrc, kMode, true, 1>(key);
  }
  return resample_scaled<kSrc, kMode, false, 1>(key);
}

// The resample kernels of one source format.
template <int kSrc>
const void* resample_for(int mode, const ResampleKey& key) {
  switch (mode) {
    case CC_NEAREST: return resample_mode<kSrc, CC_NEAREST>(key);
    case CC_BILINEAR: return resample_mode<kSrc, CC_BILINEAR>(key);
    case CC_AREA: return resample_mode<kSrc, CC_AREA>(key);
    default: return nullptr;
  }
}

const void* resample_kernel_planar(int src, int mode, const ResampleKey& key);
const void* resample_kernel_packed(int src, int mode, const ResampleKey& key);
const void* resample_kernel_rgb(int src, int mode, const ResampleKey& key);
const void* resample_kernel_other(int src, int mode, const ResampleKey& key);

}  // namespace cc_b200
