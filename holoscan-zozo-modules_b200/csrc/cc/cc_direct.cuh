// cc_direct.cuh - the converter's direct path: each destination pixel reads the
// one source pixel under it.
#pragma once

#include "cc_kernels.cuh"

namespace cc_b200 {
namespace {

using isp_b200::add2;
using isp_b200::add2_rz;
using isp_b200::bc2;
using isp_b200::exact_scale_add2;
using isp_b200::mul2;
using isp_b200::psum2;
using isp_b200::sub2;

// ---- Whole groups: four pixels in words --------------------------------------

constexpr int kRawWords = 6;  // of a group, at most (RGB16)

__host__ __device__ constexpr bool shares_chroma(int f) { return info_of(f).model == kYuv; }
// Bytes a pixel takes in plane 0, which is also the words a group takes.
__host__ __device__ constexpr int plane_bytes(int f) {
  return f == CC_YUYV || f == CC_UYVY ? 2 : info_of(f).model == kYuv ? 1 : info_of(f).channels * info_of(f).bytes;
}

// kN words from p. kShifted: p may lie at any byte; the aligned words that hold
// the bytes are read and shifted together (the last one only where it holds a
// byte of the group, so nothing outside the words of the row's own bytes is read).
template <int kN, bool kShifted>
__device__ __forceinline__ void load_words(const uint8_t* p, uint32_t* w) {
  if constexpr (kShifted) {
    const unsigned int s = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(p)) & 3U;
    const uint8_t* base = p - s;
    uint32_t raw[kN + 1];
#pragma unroll
    for (int k = 0; k < kN; ++k) raw[k] = ldw(base + 4 * k);
    raw[kN] = s != 0U ? ldw(base + 4 * kN) : 0U;
#pragma unroll
    for (int k = 0; k < kN; ++k) w[k] = __funnelshift_r(raw[k], raw[k + 1], 8U * s);
  } else {
#pragma unroll
    for (int k = 0; k < kN; ++k) w[k] = ldw(p + 4 * k);
  }
}

// Whether groups of row sy (from a column that is a multiple of four plus
// dx, dx even for shared chroma) lie on word boundaries.
template <int kF>
__device__ __forceinline__ bool source_aligned(const Image& img, int dx, int sy) {
  bool ok = aligned4(row_of(img, 0, sy) + plane_bytes(kF) * dx);
  if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    ok = ok && aligned4(row_of(img, 1, kF == CC_NV12 ? (sy >> 1) : sy) + dx);
  } else if constexpr (kF == CC_I420) {
    ok = ok && ((reinterpret_cast<uintptr_t>(row_of(img, 1, sy >> 1) + (dx >> 1)) |
                 reinterpret_cast<uintptr_t>(row_of(img, 2, sy >> 1) + (dx >> 1))) & 1U) == 0U;
  }
  return ok;
}

// The bytes of source pixels sx .. sx + 3 of row sy; of shared chroma, the two
// pairs Cb0, Cr0, Cb1, Cr1 in a word.
template <int kF, bool kShifted>
__device__ __forceinline__ void fetch4(const Image& img, int sx, int sy, uint32_t (&w)[kRawWords]) {
  load_words<plane_bytes(kF), kShifted>(row_of(img, 0, sy) + plane_bytes(kF) * sx, w);
  if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    load_words<1, kShifted>(row_of(img, 1, kF == CC_NV12 ? (sy >> 1) : sy) + sx, w + 1);
  } else if constexpr (kF == CC_I420) {
    const uint8_t* u = row_of(img, 1, sy >> 1) + (sx >> 1);
    const uint8_t* v = row_of(img, 2, sy >> 1) + (sx >> 1);
    if constexpr (kShifted) {
      w[1] = static_cast<uint32_t>(__ldg(u)) | (static_cast<uint32_t>(__ldg(v)) << 8) |
             (static_cast<uint32_t>(__ldg(u + 1)) << 16) | (static_cast<uint32_t>(__ldg(v + 1)) << 24);
    } else {
      w[1] = __byte_perm(__ldg(reinterpret_cast<const unsigned short*>(u)),
                         __ldg(reinterpret_cast<const unsigned short*>(v)), 0x5140U);
    }
  }
}

// A group's samples as lane pairs: [0] holds pixels 0 and 2, [1] pixels 1 and 3,
// so that the lanes are the group's two chroma blocks: shared chroma is one
// pair, and a block's sum is a two-lane sum. Samples of 8-bit formats stay
// biased (2^23 + sample).
struct Group {
  float2 c[3][2];
  float2 a[2];
};

__device__ __forceinline__ float2 biased2(uint32_t wa, int ka, uint32_t wb, int kb) {
  return make_float2(__uint_as_float(__byte_perm(wa, kTwo23Bits, 0x7650U | static_cast<uint32_t>(ka))),
                     __uint_as_float(__byte_perm(wb, kTwo23Bits, 0x7650U | static_cast<uint32_t>(kb))));
}

template <int kF>
__device__ __forceinline__ Group decode4(const uint32_t (&w)[kRawWords]) {
  Group g;
  if constexpr (info_of(kF).bytes == 2) {
    constexpr int kC = info_of(kF).channels;
#pragma unroll
    for (int j = 0; j < kC; ++j) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = div257((w[(kC * i + j) >> 1] >> (16 * ((kC * i + j) & 1))) & 0xFFFFU);
      g.c[j][0] = make_float2(v[0], v[2]);
      g.c[j][1] = make_float2(v[1], v[3]);
    }
  } else if constexpr (info_of(kF).model == kRgb) {
    constexpr int kC = info_of(kF).channels;
    constexpr bool kBgr = kF == CC_BGR8 || kF == CC_BGRA8;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
      for (int j = 0; j < kC; ++j) {
        const int m = kC * h + j, n = kC * (h + 2) + j;
        const float2 v = biased2(w[m >> 2], m & 3, w[n >> 2], n & 3);
        if (j == 3) {
          g.a[h] = v;
        } else {
          g.c[kBgr ? 2 - j : j][h] = v;
        }
      }
    }
  } else if constexpr (kF == CC_YUYV || kF == CC_UYVY) {
    constexpr int kY = kF == CC_YUYV ? 0 : 1;  // byte of the first luma in a pair
    constexpr int kU = kF == CC_YUYV ? 1 : 0;  // byte of Cb; Cr two later
    g.c[0][0] = biased2(w[0], kY, w[1], kY);
    g.c[0][1] = biased2(w[0], kY + 2, w[1], kY + 2);
    g.c[1][0] = g.c[1][1] = biased2(w[0], kU, w[1], kU);
    g.c[2][0] = g.c[2][1] = biased2(w[0], kU + 2, w[1], kU + 2);
  } else {
    g.c[0][0] = biased2(w[0], 0, w[0], 2);
    g.c[0][1] = biased2(w[0], 1, w[0], 3);
    if constexpr (info_of(kF).model == kYuv) {
      g.c[1][0] = g.c[1][1] = biased2(w[1], 0, w[1], 2);
      g.c[2][0] = g.c[2][1] = biased2(w[1], 1, w[1], 3);
    }
  }
  return g;
}

// Sample k of the colour map of pixels h: ((m0 c0 + m1 c1) + m2 c2) + o, every
// operation rounded. Gray sources have zeros for c1 and c2: products of zero,
// left out.
template <bool kGraySrc>
__device__ __forceinline__ float2 mapped(const Plan& p, int k, const Group& g, int h) {
  float2 t = mul2(g.c[0][h], bc2(p.m[3 * k]));
  if constexpr (!kGraySrc) {
    t = psum2(t, mul2(g.c[1][h], bc2(p.m[3 * k + 1])));
    t = psum2(mul2(g.c[2][h], bc2(p.m[3 * k + 2])), t);
    return add2(t, bc2(p.o[k]));
  }
  return psum2(t, bc2(p.o[k]));
}

// Two 8-bit codes in the halves of a word, from v + 0.5 (code8): the floor is
// 2^23 + v rounded toward zero (for a negative v, bits below those of 2^23), the
// clamp a two-half-word one of its low bits. |v| < 2^14.
__device__ __forceinline__ uint32_t codes8_of_half(float2 h) {
  const float2 r = add2_rz(h, bc2(kTwo23));
  return __vimin_s16x2_relu(__byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x5410U), 0x00FF00FFU);
}
__device__ __forceinline__ uint32_t codes8(float2 v) { return codes8_of_half(add2(v, bc2(0.5F))); }
// Two 16-bit codes (code16).
__device__ __forceinline__ uint2 codes16(float2 v) {
  const float2 r = add2_rz(psum2(mul2(v, bc2(257.0F)), bc2(0.5F)), bc2(kTwo23));
  return make_uint2(static_cast<uint32_t>(__viaddmin_s32_relu(__float_as_int(r.x), -static_cast<int>(kTwo23Bits), 65535)),
                    static_cast<uint32_t>(__viaddmin_s32_relu(__float_as_int(r.y), -static_cast<int>(kTwo23Bits), 65535)));
}

// Four 8-bit codes in pixel order, from those of pixels (0, 2) and (1, 3).
__device__ __forceinline__ uint32_t zip8(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x6240U); }

// One whole group: its plane 0 words, and for YCbCr destinations its chroma
// samples added to the blocks' sums pixel by pixel, which is the definition's
// order (first: the sums begin here).
template <int kSrc, int kDst>
__device__ __forceinline__ void convert4(const Plan& p, const uint32_t (&raw)[kRawWords], uint32_t (&w)[plane_bytes(kDst)],
                                         bool first, float2& cb, float2& cr) {
  constexpr FormatInfo from = info_of(kSrc), to = info_of(kDst);
  constexpr bool kIdentity = from.model == to.model;
  constexpr bool kBiased = from.bytes == 1;
  Group g = decode4<kSrc>(raw);
  if constexpr (!kIdentity && kBiased) {
#pragma unroll
    for (int k = 0; k < (from.model == kGray ? 1 : 3); ++k) {
#pragma unroll
      for (int h = 0; h < 2; ++h) g.c[k][h] = sub2(g.c[k][h], bc2(kTwo23));
    }
  }
  const auto value = [&](int k, int h) {
    if constexpr (!kIdentity) return mapped<from.model == kGray>(p, k, g, h);
    else if constexpr (kBiased) return sub2(g.c[k][h], bc2(kTwo23));
    else return g.c[k][h];
  };
  if constexpr (to.bytes == 2) {
    constexpr int kC = to.channels;
    uint32_t code[4 * kC];
#pragma unroll
    for (int k = 0; k < kC; ++k) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint2 q = codes16(value(k, h));
        code[kC * h + k] = q.x;
        code[kC * (h + 2) + k] = q.y;
      }
    }
#pragma unroll
    for (int i = 0; i < 2 * kC; ++i) w[i] = pack16(code[2 * i], code[2 * i + 1]);
  } else {
    const auto codes = [&](int k, int h) -> uint32_t {
      if constexpr (kIdentity && kBiased) {
        return __byte_perm(__float_as_uint(g.c[k][h].x), __float_as_uint(g.c[k][h].y), 0x5410U);
      } else {
        return codes8(value(k, h));
      }
    };
    const uint32_t a0 = codes(0, 0), b0 = codes(0, 1);
    if constexpr (to.model == kYuv) {
      cb = add2(first ? value(1, 0) : add2(cb, value(1, 0)), value(1, 1));
      cr = add2(first ? value(2, 0) : add2(cr, value(2, 0)), value(2, 1));
    }
    if constexpr (kDst == CC_YUYV || kDst == CC_UYVY) {
      const uint32_t u = codes8_of_half(exact_scale_add2(cb, bc2(0.5F), bc2(0.5F)));
      const uint32_t v = codes8_of_half(exact_scale_add2(cr, bc2(0.5F), bc2(0.5F)));
      const uint32_t x = kDst == CC_YUYV ? zip8(a0, u) : zip8(u, a0), y = kDst == CC_YUYV ? zip8(b0, v) : zip8(v, b0);
      w[0] = __byte_perm(x, y, 0x5410U);
      w[1] = __byte_perm(x, y, 0x7632U);
    } else if constexpr (to.model == kRgb) {
      const uint32_t a1 = codes(1, 0), b1 = codes(1, 1), a2 = codes(2, 0), b2 = codes(2, 1);
      constexpr bool kBgr = kDst == CC_BGR8 || kDst == CC_BGRA8;
      const uint32_t ra = kBgr ? a2 : a0, rb = kBgr ? b2 : b0, ba = kBgr ? a0 : a2, bb = kBgr ? b0 : b2;
      if constexpr (to.channels == 3) {
        // r0 g0 b0 r1 | g1 b1 r2 g2 | b2 r3 g3 b3
        const uint32_t x = zip8(ra, a1), y = zip8(ba, rb), z = zip8(b1, bb);
        w[0] = __byte_perm(x, y, 0x5410U);
        w[1] = __byte_perm(z, x, 0x7610U);
        w[2] = __byte_perm(y, z, 0x7632U);
      } else {
        uint32_t al[2] = {0x00FF00FFU, 0x00FF00FFU};
        if constexpr (from.channels == 4) {
#pragma unroll
          for (int h = 0; h < 2; ++h) al[h] = __byte_perm(__float_as_uint(g.a[h].x), __float_as_uint(g.a[h].y), 0x5410U);
        }
        const uint32_t x = zip8(ra, a1), y = zip8(ba, al[0]), z = zip8(rb, b1), t = zip8(bb, al[1]);
        w[0] = __byte_perm(x, y, 0x5410U);
        w[1] = __byte_perm(z, t, 0x5410U);
        w[2] = __byte_perm(x, y, 0x7632U);
        w[3] = __byte_perm(z, t, 0x7632U);
      }
    } else {
      w[0] = zip8(a0, b0);
    }
  }
}

// Whether the rows that groups of row y0 (and the next) store start on word
// boundaries (half-word ones of I420's chroma planes).
template <int kF>
__device__ __forceinline__ bool destination_aligned(const Image& img, int y0) {
  bool ok = aligned4(row_of(img, 0, y0));
  if constexpr (kF == CC_NV12 || kF == CC_I420) ok = ok && aligned4(row_of(img, 0, y0 + 1));
  if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    ok = ok && aligned4(row_of(img, 1, kF == CC_NV12 ? y0 >> 1 : y0));
  } else if constexpr (kF == CC_I420) {
    ok = ok && ((reinterpret_cast<uintptr_t>(row_of(img, 1, y0 >> 1)) |
                 reinterpret_cast<uintptr_t>(row_of(img, 2, y0 >> 1))) & 1U) == 0U;
  }
  return ok;
}

// A warp's row segment: lane L's kN words at q = q0 + 4 kN L, for the lanes of
// `whole`. Rows at any byte (unless kPlain): the words are shifted into the
// aligned words they span, the left neighbour's last bytes coming by a shuffle;
// the first and the last of neighbouring lanes store the ends byte by byte, so
// that no byte of another lane's is written. All lanes call.
template <int kN, bool kPlain>
__device__ __forceinline__ void store_words(uint8_t* q, const uint32_t (&w)[kN], unsigned int whole) {
  const unsigned int s = kPlain ? 0U : static_cast<unsigned int>(reinterpret_cast<uintptr_t>(q)) & 3U;
  const int lane = static_cast<int>(threadIdx.x);
  const bool mine = kPlain || ((whole >> lane) & 1U) != 0U;
  if (s == 0U) {
    if (mine) {
#pragma unroll
      for (int k = 0; k < kN; ++k) reinterpret_cast<uint32_t*>(q)[k] = w[k];
    }
    return;
  }
  const uint32_t carry = __shfl_up_sync(0xFFFFFFFFU, w[kN - 1], 1);
  if (!mine) return;
  uint32_t* base = reinterpret_cast<uint32_t*>(q - s);
  if (lane > 0 && ((whole >> (lane - 1)) & 1U) != 0U) {
    base[0] = __funnelshift_l(carry, w[0], 8U * s);
  } else {
#pragma unroll
    for (unsigned int b = 0; b < 3U; ++b) {
      if (b < 4U - s) q[b] = static_cast<uint8_t>(w[0] >> (8U * b));
    }
  }
#pragma unroll
  for (int k = 1; k < kN; ++k) base[k] = __funnelshift_l(w[k - 1], w[k], 8U * s);
  if (lane == 31 || ((whole >> (lane + 1)) & 1U) == 0U) {
#pragma unroll
    for (unsigned int b = 1; b <= 3U; ++b) {  // the group's last s bytes
      if (b <= s) q[4 * kN - static_cast<int>(b)] = static_cast<uint8_t>(w[kN - 1] >> (32U - 8U * b));
    }
  }
}

// A warp's groups of `whole` at column xs of `rows` rows, converted and stored.
template <int kSrc, int kDst, bool kPlain, int kRows>
__device__ __forceinline__ void convert_group(const Plan& p, const uint32_t (&raw)[kRows][kRawWords], int rows, int xs, int y0,
                                              unsigned int whole) {
  constexpr int kBytes = plane_bytes(kDst);
  float2 cbs = bc2(0.0F), crs = bc2(0.0F);
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    if (kPlain || r < rows) {
      uint32_t w[kBytes];
      convert4<kSrc, kDst>(p, raw[r], w, r == 0, cbs, crs);
      store_words<kBytes, kPlain>(p.dst.data[0] + static_cast<size_t>(y0 + r) * p.dst.pitch[0] + kBytes * xs, w, whole);
    }
  }
  if constexpr (kDst == CC_NV12 || kDst == CC_NV16 || kDst == CC_I420) {
    // The mean of 2 x rows samples: the product by the count's reciprocal is exact.
    const float inv = (kPlain ? kRows : rows) == 2 ? 0.25F : 0.5F;
    const uint32_t u = codes8_of_half(exact_scale_add2(cbs, bc2(inv), bc2(0.5F)));
    const uint32_t v = codes8_of_half(exact_scale_add2(crs, bc2(inv), bc2(0.5F)));
    const int cy = y0 / kRows;
    if constexpr (kDst == CC_I420) {
      if (!kPlain && ((whole >> threadIdx.x) & 1U) == 0U) return;
      uint8_t* q[2] = {p.dst.data[1] + static_cast<size_t>(cy) * p.dst.pitch[1] + (xs >> 1),
                       p.dst.data[2] + static_cast<size_t>(cy) * p.dst.pitch[2] + (xs >> 1)};
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t c = __byte_perm(k == 0 ? u : v, 0U, 0x4420U);
        if (kPlain || (reinterpret_cast<uintptr_t>(q[k]) & 1U) == 0U) {
          *reinterpret_cast<uint16_t*>(q[k]) = static_cast<uint16_t>(c);
        } else {
          q[k][0] = static_cast<uint8_t>(c);
          q[k][1] = static_cast<uint8_t>(c >> 8);
        }
      }
    } else {
      const uint32_t w[1] = {zip8(u, v)};
      store_words<1, kPlain>(p.dst.data[1] + static_cast<size_t>(cy) * p.dst.pitch[1] + xs, w, whole);
    }
  }
}

// ---- Groups at an edge ---------------------------------------------------------

// Writes n bytes held little-endian in w to q: whole words where q is
// 4-byte aligned, bytes otherwise.
template <int kWords>
__device__ __forceinline__ void put_segment(uint8_t* q, const uint32_t (&w)[kWords], int n) {
  if ((reinterpret_cast<uintptr_t>(q) & 3U) == 0U && n == 4 * kWords) {
#pragma unroll
    for (int i = 0; i < kWords; ++i) reinterpret_cast<uint32_t*>(q)[i] = w[i];
  } else {
#pragma unroll
    for (int i = 0; i < 4 * kWords; ++i) {
      if (i < n) q[i] = static_cast<uint8_t>(w[i >> 2] >> (8 * (i & 3)));
    }
  }
}

__device__ __forceinline__ void set_byte(uint32_t* w, int i, uint32_t b) { w[i >> 2] |= b << (8 * (i & 3)); }

// One row segment of up to four destination pixels (v[0..n)) of format kDst
// at (x, y); chroma of YCbCr formats is written separately, except for the
// packed 4:2:2 ones, whose row words interleave it (cb/cr per pixel pair).
template <int kDst>
__device__ __forceinline__ void store_row4(const Image& img, int x, int y, const Px (&v)[kGroupX], int n,
                                           const uint32_t (&cb)[2], const uint32_t (&cr)[2]) {
  uint8_t* row = img.data[0] + static_cast<size_t>(y) * img.pitch[0];
  constexpr FormatInfo fi = info_of(kDst);
  constexpr int kBpp = fi.model == kYuv && fi.channels == 2 ? 2 : fi.channels * fi.bytes;
  constexpr int kWords = kBpp;  // 4 pixels x kBpp bytes = kBpp words
  uint32_t w[kWords];
#pragma unroll
  for (int i = 0; i < kWords; ++i) w[i] = 0U;
#pragma unroll
  for (int i = 0; i < kGroupX; ++i) {
    if constexpr (kDst == CC_NV12 || kDst == CC_NV16 || kDst == CC_I420 || kDst == CC_MONO8) {
      set_byte(w, i, code8(v[i].c0));
    } else if constexpr (kDst == CC_YUYV) {
      set_byte(w, 2 * i, code8(v[i].c0));
      set_byte(w, 2 * i + 1, (i & 1) ? cr[i >> 1] : cb[i >> 1]);
    } else if constexpr (kDst == CC_UYVY) {
      set_byte(w, 2 * i + 1, code8(v[i].c0));
      set_byte(w, 2 * i, (i & 1) ? cr[i >> 1] : cb[i >> 1]);
    } else if constexpr (kDst == CC_RGB8 || kDst == CC_BGR8) {
      const bool bgr = kDst == CC_BGR8;
      set_byte(w, 3 * i, code8(bgr ? v[i].c2 : v[i].c0));
      set_byte(w, 3 * i + 1, code8(v[i].c1));
      set_byte(w, 3 * i + 2, code8(bgr ? v[i].c0 : v[i].c2));
    } else if constexpr (kDst == CC_RGBA8 || kDst == CC_BGRA8) {
      const bool bgr = kDst == CC_BGRA8;
      w[i] = code8(bgr ? v[i].c2 : v[i].c0) | (code8(v[i].c1) << 8) | (code8(bgr ? v[i].c0 : v[i].c2) << 16) |
             (code8(v[i].a) << 24);
    } else if constexpr (kDst == CC_MONO16) {
      const uint32_t c = code16(v[i].c0);
      set_byte(w, 2 * i, c & 0xFFU);
      set_byte(w, 2 * i + 1, c >> 8);
    } else {
      const uint32_t r = code16(v[i].c0), g = code16(v[i].c1), b = code16(v[i].c2);
      set_byte(w, 6 * i, r & 0xFFU);
      set_byte(w, 6 * i + 1, r >> 8);
      set_byte(w, 6 * i + 2, g & 0xFFU);
      set_byte(w, 6 * i + 3, g >> 8);
      set_byte(w, 6 * i + 4, b & 0xFFU);
      set_byte(w, 6 * i + 5, b >> 8);
    }
  }
  put_segment<kWords>(row + static_cast<size_t>(x) * kBpp, w, n * kBpp);
}

// The group at column xs of rows y0 (and y0 + 1 of a 4:2:0 destination), pixel
// by pixel: partial groups, fill, and sources whose chroma starts in mid-pair.
template <int kSrc, int kDst>
__device__ __noinline__ void edge_group(const Plan& p, int xs, int y0) {
  constexpr FormatInfo fi = info_of(kDst);
  constexpr bool kYuvDst = fi.model == kYuv;
  constexpr int kRows = kYuvDst ? (1 << fi.shift_y) : 1;
  const int n = p.dst.width - xs < kGroupX ? p.dst.width - xs : kGroupX;
  float cbs[2] = {0.0F, 0.0F}, crs[2] = {0.0F, 0.0F};
  int rows = 0;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const int y = y0 + r;
    if (r > 0 && y >= p.dst.height) break;
    ++rows;
    Px v[kGroupX];
    const bool row_in = y >= p.cy0 && y < p.cy1;
#pragma unroll
    for (int i = 0; i < kGroupX; ++i) {
      const int x = xs + i;
      if (i < n && row_in && x >= p.cx0 && x < p.cx1) {
        v[i] = apply_affine(p, load_px<kSrc>(p.src, x + p.sx0 - p.cx0, y + p.sy0 - p.cy0));
      } else {
        v[i] = Px{p.fill[0], p.fill[1], p.fill[2], p.fill[3]};
      }
    }
    if constexpr (kYuvDst) {
#pragma unroll
      for (int i = 0; i < kGroupX; ++i) {
        if (i < n) {
          cbs[i >> 1] = __fadd_rn(cbs[i >> 1], v[i].c1);
          crs[i >> 1] = __fadd_rn(crs[i >> 1], v[i].c2);
        }
      }
    }
    // Chroma means: a block holds 1, 2 or 4 pixels, and a sum of these
    // samples is zero or far above the subnormals, so dividing by the count
    // (as the definition does) is exactly the product by its reciprocal.
    if constexpr (kDst == CC_YUYV || kDst == CC_UYVY) {
      // One row per block: the chroma of each pixel pair is known now.
      uint32_t cb[2], cr[2];
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float inv = n - 2 * b >= 2 ? 0.5F : 1.0F;
        cb[b] = code8(__fmul_rn(cbs[b], inv));
        cr[b] = code8(__fmul_rn(crs[b], inv));
      }
      store_row4<kDst>(p.dst, xs, y, v, n, cb, cr);
    } else {
      const uint32_t none[2] = {0U, 0U};
      store_row4<kDst>(p.dst, xs, y, v, n, none, none);
    }
  }
  if constexpr (kDst == CC_NV12 || kDst == CC_NV16 || kDst == CC_I420) {
    const int cx = xs >> 1;
    const int cy = y0 >> fi.shift_y;
    const int nb = (n + 1) >> 1;  // chroma samples in this subgroup: 1 or 2
    uint32_t code[2][2];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int cnt = (n - 2 * b >= 2 ? 2 : 1) * rows;
      const float inv = cnt == 4 ? 0.25F : (cnt == 2 ? 0.5F : 1.0F);
      code[b][0] = code8(__fmul_rn(cbs[b], inv));
      code[b][1] = code8(__fmul_rn(crs[b], inv));
    }
    if constexpr (kDst == CC_I420) {
      uint8_t* u = p.dst.data[1] + static_cast<size_t>(cy) * p.dst.pitch[1] + cx;
      uint8_t* vv = p.dst.data[2] + static_cast<size_t>(cy) * p.dst.pitch[2] + cx;
      if (nb == 2 && (reinterpret_cast<uintptr_t>(u) & 1U) == 0U && (reinterpret_cast<uintptr_t>(vv) & 1U) == 0U) {
        *reinterpret_cast<uint16_t*>(u) = static_cast<uint16_t>(code[0][0] | (code[1][0] << 8));
        *reinterpret_cast<uint16_t*>(vv) = static_cast<uint16_t>(code[0][1] | (code[1][1] << 8));
      } else {
        u[0] = static_cast<uint8_t>(code[0][0]);
        vv[0] = static_cast<uint8_t>(code[0][1]);
        if (nb == 2) {
          u[1] = static_cast<uint8_t>(code[1][0]);
          vv[1] = static_cast<uint8_t>(code[1][1]);
        }
      }
    } else {
      uint8_t* q = p.dst.data[1] + static_cast<size_t>(cy) * p.dst.pitch[1] + 2 * cx;
      const uint32_t w[1] = {code[0][0] | (code[0][1] << 8) | (code[1][0] << 16) | (code[1][1] << 24)};
      put_segment<1>(q, w, 2 * nb);
    }
  }
}

// ---- The kernel ----------------------------------------------------------------
//
// A warp converts kSub x 32 four-pixel groups of rows [gy kRows, (gy + 1) kRows);
// its lane L takes groups g0 + 32 h (h < kSub), so that every load and store
// instruction of the warp covers contiguous bytes. All of a thread's whole
// groups are read first; then each is converted and stored. groups_x =
// ceil(width / 4).
//
// What bounds it at 3840x2160 is the FP32 pipes and instruction issue: RGB8 ->
// NV12, 37.3 MB (5.8 us at the copy bandwidth), executes 28 instructions a pixel,
// 12.8 of them two-lane FP32 ones that hold both pipes two cycles each (72 % of
// the active cycles). Passes before groups were lane pairs, and now (inputs
// in L2): RGB8 -> NV12 12.1 and 10.6 us, NV12 -> RGB8 13.5 and 10.7, YUYV ->
// NV12 8.0 and 5.7; rows at any byte: 3839x2159 NV12 -> RGB8 32.7 and 17.1 us,
// 2001x1500 MONO16 -> RGB16 52.5 and 12.2. The checks come before the loads, once
// for the warp: between them they cost 10 % (12.0 against 10.7 us).
template <int kSrc, int kDst, int kSub>
__global__ void __launch_bounds__(kThreadsX* kThreadsY, kDirectBlocksPerSm)
    cc_direct_kernel(const __grid_constant__ Plan p, int groups_x, int groups_y) {
  // A programmatic dependent (launch_dependent): no memory before the wait.
  isp_b200::griddep_launch_dependents();
  isp_b200::griddep_wait();
  static_assert(kThreadsX == 32, "a warp is a row of the block");
  const int gy = static_cast<int>(blockIdx.y * blockDim.y + threadIdx.y);
  if (gy >= groups_y) return;  // whole warps
  constexpr FormatInfo fi = info_of(kDst);
  constexpr int kRows = fi.model == kYuv ? (1 << fi.shift_y) : 1;
  const int first = static_cast<int>(blockIdx.x) * kThreadsX * kSub;
  const int g0 = first + static_cast<int>(threadIdx.x);
  const int y0 = gy * kRows;
  const int rows = kRows == 2 && y0 + 1 >= p.dst.height ? 1 : kRows;
  // Source offset of destination pixel (x, y) inside the content.
  const int ox = p.sx0 - p.cx0;
  const int oy = p.sy0 - p.cy0;

  bool rows_in = !shares_chroma(kSrc) || (ox & 1) == 0;
  bool aligned = true;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    if (r < rows) {
      rows_in = rows_in && y0 + r >= p.cy0 && y0 + r < p.cy1;
      aligned = aligned && source_aligned<kSrc>(p.src, ox, y0 + r + oy);
    }
  }
  uint32_t raw[kSub][kRows][kRawWords];
  // Whole warps of whole groups in whole rows on word boundaries: no checks in between.
  const int x_last = (first + kThreadsX * kSub) * kGroupX;
  if (aligned && rows_in && rows == kRows && first * kGroupX >= p.cx0 && x_last <= p.cx1 &&
      destination_aligned<kDst>(p.dst, y0)) {
#pragma unroll
    for (int h = 0; h < kSub; ++h) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        fetch4<kSrc, false>(p.src, (g0 + kThreadsX * h) * kGroupX + ox, y0 + r + oy, raw[h][r]);
      }
    }
#pragma unroll
    for (int h = 0; h < kSub; ++h) {
      convert_group<kSrc, kDst, true>(p, raw[h], kRows, (g0 + kThreadsX * h) * kGroupX, y0, 0xFFFFFFFFU);
    }
    return;
  }
  bool ok[kSub];
#pragma unroll
  for (int h = 0; h < kSub; ++h) {
    const int xs = (g0 + kThreadsX * h) * kGroupX;
    ok[h] = rows_in && xs >= p.cx0 && xs + kGroupX <= p.cx1;
  }
  if (aligned) {
#pragma unroll
    for (int h = 0; h < kSub; ++h) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        if (ok[h] && r < rows) fetch4<kSrc, false>(p.src, (g0 + kThreadsX * h) * kGroupX + ox, y0 + r + oy, raw[h][r]);
      }
    }
  } else {
#pragma unroll
    for (int h = 0; h < kSub; ++h) {
#pragma unroll
      for (int r = 0; r < kRows; ++r) {
        if (ok[h] && r < rows) fetch4<kSrc, true>(p.src, (g0 + kThreadsX * h) * kGroupX + ox, y0 + r + oy, raw[h][r]);
      }
    }
  }
#pragma unroll
  for (int h = 0; h < kSub; ++h) {
    if (first + kThreadsX * h >= groups_x) break;  // the whole warp
    const int g = g0 + kThreadsX * h;
    const unsigned int whole = __ballot_sync(0xFFFFFFFFU, ok[h]);
    if (whole != 0U) convert_group<kSrc, kDst, false>(p, raw[h], rows, g * kGroupX, y0, whole);
    if (!ok[h] && g < groups_x) edge_group<kSrc, kDst>(p, g * kGroupX, y0);
  }
}

template <int kSrc, int kDst>
const void* direct_instance(bool wide) {
  return wide ? reinterpret_cast<const void*>(&cc_direct_kernel<kSrc, kDst, direct_subgroups(kDst, true)>)
              : reinterpret_cast<const void*>(&cc_direct_kernel<kSrc, kDst, direct_subgroups(kDst, false)>);
}

}  // namespace
}  // namespace cc_b200
