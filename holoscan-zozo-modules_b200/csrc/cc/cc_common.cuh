// cc_common.cuh - the B200 colour converter's plan and per-pixel arithmetic.
//
// One conversion is defined as in holoscan::color_convert
// (modules/color-convert/include/holoscan/color_convert/conversion.hpp:9-27,
// arithmetic in src/kernel_math.hpp:70-370):
//   1. a source pixel decodes to its format's samples (Y Cb Cr, R G B or
//      luma; chroma from the chroma sample covering the pixel; 16-bit
//      samples divided by 257; alpha 255 unless stored);
//   2. a destination pixel inside the content rectangle samples the source
//      rectangle (nearest, bilinear or area); outside it takes the fill;
//   3. the samples go through one 3x4 affine map to the destination's
//      model (none between equal models), are rounded half up and clamped;
//      a subsampled destination stores the mean chroma of its block.
// Every sum and product below is a separate IEEE single operation, in the
// reference's order (the library is compiled with --fmad=false), so the
// kernels give the reference's bytes.
#pragma once

#include <cstddef>
#include <cstdint>

#include "cc_b200.h"

#if defined(__CUDACC__)
#define CC_HD __host__ __device__ __forceinline__
#else
#define CC_HD inline
#endif

namespace cc_b200 {

enum Model : int { kYuv = 0, kRgb = 1, kGray = 2 };

struct FormatInfo {
  int model, planes, shift_x, shift_y, bytes, channels;
};

// pixel_format.hpp:58-84.
CC_HD constexpr FormatInfo info_of(int f) {
  return f == CC_NV12    ? FormatInfo{kYuv, 2, 1, 1, 1, 1}
         : f == CC_NV16  ? FormatInfo{kYuv, 2, 1, 0, 1, 1}
         : f == CC_I420  ? FormatInfo{kYuv, 3, 1, 1, 1, 1}
         : f == CC_YUYV  ? FormatInfo{kYuv, 1, 1, 0, 1, 2}
         : f == CC_UYVY  ? FormatInfo{kYuv, 1, 1, 0, 1, 2}
         : f == CC_RGB8  ? FormatInfo{kRgb, 1, 0, 0, 1, 3}
         : f == CC_BGR8  ? FormatInfo{kRgb, 1, 0, 0, 1, 3}
         : f == CC_RGBA8 ? FormatInfo{kRgb, 1, 0, 0, 1, 4}
         : f == CC_BGRA8 ? FormatInfo{kRgb, 1, 0, 0, 1, 4}
         : f == CC_MONO8 ? FormatInfo{kGray, 1, 0, 0, 1, 1}
         : f == CC_MONO16 ? FormatInfo{kGray, 1, 0, 0, 2, 1}
                          : FormatInfo{kRgb, 1, 0, 0, 2, 3};
}

struct Image {
  int format, width, height;
  uint8_t* data[3];
  size_t pitch[3];
};

// Everything one conversion needs, by value in the kernel's parameters.
struct Plan {
  Image src, dst;
  int mode;
  int sx0, sy0, sx1, sy1;  // source rectangle, inclusive bounds
  float scale_x, scale_y;  // source pixels per content pixel
  int cx0, cy0, cx1, cy1;  // content rectangle [cx0, cx1) x [cy0, cy1)
  float m[9], o[3];
  int identity;
  float fill[4];  // in the destination's model
  int bsx, bsy;   // log2 of the pixels one destination chroma sample covers
};

struct Px {
  float c0, c1, c2, a;
};

#if defined(__CUDACC__)

// Integers to floats and back without the conversion unit (a quarter of the
// FP32 rate): 2^23 + k has k in its low mantissa bits for 0 <= k < 2^23, so
// a byte b becomes the float b exactly as (2^23 + b) - 2^23, and a float c in
// [0, 2^23) becomes floor(c) as the mantissa of c + 2^23 rounded down.
constexpr uint32_t kTwo23Bits = 0x4B000000U;
constexpr float kTwo23 = 8388608.0F;

__device__ __forceinline__ float byte_f(uint32_t b) { return __fsub_rn(__uint_as_float(kTwo23Bits | b), kTwo23); }

// Byte k (0..3) of w as a float, exactly.
__device__ __forceinline__ float byte_of(uint32_t w, int k) {
  return __fsub_rn(__uint_as_float(__byte_perm(w, kTwo23Bits, 0x7650U | static_cast<uint32_t>(k))), kTwo23);
}

__device__ __forceinline__ uint32_t floor_bits(float c) { return __float_as_uint(__fadd_rd(c, kTwo23)) - kTwo23Bits; }

// code8 and code16 (below) left in the bits of 2^23 + code: the code in the
// low byte (low half-word) for packing with byte permutes.
__device__ __forceinline__ uint32_t code8_bits(float v) {
  return __float_as_uint(__fadd_rd(fminf(fmaxf(__fadd_rn(v, 0.5F), 0.0F), 255.0F), kTwo23));
}
__device__ __forceinline__ uint32_t code16_bits(float v) {
  return __float_as_uint(__fadd_rd(fminf(fmaxf(__fadd_rn(__fmul_rn(v, 257.0F), 0.5F), 0.0F), 65535.0F), kTwo23));
}
// The low bytes of a, b, c, d as one little-endian word.
__device__ __forceinline__ uint32_t pack8(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040U), __byte_perm(c, d, 0x0040U), 0x5410U);
}
// The low half-words of a and b as one little-endian word.
__device__ __forceinline__ uint32_t pack16(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x5410U); }

// Rounded half up and clamped to 0..255 (kernel_math.hpp:89-92): r =
// floor(v + 0.5) then 0 where r <= 0 and 255 where r >= 255 equals the floor
// of v + 0.5 first clamped to [0, 255].
__device__ __forceinline__ uint32_t code8(float v) {
  return floor_bits(fminf(fmaxf(__fadd_rn(v, 0.5F), 0.0F), 255.0F));
}

// 16-bit codes: the floor of v * 257 + 0.5, clamped to 0..65535 (:94-97).
__device__ __forceinline__ uint32_t code16(float v) {
  return floor_bits(fminf(fmaxf(__fadd_rn(__fmul_rn(v, 257.0F), 0.5F), 0.0F), 65535.0F));
}

// v / 257 correctly rounded for an integer 0 <= v < 2^16, as the IEEE
// division the definition uses (:99-104): the product by r = RN(1/257)
// corrected once by its exact FMA residual (Markstein's correction step),
// which gives the correctly rounded quotient for every one of the 65,536
// inputs (checked exhaustively against exact rational arithmetic, and on the
// GPU against the oracle's division).
__device__ __forceinline__ float div257(uint32_t v) {
  constexpr float kR = 1.0F / 257.0F;
  const float x = byte_f(v);  // exact for v < 2^23
  const float q = __fmul_rn(x, kR);
  const float e = __fmaf_rn(-q, 257.0F, x);
  return __fmaf_rn(e, kR, q);
}

// A 16-bit little-endian sample on the 8-bit scale, read byte-wise since a
// pitched row of 16-bit samples need not be 2-byte aligned.
__device__ __forceinline__ float word_sample(const uint8_t* p) {
  return div257(static_cast<uint32_t>(__ldg(p)) | (static_cast<uint32_t>(__ldg(p + 1)) << 8));
}

__device__ __forceinline__ const uint8_t* row_of(const Image& img, int plane, int y) {
  return img.data[plane] + static_cast<size_t>(y) * img.pitch[plane];
}

// Pixel (x, y) of a source image of format kF, in its own samples (:112-161).
template <int kF>
__device__ __forceinline__ Px load_px(const Image& img, int x, int y) {
  const uint8_t* row = row_of(img, 0, y);
  if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    const uint8_t* uv = row_of(img, 1, kF == CC_NV12 ? (y >> 1) : y) + 2 * (x >> 1);
    return {byte_f(__ldg(row + x)), byte_f(__ldg(uv)), byte_f(__ldg(uv + 1)), 255.0F};
  } else if constexpr (kF == CC_I420) {
    const int cx = x >> 1, cy = y >> 1;
    return {byte_f(__ldg(row + x)), byte_f(__ldg(row_of(img, 1, cy) + cx)), byte_f(__ldg(row_of(img, 2, cy) + cx)),
            255.0F};
  } else if constexpr (kF == CC_YUYV) {
    const uint8_t* pair = row + 4 * (x >> 1);
    return {byte_f(__ldg(pair + 2 * (x & 1))), byte_f(__ldg(pair + 1)), byte_f(__ldg(pair + 3)), 255.0F};
  } else if constexpr (kF == CC_UYVY) {
    const uint8_t* pair = row + 4 * (x >> 1);
    return {byte_f(__ldg(pair + 1 + 2 * (x & 1))), byte_f(__ldg(pair)), byte_f(__ldg(pair + 2)), 255.0F};
  } else if constexpr (kF == CC_RGB8 || kF == CC_BGR8) {
    const uint8_t* p = row + 3 * x;
    const float a = byte_f(__ldg(p)), b = byte_f(__ldg(p + 1)), c = byte_f(__ldg(p + 2));
    return kF == CC_RGB8 ? Px{a, b, c, 255.0F} : Px{c, b, a, 255.0F};
  } else if constexpr (kF == CC_RGBA8 || kF == CC_BGRA8) {
    const uint8_t* p = row + 4 * x;
    const float a = byte_f(__ldg(p)), b = byte_f(__ldg(p + 1)), c = byte_f(__ldg(p + 2));
    const float al = byte_f(__ldg(p + 3));
    return kF == CC_RGBA8 ? Px{a, b, c, al} : Px{c, b, a, al};
  } else if constexpr (kF == CC_MONO8) {
    return {byte_f(__ldg(row + x)), 0.0F, 0.0F, 255.0F};
  } else if constexpr (kF == CC_MONO16) {
    return {word_sample(row + 2 * x), 0.0F, 0.0F, 255.0F};
  } else {
    const uint8_t* p = row + 6 * x;
    return {word_sample(p), word_sample(p + 2), word_sample(p + 4), 255.0F};
  }
}

__device__ __forceinline__ bool aligned4(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3U) == 0U; }

__device__ __forceinline__ uint32_t ldw(const uint8_t* p) { return __ldg(reinterpret_cast<const uint32_t*>(p)); }

// c = m s + o on the colour samples, each row summed left to right; alpha
// passes through (:236-244).
__device__ __forceinline__ Px apply_affine(const Plan& p, Px s) {
  if (p.identity) return s;
  Px r;
  r.c0 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p.m[0], s.c0), __fmul_rn(p.m[1], s.c1)), __fmul_rn(p.m[2], s.c2)),
                   p.o[0]);
  r.c1 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p.m[3], s.c0), __fmul_rn(p.m[4], s.c1)), __fmul_rn(p.m[5], s.c2)),
                   p.o[1]);
  r.c2 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p.m[6], s.c0), __fmul_rn(p.m[7], s.c1)), __fmul_rn(p.m[8], s.c2)),
                   p.o[2]);
  r.a = s.a;
  return r;
}

__device__ __forceinline__ void put_word(uint8_t* q, uint32_t w) {
  q[0] = static_cast<uint8_t>(w & 0xFFU);
  q[1] = static_cast<uint8_t>(w >> 8);
}

// Everything but chroma of pixel (x, y) of a destination of format kF (the
// luma of a YCbCr one), :256-307.
template <int kF>
__device__ __forceinline__ void store_px(const Image& img, int x, int y, const Px& v) {
  uint8_t* row = img.data[0] + static_cast<size_t>(y) * img.pitch[0];
  if constexpr (kF == CC_NV12 || kF == CC_NV16 || kF == CC_I420 || kF == CC_MONO8) {
    row[x] = static_cast<uint8_t>(code8(v.c0));
  } else if constexpr (kF == CC_YUYV) {
    row[4 * (x >> 1) + 2 * (x & 1)] = static_cast<uint8_t>(code8(v.c0));
  } else if constexpr (kF == CC_UYVY) {
    row[4 * (x >> 1) + 1 + 2 * (x & 1)] = static_cast<uint8_t>(code8(v.c0));
  } else if constexpr (kF == CC_RGB8 || kF == CC_BGR8) {
    uint8_t* q = row + 3 * x;
    const bool bgr = kF == CC_BGR8;
    q[0] = static_cast<uint8_t>(code8(bgr ? v.c2 : v.c0));
    q[1] = static_cast<uint8_t>(code8(v.c1));
    q[2] = static_cast<uint8_t>(code8(bgr ? v.c0 : v.c2));
  } else if constexpr (kF == CC_RGBA8 || kF == CC_BGRA8) {
    const bool bgr = kF == CC_BGRA8;
    const uint32_t w = code8(bgr ? v.c2 : v.c0) | (code8(v.c1) << 8) | (code8(bgr ? v.c0 : v.c2) << 16) |
                       (code8(v.a) << 24);
    uint8_t* q = row + 4 * x;
    if ((reinterpret_cast<uintptr_t>(q) & 3U) == 0U) {
      *reinterpret_cast<uint32_t*>(q) = w;
    } else {
      q[0] = static_cast<uint8_t>(w);
      q[1] = static_cast<uint8_t>(w >> 8);
      q[2] = static_cast<uint8_t>(w >> 16);
      q[3] = static_cast<uint8_t>(w >> 24);
    }
  } else if constexpr (kF == CC_MONO16) {
    put_word(row + 2 * x, code16(v.c0));
  } else {
    uint8_t* q = row + 6 * x;
    put_word(q, code16(v.c0));
    put_word(q + 2, code16(v.c1));
    put_word(q + 4, code16(v.c2));
  }
}

// Chroma sample (cx, cy) of a YCbCr destination (:311-341).
template <int kF>
__device__ __forceinline__ void store_chroma(const Image& img, int cx, int cy, float cb, float cr) {
  if constexpr (kF == CC_NV12 || kF == CC_NV16) {
    uint8_t* q = img.data[1] + static_cast<size_t>(cy) * img.pitch[1] + 2 * cx;
    q[0] = static_cast<uint8_t>(code8(cb));
    q[1] = static_cast<uint8_t>(code8(cr));
  } else if constexpr (kF == CC_I420) {
    img.data[1][static_cast<size_t>(cy) * img.pitch[1] + cx] = static_cast<uint8_t>(code8(cb));
    img.data[2][static_cast<size_t>(cy) * img.pitch[2] + cx] = static_cast<uint8_t>(code8(cr));
  } else if constexpr (kF == CC_YUYV) {
    uint8_t* q = img.data[0] + static_cast<size_t>(cy) * img.pitch[0] + 4 * cx;
    q[1] = static_cast<uint8_t>(code8(cb));
    q[3] = static_cast<uint8_t>(code8(cr));
  } else if constexpr (kF == CC_UYVY) {
    uint8_t* q = img.data[0] + static_cast<size_t>(cy) * img.pitch[0] + 4 * cx;
    q[0] = static_cast<uint8_t>(code8(cb));
    q[2] = static_cast<uint8_t>(code8(cr));
  }
}

#endif  // __CUDACC__

// Host side (cc_plan.cpp): names, geometry, checks and the plan.
int make_plan(const cc_image_c* src, const cc_image_c* dst, const cc_params_c* params, Plan* plan);
int compute_mapping(int sw, int sh, int w, int h, int dst_format, const cc_params_c* params, cc_mapping_c* out);
int validate(const cc_image_c* src, const cc_image_c* dst, const cc_params_c* params);
bool known_format(int f);

// Kernel launchers (cc_kernels*.cu).
int launch_convert(const Plan& plan, void* stream);
int launch_pattern(uint8_t* data, size_t pitch, int width, int height, uint32_t frame, void* stream);

}  // namespace cc_b200
