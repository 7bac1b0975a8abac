// cc_kernels.cuh - the colour converter's kernels.
//
// Direct path (source and content the same size on both axes, which is every
// plain format conversion): whatever the resize mode, each destination pixel
// then reads exactly the one source pixel under it (bilinear and area
// weights are exactly 1 and 0 there), so a thread converts groups of four
// pixels across (two rows of them for a 4:2:0 destination: two whole chroma
// blocks) with both formats known at compile time, in whole words whatever the
// rows' alignment (cc_direct.cuh).
//
// Resample path: a thread samples four destination pixels of a row (of two rows
// into 4:2:0 formats: two whole chroma blocks), two at a time in the lanes of
// f32x2 instructions, the source format and resize mode known at compile time,
// the destination's stores chosen at run time (cc_resample.cuh).
#pragma once

#include "../isp_ops.cuh"
#include "cc_common.cuh"

namespace cc_b200 {

constexpr int kGroupX = 4;     // pixels across per direct-path thread
constexpr int kThreadsX = 32;  // CTA shape for both paths
constexpr int kThreadsY = 8;
// Five 256-thread CTAs of the direct path per SM (at most 48 registers a
// thread): at four, a 4K frame's 2,025 CTAs ran 3.42 waves, the last 42 % full.
constexpr int kDirectBlocksPerSm = 5;
constexpr int kSms = 148;  // of a B200: a matter of balance only

// The colour map of two pixels at once: the nine products two lanes at a
// time (mul.rn.f32x2, each lane rounded as the scalar product), every sum in
// the definition's order; a two-lane product never feeds a plain two-lane
// sum, which the assembler could fuse into one rounding (psum2).
__device__ __forceinline__ void affine_pair(const Plan& p, Px& a, Px& b) {
  using isp_b200::add2;
  using isp_b200::bc2;
  using isp_b200::mul2;
  using isp_b200::psum2;
  const float2 s0 = make_float2(a.c0, b.c0), s1 = make_float2(a.c1, b.c1), s2 = make_float2(a.c2, b.c2);
  float2 out[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 t0 = mul2(bc2(p.m[3 * k]), s0);
    const float2 t1 = mul2(bc2(p.m[3 * k + 1]), s1);
    const float2 t2 = mul2(bc2(p.m[3 * k + 2]), s2);
    out[k] = add2(psum2(t2, psum2(t0, t1)), bc2(p.o[k]));
  }
  a.c0 = out[0].x;
  b.c0 = out[0].y;
  a.c1 = out[1].x;
  b.c1 = out[1].y;
  a.c2 = out[2].x;
  b.c2 = out[2].y;
}

// code8_bits of two values: the + 0.5 and the add of 2^23 rounded toward
// zero (equal to rounding down, the value being clamped to [0, 255]) two
// lanes at a time, the clamps per lane. Neither add consumes a product, so
// nothing can be fused into it.
__device__ __forceinline__ uint2 code8_bits2(float a, float b) {
  using isp_b200::add2;
  using isp_b200::add2_rz;
  using isp_b200::bc2;
  const float2 h = add2(make_float2(a, b), bc2(0.5F));
  const float2 c = make_float2(fminf(fmaxf(h.x, 0.0F), 255.0F), fminf(fmaxf(h.y, 0.0F), 255.0F));
  const float2 r = add2_rz(c, bc2(kTwo23));
  return make_uint2(__float_as_uint(r.x), __float_as_uint(r.y));
}

// One four-pixel row segment of format kDst at (x, y) from whole, aligned
// groups: every word of it stored, the row start known to be 4-byte aligned.
// Codes come as their 2^23-biased bits (code8_bits / code16_bits); cb and cr
// are the pair chroma of the packed 4:2:2 formats.
template <int kDst>
__device__ __forceinline__ void store_full4(const Image& img, int x, int y, const Px (&v)[kGroupX],
                                            const uint32_t (&cb)[2], const uint32_t (&cr)[2]) {
  uint8_t* row = img.data[0] + static_cast<size_t>(y) * img.pitch[0];
  if constexpr (kDst == CC_NV12 || kDst == CC_NV16 || kDst == CC_I420 || kDst == CC_MONO8) {
    const uint2 a = code8_bits2(v[0].c0, v[1].c0), b = code8_bits2(v[2].c0, v[3].c0);
    *reinterpret_cast<uint32_t*>(row + x) = pack8(a.x, a.y, b.x, b.y);
  } else if constexpr (kDst == CC_YUYV || kDst == CC_UYVY) {
    uint32_t* q = reinterpret_cast<uint32_t*>(row + 2 * x);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint2 yy = code8_bits2(v[2 * k].c0, v[2 * k + 1].c0);
      q[k] = kDst == CC_YUYV ? pack8(yy.x, cb[k], yy.y, cr[k]) : pack8(cb[k], yy.x, cr[k], yy.y);
    }
  } else if constexpr (kDst == CC_RGB8 || kDst == CC_BGR8) {
    const bool bgr = kDst == CC_BGR8;
    uint32_t b[12];
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      const uint2 r = code8_bits2(bgr ? v[i].c2 : v[i].c0, bgr ? v[i + 1].c2 : v[i + 1].c0);
      const uint2 g = code8_bits2(v[i].c1, v[i + 1].c1);
      const uint2 bl = code8_bits2(bgr ? v[i].c0 : v[i].c2, bgr ? v[i + 1].c0 : v[i + 1].c2);
      b[3 * i] = r.x;
      b[3 * i + 1] = g.x;
      b[3 * i + 2] = bl.x;
      b[3 * i + 3] = r.y;
      b[3 * i + 4] = g.y;
      b[3 * i + 5] = bl.y;
    }
    uint32_t* q = reinterpret_cast<uint32_t*>(row + 3 * x);
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = pack8(b[4 * k], b[4 * k + 1], b[4 * k + 2], b[4 * k + 3]);
  } else if constexpr (kDst == CC_RGBA8 || kDst == CC_BGRA8) {
    const bool bgr = kDst == CC_BGRA8;
    uint32_t* q = reinterpret_cast<uint32_t*>(row + 4 * x);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
      const uint2 r = code8_bits2(bgr ? v[i].c2 : v[i].c0, bgr ? v[i + 1].c2 : v[i + 1].c0);
      const uint2 g = code8_bits2(v[i].c1, v[i + 1].c1);
      const uint2 bl = code8_bits2(bgr ? v[i].c0 : v[i].c2, bgr ? v[i + 1].c0 : v[i + 1].c2);
      const uint2 al = code8_bits2(v[i].a, v[i + 1].a);
      q[i] = pack8(r.x, g.x, bl.x, al.x);
      q[i + 1] = pack8(r.y, g.y, bl.y, al.y);
    }
  } else if constexpr (kDst == CC_MONO16) {
    uint32_t* q = reinterpret_cast<uint32_t*>(row + 2 * x);
    q[0] = pack16(code16_bits(v[0].c0), code16_bits(v[1].c0));
    q[1] = pack16(code16_bits(v[2].c0), code16_bits(v[3].c0));
  } else {
    uint32_t h[12];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      h[3 * i] = code16_bits(v[i].c0);
      h[3 * i + 1] = code16_bits(v[i].c1);
      h[3 * i + 2] = code16_bits(v[i].c2);
    }
    uint32_t* q = reinterpret_cast<uint32_t*>(row + 6 * x);
#pragma unroll
    for (int k = 0; k < 6; ++k) q[k] = pack16(h[2 * k], h[2 * k + 1]);
  }
}

// Four-pixel subgroups a direct-path thread takes across (half as many for a
// 4:2:0 destination, whose thread also takes two rows). Large images take
// twice as many a thread, less setup for each, RGBA destinations apart, whose
// four words a group leave no registers for it; others keep more and shorter
// threads, since one wave or less of blocks lasts as long as its longest
// thread. Passes at two / one sizes: 3840x2160 YUYV -> NV12 6.0 / 7.1 us, NV12 ->
// NV16 7.4 / 7.9 us, RGB8 -> BGRA8 9.2 / 8.5 us, 669x668 I420 -> BGR8 4.9 / 3.9 us,
// 641x480 RGB8 -> I420 4.8 / 3.7 us.
__host__ __device__ constexpr int direct_subgroups(int dst, bool wide) {
  return dst == CC_RGBA8 || dst == CC_BGRA8 ? 2 : (dst == CC_NV12 || dst == CC_I420 ? 1 : 2) * (wide ? 2 : 1);
}

// Each source format's direct kernels (cc_direct_*.cu): a kernel pointer or null.
const void* direct_kernel(int src, int dst, bool wide);
const void* direct_kernel_yuv(int src, int dst, bool wide);
const void* direct_kernel_rgb(int src, int dst, bool wide);
const void* direct_kernel_gray(int src, int dst, bool wide);

}  // namespace cc_b200
