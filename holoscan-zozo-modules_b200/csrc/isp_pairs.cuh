// isp_pairs.cuh - the three phases of the fused tile pass on paired pixels.
//
// A 64x64 tile is processed as 64 rows of 32 pixel pairs: pair c of a row
// holds columns c and c + 32, which have the same Bayer colour, so one f32x2
// instruction advances both through identical IEEE operations (isp_ops.cuh).
// Shared memory keeps samples and RGB values as float2 pairs
// {v(c), v(c + 32)}; a neighbour of a pair is the neighbouring pair, loaded
// as one aligned 8- or 16-byte element.
//
//   A. samples: unpack the raw box, black level, lens shading, white balance
//      and clip (preprocess, isp_math.hpp:144-155) into the paired sample
//      plane P[kSH][kPW]: pair s holds samples s and s + 32 of the tile's
//      72 (image columns x0 - 4 + s);
//   B. (sharpening) demosaic every pixel of the tile and its one-pixel ring
//      into the paired RGB planes R, G, B [66][kCW2]: pair q holds pixels
//      q - 1 and q + 31 (isp_math.hpp:161-214; the ring outside the image is
//      the reference's virtual pixels, cpu_pipeline.cpp:22-46);
//   C. per unit of four pairs of one row: demosaic (or sharpen,
//      isp_math.hpp:219-227), colour matrix, statistics sums, tone, store and
//      histogram codes (isp_math.hpp:229-305).
//
// What bounds the pass is the shared-memory pipe: ncu counts 48 wavefronts per
// 32 pixels of a sharpened 3840x2160 RAW10 frame, 70 % of the pipe while the SMs
// work (issue slots 57 %, FMA pipe 46 %); 17 of them are bank conflicts of the
// tone table's lookups and the histogram's atomics, whose addresses the data
// decides. So the phases are shaped to touch shared memory less (A keeps its table
// rows in registers, B's units are six rows high; 57 wavefronts and 75 % before),
// and sums of products run two lanes at a time (isp_ops.cuh). The frame's pass
// went from 101.0 to 91.9 us with these, a 1920x1080 16-bit one with the same
// stages from 43.3 to 38.8 us.
#pragma once

#include "isp_common.cuh"

namespace isp_b200 {
namespace {

constexpr int kUnitsA = kPW / 4;  // phase A units per sample row: 4 pairs each

// Bank spread of the sample plane. Pair s of sample row j sits at
// j * kPW + (s ^ psw(j)): rows 2k and 2k + 1 keep their order, rows 2k + 2
// and 2k + 3 swap neighbouring 16-byte chunks, so that a quarter-warp
// reading four groups of row r and four of row r + 2 (same Bayer parity)
// meets every bank once. Accesses are whole 16-byte chunks (even s).
__device__ __forceinline__ int psw(int j) { return ((j >> 1) & 1) << 1; }

// Bank spread of the RGB planes (rows of 17 16-byte chunks): chunk c < 16 of
// row j sits at j * 17 + (c ^ csw(j)), rows 2k and 2k + 1 in order, rows
// 2k + 2 and 2k + 3 with neighbouring chunks swapped (chunk 16, the ring,
// stays), so that a quarter-warp reading four groups of each of two row
// pairs (rows r + a and r + 2 + a) meets every bank once but for chunk 16.
__device__ __forceinline__ int csw(int j) { return (j >> 1) & 1; }
__device__ __forceinline__ int cchunk(int c, int sw) { return c < kCW2 / 2 - 1 ? c ^ sw : c; }

__device__ __forceinline__ float4 lds4(Span<const float2> p) { return *span_cast<const float4>(p); }
__device__ __forceinline__ void sts4(Span<float2> p, float2 a, float2 b) {
  *span_cast<float4>(p) = make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// A. Samples of the tile and its halo as pairs; returns the saturated count
//    of the tile's own samples (raw >= white, isp_math.hpp:316), each counted
//    once.
//
//    A thread takes one unit of four pairs across and kRowsEach rows of one
//    parity, two apart: the row parity's constants, and the two rows of the
//    lens shading table that these rows lie between, stay in registers (with
//    one row per unit the table's four loads per eight samples were the
//    phase's largest share of shared-memory traffic). The two 16-byte halves
//    of a unit go to shared memory in an order that alternates every four
//    lanes (`flip`), so that a quarter-warp's stores and table loads, 32
//    bytes apart, meet every bank once.
//
//    One body serves every raw format and every tile: the unpacking branches
//    on the format, and only the units of an edge tile whose columns reach
//    past the image are unpacked sample by sample. (One copy per format, tile
//    kind and shading kept what they share alive across all of them and
//    spilled, and the batch kernel, whose CTAs mix formats, waited for
//    instructions.)
template <int kHalo, int kTileH>
__device__ __forceinline__ unsigned int phase_a2(const FrameDesc& p, const TileCtx& t, Span<float2> P, int box_bytes,
                                                 Span<const float2> quad, bool want_stats, bool interior) {
  constexpr int kSH = kTileH + 2 * kHalo;
  constexpr int kGroups = kThreads / kUnitsA / 2;  // groups of rows of each parity
  constexpr int kRowsEach = (kSH / 2 + kGroups - 1) / kGroups;
  const int tid = threadIdx.x;
  const int q = tid / kUnitsA;
  const int u = tid - q * kUnitsA;
  const int par = q & 1;  // row parity: y0 - halo is even
  const int first = 2 * (q >> 1) * kRowsEach + par;
  const int flip = ((tid >> 2) & 1) * 2;
  const int fmt = p.raw_format;
  const unsigned int white = static_cast<unsigned int>(p.white);
  unsigned int saturated = 0;
  if (q >= 2 * kGroups) return saturated;
  // The rows' two quad positions' constants.
  const float2 black = quad[par], inv = quad[2 + par], gain = quad[4 + par];
  const int pl = p.lsc_channels == 4 ? par : 0;
  // The unit's left and right columns: unpacked as they lie in the box when
  // inside the image, or when the tile has no use for them (further right
  // than any mirrored neighbour); one by one from their mirrored columns else.
  const int xl = t.x0 - 4 + 4 * u;
  const int xr = xl + kHalf;
  const bool plain_l = interior || (xl >= 0 && xl + 4 <= p.width) || xl > p.width + 3;
  const bool plain_r = interior || xr + 4 <= p.width || xr > p.width + 3;
  int cell = -1;           // the table row that top and step were read for
  float2 top[4], step[4];  // T[k] and T[k + 1] - T[k] of the unit's pairs, in the unit's (flipped) order
#pragma unroll 1
  for (int i = 0; i < kRowsEach; ++i) {
    const int j = first + 2 * i;
    if (j >= kSH) break;
    unsigned int wl[2], wr[2];  // samples 4u + k and 4u + 32 + k, as 16-bit halves
    Span<const uint8_t> row = t.box + (interior ? j : t.row_my[j] - (t.y0 - kHalo)) * box_bytes;
    if (plain_l) {
      unpack4(fmt, row, u, wl);
    } else {
      const uint2 e = unpack_edge4(fmt, row, t.col_mx + 4 * u, t.x0);
      wl[0] = e.x;
      wl[1] = e.y;
    }
    if (plain_r) {
      unpack4(fmt, row, u + kHalf / 4, wr);
    } else {
      const uint2 e = unpack_edge4(fmt, row, t.col_mx + 4 * u + kHalf, t.x0);
      wr[0] = e.x;
      wr[1] = e.y;
    }
    // Tile samples are s = 4 .. 67: the left lanes of units 1..8 hold 4..35,
    // their right lanes 36..67. Saturated samples are rare: one maximum over
    // the unit's eight samples decides whether any is counted.
    if (want_stats && any_half_at_least(__vmaxu2(__vmaxu2(wl[0], wl[1]), __vmaxu2(wr[0], wr[1])), white)) {
      if (j >= kHalo && j < kHalo + kTileH && u >= 1 && u <= kHalf / 4 && t.y0 + j - kHalo < p.height) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned int l = (wl[k >> 1] >> (16 * (k & 1))) & 0xFFFFU, r = (wr[k >> 1] >> (16 * (k & 1))) & 0xFFFFU;
          saturated += (xl + k < p.width && l >= white) ? 1U : 0U;
          saturated += (xr + k < p.width && r >= white) ? 1U : 0U;
        }
      }
    }
    // The halves in the order they are stored.
    const unsigned int al = flip ? wl[1] : wl[0], bl = flip ? wl[0] : wl[1];
    const unsigned int ar = flip ? wr[1] : wr[0], br = flip ? wr[0] : wr[1];
    // linearize (isp_math.hpp:144-148): (raw - black) * inv_range, without its
    // maximum with 0: all gains are positive, so a negative value stays
    // negative up to the saturating multiply below, which makes it the 0 that
    // the maximum would have made it.
    float2 v[4] = {magic_to_float2(magic_low(al), magic_low(ar)), magic_to_float2(magic_high(al), magic_high(ar)),
                   magic_to_float2(magic_low(bl), magic_low(br)), magic_to_float2(magic_high(bl), magic_high(br))};
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = mul2(sub2(v[k], bc2((k & 1) ? black.y : black.x)), bc2((k & 1) ? inv.y : inv.x));
    if (t.lt.rows > 0) {
      if (t.lt.rows <= kLscTableRows) {
        const int kk = t.row_k[j];
        if (kk != cell) {
          cell = kk;
          Span<const float2> r0 = t.table + (kk * 2 + pl) * kPW + 4 * u;
          Span<const float2> r1 = r0 + 2 * kPW;
          const float4 a0 = lds4(r0 + flip), b0 = lds4(r0 + (flip ^ 2)), a1 = lds4(r1 + flip), b1 = lds4(r1 + (flip ^ 2));
          top[0] = lo2(a0);
          top[1] = hi2(a0);
          top[2] = lo2(b0);
          top[3] = hi2(b0);
          step[0] = sub2(lo2(a1), top[0]);
          step[1] = sub2(hi2(a1), top[1]);
          step[2] = sub2(lo2(b1), top[2]);
          step[3] = sub2(hi2(b1), top[3]);
        }
        const float2 ty = bc2(t.row_ty[j]);
        // top + (bottom - top) * ty (isp_math.hpp:121-140).
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = mul2(v[k], psum2(mul2(step[k], ty), top[k]));
      } else {
        // A grid too dense for the table: each gain from the grid.
        const LscGrid g{t.grid, p.lsc_width, p.lsc_height, p.lsc_channels, p.lsc_sx, p.lsc_sy};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int ch = cfa_of(p.pattern, (par << 1) | (k & 1));
          const int s = 4 * u + (k ^ flip);
          v[k].x = fmul(v[k].x, lens_shading_gain_outline(g, t.col_mx[s], t.row_my[j], ch));
          v[k].y = fmul(v[k].y, lens_shading_gain_outline(g, t.col_mx[s + kHalf], t.row_my[j], ch));
        }
      }
    }
    // White balance and the clip to [0, 1]: the saturating multiply.
    Span<float2> dst = P + j * kPW;
    const int sw = psw(j) ^ flip;
    sts4(dst + ((4 * u) ^ sw), mul_sat2(v[0], bc2(gain.x)), mul_sat2(v[1], bc2(gain.y)));
    sts4(dst + ((4 * u + 2) ^ sw), mul_sat2(v[2], bc2(gain.x)), mul_sat2(v[3], bc2(gain.y)));
  }
  return saturated;
}

// B. (Sharpening) RGB of the tile and its ring into the paired planes, in
//    units of kRows rows x 2 pairs: 17 units across cover the 34 pairs, and
//    kRows divides the kTileH + 2 rows.
//    RGB pair (row cr, column q): pixels (q - 1, q + 31) of image row
//    y0 - 1 + cr, whose sample pair is P[cr + 3][q + 3] (halo 4).
//    With swap_rb the demosaic's red and blue go to the other planes: the
//    demosaic runs as the layout's canonical pattern (RGGB or GRBG), and
//    BGGR and GBRG trade red and blue.
//    The kernel's limit is the shared-memory pipe, so a unit is as high as
//    the block's threads allow: of 66 rows, 11 units of 6 (32 loads for 12
//    pairs, one round of 187 threads) instead of 33 of 2 (16 for 4 pairs,
//    three rounds). The unit's rows run one after the other through a window
//    of five sample rows that the unrolled loop keeps in registers.
template <bool kMalvar, int kPat, int kTileH>
__device__ __forceinline__ void phase_b2(Span<const float2> P, Span<float2> R, Span<float2> G, Span<float2> B) {
  constexpr int kUnitsQ = kCW2 / 2;  // 17
  constexpr int kRows = (kTileH + 2) % 6 == 0 ? 6 : 2;
  constexpr int kUnits = (kTileH + 2) / kRows * kUnitsQ;
  static_assert((kTileH + 2) % kRows == 0 && kRows % 2 == 0, "whole units, each starting at an odd image row");
  for (int unit = threadIdx.x; unit < kUnits; unit += kThreads) {
    const int ur = unit / kUnitsQ;
    const int uq = unit - ur * kUnitsQ;
    // Window row a holds P[kRows ur + 1 + a][2uq + 1 + b], b = 0 .. 5. As a
    // pixel row's own row all six columns are needed, as a neighbour only
    // columns 1 .. 4 (bilinear needs those alone, and no rows two away).
    float2 w[kRows + 4][6];
    const int base = kRows * ur + 1;
#pragma unroll
    for (int a = 0; a < kRows + 4; ++a) {
      if (!kMalvar && (a == 0 || a == kRows + 3)) continue;
      const int j = base + a;
      Span<const float2> row = P + j * kPW;  // pair 2uq is w column -1
      const int sw = psw(j);
      const float4 m1 = lds4(row + ((2 * uq + 2) ^ sw)), m2 = lds4(row + ((2 * uq + 4) ^ sw));  // w columns 1..4
      w[a][1] = lo2(m1);
      w[a][2] = hi2(m1);
      w[a][3] = lo2(m2);
      w[a][4] = hi2(m2);
      if (kMalvar && a >= 2 && a < kRows + 2) {
        w[a][0] = hi2(lds4(row + ((2 * uq) ^ sw)));
        w[a][5] = lo2(lds4(row + ((2 * uq + 6) ^ sw)));
      }
      // Pixel row dy needs window rows dy .. dy + 4 (bilinear: dy + 1 .. dy + 3).
      const int dy = kMalvar ? a - 4 : a - 3;
      if (dy < 0 || dy >= kRows) continue;
      float2 rgb[2][3];
#pragma unroll
      for (int dq = 0; dq < 2; ++dq) {
        float2 n[5][5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {
#pragma unroll
          for (int b = 0; b < 5; ++b) {
            // Taps outside the demosaic's support are never read.
            const bool used = kMalvar ? (c == 2 || (b > 0 && b < 4 && (c != 0 && c != 4)) || b == 2)
                                      : (c > 0 && c < 4 && b > 0 && b < 4);
            n[c][b] = used ? w[dy + c][dq + b] : make_float2(0.0F, 0.0F);
          }
        }
        // Pixel row y0 - 1 + kRows ur + dy, column x0 + 2uq + dq - 1: parities (dy + 1) & 1 and (dq + 1) & 1.
        demosaic2<kMalvar>(n, cfa_of(kPat, (((dy + 1) & 1) << 1) | ((dq + 1) & 1)), rgb[dq]);
      }
      const int cr = kRows * ur + dy;
      const int o = cr * kCW2 + 2 * cchunk(uq, csw(cr));
      sts4(R + o, rgb[0][0], rgb[1][0]);
      sts4(G + o, rgb[0][1], rgb[1][1]);
      sts4(B + o, rgb[0][2], rgb[1][2]);
    }
  }
}

// C (sharpening). The 3x3 windows of one plane around pairs 4uc .. 4uc + 3
// of output rows r and r + 1, sharpened: RGB rows r .. r + 3 (each loaded
// once for both output rows), pair columns 4uc .. 4uc + 5 (chunks 2uc ..
// 2uc + 2, stored at chunk ^ csw(row)).
__device__ __forceinline__ void sharpen_rows2(Span<const float2> X, int r, int uc, float2 amount, float2 (&o0)[4],
                                              float2 (&o1)[4]) {
  float2 w[4][6];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int j = r + a;
    const int s = csw(j);
    Span<const float2> row = X + j * kCW2;
    const float4 v0 = lds4(row + 2 * ((2 * uc) ^ s)), v1 = lds4(row + 2 * ((2 * uc + 1) ^ s)),
                 v2 = lds4(row + 2 * cchunk(2 * uc + 2, s));
    w[a][0] = lo2(v0);
    w[a][1] = hi2(v0);
    w[a][2] = lo2(v1);
    w[a][3] = hi2(v1);
    w[a][4] = lo2(v2);
    w[a][5] = hi2(v2);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o0[i] = sharpen_one2(w[1][i + 1], w[0][i + 1], w[2][i + 1], w[1][i], w[1][i + 2], w[0][i], w[0][i + 2], w[2][i],
                         w[2][i + 2], amount);
    o1[i] = sharpen_one2(w[2][i + 1], w[1][i + 1], w[3][i + 1], w[2][i], w[2][i + 2], w[1][i], w[1][i + 2], w[3][i],
                         w[3][i + 2], amount);
  }
}

// C (sharpening), one output row: the 3x3 windows of one plane around pairs
// 4uc .. 4uc + 3 of output row r, sharpened from RGB rows r .. r + 2 (loaded
// as in sharpen_rows2; a quarter-warp takes rows r and r + 2, which csw
// sends to different banks).
__device__ __forceinline__ void sharpen_row1(Span<const float2> X, int r, int uc, float2 amount, float2 (&o)[4]) {
  float2 w[3][6];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int j = r + a;
    const int s = csw(j);
    Span<const float2> row = X + j * kCW2;
    const float4 v0 = lds4(row + 2 * ((2 * uc) ^ s)), v1 = lds4(row + 2 * ((2 * uc + 1) ^ s)),
                 v2 = lds4(row + 2 * cchunk(2 * uc + 2, s));
    w[a][0] = lo2(v0);
    w[a][1] = hi2(v0);
    w[a][2] = lo2(v1);
    w[a][3] = hi2(v1);
    w[a][4] = lo2(v2);
    w[a][5] = hi2(v2);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    o[i] = sharpen_one2(w[1][i + 1], w[0][i + 1], w[2][i + 1], w[1][i], w[1][i + 2], w[0][i], w[0][i + 2], w[2][i],
                        w[2][i + 2], amount);
  }
}

// C (no sharpening). Demosaic pairs 4uc .. 4uc + 3 of output row r straight
// from the samples: sample rows r .. r + 4 (halo 2), pair columns 4uc + 2 ..
// 4uc + 9. kRowPar: the parity of the output row.
template <bool kMalvar, int kPat, int kRowPar>
__device__ __forceinline__ void demosaic_row4(Span<const float2> P, int r, int uc, float2 (&rgb)[4][3]) {
  float2 w[5][8] = {};
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    Span<const float2> row = P + (r + a) * kPW;
    const int sw = psw(r + a);
    const int s0 = 4 * uc + 2;
    const bool edge = a == 0 || a == 4;
    if (edge && !kMalvar) continue;
    if (edge) {  // Malvar's vertical taps: the centres only
      const float4 v1 = lds4(row + ((s0 + 2) ^ sw)), v2 = lds4(row + ((s0 + 4) ^ sw));
      w[a][2] = lo2(v1);
      w[a][3] = hi2(v1);
      w[a][4] = lo2(v2);
      w[a][5] = hi2(v2);
    } else {
      const float4 v0 = lds4(row + (s0 ^ sw)), v1 = lds4(row + ((s0 + 2) ^ sw)), v2 = lds4(row + ((s0 + 4) ^ sw)),
                   v3 = lds4(row + ((s0 + 6) ^ sw));
      w[a][0] = lo2(v0);
      w[a][1] = hi2(v0);
      w[a][2] = lo2(v1);
      w[a][3] = hi2(v1);
      w[a][4] = lo2(v2);
      w[a][5] = hi2(v2);
      w[a][6] = lo2(v3);
      w[a][7] = hi2(v3);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 n[5][5];
#pragma unroll
    for (int a = 0; a < 5; ++a) {
#pragma unroll
      for (int b = 0; b < 5; ++b) n[a][b] = w[a][i + b];
    }
    demosaic2<kMalvar>(n, cfa_of(kPat, (kRowPar << 1) | (i & 1)), rgb[i]);
  }
}

// ---- C: colour matrix, statistics, tone, codes, stores ---------------------

// The tone curve (isp_math.hpp:235-243) of one value from a table of
// (lut[i], lut[i+1] - lut[i]) pairs: lut[i] + (f - i) * diff[i] with
// f = x (N - 1) and i = trunc(f), given f's 2^23 + trunc(f) and f - i. The
// last entry's difference is -0.0, so x = 1 (t = +0) returns lut[N-1]
// exactly, as the reference's branch does, whatever the sign of lut[N-1].
template <bool kLutSmem>
__device__ __forceinline__ float tone_lookup(Span<const float2> table, float m, float frac) {
  float2 e;
#ifdef ISP_CHECKED
  // Entry trunc(f) through the checked span.
  e = table[static_cast<int>(__float_as_uint(m) - kTwo23Bits)];
#else
  if constexpr (kLutSmem) {
    // Shared address of entry trunc(f): base + 8 (bits - 2^23 bits), wrapping.
    const uint32_t addr = smem_u32(table) + (__float_as_uint(m) << 3) - (kTwo23Bits << 3);
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(e.x), "=f"(e.y) : "r"(addr));
  } else {
    e = __ldg(table + magic_int(m));
  }
#endif
  return fadd(e.x, fmul(frac, e.y));
}

// Adds one to bin `index - bias` of the block's histogram channel `channel`.
__device__ __forceinline__ void count_code(Span<unsigned int> hist, int channel, unsigned int index, unsigned int bias) {
#ifdef ISP_CHECKED
  atomicAdd(&hist[channel * kHistBins + static_cast<int>(index - bias)], 1U);
#else
  // The shared address, the bias folded into its base (mod 2^32).
  const uint32_t addr = smem_u32(hist) + 4U * channel * kHistBins - 4U * bias + 4U * index;
  asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
#endif
}

// The luma code (2126 r + 7152 g + 722 b + 5000) / 10000 (isp_math.hpp:303-305)
// of codes that carry `bias` each, as the top byte of one 32-bit sum: the
// weights in units of 2^-24 and an offset a little above one half, which gives
// the quotient for all 2^24 triples of codes (checked exhaustively) without
// the division's wide multiply and without taking the bias off the codes.
__device__ __forceinline__ unsigned int luma_of(unsigned int r, unsigned int g, unsigned int b, unsigned int bias) {
  constexpr unsigned int kR = 3566836U, kG = 11999065U, kB = 1211315U, kOffset = 8389408U;
  return (kR * r + kG * g + kB * b + (kOffset - (kR + kG + kB) * bias)) >> 24;
}

// Stores four pixels of one row, x .. x + 3 (isp_math.hpp:250-276), from
// their toned values t, their rounded integer codes c (2^23 + code as float
// bits: 8-bit codes for RGB8/RGBA8, 16-bit values for RGB16) and counts their
// 8-bit histogram codes (isp_math.hpp:279-305). `n`: pixels inside the image.
template <int kOut>
__device__ __forceinline__ void store_seg4(const FrameDesc& p, int x, int y, const float (&t)[4][3],
                                           const unsigned int (&c)[4][3], int n, bool want_hist, Span<unsigned int> hist) {
  Span<uint8_t> row = p.out + static_cast<int64_t>(y) * p.out_pitch;
  // Whole words where this row allows them: x is a multiple of four pixels, so
  // the row's own alignment decides.
  constexpr unsigned int kAlign = kOut == kOutRgb8 ? 4U : kOut == kOutRgb16 ? 8U : 16U;
  const bool vec = n == 4 && (static_cast<unsigned int>(reinterpret_cast<uintptr_t>(span_ptr(row))) & (kAlign - 1U)) == 0U;
  if constexpr (kOut == kOutRgb8 || kOut == kOutRgba8) {
    if constexpr (kOut == kOutRgb8) {
      if (vec) {
        Span<unsigned int> o = span_cast<unsigned int>(row + 3 * x);
        o[0] = __byte_perm(__byte_perm(c[0][0], c[0][1], 0x0040), __byte_perm(c[0][2], c[1][0], 0x0040), 0x5410);
        o[1] = __byte_perm(__byte_perm(c[1][1], c[1][2], 0x0040), __byte_perm(c[2][0], c[2][1], 0x0040), 0x5410);
        o[2] = __byte_perm(__byte_perm(c[2][2], c[3][0], 0x0040), __byte_perm(c[3][1], c[3][2], 0x0040), 0x5410);
      } else {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          if (d >= n) break;
#pragma unroll
          for (int k = 0; k < 3; ++k) row[3 * (x + d) + k] = static_cast<uint8_t>(c[d][k]);
        }
      }
    } else {
      unsigned int w[4];
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        w[d] = __byte_perm(__byte_perm(c[d][0], c[d][1], 0x0040), c[d][2], 0x7410) | 0xFF000000U;
      }
      if (vec) {
        *span_cast<uint4>(row + 4 * x) = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
#pragma unroll
        for (int d = 0; d < 4; ++d) {
          if (d >= n) break;
#pragma unroll
          for (int k = 0; k < 4; ++k) row[4 * (x + d) + k] = static_cast<uint8_t>(w[d] >> (8 * k));
        }
      }
    }
  } else if constexpr (kOut == kOutRgb16) {
    if (vec) {
      Span<uint2> o = span_cast<uint2>(row + 6 * x);
      o[0] = make_uint2(__byte_perm(c[0][0], c[0][1], 0x5410), __byte_perm(c[0][2], c[1][0], 0x5410));
      o[1] = make_uint2(__byte_perm(c[1][1], c[1][2], 0x5410), __byte_perm(c[2][0], c[2][1], 0x5410));
      o[2] = make_uint2(__byte_perm(c[2][2], c[3][0], 0x5410), __byte_perm(c[3][1], c[3][2], 0x5410));
    } else {
      Span<uint16_t> o = span_cast<uint16_t>(row);
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        if (d >= n) break;
#pragma unroll
        for (int k = 0; k < 3; ++k) o[3 * (x + d) + k] = static_cast<uint16_t>(c[d][k]);
      }
    }
  } else {
    if (vec) {
      Span<float4> o = span_cast<float4>(row + 12 * x);
      o[0] = make_float4(t[0][0], t[0][1], t[0][2], t[1][0]);
      o[1] = make_float4(t[1][1], t[1][2], t[2][0], t[2][1]);
      o[2] = make_float4(t[2][2], t[3][0], t[3][1], t[3][2]);
    } else {
      Span<float> o = span_cast<float>(row);
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        if (d >= n) break;
#pragma unroll
        for (int k = 0; k < 3; ++k) o[3 * (x + d) + k] = t[d][k];
      }
    }
  }
  if (want_hist) {
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      if (d >= n) break;
      // The 8-bit codes, with the 2^23 bits still on them where they are the
      // stored codes themselves.
      constexpr unsigned int kBias = kOut == kOutRgb16 ? 0U : kTwo23Bits;
      unsigned int q[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        // 16-bit values: (v * 255 + 32767) / 65535 == ((v + 128) * 0xFF01) >> 24
        // for v < 2^16 (checked for every v); c = 2^23 bits + v, and the
        // product of (c + 128 - 2^23 bits) stays below 2^32.
        q[k] = kOut == kOutRgb16 ? ((c[d][k] + (128U - kTwo23Bits)) * 0xFF01U) >> 24 : c[d][k];
      }
      count_code(hist, 0, luma_of(q[0], q[1], q[2], kBias), 0U);
#pragma unroll
      for (int k = 0; k < 3; ++k) count_code(hist, 1 + k, q[k], kBias);
    }
  }
}

// The per-pixel tail of four pairs of one row (pixels x .. x + 3 and
// x + 32 .. x + 35 of image row y): colour matrix, statistics sums, tone,
// codes, stores. nl, nr: pixels of the left and right groups inside the
// image (0..4); kFull: both are 4 (the interior units, compiled without the
// per-pixel guards). sums:
// 2^23 bits + to_fixed summed mod 2^32, npix the number of terms, so that the
// caller subtracts npix x 2^23 bits. The sums are formed whether the frame
// wants them or not: a test per value cut the twelve values of a unit into as
// many blocks of code, and two versions of the function overran the
// instruction cache of the batch kernel.
template <int kOut, bool kLutSmem, bool kFull>
__device__ __forceinline__ void finish_pairs(const FrameDesc& p, const float2 (&rgb)[4][3], int x, int y, int nl_,
                                             int nr_, Span<const float2> lut, float lut_scale,
                                             bool want_hist, Span<unsigned int> hist, unsigned int (&sums)[3],
                                             unsigned int& npix) {
  const int nl = kFull ? 4 : nl_;
  const int nr = kFull ? 4 : nr_;
  float tl[4][3], tr[4][3];
  unsigned int cl[4][3], cr[4][3];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2* c = rgb[i];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      // clamp01((m0 r + m1 g) + m2 b), isp_math.hpp:229-233.
      const float2 lin = add_sat2(psum2(mul2(bc2(p.ccm[3 * k]), c[0]), mul2(bc2(p.ccm[3 * k + 1]), c[1])),
                                  mul2(bc2(p.ccm[3 * k + 2]), c[2]));
      // to_fixed (isp_math.hpp:245-247): trunc(lin 2^20 + 0.5). lin 2^20 is
      // exact and so is the sum below 2^20 + 1; above it both roundings
      // truncate to 2^20.
      const float2 fixed = magic_trunc2(exact_scale_add2(lin, bc2(kFixedOne), bc2(0.5F)));
      sums[k] += (i < nl ? __float_as_uint(fixed.x) : 0U) + (i < nr ? __float_as_uint(fixed.y) : 0U);
      // f = lin (N - 1), a product; i = trunc(f); f - i.
      const float2 f = mul2(lin, bc2(lut_scale));
      const float2 m = magic_trunc_product2(f);
      const float2 frac = psum2(f, sub2(bc2(kTwo23), m));
      const float2 toned = make_float2(tone_lookup<kLutSmem>(lut, m.x, frac.x), tone_lookup<kLutSmem>(lut, m.y, frac.y));
      tl[i][k] = toned.x;
      tr[i][k] = toned.y;
      float2 code;
      // trunc(t scale + 0.5). RGB32F stores t itself; its code is of t clamped.
      if constexpr (kOut == kOutRgb16) {
        code = magic_trunc2(psum2(mul2(toned, bc2(65535.0F)), bc2(0.5F)));
      } else if constexpr (kOut == kOutRgb32f) {
        const float2 clamped = mul_sat2(toned, bc2(1.0F));
        code = magic_trunc2(psum2(mul2(clamped, bc2(255.0F)), bc2(0.5F)));
      } else {
        code = magic_trunc2(psum2(mul2(toned, bc2(255.0F)), bc2(0.5F)));
      }
      cl[i][k] = __float_as_uint(code.x);
      cr[i][k] = __float_as_uint(code.y);
    }
  }
  npix += static_cast<unsigned int>(nl + nr);
  if (kFull || nl > 0) store_seg4<kOut>(p, x, y, tl, cl, nl, want_hist, hist);
  if (kFull || nr > 0) store_seg4<kOut>(p, x + kHalf, y, tr, cr, nr, want_hist, hist);
}

template <bool kLutSmem, bool kFull>
__device__ __forceinline__ void finish_pairs_any(const FrameDesc& p, const float2 (&rgb)[4][3], int x, int y, int nl,
                                                 int nr, Span<const float2> lut, float lut_scale, bool want_hist,
                                                 Span<unsigned int> hist, unsigned int (&sums)[3],
                                                 unsigned int& npix) {
  switch (p.out_format) {
    case kOutRgb8:
      finish_pairs<kOutRgb8, kLutSmem, kFull>(p, rgb, x, y, nl, nr, lut, lut_scale, want_hist, hist, sums, npix);
      break;
    case kOutRgba8:
      finish_pairs<kOutRgba8, kLutSmem, kFull>(p, rgb, x, y, nl, nr, lut, lut_scale, want_hist, hist, sums, npix);
      break;
    case kOutRgb16:
      finish_pairs<kOutRgb16, kLutSmem, kFull>(p, rgb, x, y, nl, nr, lut, lut_scale, want_hist, hist, sums, npix);
      break;
    default:
      finish_pairs<kOutRgb32f, kLutSmem, kFull>(p, rgb, x, y, nl, nr, lut, lut_scale, want_hist, hist, sums, npix);
      break;
  }
}

}  // namespace
}  // namespace isp_b200
