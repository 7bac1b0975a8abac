// isp_awb.cuh - the white balance statistics pass as device templates: the
// sums of one 64x64-sample tile, and a frame's flush by a CTA with the
// last-tile finish. The single-frame kernel (isp_awb.cu) and the batch kernel
// (isp_batch.cu) are both built from them.
#pragma once

#include "isp_common.cuh"

namespace isp_b200 {
namespace {

__host__ __device__ constexpr int awb_box_bytes(int fmt) {
  return fmt == kRawU8 ? 64 : fmt == kRawU16 ? 128 : fmt == kRawRaw10 ? 80 : 96;
}

// TMA x coordinate (bytes, or uint16 samples) of the statistics box of a
// tile at column x0 (x0 % 64 == 0): 16-byte aligned.
__device__ __forceinline__ int awb_box_x(int fmt, int x0) {
  return fmt == kRawRaw10 ? 5 * (x0 >> 2) : fmt == kRawRaw12 ? 3 * (x0 >> 1) : x0;
}

// ---- Shared memory of a CTA of the statistics pass ---------------------------

constexpr int kAwbTableAt = 2 * 64 * 128;                             // boxes: [2][64][128], a double buffer
constexpr int kAwbColsAt = kAwbTableAt + kLscTableRows * 2 * kSW * 4;  // table: [kLscTableRows][2][kSW]
constexpr int kAwbRowsAt = kAwbColsAt + 2 * 64 * 4;                    // col_ix, col_tx: [64] each
constexpr int kAwbHistAt = kAwbRowsAt + 2 * kAwbBandRows * 4;          // row_k, row_ty: [kAwbBandRows] each
constexpr int kAwbGridAt = kAwbHistAt + 3 * kAwbBins * 4;              // hist: [3][kAwbBins]
constexpr int kAwbSmem = kAwbGridAt + kGridSmemGains * 4;              // grid: [kGridSmemGains]

struct AwbSmem {
  Span<uint8_t> boxes;
  Span<float> table;
  Span<int> col_ix;
  Span<float> col_tx;
  Span<int> row_k;
  Span<float> row_ty;
  Span<unsigned int> hist;
  Span<float> grid;
};

__device__ __forceinline__ AwbSmem carve_awb(unsigned char* smem, CheckRecord* rec) {
  AwbSmem m;
  m.boxes = carve_span<uint8_t>(smem, 0, kAwbTableAt, rec);
  m.table = carve_span<float>(smem, kAwbTableAt, kAwbColsAt - kAwbTableAt, rec);
  m.col_ix = carve_span<int>(smem, kAwbColsAt, 64 * 4, rec);
  m.col_tx = carve_span<float>(smem, kAwbColsAt + 64 * 4, 64 * 4, rec);
  m.row_k = carve_span<int>(smem, kAwbRowsAt, kAwbBandRows * 4, rec);
  m.row_ty = carve_span<float>(smem, kAwbRowsAt + kAwbBandRows * 4, kAwbBandRows * 4, rec);
  m.hist = carve_span<unsigned int>(smem, kAwbHistAt, 3 * kAwbBins * 4, rec);
  m.grid = carve_span<float>(smem, kAwbGridAt, kGridSmemGains * 4, rec);
  return m;
}

// A band's lens shading maps and table: build_lsc's columns, rows, grid-row
// range and table (the same arithmetic: top + (bottom - top) * ty from
// T[k] = g + (g' - g) * tx, isp_math.hpp:121-140), for 64 columns and up to
// kAwbBandRows rows, the rows looped over the block's threads.
__device__ LscTile build_band_lsc(const FrameDesc& p, Span<const float> grid, int pattern, int x_first, int y_first,
                                  int nrows, const AwbSmem& m, int* minmax) {
  constexpr int kCols = 64;
  const Span<int> col_ix = m.col_ix, row_k = m.row_k;
  const Span<float> col_tx = m.col_tx, row_ty = m.row_ty, table = m.table;
  const int t = threadIdx.x;
  if (t == 0) {
    minmax[0] = 0x7FFFFFFF;
    minmax[1] = -1;
  }
  __syncthreads();
  if (t < kCols) {
    const int x = x_first + t;
    if (p.lsc != nullptr) {
      const float fx = static_cast<float>(x) * p.lsc_sx;
      int ix = static_cast<int>(fx);
      ix = ix > p.lsc_width - 2 ? p.lsc_width - 2 : ix;
      col_ix[t] = ix;
      col_tx[t] = fx - static_cast<float>(ix);
    }
  }
  int iy_lo = 0x7FFFFFFF;
  int iy_hi = -1;
  for (int j = t; j < nrows; j += kThreads) {
    const int y = y_first + j;
    if (p.lsc != nullptr) {
      const float fy = static_cast<float>(y) * p.lsc_sy;
      int iy = static_cast<int>(fy);
      iy = iy > p.lsc_height - 2 ? p.lsc_height - 2 : iy;
      row_k[j] = iy;
      row_ty[j] = fy - static_cast<float>(iy);
      iy_lo = iy < iy_lo ? iy : iy_lo;
      iy_hi = iy > iy_hi ? iy : iy_hi;
    }
  }
  if (p.lsc != nullptr) {
    iy_lo = __reduce_min_sync(0xFFFFFFFFU, iy_lo);
    iy_hi = __reduce_max_sync(0xFFFFFFFFU, iy_hi);
    if ((t & 31) == 0 && iy_hi >= 0) {
      atomicMin(&minmax[0], iy_lo);
      atomicMax(&minmax[1], iy_hi);
    }
  }
  __syncthreads();
  LscTile lt{0, 0};
  if (p.lsc == nullptr) return lt;
  lt.iy0 = minmax[0];
  lt.rows = minmax[1] - minmax[0] + 2;
  if (lt.rows > kLscTableRows) return lt;
  const int step = p.lsc_channels;
  const int odd = step == 4 ? 1 : 0;  // two rows of the table per grid row, or one
  for (int e = t; e < (lt.rows << odd) * kCols; e += kThreads) {
    const int i = e % kCols;
    const int kp = e / kCols;
    const int par = kp & odd;
    const int k = kp >> odd;
    const int ch = step == 4 ? cfa_of(pattern, (par << 1) | (i & 1)) : 0;
    Span<const float> g = grid + ((lt.iy0 + k) * p.lsc_width + col_ix[i]) * step + ch;
    table[(k * 2 + par) * kSW + i] = g[0] + (g[step] - g[0]) * col_tx[i];
  }
  for (int j = t; j < nrows; j += kThreads) row_k[j] -= lt.iy0;
  __syncthreads();
  return lt;
}

// The two rows of the lens shading table that a thread's current samples lie
// between: T[k] and T[k + 1] - T[k] per row parity and column pair. A thread
// keeps its four columns through a band, so they are read again only where
// its rows cross into another cell of the grid.
struct AwbCell {
  int k = -1;
  float2 top[2][2];
  float2 step[2][2];
};

// Units of two complete quads (4 samples across, 2 rows) of one tile: the
// white balance sums (white_balance_quad, isp_math.hpp:311-332) into 32-bit
// per-tile sums (at most 8 samples of 2^22 per colour and thread) and, for
// white patch, the block's bins. The samples come from the tile's box.
template <bool kWhitePatch, int kPat>
__device__ __forceinline__ void awb_tile(const FrameDesc& p, Span<const float> grid, Span<const uint8_t> box, int box_bytes,
                                         int x0, int y0, const LscTile& lt, Span<const int> row_k,
                                         Span<const float> row_ty, Span<const float> table, const float (&black)[4],
                                         const float (&inv)[4], Span<unsigned int> hist, AwbCell& cell,
                                         unsigned int (&sum)[3], unsigned int& quads) {
  const int quads_x = p.width / 2;
  const int quads_y = p.height / 2;
  const int fmt = p.raw_format;
  const unsigned int white = static_cast<unsigned int>(p.white);
  const int u = threadIdx.x & 15;
  const int qx0 = (x0 >> 1) + 2 * u;
  unsigned int counted = 0;  // quads summed by this call
  static_assert(512 % kThreads == 0, "a tile's units split evenly over the block");
  if (qx0 < quads_x) {
#pragma unroll 1
    for (int a = threadIdx.x >> 4; a < 32; a += kThreads / 16) {
      if ((y0 >> 1) + a >= quads_y) break;
      unsigned int top[2], bot[2];  // samples 4u .. 4u + 3 of both rows, as 16-bit halves
      // unpack4 reads sample x0 - 4 + 4u' from a box starting at box_x; this
      // box starts at x0: step the row back to there, u' = u + 1.
      Span<const uint8_t> r0 = box + (2 * a) * box_bytes - 16;
      unpack4(fmt, r0, u + 1, top);
      unpack4(fmt, r0 + box_bytes, u + 1, bot);
      // Linear values before white balance, capped at 4 (isp_math.hpp:320-330).
      // The two quads of the unit run as the two lanes of f32x2 instructions:
      // lane x holds sample j of quad 0, lane y sample j of quad 1 (columns
      // 4u + j and 4u + j + 2, the same Bayer colour). The clamp to [0, 4] is
      // the saturating multiply by 1/4 below (all gains are positive, so a value
      // below black stays negative up to there).
      float2 v[2][2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const unsigned int* s = r == 0 ? top : bot;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int q = (r << 1) | j;
          const float2 raw = j == 0 ? magic_to_float2(magic_low(s[0]), magic_low(s[1]))
                                    : magic_to_float2(magic_high(s[0]), magic_high(s[1]));
          v[r][j] = mul2(sub2(raw, bc2(black[q])), bc2(inv[q]));
        }
      }
      if (lt.rows > 0) {
        if (lt.rows <= kLscTableRows) {
          // gain = T[k] + (T[k + 1] - T[k]) ty (lens_shading_gain, isp_math.hpp:121-140).
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const int k = row_k[2 * a + r];
            if (k != cell.k) {
              cell.k = k;
#pragma unroll
              for (int par = 0; par < 2; ++par) {
                const int pl = p.lsc_channels == 4 ? par : 0;
                const float4 t0 = *span_cast<const float4>(table + (k * 2 + pl) * kSW + 4 * u);
                const float4 t1 = *span_cast<const float4>(table + ((k + 1) * 2 + pl) * kSW + 4 * u);
                cell.top[par][0] = make_float2(t0.x, t0.z);
                cell.top[par][1] = make_float2(t0.y, t0.w);
                cell.step[par][0] = sub2(make_float2(t1.x, t1.z), cell.top[par][0]);
                cell.step[par][1] = sub2(make_float2(t1.y, t1.w), cell.top[par][1]);
              }
            }
            const float2 ty = bc2(row_ty[2 * a + r]);
            v[r][0] = mul2(v[r][0], psum2(mul2(cell.step[r][0], ty), cell.top[r][0]));
            v[r][1] = mul2(v[r][1], psum2(mul2(cell.step[r][1], ty), cell.top[r][1]));
          }
        } else {
          const LscGrid g{grid, p.lsc_width, p.lsc_height, p.lsc_channels, p.lsc_sx, p.lsc_sy};
#pragma unroll
          for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int channel = cfa_of(kPat, (r << 1) | j);
              v[r][j].x = fmul(v[r][j].x, lens_shading_gain_outline(g, x0 + 4 * u + j, y0 + 2 * a + r, channel));
              v[r][j].y = fmul(v[r][j].y, lens_shading_gain_outline(g, x0 + 4 * u + j + 2, y0 + 2 * a + r, channel));
            }
          }
        }
      }
      // The quad test per lane: no sample at or above white (isp_math.hpp:316-318).
      const bool ok0 = !any_half_at_least(__vmaxu2(top[0], bot[0]), white);
      const bool ok1 = qx0 + 1 < quads_x && !any_half_at_least(__vmaxu2(top[1], bot[1]), white);
      unsigned int m0[4], m1[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        // x / 4 in [0, 1], the scale exact; to_fixed: trunc(x 2^20 + 0.5), the
        // product exact. Summed as 2^23 bits + value; the 2^23 bits come off
        // once, after the units.
        const float2 x = mul_sat2(v[k >> 1][k & 1], bc2(0.25F));
        const float2 m = magic_trunc2(exact_scale_add2(x, bc2(4.0F * kFixedOne), bc2(0.5F)));
        m0[k] = __float_as_uint(m.x);
        m1[k] = __float_as_uint(m.y);
        if constexpr (kWhitePatch) {
          // trunc(x 1024): an exact product, so its two-lane truncation is safe.
          const float2 b = magic_trunc2(mul2(x, bc2(4.0F * kAwbBins)));
          const unsigned int b0 = magic_int(b.x), b1 = magic_int(b.y);
          Span<unsigned int> h = hist + color_of(cfa_of(kPat, k)) * kAwbBins;
          if (ok0) atomicAdd(&h[b0 < kAwbBins - 1 ? b0 : kAwbBins - 1], 1U);
          if (ok1) atomicAdd(&h[b1 < kAwbBins - 1 ? b1 : kAwbBins - 1], 1U);
        }
      }
      if (ok0 && ok1) {
#pragma unroll
        for (int k = 0; k < 4; ++k) sum[color_of(cfa_of(kPat, k))] += m0[k] + m1[k];
        counted += 2U;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) sum[color_of(cfa_of(kPat, k))] += (ok0 ? m0[k] : 0U) + (ok1 ? m1[k] : 0U);
        counted += (ok0 ? 1U : 0U) + (ok1 ? 1U : 0U);
      }
    }
  }
  // Every counted quad added one red, two green and one blue sample, each
  // with 2^23 bits on top (sums mod 2^32; the true sums fit 32 bits).
  sum[0] -= counted * kTwo23Bits;
  sum[1] -= 2U * counted * kTwo23Bits;
  sum[2] -= counted * kTwo23Bits;
  quads += counted;
}

// A frame's flush by one CTA after it summed `tiles_done` of the frame's
// `tiles_total` statistics tiles: block sums and bins into the frame's
// scratch; the CTA that completes the count forms the frame's estimate
// (awb_finish). The block's bins are left for the caller to clear.
// With kAfterPrevious, the last CTA first waits (griddepcontrol.wait) for the
// kernel this pass was launched behind: the single-frame pass may begin
// while the previous frame's tile pass finishes, and only the estimate
// (which reads and writes the white balance state that tile pass read) must
// follow it.
template <bool kAfterPrevious = false>
__device__ void awb_flush(const FrameDesc& p, const u64 (&acc)[4], Span<const unsigned int> hist, bool white_patch,
                          u64* red, bool* last, unsigned int tiles_done, unsigned int tiles_total) {
  Span<Scratch> s = p.scratch;
  const int tid = threadIdx.x;
  u64 total[4];
  block_sum4(acc, red, total);  // its barrier also closes the block's bins
  if (tid < 4 && total[tid] != 0) atomicAdd(tid < 3 ? &s->awb_sum[tid] : &s->awb_quads, total[tid]);
  if (white_patch) {
    // Two bins per 64-bit atomic: a bin's count over a frame stays below 2^32.
    static_assert(offsetof(Scratch, awb_hist) % 8 == 0, "bin pairs are 8-byte aligned");
    const Span<unsigned long long> pairs = span_cast<unsigned long long>(sub_span(s, &s->awb_hist[0][0], 3 * kAwbBins));
    for (int i = tid; i < 3 * kAwbBins / 2; i += kThreads) {
      const uint2 h = span_cast<const uint2>(hist)[i];
      if ((h.x | h.y) != 0U) atomicAdd(&pairs[i], (static_cast<unsigned long long>(h.y) << 32) | h.x);
    }
  }
  __syncthreads();
  if (tid == 0) {
    // The block's atomics come before the count that hands the frame over
    // (the barrier above orders them before this thread's fence).
    __threadfence();
    *last = atomicAdd(&s->awb_done, tiles_done) + tiles_done == tiles_total;
  }
  __syncthreads();
  if (*last) {
    if constexpr (kAfterPrevious) griddep_wait();
    __threadfence();
    awb_finish(p, s);
  }
  __syncthreads();
}

}  // namespace
}  // namespace isp_b200
