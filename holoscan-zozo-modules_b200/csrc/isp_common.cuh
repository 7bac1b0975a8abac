// isp_common.cuh - device building blocks shared by the ISP's kernels: tile
// geometry and shared-memory layout, TMA and mbarrier helpers, raw unpacking,
// lens shading tables, stores, block reductions and the last-CTA finishers.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "isp_device.cuh"
#include "isp_kernels.cuh"
#include "isp_ops.cuh"

namespace isp_b200 {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTW = 64;  // tile: output pixels across
constexpr int kTH = 64;  // and down
constexpr int kSW = 72;  // samples per tile row: x0 - 4 .. x0 + 67
constexpr int kUnitsRow = kSW / 4;
constexpr unsigned int kWaitLimit = 1U << 22;  // bounded mbarrier polls
// Grid rows a tile's lens shading table holds; tiles that need more compute
// each gain from the grid directly.
constexpr int kLscTableRows = 8;

// The channel (kChR, kChGr, kChGb, kChB) at quad position (y & 1) * 2 + (x & 1)
// of each Bayer pattern, packed two bits per entry so that a run-time lookup
// is a shift (a constant array indexed at run time would live in local memory).
__host__ __device__ constexpr unsigned int cfa_word() {
  constexpr int t[4][4] = {{kChR, kChGr, kChGb, kChB},
                           {kChB, kChGb, kChGr, kChR},
                           {kChGr, kChR, kChB, kChGb},
                           {kChGb, kChB, kChR, kChGr}};
  unsigned int w = 0;
  for (int p = 0; p < 4; ++p) {
    for (int q = 0; q < 4; ++q) w |= static_cast<unsigned int>(t[p][q]) << (8 * p + 2 * q);
  }
  return w;
}
constexpr unsigned int kCfaWord = cfa_word();
__host__ __device__ constexpr int cfa_of(int pattern, int pos) {
  return static_cast<int>((kCfaWord >> (8 * pattern + 2 * pos)) & 3U);
}
static_assert(cfa_of(0, 0) == kChR && cfa_of(1, 3) == kChR && cfa_of(2, 1) == kChR && cfa_of(3, 2) == kChR &&
                  cfa_of(2, 0) == kChGr && cfa_of(3, 1) == kChB && cfa_of(1, 1) == kChGb,
              "Bayer channel table");

// Lens shading grids of at most this many gains are kept in shared memory
// for the frame (a 17 x 13 x 4 grid is 884).
constexpr int kGridSmemGains = 1024;

// A frame's constants per quad position (3 x 4) and its gains.
constexpr int kQuadFloats = 15;

// Paired pixels. The tile pass computes two pixels in the two lanes of every
// f32x2 operation: columns c and c + kHalf of the same row, which have the
// same Bayer colour and so the same arithmetic. Samples and RGB values live
// in shared memory as float2 pairs {v(c), v(c + kHalf)}, so that each operand
// is one aligned 8-byte element and neighbours are neighbouring pairs.
constexpr int kHalf = 32;
// Paired sample columns: pair s (0..39) holds tile samples s and s + 32
// (sample s is image column x0 - 4 + s).
constexpr int kPW = 40;
// Paired RGB columns (sharpening): pair q (0..33) holds pixels q - 1 and q + 31.
constexpr int kCW2 = 34;

// Tile heights the kernels are compiled for: kTH rows (the default) or
// kTHShort rows (more, smaller tiles: a frame of few tiles spreads over more
// SMs, and three CTAs share an SM).
constexpr int kTHShort = 32;

template <bool kSharpen, int kTileH = kTH>
struct Geom {
  static constexpr int kHalo = kSharpen ? 4 : 2;  // sample rows above and below the tile
  static constexpr int kSH = kTileH + 2 * kHalo;
  static constexpr int kCH = kTileH + 2;  // RGB rows: y0 - 1 .. y0 + kTileH
};

// ---- Shared memory layout -------------------------------------------------

// The regions whose size a kernel instance knows come first, so that their
// offsets from the one base register are constants; the TMA box (its size
// depends on the raw format) and the tone table follow.
struct Layout {
  int samples;  // float2 [kSH][kPW]
  int r, g, b;  // float2 [kCH][kCW2] each (sharpening)
  int lsc;      // float2 [kLscTableRows][2][kPW]
  int cols;     // int col_mx[kSW]; int col_ix[kSW]; float col_tx[kSW]
  int rows;     // int row_my[kSH]; int row_k[kSH]; float row_ty[kSH]
  int quad;     // float [kQuadFloats]: the frame's constants per quad position
  int hist;     // u32 [4][256]
  int grid;     // float [kGridSmemGains]: the frame's lens shading grid, when it fits
  int raw;      // TMA box: box rows x box bytes
  int lut;      // float2 [tone_size] when in shared memory
  int total;
};

__host__ __device__ constexpr int align128(int v) { return (v + 127) & ~127; }

__host__ __device__ constexpr Layout layout_of(bool sharpen, int box_bytes_row, int lut_entries, int tile_h = kTH) {
  const int halo = sharpen ? 4 : 2;
  const int sh = tile_h + 2 * halo;
  const int plane = align128((tile_h + 2) * kCW2 * 8);
  Layout l{};
  int o = 0;
  l.samples = o;
  o = align128(o + sh * kPW * 8);
  l.r = o;
  l.g = o + (sharpen ? plane : 0);
  l.b = o + (sharpen ? 2 * plane : 0);
  if (sharpen) o += 3 * plane;
  l.lsc = o;
  o = align128(o + kLscTableRows * 2 * kPW * 8);
  l.cols = o;
  o = align128(o + 3 * kSW * 4);
  l.rows = o;
  o = align128(o + 3 * sh * 4);
  l.quad = o;
  o = align128(o + kQuadFloats * 4);
  l.hist = o;
  o = align128(o + kHistChannels * kHistBins * 4);
  l.grid = o;
  o = align128(o + kGridSmemGains * 4);
  l.raw = o;
  o = align128(o + sh * box_bytes_row);
  l.lut = o;
  o = align128(o + lut_entries * 8);
  l.total = o;
  return l;
}

// Bytes per box row of each raw format (TMA inner extent, multiple of 16),
// and the byte of the box row where sample x0 - 4 starts.
__host__ __device__ constexpr int box_row_bytes(int fmt) {
  return fmt == kRawU8 ? 96 : fmt == kRawU16 ? 160 : fmt == kRawRaw10 ? 112 : 128;
}

// ---- TMA and mbarrier -----------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Requests a box of `bytes` bytes into dst, completing on bar. (The checked
// build makes no copy whose box would leave dst's region: it arrives on the
// barrier without one, so that the wait still ends.)
__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, Span<uint8_t> dst, uint64_t* bar, int x, int y,
                                            unsigned int bytes) {
#ifdef ISP_CHECKED
  if (span_range(dst, bytes) != span_ptr(dst)) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    return;
  }
#endif
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
      "[%4];" ::"r"(smem_u32(span_ptr(dst))),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}

// Waits for the barrier's phase `parity` to complete; false after `limit` polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned int limit = kWaitLimit) {
  for (unsigned int i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// A bounded wait gave up: the frame's outputs are not trustworthy. The flag
// stays set until isp_b200_device_status reads and clears it.
__device__ __forceinline__ void report_wait_timeout(Span<Scratch> s) { atomicExch(&s->error, 1); }

__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Copies of 4 or 8 bytes from global to shared memory that bypass the
// registers: a thread's copies are all in flight at once (a fill loop of
// plain loads and stores waits out one L2 round trip per iteration), and
// cp_async_wait_all() returns once this thread's copies have landed.
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
#ifdef ISP_CHECKED
  if (!__isShared(dst)) {  // a refused destination: the check's sink in global memory
    *static_cast<uint32_t*>(dst) = *static_cast<const uint32_t*>(src);
    return;
  }
#endif
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(__cvta_generic_to_global(src))
               : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
#ifdef ISP_CHECKED
  if (!__isShared(dst)) {
    *static_cast<uint2*>(dst) = *static_cast<const uint2*>(src);
    return;
  }
#endif
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(__cvta_generic_to_global(src))
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The TMA coordinates of the box for a tile at (x0, y0) (x in the tensor's
// elements: bytes, or uint16 samples), 16-byte aligned for any x0 % 64 == 0.
__device__ __forceinline__ int box_x(int fmt, int x0) {
  return fmt == kRawU8 ? x0 - 16 : fmt == kRawU16 ? x0 - 8 : fmt == kRawRaw10 ? 5 * (x0 >> 2) - 16 : 3 * (x0 >> 1) - 16;
}

// ---- Raw unpacking from a box row ----------------------------------------

// Samples x0 - 4 + 4u .. + 3 of a box row (box starting at box_x(fmt, x0)) as
// 16-bit halves: w[0] holds the first two, w[1] the last two. Packed halves
// cost 2.5 (RAW10) or 3 (RAW12) integer operations a sample where extracting
// each sample on its own took 4, and the saturation tests take a maximum of
// two samples per instruction.
__device__ __forceinline__ void unpack4(int fmt, Span<const uint8_t> row, int u, unsigned int (&w)[2]) {
  if (fmt == kRawU8) {
    const unsigned int v = *span_cast<const unsigned int>(row + 12 + 4 * u);
    w[0] = __byte_perm(v, 0U, 0x4140);
    w[1] = __byte_perm(v, 0U, 0x4342);
  } else if (fmt == kRawU16) {
    const uint2 v = *span_cast<const uint2>(row + 8 + 8 * u);
    w[0] = v.x;
    w[1] = v.y;
  } else if (fmt == kRawRaw10) {
    // Group g0 - 1 + u at byte 11 + 5u: four high bytes, then the low bits.
    const int b = 11 + 5 * u;
    Span<const unsigned int> v = span_cast<const unsigned int>(row + (b & ~3));
    const unsigned int at = static_cast<unsigned int>(b & 3);
    const unsigned int next = v[1];
    const unsigned int hi4 = __funnelshift_r(v[0], next, 8U * at);
    // The four 2-bit fields: t holds the low byte at bits 0 and 14, so that
    // fields 0 and 1 (2 and 3 after >> 4) lie at bits 0 and 16.
    const unsigned int t = __byte_perm(next, 0U, 0x4440U + at) * 0x4001U;
    w[0] = __byte_perm(hi4, 0U, 0x4140) * 4U + (t & 0x00030003U);
    w[1] = __byte_perm(hi4, 0U, 0x4342) * 4U + ((t >> 4) & 0x00030003U);
  } else {
    // Two groups of three bytes at byte 10 + 6u: two high bytes, then the low
    // nibbles, copied to bits 0 and 12 so that they lie at bits 0 and 16.
    const int b = 10 + 6 * u;
    Span<const unsigned int> v = span_cast<const unsigned int>(row + (b & ~3));
    const unsigned int sh = 8U * static_cast<unsigned int>(b & 3);
    const unsigned int next = v[1];
    const unsigned int v0 = __funnelshift_r(v[0], next, sh);  // a0 a1 a2 b0
    const unsigned int v1 = next >> sh;                        // b1 b2 ..
    w[0] = __byte_perm(v0, 0U, 0x4140) * 16U + ((__byte_perm(v0, 0U, 0x4442) * 0x1001U) & 0x000F000FU);
    w[1] = (__byte_perm(v0, v1, 0x0403) & 0x00FF00FFU) * 16U +
           ((__byte_perm(v1, 0U, 0x4441) * 0x1001U) & 0x000F000FU);
  }
}

// 2^23 + a 16-bit half of w, as the bits of a float.
__device__ __forceinline__ unsigned int magic_low(unsigned int w) { return __byte_perm(w, kTwo23Bits, 0x7610); }
__device__ __forceinline__ unsigned int magic_high(unsigned int w) { return __byte_perm(w, kTwo23Bits, 0x7632); }
// Whether a 16-bit half of w is at least `white`.
__device__ __forceinline__ bool any_half_at_least(unsigned int w, unsigned int white) {
  return max(w & 0xFFFFU, w >> 16) >= white;
}

// One sample at image column mx of a box row (box starting at box_x(fmt, x0)).
__device__ __forceinline__ unsigned int unpack1(int fmt, Span<const uint8_t> row, int mx, int x0) {
  if (fmt == kRawU8) return row[mx - x0 + 16];
  if (fmt == kRawU16) return *span_cast<const uint16_t>(row + 2 * (mx - x0 + 8));
  if (fmt == kRawRaw10) {
    Span<const uint8_t> g = row + 5 * ((mx >> 2) - (x0 >> 2)) + 16;
    const int k = mx & 3;
    return (static_cast<unsigned int>(g[k]) << 2) | ((g[4] >> (2 * k)) & 3U);
  }
  Span<const uint8_t> g = row + 3 * ((mx >> 1) - (x0 >> 1)) + 16;
  const int k = mx & 1;
  return (static_cast<unsigned int>(g[k]) << 4) | ((g[2] >> (4 * k)) & 15U);
}

// The four samples whose mirrored columns col_mx holds, from a box row, as
// unpack4's halves. For the few units of an edge tile that reach past the
// image; out of line, so that they cost the others no registers or code.
__device__ __noinline__ uint2 unpack_edge4(int fmt, Span<const uint8_t> row, Span<const int> col_mx, int x0) {
  unsigned int s[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) s[k] = unpack1(fmt, row, col_mx[k], x0);
  return make_uint2(s[0] | (s[1] << 16), s[2] | (s[3] << 16));
}

// ---- Boxes without TMA -----------------------------------------------------

// The bytes of a raw row (raw_row_bytes, isp_params.cpp:184-197).
__device__ __forceinline__ int raw_bytes_of(int fmt, int width) {
  return fmt == kRawU8 ? width : fmt == kRawU16 ? 2 * width : fmt == kRawRaw10 ? 5 * ((width + 3) >> 2) : 3 * ((width + 1) >> 1);
}

// Fills a box as TMA would, for a frame whose rows are not 16-byte aligned:
// `rows` rows of `box_bytes` bytes from byte bx (a multiple of 16) of image
// rows y0 .., zero outside the image. Warps take rows, lanes 4-byte words:
// asynchronous copies where rows are 4-byte aligned, else two aligned words
// shifted together; the words at a row's ends byte by byte, so that nothing
// outside the frame's rows is read. The caller waits (box_filled) and
// synchronises the block. The copies are in flight while the tile's lens
// shading table is built. A 1366x768 16-bit frame with packed rows (white
// patch, RGB32F) takes 31.6 us this way; with a load from global memory per
// sample in both passes it took 42.9.
__device__ void fill_box(const FrameDesc& p, Span<uint8_t> box, int box_bytes, int rows, int bx, int y0) {
  const int row_bytes = raw_bytes_of(p.raw_format, p.width);
  const int words = box_bytes >> 2;
  const bool aligned = ((reinterpret_cast<uintptr_t>(span_ptr(p.raw)) | static_cast<uintptr_t>(p.raw_pitch)) & 3U) == 0U;
  for (int j = threadIdx.x >> 5; j < rows; j += kWarps) {
    const int y = y0 + j;
    const bool inside = y >= 0 && y < p.height;
    Span<const uint8_t> row = p.raw + static_cast<int64_t>(inside ? y : 0) * p.raw_pitch;
    for (int c = threadIdx.x & 31; c < words; c += 32) {
      const int o = bx + 4 * c;
      Span<uint8_t> dst = box + j * box_bytes + 4 * c;
      unsigned int v = 0U;
      if (inside && o > -4 && o < row_bytes) {
        if (aligned && o >= 0 && o + 4 <= row_bytes) {
          cp_async4(span_range(dst, 4), span_range(row + o, 4));
          continue;
        }
        if (o >= 4 && o + 8 <= row_bytes) {
          const unsigned int back = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(span_ptr(row + o)) & 3U);
          Span<const unsigned int> w = span_cast<const unsigned int>(row + (o - static_cast<int>(back)));
          v = __funnelshift_r(__ldg(&w[0]), __ldg(&w[1]), 8U * back);
        } else {
          for (int b = 0; b < 4; ++b) {
            if (o + b >= 0 && o + b < row_bytes) v |= static_cast<unsigned int>(__ldg(&row[o + b])) << (8 * b);
          }
        }
      }
      *span_cast<unsigned int>(dst) = v;
    }
  }
}

// Waits for this thread's part of fill_box and orders it before a later TMA
// copy into the same box (a batch mixes both); the block barrier is the caller's.
__device__ __forceinline__ void box_filled() {
  cp_async_wait_all();
  fence_async_shared();
}

// ---- Lens shading tables --------------------------------------------------

// Per tile: for every column the grid cell and fraction across, for every
// row the cell and fraction down, and the interpolated "top" rows
//   T[k][parity][i] = g(iy0 + k, ix_i) + (g(iy0 + k, ix_i + 1) - g(iy0 + k, ix_i)) * tx_i
// for the grid rows iy0 .. iy0 + K - 1 the tile's rows use, so that a
// sample's gain is T[k] + (T[k + 1] - T[k]) * ty: the reference's
// top + (bottom - top) * ty (isp_math.hpp:121-140), same operands, same order.
struct LscTile {
  int iy0;
  int rows;  // K; 0 when there is no grid, > kLscTableRows when the table does not fit
};

// Fills the column and row maps (mirrored coordinates, grid cells) and, when
// it fits, the table. Threads 0..ncols-1 do columns, the next nrows do rows.
// The table holds float2 pairs {T(s), T(s + kHalf)} for s < kPW (the tile pass's
// paired columns).
// `grid`: the frame's lens shading gains (the frame's own, or a copy in
// shared memory).
__device__ LscTile build_lsc(const FrameDesc& p, Span<const float> grid, int pattern, int x_first, int ncols, int y_first,
                             int nrows,
                             bool mirror_xy, int xclamp, int yclamp, Span<int> col_mx, Span<int> col_ix, Span<float> col_tx,
                             Span<int> row_my, Span<int> row_k, Span<float> row_ty, Span<float> table, int* minmax) {
  const int t = threadIdx.x;
  if (t == 0) {
    minmax[0] = 0x7FFFFFFF;
    minmax[1] = -1;
  }
  int iy_lo = 0x7FFFFFFF;  // this thread's row's grid row, if it has one
  int iy_hi = -1;
  __syncthreads();
  if (t < ncols) {
    int x = x_first + t;
    if (mirror_xy) x = mirror(x < xclamp ? x : xclamp, p.width);
    col_mx[t] = x;
    if (p.lsc != nullptr) {
      const float fx = static_cast<float>(x) * p.lsc_sx;
      int ix = static_cast<int>(fx);
      ix = ix > p.lsc_width - 2 ? p.lsc_width - 2 : ix;
      col_ix[t] = ix;
      col_tx[t] = fx - static_cast<float>(ix);
    }
  } else if (t < ncols + nrows) {
    const int j = t - ncols;
    int y = y_first + j;
    if (mirror_xy) y = mirror(y < yclamp ? y : yclamp, p.height);
    row_my[j] = y;
    if (p.lsc != nullptr) {
      const float fy = static_cast<float>(y) * p.lsc_sy;
      int iy = static_cast<int>(fy);
      iy = iy > p.lsc_height - 2 ? p.lsc_height - 2 : iy;
      row_k[j] = iy;
      row_ty[j] = fy - static_cast<float>(iy);
      iy_lo = iy;
      iy_hi = iy;
    }
  }
  // The rows' grid range: a warp reduction, then one shared atomic per warp
  // (same-address shared atomics from every row thread would serialise).
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
  const int planes = step == 4 ? 2 : 1;
  const auto entry = [&](int k, int par, int i) {
    const int ch = step == 4 ? cfa_of(pattern, (par << 1) | (col_mx[i] & 1)) : 0;
    Span<const float> g = grid + ((lt.iy0 + k) * p.lsc_width + col_ix[i]) * step + ch;
    return g[0] + (g[step] - g[0]) * col_tx[i];
  };
  Span<float2> table2 = span_cast<float2>(table);
  for (int e = t; e < lt.rows * planes * kPW; e += kThreads) {
    const int i = e % kPW;
    const int kp = e / kPW;
    const int par = kp % planes;
    const int k = kp / planes;
    table2[(k * 2 + par) * kPW + i] = make_float2(entry(k, par, i), entry(k, par, i + kHalf));
  }
  if (t < nrows) row_k[t] -= lt.iy0;
  __syncthreads();
  return lt;
}

// build_lsc for a tile none of whose rows and columns is mirrored:
// the grid rows it spans follow from its first and last rows (a row's grid
// cell never decreases down the frame), so the row maps and the paired table
// are written in one pass behind one block barrier, each table entry working
// out its own column's cell (the same operations as build_lsc's column maps).
// Tiles whose table would not fit take build_lsc. The mirrored rows and columns
// are not written: phase A reads those of edge tiles and of grids too dense for
// the table only.
__device__ LscTile build_lsc_inner(const FrameDesc& p, Span<const float> grid, int pattern, int x_first, int y_first,
                                   int nrows, Span<int> col_mx, Span<int> col_ix, Span<float> col_tx, Span<int> row_my, Span<int> row_k,
                                   Span<float> row_ty, Span<float> table, int* minmax) {
  LscTile lt{0, 0};
  const int t = threadIdx.x;
  if (p.lsc == nullptr) {
    return lt;
  }
  const auto row_cell = [&](int y) {
    const int iy = static_cast<int>(static_cast<float>(y) * p.lsc_sy);
    return iy > p.lsc_height - 2 ? p.lsc_height - 2 : iy;
  };
  lt.iy0 = row_cell(y_first);
  lt.rows = row_cell(y_first + nrows - 1) - lt.iy0 + 2;
  if (lt.rows > kLscTableRows) {
    return build_lsc(p, grid, pattern, x_first, kSW, y_first, nrows, false, 0, 0, col_mx, col_ix, col_tx, row_my,
                           row_k, row_ty, table, minmax);
  }
  if (t < nrows) {
    const int y = y_first + t;
    const float fy = static_cast<float>(y) * p.lsc_sy;
    int iy = static_cast<int>(fy);
    iy = iy > p.lsc_height - 2 ? p.lsc_height - 2 : iy;
    row_k[t] = iy - lt.iy0;
    row_ty[t] = fy - static_cast<float>(iy);
  }
  const int step = p.lsc_channels;
  const int planes = step == 4 ? 2 : 1;
  const auto entry = [&](int k, int par, int i) {
    const int x = x_first + i;
    const float fx = static_cast<float>(x) * p.lsc_sx;
    int ix = static_cast<int>(fx);
    ix = ix > p.lsc_width - 2 ? p.lsc_width - 2 : ix;
    const float tx = fx - static_cast<float>(ix);
    const int ch = step == 4 ? cfa_of(pattern, (par << 1) | (x & 1)) : 0;
    Span<const float> g = grid + ((lt.iy0 + k) * p.lsc_width + ix) * step + ch;
    return g[0] + (g[step] - g[0]) * tx;
  };
  Span<float2> table2 = span_cast<float2>(table);
  for (int e = t; e < lt.rows * planes * kPW; e += kThreads) {
    const int i = e % kPW;
    const int kp = e / kPW;
    const int par = kp % planes;
    const int k = kp / planes;
    table2[(k * 2 + par) * kPW + i] = make_float2(entry(k, par, i), entry(k, par, i + kHalf));
  }
  __syncthreads();
  return lt;
}

__device__ __forceinline__ u64 warp_sum(u64 v) {
#pragma unroll
  for (int offset = 16; offset > 0; offset >>= 1) v += __shfl_down_sync(0xFFFFFFFFU, v, offset);
  return v;
}

// Sums of four u64 per thread over the block, in `out` of thread 0; `red`
// holds 4 x kWarps values.
__device__ __forceinline__ void block_sum4(const u64 (&v)[4], u64* red, u64 (&out)[4]) {
  u64 w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = warp_sum(v[k]);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) red[k * kWarps + (threadIdx.x >> 5)] = w[k];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    u64 total = 0;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) total += red[k * kWarps + i];
    out[k] = total;
  }
}

// histogram_percentile (isp_math.hpp:336-352) by one warp: lane l owns bins
// 32l .. 32l + 31; the prefix counts are exact integers, so every comparison is
// the reference's. The result in every lane. (Three warps take the three
// colours side by side, without block barriers: one colour after the other by
// the whole block took two dozen of them at the end of every frame.)
__device__ float warp_percentile(Span<const unsigned int> hist, float percentile) {
  constexpr int kPerLane = kAwbBins / 32;
  const int lane = threadIdx.x & 31;
  uint4 h[kPerLane / 4];
  u64 mine = 0;
#pragma unroll
  for (int k = 0; k < kPerLane / 4; ++k) {
    h[k] = __ldcg(&span_cast<const uint4>(hist)[lane * (kPerLane / 4) + k]);
    mine += static_cast<u64>(h[k].x) + h[k].y + h[k].z + h[k].w;
  }
  u64 inc = mine;
#pragma unroll
  for (int offset = 1; offset < 32; offset <<= 1) {
    const u64 up = __shfl_up_sync(0xFFFFFFFFU, inc, offset);
    if (lane >= offset) inc += up;
  }
  const u64 total = __shfl_sync(0xFFFFFFFFU, inc, 31);
  if (total == 0) return 0.0F;
  const double target = static_cast<double>(percentile) * static_cast<double>(total);
  // This lane's first counted bin that reaches the target; the lowest such
  // lane holds the answer.
  u64 below = inc - mine;
  int bin = -1;
  u64 bin_below = 0;
  unsigned int bin_count = 0;
#pragma unroll
  for (int k = 0; k < kPerLane; ++k) {
    const uint4 w = h[k >> 2];
    const unsigned int n = (k & 3) == 0 ? w.x : (k & 3) == 1 ? w.y : (k & 3) == 2 ? w.z : w.w;
    if (bin < 0 && n != 0U && static_cast<double>(below + n) >= target) {
      bin = lane * kPerLane + k;
      bin_below = below;
      bin_count = n;
    }
    below += n;
  }
  const unsigned int found = __ballot_sync(0xFFFFFFFFU, bin >= 0);
  if (found == 0U) return 1.0F;
  float result = 1.0F;
  if (bin >= 0) {
    const double within = (target - static_cast<double>(bin_below)) / static_cast<double>(bin_count);
    result = static_cast<float>((static_cast<double>(bin) + within) / kAwbBins);
  }
  return __shfl_sync(0xFFFFFFFFU, result, __ffs(static_cast<int>(found)) - 1);
}

// finish_white_balance (isp_math.hpp:357-384) in the statistics pass's last
// CTA; then the sums are cleared for the next frame.
__device__ void awb_finish(const FrameDesc& p, Span<Scratch> s) {
  __shared__ float level[3];
  const int warp = threadIdx.x >> 5;
  const u64 nquads = __ldcg(&s->awb_quads);
  if (nquads != 0 && warp < 3) {
    float v;
    if (p.awb_mode == kWbGrayWorld) {
      const double q = static_cast<double>(nquads);
      const double sum = static_cast<double>(__ldcg(&s->awb_sum[warp]));
      v = static_cast<float>(warp == 1 ? sum / (2.0 * q) : sum / q);
    } else {
      v = warp_percentile(sub_span(s, &s->awb_hist[warp][0], kAwbBins), p.awb_percentile);
    }
    if ((threadIdx.x & 31) == 0) level[warp] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0 && nquads != 0 && level[0] > 0.0F && level[1] > 0.0F && level[2] > 0.0F) {
    const float target[3] = {level[1] / level[0], 1.0F, level[1] / level[2]};
    const bool smooth = s->awb_valid != 0 && p.awb_smoothing < 1.0F;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      const float t = target[k] < 0.0625F ? 0.0625F : target[k] > 16.0F ? 16.0F : target[k];
      const float g = s->awb_gains[k];
      s->awb_gains[k] = smooth ? g + p.awb_smoothing * (t - g) : t;
    }
    s->awb_valid = 1;
  }
  if (p.awb_mode == kWbWhitePatch) {
    static_assert(offsetof(Scratch, awb_hist) % 16 == 0, "bins are cleared 16 bytes at a time");
    const Span<uint4> bins = span_cast<uint4>(sub_span(s, &s->awb_hist[0][0], 3 * kAwbBins));
    for (int i = threadIdx.x; i < 3 * kAwbBins / 4; i += kThreads) bins[i] = make_uint4(0U, 0U, 0U, 0U);
  }
  if (threadIdx.x < 3) s->awb_sum[threadIdx.x] = 0;
  if (threadIdx.x == 3) s->awb_quads = 0;
  if (threadIdx.x == 4) s->awb_done = 0;
}

// finish_stats (isp_math.hpp:387-425) from the main pass's sums.
__device__ void finish_stats(const FrameDesc& p, const u64 sum[3], u64 saturated, const float gains[3]) {
  const int64_t pixels = static_cast<int64_t>(p.width) * p.height;
  const double n = static_cast<double>(pixels) * static_cast<double>(kFixedOne);
  const double mean[3] = {static_cast<double>(sum[0]) / n, static_cast<double>(sum[1]) / n,
                          static_cast<double>(sum[2]) / n};
  const double luma = 0.2126 * mean[0] + 0.7152 * mean[1] + 0.0722 * mean[2];
  double error = luma > 0.0 ? log2(static_cast<double>(p.ae.target) / luma) : 8.0;
  error = error < -8.0 ? -8.0 : error > 8.0 ? 8.0 : error;
  const double scale = exp2(static_cast<double>(p.ae.damping) * error);
  double next_exposure = 0.0;
  double next_gain = 0.0;
  if (p.exposure_ns > 0) {
    const double gain = p.exposure_gain > 0.0F ? p.exposure_gain : p.ae.min_gain;
    const double wanted = static_cast<double>(p.exposure_ns) * gain * scale;
    next_exposure = wanted / p.ae.min_gain;
    const double low = static_cast<double>(p.ae.min_exposure_ns);
    const double high = static_cast<double>(p.ae.max_exposure_ns);
    next_exposure = next_exposure < low ? low : next_exposure > high ? high : next_exposure;
    next_gain = wanted / next_exposure;
    next_gain = next_gain < p.ae.min_gain ? p.ae.min_gain : next_gain > p.ae.max_gain ? p.ae.max_gain : next_gain;
  }
  Span<float> out = p.stats_out;
  out[0] = static_cast<float>(mean[0]);
  out[1] = static_cast<float>(mean[1]);
  out[2] = static_cast<float>(mean[2]);
  out[3] = static_cast<float>(luma);
  out[4] = static_cast<float>(error);
  out[5] = static_cast<float>(scale);
  out[6] = static_cast<float>(next_exposure);
  out[7] = static_cast<float>(next_gain);
  out[8] = gains[0];
  out[9] = gains[1];
  out[10] = gains[2];
  out[11] = static_cast<float>(static_cast<double>(saturated) / static_cast<double>(pixels));
}

// ---- The fused tile pass --------------------------------------------------

// Per-tile state the phases share.
struct TileCtx {
  int x0, y0;
  Span<const uint8_t> box;
  Span<const int> col_mx;
  Span<const int> row_my;
  Span<const int> row_k;
  Span<const float> row_ty;
  Span<const float2> table;  // paired lens shading table
  Span<const float> grid;     // the frame's lens shading gains
  LscTile lt;
};

}  // namespace
}  // namespace isp_b200
