// isp_awb.cu - the white balance statistics kernel of the B200 ISP
// (gray world and white patch): each CTA takes one band of a 64-column strip,
// whose tiles of 64x64 samples arrive by TMA; the complete 2x2 quads without
// a saturated sample are summed per colour (and binned for white patch) in
// the block, then flushed once; the last CTA to finish forms the frame's
// estimate (finish_white_balance, isp_math.hpp:357-384) and clears the sums
// for the next frame.
#include "isp_awb.cuh"

namespace isp_b200 {
namespace {

// One CTA per band of a strip: columns [64 s, 64 s + 64) of the complete
// quads, tiles [b band_tiles, (b + 1) band_tiles) of 64 rows. The band's lens
// shading maps and table are built once; its tiles then stream through a
// double-buffered TMA box with one block barrier each (buffer reuse).
template <bool kWhitePatch, int kPat>
__global__ void __launch_bounds__(kThreads, 3) isp_awb_kernel(const __grid_constant__ CUtensorMap map, FrameDesc p,
                                                         int strips, int tiles_y, int band_tiles, int use_tma) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128U - (smem_u32(smem_raw) & 127U)) & 127U);
  constexpr int kBoxRows = 64;
  const AwbSmem m = carve_awb(smem, span_rec(p.scratch));
  const Span<uint8_t> boxes = m.boxes;
  const Span<unsigned int> hist = m.hist;
  __shared__ uint64_t bars[2];
  __shared__ u64 red[4 * kWarps];
  __shared__ int minmax[2];
  __shared__ bool last;
  Span<Scratch> s = p.scratch;
  const int tid = threadIdx.x;
  const int box_bytes = awb_box_bytes(p.raw_format);
  // The tile pass that follows may launch now: it waits (griddepcontrol.wait)
  // for this grid's completion before it does anything, but its CTAs become
  // resident on the SMs this pass leaves while the last bands are summed.
  griddep_launch_dependents();
  if constexpr (kWhitePatch) {
    for (int i = tid; i < 3 * kAwbBins; i += kThreads) hist[i] = 0U;
  }
  // The lens shading gains in shared memory for the frame, when they fit.
  Span<const float> grid = p.lsc;
  const int gains = p.lsc_width * p.lsc_height * p.lsc_channels;
  if (p.lsc != nullptr && gains <= kGridSmemGains) {
    for (int i = tid; i < gains; i += kThreads) cp_async4(&m.grid[i], &p.lsc[i]);
    grid = m.grid;
  }
  if (tid == 0 && use_tma) {
    mbar_init(&bars[0]);
    mbar_init(&bars[1]);
  }
  float black[4], inv[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    black[k] = p.black[cfa_of(kPat, k)];
    inv[k] = p.inv_range[cfa_of(kPat, k)];
  }
  const int strip = static_cast<int>(blockIdx.x) % strips;
  const int ty0 = (static_cast<int>(blockIdx.x) / strips) * band_tiles;
  const int ty1 = min(ty0 + band_tiles, tiles_y);
  const int x0 = strip * 64;
  const auto issue = [&](int ty, int b) {
    if (!use_tma) {
      fill_box(p, boxes + b * 64 * 128, box_bytes, kBoxRows,
               awb_box_x(p.raw_format, x0) * (p.raw_format == kRawU16 ? 2 : 1), ty * 64);
    } else if (tid == 0) {
      fence_async_shared();
      tma_load_2d(&map, boxes + b * 64 * 128, &bars[b], awb_box_x(p.raw_format, x0), ty * 64,
                  static_cast<unsigned int>(kBoxRows * box_bytes));
    }
  };
  cp_async_wait_all();
  __syncthreads();  // barriers initialised, the gains in shared memory
  if (ty0 < ty1) issue(ty0, 0);
  // The band's maps and table (block-synchronised inside), while the first
  // box is in flight.
  const LscTile lt = build_band_lsc(p, grid, kPat, x0, ty0 * 64, (ty1 - ty0) * 64, m, minmax);
  u64 acc[4] = {0, 0, 0, 0};
  uint32_t phases = 0;  // bit b: parity of buffer b's next completion
  AwbCell cell;
  for (int ty = ty0; ty < ty1; ++ty) {
    const int buf = (ty - ty0) & 1;
    if (!use_tma) {
      box_filled();
      __syncthreads();
    }
    // The other buffer was read by the previous tile (the block synchronised
    // since): load the next tile into it while this one is summed.
    if (ty + 1 < ty1) issue(ty + 1, buf ^ 1);
    if (use_tma && !mbar_wait(&bars[buf], (phases >> buf) & 1U)) {
      if (tid == 0) report_wait_timeout(s);
    }
    phases ^= 1U << buf;
    const int rows = (ty - ty0) * 64;  // the tile's first row within the band
    unsigned int sum[3] = {0U, 0U, 0U};
    unsigned int quads = 0;
    awb_tile<kWhitePatch, kPat>(p, grid, boxes + buf * 64 * 128, box_bytes, x0, ty * 64, lt, m.row_k + rows, m.row_ty + rows,
                                m.table, black, inv, hist, cell, sum, quads);
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[k] += sum[k];
    acc[3] += quads;
    __syncthreads();
  }
  awb_flush<true>(p, acc, hist, kWhitePatch, red, &last, static_cast<unsigned int>(ty1 > ty0 ? ty1 - ty0 : 0),
            static_cast<unsigned int>(strips * tiles_y));
}

template <bool kWhitePatch>
const void* awb_by_pattern(int pattern) {
  switch (pattern) {
    case 0: return reinterpret_cast<const void*>(&isp_awb_kernel<kWhitePatch, 0>);
    case 1: return reinterpret_cast<const void*>(&isp_awb_kernel<kWhitePatch, 1>);
    case 2: return reinterpret_cast<const void*>(&isp_awb_kernel<kWhitePatch, 2>);
    default: return reinterpret_cast<const void*>(&isp_awb_kernel<kWhitePatch, 3>);
  }
}

}  // namespace

const void* awb_kernel(bool white_patch, int pattern) {
  return white_patch ? awb_by_pattern<true>(pattern) : awb_by_pattern<false>(pattern);
}

}  // namespace isp_b200
