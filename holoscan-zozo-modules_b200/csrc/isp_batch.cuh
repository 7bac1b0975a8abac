// isp_batch.cuh - frames of uneven size, format, Bayer pattern and settings
// in one launch per pass: the statistics pass over the auto-white-balance
// frames' tiles, then the tile pass over every frame's tiles.
//
// Each pass is a persistent kernel over a work list: CTA i owns the
// contiguous items ranges[i] (sized by the host so the estimated cost is
// even; the last part of the work is claimed range by range from a queue
// instead), walks them frame by frame, keeps the frame's FrameDesc and tone
// table in shared memory, prefetches the next item's raw box by TMA
// (whichever frame it belongs to), and flushes a frame's sums when it leaves
// it; the CTA that completes a frame's count of tiles finishes that frame
// (its statistics and histogram, or its white balance estimate). Every tile
// runs the same device code as the single-frame kernels (isp_main.cuh,
// isp_awb.cuh), so a frame's bytes are the same alone or in a batch.
#pragma once

#include "isp_awb.cuh"
#include "isp_bands.hpp"
#include "isp_main.cuh"

namespace isp_b200 {
namespace {

__device__ __forceinline__ void tensormap_acquire(const CUtensorMap* map) {
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map))
               : "memory");
}

// Copies a frame's FrameDesc to shared memory (all threads; the caller syncs).
__device__ __forceinline__ void load_desc(FrameDesc* dst, const FrameDesc* src) {
  constexpr int kWords = sizeof(FrameDesc) / 4;
  static_assert(sizeof(FrameDesc) % 4 == 0, "FrameDesc words");
  const unsigned int* s = reinterpret_cast<const unsigned int*>(src);
  unsigned int* d = reinterpret_cast<unsigned int*>(dst);
  for (int i = threadIdx.x; i < kWords; i += kThreads) d[i] = s[i];
}

// The frame holding work item `item`, searching forward from frame `from`.
__device__ __forceinline__ int frame_of_item(Span<const BatchFrame> frames, int nframes, int from, int item, bool awb) {
  int f = from;
  while (f + 1 < nframes && item >= (awb ? frames[f + 1].awb_begin : frames[f + 1].tile_begin)) ++f;
  return f;
}

// The queue's count and first: read once at a CTA's start, beside its own range,
// and kept in shared memory, since a read at each claim holds up the thread that
// claims, and the block behind it, for a round trip to L2.
__device__ __forceinline__ int2 queue_head(const BatchQueue* queue) { return make_int2(queue->count, queue->first); }

// The item after `item` for a CTA (one thread calls): the next of its range
// r, or the first of a range claimed from the queue, which is left in `claim`
// (empty when none is left). -1: none. Queued items come after every CTA's own,
// and claims only move forward.
__device__ __forceinline__ int next_item(BatchQueue* queue, int2 head, int item, int2 r, int2& claim, CheckRecord* rec) {
  if (item + 1 < r.y) return item + 1;
  claim = make_int2(0, 0);
  if (head.x > 0) {
    const unsigned int c = atomicAdd(&queue->claimed, 1U);
    if (c < static_cast<unsigned int>(head.x)) {
      const int2* entries = reinterpret_cast<const int2*>(queue) + head.y;
      claim = make_span(entries, static_cast<size_t>(head.x), rec)[static_cast<int>(c)];
    }
  }
  return claim.x < claim.y ? claim.x : -1;
}

// Adds a tile's four sums over the warp to the totals its lanes 0..3 keep: two
// registers a thread across the tiles instead of eight. A tile has at most
// 16 samples a thread of at most 2^22, so a warp's sum is below 2^32.
__device__ __forceinline__ void add_tile_sums(u64& acc, unsigned int a, unsigned int b, unsigned int c, unsigned int d) {
  a = __reduce_add_sync(0xffffffffU, a);
  b = __reduce_add_sync(0xffffffffU, b);
  c = __reduce_add_sync(0xffffffffU, c);
  d = __reduce_add_sync(0xffffffffU, d);
  const int lane = threadIdx.x & 31;
  const unsigned int lo = (lane & 1) ? b : a, hi = (lane & 1) ? d : c;
  acc += (lane & 2) ? hi : lo;
}

// The warp's totals as the flushes take them: per thread, summed over the block.
__device__ __forceinline__ void totals_of(u64 acc, u64 (&total)[4]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 4; ++k) total[k] = lane == k ? acc : 0;
}

// One tile of a frame of any settings (BatchFrame::variant). Only what differs
// between the variants is compiled per variant: the demosaics. With one copy
// of the whole tile per variant (eight, each with the finish of four output
// formats) the CTAs of an SM, at work on different variants, waited for
// instructions more than for anything else (1.3 of 7.4 cycles per
// instruction). kSharpen: whether any frame of the batch sharpens.
template <bool kLutSmem, int kTileH, bool kSharpen, class AfterA>
__device__ __forceinline__ void run_tile_any(const FrameDesc& p, const FrameSetup& f, const TileSmem& m, int* minmax,
                                             int variant, int x0, int y0, bool use_tma, uint64_t* bar, uint32_t& phase,
                                             u64& acc, AfterA after_a) {
  const bool sharpen = kSharpen && (variant & 2) != 0;
  unsigned int saturated = 0;
  const auto no_wait = [] {};
  if (kSharpen && sharpen) {
    saturated = tile_samples<Geom<true, kTileH>::kHalo, kTileH>(p, f, m, minmax, x0, y0, use_tma, bar, phase, no_wait);
  } else {
    saturated = tile_samples<Geom<false, kTileH>::kHalo, kTileH>(p, f, m, minmax, x0, y0, use_tma, bar, phase, no_wait);
  }
  __syncthreads();
  after_a();
  if (kSharpen && sharpen) {
    const Span<float2> red = f.swap_rb ? m.B : m.R, blue = f.swap_rb ? m.R : m.B;
    switch (variant) {
      case 2: phase_b2<false, 0, kTileH>(m.P, red, m.G, blue); break;
      case 3: phase_b2<true, 0, kTileH>(m.P, red, m.G, blue); break;
      case 6: phase_b2<false, 2, kTileH>(m.P, red, m.G, blue); break;
      default: phase_b2<true, 2, kTileH>(m.P, red, m.G, blue); break;
    }
    __syncthreads();
  }
  unsigned int sums[3] = {0U, 0U, 0U};
  unsigned int npix = 0;
#pragma unroll 1
  for (int k = 0; k < kTileH / 32; ++k) {
    int r, uc;
    unit_rc(threadIdx.x + k * kThreads, r, uc);
    float2 rgb[4][3];
    if (kSharpen && sharpen) {
      sharpened_row(m, r, uc, p.sharpen, rgb);
    } else {
      switch (variant) {
        case 0: demosaiced_row<false, 0>(m, r, uc, rgb); break;
        case 1: demosaiced_row<true, 0>(m, r, uc, rgb); break;
        case 4: demosaiced_row<false, 2>(m, r, uc, rgb); break;
        default: demosaiced_row<true, 2>(m, r, uc, rgb); break;
      }
      if (f.swap_rb) swap_red_blue(rgb);
    }
    finish_row<-1, kLutSmem>(p, f, m.hist, rgb, x0 + 4 * uc, y0 + r, sums, npix);
  }
  add_tile_sums(acc, sums[0] - npix * kTwo23Bits, sums[1] - npix * kTwo23Bits, sums[2] - npix * kTwo23Bits,
                saturated);  // mod 2^32: the true sums
  __syncthreads();  // the next tile overwrites the tables, P and the planes
}

// Without sharpening three CTAs share an SM (80 registers a thread, no RGB
// planes), with it two: the tile pass of a 48-camera batch took 1497 us at two
// with all its work dealt out, 1313 at three with the queue. The shared-memory
// pipe bounds it (73 % of its cycles: the planes, the tone table's gathers and
// the histogram's atomics).
template <bool kLutSmem, int kTileH, bool kSharpen>
__global__ void __launch_bounds__(kThreads, kSharpen && kTileH == kTH ? 2 : 3)
    isp_batch_kernel(const BatchFrame* frames_in, int nframes, const int2* ranges_in, BatchQueue* queue) {
  using GS = Geom<kSharpen, kTileH>;  // the sharpening geometry holds every variant's
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128U - (smem_u32(smem_raw) & 127U)) & 127U);
#ifdef ISP_CHECKED
  CheckRecord* const rec = span_rec(frames_in[0].desc.scratch);
#else
  CheckRecord* const rec = nullptr;
#endif
  const Span<const BatchFrame> frames = make_span(frames_in, static_cast<size_t>(nframes), rec);
  const Span<const int2> ranges = make_span(ranges_in, static_cast<size_t>(gridDim.x), rec);
  const TileSmem m =
      carve(smem, layout_of(kSharpen, box_row_bytes(kRawU16), kLutSmem ? kBatchLutEntries : 0, kTileH), GS::kSH, rec);
  __shared__ int2 next_range;
  __shared__ int2 head;
  __shared__ uint64_t bar;
  __shared__ u64 red[4 * kWarps];
  __shared__ int minmax[2];
  __shared__ bool last;
  __shared__ __align__(16) FrameDesc fd;
  // A programmatic dependent of the statistics batch: resident early, it
  // waits here for that batch's completion (and the gains it wrote).
  griddep_wait();
  const int2 queued = queue_head(queue);
  int2 r = ranges[blockIdx.x];
  if (r.x >= r.y) return;
  const int tid = threadIdx.x;
  if (tid == 0) {
    head = queued;
    mbar_init(&bar);
  }
  int f = frame_of_item(frames, nframes, 0, r.x, false);
  load_desc(&fd, &frames[f].desc);
  __syncthreads();
  setup_frame<kLutSmem>(fd, m);
  __syncthreads();

  const auto issue = [&](int g, int item) {
    const BatchFrame& bf = frames[g];
    const int local = item - bf.tile_begin;
    const int ty = local / bf.tiles_x;
    const int x0 = (local - ty * bf.tiles_x) * kTW;
    const int halo = (bf.variant & 2) ? 4 : 2;
    const int fmt = bf.desc.raw_format;
    tensormap_acquire(&bf.main_map);
    tma_load_2d(&bf.main_map, m.box, &bar, box_x(fmt, x0), ty * kTileH - halo,
                static_cast<unsigned int>((kTileH + 2 * halo) * box_row_bytes(fmt)));
  };
  if (tid == 0 && frames[f].use_tma) issue(f, r.x);
  uint32_t phase = 0;
  u64 acc = 0;
  unsigned int done = 0;
  const auto flush = [&] {
    u64 total[4];
    totals_of(acc, total);
    flush_frame(fd, frame_setup<kLutSmem>(fd, m), total, m, red, &last, done, static_cast<unsigned int>(frames[f].tiles));
  };
  int item = r.x;
  while (true) {
    if (item >= frames[f].tile_begin + frames[f].tiles) {
      flush();
      __syncthreads();
      f = frame_of_item(frames, nframes, f, item, false);
      load_desc(&fd, &frames[f].desc);
      __syncthreads();
      setup_frame<kLutSmem>(fd, m);
      __syncthreads();
      acc = 0;
      done = 0;
    }
    const BatchFrame& bf = frames[f];
    const int local = item - bf.tile_begin;
    const int ty = local / bf.tiles_x;
    const int x0 = (local - ty * bf.tiles_x) * kTW;
    const bool use_tma = bf.use_tma != 0;
    const auto prefetch = [&] {
      if (tid != 0) return;
      const int next = next_item(queue, head, item, r, next_range, rec);
      if (next < 0) return;
      const int g = frame_of_item(frames, nframes, f, next, false);
      if (frames[g].use_tma) {
        fence_async_shared();
        issue(g, next);
      }
    };
    run_tile_any<kLutSmem, kTileH, kSharpen>(fd, frame_setup<kLutSmem>(fd, m), m, minmax, bf.variant, x0, ty * kTileH, use_tma, &bar, phase, acc,
                                             prefetch);
    ++done;
    if (++item == r.y) {
      r = next_range;  // written before run_tile_any's closing barrier
      if (r.x >= r.y) break;
      item = r.x;
    }
  }
  flush();
}

// The statistics tile of a frame for its Bayer pattern and mode.
__device__ __forceinline__ void awb_tile_any(const FrameDesc& p, int pattern, bool white_patch, Span<const uint8_t> box,
                                             int box_bytes, int x0, int y0, const LscTile& lt, Span<const int> row_k,
                                             Span<const float> row_ty, Span<const float> table, const float (&black)[4],
                                             const float (&inv)[4], Span<unsigned int> hist, AwbCell& cell,
                                             unsigned int (&sum)[3], unsigned int& quads) {
#define ISP_AWB_CASE(P, W) \
  awb_tile<W, P>(p, p.lsc, box, box_bytes, x0, y0, lt, row_k, row_ty, table, black, inv, hist, cell, sum, quads)
  switch (pattern * 2 + (white_patch ? 1 : 0)) {
    case 0: ISP_AWB_CASE(0, false); break;
    case 1: ISP_AWB_CASE(0, true); break;
    case 2: ISP_AWB_CASE(1, false); break;
    case 3: ISP_AWB_CASE(1, true); break;
    case 4: ISP_AWB_CASE(2, false); break;
    case 5: ISP_AWB_CASE(2, true); break;
    case 6: ISP_AWB_CASE(3, false); break;
    default: ISP_AWB_CASE(3, true); break;
  }
#undef ISP_AWB_CASE
}

__global__ void __launch_bounds__(kThreads, 3) isp_awb_batch_kernel(const BatchFrame* frames_in, int nframes,
                                                               const int2* ranges_in, BatchQueue* queue) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((128U - (smem_u32(smem_raw) & 127U)) & 127U);
#ifdef ISP_CHECKED
  CheckRecord* const rec = span_rec(frames_in[0].desc.scratch);
#else
  CheckRecord* const rec = nullptr;
#endif
  const Span<const BatchFrame> frames = make_span(frames_in, static_cast<size_t>(nframes), rec);
  const Span<const int2> ranges = make_span(ranges_in, static_cast<size_t>(gridDim.x), rec);
  const AwbSmem m = carve_awb(smem, rec);
  const Span<uint8_t> boxes = m.boxes;
  const Span<unsigned int> hist = m.hist;
  __shared__ uint64_t bars[2];
  __shared__ u64 red[4 * kWarps];
  __shared__ int minmax[2];
  __shared__ bool last;
  __shared__ __align__(16) FrameDesc fd;
  griddep_launch_dependents();  // the tile batch may become resident as this one finishes
  __shared__ int2 next_range[2];
  __shared__ int2 head;
  const int2 queued = queue_head(queue);
  int2 r = ranges[blockIdx.x];
  if (r.x >= r.y) return;
  const int tid = threadIdx.x;
  if (tid == 0) {
    head = queued;
    mbar_init(&bars[0]);
    mbar_init(&bars[1]);
  }
  for (int i = tid; i < 3 * kAwbBins; i += kThreads) hist[i] = 0U;
  int f = frame_of_item(frames, nframes, 0, r.x, true);
  load_desc(&fd, &frames[f].desc);
  __syncthreads();
  const auto issue = [&](int g, int item, int b) {
    const BatchFrame& bf = frames[g];
    const int tiles_y = bf.awb_tiles / bf.awb_tiles_x;
    const int strip = (item - bf.awb_begin) / tiles_y;
    const int ty = item - bf.awb_begin - strip * tiles_y;
    const int x0 = strip * 64;
    const int fmt = bf.desc.raw_format;
    tensormap_acquire(&bf.awb_map);
    tma_load_2d(&bf.awb_map, boxes + b * 64 * 128, &bars[b], awb_box_x(fmt, x0), ty * 64,
                static_cast<unsigned int>(64 * awb_box_bytes(fmt)));
  };
  if (tid == 0 && frames[f].use_tma) issue(f, r.x, 0);
  // Items alternate between the buffers, whether or not their frame uses TMA,
  // so the prefetching thread and the waiting block always agree.
  uint32_t phases = 0;  // bit b: parity of buffer b's next completion
  u64 acc = 0;
  unsigned int done = 0;
  // Tiles run down the 64-column strips of a frame; the lens shading maps and
  // table are built for as many of a strip's next tiles as one table serves (a
  // band).
  int band_begin = 0, band_end = 0;
  LscTile lt{0, 0};
  AwbCell cell;
  const auto flush = [&] {
    u64 total[4];
    totals_of(acc, total);
    awb_flush(fd, total, hist, fd.awb_mode == kWbWhitePatch, red, &last, done,
              static_cast<unsigned int>(frames[f].awb_tiles));
  };
  int item = r.x;
  int buf = 0;
  while (true) {
    if (item >= frames[f].awb_begin + frames[f].awb_tiles) {
      flush();
      f = frame_of_item(frames, nframes, f, item, true);
      load_desc(&fd, &frames[f].desc);
      for (int i = tid; i < 3 * kAwbBins; i += kThreads) hist[i] = 0U;
      acc = 0;
      done = 0;
      __syncthreads();
    }
    const BatchFrame& bf = frames[f];
    // The other buffer was read by the previous item (the block synchronised
    // since): load the next item into it while this one is summed. The claimed
    // range's slot alternates too: the next claim may follow within the next
    // item, before every thread has read this one.
    if (tid == 0) {
      const int next = next_item(queue, head, item, r, next_range[buf], rec);
      if (next >= 0) {
        const int g = frame_of_item(frames, nframes, f, next, true);
        if (frames[g].use_tma) {
          fence_async_shared();
          issue(g, next, buf ^ 1);
        }
      }
    }
    const int tiles_y = bf.awb_tiles / bf.awb_tiles_x;
    const int strip = (item - bf.awb_begin) / tiles_y;
    const int ty = item - bf.awb_begin - strip * tiles_y;
    const int x0 = strip * 64;
    const int y0 = ty * 64;
    const bool use_tma = bf.use_tma != 0;
    const int box_bytes = awb_box_bytes(fd.raw_format);
    if (!use_tma) {
      fill_box(fd, boxes + buf * 64 * 128, box_bytes, 64, awb_box_x(fd.raw_format, x0) * (fd.raw_format == kRawU16 ? 2 : 1), y0);
    }
    if (item >= band_end) {
      band_begin = item;
      int most = min(min(tiles_y - ty, r.y - item), kAwbBandRows / 64);
      if (fd.lsc != nullptr) most = lsc_band_tiles(y0, most, fd.lsc_sy, fd.lsc_height, kLscTableRows);
      band_end = item + most;
      lt = build_band_lsc(fd, fd.lsc, fd.pattern, x0, y0, (band_end - band_begin) * 64, m, minmax);
      cell.k = -1;
    }
    const int rows = (item - band_begin) * 64;
    if (use_tma) {
      if (!mbar_wait(&bars[buf], (phases >> buf) & 1U) && tid == 0) report_wait_timeout(fd.scratch);
      phases ^= 1U << buf;
    } else {
      box_filled();
      __syncthreads();
    }
    float black[4], inv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      black[k] = fd.black[fd.cfa[k]];
      inv[k] = fd.inv_range[fd.cfa[k]];
    }
    unsigned int sum[3] = {0U, 0U, 0U};
    unsigned int quads = 0;
    awb_tile_any(fd, fd.pattern, fd.awb_mode == kWbWhitePatch, boxes + buf * 64 * 128, box_bytes, x0, y0, lt, m.row_k + rows,
                 m.row_ty + rows, m.table, black, inv, hist, cell, sum, quads);
    add_tile_sums(acc, sum[0], sum[1], sum[2], quads);
    __syncthreads();
    ++done;
    if (++item == r.y) {
      r = next_range[buf];
      if (r.x >= r.y) break;
      item = r.x;
    }
    buf ^= 1;
  }
  flush();
}

}  // namespace
}  // namespace isp_b200
