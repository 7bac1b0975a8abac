// isp_view.cu - the demo's side-by-side view of raw and processed frames
// (applications/isp/src/view_op.cu:35-75), as a headless device image: the
// raw mosaic as square-rooted gray on the left, the ISP's RGB8 image on the
// right. One thread converts a run of sixteen pixels of a row.
//
// The bytes that move (9 per pixel and the raw frame) take 13.2 us of a
// 3840x2160 RAW10 frame at the measured copy bandwidth. What kept the kernel at
// twice that was instruction issue (71 % of the slots, 62 instructions per
// pixel: two byte loads and an exact square root for every sample), so that
//   - a warp takes 32 runs of a row and moves their bytes in whole, contiguous
//     words of the row: the RGB pixels straight across, the raw samples and the
//     gray pixels by way of shared memory (three 16-byte accesses 48 bytes apart
//     per thread left the load and store units the limit);
//   - the gray codes of 8- to 12-bit samples, at most 4096 of them, are worked
//     out once per block into shared memory, and blocks stay for several rows
//     (kTableMax; deeper samples are computed one by one).
// The frame then takes 16.0 us, of 24.7.
#include <cuda_runtime.h>

#include <string>

#include "isp_host.hpp"
#include "isp_ops.cuh"
#include "isp_trace.hpp"

namespace isp_b200 {
namespace {

struct ViewArgs {
  const uint8_t* raw;
  size_t raw_pitch;
  int width, height, format;
  float black, scale;
  const uint8_t* rgb;
  size_t rgb_pitch;
  uint8_t* out;
  size_t out_pitch;
};

// Bytes of n samples of a row, from a run's start.
template <int kFormat>
__device__ __forceinline__ int raw_bytes(int n) {
  return kFormat == ISP_RAW_U8 ? n : kFormat == ISP_RAW_U16 ? 2 * n : kFormat == ISP_RAW_RAW10 ? (n + 3) / 4 * 5 : (n + 1) / 2 * 3;
}

// The gray code of one sample: (s - black) * scale clamped to [0, 1], its
// square root, times 255, plus 0.5, truncated; every step rounded once.
__device__ __forceinline__ uint32_t view_gray(int s, float black, float scale) {
  float v = __fmul_rn(__fsub_rn(static_cast<float>(s), black), scale);
  v = v < 0.0F ? 0.0F : (v > 1.0F ? 1.0F : v);
  return __float2uint_rz(__fadd_rn(__fmul_rn(__fsqrt_rn(v), 255.0F), 0.5F));
}

constexpr int kRun = 16;             // pixels of a thread
constexpr int kTableMax = 4096;      // gray codes kept per block
constexpr int kViewThreads = 256;
constexpr int kViewBlocksPerSm = 5;

// 32-bit words of sixteen samples.
__host__ __device__ constexpr int run_words(int format) {
  return format == ISP_RAW_U8 ? 4 : format == ISP_RAW_U16 ? 8 : format == ISP_RAW_RAW10 ? 5 : 6;
}

// The sixteen samples of a run's words (view_op.cu:35-51; isp_math.hpp:101-119). Packed formats as in load_raw: RAW10
// holds four pixels in five bytes, RAW12 two in three.
template <int kFormat>
__device__ __forceinline__ void view_samples(const uint32_t (&w)[run_words(kFormat)], uint32_t (&s)[kRun]) {
  const auto byte_of = [&](int i) { return (w[i >> 2] >> (8 * (i & 3))) & 0xFFU; };
#pragma unroll
  for (int i = 0; i < kRun; ++i) {
    if constexpr (kFormat == ISP_RAW_U8) {
      s[i] = byte_of(i);
    } else if constexpr (kFormat == ISP_RAW_U16) {
      s[i] = (w[i >> 1] >> (16 * (i & 1))) & 0xFFFFU;
    } else if constexpr (kFormat == ISP_RAW_RAW10) {
      const int g = 5 * (i >> 2);
      s[i] = (byte_of(g + (i & 3)) << 2) | ((w[(g + 4) >> 2] >> (8 * ((g + 4) & 3) + 2 * (i & 3))) & 3U);
    } else {
      const int g = 3 * (i >> 1);
      s[i] = (byte_of(g + (i & 1)) << 4) | ((w[(g + 2) >> 2] >> (8 * ((g + 2) & 3) + 4 * (i & 1))) & 15U);
    }
  }
}

// The 32-bit word at any address, from the aligned words that hold its bytes.
__device__ __forceinline__ uint32_t word_at(const uint8_t* p) {
  const unsigned int s = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(p)) & 3U;
  const uint32_t* base = reinterpret_cast<const uint32_t*>(p - s);
  return __funnelshift_r(__ldg(base), s != 0U ? __ldg(base + 1) : 0U, 8U * s);
}

// A warp writes `bytes` bytes at dst, wherever it starts: aligned words from
// word(offset), the few bytes before and after them from byte(offset).
template <class Word, class Byte>
__device__ __forceinline__ void put_bytes(uint8_t* dst, int bytes, Word word, Byte byte) {
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int head = min(static_cast<int>(-reinterpret_cast<uintptr_t>(dst) & 3U), bytes);
  const int n = (bytes - head) >> 2;
  const int end = head + 4 * n;
#pragma unroll 2
  for (int j = lane; j < n; j += 32) *reinterpret_cast<uint32_t*>(dst + head + 4 * j) = word(head + 4 * j);
  if (lane < head) dst[lane] = byte(lane);
  if (lane < bytes - end) dst[end + lane] = byte(end + lane);
}

// A warp takes `tiles` of 32 runs of 16 pixels (tiles_x across the frame's
// width), striding over the frame with the grid's other warps. Where the rows
// allow it (16-byte aligned RGB and view rows, 4-byte aligned raw rows) the
// runs move as 16-byte words; elsewhere as the aligned 4-byte words that hold
// them, shifted on the way (1646x1647 U8: 116 us pixel by pixel, 12 now; 3119x2338
// RAW12 267 and 22 us).
template <int kFormat, bool kTable>
__global__ void __launch_bounds__(kViewThreads, kViewBlocksPerSm) isp_view_kernel(const __grid_constant__ ViewArgs a, int tiles_x,
                                                                int tiles, int table_size) {
  constexpr int kWords = run_words(kFormat);
  __shared__ uint8_t table[kTable ? kTableMax : 4];
  __shared__ uint4 staged[kViewThreads / 32][96];  // a tile's gray pixels; its raw words before them
  // A programmatic dependent (launch_dependent): no global memory before the wait.
  griddep_launch_dependents();
  if constexpr (kTable) {
    for (int i = threadIdx.x; i < table_size; i += kViewThreads) table[i] = static_cast<uint8_t>(view_gray(i, a.black, a.scale));
    __syncthreads();
  }
  griddep_wait();
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const int warp = static_cast<int>(threadIdx.x) >> 5;
  uint4* const stage = staged[warp];
  uint32_t* const words = reinterpret_cast<uint32_t*>(stage);
  const auto gray = [&](uint32_t s) -> uint32_t {
    if constexpr (kTable) {
      // A 16-bit container may hold more than its bit depth says.
      if (kFormat != ISP_RAW_U16 || s < static_cast<uint32_t>(table_size)) return table[s];
    }
    return view_gray(static_cast<int>(s), a.black, a.scale);
  };
  constexpr int kWarps = kViewThreads / 32;
  for (int tile = static_cast<int>(blockIdx.x) * kWarps + warp; tile < tiles; tile += static_cast<int>(gridDim.x) * kWarps) {
    const int y = tile / tiles_x;
    const int run0 = 32 * (tile - y * tiles_x);
    const uint8_t* raw = a.raw + static_cast<size_t>(y) * a.raw_pitch;
    const uint8_t* rgb = a.rgb + static_cast<size_t>(y) * a.rgb_pitch;
    uint8_t* left = a.out + static_cast<size_t>(y) * a.out_pitch;
    uint8_t* right = left + 3 * static_cast<size_t>(a.width);
    const bool vec = ((reinterpret_cast<uintptr_t>(rgb) | reinterpret_cast<uintptr_t>(left) |
                       reinterpret_cast<uintptr_t>(right)) & 15U) == 0U && (reinterpret_cast<uintptr_t>(raw) & 3U) == 0U;
    const int pixels_here = min(a.width - kRun * run0, 32 * kRun);
    const int whole = pixels_here / kRun;  // all of the tile's, where vec
    raw += static_cast<size_t>(run0) * (4 * kWords);
    rgb += static_cast<size_t>(run0) * (3 * kRun);
    left += static_cast<size_t>(run0) * (3 * kRun);
    right += static_cast<size_t>(run0) * (3 * kRun);
    const uint4* pixels = reinterpret_cast<const uint4*>(rgb);
    uint4* beside = reinterpret_cast<uint4*>(right);
    uint4* below = reinterpret_cast<uint4*>(left);
    uint32_t w[kWords];
    uint4 c[3];
    if (vec) {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(raw);
#pragma unroll
      for (int k = 0; k < kWords; ++k) w[k] = lane + 32 * k < whole * kWords ? __ldg(from + lane + 32 * k) : 0U;
#pragma unroll
      for (int k = 0; k < 3; ++k) c[k] = lane + 32 * k < 3 * whole ? __ldg(pixels + lane + 32 * k) : make_uint4(0U, 0U, 0U, 0U);
    } else {
      // Aligned words that hold at least a byte of the row's; zeros past its end.
      const int bytes = raw_bytes<kFormat>(pixels_here);
      const unsigned int s = static_cast<unsigned int>(reinterpret_cast<uintptr_t>(raw)) & 3U;
      const uint32_t* from = reinterpret_cast<const uint32_t*>(raw - s);
#pragma unroll
      for (int k = 0; k < kWords; ++k) {
        const int i = lane + 32 * k;
        const uint32_t lo = 4 * i < bytes + static_cast<int>(s) ? __ldg(from + i) : 0U;
        const uint32_t hi = s != 0U && 4 * i + 4 < bytes + static_cast<int>(s) ? __ldg(from + i + 1) : 0U;
        w[k] = __funnelshift_r(lo, hi, 8U * s);
      }
    }
#pragma unroll
    for (int k = 0; k < kWords; ++k) words[lane + 32 * k] = w[k];
    __syncwarp();
    if constexpr (kWords % 4 == 0) {
#pragma unroll
      for (int k = 0; k < kWords / 4; ++k) {
        const uint4 v = stage[lane * (kWords / 4) + k];
        w[4 * k] = v.x;
        w[4 * k + 1] = v.y;
        w[4 * k + 2] = v.z;
        w[4 * k + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < kWords; ++k) w[k] = words[lane * kWords + k];
    }
    __syncwarp();
    if (vec) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (lane + 32 * k < 3 * whole) beside[lane + 32 * k] = c[k];
      }
    }
    uint32_t g[kRun];
    view_samples<kFormat>(w, g);
#pragma unroll
    for (int i = 0; i < kRun; ++i) g[i] = gray(g[i]);
    // Gray pixels: bytes g, g, g per pixel; four of them, a b c d, as the
    // words aaab bbcc cddd.
    uint32_t o[12];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      o[3 * k] = __byte_perm(g[4 * k], g[4 * k + 1], 0x4000U);
      o[3 * k + 1] = __byte_perm(g[4 * k + 1], g[4 * k + 2], 0x4400U);
      o[3 * k + 2] = __byte_perm(g[4 * k + 2], g[4 * k + 3], 0x4440U);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) stage[3 * lane + k] = make_uint4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
    __syncwarp();
    if (vec) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (lane + 32 * k < 3 * whole) below[lane + 32 * k] = stage[lane + 32 * k];
      }
    } else {
      put_bytes(right, 3 * pixels_here, [&](int at) { return word_at(rgb + at); }, [&](int at) { return __ldg(rgb + at); });
      put_bytes(
          left, 3 * pixels_here,
          [&](int at) {
            const int k = at >> 2;
            return (at & 3) == 0 ? words[k] : __funnelshift_r(words[k], words[k + 1], 8U * (static_cast<unsigned int>(at) & 3U));
          },
          [&](int at) { return static_cast<uint8_t>(words[at >> 2] >> (8 * (at & 3))); });
    }
    __syncwarp();
  }
}

const void* view_kernel(int format, bool table) {
  switch (format) {
    case ISP_RAW_U8: return reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_U8, true>);
    case ISP_RAW_U16:
      return table ? reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_U16, true>)
                   : reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_U16, false>);
    case ISP_RAW_RAW10: return reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_RAW10, true>);
    default:
      return table ? reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_RAW12, true>)
                   : reinterpret_cast<const void*>(&isp_view_kernel<ISP_RAW_RAW12, false>);
  }
}

}  // namespace
}  // namespace isp_b200

extern "C" ISP_B200_API int isp_b200_view_compose(const isp_raw_view_c* raw, float black_level, const void* rgb8,
                                                  size_t rgb8_pitch, void* view, size_t view_pitch, void* stream) {
  using namespace isp_b200;
  const TraceRange range("isp.view", kTraceKernel);
  clear_error();
  if (raw == nullptr || raw->data == nullptr || rgb8 == nullptr || view == nullptr) {
    return fail(ISP_EINVAL, "view_compose: a buffer is missing");
  }
  if (raw->width <= 0 || raw->height <= 0) return fail(ISP_EINVAL, "raw image size must be positive");
  if (raw->format < ISP_RAW_U8 || raw->format > ISP_RAW_RAW12) return fail(ISP_EINVAL, "unknown raw format");
  const int max_bits = raw->format == ISP_RAW_U8 ? 8 : raw->format == ISP_RAW_U16 ? 16 : raw->format == ISP_RAW_RAW10 ? 10 : 12;
  if (raw->bit_depth < 1 || raw->bit_depth > max_bits) {
    return fail(ISP_EINVAL, "raw bit depth " + std::to_string(raw->bit_depth) + " does not fit the raw format");
  }
  if (raw->pitch < raw_row_bytes(raw->format, raw->width)) return fail(ISP_EINVAL, "raw pitch is shorter than a row");
  const size_t rgb_row = 3 * static_cast<size_t>(raw->width);
  if (rgb8_pitch < rgb_row) return fail(ISP_EINVAL, "RGB8 pitch is shorter than a row");
  if (view_pitch < 2 * rgb_row) return fail(ISP_EINVAL, "view pitch is shorter than a row of the double-width image");
  // view_op.cu:143-149: white and the scale in single precision on the host.
  const float white = static_cast<float>((1U << static_cast<unsigned>(raw->bit_depth)) - 1U);
  ViewArgs a{static_cast<const uint8_t*>(raw->data), raw->pitch, raw->width, raw->height, raw->format, black_level,
             1.0F / (white - black_level), static_cast<const uint8_t*>(rgb8), rgb8_pitch,
             static_cast<uint8_t*>(view), view_pitch};
  // Rows beyond this were never taken (a grid of one block per eight rows).
  if ((static_cast<int64_t>(raw->height) + 7) / 8 > 65535) return fail_cuda(cudaErrorInvalidConfiguration, "view kernel");
  cudaError_t e = cudaSuccess;
  const LaunchShapes& shapes = shapes_for_current_device(&e);
  if (e != cudaSuccess) return fail_cuda(e, "view kernel");
  // As many blocks as are resident at once, each with the same number of
  // rounds over the frame's tiles.
  constexpr int64_t kWarps = kViewThreads / 32;
  int tiles_x = (raw->width + 32 * kRun - 1) / (32 * kRun);
  const int64_t total = static_cast<int64_t>(tiles_x) * raw->height;
  const int64_t needed = (total + kWarps - 1) / kWarps;
  const int64_t rounds = (needed + shapes.sm_count * int64_t{kViewBlocksPerSm} - 1) / (shapes.sm_count * int64_t{kViewBlocksPerSm});
  const int64_t blocks = (needed + rounds - 1) / rounds;
  // The table costs each thread table_size / 256 codes; a 12-bit one pays from
  // the second round on (of two: 16 codes instead of 32). Every sample a packed
  // format can hold has its entry, whatever the bit depth.
  int table_size = 1 << (raw->format == ISP_RAW_U16 ? raw->bit_depth : max_bits);
  const bool table = table_size <= kTableMax && (table_size <= 1024 || rounds >= 2);
  int tiles = static_cast<int>(total);
  void* args[] = {&a, &tiles_x, &tiles, &table_size};
  e = launch_dependent(view_kernel(raw->format, table), dim3(static_cast<unsigned>(blocks)), dim3(kViewThreads), args,
                       static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail_cuda(e, "view kernel");
  return ISP_OK;
}
