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

// One raw sample's counts (view_op.cu:35-51; isp_math.hpp:101-119).
__device__ __forceinline__ int view_sample(const uint8_t* row, int format, int x) {
  switch (format) {
    case ISP_RAW_U8: return __ldg(row + x);
    case ISP_RAW_U16: return __ldg(row + 2 * x) | (__ldg(row + 2 * x + 1) << 8);
    case ISP_RAW_RAW10: {
      const uint8_t* g = row + 5 * (x >> 2);
      return (__ldg(g + (x & 3)) << 2) | ((__ldg(g + 4) >> (2 * (x & 3))) & 3);
    }
    default: {
      const uint8_t* g = row + 3 * (x >> 1);
      return (__ldg(g + (x & 1)) << 4) | ((__ldg(g + 2) >> (4 * (x & 1))) & 15);
    }
  }
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

// 32-bit words of sixteen samples.
__host__ __device__ constexpr int run_words(int format) {
  return format == ISP_RAW_U8 ? 4 : format == ISP_RAW_U16 ? 8 : format == ISP_RAW_RAW10 ? 5 : 6;
}

// The sixteen samples of a run's words. Packed formats as in load_raw: RAW10
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

// A warp takes `tiles` of 32 runs of 16 pixels (tiles_x across the frame's
// runs_x runs), striding over the frame with the grid's other warps. Where the
// rows allow it (16-byte aligned RGB and view rows, 4-byte aligned raw rows)
// whole runs move as described above; a row's last, shorter run and the runs of
// other rows byte by byte.
template <int kFormat, bool kTable>
__global__ void __launch_bounds__(kViewThreads) isp_view_kernel(const __grid_constant__ ViewArgs a, int runs_x, int tiles_x,
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
    const int whole = vec ? min(a.width / kRun - run0, 32) : 0;  // the tile's runs moved as words
    if (whole > 0) {
      const uint32_t* from = reinterpret_cast<const uint32_t*>(raw) + static_cast<size_t>(run0) * kWords;
      const uint4* pixels = reinterpret_cast<const uint4*>(rgb) + static_cast<size_t>(run0) * 3;
      uint4* beside = reinterpret_cast<uint4*>(right) + static_cast<size_t>(run0) * 3;
      uint4* below = reinterpret_cast<uint4*>(left) + static_cast<size_t>(run0) * 3;
      uint32_t w[kWords];
#pragma unroll
      for (int k = 0; k < kWords; ++k) w[k] = lane + 32 * k < whole * kWords ? __ldg(from + lane + 32 * k) : 0U;
      uint4 c[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) c[k] = lane + 32 * k < 3 * whole ? __ldg(pixels + lane + 32 * k) : make_uint4(0U, 0U, 0U, 0U);
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
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (lane + 32 * k < 3 * whole) beside[lane + 32 * k] = c[k];
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
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (lane + 32 * k < 3 * whole) below[lane + 32 * k] = stage[lane + 32 * k];
      }
      __syncwarp();
    }
    if (lane >= whole && run0 + lane < runs_x) {
      const int x0 = kRun * (run0 + lane);
      const int x1 = min(x0 + kRun, a.width);
      for (int x = x0; x < x1; ++x) {
        const uint8_t g = static_cast<uint8_t>(gray(static_cast<uint32_t>(view_sample(raw, kFormat, x))));
        left[3 * static_cast<size_t>(x)] = left[3 * static_cast<size_t>(x) + 1] = left[3 * static_cast<size_t>(x) + 2] = g;
#pragma unroll
        for (int k = 0; k < 3; ++k) right[3 * static_cast<size_t>(x) + k] = __ldg(rgb + 3 * static_cast<size_t>(x) + k);
      }
    }
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
  constexpr int64_t kBlocksPerSm = 5;
  constexpr int64_t kWarps = kViewThreads / 32;
  int runs_x = (raw->width + kRun - 1) / kRun;
  int tiles_x = (runs_x + 31) / 32;
  const int64_t total = static_cast<int64_t>(tiles_x) * raw->height;
  const int64_t needed = (total + kWarps - 1) / kWarps;
  const int64_t rounds = (needed + shapes.sm_count * kBlocksPerSm - 1) / (shapes.sm_count * kBlocksPerSm);
  const int64_t blocks = (needed + rounds - 1) / rounds;
  // The table costs each thread table_size / 256 codes; a 12-bit one pays from
  // the second round on (of two: 16 codes instead of 32). Every sample a packed
  // format can hold has its entry, whatever the bit depth.
  int table_size = 1 << (raw->format == ISP_RAW_U16 ? raw->bit_depth : max_bits);
  const bool table = table_size <= kTableMax && (table_size <= 1024 || rounds >= 2);
  int tiles = static_cast<int>(total);
  void* args[] = {&a, &runs_x, &tiles_x, &tiles, &table_size};
  e = launch_dependent(view_kernel(raw->format, table), dim3(static_cast<unsigned>(blocks)), dim3(kViewThreads), args,
                       static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return fail_cuda(e, "view kernel");
  return ISP_OK;
}
