// cc_direct_gray.cu - direct-path kernels (same-size conversions) of the
// MONO8, MONO16 and RGB16 sources into every destination format;
// split from the other source formats so that they compile in parallel.
#include "cc_direct.cuh"

namespace cc_b200 {
namespace {

template <int kSrc>
const void* for_destination(int dst, bool wide) {
  switch (dst) {
    case CC_NV12: return direct_instance<kSrc, CC_NV12>(wide);
    case CC_NV16: return direct_instance<kSrc, CC_NV16>(wide);
    case CC_I420: return direct_instance<kSrc, CC_I420>(wide);
    case CC_YUYV: return direct_instance<kSrc, CC_YUYV>(wide);
    case CC_UYVY: return direct_instance<kSrc, CC_UYVY>(wide);
    case CC_RGB8: return direct_instance<kSrc, CC_RGB8>(wide);
    case CC_BGR8: return direct_instance<kSrc, CC_BGR8>(wide);
    case CC_RGBA8: return direct_instance<kSrc, CC_RGBA8>(wide);
    case CC_BGRA8: return direct_instance<kSrc, CC_BGRA8>(wide);
    case CC_MONO8: return direct_instance<kSrc, CC_MONO8>(wide);
    case CC_MONO16: return direct_instance<kSrc, CC_MONO16>(wide);
    case CC_RGB16: return direct_instance<kSrc, CC_RGB16>(wide);
    default: return nullptr;
  }
}

}  // namespace

const void* direct_kernel_gray(int src, int dst, bool wide) {
  switch (src) {
    case CC_MONO8: return for_destination<CC_MONO8>(dst, wide);
    case CC_MONO16: return for_destination<CC_MONO16>(dst, wide);
    case CC_RGB16: return for_destination<CC_RGB16>(dst, wide);
    default: return nullptr;
  }
}

}  // namespace cc_b200
