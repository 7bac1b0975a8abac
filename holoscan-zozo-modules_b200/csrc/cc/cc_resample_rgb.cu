// cc_resample_rgb.cu - resample kernels of the three- and four-byte RGB sources.
#include "cc_resample.cuh"

namespace cc_b200 {

const void* resample_kernel_rgb(int src, int mode, const ResampleKey& key) {
  switch (src) {
    case CC_RGB8: return resample_for<CC_RGB8>(mode, key);
    case CC_BGR8: return resample_for<CC_BGR8>(mode, key);
    case CC_RGBA8: return resample_for<CC_RGBA8>(mode, key);
    case CC_BGRA8: return resample_for<CC_BGRA8>(mode, key);
    default: return nullptr;
  }
}

}  // namespace cc_b200
