// cc_resample_packed.cu - resample kernels of the packed YCbCr sources.
#include "cc_resample.cuh"

namespace cc_b200 {

const void* resample_kernel_packed(int src, int mode, const ResampleKey& key) {
  switch (src) {
    case CC_YUYV: return resample_for<CC_YUYV>(mode, key);
    case CC_UYVY: return resample_for<CC_UYVY>(mode, key);
    default: return nullptr;
  }
}

}  // namespace cc_b200
