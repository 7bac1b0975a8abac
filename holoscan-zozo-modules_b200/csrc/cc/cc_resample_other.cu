// cc_resample_other.cu - resample kernels of the gray and 16-bit sources.
#include "cc_resample.cuh"

namespace cc_b200 {

const void* resample_kernel_other(int src, int mode, const ResampleKey& key) {
  switch (src) {
    case CC_MONO8: return resample_for<CC_MONO8>(mode, key);
    case CC_MONO16: return resample_for<CC_MONO16>(mode, key);
    case CC_RGB16: return resample_for<CC_RGB16>(mode, key);
    default: return nullptr;
  }
}

}  // namespace cc_b200
