// cc_resample_planar.cu - resample kernels of the planar YCbCr sources.
#include "cc_resample.cuh"

namespace cc_b200 {

const void* resample_kernel_planar(int src, int mode, const ResampleKey& key) {
  switch (src) {
    case CC_NV12: return resample_for<CC_NV12>(mode, key);
    case CC_NV16: return resample_for<CC_NV16>(mode, key);
    case CC_I420: return resample_for<CC_I420>(mode, key);
    default: return nullptr;
  }
}

}  // namespace cc_b200
