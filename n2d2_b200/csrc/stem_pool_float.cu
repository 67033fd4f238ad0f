// The pooled first layer with the floating-point form of the rescale
#include "stem_pool_kernel.cuh"

namespace n2d2b {

const StemPoolKernel stem_pool_float[2][3][4] = N2D2B_STEM_POOL_KERNELS(false, EF_FLOAT);
const StemPoolKernel stem_pool_float_clamped[2][3][4] = N2D2B_STEM_POOL_KERNELS(true, EF_FLOAT);

}  // namespace n2d2b
