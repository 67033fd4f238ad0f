// The pooled first layer with the 64-bit form of the rescale
#include "stem_pool_kernel.cuh"

namespace n2d2b {

const StemPoolKernel stem_pool_wide[2][3][4] = N2D2B_STEM_POOL_KERNELS(false, EF_WIDE);
const StemPoolKernel stem_pool_wide_clamped[2][3][4] = N2D2B_STEM_POOL_KERNELS(true, EF_WIDE);

}  // namespace n2d2b
