// The pooled first layer with the 32-bit form of the rescale
#include "stem_pool_kernel.cuh"

namespace n2d2b {

const StemPoolKernel stem_pool_int[2][3][4] = N2D2B_STEM_POOL_KERNELS(false, 0);
const StemPoolKernel stem_pool_int_clamped[2][3][4] = N2D2B_STEM_POOL_KERNELS(true, 0);

}  // namespace n2d2b
