// First layer by space-to-depth with a pooling of its bytes behind it
#include "stem_s2d_kernel.cuh"

namespace n2d2b {

const StemS2dKernel stem_s2d_pool_kernels[6][3] = N2D2B_STEM_S2D_KERNELS(true);

}  // namespace n2d2b
