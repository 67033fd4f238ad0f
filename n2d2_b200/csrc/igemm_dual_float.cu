// A branch, its projection and their sum with the floating-point form of the rescale (which has no dot-product sum)
#include "igemm_dual_kernel.cuh"

namespace n2d2b {

const DualKernel dual_float[3] = {igemm_dual_tcgen05_kernel<2, DUAL_FLOAT>, igemm_dual_tcgen05_kernel<4, DUAL_FLOAT>, nullptr};

}  // namespace n2d2b
