// A branch, its projection and their sum where one of them has the 64-bit form of the rescale or their forms differ
#include "igemm_dual_kernel.cuh"

namespace n2d2b {

const DualKernel dual_any[3] = {igemm_dual_tcgen05_kernel<2, DUAL_ANY>, igemm_dual_tcgen05_kernel<4, DUAL_ANY>, igemm_dual_tcgen05_kernel<5, DUAL_ANY>};

}  // namespace n2d2b
