// The patch kernel with the 64-bit form of the rescale
#include "patch_kernel.cuh"

namespace n2d2b {

const PatchKernel patch_wide[2][6] = N2D2B_PATCH_KERNELS(EF_WIDE);

}  // namespace n2d2b
