// The patch kernel with the floating-point form of the rescale
#include "patch_kernel.cuh"

namespace n2d2b {

const PatchKernel patch_float[2][6] = N2D2B_PATCH_KERNELS(EF_FLOAT);

}  // namespace n2d2b
