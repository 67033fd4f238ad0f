// Implicit GEMM of packed 4-bit weights
#include "igemm_kernel.cuh"

namespace n2d2b {

const IgemmKernel igemm_w4_kernels[6] = {igemm_i8_tcgen05_kernel<0, true, false>, igemm_i8_tcgen05_kernel<1, true, false>,
                                         igemm_i8_tcgen05_kernel<2, true, false>, igemm_i8_tcgen05_kernel<3, true, false>,
                                         igemm_i8_tcgen05_kernel<4, true, false>, igemm_i8_tcgen05_kernel<5, true, false>};

}  // namespace n2d2b
