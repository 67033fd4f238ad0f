// An expansion with its residual sum and the 1x1 layer behind it: the floating-point form of the rescale (which has no dot-product sum)
#include "igemm_chain_kernel.cuh"

namespace n2d2b {

const ChainKernel chain_float[3] = {igemm_chain_tcgen05_kernel<2, CHAIN_FLOAT>, igemm_chain_tcgen05_kernel<4, CHAIN_FLOAT>, nullptr};

}  // namespace n2d2b
