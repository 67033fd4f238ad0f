// An expansion with its residual sum and the 1x1 layer behind it: the 64-bit form of the rescale in one of its two layers, or different forms
#include "igemm_chain_kernel.cuh"

namespace n2d2b {

const ChainKernel chain_any[3] = {igemm_chain_tcgen05_kernel<2, CHAIN_ANY>, igemm_chain_tcgen05_kernel<4, CHAIN_ANY>, igemm_chain_tcgen05_kernel<5, CHAIN_ANY>};

}  // namespace n2d2b
