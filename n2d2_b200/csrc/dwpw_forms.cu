// The depthwise + 1x1 kernel with the 64-bit form of the rescale
#include "dwpw_kernel.cuh"

namespace n2d2b {

const DwPwKernel dwpw_wide[2] = {dwpw_i8_tcgen05_kernel<1, DPF_WIDE, DPF_WIDE>, dwpw_i8_tcgen05_kernel<2, DPF_WIDE, DPF_WIDE>};
const DwPwKernel dwpw_wide_1x1[2] = {dwpw_i8_tcgen05_kernel<1, DPF_CLAMP, DPF_WIDE>, dwpw_i8_tcgen05_kernel<2, DPF_CLAMP, DPF_WIDE>};
const DwPwKernel dwpw_wide_depthwise[2] = {dwpw_i8_tcgen05_kernel<1, DPF_WIDE, DPF_CLAMP>, dwpw_i8_tcgen05_kernel<2, DPF_WIDE, DPF_CLAMP>};

}  // namespace n2d2b
