// Instantiations of the persistent convolution kernel: a fused residual add.
#include "conv_igemm_kernel.cuh"

namespace b200 {

IgemmKernel igemm_kernel_residual(int epi)
{
    switch (epi) {
    case kEpiFpOne: return conv_igemm_i8_kernel<kEpiFpOne, true, false, 0>;
    case kEpiFpMany: return conv_igemm_i8_kernel<kEpiFpMany, true, false, 0>;
    case kEpiIntOne: return conv_igemm_i8_kernel<kEpiIntOne, true, false, 0>;
    case kEpiIntMany: return conv_igemm_i8_kernel<kEpiIntMany, true, false, 0>;
    default: return nullptr;
    }
}

}  // namespace b200
