// Instantiations of the persistent convolution kernel: tile by tile.
#include "conv_igemm_kernel.cuh"

namespace b200 {

IgemmKernel igemm_kernel_mode0(int epi)
{
    switch (epi) {
    case kEpiFpOne: return conv_igemm_i8_kernel<kEpiFpOne, false, false, 0, false>;
    case kEpiFpOneFull: return conv_igemm_i8_kernel<kEpiFpOneFull, false, false, 0, false>;
    case kEpiFpMany: return conv_igemm_i8_kernel<kEpiFpMany, false, false, 0, false>;
    case kEpiFpManyFull: return conv_igemm_i8_kernel<kEpiFpManyFull, false, false, 0, false>;
    case kEpiIntOne: return conv_igemm_i8_kernel<kEpiIntOne, false, false, 0, false>;
    case kEpiIntOneFull: return conv_igemm_i8_kernel<kEpiIntOneFull, false, false, 0, false>;
    case kEpiIntMany: return conv_igemm_i8_kernel<kEpiIntMany, false, false, 0, false>;
    case kEpiIntManyFull: return conv_igemm_i8_kernel<kEpiIntManyFull, false, false, 0, false>;
    case kEpiAny: return conv_igemm_i8_kernel<kEpiAny, false, false, 0, false>;
    default: return nullptr;
    }
}

}  // namespace b200
