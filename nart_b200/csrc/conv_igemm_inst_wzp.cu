// Instantiations of the persistent convolution kernel: a weight zero point other than 128.
#include "conv_igemm_kernel.cuh"

namespace b200 {

IgemmKernel igemm_kernel_wzp(int epi)
{
    switch (epi) {
    case kEpiFpOne: return conv_igemm_i8_kernel<kEpiFpOne, false, true, 0>;
    case kEpiFpOneFull: return conv_igemm_i8_kernel<kEpiFpOneFull, false, true, 0>;
    case kEpiFpMany: return conv_igemm_i8_kernel<kEpiFpMany, false, true, 0>;
    case kEpiFpManyFull: return conv_igemm_i8_kernel<kEpiFpManyFull, false, true, 0>;
    case kEpiIntOne: return conv_igemm_i8_kernel<kEpiIntOne, false, true, 0>;
    case kEpiIntOneFull: return conv_igemm_i8_kernel<kEpiIntOneFull, false, true, 0>;
    case kEpiIntMany: return conv_igemm_i8_kernel<kEpiIntMany, false, true, 0>;
    case kEpiIntManyFull: return conv_igemm_i8_kernel<kEpiIntManyFull, false, true, 0>;
    case kEpiAny: return conv_igemm_i8_kernel<kEpiAny, false, true, 0>;
    default: return nullptr;
    }
}

}  // namespace b200
