// Instantiations of the persistent convolution kernel: output channels not a multiple of 16.
#include "conv_igemm_kernel.cuh"

namespace b200 {

IgemmKernel igemm_kernel_ragged(int epi, bool two_pipelines)
{
    switch (epi) {
    case kEpiFpOne: return two_pipelines ? conv_igemm_i8_kernel<kEpiFpOne, false, false, 1> : conv_igemm_i8_kernel<kEpiFpOne, false, false, 0>;
    case kEpiFpOneFull: return two_pipelines ? conv_igemm_i8_kernel<kEpiFpOneFull, false, false, 1> : conv_igemm_i8_kernel<kEpiFpOneFull, false, false, 0>;
    case kEpiFpMany: return two_pipelines ? conv_igemm_i8_kernel<kEpiFpMany, false, false, 1> : conv_igemm_i8_kernel<kEpiFpMany, false, false, 0>;
    case kEpiFpManyFull: return two_pipelines ? conv_igemm_i8_kernel<kEpiFpManyFull, false, false, 1> : conv_igemm_i8_kernel<kEpiFpManyFull, false, false, 0>;
    case kEpiIntOne: return two_pipelines ? conv_igemm_i8_kernel<kEpiIntOne, false, false, 1> : conv_igemm_i8_kernel<kEpiIntOne, false, false, 0>;
    case kEpiIntOneFull: return two_pipelines ? conv_igemm_i8_kernel<kEpiIntOneFull, false, false, 1> : conv_igemm_i8_kernel<kEpiIntOneFull, false, false, 0>;
    case kEpiIntMany: return two_pipelines ? conv_igemm_i8_kernel<kEpiIntMany, false, false, 1> : conv_igemm_i8_kernel<kEpiIntMany, false, false, 0>;
    case kEpiIntManyFull: return two_pipelines ? conv_igemm_i8_kernel<kEpiIntManyFull, false, false, 1> : conv_igemm_i8_kernel<kEpiIntManyFull, false, false, 0>;
    case kEpiAny: return two_pipelines ? conv_igemm_i8_kernel<kEpiAny, false, false, 1> : conv_igemm_i8_kernel<kEpiAny, false, false, 0>;
    default: return nullptr;
    }
}

}  // namespace b200
