// Instantiations of the persistent convolution kernel: one box of activations for all taps, two pipelines.
#include "conv_igemm_kernel.cuh"

namespace b200 {

template <bool WZP>
static IgemmBoxKernel pick(int epi)
{
    switch (epi) {
    case kEpiFpOne: return conv_igemm_i8_kernel<kEpiFpOne, false, WZP, 5, false>;
    case kEpiFpOneFull: return conv_igemm_i8_kernel<kEpiFpOneFull, false, WZP, 5, false>;
    case kEpiFpMany: return conv_igemm_i8_kernel<kEpiFpMany, false, WZP, 5, false>;
    case kEpiFpManyFull: return conv_igemm_i8_kernel<kEpiFpManyFull, false, WZP, 5, false>;
    case kEpiIntOne: return conv_igemm_i8_kernel<kEpiIntOne, false, WZP, 5, false>;
    case kEpiIntOneFull: return conv_igemm_i8_kernel<kEpiIntOneFull, false, WZP, 5, false>;
    case kEpiIntMany: return conv_igemm_i8_kernel<kEpiIntMany, false, WZP, 5, false>;
    case kEpiIntManyFull: return conv_igemm_i8_kernel<kEpiIntManyFull, false, WZP, 5, false>;
    case kEpiAny: return conv_igemm_i8_kernel<kEpiAny, false, WZP, 5, false>;
    default: return nullptr;
    }
}
IgemmBoxKernel igemm_kernel_mode5(int epi, bool wzp) { return wzp ? pick<true>(epi) : pick<false>(epi); }

}  // namespace b200
