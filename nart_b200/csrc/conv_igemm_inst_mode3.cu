// Instantiations of the persistent convolution kernel: CTA pairs, which long reductions take.
#include "conv_igemm_kernel.cuh"

namespace b200 {

IgemmKernel igemm_kernel_mode3(int epi)
{
    switch (epi) {
    case kEpiIntOne: return conv_igemm_i8_kernel<kEpiIntOne, false, false, 3>;
    case kEpiIntOneFull: return conv_igemm_i8_kernel<kEpiIntOneFull, false, false, 3>;
    case kEpiIntMany: return conv_igemm_i8_kernel<kEpiIntMany, false, false, 3>;
    case kEpiIntManyFull: return conv_igemm_i8_kernel<kEpiIntManyFull, false, false, 3>;
    default: return nullptr;
    }
}

}  // namespace b200
