// resident_m.cuh -- body of the translation units resident_m1.cu ..
// resident_m6.cu: instantiates resident_kernel<FOMO_RESIDENT_M> and its host
// entry points.
#pragma once

#include "step_resident.cuh"

namespace fomo {

template <>
const void* resident_kernel_fn<FOMO_RESIDENT_M>(int h_max) {
    return h_max > kRRowsOne ? reinterpret_cast<const void*>(&resident_kernel<FOMO_RESIDENT_M, 2>)
                             : reinterpret_cast<const void*>(&resident_kernel<FOMO_RESIDENT_M, 1>);
}

template <>
cudaError_t resident_launch<FOMO_RESIDENT_M>(int blocks, size_t smem, cudaStream_t st, const StepParams& P,
                                             const ResidentArgs& A) {
    void* args[2] = {const_cast<StepParams*>(&P), const_cast<ResidentArgs*>(&A)};
    return cudaLaunchCooperativeKernel(resident_kernel_fn<FOMO_RESIDENT_M>(A.L.h_max), dim3(blocks), dim3(kRThreads),
                                       args, smem, st);
}

}  // namespace fomo
