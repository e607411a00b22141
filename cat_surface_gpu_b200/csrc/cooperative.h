// Cooperative launches of kernels whose CTAs wait on one another.
#pragma once

#include <cuda_runtime.h>

#include "errors.h"

namespace csg {

// Launches `kernel` cooperatively if all its CTAs can be resident at once; `launched` says whether it did.
inline int launch_if_resident(const void* kernel, int n_ctas, int threads, size_t smem, void** args, cudaStream_t s,
                              bool& launched) {
    int device = 0, sms = 0, per_sm = 0;
    launched = false;
    CSG_CUDA_CHECK(cudaGetDevice(&device));
    CSG_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    if (smem > 0)
        CSG_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CSG_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1 || n_ctas > per_sm * sms) return CSG_OK;
    CSG_CUDA_CHECK(cudaLaunchCooperativeKernel(kernel, dim3(n_ctas), dim3(threads), args, smem, s));
    note_launch();
    launched = true;
    return CSG_OK;
}

}  // namespace csg
