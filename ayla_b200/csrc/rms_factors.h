// Row factors of an RMS norm; see rms_factors.cu.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace ayla_b200 {
cudaError_t launch_rms_factors(const void* x, void* factors, int rows, int k, float eps, int is_bf16, int overlap,
                               cudaStream_t stream);
}  // namespace ayla_b200
