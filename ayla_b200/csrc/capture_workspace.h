// Workspaces that belong to CUDA graphs; see capture_workspace.cu.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace ayla_b200 {
// The workspace of launches captured on `stream`, at least `bytes` with the first `zero_bytes` zero; the graph being
// captured keeps it.  The current device is the stream's.
cudaError_t capture_workspace(cudaStream_t stream, size_t bytes, size_t zero_bytes, void** workspace);
}  // namespace ayla_b200
