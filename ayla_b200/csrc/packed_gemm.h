// Products with few columns and a shallow depth; see packed_gemm.cu.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

namespace ayla_b200 {

struct PackedProblem {
  const void* a;     // [batch][m][k]
  const void* b;     // [batch][n][k]
  const void* bias;  // [n], or null
  void* out;         // [batch][m][n]
  int64_t batch, m, n, k;
  int is_bf16;
  uint32_t idesc_base;  // instruction descriptor without its N field
  unsigned* status;
  unsigned long long timeout_ns;
  int debug_flags;
  int sm_count;
  int overlap;
  cudaStream_t stream;
};

// Largest column count and depth the kernel takes (both in multiples of 8).
constexpr int kPackedMaxN = 128;
constexpr int kPackedMaxK = 128;

cudaError_t init_packed_gemm();
// Whether `out` starts on a 32-byte sector: else its rows go through staging, whatever they are.
inline bool on_sectors(const void* out) { return (reinterpret_cast<uintptr_t>(out) & 31) == 0; }
bool packed_preferred(int64_t batch, int64_t m, int64_t n, int64_t k, int sm_count, bool on_sectors);
cudaError_t launch_packed_gemm(const PackedProblem& problem);

}  // namespace ayla_b200
