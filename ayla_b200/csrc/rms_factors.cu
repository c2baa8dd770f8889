// factors[r] = 1 / sqrt(mean(x[r]^2) + eps) for the rows of a 16-bit matrix, squares and sums in fp32, one
// rounding to the operands' type: what a projection behind an RMS norm multiplies its fp32 rows by.
//
// Bound by the one read of x.  The elementwise form it replaces (cast, square, mean, add, rsqrt, cast) wrote and
// re-read two fp32 copies of x: 4096 x 4096 bf16, us per call: six
// elementwise launches some 75, this kernel 6.7 (5.0 TB/s, the copy peak being 6.55).
#include "rms_factors.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "sm100_prims.cuh"

namespace ayla_b200 {
namespace {

__device__ __forceinline__ float square_sum(uint4 v, bool is_bf16, float sum) {
  const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = is_bf16 ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&words[j]))
                             : __half22float2(*reinterpret_cast<const __half2*>(&words[j]));
    sum = fmaf(f.x, f.x, sum);
    sum = fmaf(f.y, f.y, sum);
  }
  return sum;
}

constexpr int kThreads = 256;
constexpr int kUnroll = 4;  // 16-byte loads a thread has in flight

// ROW_THREADS threads (one to eight warps) share a row.  x is read through L2 (ld.global.cg), not as read-only data:
// this launch may begin while the one that writes x still runs, so x does change during the kernel's lifetime.
template <int ROW_THREADS>
__global__ void __launch_bounds__(kThreads)
rms_factors_kernel(const uint4* x, void* factors, int rows, int chunks, float k, float eps,
                   int is_bf16) {
  grid_launch_dependents();
  grid_dependency_wait();
  const int row = blockIdx.x * (kThreads / ROW_THREADS) + static_cast<int>(threadIdx.x) / ROW_THREADS;
  const int at = static_cast<int>(threadIdx.x) % ROW_THREADS;
  float sum = 0.0f;
  if (row < rows) {
    const uint4* src = x + static_cast<size_t>(row) * chunks;
    float part[kUnroll] = {};
    int c = at;
    for (; c + (kUnroll - 1) * ROW_THREADS < chunks; c += kUnroll * ROW_THREADS) {
      uint4 v[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) v[u] = __ldcg(src + c + u * ROW_THREADS);
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) part[u] = square_sum(v[u], is_bf16 != 0, part[u]);
    }
    for (; c < chunks; c += ROW_THREADS) part[0] = square_sum(__ldcg(src + c), is_bf16 != 0, part[0]);
    sum = (part[0] + part[1]) + (part[2] + part[3]);
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
  if constexpr (ROW_THREADS > 32) {
    __shared__ float warp_sums[kThreads / 32];
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (at == 0) {
      sum = 0.0f;
#pragma unroll
      for (int w = 0; w < ROW_THREADS / 32; ++w) sum += warp_sums[(threadIdx.x >> 5) + w];
    }
  }
  if (at == 0 && row < rows) {
    const float factor = rsqrtf(sum / k + eps);
    if (is_bf16 != 0) {
      static_cast<__nv_bfloat16*>(factors)[row] = __float2bfloat16_rn(factor);
    } else {
      static_cast<__half*>(factors)[row] = __float2half_rn(factor);
    }
  }
}

}  // namespace

cudaError_t launch_rms_factors(const void* x, void* factors, int rows, int k, float eps, int is_bf16, int overlap,
                               cudaStream_t stream) {
  // The most threads to a row that still have kUnroll loads each; fewer on short rows, so that a block's fixed cost
  // (launch, reduction) is shared by several: 2400 rows of 8192 with one warp a row 9.0 us, with eight 7.4;
  // 2300 rows of 1024 with eight warps a row 3.5 us, with one 2.1.
  const int chunks = k / 8;
  const int row_threads = chunks >= 256 * kUnroll ? 256 : chunks >= 128 * kUnroll ? 128 : chunks >= 64 * kUnroll ? 64 : 32;
  const auto kernel = row_threads == 256   ? rms_factors_kernel<256>
                      : row_threads == 128 ? rms_factors_kernel<128>
                      : row_threads == 64  ? rms_factors_kernel<64>
                                           : rms_factors_kernel<32>;
  const int block_rows = kThreads / row_threads;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((rows + block_rows - 1) / block_rows));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<const uint4*>(x), factors, rows, chunks, static_cast<float>(k),
                            eps, is_bf16);
}

}  // namespace ayla_b200
