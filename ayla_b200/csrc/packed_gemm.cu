// out[b, m, n] = [bias[n] +] sum_k a[b, m, k] * b[b, n, k] for n, k <= 128: window attention, pointwise
// convolutions, any product whose work is reading a and writing out.
//
// What bounds these is memory, and on the way to it the fixed cost of a tile.  The general kernel spends some
// 0.8 us of one SM on a tile however little it holds (one CTA per SM, half of the epilogue warps idle at 64
// columns), and its TMA boxes are 64 elements deep: rows of 24 elements take four times as long as rows of 64.
// Here
//  * a unit is one 128-row accumulator: 128 rows of one matrix, or two or four small matrices side by side (their
//    rows stacked in A, their columns in B; the products of one matrix's rows with another's columns are computed
//    along and dropped, a tcgen05.mma of 128 rows takes the same 39 cycles up to 32 columns);
//  * operands come through cp.async in 16-byte pieces, which read the contiguous rows as one stream whatever
//    their length and put each piece where the swizzle wants it;
//  * the accumulator leaves through shared memory as one contiguous run of 16-byte pieces, or row by row (writes_rows).
// Two kernels do this.  In the chained one two to four CTAs share an SM and hide each other's waits; inside one, the next
// unit's loads run under the MMAs and the epilogue.  In the piped one, for units too large for that (piped_pays), the
// stages overlap inside a CTA.
// us per launch (graph replay, operands past L2), general kernel -> this: chained, bmm 8192 x 56x32x56 45.9 -> 22.4
// (110 MB: 16.8 at the copy peak), 8192 x 16x16x16 44.9 -> 7.1, mm 153718x32x16 18.5 -> 6.2; piped, mm 200704x96x24 37.3 ->
// 13.4 (7.4 at the peak).  What is left is latency: in the chained form a unit takes some 5000 cycles from its
// load to its last store, over half of them in the epilogue's chain of TMEM load, conversion, staging and copy.  Measured
// and left out there: 256 threads per CTA (bmm 22.4 -> 35.8), a third ring slot (25.6, it costs a resident CTA), two
// accumulators per CTA (25.5: half the CTAs find room in TMEM).
#include "packed_gemm.h"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "gemm_sm100.cuh"

namespace ayla_b200 {
namespace {

constexpr int kThreads = 128;     // the chained kernel: a warp per quarter of the accumulator's rows
constexpr int kStages = 2;
constexpr int kMaxCtasPerSm = 4;  // each may hold 128 of the 512 TMEM columns
constexpr int kRows = 128;        // accumulator rows

// The piped kernel: warps of its own for the epilogue (one per quarter), the loads and the MMAs.
constexpr int kEpilogueThreads = 128;
constexpr int kLoadThreads = 128;
constexpr int kPipedThreads = kEpilogueThreads + kLoadThreads + 32;
constexpr int kPipedMaxStages = 4;
constexpr int kPipedCtasPerSm = 2;
constexpr int kAccs = 2;              // accumulators in TMEM: the MMAs of a unit run under the epilogue of the one before

struct PackedParams {
  const uint8_t* a;
  const uint8_t* b;
  const void* bias;
  uint8_t* out;
  int units, row_tiles, batch, m, n;
  int matrices;   // small matrices per unit (1, 2 or 4)
  int slot_rows;  // accumulator rows each of them has
  int k_chunks;   // 16-byte pieces of one operand row
  int k_blocks;   // 64-deep blocks of an operand in shared memory
  int narrow;     // operand rows of 128 >> narrow bytes per block (a depth of at most 64 >> narrow)
  int mma_n;      // accumulator columns
  int shared_b;   // 1: every unit multiplies by the same B, loaded once
  int stages;     // ring slots of the piped kernel
  int tmem_cols;
  uint32_t idesc;
  uint32_t staging_pitch;
  int load_rows;     // operand rows the CTA loads at a time: each thread keeps to one piece of its row
  int load_threads;  // load_rows * k_chunks
  FastDiv div_k_chunks, div_n_chunks, div_row_tiles;
  unsigned* status;
  unsigned long long timeout_ns;
  int debug_flags;
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

__device__ __forceinline__ void store_32_bytes(void* dst, const uint32_t (&x)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst), "r"(x[0]), "r"(x[1]), "r"(x[2]),
               "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7])
               : "memory");
}

// Offset of 16-byte piece `c` of row `row` in an operand tile of 64-deep blocks of `block_bytes`, in the
// 128-, 64- or 32-byte swizzle (rows of 128 >> narrow bytes, a single block where narrow > 0).
__device__ __forceinline__ uint32_t piece_offset(int row, int c, uint32_t block_bytes, int narrow) {
  const int swizzle = (row >> narrow) & (7 >> narrow);
  return static_cast<uint32_t>(c >> 3) * block_bytes + (static_cast<uint32_t>(row) << (7 - narrow)) +
         static_cast<uint32_t>(((c & 7) ^ swizzle) << 4);
}

__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr, int narrow) {
  // As umma_smem_desc_sw128, with eight rows 1024 >> narrow bytes apart and layout type 2, 4 or 6.
  uint64_t d = umma_smem_desc_sw128(smem_addr);
  d &= ~((static_cast<uint64_t>(0x3FFF) << 32) | (static_cast<uint64_t>(7) << 61));
  d |= static_cast<uint64_t>(64 >> narrow) << 32;
  d |= static_cast<uint64_t>(2 + 2 * narrow) << 61;
  return d;
}

template <bool BF16>
__device__ __forceinline__ uint32_t pack_pair(float lo, float hi) {
  return pack2(lo, hi, BF16 ? 1 : 0);
}

// Loads of one unit's operands by a group of threads, each keeping to one 16-byte piece of its rows.
struct UnitLoader {
  const PackedParams& p;
  const int tid, load_row, load_c;
  const bool loads;
  const uint32_t a_block, b_block;

  __device__ UnitLoader(const PackedParams& p_, int tid_, uint32_t a_block_, uint32_t b_block_)
      : p(p_), tid(tid_), load_row(p_.div_k_chunks.div(tid_)), load_c(tid_ - load_row * p_.k_chunks),
        loads(tid_ < p_.load_threads), a_block(a_block_), b_block(b_block_) {}

  __device__ __forceinline__ void load_operand(uint32_t dst, const uint8_t* src, int rows, uint32_t block_bytes,
                                               int rows_per_matrix, int gap) const {
    src += static_cast<uint32_t>(tid) * 16u;
    const uint32_t step = static_cast<uint32_t>(p.load_threads) * 16u;
    int slot_row = load_row, left = rows_per_matrix - load_row;  // rows of this matrix still ahead
    for (int row = load_row; row < rows; row += p.load_rows) {
      while (left <= 0) {
        left += rows_per_matrix;
        slot_row += gap;
      }
      cp_async_16(dst + piece_offset(slot_row, load_c, block_bytes, p.narrow), src);
      src += step;
      slot_row += p.load_rows;
      left -= p.load_rows;
    }
  }

  // `first`: also the B that all units share.
  __device__ __forceinline__ void load(int unit, uint32_t dst_a, uint32_t dst_b, bool first) const {
    if (!loads) return;
    int first_matrix, matrices, row0, rows;  // rows: of A, over all of the unit's matrices
    if (p.matrices == 1) {
      first_matrix = p.div_row_tiles.div(unit);
      matrices = 1;
      row0 = (unit - first_matrix * p.row_tiles) * kRows;
      rows = min(kRows, p.m - row0);
    } else {
      first_matrix = unit * p.matrices;
      matrices = min(p.matrices, p.batch - first_matrix);
      row0 = 0;
      rows = matrices * p.m;
    }
    load_operand(dst_a, p.a + (static_cast<size_t>(first_matrix) * p.m + row0) * p.k_chunks * 16, rows, a_block,
                 p.matrices == 1 ? kRows : p.m, p.slot_rows - p.m);
    if (!p.shared_b || first) {
      load_operand(dst_b, p.b + static_cast<size_t>(first_matrix) * p.n * p.k_chunks * 16, matrices * p.n, b_block,
                   kPackedMaxN, 0);
    }
  }
};

// A warp's share of one unit's results: a quarter of the accumulator's rows, through its staging rows into `out` or straight
// (DIRECT kernels, see writes_rows).
template <bool BF16>
struct UnitWriter {
  const PackedParams& p;
  const int quarter, lane, my_matrix, my_row, n_chunks;
  uint8_t* const staging;
  const float* const smem_bias;
  // This lane's first piece of the warp's staged rows, and the steps to the one 32 pieces on.
  int out_c, out_c_step;
  uint32_t out_offset, out_step, out_wrap;
  mutable int matrix = 0, row0 = 0, rows = 0;

  // `staging_`: the warp's own rows (their offset added up in here, the piped kernel took 15.5 us instead of 14.2 for mm
  // 200704x96x24).
  __device__ UnitWriter(const PackedParams& p_, int quarter_, int lane_, uint8_t* staging_, const float* smem_bias_)
      : p(p_), quarter(quarter_), lane(lane_), my_matrix(quarter_ / (p_.slot_rows / 32)),
        my_row((quarter_ % (p_.slot_rows / 32)) * 32), n_chunks(p_.n >> 3),
        staging(staging_), smem_bias(smem_bias_) {
    const int out_row = p.div_n_chunks.div(lane), out_row_step = p.div_n_chunks.div(32);
    out_c = lane - out_row * n_chunks;
    out_c_step = 32 - out_row_step * n_chunks;
    out_offset = static_cast<uint32_t>(out_row) * p.staging_pitch + static_cast<uint32_t>(out_c) * 16u;
    out_step = static_cast<uint32_t>(out_row_step) * p.staging_pitch + static_cast<uint32_t>(out_c_step) * 16u;
    out_wrap = p.staging_pitch - static_cast<uint32_t>(n_chunks) * 16u;
  }

  // Matrix `my_matrix` of the unit, from its row `my_row` on; false where there is none.
  __device__ __forceinline__ bool locate(int unit) const {
    if (p.matrices == 1) {
      matrix = p.div_row_tiles.div(unit);
      row0 = (unit - matrix * p.row_tiles) * kRows + my_row;
    } else {
      matrix = unit * p.matrices + my_matrix;
      row0 = my_row;
    }
    rows = matrix < p.batch ? min(32, p.m - row0) : 0;
    return rows > 0;
  }

  __device__ __forceinline__ void stage(uint32_t accumulator) const {
    const uint32_t t = accumulator + (static_cast<uint32_t>(quarter * 32) << 16) +
                       static_cast<uint32_t>(p.matrices > 1 ? my_matrix * p.n : 0);
    for (int c0 = 0; c0 < n_chunks; c0 += 4) {
      uint32_t r[32];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c0 + j < n_chunks) tmem_ld_32x8(t + (c0 + j) * 8, r + 8 * j);
      }
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c0 + j < n_chunks) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * j + e]);
          if (p.bias != nullptr) {
            const float4* b4 = reinterpret_cast<const float4*>(smem_bias + (c0 + j) * 8);
            const float4 lo = b4[0], hi = b4[1];
            v[0] += lo.x;
            v[1] += lo.y;
            v[2] += lo.z;
            v[3] += lo.w;
            v[4] += hi.x;
            v[5] += hi.y;
            v[6] += hi.z;
            v[7] += hi.w;
          }
          *reinterpret_cast<uint4*>(staging + lane * p.staging_pitch + (c0 + j) * 16) =
              make_uint4(pack_pair<BF16>(v[0], v[1]), pack_pair<BF16>(v[2], v[3]), pack_pair<BF16>(v[4], v[5]),
                         pack_pair<BF16>(v[6], v[7]));
        }
      }
    }
  }

  // Without staging: each lane writes its row, two pieces (a 32-byte sector) an instruction.
  __device__ __forceinline__ void write(uint32_t accumulator) const {
    const uint32_t t = accumulator + (static_cast<uint32_t>(quarter * 32) << 16) +
                       static_cast<uint32_t>(p.matrices > 1 ? my_matrix * p.n : 0);
    uint8_t* dst = p.out + ((static_cast<size_t>(matrix) * p.m + row0 + lane) * n_chunks) * 16;
    const bool mine = lane < rows;
    for (int c0 = 0; c0 < n_chunks; c0 += 4) {
      uint32_t r[32];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (c0 + j < n_chunks) tmem_ld_32x8(t + (c0 + j) * 8, r + 8 * j);
      }
      tmem_ld_wait();
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        if (c0 + j < n_chunks) {
          uint32_t x[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            float lo = __uint_as_float(r[8 * j + 2 * e]), hi = __uint_as_float(r[8 * j + 2 * e + 1]);
            if (p.bias != nullptr) {
              const float2 b = *reinterpret_cast<const float2*>(smem_bias + (c0 + j) * 8 + 2 * e);
              lo += b.x;
              hi += b.y;
            }
            x[e] = pack_pair<BF16>(lo, hi);
          }
          if (mine) store_32_bytes(dst + (c0 + j) * 16, x);
        }
      }
    }
  }

  // The staged rows follow one another in `out` without a gap.
  __device__ __forceinline__ void copy_out() const {
    uint8_t* dst = p.out + ((static_cast<size_t>(matrix) * p.m + row0) * n_chunks + lane) * 16;
    const int pieces = rows * n_chunks;
    int c = out_c;
    const uint8_t* src = staging + out_offset;
    for (int j = lane; j < pieces; j += 128) {
      uint4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j + 32 * u < pieces) x[u] = *reinterpret_cast<const uint4*>(src);
        src += out_step;
        c += out_c_step;
        if (c >= n_chunks) {
          c -= n_chunks;
          src += out_wrap;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        if (j + 32 * u < pieces) *reinterpret_cast<uint4*>(dst + 512 * u) = x[u];
      }
      dst += 2048;
    }
  }
};

template <bool BF16, bool DIRECT>
__global__ void __launch_bounds__(kThreads, kMaxCtasPerSm) packed_gemm_kernel(const PackedParams p) {
#if defined(__CUDA_ARCH_FEAT_SM100_ALL) || defined(__CUDA_ARCH_FEAT_SM101_ALL)
  extern __shared__ __align__(1024) uint8_t packed_smem[];
  const int narrow = p.narrow;
  const uint32_t a_block = static_cast<uint32_t>(kRows * 128) >> narrow;
  const uint32_t a_bytes = static_cast<uint32_t>(p.k_blocks) * a_block;
  const uint32_t b_block = static_cast<uint32_t>(p.mma_n * 128) >> narrow;
  const uint32_t b_bytes = static_cast<uint32_t>(p.k_blocks) * b_block;
  const int b_copies = p.shared_b ? 1 : kStages;
  uint8_t* smem_b = packed_smem + kStages * a_bytes;
  uint8_t* smem_staging = smem_b + b_copies * b_bytes;
  float* smem_bias = reinterpret_cast<float*>(smem_staging + kRows * p.staging_pitch);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_bias + kPackedMaxN);
  const uint32_t bar_done = smem_u32(bars);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int tid = static_cast<int>(threadIdx.x);
  const int warp = tid >> 5, lane = tid & 31;
  const BoundedWait bw{abort_flag, p.status, p.timeout_ns};

  if (tid == 0) {
    *abort_flag = 0;
    if ((smem_u32(packed_smem) & 1023u) != 0) bw.give_up(ST_BAD_SMEM_ALIGN);
    mbar_init(bar_done, 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc<1>(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish<1>();
  }
  // A depth that is an odd number of pieces is read one piece further by the MMAs: zero in both operands.
  if ((p.k_chunks & 1) != 0) {
    for (int i = tid; i < kStages * kRows; i += kThreads) {
      const int s = i / kRows, row = i % kRows;
      *reinterpret_cast<uint4*>(packed_smem + s * a_bytes + piece_offset(row, p.k_chunks, a_block, narrow)) =
          make_uint4(0, 0, 0, 0);
    }
    for (int s = 0; s < b_copies; ++s) {
      for (int row = tid; row < p.mma_n; row += kThreads) {
        *reinterpret_cast<uint4*>(smem_b + s * b_bytes + piece_offset(row, p.k_chunks, b_block, narrow)) =
            make_uint4(0, 0, 0, 0);
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();
  grid_dependency_wait();
  if (p.bias != nullptr && tid < p.n) smem_bias[tid] = load_elem(p.bias, tid, BF16 ? 1 : 0);

  const int first = static_cast<int>(blockIdx.x), stride = static_cast<int>(gridDim.x);
  const int count = (p.units - first + stride - 1) / stride;  // the grid is no larger than `units`

  // Loads of this CTA's i-th unit into ring slot `s`: one commit group per unit, empty past the last.
  const UnitLoader loader(p, tid, a_block, b_block);
  auto load_unit = [&](int i, int s) {
    if (i < count) {
      loader.load(first + i * stride, smem_u32(packed_smem) + static_cast<uint32_t>(s) * a_bytes,
                  smem_u32(smem_b) + (p.shared_b ? 0u : static_cast<uint32_t>(s) * b_bytes), i == 0);
    }
    cp_async_commit();
  };
  const UnitWriter<BF16> writer(p, warp, lane, smem_staging + warp * 32 * p.staging_pitch, smem_bias);
  auto epilogue = [&](int i) {
    if (!writer.locate(first + i * stride)) return;
    if constexpr (DIRECT) {
      writer.write(tmem_base);
    } else {
      writer.stage(tmem_base);
      __syncwarp();
      writer.copy_out();
    }
  };

#pragma unroll
  for (int s = 0; s < kStages; ++s) load_unit(s, s);

  int slot = 0;
  for (int i = 0; i < count; ++i) {
    // Groups are committed in the order of the units: all but the kStages - 1 newest are in.
    cp_async_wait<kStages - 1>();
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();  // the unit's operands are in; everyone is done with the accumulator and the staging rows
    if (warp == 0) {
      tc_fence_after_sync();
      if (elect_one() && (p.debug_flags & 1) == 0) {
        const uint64_t desc_a = operand_desc(smem_u32(packed_smem) + static_cast<uint32_t>(slot) * a_bytes, narrow);
        const uint64_t desc_b =
            operand_desc(smem_u32(smem_b) + (p.shared_b ? 0u : static_cast<uint32_t>(slot) * b_bytes), narrow);
        const int steps = (p.k_chunks + 1) >> 1;
        for (int ks = 0; ks < steps; ++ks) {
          const uint32_t kb = static_cast<uint32_t>(ks >> 2), in_block = 2u * static_cast<uint32_t>(ks & 3);
          umma_f16<1>(tmem_base, desc_a + kb * (a_block >> 4) + in_block, desc_b + kb * (b_block >> 4) + in_block,
                      p.idesc, ks > 0 ? 1u : 0u);
        }
        umma_commit_1cta(bar_done);
      }
      __syncwarp();
      bw.wait(bar_done, static_cast<uint32_t>(i) & 1u, ST_TIMEOUT_FULL);
    }
    __syncthreads();
    tc_fence_after_sync();
    load_unit(i + kStages, slot);  // the MMAs have read the slot
    if (++slot == kStages) slot = 0;
    epilogue(i);
  }

  cp_async_wait<0>();
  if (bw.aborted()) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // MMAs still in flight
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
#endif
}

// The same units through a pipeline inside each CTA: four warps load, one issues MMAs, the others write results, and
// they meet at mbarriers only, so that the loads run several units ahead and the MMAs and the epilogue of consecutive
// units overlap.  In the kernel above a unit is a chain (load, MMA, epilogue, 5000 cycles) that only other CTAs of the SM
// hide: with units of 24 KB and more fewer of those fit, and the chain shows; with small ones its smaller CTAs win.
// us per launch, the kernel above -> this one: mm 200704x96x24 16.3 -> 14.3, 171761x24x40 11.0 -> 8.2, 131072x64x8 13.9 ->
// 8.8, 250000x128x40 25.7 -> 20.5, bmm 3000 x 128x64x40 21.3 -> 19.3, 5332 x 45x16x120 22.3 -> 18.9.  What is left is
// the epilogue's chain (a second set of epilogue warps made no more than 3 %, or lost as much to its staging rows) and,
// from 30 KB a unit on, the SM's store rate.
template <bool BF16, bool DIRECT>
__global__ void __launch_bounds__(kPipedThreads, kPipedCtasPerSm) packed_piped_kernel(const PackedParams p) {
#if defined(__CUDA_ARCH_FEAT_SM100_ALL) || defined(__CUDA_ARCH_FEAT_SM101_ALL)
  extern __shared__ __align__(1024) uint8_t packed_smem[];
  const int narrow = p.narrow;
  const uint32_t a_block = static_cast<uint32_t>(kRows * 128) >> narrow;
  const uint32_t a_bytes = static_cast<uint32_t>(p.k_blocks) * a_block;
  const uint32_t b_block = static_cast<uint32_t>(p.mma_n * 128) >> narrow;
  const uint32_t b_bytes = static_cast<uint32_t>(p.k_blocks) * b_block;
  const int b_copies = p.shared_b ? 1 : p.stages;
  uint8_t* smem_b = packed_smem + p.stages * a_bytes;
  uint8_t* smem_staging = smem_b + b_copies * b_bytes;
  float* smem_bias = reinterpret_cast<float*>(smem_staging + kRows * p.staging_pitch);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_bias + kPackedMaxN);
  // full[kPipedMaxStages], empty[kPipedMaxStages], acc_full[kAccs], acc_empty[kAccs]
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = bar_full + kPipedMaxStages * 8;
  const uint32_t bar_acc_full = bar_empty + kPipedMaxStages * 8;
  const uint32_t bar_acc_empty = bar_acc_full + kAccs * 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kPipedMaxStages + 2 * kAccs);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  constexpr int kFirstLoadWarp = kEpilogueThreads / 32, kMmaWarp = kFirstLoadWarp + kLoadThreads / 32;
  const BoundedWait bw{abort_flag, p.status, p.timeout_ns};

  if (threadIdx.x == 0) {
    *abort_flag = 0;
    if ((smem_u32(packed_smem) & 1023u) != 0) bw.give_up(ST_BAD_SMEM_ALIGN);
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(bar_full + s * 8, kLoadThreads);
      mbar_init(bar_empty + s * 8, 1);
    }
    for (int i = 0; i < kAccs; ++i) {
      mbar_init(bar_acc_full + i * 8, 1);
      mbar_init(bar_acc_empty + i * 8, 4);
    }
    fence_mbar_init();
  }
  if (warp == kMmaWarp) {
    tmem_alloc<1>(smem_u32(tmem_slot), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish<1>();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  grid_launch_dependents();

  const int first = static_cast<int>(blockIdx.x), stride = static_cast<int>(gridDim.x);
  const int count = (p.units - first + stride - 1) / stride;  // the grid is no larger than `units`

  if (warp >= kFirstLoadWarp && warp < kMmaWarp) {
    // ---------------------------------------------------------------- loads
    const int tid = static_cast<int>(threadIdx.x) - kFirstLoadWarp * 32;
    // A depth that is an odd number of pieces is read one piece further by the MMAs: zero in both operands.
    if ((p.k_chunks & 1) != 0) {
      for (int s = 0; s < p.stages; ++s) {
        *reinterpret_cast<uint4*>(packed_smem + s * a_bytes + piece_offset(tid, p.k_chunks, a_block, narrow)) =
            make_uint4(0, 0, 0, 0);
      }
      for (int s = 0; s < b_copies; ++s) {
        if (tid < p.mma_n) {
          *reinterpret_cast<uint4*>(smem_b + s * b_bytes + piece_offset(tid, p.k_chunks, b_block, narrow)) =
              make_uint4(0, 0, 0, 0);
        }
      }
    }
    grid_dependency_wait();
    const bool loads = (p.debug_flags & 1) == 0;
    const UnitLoader loader(p, tid, a_block, b_block);
    // A unit is announced once this thread's pieces of it have landed, when the loads of the next `behind` units have
    // been issued: commit groups complete in order.
    const int behind = p.stages - 1;
    int slot = 0, done_slot = 0;
    uint32_t phase = 1;
    for (int i = 0; i < count + behind; ++i) {
      if (i < count) {
        bw.wait(bar_empty + slot * 8, phase, ST_TIMEOUT_EMPTY);
        if (loads && !bw.aborted()) {
          loader.load(first + i * stride, smem_u32(packed_smem) + static_cast<uint32_t>(slot) * a_bytes,
                      smem_u32(smem_b) + (p.shared_b ? 0u : static_cast<uint32_t>(slot) * b_bytes), i == 0);
        }
        if (++slot == p.stages) {
          slot = 0;
          phase ^= 1;
        }
      }
      cp_async_commit();
      if (i >= behind) {
        switch (behind) {
          case 1: cp_async_wait<1>(); break;
          case 2: cp_async_wait<2>(); break;
          default: cp_async_wait<3>(); break;
        }
        fence_proxy_async_smem();
        if (loads) mbar_arrive(bar_full + done_slot * 8);
        if (++done_slot == p.stages) done_slot = 0;
      }
    }
    cp_async_wait<0>();
  } else if (warp == kMmaWarp) {
    // ----------------------------------------------------------------- MMAs
    const bool issuer = elect_one();
    const uint64_t desc_a0 = operand_desc(smem_u32(packed_smem), narrow);
    const uint64_t desc_b0 = operand_desc(smem_u32(smem_b), narrow);
    const int steps = (p.k_chunks + 1) >> 1;
    int slot = 0;
    uint32_t phase = 0, acc = 0, acc_phase = 1;
    for (int i = 0; i < count; ++i) {
      bw.wait(bar_acc_empty + acc * 8, acc_phase, ST_TIMEOUT_ACC_EMPTY);
      bw.wait(bar_full + slot * 8, phase, ST_TIMEOUT_FULL);
      if (__any_sync(0xffffffffu, bw.aborted())) break;  // lanes whose wait ran out, and the others with them
      tc_fence_after_sync();
      if (issuer) {
        const uint64_t desc_a = desc_a0 + static_cast<uint32_t>(slot) * (a_bytes >> 4);
        const uint64_t desc_b = desc_b0 + (p.shared_b ? 0u : static_cast<uint32_t>(slot) * (b_bytes >> 4));
        for (int ks = 0; ks < steps; ++ks) {
          const uint32_t kb = static_cast<uint32_t>(ks >> 2), in_block = 2u * static_cast<uint32_t>(ks & 3);
          umma_f16<1>(tmem_base + acc * static_cast<uint32_t>(p.mma_n), desc_a + kb * (a_block >> 4) + in_block,
                      desc_b + kb * (b_block >> 4) + in_block, p.idesc, ks > 0 ? 1u : 0u);
        }
        umma_commit_1cta(bar_empty + slot * 8);
        umma_commit_1cta(bar_acc_full + acc * 8);
      }
      __syncwarp();
      if (++slot == p.stages) {
        slot = 0;
        phase ^= 1;
      }
      if (++acc == kAccs) {
        acc = 0;
        acc_phase ^= 1;
      }
    }
  } else {
    // ------------------------------------------------------------- epilogue
    grid_dependency_wait();
    if (p.bias != nullptr) {
      if (static_cast<int>(threadIdx.x) < p.n) smem_bias[threadIdx.x] = load_elem(p.bias, threadIdx.x, BF16 ? 1 : 0);
      named_bar_sync(1, kEpilogueThreads);
    }
    const UnitWriter<BF16> writer(p, warp, lane, smem_staging + warp * 32 * p.staging_pitch, smem_bias);
    for (int i = 0; i < count; ++i) {
      const uint32_t acc = static_cast<uint32_t>(i) & 1u, acc_phase = (static_cast<uint32_t>(i) >> 1) & 1u;
      bw.wait(bar_acc_full + acc * 8, acc_phase, ST_TIMEOUT_ACC_FULL);
      // TMEM is read by whole warps: a wait that ran out for some lanes ends the unit for all.
      const bool aborted = __any_sync(0xffffffffu, bw.aborted());
      tc_fence_after_sync();
      const bool live = writer.locate(first + i * stride) && !aborted;
      if (live) {
        if constexpr (DIRECT) {
          writer.write(tmem_base + acc * static_cast<uint32_t>(p.mma_n));
        } else {
          writer.stage(tmem_base + acc * static_cast<uint32_t>(p.mma_n));
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_acc_empty + acc * 8);
      if constexpr (!DIRECT) {
        if (live) writer.copy_out();
        __syncwarp();  // the staging rows are free again
      }
    }
  }

  if (bw.aborted()) {
    for (int i = 0; i < 64; ++i) __nanosleep(2000);  // MMAs still in flight
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after_sync();
    tmem_dealloc<1>(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
#endif
}

constexpr int kSmemPerSm = 233472, kSmemPerCta = 232448, kCtaReserve = 1024;

// How a problem lies in shared memory and how many CTAs of it an SM holds.
struct Footprint {
  int matrices;  // small matrices per unit: as many as the accumulator's quarters of 32 rows and its columns hold
  int mma_n, narrow, k_blocks;
  int staging_pitch;
  int smem, ctas;
  int64_t units;
  bool piped;     // the piped kernel
  int stages, piped_smem, piped_ctas, piped_tmem_cols;
};

// Where the piped kernel is the faster one (350 shapes timed on both; over the 64 of the packed kernel's that it takes, 0.914
// of the time, the slowest 1.04): with rows that start inside a 32-byte sector and one B for all units, whose loads take
// longest (247747x48x24 18.5 -> 14.0, 33392x64x24 6.7 -> 5.7); otherwise where an SM would hold two CTAs of the other or
// fewer, which leaves a unit's chain bare (204363x40x88 17.0 -> 14.9), and every CTA has a unit at least (36745x32x128, 288
// units, 5.0 -> 5.2).  Three CTAs hide it as well or better, far better with few rows to a unit (2984 x 19x112x32 15.1 ->
// 17.4, 2099 x 10x104x24 11.0 -> 12.7, 381 x 1239x64x56 25.1 -> 26.0).
bool piped_pays(int64_t units, int64_t k, bool shared_b, int chained_ctas) {
  if (shared_b && k % 16 != 0) return units >= 256;
  return chained_ctas <= 2 && units >= 300;
}

// Where the lanes write their rows themselves, without staging: rows of whole sectors, but not of whole lines, whose stores
// meet in one another's way.  What it saves is the way through shared memory, and its rows there, which makes room for more
// CTAs.  Over 140 shapes of 16 to 112 columns timed both ways it takes 0.90 of the time (us, staged -> direct: mm 200704x96x24
// 14.6 -> 13.7, 262144x48x32 11.7 -> 8.9, bmm 3194 x 13x80x112 25.6 -> 16.8, 8149 x 32x48x8 12.3 -> 10.8); of 64 and 128
// columns 1.0 to 1.2 (mm 121018x64x32 7.0 -> 8.3).  Rows of 64 bytes are half lines, which only shallow products make up for
// (bmm 2500 x 100x32x32 10.0 -> 9.0, x40 10.6 -> 11.1, x56 12.5 -> 13.5, 8192 x 56x32x56 21.1 -> 21.8), and those of 192 are a
// line and a half (bmm 2500 x 100x96x56 20.4 -> 21.5, x40 18.1 -> 18.5; with one B or another depth they gain).
bool writes_rows(int64_t n, int64_t k, bool shared_b) {
  if (n % 16 != 0 || n % 64 == 0) return false;
  if (n == 32) return k <= 32;
  return n != 96 || shared_b || k <= 32 || k > 64;
}

// `staged`: with room for the results on their way out.
Footprint footprint(int64_t batch, int64_t m, int64_t n, int64_t k, bool staged = true) {
  Footprint f;
  f.matrices = 1;
  while (batch > 1 && f.matrices < 4 && m * f.matrices * 2 <= kRows && n * f.matrices * 2 <= kPackedMaxN) f.matrices *= 2;
  f.mma_n = static_cast<int>((n * f.matrices + 15) / 16 * 16);
  f.narrow = k <= 16 ? 2 : k <= 32 ? 1 : 0;
  f.k_blocks = static_cast<int>((k + 63) / 64);
  // An odd number of 16-byte pieces per staging row: eight lanes writing a piece of eight rows meet eight banks.
  f.staging_pitch = staged ? 16 * static_cast<int>((n / 8) | 1) : 0;
  const int a_bytes = (f.k_blocks * kRows * 128) >> f.narrow, b_bytes = (f.k_blocks * f.mma_n * 128) >> f.narrow;
  f.smem = kStages * a_bytes + (batch == 1 ? 1 : kStages) * b_bytes + kRows * f.staging_pitch + kPackedMaxN * 4 + 64;
  f.ctas = kSmemPerSm / (f.smem + kCtaReserve);
  if (f.ctas > kMaxCtasPerSm) f.ctas = kMaxCtasPerSm;

  // Two CTAs, or one, and then as many ring slots as still fit.
  const bool shared_b = batch == 1;
  auto piped_smem = [&](int stages) {
    return stages * a_bytes + (shared_b ? 1 : stages) * b_bytes + kRows * f.staging_pitch + kPackedMaxN * 4 + 128;
  };
  f.piped_tmem_cols = 32;
  while (f.piped_tmem_cols < kAccs * f.mma_n) f.piped_tmem_cols *= 2;
  f.piped_ctas = kPipedCtasPerSm;
  while (f.piped_ctas > 1 && kSmemPerSm / (piped_smem(2) + kCtaReserve) < f.piped_ctas) --f.piped_ctas;
  f.stages = 2;
  while (f.stages < kPipedMaxStages && piped_smem(f.stages + 1) <= kSmemPerCta &&
         kSmemPerSm / (piped_smem(f.stages + 1) + kCtaReserve) >= f.piped_ctas) {
    ++f.stages;
  }
  f.piped_smem = piped_smem(f.stages);
  f.units = f.matrices == 1 ? batch * ((m + kRows - 1) / kRows) : (batch + f.matrices - 1) / f.matrices;
  f.piped = piped_pays(f.units, k, shared_b, f.ctas);
  return f;
}

bool one_piece_round(int64_t k, int64_t n, bool shared_b, const Footprint& f, int64_t tiles, int sm_count) {
  const double rounds = static_cast<double>(tiles) / (static_cast<double>(f.ctas) * sm_count);
  return f.ctas >= 4 && shared_b && k < 16 && n > 40 && n <= 64 && rounds > 0.5 && rounds < 1.35;
}

bool preferred_by_rounds(int64_t batch, int64_t n, int64_t k, int64_t tiles, const Footprint& f, int sm_count) {
  if (f.matrices > 1) return f.matrices == 4 || f.ctas >= 2;
  if (f.ctas < 2) return false;
  const bool shared_b = batch == 1, mid_sector = k % 16 != 0;
  if (n <= 32) return shared_b || f.ctas >= 3 || mid_sector;
  const double rounds = static_cast<double>(tiles) / (static_cast<double>(f.ctas) * sm_count);
  if (k >= 48 && rounds < 0.5) return false;
  if (f.ctas >= 4) return !one_piece_round(k, n, shared_b, f, tiles, sm_count);
  const bool settled = rounds <= 0.95 || rounds >= 1.35;
  if (f.ctas == 3) {
    if (n <= 64) return settled || k < 48;
    if (shared_b) return rounds >= 1.25 || (mid_sector && k < 48);
    return settled && (mid_sector || (n <= 80 && rounds >= 1.35) || (k <= 32 && rounds >= 2.0));
  }
  if (!shared_b) return n <= 64 ? settled && mid_sector : k < 64 && rounds <= 0.95;
  if (mid_sector) return (k > 64 && n <= 96) || (settled && (n <= 96 || rounds >= 1.35 || k < 64));
  return n <= 64 ? rounds >= 2.4 : k < 64 && n % 16 != 0 && rounds >= 1.35;
}

}  // namespace

cudaError_t init_packed_gemm() {
  const void* const kernels[] = {
      reinterpret_cast<const void*>(&packed_gemm_kernel<false, false>),
      reinterpret_cast<const void*>(&packed_gemm_kernel<true, false>),
      reinterpret_cast<const void*>(&packed_gemm_kernel<false, true>),
      reinterpret_cast<const void*>(&packed_gemm_kernel<true, true>),
      reinterpret_cast<const void*>(&packed_piped_kernel<false, false>),
      reinterpret_cast<const void*>(&packed_piped_kernel<true, false>),
      reinterpret_cast<const void*>(&packed_piped_kernel<false, true>),
      reinterpret_cast<const void*>(&packed_piped_kernel<true, true>),
  };
  for (const void* kernel : kernels) {
    const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemPerCta);
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

// Where these kernels are faster than the general one.  The edges come from 1606 shapes of up to 128 columns and a depth of
// up to 128, timed with the chained form alone (0.726 of the general kernel's time).  With the form that runs now, over 350
// others: 276 are taken, in 0.575 of the time, five of them slower by 4 to 20 % (285 x 422x128x32 10.4 -> 12.1); of the 74
// left, 28 would take less than 0.9, most of them piped with one or two CTAs per SM (103219x88x80 16.9, 11.1 piped).
// What it goes by (us, general -> chained; or chained over general):
//  * a 128-row tile for every SM; below, both are a launch and one pass (bmm 8 x 1024x64x64 2.8 -> 3.5).
//  * Small matrices that share an accumulator gain most (1024 x 64x64x64 8.7 -> 7.3, 574 x 15x16x32 5.4 -> 2.6), as
//    long as two CTAs fit an SM or four matrices a unit (7467 x 17x48x104, one CTA: 42.5 -> 47.9).
//  * Otherwise resident CTAs hide a unit's chain of load, MMA and epilogue: with one per SM nothing does (512 x
//    128x72x104 8.4 -> 10.3), with four nearly every product gains, and with three or two it takes an advantage
//    besides: few columns, rows that start in the middle of a 32-byte sector, which cost the general kernel's TMA
//    loads twice (200 x 500x56x72 10.1 -> 9.1, but 200 x 500x48x128 9.1 -> 10.0 and 200 x 500x128x56 9.3 -> 12.9),
//    or one B for all units (162131x72x48 0.60, but 4252 x 85x112x48 1.46), for aligned rows at two CTAs from the third
//    round on (159590x40x80, 4.2 rounds, 0.53; 42849x48x96, 1.1, 1.14) or with output rows that start inside a sector
//    (70938x120x48 0.85, 72817x112x48 1.16).
//  * A second round of units that fills less than a third of the resident CTAs is a round all the same (512 x
//    128x72x56, 1.15 rounds: 7.6 -> 8.2), and so is a first one that leaves half of them without work (19815x64x48 1.09,
//    170 x 110x64x56 1.10); up to a depth of 40 the general kernel's 64-deep boxes cost it more than that (37 x
//    473x56x40 0.81, 512 x 128x48x40 0.83).
//  * A product of one 16-byte piece in depth with shared B, in a single round (60000x64x8 8.6 -> 10.8; 131072x64x8, in
//    two, 16.0 -> 13.7).
//
// Where two CTAs and more of the form that runs fit an SM (without staging rows where the lanes write their own, for which
// `out` has to be `on_sectors`: with staging rows and one CTA, bmm 7653 x 22x96x120 general 52.8, packed 74.2; 156 x
// 726x80x80 11.0 and 14.9), these besides, from 1100 shapes timed on both kernels:
//  * up to a depth of 40, from 64 tiles on: 98 shapes, 0.80 of the time, the slowest 1.01; of 120 columns, where every SM has a
//    tile (bmm 73 x 72x120x40 3.4 -> 3.6), one to a unit with few rows or five tiles to an SM (17 shapes: 283 x 24x120x32 5.5 ->
//    3.6, 2557 x 186x120x40 55 -> 41, 561 x 661x120x40 30.5 -> 28.6, but in two or three rounds of full tiles 153 x 238x120x40 5.5 ->
//    6.5, 250 x 174x120x32 8.6 -> 9.4); not of 128 (mm 11964x128x40 4.6 -> 4.9);
//  * deeper, with few rows to a unit or one B, from 950 tiles on: 13 shapes, 0.78, 0.93 (1226 x 26x80x80 10.7 -> 8.5, mm
//    246943x72x96 0.54);
//  * up to 80 columns and a depth of 88, with a tile for every SM: 41 shapes, 0.88, 1.06 (59 x 635x80x64 0.75, but 24 x
//    1677x80x120 1.24), four tenths of a round and thin second rounds aside.
// Of 547 shapes drawn afterwards among those that these three take: 0.80 of the time of the general kernel with the ops'
// schedule, eight slower by 2 %, at most 1.09 (43 x 786x48x80).
bool packed_preferred(int64_t batch, int64_t m, int64_t n, int64_t k, int sm_count, bool on_sectors) {
  if (n > kPackedMaxN || k > kPackedMaxK) return false;
  const int64_t tiles = batch * ((m + kRows - 1) / kRows);
  if (tiles > 0x7FFFFFFF) return false;
  const Footprint f = footprint(batch, m, n, k);
  if (tiles >= sm_count && preferred_by_rounds(batch, n, k, tiles, f, sm_count)) return true;
  if (f.matrices > 1 && f.matrices < 4 && f.ctas < 2) return false;
  const bool shared_b = batch == 1, direct = on_sectors && writes_rows(n, k, shared_b);
  if ((direct ? footprint(batch, m, n, k, false).ctas : f.ctas) < 2 || one_piece_round(k, n, shared_b, f, tiles, sm_count)) return false;
  if (k <= 40) {
    return tiles >= 64 && (n <= 112 || (n < 128 && tiles >= sm_count && (m <= 65 || tiles >= 5 * sm_count)));
  }
  if (tiles > 950) return m <= 65 || (shared_b && n <= 112);
  if (tiles < sm_count || n > 80 || k > 88) return false;
  const double rounds = static_cast<double>(tiles) / (static_cast<double>(f.ctas) * sm_count);
  return direct || (rounds >= 0.4 && (rounds <= 0.95 || rounds >= 1.35));
}

cudaError_t launch_packed_gemm(const PackedProblem& pr) {
  Footprint f = footprint(pr.batch, pr.m, pr.n, pr.k);
  const bool direct = writes_rows(pr.n, pr.k, pr.batch == 1) && on_sectors(pr.out);
  if (direct) {
    const Footprint staged = f;
    f = footprint(pr.batch, pr.m, pr.n, pr.k, false);
    f.piped = staged.piped;  // by the CTAs that staging leaves: the form was chosen between with them
    if (f.units <= static_cast<int64_t>(staged.ctas) * pr.sm_count) {
      // A single round as it was: the room would let some SMs take more units than others (see below; mm 56229x80x48 5.4 ->
      // 6.3, 28359x112x40 6.5 -> 7.3).
      f.smem = staged.smem;
      f.ctas = staged.ctas;
    }
  }
  PackedParams p = {};
  p.a = static_cast<const uint8_t*>(pr.a);
  p.b = static_cast<const uint8_t*>(pr.b);
  p.bias = pr.bias;
  p.out = static_cast<uint8_t*>(pr.out);
  p.batch = static_cast<int>(pr.batch);
  p.m = static_cast<int>(pr.m);
  p.n = static_cast<int>(pr.n);
  p.k_chunks = static_cast<int>(pr.k / 8);
  p.k_blocks = f.k_blocks;
  p.matrices = f.matrices;
  p.slot_rows = kRows / p.matrices;
  p.row_tiles = (p.m + kRows - 1) / kRows;
  p.units = p.matrices == 1 ? p.batch * p.row_tiles : (p.batch + p.matrices - 1) / p.matrices;
  p.mma_n = f.mma_n;
  p.shared_b = p.batch == 1 ? 1 : 0;
  p.narrow = f.narrow;
  p.idesc = pr.idesc_base | (static_cast<uint32_t>(p.mma_n >> 3) << 17);
  p.staging_pitch = static_cast<uint32_t>(f.staging_pitch);
  p.load_rows = kThreads / p.k_chunks;
  p.load_threads = p.load_rows * p.k_chunks;
  p.div_k_chunks = FastDiv::make(static_cast<uint32_t>(p.k_chunks));
  p.div_n_chunks = FastDiv::make(static_cast<uint32_t>(p.n / 8));
  p.div_row_tiles = FastDiv::make(static_cast<uint32_t>(p.row_tiles));
  p.status = pr.status;
  p.timeout_ns = pr.timeout_ns;
  p.debug_flags = pr.debug_flags;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.mma_n) p.tmem_cols *= 2;
  if (f.piped) p.tmem_cols = f.piped_tmem_cols;
  p.stages = f.stages;

  const int64_t room = static_cast<int64_t>(f.piped ? f.piped_ctas : f.ctas) * pr.sm_count;

  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(p.units < room ? p.units : room));
  cfg.blockDim = dim3(f.piped ? kPipedThreads : kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(f.piped ? f.piped_smem : f.smem);
  // The launch hardware deals CTAs out by shared memory, registers and threads: with little of them an SM may get five and
  // another three, and TMEM, which it does not count, may hold only four, so that the fifth starts when another has done all
  // its units.  From 1.6 rounds on each takes its share of the SM's shared memory, and no SM gets more (us: bmm 5400 x
  // 26x96x8 23.8 -> 17.4, 2500 x 64x96x16 14.2 -> 11.6, mm 262144x48x32 11.7 -> 10.5, 125610x80x16 8.2 -> 7.3).  With fewer
  // units the next launch's CTAs better set up beside them (mm 21517x72x24 5.0 -> 5.6, bmm 444 x 31x88x8 3.3 -> 4.0, 1776 x
  // 15x48x8 4.1 -> 4.5), and accumulators of 32 columns are too small to matter (4576 x 47x16x16 6.9 -> 7.0).
  if (!f.piped && p.tmem_cols >= 64 && f.units * 5 >= room * 8 && kSmemPerSm / (f.smem + kCtaReserve) > f.ctas) {
    cfg.dynamicSmemBytes = static_cast<size_t>(kSmemPerSm / f.ctas - kCtaReserve);
  }
  cfg.stream = pr.stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pr.overlap ? 1 : 0;
  using Kernel = void (*)(PackedParams);
  static const Kernel kernels[2][2][2] = {  // [piped][direct][bf16]
      {{packed_gemm_kernel<false, false>, packed_gemm_kernel<true, false>},
       {packed_gemm_kernel<false, true>, packed_gemm_kernel<true, true>}},
      {{packed_piped_kernel<false, false>, packed_piped_kernel<true, false>},
       {packed_piped_kernel<false, true>, packed_piped_kernel<true, true>}},
  };
  return cudaLaunchKernelEx(&cfg, kernels[f.piped ? 1 : 0][direct ? 1 : 0][pr.is_bf16 ? 1 : 0], p);
}

}  // namespace ayla_b200
