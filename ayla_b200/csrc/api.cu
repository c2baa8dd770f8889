// C ABI of the sm_100a GEMM backend: argument checks, schedule choice, tensor-map
// encoding and the kernel launch.  Nothing here allocates device memory or
// synchronises but ayla_b200_capture_workspace, which is for captures, so every entry
// point except ayla_b200_init can run inside CUDA graph capture.
#include "../../include/ayla_b200.h"

#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <unordered_map>
#include <vector>

#include "capture_workspace.h"
#include "kernel_registry.h"
#include "packed_gemm.h"
#include "rms_factors.h"

namespace ayla_b200 {
namespace {

thread_local std::string g_last_error;

int fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  g_last_error = buf;
  return code;
}

constexpr int kMaxDevices = 64;

struct Registry {
  std::vector<KernelEntry> entries;
  Registry() {
    append_variants_cg1(&entries);
    append_variants_cg2(&entries);
    append_variants_trans(&entries);
    append_variants_swiglu(&entries);
    base_count = static_cast<int>(entries.size());
    append_variants_swiglu_trans(&entries);
    append_variants_act_cg1(&entries);
    append_variants_act_cg2(&entries);
    append_variants_act_trans(&entries);
    append_variants_lean_cg1(&entries);
    append_variants_lean_cg2(&entries);
    append_variants_lean_trans(&entries);
    append_variants_lean_act_cg1(&entries);
    append_variants_lean_act_cg2(&entries);
    append_variants_lean_act_trans(&entries);
    append_variants_paired_cg1(&entries);
    append_variants_paired_cg2(&entries);
    append_variants_shared_cg1(&entries);
    append_variants_shared_cg2(&entries);
    append_variants_shared_act_cg1(&entries);
    append_variants_shared_act_cg2(&entries);
    append_variants_gated_cg1(&entries);
    append_variants_gated_cg2(&entries);
    append_variants_flat(&entries);
  }
  int base_count = 0;  // the variants without the activation epilogue come first
  // Where there is no variant of the form asked for, the one with all epilogues serves.
  const KernelEntry* find(int tile_n, int cta_group, int epilogue, int transposed, int activation = 0,
                          int form = FORM_FULL) const {
    const KernelEntry* full = nullptr;
    for (const KernelEntry& e : entries) {
      if (e.tile_n == tile_n && e.cta_group == cta_group && e.epilogue == epilogue &&
          e.transposed_out == transposed && e.activation == activation) {
        if (e.form == form) return &e;
        if (e.form == FORM_FULL) full = &e;
      }
    }
    return full;
  }
};

const Registry& registry() {
  static const Registry& r = *new Registry;  // kept for good: threads may launch while the process exits
  return r;
}

// SMs, and how many clusters of four and of eight CTAs with a ring of shared memory each run at the same time: fewer
// than the SMs would hold, since a cluster lies within one GPC (33 and 15 on a B200 of 148 SMs).
struct Machine {
  int sm_count = 148, clusters4 = 33, clusters8 = 15;
  int clusters(int ctas) const { return ctas >= 8 ? clusters8 : ctas >= 4 ? clusters4 : sm_count / ctas; }
};
struct DeviceState {
  std::atomic<bool> ready{false};
  int sm_count = 0;
  Machine machine;
};
DeviceState g_devices[kMaxDevices];
std::mutex g_init_mutex;
PFN_cuTensorMapEncodeTiled g_encode_tiled = nullptr;
std::atomic<long long> g_timeout_ns{2000000000ll};
std::atomic<int> g_debug_flags{0};
std::atomic<int> g_launch_overlap{1};

// ------------------------------------------------------------- tensor maps

struct MapKey {
  const void* ptr;
  uint64_t d0, d1, d2;
  uint32_t b0, b1, b2;
  bool operator==(const MapKey& o) const {
    return ptr == o.ptr && d0 == o.d0 && d1 == o.d1 && d2 == o.d2 && b0 == o.b0 && b1 == o.b1 &&
           b2 == o.b2;
  }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    uint64_t h = reinterpret_cast<uint64_t>(k.ptr) * 0x9E3779B97F4A7C15ull;
    h ^= (k.d0 + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2));
    h ^= (k.d1 + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2));
    h ^= (k.d2 + 0x9E3779B97F4A7C15ull + (h << 6) + (h >> 2));
    h ^= ((static_cast<uint64_t>(k.b0) << 40) ^ (static_cast<uint64_t>(k.b1) << 20) ^ k.b2) +
         (h << 6) + (h >> 2);
    return static_cast<size_t>(h);
  }
};

// Descriptors are pure functions of (pointer, extents, box); cache them by value
// as the reference's launcher does (ayla/ptx_runtime.py:185-235), behind a mutex
// because this library does not rely on the GIL.
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_map_cache;
std::mutex g_map_mutex;

// 3-D map over a row-major [d2][d1][d0] tensor of 16-bit elements, box
// [b2][b1][b0], 128-byte swizzle (b0 must be 64 elements).
int encode_map(CUtensorMap* out, const void* ptr, uint64_t d0, uint64_t d1, uint64_t d2, uint32_t b0,
               uint32_t b1, uint32_t b2) {
  const MapKey key{ptr, d0, d1, d2, b0, b1, b2};
  {
    std::lock_guard<std::mutex> lock(g_map_mutex);
    auto it = g_map_cache.find(key);
    if (it != g_map_cache.end()) {
      *out = it->second;
      return AYLA_B200_OK;
    }
  }
  const cuuint64_t dims[3] = {d0, d1, d2};
  const cuuint64_t strides[2] = {d0 * 2, d0 * d1 * 2};
  const cuuint32_t box[3] = {b0, b1, b2};
  const cuuint32_t elem_strides[3] = {1, 1, 1};
  auto encode = [&] {
    return g_encode_tiled(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box,
                          elem_strides, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = encode();
  if (r == CUDA_ERROR_INVALID_CONTEXT) {
    // A thread's first CUDA call may be this one, which wants a current context: selecting the current
    // device makes its primary context current.
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && cudaSetDevice(device) == cudaSuccess) r = encode();
  }
  if (r != CUDA_SUCCESS) {
    return fail(AYLA_B200_E_CUDA,
                "cuTensorMapEncodeTiled failed (%d) for ptr=%p dims=[%llu,%llu,%llu] box=[%u,%u,%u]",
                static_cast<int>(r), ptr, (unsigned long long)d0, (unsigned long long)d1,
                (unsigned long long)d2, b0, b1, b2);
  }
  std::lock_guard<std::mutex> lock(g_map_mutex);
  if (g_map_cache.size() > 8192) g_map_cache.clear();
  g_map_cache.emplace(key, *out);
  return AYLA_B200_OK;
}

// ------------------------------------------------------------ the schedule

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// The problem as the kernel sees it after an optional swap of the operands.
struct Problem {
  int64_t rows, cols, k, batch;  // rows fill the 128-row tile, cols the accumulator width
  const void* row_operand;       // [batch][rows][k]
  const void* col_operand;       // [batch][cols][k]
};

struct Plan {
  const KernelEntry* kernel;
  int m_tiles, n_tiles, k_blocks, splits, kb_per_split, total_units, group_m, grid;
  int split_from_tile;  // first k-split tile (0 = all tiles split, == tiles when none is)
  int narrow_from_tile; // first tile done as two half-width units (== tiles when none is)
  int stream_k, kb_per_cta;
  int cluster_split;    // cluster size of the cluster split-K schedule (0 = not used)
  long long slabs;      // fp32 partial-sum slabs of 128 x tile_n the schedule may write
  int row_tiles;  // 128-row x tile_n tiles (split-K counters, slabs)
  int shared_reduce;  // the CTAs that split a tile's depth through the workspace share the sum
  int tile_rows;  // rows of the row operand per tile (128 unless the swapped form trims it)
};

int check_shape(int op, int dtype, int64_t batch, int64_t m, int64_t n, int64_t k) {
  if (op != AYLA_B200_OP_MM && op != AYLA_B200_OP_ADDMM && op != AYLA_B200_OP_BMM) {
    return fail(AYLA_B200_E_INVALID, "unknown op %d", op);
  }
  if (dtype != AYLA_B200_F16 && dtype != AYLA_B200_BF16) {
    return fail(AYLA_B200_E_INVALID, "unknown dtype %d (0 = float16, 1 = bfloat16)", dtype);
  }
  if (batch <= 0 || m <= 0 || n <= 0 || k <= 0) {
    return fail(AYLA_B200_E_INVALID, "non-positive extent batch=%lld m=%lld n=%lld k=%lld",
                (long long)batch, (long long)m, (long long)n, (long long)k);
  }
  if (op != AYLA_B200_OP_BMM && batch != 1) {
    return fail(AYLA_B200_E_INVALID, "batch must be 1 for mm/addmm, got %lld", (long long)batch);
  }
  if (n % 8 != 0) {
    return fail(AYLA_B200_E_UNSUPPORTED, "n=%lld must be a multiple of 8 (16-byte output rows)",
                (long long)n);
  }
  if (k % 8 != 0) {
    return fail(AYLA_B200_E_UNSUPPORTED, "k=%lld must be a multiple of 8 (16-byte operand rows)",
                (long long)k);
  }
  if (m > 0x7FFFFFFF / 2 || n > 0x7FFFFFFF / 2 || k > 0x7FFFFFFF / 2 || batch > 65535 * 16) {
    return fail(AYLA_B200_E_UNSUPPORTED, "extent too large for 32-bit tile coordinates");
  }
  return AYLA_B200_OK;
}

int check_config(const ayla_b200_config& c, bool swiglu) {
  if (c.cta_group != 1 && c.cta_group != 2) {
    return fail(AYLA_B200_E_UNSUPPORTED, "cta_group must be 1 or 2, got %d", c.cta_group);
  }
  if (c.split_k < 1 || c.group_m < 1 || c.grid_ctas < 0) {
    return fail(AYLA_B200_E_UNSUPPORTED, "split_k and group_m must be >= 1, grid_ctas >= 0");
  }
  if (c.split_tail < 0 || c.split_tail > 2) {
    return fail(AYLA_B200_E_UNSUPPORTED, "split_tail must be 0, 1 or 2");
  }
  if (c.cluster_split != 0 && c.cluster_split != 1) {
    return fail(AYLA_B200_E_UNSUPPORTED, "cluster_split must be 0 or 1");
  }
  if (c.cluster_split) {
    if (swiglu || c.stream_k || c.split_tail) {
      return fail(AYLA_B200_E_UNSUPPORTED,
                  "cluster_split excludes stream_k, split_tail and the SwiGLU kernel");
    }
    // The cluster has split_k * cta_group CTAs, 8 at most.
    if (c.split_k != 2 && c.split_k != 4 && !(c.split_k == 8 && c.cta_group == 1)) {
      return fail(AYLA_B200_E_UNSUPPORTED,
                  "cluster_split needs split_k in {2, 4, 8} and a cluster (split_k * cta_group) of at most 8 CTAs");
    }
    if (c.tile_n % (4 * c.split_k) != 0 || (c.tile_n & (c.tile_n - 1)) != 0) {
      return fail(AYLA_B200_E_UNSUPPORTED,
                  "cluster_split needs a power-of-two tile_n that is a multiple of 4 * split_k");
    }
  }
  if (c.l2_prefetch < 0 || c.l2_prefetch > 256) {
    return fail(AYLA_B200_E_UNSUPPORTED, "l2_prefetch must be between 0 and 256 k-blocks");
  }
  if (c.early_prefetch < 0 || c.early_prefetch > 32) {
    return fail(AYLA_B200_E_UNSUPPORTED, "early_prefetch must be between 0 and 32 k-blocks");
  }
  if (c.stream_k != 0 && c.stream_k != 1) {
    return fail(AYLA_B200_E_UNSUPPORTED, "stream_k must be 0 or 1");
  }
  if (c.stream_k && (swiglu || c.split_k != 1 || c.split_tail != 0)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "stream_k excludes split_k > 1, split_tail and the SwiGLU kernel");
  }
  if (c.split_tail == 2 && (swiglu || c.swap_ab || c.split_k != 1 || c.tile_n % 128 != 0)) {
    return fail(AYLA_B200_E_UNSUPPORTED,
                "split_tail = 2 (half-width last wave) needs tile_n of 128 or 256, split_k = 1 and no swap_ab");
  }
  if (c.l2_hint_a < 0 || c.l2_hint_a > 2 || c.l2_hint_b < 0 || c.l2_hint_b > 2) {
    return fail(AYLA_B200_E_UNSUPPORTED, "L2 hints must be 0, 1 or 2");
  }
  if (swiglu) {
    if (c.split_k != 1 || c.swap_ab != 0) {
      return fail(AYLA_B200_E_UNSUPPORTED, "the SwiGLU kernel has no split-K or swapped form");
    }
    return AYLA_B200_OK;
  }
  if (c.tile_rows != 0 && (!c.swap_ab || c.tile_rows < 8 || c.tile_rows > 128)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "tile_rows needs swap_ab = 1 and a value between 8 and 128 (0 = 128)");
  }
  if (c.swap_ab) {
    if (c.cta_group != 1) {
      return fail(AYLA_B200_E_UNSUPPORTED, "swap_ab is only built with cta_group == 1");
    }
    if (c.tile_n != 16 && c.tile_n != 32 && c.tile_n != 64 && c.tile_n != 128) {
      return fail(AYLA_B200_E_UNSUPPORTED, "swap_ab needs tile_n in {16,32,64,128}, got %d", c.tile_n);
    }
  } else if (c.tile_n != 64 && c.tile_n != 128 && c.tile_n != 192 && c.tile_n != 256) {
    return fail(AYLA_B200_E_UNSUPPORTED, "tile_n must be 64, 128, 192 or 256, got %d", c.tile_n);
  }
  return AYLA_B200_OK;
}

// The arrival counters live in a header of fixed size at the start of the
// workspace, whatever the shape, so one zero-initialised workspace can serve
// launches of different shapes: data slabs never overlay a counter.
constexpr int kMaxSplitKTiles = 16384;
constexpr size_t kCounterBytes = static_cast<size_t>(kMaxSplitKTiles) * 4;

// How long the owner of a piece of a split tile waits for the other partials before it leaves the piece to the last
// of them: far above the few microseconds by which CTAs that run together differ, and little where they do not.
constexpr unsigned kHandoverNs = 20000;

// Fills `plan` for a validated config.  `epilogue` is one of EPI_*.
int make_plan(const ayla_b200_config& c, int epilogue, int64_t batch, int64_t rows, int64_t cols,
              int64_t k, int sm_count, Plan* plan, int activation = 0) {
  const int transposed = c.swap_ab ? 1 : 0;
  const bool swiglu_cols = epilogue == EPI_SWIGLU && !c.swap_ab;
  const int tile_n = swiglu_cols ? 256 : c.tile_n;
  const int form = (c.split_k <= 1 && c.stream_k == 0) ? FORM_LEAN : FORM_FULL;
  // `activation` 3: one that is more than a comparison, for which those launches have kernels with sixteen epilogue
  // warps (see GemmTraits::PAIRED; with a comparison or a row factor alone eight do as well or better: RMS norm and
  // projection 4096x6144x4096 172 against 173 us).
  // `activation` 2: a gate operand shaped like the output, for which the launches without a k-split have kernels of
  // their own (us per launch, before -> with them: 16384x2048x256 71.4 -> 38.1, 6983x1472x1312 43.8 -> 32.2,
  // 1024x4096x512 15.3 -> 12.0, 64x8192x1024 10.4 -> 8.9); the k-split and swapped forms load it directly.
  const KernelEntry* e = nullptr;
  if (activation == 2 && form == FORM_LEAN) e = registry().find(tile_n, c.cta_group, epilogue, transposed, 2, FORM_LEAN);
  if (e == nullptr && rows <= 128 && c.cta_group == 2 && !transposed && c.stream_k == 0 && c.split_tail == 0 &&
      (c.split_k <= 1 || c.cluster_split)) {
    const KernelEntry* flat = registry().find(tile_n, 2, epilogue, transposed, activation != 0 ? 1 : 0, FORM_FLAT);
    if (flat != nullptr && flat->form == FORM_FLAT) e = flat;
  }
  if (e == nullptr && activation == 3 && form == FORM_LEAN) {
    e = registry().find(tile_n, c.cta_group, epilogue, transposed, 3, FORM_LEAN);
  }
  if (e == nullptr) e = registry().find(tile_n, c.cta_group, epilogue, transposed, activation != 0 ? 1 : 0, form);
  if (e == nullptr) {
    return fail(AYLA_B200_E_UNSUPPORTED, "no kernel variant tile_n=%d cta_group=%d epilogue=%d swap=%d",
                tile_n, c.cta_group, epilogue, transposed);
  }
  const int out_tile_n = swiglu_cols ? 128 : tile_n;
  plan->kernel = e;
  plan->tile_rows = (c.swap_ab && c.tile_rows > 0) ? c.tile_rows : 128;
  plan->m_tiles = static_cast<int>(ceil_div(rows, c.swap_ab ? plan->tile_rows : e->cta_rows * c.cta_group));
  plan->n_tiles = static_cast<int>(ceil_div(cols, out_tile_n));
  plan->k_blocks = static_cast<int>(ceil_div(k, 64));
  int splits = c.split_k;
  if (splits > plan->k_blocks) splits = plan->k_blocks;
  plan->kb_per_split = static_cast<int>(ceil_div(plan->k_blocks, splits));
  plan->splits = static_cast<int>(ceil_div(plan->k_blocks, plan->kb_per_split));
  const int64_t tiles = static_cast<int64_t>(batch) * plan->m_tiles * plan->n_tiles;
  if (tiles * c.cta_group > 0x7FFFFFFF) {
    return fail(AYLA_B200_E_UNSUPPORTED, "too many tiles (%lld)", (long long)tiles);
  }
  int grid = (c.grid_ctas > 0) ? c.grid_ctas : sm_count;
  if (c.cta_group == 2) {
    grid &= ~1;
    if (grid < 2) grid = 2;
  } else if (grid < 1) {
    grid = 1;
  }
  plan->stream_k = 0;
  plan->kb_per_cta = 0;
  plan->cluster_split = 0;  // also for the stream-K plan below, which returns before the cluster branch
  plan->shared_reduce = 0;
  if (c.stream_k) {
    // Equal contiguous shares of the (tile, k-block) sequence; a share is never shorter
    // than four k-blocks so that a segment is worth its epilogue.
    const int64_t total_kb = tiles * plan->k_blocks;
    if (total_kb > 0x7FFFFFFF) {
      return fail(AYLA_B200_E_UNSUPPORTED, "too much work for the stream-K schedule (%lld k-blocks)",
                  (long long)total_kb);
    }
    int64_t ctas = grid / c.cta_group;
    int64_t share = ceil_div(total_kb, ctas);
    const int64_t min_share = plan->k_blocks < 4 ? plan->k_blocks : 4;
    if (share < min_share) share = min_share;
    ctas = ceil_div(total_kb, share);
    if (ctas * c.cta_group > kMaxSplitKTiles) {
      return fail(AYLA_B200_E_UNSUPPORTED, "stream_k over %lld CTAs (limit %d arrival counters)",
                  (long long)(ctas * c.cta_group), kMaxSplitKTiles);
    }
    plan->stream_k = 1;
    plan->kb_per_cta = static_cast<int>(share);
    plan->splits = 1;
    plan->kb_per_split = plan->k_blocks;
    plan->split_from_tile = static_cast<int>(tiles);
    plan->narrow_from_tile = 0x7FFFFFFF;
    plan->total_units = static_cast<int>(total_kb);
    plan->row_tiles = static_cast<int>(ctas * c.cta_group);
    // No tile is cut when every share is a whole number of tiles.
    plan->slabs = (share % plan->k_blocks == 0) ? 0 : 2 * ctas * c.cta_group;
    plan->group_m = c.group_m;
    plan->grid = static_cast<int>(ctas * c.cta_group);
    return AYLA_B200_OK;
  }
  plan->cluster_split = 0;
  if (c.cluster_split) {
    // One cluster of split_k CTAs (CTA pairs) per tile, one tile per cluster; every k-split
    // must be non-empty.
    const int s_k = c.split_k;
    const int per = static_cast<int>(ceil_div(plan->k_blocks, s_k));
    if (static_cast<int64_t>(s_k - 1) * per >= plan->k_blocks) {
      return fail(AYLA_B200_E_UNSUPPORTED, "cluster_split: %d k-blocks cannot be shared by %d CTAs",
                  plan->k_blocks, s_k);
    }
    if (tiles * s_k * c.cta_group > 0x7FFFFFFF) {
      return fail(AYLA_B200_E_UNSUPPORTED, "too many tiles (%lld)", (long long)tiles);
    }
    plan->cluster_split = s_k;
    plan->splits = s_k;
    plan->kb_per_split = per;
    plan->split_from_tile = 0;
    plan->narrow_from_tile = 0x7FFFFFFF;
    plan->total_units = static_cast<int>(tiles);
    plan->row_tiles = 0;
    plan->slabs = 0;
    plan->group_m = c.group_m;
    plan->grid = static_cast<int>(tiles * s_k * c.cta_group);
    return AYLA_B200_OK;
  }
  // Tiles processed at the same time by the persistent grid.
  const int64_t wave = grid / c.cta_group;
  int64_t split_from = 0;
  if (plan->splits <= 1) {
    split_from = tiles;
  } else if (c.split_tail) {
    // Only the tiles of the last, partial wave are k-split; with less than one wave of
    // tiles that is all of them, with a whole number of waves none.
    split_from = (tiles / wave) * wave;
    if (split_from == tiles) {
      plan->splits = 1;
      plan->kb_per_split = plan->k_blocks;
    }
  }
  plan->split_from_tile = static_cast<int>(split_from);
  int64_t narrow_from = tiles;
  if (c.split_tail == 2 && tiles > wave && tiles % wave != 0) {
    // The tiles of the last, partial wave are done as two half-width units each.
    narrow_from = (tiles / wave) * wave;
  }
  // INT_MAX = no narrow units (unit indices of k-split tiles run past `tiles`).
  plan->narrow_from_tile = (narrow_from == tiles) ? 0x7FFFFFFF : static_cast<int>(narrow_from);
  const int64_t units = split_from + (tiles - split_from) * plan->splits + (tiles - narrow_from);
  if (units > 0x7FFFFFFF) {
    return fail(AYLA_B200_E_UNSUPPORTED, "too many work units (%lld)", (long long)units);
  }
  plan->total_units = static_cast<int>(units);
  plan->row_tiles = static_cast<int>((tiles - split_from) * c.cta_group);
  if (plan->splits > 1 && plan->row_tiles > kMaxSplitKTiles) {
    return fail(AYLA_B200_E_UNSUPPORTED, "split_k with %d output tiles (limit %d); use split_k = 1",
                plan->row_tiles, kMaxSplitKTiles);
  }
  plan->slabs = (plan->splits > 1) ? static_cast<long long>(plan->row_tiles) * plan->splits : 0;
  plan->group_m = c.group_m;
  if (wave > units) grid = static_cast<int>(units * c.cta_group);
  plan->grid = grid;
  // At most one split unit per CTA, its last: those of a tile share its sum.  With more of them a CTA would wait for
  // partials that it, or one that waits as well, has yet to compute; there the last arriver sums.  (320 schedules timed
  // both ways, two to sixteen splits: 0.74 of the last arriver's time, none slower; 0.99 to 0.78 with two.)
  if (plan->splits > 1 && split_from % wave == 0 && (tiles - split_from) * plan->splits <= wave && !transposed &&
      static_cast<int64_t>(plan->row_tiles) * (tile_n / 32) * 4 <= kMaxSplitKTiles) {
    const KernelEntry* shared =
        registry().find(tile_n, c.cta_group, epilogue, transposed, activation != 0 ? 1 : 0, FORM_SHARED);
    if (shared != nullptr && shared->form == FORM_SHARED) {
      plan->kernel = shared;
      plan->shared_reduce = 1;
    }
  }
  return AYLA_B200_OK;
}

size_t counter_bytes_for(const Plan& p) {
  if (p.slabs <= 0) return 0;
  return kCounterBytes;
}

size_t workspace_bytes_for(const Plan& p) {
  if (p.slabs <= 0) return 0;
  return counter_bytes_for(p) + static_cast<size_t>(p.slabs) * 128 * p.kernel->tile_n * sizeof(float);
}

uint32_t make_idesc(int is_bf16, int mma_m, int mma_n) {
  // tcgen05 .kind::f16 instruction descriptor: fp32 accumulator (bits 4-5 = 1),
  // A/B element format (bits 7-9 / 10-12: 0 = f16, 1 = bf16), both operands
  // K-major (bits 15, 16 = 0), N >> 3 in bits 17-22, M >> 4 in bits 24-28.
  uint32_t d = 0;
  d |= 1u << 4;
  d |= static_cast<uint32_t>(is_bf16 ? 1 : 0) << 7;
  d |= static_cast<uint32_t>(is_bf16 ? 1 : 0) << 10;
  d |= static_cast<uint32_t>(mma_n >> 3) << 17;
  d |= static_cast<uint32_t>(mma_m >> 4) << 24;
  return d;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int current_device_state(DeviceState** out, int* device) {
  int dev = -1;
  const cudaError_t err = cudaGetDevice(&dev);
  if (err != cudaSuccess) {
    return fail(AYLA_B200_E_CUDA, "cudaGetDevice: %s", cudaGetErrorString(err));
  }
  if (dev < 0 || dev >= kMaxDevices || !g_devices[dev].ready.load(std::memory_order_acquire)) {
    return fail(AYLA_B200_E_NOT_INIT, "ayla_b200_init(%d) has not been called", dev);
  }
  *out = &g_devices[dev];
  *device = dev;
  return AYLA_B200_OK;
}

// For queries, which need no device: the current device's where it has been set up, else a B200's.
Machine current_machine() {
  int dev = -1;
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices &&
      g_devices[dev].ready.load(std::memory_order_acquire)) {
    return g_devices[dev].machine;
  }
  (void)cudaGetLastError();
  return Machine{};
}
int current_sm_count() { return current_machine().sm_count; }

// Whether the tiles chosen for a product of at most four k-blocks are better run by CTA pairs, which read half as much
// of B.  170 shapes timed in both forms: with this rule the paired ones take 0.946 of the time without an activation
// (the slowest 1.05), the others would take 1.035.  us, single -> pair:
//  * from two waves of 256-wide tiles on, and of 128-wide ones of three or four k-blocks (mm 8216x4976x104 29.1 -> 24.1,
//    15515x1592x128 14.8 -> 14.1, addmm 12010x552x192 8.8 -> 8.6; in one wave pairing only adds set-up: mm
//    1236x6728x192 7.5 -> 7.7, 3755x816x192 5.1 -> 5.3; 128-wide tiles of two k-blocks: mm 2437x1696x96 5.0 -> 5.3);
//  * from one wave on where rows start in the middle of a 32-byte sector, so that B's are read twice (addmm
//    10684x280x216 8.7 -> 7.3, mm 9609x552x120 7.7 -> 6.6);
//  * not where 256-row tiles add much padding to the rows (bmm 28 x 1873x1576x128, 7 %: 40.5 -> 46.6; 82 x
//    1335x1064x128, 9 %: 58.5 -> 72.8), more of which a deeper or misaligned product bears (bmm 26 x 830x1264x256, 14 %:
//    21.4 -> 19.6);
//  * behind an activation only without padding: its rows pass through the epilogue too (bmm 26 x 830x1264x256 with
//    SiLU 1.12).  There pairs take 0.96 of the time with SiLU and GELU, 0.99 with sigmoid and GELU-tanh, 0.81 to 1.04.
bool shallow_pairs_pay(int64_t batch, int64_t m, int64_t n, int64_t k, int tile_n, int activation, int sm_count) {
  const int64_t k_blocks = ceil_div(k, 64);
  if (k_blocks > 4 || m < 256 || tile_n < 128) return false;
  const bool mid_sector = k % 16 != 0;
  const int64_t row_tiles = ceil_div(m, 128);
  const double growth = static_cast<double>(2 * ceil_div(m, 256)) / static_cast<double>(row_tiles);
  if (growth > (activation == AYLA_B200_ACT_NONE && (k_blocks >= 3 || mid_sector) ? 1.2 : 1.03)) return false;
  const double waves = static_cast<double>(batch * row_tiles * ceil_div(n, tile_n)) / sm_count;
  return mid_sector ? waves >= 1.0 : waves >= 2.0 && (tile_n == 256 || k_blocks >= 3);
}

void default_config(int64_t batch, int64_t m, int64_t n, int64_t k, int activation, const Machine& machine,
                    ayla_b200_config* c) {
  const int sm_count = machine.sm_count;
  memset(c, 0, sizeof(*c));
  c->cta_group = 1;
  c->split_k = 1;
  c->group_m = 8;
  // L2 eviction hints: `a` (re-read by every column tile) is kept, `bt` (streamed) goes first.
  // In the sweep almost any hint beat none (2-10 % on mid-size shapes); this pair won most often.
  c->l2_hint_a = 2;
  c->l2_hint_b = 1;
  const int64_t k_blocks = ceil_div(k, 64);
  if (m <= 64 && n >= 128) {
    // Weight-streaming regime: put bt's rows on the 128-row tile and M on the
    // narrow accumulator, then split K until every SM has a share of the stream.
    c->swap_ab = 1;
    c->tile_n = m <= 16 ? 16 : (m <= 32 ? 32 : 64);
    const int64_t tiles = batch * ceil_div(n, 128);
    // Split K across a cluster of 8, 4 or 2 (summed through distributed shared memory) while all the clusters run at
    // once and every CTA keeps a few k-blocks.  us, all at once -> in two waves: 12x4608x5504, 36 tiles, clusters of
    // two 12.2, of four 17.0; 17x4568x2520, 36 tiles, 8.9 and 12.7; 2x4160x8704, 33 tiles, clusters of four 13.2, of
    // two 15.9.  Eight for deep products of the fewest tiles (28x1824x9144, 15 tiles, clusters of eight 9.8, of four
    // 12.6; 32x2112x2560, 17 tiles, 9.6 and 5.7).
    for (int s = 8; s >= 2; s /= 2) {
      const int width = s == 8 && c->tile_n < 32 ? 32 : c->tile_n;
      if (tiles <= machine.clusters(s) && k_blocks >= (s == 8 ? 140 : 4 * s) && width % (4 * s) == 0) {
        c->tile_n = width;
        c->split_k = s;
        c->cluster_split = 1;
        break;
      }
    }
    c->group_m = 1;
    // Weight streaming is what early_prefetch is for: half of the CTA's share of K, 16 k-blocks at most.
    {
      const int64_t share = k_blocks / c->split_k / 2;
      // (Eight blocks of a wider accumulator's, whose loads come with more of `a`: 62x6656x5440 with a gate 16 blocks 27.0,
      // 12 24.9, 8 24.1; without 17.0, 16.8, 16.9.)
      const int64_t most = c->tile_n >= 64 ? 8 : 16;
      c->early_prefetch = static_cast<int>(share < most ? share : most);
    }
    // One wave of tiles that would leave SMs idle is cut into as many as there are SMs (3x13056x1728, 102 -> 136 tiles,
    // 9.7 -> 9.1; 7x13696x5504, 107 -> 143, 24.5 -> 23.6; 44x12216x4760, 96 -> 139, 30.8 -> 27.5), a split one where the
    // stream is long (2x5888x7200, 46 -> 74, 17.0 -> 16.0; 9x6208x11200, 49 -> 71, 25.6 -> 24.4; but 14x7552x1536,
    // 59 -> 73, 6.3 -> 6.6).
    if (c->split_k <= 2 && batch == 1) {
      const int64_t rows = ceil_div(ceil_div(n, sm_count / c->split_k), 8) * 8;
      if (rows >= 72 && rows <= 96 && k_blocks / c->split_k >= (c->split_k == 1 ? 20 : 48)) {
        c->tile_rows = static_cast<int>(rows);
      }
    }
    if (c->split_k == 1 && m > 16 && (c->tile_rows == 0 || k_blocks < 40 || (activation != AYLA_B200_ACT_NONE && m > 32))) {
      // No room to split K (bt alone fills the SMs): with a few dozen rows of `a` the plain
      // row-major 128-wide tile, its `a` box trimmed to the rows that exist, measures 1.2-1.3x
      // faster than the swapped form (M = 32, 64 at N = 14336).  Trimmed tiles are faster still for deep
      // products (above), but not over a 64-wide accumulator before a gate, which the swapped form reads
      // with direct loads and the row-major kernels through their staging rows (38x11512x2952 row-major
      // 22.0, swapped 25.7; 40x10752x8704 39.8 and 41.6; of 32 rows and fewer 20x11136x5312 27.1 and 25.9).
      // Gates come with an activation.
      c->swap_ab = 0;
      c->tile_rows = 0;
      c->tile_n = (batch * ceil_div(n, 128) <= static_cast<int64_t>(sm_count)) ? 128 : 256;  // one wave if it fits
      c->group_m = 8;
      c->split_tail = 2;
    }
    return;
  }
  // Row-major form: pick (tile width, CTA pairing, k-split) by a small cost model fitted to
  // the B200 sweep.  Costs are in units of "one 64-deep k-block of a paired 256-wide tile at
  // full tensor rate" (about 0.28 us): a tile costs its width over the measured efficiency of
  // its shape, waves are whole, a k-split pays a fixed fix-up and every launch a fixed
  // prologue/epilogue that grows with the tile width.
  struct Shape { int tile_n, cta_group; double eff; };
  static const Shape kShapes[6] = {{256, 2, 1.00}, {256, 1, 0.88}, {128, 2, 0.80},
                                   {128, 1, 0.62}, {64, 2, 0.50}, {64, 1, 0.40}};
  double best_cost = 1e300;
  for (const Shape& sh : kShapes) {
    if (sh.cta_group == 2 && (m <= 128 || k_blocks <= 4)) continue;  // shallow K: see shallow_pairs_pay
    if (sh.tile_n > 64 && n * 2 <= sh.tile_n) continue;
    const int64_t ctas = sm_count / sh.cta_group;
    const int64_t tiles = batch * ceil_div(m, 128 * sh.cta_group) * ceil_div(n, sh.tile_n);
    const double tile_cost = (sh.tile_n / 256.0) / sh.eff * static_cast<double>(k_blocks);
    const double launch_cost = 6.0 + sh.tile_n / 64.0;
    for (int split = 1; split <= 16; split *= 2) {
      if (split > 1 && (k_blocks < 8 * split || tiles * split > ctas)) break;
      const int64_t units = tiles * split;
      double waves = static_cast<double>(ceil_div(units, ctas));
      int tail = 0;
      if (split == 1 && units > ctas && sh.tile_n >= 128) {
        const int64_t rest = units % ctas;
        if (rest != 0 && rest * 2 <= ctas) {
          waves -= 0.45;  // the thin last wave runs at half width
          tail = 2;
        }
      }
      // Up to four CTAs (two pairs) split K across a cluster (cheap exchange through
      // distributed shared memory); deeper splits go through the workspace, where the last
      // arriver sums `split` partial tiles one after the other.
      const bool cluster = split > 1 && split * sh.cta_group <= 4;
      // Cluster exchange: two cluster barriers plus the partial columns each CTA sends,
      // 128 x tile_n x 4 bytes x (split - 1) / split, at about 16 KB per cost unit.
      const double exchange_kb = 0.5 * sh.tile_n * (split - 1) / split;
      const double fixup = split == 1 ? 0.0 : (cluster ? 2.5 + exchange_kb / 16.0
                                                       : 4.0 + 0.9 * split * (sh.tile_n / 64.0));
      const double cost = waves * tile_cost / split + fixup + launch_cost;
      if (cost < best_cost) {
        best_cost = cost;
        c->tile_n = sh.tile_n;
        c->cta_group = sh.cta_group;
        c->split_k = split;
        c->split_tail = tail;
        c->cluster_split = cluster ? 1 : 0;
      }
    }
  }
  if (c->cta_group == 1 && c->split_k == 1 && shallow_pairs_pay(batch, m, n, k, c->tile_n, activation, sm_count)) {
    c->cta_group = 2;
    const int64_t pairs = sm_count / 2, tiles = batch * ceil_div(m, 256) * ceil_div(n, c->tile_n), rest = tiles % pairs;
    c->split_tail = tiles > pairs && rest != 0 && rest * 2 <= pairs ? 2 : 0;
  }
  // bt is streamed (evict-first) only while every row tile that needs a column tile's slab runs
  // in the same raster group; with more row tiles than that it is read again later and is kept.
  if (ceil_div(m, 128 * c->cta_group) > c->group_m) c->l2_hint_b = 2;
}

// Microseconds that a product without an activation takes where its units run in one wave: a launch, then k-blocks at a
// rate that falls with the share of the SMs at work, then, for a split depth, the sum.  Fitted to 2600 timings of 310
// shapes (tile widths of 192 between their neighbours), median error 4 %; k-blocks of rows that start inside a 32-byte
// sector take about 1.35 times as long.  One rate per tile stands for all depths: 256-wide pairs split four ways take 0.31
// us a k-block from 4096 to 8192 deep at 1024x1024 and 0.49 from there to 16384, the model 0.38.
struct Rate { double launch, block, block_busy, per_split; };
enum { RATE_WHOLE = 0, RATE_SHARED = 1, RATE_CLUSTER = 2 };
double modelled_us(int tile_n, int cta_group, int splits, int kind, int64_t tiles, int64_t k, const Machine& machine) {
  static const Rate kRates[3][4][2] = {
      {{{3.80, .147, .078, 0}, {3.20, .137, .076, 0}}, {{4.05, .221, .081, 0}, {3.80, .163, .073, 0}},
       {{4.10, .260, .130, 0}, {4.10, .210, .100, 0}}, {{4.25, .298, .180, 0}, {4.35, .256, .131, 0}}},
      {{{5.24, .156, .068, .30}, {5.16, .127, .097, .32}}, {{5.44, .203, .149, .265}, {5.87, .152, .118, .28}},
       {{6.50, .250, .210, .20}, {7.00, .200, .130, .20}}, {{7.40, .289, .281, .17}, {8.25, .260, .143, .20}}},
      {{{5.10, .170, .086, 0}, {5.10, .127, .097, 0}}, {{6.30, .262, .064, 0}, {4.30, .262, .019, 0}},
       {{6.50, .250, .210, 0}, {7.00, .200, .130, 0}}, {{7.40, .289, .281, 0}, {8.25, .260, .143, 0}}},
  };
  const Rate& r = kRates[kind][tile_n / 64 - 1][cta_group - 1];
  const int64_t at_once = kind == RATE_CLUSTER ? machine.clusters(splits * cta_group) : machine.sm_count / cta_group / splits;
  const int64_t waves = ceil_div(tiles, at_once < 1 ? 1 : at_once);
  double busy = static_cast<double>(tiles * splits * cta_group) / static_cast<double>(waves * machine.sm_count);
  if (busy > 1.0) busy = 1.0;
  const double blocks = static_cast<double>(waves * ceil_div(ceil_div(k, 64), splits)) * (k % 16 != 0 ? 1.35 : 1.0);
  return r.launch + blocks * (r.block + r.block_busy * busy) + r.per_split * splits + 4.5 * static_cast<double>(waves - 1);
}

// Microseconds that a product of more than one wave of 128- to 256-wide tiles takes, launch aside, and the number of ways its
// last wave's tiles are best split (1: not at all).  A k-block of 256-wide pairs takes 0.39 us, of 192 and 128 columns 0.34
// and 0.25 (0.23 to 0.27 in eleven products 400 to 1000 k-blocks deep); tiles of half the width two thirds of a whole one's time, as long as it where rows start inside a
// sector; the sum of S parts 4.8 us (5.8 of 192 columns) and 0.4 per part.  Fitted to 330 timings of 110 shapes.  A split has to
// gain 1 us, and 4.5 % or 3 us, by this (by 3.5 %: addmm 640x8160x3968, 1 + 22/74, halves 43.9 -> 47.0 with 3; not without the
// 3 us: 8071x2944x4480, 5 + 14/74, split five ways 171 -> halves 189).  Of 1000 shapes drawn over all kinds 61 get another
// schedule than by the bounds before, half of them whole tiles for halves that did not fit; they take 0.91 of the time.
double block_us(int tile_n) { return tile_n == 256 ? 0.39 : tile_n == 192 ? 0.34 : 0.25; }
struct LastWave { double us; int splits; };
LastWave last_wave(int64_t tiles, int64_t wave, int64_t k, int tile_n) {
  const int64_t k_blocks = ceil_div(k, 64), whole = tiles / wave, rest = tiles % wave;
  const double tile = static_cast<double>(k_blocks) * block_us(tile_n);
  LastWave best{static_cast<double>(whole) * tile, 1};
  if (rest == 0) return best;
  const double unsplit = tile_n % 128 == 0 && rest * 2 <= wave && k % 16 == 0 ? 0.66 * tile : tile;
  const double bound = 0.045 * static_cast<double>(whole + 1) * tile;
  const double sum = tile_n == 192 ? 5.8 : 4.8;
  double least = unsplit - (bound > 3.0 ? 3.0 : bound > 1.0 ? bound : 1.0);
  double last = unsplit;
  for (int s = 2; s <= 16 && s * rest <= wave && s * 5 <= k_blocks; ++s) {
    const double us = tile / s + sum + 0.4 * s;
    if (us >= least) continue;
    least = last = us;
    best.splits = s;
  }
  best.us += last;
  return best;
}

// A row-major schedule's time by the two models, roughly.
double scheduled_us(int64_t batch, int64_t m, int64_t n, int64_t k, const Machine& machine, const ayla_b200_config& c) {
  const int64_t wave = machine.sm_count / c.cta_group;
  const int64_t tiles = batch * ceil_div(m, 128 * c.cta_group) * ceil_div(n, c.tile_n);
  if (tiles > wave && !c.cluster_split) {
    return last_wave(tiles, wave, k, c.tile_n).us * (c.cta_group == 2 ? 1.0 : 1.2) * (k % 16 != 0 ? 1.2 : 1.0) + 4.3;
  }
  return modelled_us(c.tile_n, c.cta_group, c.split_k,
                     c.cluster_split ? RATE_CLUSTER : c.split_k > 1 ? RATE_SHARED : RATE_WHOLE, tiles, k, machine);
}

// Whether wider tiles in one wave pay for 128-wide pairs in more (whole sectors).  Those hide a tile's results under the next one's
// MMAs, and take less than the model says when shallow; what a lone wide tile shows of its results depends on the activation, and
// rows that start inside a 128-byte line cost the narrower tiles more.  2873 shapes timed both ways, of their time where taken, and
// where not (us, 128-wide pairs -> one wave: mm 9457x384x1280 13.7 -> 12.0; addmm 1147x1920x1408 + GELU 10.1 -> 11.6):
//   none                 578 taken, 0.893, nine of them slower by 2 %; 35 not, 1.01
//   ReLU or row factors  721, 0.916, 15; 226, 1.04
//   others               552, 0.916, 12; 761, 1.06
bool wider_tiles_pay(int64_t tiles, int64_t wave, int64_t k, int activation) {
  const int64_t k_blocks = ceil_div(k, 64), rest = tiles % wave;
  const bool lines = k % 64 == 0, many = rest * 10 > wave * 3;
  if (activation == AYLA_B200_ACT_NONE) return !lines || k_blocks >= 14 || many;
  if (activation == AYLA_B200_ACT_RELU) return k_blocks >= (lines && !many ? 18 : 15);
  return k_blocks >= (lines && rest * 2 <= wave ? 33 : 21);
}

// Whole tiles of the best other width or pairing that all run at once, for a schedule measured on another shape whose tiles
// fit this one badly; false where there is none 8 % faster by the model.  (us, the schedule -> this: 5539x384x4096 + GELU,
// 256-wide pairs in 1 + 14/74 waves -> 128-wide ones, 30.4 -> 19.9; 1240x2176x28672, 45 pairs of 256 columns -> 60 of 192, 157
// -> 137; 620x7232x1664, three rows of pairs -> five of single CTAs, 19.8 -> 16.8; 119x5312x832, clusters in two waves -> 64
// columns, 7.5 -> 5.7.)  Not for the shallowest (mm 1759x1344x640 7.0 -> 8.0).  No pairs in place of single CTAs of the same 256
// columns up to 23 k-blocks of whole lines (182 shapes 1.03 of the time, addmm 1722x2560x768 8.2 -> 8.5; 61 whose rows start inside
// a 128-byte line 0.93, none slower).
// Not in place of clusters whose rows start inside a sector (mm 200x3208x2456 13.1 -> 14.6), of one product's 64-wide ones whose rows
// start inside a line from 21 k-blocks on (seven shapes 0.90 to 1.06, whole lines and fewer 0.76 to 0.96: addmm 179x768x1296 +
// ReLU 6.6 -> 7.0), nor of 256-wide ones of single CTAs (addmm 282x5440x3776 21.3 -> 23.8).
bool one_wave(int64_t batch, int64_t m, int64_t n, int64_t k, int activation, const Machine& machine, ayla_b200_config* c) {
  const bool mid_sector = k % 16 != 0;
  if (m <= 64 || k <= 704) return false;
  if (c->cluster_split && (mid_sector || (c->tile_n == 256 && c->cta_group == 1))) return false;
  if (c->cluster_split && c->tile_n == 64 && batch == 1 && k % 64 != 0 && k > 20 * 64) return false;
  const int64_t wave = machine.sm_count / c->cta_group;
  const int64_t own_tiles = batch * ceil_div(m, 128 * c->cta_group) * ceil_div(n, c->tile_n);
  if (own_tiles > wave && (c->split_k > 1 || c->cluster_split || c->tile_n < 128)) return false;
  const bool no_wider = !mid_sector && c->tile_n == 128 && c->cta_group == 2 && own_tiles > wave &&
                        !wider_tiles_pay(own_tiles, wave, k, activation);
  const bool no_pairs = k % 64 == 0 && c->tile_n == 256 && c->cta_group == 1 && k <= 23 * 64;
  double best = 0.92 * scheduled_us(batch, m, n, k, machine, *c);
  ayla_b200_config chosen = *c;
  chosen.split_k = 1;
  chosen.split_tail = 0;
  chosen.cluster_split = 0;
  bool found = false;
  for (int tile_n = 64; tile_n <= 256; tile_n += 64) {
    for (int cta_group = 1; cta_group <= 2; ++cta_group) {
      if (cta_group == 2 && m <= 128) continue;
      const int64_t tiles = batch * ceil_div(m, 128 * cta_group) * ceil_div(n, tile_n);
      if (tiles > machine.sm_count / cta_group) continue;
      if ((no_wider && tile_n > 128) || (no_pairs && tile_n == 256 && cta_group == 2)) continue;
      const double us = modelled_us(tile_n, cta_group, 1, RATE_WHOLE, tiles, k, machine);
      if (us >= best) continue;
      best = us;
      found = true;
      chosen.tile_n = tile_n;
      chosen.cta_group = cta_group;
    }
  }
  if (found) *c = chosen;
  return found;
}

// What a schedule measured elsewhere, or here by bursts, is corrected in.
//
// Shallow products of 256-wide tiles become pairs where no rows are padded: they read B half as often, and under the
// power cap, which a burst does not reach, that is time (us per call, bmm 64 x 2048x2048x128 133.2 -> 122.7, 106 x
// 1872x1456x96 152.7 -> 142.1, 35 x 1219x1960x128 50.0 -> 45.4; of one k-block they do not gain: 55 x 2043x1208x64 80.1 ->
// 81.1).
//
// Splits the depth where a row-major schedule leaves SMs idle through a long product: the CTAs of a tile share its sum
// (see the kernel), so any number of them may work on it.  Two places:
//  * The last, partial wave of tiles, see last_wave: its tiles whole, as two halves each, or split S ways (us, whole -> half
//    -> split: 2744x2112x29248, 1 + 25/74 waves, 332 -> 316 -> 266 with 2; 4156x1088x3712, 1 + 11/74, 46 -> 40 -> 34 with 6;
//    4451x2240x7040, 2 + 14/74, 124 -> 112 -> 103 with 5; rows inside a sector: 1128x7488x7928, 2 + 2/74, 176 -> 175 ->
//    139 with 6; 3915x1088x5032, 1 + 6/74, 70 -> 70 -> 52 with 8).
//    Otherwise half width where two halves fit (1260x4480x768 12.0 -> 10.6, 1221x4160x1728 21.5 -> 18.8; nothing with rows
//    inside a sector), in shallow products where the rest is below three tenths of a wave: there the results that the SMs
//    write set the pace, not their number (bmm 71 x 324x128x272, 0.44 waves, 8.3 -> 8.8; mm 4546x1408x256, 0.46, 7.5 -> 7.8;
//    but 3266x1600x512, 0.23, 9.7 -> 8.6).  192 shapes timed with whole tiles and halves: 154 take them by this, the
//    geometric mean is 0.963 of the time, three are slower, by 4 to 5 %.  Where two do not fit, halves take two rounds:
//    whole instead (37 shapes, 0.74 to 1.0 of the time, all but three below 0.97: 1647x7520x1352, 2 + 62/74, 47 -> 37).
//  * A single wave with SMs to spare, or with clusters that do not all run at once.  By the model the shared sum has to
//    take 0.97 of the time for pairs and a deep product, 0.9 otherwise (536x896x59968 132 -> 67, 1064x192x38720 53 -> 29,
//    175x2304x8000 28.7 -> 16.2, 1896x320x8576 23.0 -> 18.0, 1024x1024x8192 23.8 -> 22.4; by less than that others lose:
//    128x4096x4096 12.1 -> 13.5, 433x1280x3584 with row factors 12.9 -> 13.7).  Not 0.97 where the pairs pad a row tile
//    that single CTAs did not (296x1088x14016 22.6 -> 24.2, 288x576x37248 36.8 -> 40.2), 0.85 for short products whose
//    rows start inside a sector (332x960x2568 11.8 -> 12.6), and never single CTAs for pairs there, which read B twice as
//    often (524x3200x13656 88 -> 99).  Over 191 shapes that are split by these bounds it takes 0.81 of the time, the slowest
//    1.02.
//
// `cautious`: ayla_b200_share_depth keeps the bounds that it has for last waves whose rows start inside a sector: two ways at
// most, behind one whole wave, behind two with a quarter of a wave left, or where the schedule has halves.  No op asks for that
// entry's answers; callers of the library may.
void share_depth(int64_t batch, int64_t m, int64_t n, int64_t k, const Machine& machine, bool cautious, ayla_b200_config* c) {
  if (c->swap_ab || c->stream_k || c->grid_ctas != 0 || c->split_tail == 1) return;
  if (c->split_k > 1 && !c->cluster_split && c->split_tail != 0) return;
  const int64_t k_blocks = ceil_div(k, 64);
  const bool mid_sector = k % 16 != 0;
  if (c->cta_group == 1 && c->split_k == 1 && c->tile_n == 256 && k_blocks >= 2 &&
      shallow_pairs_pay(batch, m, n, k, 256, AYLA_B200_ACT_RELU, machine.sm_count)) {
    c->cta_group = 2;
    c->split_tail = 0;
  }
  const int64_t wave = machine.sm_count / c->cta_group;
  int64_t tiles = batch * ceil_div(m, 128 * c->cta_group) * ceil_div(n, c->tile_n);
  if (tiles > wave) {
    if (c->split_k > 1 || c->cluster_split || tiles % wave == 0 || c->tile_n < 128) return;
    LastWave last = last_wave(tiles, wave, k, c->tile_n);
    if (cautious && mid_sector) {
      const int64_t rest = tiles % wave;
      const bool lone = tiles < 2 * wave || (tiles < 3 * wave && rest * 4 <= wave) || c->split_tail == 2;
      const double block = c->tile_n == 256 ? 0.38 : c->tile_n == 192 ? 0.33 : 0.275;
      if (lone && rest * 2 <= wave && k_blocks >= 32 && static_cast<double>(k_blocks) * 0.2 * block > 8.5) {
        c->split_k = 2;
        c->split_tail = 1;
      }
      return;
    }
    if (c->tile_n == 192 && c->cta_group == 2) {
      // 256-wide tiles may leave a thinner last wave, and a split one (2100x2368x7824 90 -> 67, 7328x640x5168 60 -> 50; by
      // less than 7 % of the model's time the 192-wide ones stay: 6690x1408x3200 0.99, 53 -> 56).
      const int64_t wider = batch * ceil_div(m, 256) * ceil_div(n, 256);
      const LastWave there = wider > wave ? last_wave(wider, wave, k, 256) : last;
      if (there.splits > 1 && there.us < 0.93 * last.us) {
        c->tile_n = 256;
        tiles = wider;
        last = there;
      }
    }
    const int64_t rest = tiles % wave;
    const bool halves_fit = c->tile_n % 128 == 0 && rest * 2 <= wave;
    if (last.splits > 1) {
      c->split_k = last.splits;
      c->split_tail = 1;
    } else if (!halves_fit) {
      c->split_tail = 0;
    } else if (!mid_sector && (k_blocks > 8 || rest * 10 <= wave * 3)) {
      c->split_tail = 2;
    }
    return;
  }
  if (m <= 64 || k_blocks < 16) return;
  const double now = modelled_us(c->tile_n, c->cta_group, c->split_k,
                                 c->cluster_split ? RATE_CLUSTER : c->split_k > 1 ? RATE_SHARED : RATE_WHOLE, tiles, k, machine);
  double best = now;
  ayla_b200_config chosen = *c;
  static const int kWidths[3] = {64, 128, 256};
  for (int tile_n : kWidths) {
    if (tile_n > 64 && n * 2 <= tile_n) continue;
    for (int cta_group = 1; cta_group <= 2; ++cta_group) {
      if ((cta_group == 2 && m <= 128) || (mid_sector && cta_group < c->cta_group)) continue;
      const int64_t there = batch * ceil_div(m, 128 * cta_group) * ceil_div(n, tile_n);
      int64_t most = machine.sm_count / cta_group / there;
      if (most > 48) most = 48;
      if (most > k_blocks / 4) most = k_blocks / 4;
      for (int64_t splits = most; splits >= 2; --splits) {
        const bool pads = cta_group > c->cta_group && ceil_div(m, 128) % 2 != 0;
        const double bound = cta_group == 2 && tile_n >= 128 && k_blocks >= 96 && !pads ? 0.97
                             : mid_sector && k_blocks < 48                               ? 0.85
                                                                                         : 0.9;
        const double us = modelled_us(tile_n, cta_group, static_cast<int>(splits), RATE_SHARED, there, k, machine);
        if (us >= best || us > bound * now) continue;
        best = us;
        chosen.tile_n = tile_n;
        chosen.cta_group = cta_group;
        chosen.split_k = static_cast<int>(splits);
        chosen.split_tail = 0;
        chosen.cluster_split = 0;
      }
    }
  }
  *c = chosen;
}

// Products of 33 to 128 rows on pairs (FORM_FLAT) instead, where by the models they take 0.95 of the schedule's time; all of
// their tiles at once.  Their times are a launch and the k-blocks, at rates fitted to 1340 timings of 730 shapes (6 % rms); rows
// that start inside a sector take 1.4 times as long.  The factors on the schedule's own model are what it lacks for 128 rows: a
// pair's rates do not change with the tile's height, and wide tiles read 128 rows per 128 or 256 columns.  us, before -> with
// it: mm 128x4096x4096 11.8 -> 10.4, 128x8192x2048 11.4 -> 9.5, addmm 100x3584x2560 9.3 -> 7.8, 128x1024x1024 6.1 -> 5.4.  Not
// where depth is short and tiles are narrow already.
// Of 33 to 64 rows only in place of a split depth: single CTAs on whole tiles load just the rows that exist (36x5632x1664 7.7 ->
// 8.3).  The swapped form's own model is fitted to 200 timings (4 to 6 % rms; eight-way clusters and narrower accumulators stay, pairs
// take 1.1 to 1.4 of their time).
// Besides, what the models miss, from 6700 shapes timed both ways, thin and batched ones and every measured schedule that
// changes among them: `amiss` is how much the log of the modelled ratio falls short, by terms of
//  * rows: single CTAs load the rows that exist, a pair's second CTA a box of 64 whatever is in it, the more so where rows start
//    inside a sector (clusters of four pairs for those of four 64-wide CTAs: of 33 to 64 rows 0.93 of the time and of more than 96
//    0.895, inside a sector 1.00 and 0.91);
//  * clusters nearly as many as run at once, mostly of padding in particular (bmm 33 x 72x72x1512 7.0 -> 7.9);
//  * depths split twelve ways and more (mm 65x32x15984 10.4 -> 11.6, 64x104x13320, inside a sector, 10.7 -> 14.1), inside a sector
//    eight ways (addmm 64x104x10520 10.4 -> 12.3), whole tiles of a batch (17 x 78x944x392 5.8 -> 6.5; but of one product they
//    gain more than modelled) and whole tiles for clusters;
//  * an activation (0.04 of the log, no more is known of it).
// No split depth in place of whole 64-wide tiles up to 16 k-blocks (mm 128x4096x1024 split in two 1.09 of the time, whole 0.85).
// By them 5724 of those shapes are taken, in 0.90 of the time, 103 slower by 2 %, at most 1.11; the others took 1.02, up to 1.31.  The
// swapped form needs none (430 shapes 0.87, one slower by 2 %).
bool flat_pairs(int64_t batch, int64_t m, int64_t n, int64_t k, int activation, const Machine& machine, ayla_b200_config* c) {
  const int64_t k_blocks = ceil_div(k, 64);
  if (m <= 32 || m > 128 || c->stream_k || c->grid_ctas != 0) return false;
  if (m <= 64 ? c->split_k == 1 || k_blocks < 16 : c->swap_ab || k_blocks < (c->tile_n == 64 ? 12 : 7)) return false;
  const bool mid_sector = k % 16 != 0;
  const int64_t own_tiles = batch * ceil_div(n, c->swap_ab ? (c->tile_rows > 0 ? c->tile_rows : 128) : c->tile_n);
  if (c->split_tail != 0 && own_tiles > machine.sm_count) return false;
  double own;
  if (c->swap_ab) {
    if (c->tile_n != 64 || !c->cluster_split || c->split_k > 4) return false;
    const bool two = c->split_k == 2;
    const int64_t ctas = own_tiles * c->split_k, waves = ceil_div(ctas, machine.sm_count);
    const double busy = static_cast<double>(ctas * (c->tile_rows > 0 ? c->tile_rows : 128)) /
                        static_cast<double>(128 * waves * machine.sm_count);
    own = (two ? 5.70 : 5.23) + static_cast<double>(waves * ceil_div(k_blocks, c->split_k)) *
                                    (mid_sector ? (two ? 1.25 : 1.18) : 1.0) * (two ? .136 + .191 * busy : .149 + .172 * busy);
  } else {
    own = modelled_us(c->tile_n, c->cta_group, c->split_k,
                      c->cluster_split ? RATE_CLUSTER : c->split_k > 1 ? RATE_SHARED : RATE_WHOLE, own_tiles, k, machine);
    if (c->split_k == 1) {
      own *= c->tile_n != 128 || c->cta_group != 1 ? 1.0 : mid_sector ? 1.25 : k_blocks < 20 ? 1.05 : 1.2;
    } else if (c->tile_n == 256) {
      own *= mid_sector ? 1.06 : 1.24;
    } else if (c->tile_n == 64) {
      own *= 1.05;
    } else if (c->tile_n == 128) {
      own *= c->cluster_split ? (c->split_k == 2 ? 1.02 : 1.0) : mid_sector ? 1.0 : 1.05;
    }
  }
  struct Flat { int tile_n, split; double launch, block, block_busy; };
  static const Flat kFlat[5] = {{128, 1, 4.17, .099, .077}, {128, 2, 4.85, .105, .082}, {128, 4, 5.69, .095, .091},
                                {256, 1, 4.44, .126, .227}, {256, 2, 5.08, .163, .247}};
  const int64_t pairs = machine.sm_count / 2;
  double best = 0.95 * own;
  const Flat* chosen = nullptr;
  for (const Flat& f : kFlat) {
    const int64_t tiles = batch * ceil_div(n, f.tile_n);
    if (tiles > machine.clusters(2 * f.split) || (f.split > 1 && k_blocks < 4 * f.split)) continue;
    if (f.split > 1 && c->split_k == 1 && c->tile_n == 64 && k_blocks <= 16 && !mid_sector) continue;
    const double busy = static_cast<double>(tiles * f.split) / static_cast<double>(pairs);
    const double us = f.launch + static_cast<double>(ceil_div(k_blocks, f.split)) * (mid_sector ? 1.4 : 1.0) *
                                     (f.block + f.block_busy * busy);
    if (us >= best) continue;
    best = us;
    chosen = &f;
  }
  if (chosen == nullptr) return false;
  if (!c->swap_ab) {
    const int64_t tiles = batch * ceil_div(n, chosen->tile_n);
    const bool shared = c->split_k > 1 && !c->cluster_split;
    double amiss = (mid_sector ? 0.40 : 0.17) * static_cast<double>(128 - m) / 128.0;
    if ((chosen->split == 2 && tiles * 3 > machine.clusters4 * 2) || (chosen->split == 4 && tiles * 2 > machine.clusters8)) {
      amiss += (mid_sector ? 0.085 : 0.05) + (n * 8 <= chosen->tile_n * 5 ? 0.1 : 0.0);
    }
    if (shared && c->split_k >= 12) amiss += mid_sector ? 0.31 : k_blocks > 213 ? 0.17 : 0.12;
    if (mid_sector && shared && c->tile_n == 64 && c->split_k >= 8 && c->split_k < 12) amiss += 0.085;
    if (mid_sector && c->tile_n == 128 && c->split_k == 1) amiss += batch > 1 ? 0.17 : -0.16;
    if (mid_sector && c->tile_n == 64 && c->cluster_split && c->split_k == 2 && chosen->split == 1) amiss += 0.12;
    if (activation != AYLA_B200_ACT_NONE) amiss += 0.04;
    if (best * std::exp(amiss) >= 1.1 * own) return false;
  }
  c->tile_n = chosen->tile_n;
  c->cta_group = 2;
  c->swap_ab = 0;
  c->tile_rows = 0;
  c->split_k = chosen->split;
  c->cluster_split = chosen->split > 1 ? 1 : 0;
  c->split_tail = 0;
  c->group_m = 8;
  // Of 730 schedules faster than before: 1.009 of the best pair of hints with these, 1.013 with none; 1.019 without a prefetch.
  c->l2_hint_a = 2;
  c->l2_hint_b = 1;
  const int64_t share = k_blocks / chosen->split / 2;
  c->early_prefetch = static_cast<int>(share < 8 ? share : 8);
  return true;
}

// A schedule that was measured elsewhere, or here without what this knows: with its depth shared out, or with tiles that fit
// the shape in one wave, and their depth shared out, where that takes 0.92 of the time by the models; or on flat pairs.  Beside
// 128-wide pairs whose last wave is split, whole wider ones count with the k-blocks of a last wave's model: their operands outgrow
// L2, and by the rate of a single wave mm 2200x1216x35136 took them, 174 -> 191, and 1304x1808x33888, 179 -> 204 (of eleven such
// shapes the four still taken 0.75 to 0.94, the others 0.97 to 1.13; of 63 that are 64 to 100 k-blocks deep, none of them taken,
// 1.03).  An activation of RELU stands for row factors too.  Of 12000 shapes drawn over all kinds when these rules stood, 3300 change; 883
// of them timed take 0.914 of the time, 13 are slower by 2 %, at most 1.06.
void fit_depth(int64_t batch, int64_t m, int64_t n, int64_t k, int activation, const Machine& machine, ayla_b200_config* c) {
  ayla_b200_config fitted = *c;
  share_depth(batch, m, n, k, machine, false, c);
  if (!fitted.swap_ab && !fitted.stream_k && fitted.grid_ctas == 0 && one_wave(batch, m, n, k, activation, machine, &fitted)) {
    share_depth(batch, m, n, k, machine, false, &fitted);
    double us = scheduled_us(batch, m, n, k, machine, fitted);
    if (c->tile_n == 128 && c->split_tail == 1 && fitted.tile_n > 128 && fitted.split_k == 1) {
      const double deep = 4.3 + static_cast<double>(ceil_div(k, 64)) * block_us(fitted.tile_n) * (k % 16 != 0 ? 1.2 : 1.0);
      if (us < deep) us = deep;
    }
    if (us < 0.92 * scheduled_us(batch, m, n, k, machine, *c)) *c = fitted;
  }
  flat_pairs(batch, m, n, k, activation, machine, c);
}

// The swapped SwiGLU schedule for a product that does not fill the SMs with 128-column row-major tiles (which
// leave 32 of them working at n = 4096): 64 output columns per tile, M on the narrow accumulator, k split across
// a cluster, all in one wave.  False where no such schedule exists; where one does it measured the faster in 168
// shapes (us, row-major -> swapped: 8x1024x4096 25.0 -> 6.5, 8x4096x4096 26.7 -> 13.0, 64x8192x4096 30.4 -> 24.3,
// 128x4096x4096 27.9 -> 17.9, 512x1024x4096 23.5 -> 15.6, 1024x1024x4096 24.1 -> 21.9; in more than one wave it
// loses: 64x14336x4096 41.7 -> 42.6, 769x1472x3008 20.0 -> 29.4).  A 128-wide accumulator that no cluster shares is
// written out by its one CTA in 4 us and more, two bytes at a time, which only a deep product earns back.  Against
// pairs (256 rows and more): 740x1504x896, 14 k-blocks, 9.3 -> 10.4, 595x1024x2112, 33, 15.6 -> 17.6, but
// 659x896x2432, 38, 16.0 -> 15.2, 374x2944x3200, 50, 21.9 -> 20.7; against single CTAs: 109x6080x960, 15, 10.5 ->
// 11.4, but 150x3304x1664, 26, 14.0 -> 12.8; with rows that start inside a 32-byte sector 381x3136x3208, 51,
// 25.1 -> 29.2, but 68x5232x11720, 184, 92.4 -> 72.8.
bool swapped_swiglu_config(int64_t m, int64_t n, int64_t k, const Machine& machine, ayla_b200_config* c) {
  // us per k-block and per cluster exchange, fitted to the same measurements.
  struct Width { int tile_n; double per_kb, exchange2, exchange4; };
  static const Width kWidths[4] = {{16, 0.160, 0.9, 1.4}, {32, 0.170, 0.9, 1.4}, {64, 0.20, 1.5, 3.0}, {128, 0.28, 2.7, 4.6}};
  const int64_t k_blocks = ceil_div(k, 64), row_tiles = ceil_div(n, 64);
  double best = 1e300;
  memset(c, 0, sizeof(*c));
  for (const Width& w : kWidths) {
    const int64_t tiles = row_tiles * ceil_div(m, w.tile_n);
    for (int split = 1; split <= 4; split *= 2) {
      if (tiles > machine.clusters(split) || (split > 1 && k_blocks < 4 * split)) break;
      if (w.tile_n == 128 && split == 1 && k_blocks < (k % 16 != 0 ? 60 : m < 256 ? 20 : 36)) continue;
      const double cost = static_cast<double>(ceil_div(k_blocks, split)) * w.per_kb +
                          (split == 1 ? 0.0 : split == 2 ? w.exchange2 : w.exchange4);
      if (cost < best && static_cast<int64_t>(split - 1) * ceil_div(k_blocks, split) < k_blocks) {
        best = cost;
        c->tile_n = w.tile_n;
        c->split_k = split;
      }
    }
  }
  if (best == 1e300) return false;
  c->swap_ab = 1;
  c->cta_group = 1;
  c->group_m = 1;
  c->tile_rows = 64;
  c->cluster_split = c->split_k > 1 ? 1 : 0;
  c->l2_hint_a = 2;
  c->l2_hint_b = 1;
  // The weights' first blocks are asked into L2 under the preceding launch's tail (8x4096x4096 13.6 -> 13.0).
  const int64_t share = k_blocks / c->split_k / 2;
  c->early_prefetch = m > 64 ? 0 : static_cast<int>(share < 8 ? share : 8);
  return true;
}

ayla_b200_config row_major_swiglu_config(int64_t m) {
  ayla_b200_config c;
  memset(&c, 0, sizeof(c));
  c.tile_n = 256;
  c.cta_group = (m >= 256) ? 2 : 1;
  c.split_k = 1;
  c.group_m = 8;
  c.l2_hint_a = 2;  // x is re-read by every column tile,
  c.l2_hint_b = 1;  // the weights stream through once
  return c;
}

int launch_plan(const Plan& plan, const ayla_b200_config& c, const Problem& pr, int is_bf16,
                const void* bias, const void* b2_operand, void* out, int64_t out_rows,
                int64_t out_cols, void* workspace, size_t workspace_bytes, uint32_t* status,
                cudaStream_t stream, int activation = 0, const void* mul = nullptr, int mul_per_row = 0) {
  const KernelEntry& e = *plan.kernel;
  LaunchArgs la;
  memset(&la, 0, sizeof(la));
  const bool swiglu_cols = e.epilogue == EPI_SWIGLU && !e.transposed_out;
  const bool swiglu_rows = e.epilogue == EPI_SWIGLU && e.transposed_out;
  int b_box_rows = swiglu_cols ? 128 : e.tile_n / e.cta_group;
  int b_stage_rows = e.tile_n / e.cta_group;  // rows of the column operand one CTA receives per stage
  int a_box_rows = e.cta_rows < plan.tile_rows ? e.cta_rows : plan.tile_rows;
  // An operand that fits in a single tile is loaded with a box of just its own rows (rounded
  // up to the 8-row swizzle atom): rows of the box that lie outside the tensor are zero-filled
  // by TMA at a cost comparable to real rows, and a GEMM with a handful of rows would spend
  // most of its load time on them.  The shared-memory rows the smaller box leaves untouched
  // feed only accumulator rows / columns that are never stored.
  if (e.cta_group == 1) {
    const int rows8 = static_cast<int>(ceil_div(pr.rows, 8) * 8);
    const int cols8 = static_cast<int>(ceil_div(pr.cols, 8) * 8);
    if (plan.m_tiles == 1 && rows8 < a_box_rows) a_box_rows = rows8;
    if (plan.n_tiles == 1 && !swiglu_cols && plan.narrow_from_tile == 0x7FFFFFFF && cols8 < b_box_rows) {
      b_box_rows = cols8;
      b_stage_rows = cols8;
    }
  }
  int rc = encode_map(&la.tm_a, pr.row_operand, pr.k, pr.rows, pr.batch, 64, a_box_rows, 1);
  if (rc) return rc;
  rc = encode_map(&la.tm_b, pr.col_operand, pr.k, pr.cols, pr.batch, 64, b_box_rows, 1);
  if (rc) return rc;
  if (e.epilogue == EPI_SWIGLU) {
    rc = swiglu_rows ? encode_map(&la.tm_b2, b2_operand, pr.k, pr.rows, pr.batch, 64, a_box_rows, 1)
                     : encode_map(&la.tm_b2, b2_operand, pr.k, pr.cols, pr.batch, 64, b_box_rows, 1);
    if (rc) return rc;
  } else if (e.activation == 2) {
    rc = encode_map(&la.tm_b2, mul, out_cols, out_rows, pr.batch, 64, 32, 1);
    if (rc) return rc;
  } else {
    la.tm_b2 = la.tm_b;
  }
  if (!e.transposed_out) {
    rc = encode_map(&la.tm_d, out, out_cols, out_rows, pr.batch, 64, 32, 1);
    if (rc) return rc;
  } else {
    la.tm_d = la.tm_a;
  }

  KernelParams& p = la.p;
  p.m = static_cast<int>(pr.rows);
  p.n = static_cast<int>(pr.cols);
  p.k = static_cast<int>(pr.k);
  p.batch = static_cast<int>(pr.batch);
  p.m_tiles = plan.m_tiles;
  p.n_tiles = plan.n_tiles;
  p.k_blocks = plan.k_blocks;
  p.splits = plan.splits;
  p.kb_per_split = plan.kb_per_split;
  p.split_from_tile = plan.split_from_tile;
  p.narrow_from_tile = plan.narrow_from_tile;
  p.cluster_split = plan.cluster_split;
  p.stream_k = plan.stream_k;
  p.kb_per_cta = plan.kb_per_cta;
  p.idesc_narrow = make_idesc(is_bf16, e.cta_rows * e.cta_group, e.tile_n / 2);
  p.total_units = plan.total_units;
  p.group_m = plan.group_m;
  p.is_bf16 = is_bf16;
  p.idesc = make_idesc(is_bf16, e.cta_rows * e.cta_group, e.tile_n);
  // Hints are given for a/bt as the caller passed them.
  p.l2_hint_a = static_cast<uint32_t>(c.swap_ab ? c.l2_hint_b : c.l2_hint_a);
  p.l2_hint_b = static_cast<uint32_t>(c.swap_ab ? c.l2_hint_a : c.l2_hint_b);
  p.bias = bias;
  p.out = out;
  p.out_ld = out_cols;               // direct stores: out[batch][col][row], row-major [M][N]
  p.out_batch_stride = out_rows * out_cols;
  p.status = status;
  p.timeout_ns = static_cast<unsigned long long>(g_timeout_ns.load());
  p.debug_flags = g_debug_flags.load();
  p.l2_prefetch = c.l2_prefetch;
  p.early_prefetch = c.early_prefetch;
  // The early prefetch covers the operand that carries the bytes (a weight against a few rows of
  // activations); both when they are within a factor of four of each other.
  p.early_operands = (pr.rows * 4 >= pr.cols ? 1 : 0) | (pr.cols * 4 >= pr.rows ? 2 : 0);
  p.div_tiles_per_batch = FastDiv::make(static_cast<uint32_t>(plan.m_tiles) * static_cast<uint32_t>(plan.n_tiles));
  p.div_group_size = FastDiv::make(static_cast<uint32_t>(plan.group_m) * static_cast<uint32_t>(plan.n_tiles));
  p.div_group_m = FastDiv::make(static_cast<uint32_t>(plan.group_m));
  p.div_last_group_rows = FastDiv::make(static_cast<uint32_t>(plan.m_tiles % plan.group_m));
  p.div_splits = FastDiv::make(static_cast<uint32_t>(plan.splits));
  {
    int per_unit = e.cta_group * (plan.cluster_split > 0 ? plan.cluster_split : 1), log2 = 0;
    while ((1 << log2) < per_unit) ++log2;
    p.ctas_per_unit_log2 = log2;
  }
  p.stages = e.stages;
  if (plan.cluster_split > 0) {
    // Cluster split-K: every CTA receives the other k-splits' partials of the columns it owns in an
    // inbox of shared memory.  The inbox takes the top of the ring region; the ring gives up the
    // slots it covers as long as three remain, otherwise the inbox overlays live slots and the
    // kernel holds the partials back until the whole cluster is done with its MMAs.
    const int csk = plan.cluster_split;
    const int slice_cols = e.acc_cols / csk;
    const int chunk_cols = e.acc_cols < 32 ? e.acc_cols : 32;
    const int slots = (slice_cols >= chunk_cols) ? csk - 1 : csk;
    const int inbox_bytes = slots * 128 * slice_cols * 4;
    const int stage_bytes = e.kb_per_slot * (e.cta_rows * 64 * 2 + (e.tile_n / e.cta_group) * 64 * 2);  // one ring slot
    const int ring_bytes = e.stages * stage_bytes;
    if (inbox_bytes > ring_bytes) {
      return fail(AYLA_B200_E_UNSUPPORTED, "cluster_split: the %d-byte inbox does not fit the %d-byte ring", inbox_bytes,
                  ring_bytes);
    }
    const int free_stages = (ring_bytes - inbox_bytes) / stage_bytes;
    p.inbox_tx = static_cast<uint32_t>(inbox_bytes);
    p.inbox_offset = static_cast<uint32_t>(ring_bytes - inbox_bytes);
    if (free_stages >= 3 && (g_debug_flags.load() & 2) == 0) {
      p.stages = free_stages;
      p.inbox_in_ring = 0;
    } else {
      p.inbox_in_ring = 1;
    }
  }
  p.handover_ns = (g_debug_flags.load() & 32) != 0 ? 0u : kHandoverNs;
  p.tile_rows = plan.tile_rows;
  p.act = activation;
  p.mul = mul;
  p.mul_per_row = mul_per_row;
  // One stage receives this CTA's rows of the row operand and its share of the column
  // operand; the leader of a pair counts both CTAs' bytes.
  p.stage_tx = static_cast<uint32_t>((a_box_rows * (swiglu_rows ? 2 : 1) + b_stage_rows) * 128 * e.cta_group);
  if (plan.slabs > 0) {
    const size_t need = workspace_bytes_for(plan);
    if (workspace == nullptr || workspace_bytes < need) {
      return fail(AYLA_B200_E_WORKSPACE, "this schedule (split_k=%d, stream_k=%d) needs a workspace of %zu bytes, got %zu",
                  plan.splits, plan.stream_k, need, workspace == nullptr ? size_t(0) : workspace_bytes);
    }
    if (!aligned16(workspace)) {
      return fail(AYLA_B200_E_INVALID, "workspace must be 16-byte aligned");
    }
    p.counters = reinterpret_cast<unsigned*>(workspace);
    p.ws = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(workspace) + counter_bytes_for(plan));
  }
#ifdef AYLA_B200_TRACE
  // Tuning builds: a schedule that needs no scratch lends the workspace to the per-CTA cycle counters.
  if (plan.slabs == 0 && workspace != nullptr && workspace_bytes >= (4096 + static_cast<size_t>(plan.grid) * 64) * 8) {
    p.trace = reinterpret_cast<long long*>(workspace);
  }
#endif
  la.grid = plan.grid;
  la.cluster_x = plan.cluster_split * e.cta_group;
  la.overlap = g_launch_overlap.load();
  la.stream = stream;
  const cudaError_t err = e.launch(la);
  if (err != cudaSuccess) {
    return fail(AYLA_B200_E_CUDA, "kernel launch failed: %s", cudaGetErrorString(err));
  }
  return AYLA_B200_OK;
}

// ----------------------------------------------------- built-in split-K scratch
//
// Scratch for ayla_b200_gemm_static_scratch: a fixed array in device memory that is
// part of the loaded library image on every GPU, so that entry point never has to
// ask anyone for memory.  In host code `g_static_scratch` is only a handle for
// the runtime (not a device address); the address a kernel can use comes from
// cudaGetSymbolAddress, looked up once per device with that device current.
static __device__ __align__(256) unsigned char g_static_scratch[AYLA_B200_STATIC_SCRATCH_BYTES];

std::mutex g_scratch_mutex;
void* g_scratch_ptr[kMaxDevices] = {};

int static_scratch_for_current_device(int device, void** out) {
  std::lock_guard<std::mutex> lock(g_scratch_mutex);
  if (g_scratch_ptr[device] == nullptr) {
    void* ptr = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&ptr, g_static_scratch);
    if (err != cudaSuccess || ptr == nullptr) {
      return fail(AYLA_B200_E_CUDA, "cudaGetSymbolAddress(static scratch) on device %d: %s", device,
                  cudaGetErrorString(err));
    }
    g_scratch_ptr[device] = ptr;
  }
  *out = g_scratch_ptr[device];
  return AYLA_B200_OK;
}

}  // namespace
}  // namespace ayla_b200

using namespace ayla_b200;

extern "C" {

int ayla_b200_init(int device) {
  if (device < 0 || device >= kMaxDevices) {
    return fail(AYLA_B200_E_INVALID, "device %d out of range", device);
  }
  std::lock_guard<std::mutex> lock(g_init_mutex);
  if (g_devices[device].ready.load(std::memory_order_acquire)) return AYLA_B200_OK;
  int prev = -1;
  cudaError_t err = cudaGetDevice(&prev);
  if (err != cudaSuccess) return fail(AYLA_B200_E_CUDA, "cudaGetDevice: %s", cudaGetErrorString(err));
  err = cudaSetDevice(device);
  if (err != cudaSuccess) return fail(AYLA_B200_E_CUDA, "cudaSetDevice: %s", cudaGetErrorString(err));
  int rc = AYLA_B200_OK;
  do {
    cudaDeviceProp prop;
    err = cudaGetDeviceProperties(&prop, device);
    if (err != cudaSuccess) {
      rc = fail(AYLA_B200_E_CUDA, "cudaGetDeviceProperties: %s", cudaGetErrorString(err));
      break;
    }
    if (prop.major != 10) {
      rc = fail(AYLA_B200_E_UNSUPPORTED, "device %d is sm_%d%d; this library is sm_100a only", device,
                prop.major, prop.minor);
      break;
    }
    if (g_encode_tiled == nullptr) {
      void* fn = nullptr;
      cudaDriverEntryPointQueryResult qres;
      err = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres);
      if (err != cudaSuccess || fn == nullptr || qres != cudaDriverEntryPointSuccess) {
        rc = fail(AYLA_B200_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
        break;
      }
      g_encode_tiled = reinterpret_cast<PFN_cuTensorMapEncodeTiled>(fn);
    }
    const Registry& reg = registry();
    for (size_t i = 0; i < reg.entries.size(); ++i) {
      const KernelEntry& e = reg.entries[i];
      err = cudaFuncSetAttribute(e.func, cudaFuncAttributeMaxDynamicSharedMemorySize, e.smem_bytes);
      if (err != cudaSuccess) {
        rc = fail(AYLA_B200_E_CUDA, "cudaFuncSetAttribute(smem=%d) for variant %zu: %s", e.smem_bytes, i,
                  cudaGetErrorString(err));
        break;
      }
    }
    if (rc) break;
    err = init_packed_gemm();
    if (err != cudaSuccess) {
      rc = fail(AYLA_B200_E_CUDA, "cudaFuncSetAttribute for the packed kernel: %s", cudaGetErrorString(err));
      break;
    }
    {
      // Resolve the built-in scratch array here as well, with `device` current: the query loads the
      // library's device image if nothing has yet, which is better done at set-up than inside the
      // first ayla_b200_gemm_static_scratch call.
      void* scratch = nullptr;
      rc = static_scratch_for_current_device(device, &scratch);
      if (rc) break;
    }
    g_devices[device].sm_count = prop.multiProcessorCount;
    Machine& machine = g_devices[device].machine;
    machine.sm_count = prop.multiProcessorCount;
    const KernelEntry* clustered = registry().find(128, 1, EPI_PLAIN, 0);
    for (int ctas = 4; ctas <= 8; ctas *= 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(static_cast<unsigned>(machine.sm_count / ctas * ctas));
      cfg.blockDim = dim3(static_cast<unsigned>(clustered->threads));
      cfg.dynamicSmemBytes = static_cast<size_t>(clustered->smem_bytes);
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = static_cast<unsigned>(ctas);
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      int at_once = 0;
      if (cudaOccupancyMaxActiveClusters(&at_once, clustered->func, &cfg) != cudaSuccess || at_once < 1) {
        (void)cudaGetLastError();
        continue;  // what a B200 holds stays
      }
      (ctas == 4 ? machine.clusters4 : machine.clusters8) = at_once;
    }
    g_devices[device].ready.store(true, std::memory_order_release);
  } while (false);
  if (prev >= 0 && prev != device) cudaSetDevice(prev);
  return rc;
}

int ayla_b200_default_config(int op, int dtype, int64_t batch, int64_t m, int64_t n, int64_t k,
                             ayla_b200_config* cfg_out) {
  return ayla_b200_default_config_act(op, dtype, AYLA_B200_ACT_NONE, batch, m, n, k, cfg_out);
}

int ayla_b200_default_config_act(int op, int dtype, int activation, int64_t batch, int64_t m, int64_t n, int64_t k,
                                 ayla_b200_config* cfg_out) {
  if (cfg_out == nullptr) return fail(AYLA_B200_E_INVALID, "cfg_out is null");
  const int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  if (activation < AYLA_B200_ACT_NONE || activation > AYLA_B200_ACT_GELU_TANH) {
    return fail(AYLA_B200_E_INVALID, "unknown activation %d", activation);
  }
  default_config(batch, m, n, k, activation, current_machine(), cfg_out);
  return AYLA_B200_OK;
}

int ayla_b200_share_depth(int op, int dtype, int64_t batch, int64_t m, int64_t n, int64_t k, ayla_b200_config* cfg) {
  if (cfg == nullptr) return fail(AYLA_B200_E_INVALID, "cfg is null");
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  rc = check_config(*cfg, false);
  if (rc) return rc;
  share_depth(batch, m, n, k, current_machine(), true, cfg);
  return AYLA_B200_OK;
}

int ayla_b200_fit_depth(int op, int dtype, int64_t batch, int64_t m, int64_t n, int64_t k, ayla_b200_config* cfg) {
  return ayla_b200_fit_depth_act(op, dtype, AYLA_B200_ACT_NONE, batch, m, n, k, cfg);
}

int ayla_b200_fit_depth_act(int op, int dtype, int activation, int64_t batch, int64_t m, int64_t n, int64_t k,
                            ayla_b200_config* cfg) {
  if (cfg == nullptr) return fail(AYLA_B200_E_INVALID, "cfg is null");
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  if (activation < AYLA_B200_ACT_NONE || activation > AYLA_B200_ACT_GELU_TANH) {
    return fail(AYLA_B200_E_INVALID, "unknown activation %d", activation);
  }
  rc = check_config(*cfg, false);
  if (rc) return rc;
  fit_depth(batch, m, n, k, activation, current_machine(), cfg);
  return AYLA_B200_OK;
}

int ayla_b200_swiglu_default_config(int dtype, int64_t m, int64_t n, int64_t k, ayla_b200_config* cfg_out) {
  if (cfg_out == nullptr) return fail(AYLA_B200_E_INVALID, "cfg_out is null");
  const int rc = check_shape(AYLA_B200_OP_MM, dtype, 1, m, n, k);
  if (rc) return rc;
  if (!swapped_swiglu_config(m, n, k, current_machine(), cfg_out)) *cfg_out = row_major_swiglu_config(m);
  return AYLA_B200_OK;
}

int ayla_b200_config_valid(const ayla_b200_config* cfg, int op, int dtype, int64_t batch, int64_t m,
                           int64_t n, int64_t k) {
  if (cfg == nullptr) return fail(AYLA_B200_E_INVALID, "cfg is null");
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  rc = check_config(*cfg, false);
  if (rc) return rc;
  Plan plan{};
  const int epi = (op == AYLA_B200_OP_ADDMM) ? EPI_BIAS : EPI_PLAIN;
  return make_plan(*cfg, epi, batch, cfg->swap_ab ? n : m, cfg->swap_ab ? m : n, k, 148, &plan);
}

size_t ayla_b200_workspace_bytes(const ayla_b200_config* cfg, int op, int64_t batch, int64_t m,
                                 int64_t n, int64_t k) {
  if (cfg == nullptr || check_config(*cfg, false) != AYLA_B200_OK) return 0;
  if (batch <= 0 || m <= 0 || n <= 0 || k <= 0) return 0;
  Plan plan{};
  const int epi = (op == AYLA_B200_OP_ADDMM) ? EPI_BIAS : EPI_PLAIN;
  if (make_plan(*cfg, epi, batch, cfg->swap_ab ? n : m, cfg->swap_ab ? m : n, k, 148, &plan)) return 0;
  return workspace_bytes_for(plan);
}

size_t ayla_b200_workspace_counter_bytes(const ayla_b200_config* cfg, int op, int64_t batch,
                                         int64_t m, int64_t n, int64_t k) {
  if (cfg == nullptr || check_config(*cfg, false) != AYLA_B200_OK) return 0;
  if (batch <= 0 || m <= 0 || n <= 0 || k <= 0) return 0;
  Plan plan{};
  const int epi = (op == AYLA_B200_OP_ADDMM) ? EPI_BIAS : EPI_PLAIN;
  if (make_plan(*cfg, epi, batch, cfg->swap_ab ? n : m, cfg->swap_ab ? m : n, k, 148, &plan)) return 0;
  return counter_bytes_for(plan);
}

int ayla_b200_capture_workspace(void* stream, size_t bytes, void** workspace) {
  if (workspace == nullptr || bytes < kCounterBytes) {
    return fail(AYLA_B200_E_INVALID, "a workspace has at least its %zu bytes of counters", kCounterBytes);
  }
  const cudaError_t err =
      capture_workspace(reinterpret_cast<cudaStream_t>(stream), bytes, kCounterBytes, workspace);
  if (err != cudaSuccess) {
    (void)cudaGetLastError();
    return fail(AYLA_B200_E_CUDA, "a workspace for the graph being captured: %s", cudaGetErrorString(err));
  }
  return AYLA_B200_OK;
}

int ayla_b200_gemm(int op, int dtype, const void* bias, const void* a, const void* bt, void* out,
                   int64_t batch, int64_t m, int64_t n, int64_t k, const ayla_b200_config* cfg,
                   void* workspace, size_t workspace_bytes, uint32_t* status, void* stream) {
  return ayla_b200_gemm_act(op, dtype, AYLA_B200_ACT_NONE, bias, a, bt, out, batch, m, n, k, cfg, workspace,
                            workspace_bytes, status, stream);
}

int ayla_b200_gemm_act(int op, int dtype, int activation, const void* bias, const void* a, const void* bt,
                       void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                       const ayla_b200_config* cfg, void* workspace, size_t workspace_bytes,
                       uint32_t* status, void* stream) {
  return ayla_b200_gemm_act_mul(op, dtype, activation, bias, a, bt, nullptr, out, batch, m, n, k, cfg, workspace,
                                workspace_bytes, status, stream);
}

static int gemm_fused(int op, int dtype, int activation, const void* bias, const void* a, const void* bt,
                      const void* mul, int mul_per_row, void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                      const ayla_b200_config* cfg, void* workspace, size_t workspace_bytes, uint32_t* status,
                      void* stream);

int ayla_b200_gemm_act_mul(int op, int dtype, int activation, const void* bias, const void* a, const void* bt,
                           const void* mul, void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                           const ayla_b200_config* cfg, void* workspace, size_t workspace_bytes,
                           uint32_t* status, void* stream) {
  if (mul != nullptr && !aligned16(mul)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "mul must be 16-byte aligned");
  }
  return gemm_fused(op, dtype, activation, bias, a, bt, mul, 0, out, batch, m, n, k, cfg, workspace,
                    workspace_bytes, status, stream);
}

int ayla_b200_gemm_act_rowmul(int op, int dtype, int activation, const void* bias, const void* a, const void* bt,
                              const void* row_mul, void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                              const ayla_b200_config* cfg, void* workspace, size_t workspace_bytes,
                              uint32_t* status, void* stream) {
  if (row_mul == nullptr || (reinterpret_cast<uintptr_t>(row_mul) & 1) != 0) {
    return fail(AYLA_B200_E_INVALID, "row_mul must be a non-null, 2-byte aligned pointer");
  }
  return gemm_fused(op, dtype, activation, bias, a, bt, row_mul, 1, out, batch, m, n, k, cfg, workspace,
                    workspace_bytes, status, stream);
}

static int gemm_fused(int op, int dtype, int activation, const void* bias, const void* a, const void* bt,
                      const void* mul, int mul_per_row, void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                      const ayla_b200_config* cfg, void* workspace, size_t workspace_bytes, uint32_t* status,
                      void* stream) {
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  if (activation < AYLA_B200_ACT_NONE || activation > AYLA_B200_ACT_GELU_TANH) {
    return fail(AYLA_B200_E_INVALID, "unknown activation %d", activation);
  }
  if (a == nullptr || bt == nullptr || out == nullptr) {
    return fail(AYLA_B200_E_INVALID, "a, bt and out must be non-null");
  }
  if (op == AYLA_B200_OP_ADDMM && bias == nullptr) {
    return fail(AYLA_B200_E_INVALID, "addmm needs a bias pointer");
  }
  if (!aligned16(a) || !aligned16(bt) || !aligned16(out)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "a, bt and out must be 16-byte aligned");
  }
  DeviceState* ds = nullptr;
  int dev = -1;
  rc = current_device_state(&ds, &dev);
  if (rc) return rc;

  ayla_b200_config c;
  if (cfg != nullptr) {
    c = *cfg;
  } else if (activation == AYLA_B200_ACT_NONE && mul == nullptr &&
             packed_preferred(batch, m, n, k, ds->sm_count, on_sectors(out))) {
    return ayla_b200_gemm_packed(op, dtype, bias, a, bt, out, batch, m, n, k, status, stream);
  } else {
    default_config(batch, m, n, k, activation, ds->machine, &c);
  }
  rc = check_config(c, false);
  if (rc) return rc;

  Problem pr;
  pr.k = k;
  pr.batch = batch;
  if (c.swap_ab) {
    pr.rows = n;
    pr.cols = m;
    pr.row_operand = bt;
    pr.col_operand = a;
  } else {
    pr.rows = m;
    pr.cols = n;
    pr.row_operand = a;
    pr.col_operand = bt;
  }
  const int epi = (op == AYLA_B200_OP_ADDMM) ? EPI_BIAS : EPI_PLAIN;
  Plan plan{};
  rc = make_plan(c, epi, batch, pr.rows, pr.cols, k, ds->sm_count, &plan,
                 (mul != nullptr && mul_per_row == 0)  ? 2
                 : activation > AYLA_B200_ACT_RELU       ? 3
                 : activation != 0 || mul != nullptr     ? 1
                                                         : 0);
  if (rc) return rc;
  return launch_plan(plan, c, pr, dtype == AYLA_B200_BF16 ? 1 : 0, bias, nullptr, out, m, n, workspace,
                     workspace_bytes, status, reinterpret_cast<cudaStream_t>(stream), activation, mul, mul_per_row);
}

int ayla_b200_gemm_packed(int op, int dtype, const void* bias, const void* a, const void* bt, void* out,
                          int64_t batch, int64_t m, int64_t n, int64_t k, uint32_t* status, void* stream) {
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  if (a == nullptr || bt == nullptr || out == nullptr) {
    return fail(AYLA_B200_E_INVALID, "a, bt and out must be non-null");
  }
  if (op == AYLA_B200_OP_ADDMM && bias == nullptr) {
    return fail(AYLA_B200_E_INVALID, "addmm needs a bias pointer");
  }
  if (!aligned16(a) || !aligned16(bt) || !aligned16(out)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "a, bt and out must be 16-byte aligned");
  }
  if (n > kPackedMaxN || k > kPackedMaxK || batch * ceil_div(m, 128) > 0x7FFFFFFF) {
    return fail(AYLA_B200_E_UNSUPPORTED, "the packed kernel takes n <= %d and k <= %d, got n=%lld k=%lld", kPackedMaxN,
                kPackedMaxK, (long long)n, (long long)k);
  }
  DeviceState* ds = nullptr;
  int dev = -1;
  rc = current_device_state(&ds, &dev);
  if (rc) return rc;
  PackedProblem pr = {};
  pr.a = a;
  pr.b = bt;
  pr.bias = op == AYLA_B200_OP_ADDMM ? bias : nullptr;
  pr.out = out;
  pr.batch = batch;
  pr.m = m;
  pr.n = n;
  pr.k = k;
  pr.is_bf16 = dtype == AYLA_B200_BF16 ? 1 : 0;
  pr.idesc_base = make_idesc(pr.is_bf16, 128, 0);
  pr.status = status;
  pr.timeout_ns = static_cast<unsigned long long>(g_timeout_ns.load());
  pr.debug_flags = g_debug_flags.load();
  pr.sm_count = ds->sm_count;
  pr.overlap = g_launch_overlap.load();
  pr.stream = reinterpret_cast<cudaStream_t>(stream);
  const cudaError_t err = launch_packed_gemm(pr);
  if (err != cudaSuccess) return fail(AYLA_B200_E_CUDA, "kernel launch failed: %s", cudaGetErrorString(err));
  return AYLA_B200_OK;
}

int ayla_b200_packed_preferred(int op, int64_t batch, int64_t m, int64_t n, int64_t k) {
  return ayla_b200_packed_preferred_at(op, batch, m, n, k, nullptr);
}

int ayla_b200_packed_preferred_at(int op, int64_t batch, int64_t m, int64_t n, int64_t k, const void* out) {
  if (check_shape(op, AYLA_B200_BF16, batch, m, n, k) != AYLA_B200_OK) return 0;
  return packed_preferred(batch, m, n, k, current_sm_count(), on_sectors(out)) ? 1 : 0;
}

int ayla_b200_gemm_static_scratch(int op, int dtype, const void* bias, const void* a, const void* bt,
                                  void* out, int64_t batch, int64_t m, int64_t n, int64_t k,
                                  const ayla_b200_config* cfg, uint32_t* status, void* stream) {
  int rc = check_shape(op, dtype, batch, m, n, k);
  if (rc) return rc;
  if (a == nullptr || bt == nullptr || out == nullptr) {
    return fail(AYLA_B200_E_INVALID, "a, bt and out must be non-null");
  }
  if (op == AYLA_B200_OP_ADDMM && bias == nullptr) {
    return fail(AYLA_B200_E_INVALID, "addmm needs a bias pointer");
  }
  if (!aligned16(a) || !aligned16(bt) || !aligned16(out)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "a, bt and out must be 16-byte aligned");
  }
  DeviceState* ds = nullptr;
  int dev = -1;
  rc = current_device_state(&ds, &dev);
  if (rc) return rc;
  ayla_b200_config c;
  if (cfg != nullptr) {
    c = *cfg;
  } else {
    default_config(batch, m, n, k, AYLA_B200_ACT_NONE, ds->machine, &c);
  }
  rc = check_config(c, false);
  if (rc) return rc;
  Problem pr;
  pr.k = k;
  pr.batch = batch;
  pr.rows = c.swap_ab ? n : m;
  pr.cols = c.swap_ab ? m : n;
  pr.row_operand = c.swap_ab ? bt : a;
  pr.col_operand = c.swap_ab ? a : bt;
  const int epi = (op == AYLA_B200_OP_ADDMM) ? EPI_BIAS : EPI_PLAIN;
  Plan plan{};
  rc = make_plan(c, epi, batch, pr.rows, pr.cols, k, ds->sm_count, &plan);
  if (rc) return rc;
  const size_t need = workspace_bytes_for(plan);
  if (need > static_cast<size_t>(AYLA_B200_STATIC_SCRATCH_BYTES)) {
    return fail(AYLA_B200_E_WORKSPACE,
                "this schedule needs %zu bytes of split-K scratch; the built-in array holds %zu "
                "(use ayla_b200_gemm with a caller workspace, or a smaller split_k)",
                need, static_cast<size_t>(AYLA_B200_STATIC_SCRATCH_BYTES));
  }
  void* scratch = nullptr;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (need > 0) {
    rc = static_scratch_for_current_device(dev, &scratch);
    if (rc) return rc;
    // The array keeps whatever the previous call left behind.  Only the arrival
    // counters must start at zero; partial sums are fully rewritten before they are read.
    const int counters = plan.row_tiles * (plan.shared_reduce ? plan.kernel->tile_n / 32 * 4 : 1);
    const cudaError_t err = cudaMemsetAsync(scratch, 0, static_cast<size_t>(counters) * 4, s);
    if (err != cudaSuccess) {
      return fail(AYLA_B200_E_CUDA, "clearing the split-K counters: %s", cudaGetErrorString(err));
    }
  }
  return launch_plan(plan, c, pr, dtype == AYLA_B200_BF16 ? 1 : 0, bias, nullptr, out, m, n, scratch, need,
                     status, s);
}

int ayla_b200_swiglu(int dtype, const void* x, const void* w_gate, const void* w_up, void* out,
                     int64_t m, int64_t n, int64_t k, const ayla_b200_config* cfg, uint32_t* status,
                     void* stream) {
  int rc = check_shape(AYLA_B200_OP_MM, dtype, 1, m, n, k);
  if (rc) return rc;
  if (x == nullptr || w_gate == nullptr || w_up == nullptr || out == nullptr) {
    return fail(AYLA_B200_E_INVALID, "x, w_gate, w_up and out must be non-null");
  }
  if (!aligned16(x) || !aligned16(w_gate) || !aligned16(w_up) || !aligned16(out)) {
    return fail(AYLA_B200_E_UNSUPPORTED, "x, w_gate, w_up and out must be 16-byte aligned");
  }
  DeviceState* ds = nullptr;
  int dev = -1;
  rc = current_device_state(&ds, &dev);
  if (rc) return rc;
  ayla_b200_config c;
  const bool swapped = cfg == nullptr && swapped_swiglu_config(m, n, k, ds->machine, &c);
  if (!swapped) {
    c = cfg != nullptr ? *cfg : row_major_swiglu_config(m);
    c.tile_n = 256;
    c.split_k = 1;
    c.swap_ab = 0;
    rc = check_config(c, true);
    if (rc) return rc;
  }
  Problem pr;
  pr.rows = swapped ? n : m;
  pr.cols = swapped ? m : n;
  pr.k = k;
  pr.batch = 1;
  pr.row_operand = swapped ? w_gate : x;
  pr.col_operand = swapped ? x : w_gate;
  Plan plan{};
  rc = make_plan(c, EPI_SWIGLU, 1, pr.rows, pr.cols, k, ds->sm_count, &plan);
  if (rc) return rc;
  return launch_plan(plan, c, pr, dtype == AYLA_B200_BF16 ? 1 : 0, nullptr, w_up, out, m, n, nullptr, 0,
                     status, reinterpret_cast<cudaStream_t>(stream));
}

int ayla_b200_rms_factors(int dtype, const void* x, void* factors, int64_t rows, int64_t k, float eps, void* stream) {
  const int rc = check_shape(AYLA_B200_OP_MM, dtype, 1, rows, 8, k);
  if (rc) return rc;
  if (x == nullptr || factors == nullptr) return fail(AYLA_B200_E_INVALID, "x and factors must be non-null");
  if (!aligned16(x) || (reinterpret_cast<uintptr_t>(factors) & 1) != 0) {
    return fail(AYLA_B200_E_UNSUPPORTED, "x must be 16-byte aligned and factors 2-byte aligned");
  }
  const cudaError_t err =
      launch_rms_factors(x, factors, static_cast<int>(rows), static_cast<int>(k), eps, dtype == AYLA_B200_BF16 ? 1 : 0,
                         g_launch_overlap.load(), reinterpret_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(AYLA_B200_E_CUDA, "kernel launch failed: %s", cudaGetErrorString(err));
  return AYLA_B200_OK;
}

// The listing covers the variants without the activation epilogue; each of them except the
// SwiGLU pair exists a second time with it.
int ayla_b200_kernel_count(void) { return registry().base_count; }

int ayla_b200_kernel_info(int i, int32_t* tile_n, int32_t* cta_group, int32_t* epilogue,
                          int32_t* transposed_out, int32_t* stages, int32_t* smem_bytes) {
  const Registry& reg = registry();
  if (i < 0 || i >= reg.base_count) return fail(AYLA_B200_E_INVALID, "variant index %d out of range", i);
  const KernelEntry& e = reg.entries[i];
  if (tile_n) *tile_n = e.tile_n;
  if (cta_group) *cta_group = e.cta_group;
  if (epilogue) *epilogue = e.epilogue;
  if (transposed_out) *transposed_out = e.transposed_out;
  if (stages) *stages = e.stages;
  if (smem_bytes) *smem_bytes = e.smem_bytes;
  return AYLA_B200_OK;
}

void ayla_b200_set_wait_timeout_ms(int64_t ms) {
  if (ms < 1) ms = 1;
  g_timeout_ns.store(ms * 1000000ll);
}

int ayla_b200_copy_2d(void* dst, size_t dst_pitch, const void* src, size_t src_pitch, size_t width_bytes,
                      size_t rows, void* stream) {
  if (dst == nullptr || src == nullptr) return fail(AYLA_B200_E_INVALID, "dst and src must be non-null");
  if (width_bytes == 0 || rows == 0) return AYLA_B200_OK;
  if (dst_pitch < width_bytes || src_pitch < width_bytes) {
    return fail(AYLA_B200_E_INVALID, "pitches must be at least the row width");
  }
  const cudaError_t err = cudaMemcpy2DAsync(dst, dst_pitch, src, src_pitch, width_bytes, rows,
                                            cudaMemcpyDeviceToDevice, reinterpret_cast<cudaStream_t>(stream));
  if (err != cudaSuccess) return fail(AYLA_B200_E_CUDA, "cudaMemcpy2DAsync: %s", cudaGetErrorString(err));
  return AYLA_B200_OK;
}

void ayla_b200_debug_set_flags(int flags) { g_debug_flags.store(flags); }

void ayla_b200_set_launch_overlap(int enabled) { g_launch_overlap.store(enabled ? 1 : 0); }

const char* ayla_b200_last_error(void) { return g_last_error.c_str(); }

const char* ayla_b200_version(void) { return "ayla_b200 0.1 (sm_100a, tcgen05)"; }

}  // extern "C"
