// Fused SwiGLU in the swapped (small-M) form: 64 rows of the gate weight and the same 64 of the up weight fill
// the 128-row tile, the narrow accumulator width covers M.
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_swiglu_trans(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<16, 1, EPI_SWIGLU, true>());
  out->push_back(make_entry<32, 1, EPI_SWIGLU, true>());
  out->push_back(make_entry<64, 1, EPI_SWIGLU, true>());
  out->push_back(make_entry<128, 1, EPI_SWIGLU, true>());
  out->push_back(make_entry<16, 1, EPI_SWIGLU, true, false, true>());
  out->push_back(make_entry<32, 1, EPI_SWIGLU, true, false, true>());
  out->push_back(make_entry<64, 1, EPI_SWIGLU, true, false, true>());
  out->push_back(make_entry<128, 1, EPI_SWIGLU, true, false, true>());
}
}  // namespace ayla_b200
