// Fused SwiGLU variants: gate and up weights share one stream of x.
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_swiglu(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<256, 1, EPI_SWIGLU, false>());
  out->push_back(make_entry<256, 2, EPI_SWIGLU, false>());
}
}  // namespace ayla_b200
