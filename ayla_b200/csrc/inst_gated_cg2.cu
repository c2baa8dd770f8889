// Row-major-output variants for a gate operand shaped like the output, a CTA pair per 256-row tile.
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_gated_cg2(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<64, 2, EPI_PLAIN, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<128, 2, EPI_PLAIN, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<192, 2, EPI_PLAIN, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<256, 2, EPI_PLAIN, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<64, 2, EPI_BIAS, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<128, 2, EPI_BIAS, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<192, 2, EPI_BIAS, false, true, FORM_LEAN, true>());
  out->push_back(make_entry<256, 2, EPI_BIAS, false, true, FORM_LEAN, true>());
}
}  // namespace ayla_b200
