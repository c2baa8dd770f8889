// Row-major-output activation variants with sixteen epilogue warps, one CTA per 128-row tile: the kernels of
// launches that do not split k and whose activation is more than a comparison.
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_paired_cg1(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<64, 1, EPI_PLAIN, false, 2, FORM_LEAN>());
  out->push_back(make_entry<128, 1, EPI_PLAIN, false, 2, FORM_LEAN>());
  out->push_back(make_entry<192, 1, EPI_PLAIN, false, 2, FORM_LEAN>());
  out->push_back(make_entry<256, 1, EPI_PLAIN, false, 2, FORM_LEAN>());
  out->push_back(make_entry<64, 1, EPI_BIAS, false, 2, FORM_LEAN>());
  out->push_back(make_entry<128, 1, EPI_BIAS, false, 2, FORM_LEAN>());
  out->push_back(make_entry<192, 1, EPI_BIAS, false, 2, FORM_LEAN>());
  out->push_back(make_entry<256, 1, EPI_BIAS, false, 2, FORM_LEAN>());
}
}  // namespace ayla_b200
