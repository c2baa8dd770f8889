// Row-major-output variants, one CTA per 128-row tile: the kernels of launches whose
// k-splits share their sum through the workspace.
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_shared_cg1(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<64, 1, EPI_PLAIN, false, false, FORM_SHARED>());
  out->push_back(make_entry<128, 1, EPI_PLAIN, false, false, FORM_SHARED>());
  out->push_back(make_entry<192, 1, EPI_PLAIN, false, false, FORM_SHARED>());
  out->push_back(make_entry<256, 1, EPI_PLAIN, false, false, FORM_SHARED>());
  out->push_back(make_entry<64, 1, EPI_BIAS, false, false, FORM_SHARED>());
  out->push_back(make_entry<128, 1, EPI_BIAS, false, false, FORM_SHARED>());
  out->push_back(make_entry<192, 1, EPI_BIAS, false, false, FORM_SHARED>());
  out->push_back(make_entry<256, 1, EPI_BIAS, false, false, FORM_SHARED>());
}
}  // namespace ayla_b200
