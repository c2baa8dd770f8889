// Row-major-output variants for products of at most 128 rows: a CTA pair per 128-row tile (tcgen05 cta_group::2).
#include "kernel_registry.h"

namespace ayla_b200 {
void append_variants_flat(std::vector<KernelEntry>* out) {
  out->push_back(make_entry<128, 2, EPI_PLAIN, false, 0, FORM_FLAT>());
  out->push_back(make_entry<256, 2, EPI_PLAIN, false, 0, FORM_FLAT>());
  out->push_back(make_entry<128, 2, EPI_BIAS, false, 0, FORM_FLAT>());
  out->push_back(make_entry<256, 2, EPI_BIAS, false, 0, FORM_FLAT>());
  out->push_back(make_entry<128, 2, EPI_PLAIN, false, 1, FORM_FLAT>());
  out->push_back(make_entry<256, 2, EPI_PLAIN, false, 1, FORM_FLAT>());
  out->push_back(make_entry<128, 2, EPI_BIAS, false, 1, FORM_FLAT>());
  out->push_back(make_entry<256, 2, EPI_BIAS, false, 1, FORM_FLAT>());
}
}  // namespace ayla_b200
