// Two-register-stage kernels, complex128: inverse (Y^-1, Z^-1) passes, lengths 140 to 320.
#include "bdda_line.cuh"

namespace bdda {

#define BDDA_LINE_ENTRY(MM) {MM, line_entry<double2, K_INV, MM, false>()},
static const LineKernel kTable[] = {BDDA_LINE_MID(BDDA_LINE_ENTRY)};

const LineKernel* line_inv_c128_b(int* n) {
  *n = (int)(sizeof(kTable) / sizeof(kTable[0]));
  return kTable;
}

}  // namespace bdda
