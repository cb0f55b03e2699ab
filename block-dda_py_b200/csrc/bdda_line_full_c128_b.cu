// Two-register-stage kernels, complex128: forward passes of a pencil full of data (the Green's tensor), lengths 140 to 320.
#include "bdda_line.cuh"

namespace bdda {

#define BDDA_LINE_ENTRY(MM) {MM, line_entry<double2, K_FWD, MM, true>()},
static const LineKernel kTable[] = {BDDA_LINE_MID(BDDA_LINE_ENTRY)};

const LineKernel* line_full_c128_b(int* n) {
  *n = (int)(sizeof(kTable) / sizeof(kTable[0]));
  return kTable;
}

}  // namespace bdda
