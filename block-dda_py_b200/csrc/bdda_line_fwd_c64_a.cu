// Two-register-stage kernels, complex64: forward (Z, Y) passes, lengths up to 128.
#include "bdda_line.cuh"

namespace bdda {

#define BDDA_LINE_ENTRY(MM) {MM, line_entry<float2, K_FWD, MM, false>()},
static const LineKernel kTable[] = {BDDA_LINE_SHORT(BDDA_LINE_ENTRY)};

const LineKernel* line_fwd_c64_a(int* n) {
  *n = (int)(sizeof(kTable) / sizeof(kTable[0]));
  return kTable;
}

}  // namespace bdda
