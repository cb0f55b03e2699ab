// Two-register-stage kernels, complex64: X passes, lengths 140 to 320.
#include "bdda_line.cuh"

namespace bdda {

#define BDDA_LINE_ENTRY(MM) {MM, conv_entry<float2, MM>()},
static const LineKernel kTable[] = {BDDA_LINE_MID(BDDA_LINE_ENTRY)};

const LineKernel* line_conv_c64_b(int* n) {
  *n = (int)(sizeof(kTable) / sizeof(kTable[0]));
  return kTable;
}

}  // namespace bdda
