// passes_z64.cu -- the FP64 Z passes.
#include "passes_z.cuh"

namespace gb {
GB_INST(double)
}  // namespace gb
