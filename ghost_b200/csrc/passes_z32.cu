// passes_z32.cu -- the FP32 Z passes.
#include "passes_z.cuh"

namespace gb {
GB_INST(float)
}  // namespace gb
