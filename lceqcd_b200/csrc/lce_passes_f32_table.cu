// lce_passes_f32_table.cu -- the FP32 update passes of batches with their table in memory.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, float, kTable)
}  // namespace lce
