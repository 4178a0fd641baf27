// lce_passes_f64_table.cu -- the FP64 update passes of batches with their table in memory.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, double, kTable)
}  // namespace lce
