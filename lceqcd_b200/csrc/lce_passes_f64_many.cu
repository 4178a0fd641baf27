// lce_passes_f64_many.cu -- the FP64 update passes of batches with their table in the arguments.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, double, kMany)
}  // namespace lce
