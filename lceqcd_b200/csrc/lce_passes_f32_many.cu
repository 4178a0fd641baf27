// lce_passes_f32_many.cu -- the FP32 update passes of batches with their table in the arguments.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, float, kMany)
}  // namespace lce
