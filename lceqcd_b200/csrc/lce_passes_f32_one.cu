// lce_passes_f32_one.cu -- the FP32 update passes of contexts with one chain.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, float, kOne)
LCE_PASSES_FIN(template, float)
}  // namespace lce
