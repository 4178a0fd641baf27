// lce_passes_f64_one.cu -- the FP64 update passes of contexts with one chain.
#include "lce_passes.cuh"

namespace lce {
LCE_PASSES(template, double, kOne)
LCE_PASSES_FIN(template, double)
}  // namespace lce
