// engine_pass.cu -- the pass kernels of one precision and size, compiled once
// per (MLQ_PASS_T, MLQ_PASS_N) (build.py).
#include "engine_pass.cuh"

namespace mlq {
MLQ_PASS_UNIT(, MLQ_PASS_T, MLQ_PASS_N)
}  // namespace mlq
