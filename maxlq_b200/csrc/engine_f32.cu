// engine_f32.cu -- Engine<float>: the mixed-precision (FP32 fields) pipelines.
#include "engine_pass.cuh"

namespace mlq {
MLQ_PASS_EXTERN(float)
template class Engine<float>;
}  // namespace mlq
