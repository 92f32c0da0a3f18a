// engine_f64.cu -- Engine<double>: the all-FP64 pipelines.
#include "engine_pass.cuh"

namespace mlq {
MLQ_PASS_EXTERN(double)
template class Engine<double>;
}  // namespace mlq
