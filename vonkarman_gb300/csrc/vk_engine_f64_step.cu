// FP64 instances of the nonlinear evaluation (P1..P5).  The FP64 form is split
// over several units so that they compile in parallel.
#include "vk_engine.cuh"

namespace vk {
template cudaError_t Engine<double>::nle(const NleParams<double>&, cudaStream_t);
}
