// FP64 instances of the N-grid maxima and the diagnostics reductions.
#include "vk_engine.cuh"

namespace vk {
template cudaError_t Engine<double>::ngrid_max(const NgridParams<double>&, cudaStream_t);
template cudaError_t Engine<double>::tier1_partial(const double2*, size_t, int, double, double*, int, cudaStream_t);
template cudaError_t Engine<double>::spectrum_partial(const double2*, size_t, int, double, int, double*, int, cudaStream_t);
}
