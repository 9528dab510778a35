// FP64 instances of the discrete adjoint.
#include "vk_engine.cuh"

namespace vk {
template cudaError_t Engine<double>::nle_adjoint(const NlaParams<double>&, cudaStream_t);
template cudaError_t Engine<double>::adj_mode(int, double, size_t, const double2*, double2*, int, cudaStream_t);
template cudaError_t Engine<double>::hermitian_avg(int, size_t, const double2*, double2*, cudaStream_t);
}
