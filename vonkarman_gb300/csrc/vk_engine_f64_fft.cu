// FP64 instances of the standalone FFT backend.
#include "vk_engine.cuh"

namespace vk {
template cudaError_t Engine<double>::fft_r2c(const FftParams<double>&, cudaStream_t);
template cudaError_t Engine<double>::fft_c2r(const FftParams<double>&, cudaStream_t);
}
