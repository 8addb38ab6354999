// fft_f32.cu -- the ComplexF32 FFT passes.
#include "fft_line.cuh"

namespace qob {

template void fft_axis<float>(const FftAxis&, int64_t, const void*, int64_t, int64_t, const FftOut&, int64_t, void*,
                               int, cudaStream_t);
template void fft_turn<float>(const FftAxis&, const FftAxis&, const GatherPlan&, const void*, int64_t, const void*,
                               int64_t, int64_t, const FftOut&, int64_t, void*, void*, int, cudaStream_t);

}  // namespace qob
