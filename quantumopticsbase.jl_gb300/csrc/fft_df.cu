// fft_df.cu -- the double-float FFT passes.
#include "fft_line.cuh"

namespace qob {

template void fft_axis<gather::DF>(const FftAxis&, int64_t, const void*, int64_t, int64_t, const FftOut&, int64_t, void*,
                               int, cudaStream_t);
template void fft_turn<gather::DF>(const FftAxis&, const FftAxis&, const GatherPlan&, const void*, int64_t, const void*,
                               int64_t, int64_t, const FftOut&, int64_t, void*, void*, int, cudaStream_t);

}  // namespace qob
