// k_multi_f32.cu -- the several-index gather (k_multi.cuh) for ComplexF32.
#include "k_multi_launch.cuh"

namespace qob {
namespace gather {
template void launch_multi<float, kReal>(const GatherView&, const void*, int64_t, int64_t, void*, int64_t, int64_t, int64_t, c128, c128, cudaStream_t);
template void launch_multi<float, kPhased>(const GatherView&, const void*, int64_t, int64_t, void*, int64_t, int64_t, int64_t, c128, c128, cudaStream_t);
}  // namespace gather
}  // namespace qob
