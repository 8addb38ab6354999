// k_multi_df.cu -- the several-index gather (k_multi.cuh) for double-float.
#include "k_multi_launch.cuh"

namespace qob {
namespace gather {
template void launch_multi<DF, kReal>(const GatherView&, const void*, int64_t, int64_t, void*, int64_t, int64_t, int64_t, c128, c128, cudaStream_t);
template void launch_multi<DF, kPhased>(const GatherView&, const void*, int64_t, int64_t, void*, int64_t, int64_t, int64_t, c128, c128, cudaStream_t);
}  // namespace gather
}  // namespace qob
