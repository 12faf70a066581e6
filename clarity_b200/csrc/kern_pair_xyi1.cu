// kern_pair_xyi1.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_inverse<EpiClip, false>(const PlanEntry&, cudaStream_t, const EpiClip&, float2*, cudaError_t*);
template bool pair_xy_inverse<EpiWork, false>(const PlanEntry&, cudaStream_t, const EpiWork&, float2*, cudaError_t*);
}  // namespace clarity
