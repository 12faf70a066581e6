// kern_pair_xyif3.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_inverse<EpiJVC, true>(const PlanEntry&, cudaStream_t, const EpiJVC&, float2*, cudaError_t*);
template bool pair_xy_inverse<EpiWork, true>(const PlanEntry&, cudaStream_t, const EpiWork&, float2*, cudaError_t*);
}  // namespace clarity
