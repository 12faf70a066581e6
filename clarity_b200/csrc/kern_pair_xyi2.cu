// kern_pair_xyi2.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_inverse<EpiRLProduct, false>(const PlanEntry&, cudaStream_t, const EpiRLProduct&, float2*, cudaError_t*);
template bool pair_xy_inverse<MidRLRatio, false>(const PlanEntry&, cudaStream_t, const MidRLRatio&, float2*, cudaError_t*);
template bool pair_xy_inverse<EpiJVC, false>(const PlanEntry&, cudaStream_t, const EpiJVC&, float2*, cudaError_t*);
}  // namespace clarity
