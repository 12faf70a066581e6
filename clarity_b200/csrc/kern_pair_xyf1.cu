// kern_pair_xyf1.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_forward<ProWork>(const PlanEntry&, cudaStream_t, const ProWork&, float2*, cudaError_t*);
template bool pair_xy_forward<ProPadded>(const PlanEntry&, cudaStream_t, const ProPadded&, float2*, cudaError_t*);
}  // namespace clarity
