// kern_pair_xyf2.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_forward<ProImage>(const PlanEntry&, cudaStream_t, const ProImage&, float2*, cudaError_t*);
template bool pair_xy_forward<ProAccel>(const PlanEntry&, cudaStream_t, const ProAccel&, float2*, cudaError_t*);
}  // namespace clarity
