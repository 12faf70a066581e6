// kern_pair_xyif2.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_inverse<MidRLRatio, true>(const PlanEntry&, cudaStream_t, const MidRLRatio&, float2*, cudaError_t*);
}  // namespace clarity
