// kern_pair_xyif1.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_xy_inverse<EpiRLProduct, true>(const PlanEntry&, cudaStream_t, const EpiRLProduct&, float2*, cudaError_t*);
}  // namespace clarity
