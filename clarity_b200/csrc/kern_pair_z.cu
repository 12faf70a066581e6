// kern_pair_z.cu -- column-pair pass kernels (pair_dispatch.cuh).
#include "pair_dispatch.cuh"

namespace clarity {
template bool pair_z<ModOTF>(const PlanEntry&, cudaStream_t, const ModOTF&, const float2*, float2*, cudaError_t*);
template bool pair_z<ModWiener>(const PlanEntry&, cudaStream_t, const ModWiener&, const float2*, float2*, cudaError_t*);
template bool pair_z<ModForward>(const PlanEntry&, cudaStream_t, const ModForward&, const float2*, float2*, cudaError_t*);
}  // namespace clarity
