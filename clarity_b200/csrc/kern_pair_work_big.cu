// kern_pair_work_big.cu -- column-pair passes (pair_dispatch.cuh): work-box results and the trace of a result, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiWork, true, true)
CLARITY_PAIR_INVERSE(EpiWork, false, true)
CLARITY_PAIR_INVERSE(MidRLRatio, false, true)
}  // namespace clarity
