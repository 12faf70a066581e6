// kern_pair_work.cu -- column-pair passes (pair_dispatch.cuh): work-box results and the trace of a result.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiWork, true, false)
CLARITY_PAIR_INVERSE(EpiWork, false, false)
CLARITY_PAIR_INVERSE(MidRLRatio, false, false)
}  // namespace clarity
#endif
