// kern_pair_ratio.cu -- column-pair passes (pair_dispatch.cuh): the RL ratio.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(MidRLRatio, true, false)
}  // namespace clarity
#endif
