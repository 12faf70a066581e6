// kern_pair_ratio_big.cu -- column-pair passes (pair_dispatch.cuh): the RL ratio, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(MidRLRatio, true, true)
}  // namespace clarity
