// kern_pair_jvc_big.cu -- column-pair passes (pair_dispatch.cuh): the JVC update, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiJVC, true, true)
CLARITY_PAIR_INVERSE(EpiJVC, false, true)
}  // namespace clarity
