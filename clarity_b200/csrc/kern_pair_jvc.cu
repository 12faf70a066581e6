// kern_pair_jvc.cu -- column-pair passes (pair_dispatch.cuh): the JVC update.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiJVC, true, false)
CLARITY_PAIR_INVERSE(EpiJVC, false, false)
}  // namespace clarity
#endif
