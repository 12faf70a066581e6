// kern_pair_product.cu -- column-pair passes (pair_dispatch.cuh): the RL product.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiRLProduct, true, false)
CLARITY_PAIR_INVERSE(EpiRLProduct, false, false)
}  // namespace clarity
#endif
