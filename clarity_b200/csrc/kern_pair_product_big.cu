// kern_pair_product_big.cu -- column-pair passes (pair_dispatch.cuh): the RL product, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiRLProduct, true, true)
CLARITY_PAIR_INVERSE(EpiRLProduct, false, true)
}  // namespace clarity
