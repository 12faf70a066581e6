// kern_pair_fwd_big.cu -- column-pair passes (pair_dispatch.cuh): the forward passes of every call, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_FORWARD(ProPadded, true)
CLARITY_PAIR_FORWARD(ProImage, true)
}  // namespace clarity
