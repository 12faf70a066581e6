// kern_pair_fwd.cu -- column-pair passes (pair_dispatch.cuh): the forward passes of every call.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_FORWARD(ProPadded, false)
CLARITY_PAIR_FORWARD(ProImage, false)
}  // namespace clarity
#endif
