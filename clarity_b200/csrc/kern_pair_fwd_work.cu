// kern_pair_fwd_work.cu -- column-pair passes (pair_dispatch.cuh): the forward passes of work-box and extrapolated estimates.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_FORWARD(ProWork, false)
CLARITY_PAIR_FORWARD(ProAccel, false)
}  // namespace clarity
#endif
