// kern_pair_fwd_work_big.cu -- column-pair passes (pair_dispatch.cuh): the forward passes of work-box and extrapolated estimates, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_FORWARD(ProWork, true)
CLARITY_PAIR_FORWARD(ProAccel, true)
}  // namespace clarity
