// kern_pair_clip_big.cu -- column-pair passes (pair_dispatch.cuh): the last pass of the single-pass filters, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiClip, false, true)
}  // namespace clarity
