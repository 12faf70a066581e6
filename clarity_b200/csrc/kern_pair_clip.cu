// kern_pair_clip.cu -- column-pair passes (pair_dispatch.cuh): the last pass of the single-pass filters.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_INVERSE(EpiClip, false, false)
}  // namespace clarity
#endif
