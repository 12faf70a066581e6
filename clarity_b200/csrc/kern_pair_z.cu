// kern_pair_z.cu -- column-pair passes (pair_dispatch.cuh): the z passes of every call.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_Z(ModForward, false)
CLARITY_PAIR_Z(ModOTF, false)
}  // namespace clarity
#endif
