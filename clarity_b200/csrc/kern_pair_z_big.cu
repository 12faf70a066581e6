// kern_pair_z_big.cu -- column-pair passes (pair_dispatch.cuh): the z passes of every call, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_Z(ModForward, true)
CLARITY_PAIR_Z(ModOTF, true)
}  // namespace clarity
