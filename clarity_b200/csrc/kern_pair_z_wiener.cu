// kern_pair_z_wiener.cu -- column-pair passes (pair_dispatch.cuh): the Wiener filter.
#ifndef CLARITY_HOST_EMULATION  // one register class there
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_Z(ModWiener, false)
}  // namespace clarity
#endif
