// kern_pair_z_wiener_big.cu -- column-pair passes (pair_dispatch.cuh): the Wiener filter, radices above 16.
#include "pair_dispatch.cuh"

namespace clarity {
CLARITY_PAIR_Z(ModWiener, true)
}  // namespace clarity
