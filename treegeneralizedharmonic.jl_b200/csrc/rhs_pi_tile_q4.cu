// The tile Pi kernel's instantiations for finite-difference order q = 4.
#include "rhs_pi_tile.cuh"

namespace tgh {
TGH_DEFINE_PI_TILE(4)
}  // namespace tgh
