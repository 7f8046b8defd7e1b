// The tile Pi kernel's instantiations for finite-difference order q = 8.
#include "rhs_pi_tile.cuh"

namespace tgh {
TGH_DEFINE_PI_TILE(8)
}  // namespace tgh
