// Pencil-kernel instantiations: double bulk storage, 15x5-oct XY tiles (a ring
// of 32 x 12 columns: 12 full warps), registers sized for 1 CTA per SM; slope
// types 0-3 x llf/hll/hllc.
#include "rh_launch.h"
namespace rh {
static TileRegistrar<double, 15, 5, 1> reg_f64_15x5_b1;
}
