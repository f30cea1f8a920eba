// Coarse-fine pencil-kernel instantiations: double bulk storage, 7x11-oct XY
// tiles (a ring of 16 x 24 columns: 12 full warps), registers sized for 1 CTA
// per SM.
#include "rh_launch.h"
namespace rh {
static TileRegistrar<double, 7, 11, 1, true> reg_amr_f64_7x11_b1;
}
