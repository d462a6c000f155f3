// Step plane passes of 96-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 96)
}  // namespace psb
