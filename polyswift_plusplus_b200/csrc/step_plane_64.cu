// Step plane passes of 64-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 64)
}  // namespace psb
