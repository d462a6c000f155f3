// Step plane passes of 24-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 24)
}  // namespace psb
