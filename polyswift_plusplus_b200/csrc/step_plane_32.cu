// Step plane passes of 32-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 32)
}  // namespace psb
