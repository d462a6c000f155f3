// Step plane passes of 128-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 128)
}  // namespace psb
