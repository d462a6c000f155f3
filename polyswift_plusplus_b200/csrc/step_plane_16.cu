// Step plane passes of 16-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 16)
}  // namespace psb
