// Step plane passes of 48-row planes.
#include "step_plane.cuh"

namespace psb {
PSB_STEP_PLANE_NY(, 48)
}  // namespace psb
