// Dispatch of the step plane pass (step_plane.cuh) over the plane's extents.
#include "step_plane.cuh"

namespace psb {

PSB_STEP_PLANE_NY(extern, 16)
PSB_STEP_PLANE_NY(extern, 24)
PSB_STEP_PLANE_NY(extern, 32)
PSB_STEP_PLANE_NY(extern, 48)
PSB_STEP_PLANE_NY(extern, 64)
PSB_STEP_PLANE_NY(extern, 96)
PSB_STEP_PLANE_NY(extern, 128)

// Every plane of two listed extents: its packed rows fit one CTA's shared memory
// in both precisions (128 x 128 in FP64: 141 KB).
bool step_plane_supported(int ny, int nz) {
  bool y = false, z = false;
  for (int e : kStepExtents) {
    y |= (e == ny);
    z |= (e == nz);
  }
  return y && z;
}

template <typename T>
cudaError_t launch_step_plane(const PlaneWork<T>* w, int nw, int nx, int ny, int nz, bool early,
                              const c2_t<T>* ty, const c2_t<T>* tz, cudaStream_t st) {
  switch (ny) {
    case 16: return launch_step_plane_ny<T, 16>(w, nw, nx, nz, early, ty, tz, st);
    case 24: return launch_step_plane_ny<T, 24>(w, nw, nx, nz, early, ty, tz, st);
    case 32: return launch_step_plane_ny<T, 32>(w, nw, nx, nz, early, ty, tz, st);
    case 48: return launch_step_plane_ny<T, 48>(w, nw, nx, nz, early, ty, tz, st);
    case 64: return launch_step_plane_ny<T, 64>(w, nw, nx, nz, early, ty, tz, st);
    case 96: return launch_step_plane_ny<T, 96>(w, nw, nx, nz, early, ty, tz, st);
    case 128: return launch_step_plane_ny<T, 128>(w, nw, nx, nz, early, ty, tz, st);
  }
  return cudaErrorInvalidValue;
}
template cudaError_t launch_step_plane<float>(const PlaneWork<float>*, int, int, int, int, bool, const float2*,
                                              const float2*, cudaStream_t);
template cudaError_t launch_step_plane<double>(const PlaneWork<double>*, int, int, int, int, bool, const double2*,
                                               const double2*, cudaStream_t);

}  // namespace psb
