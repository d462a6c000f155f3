// Dispatch of the split step (step_split.cuh): 256 x 256 y-z planes, any x extent.
#include "step_split.cuh"

namespace psb {

bool step_split_supported(int ny, int nz) { return ny == 256 && nz == 256; }

size_t step_split_spectrum(int prec_bytes, int nx, int ny, int nz) {
  return (size_t)nx * ny * (nz / 2 + 32 / (2 * prec_bytes));
}

template <typename T>
cudaError_t launch_split_plane(const PlaneWork<T>* w, int nw, int nx, const c2_t<T>* ty, const c2_t<T>* tz,
                               cudaStream_t st) {
  return launch_split_plane_t<T, 256, 256>(w, nw, nx, ty, tz, st);
}

template <typename T>
cudaError_t launch_split_pencil(const PencilWork<T>* w, int nw, int nx, int nz, const c2_t<T>* tx, cudaStream_t st) {
#define PSB_X(NX) \
  if (nx == NX) return launch_split_pencil_t<T, NX, 256>(w, nw, nz, tx, st);
  PSB_X(1) PSB_X(4) PSB_X(8) PSB_X(12) PSB_X(16) PSB_X(24) PSB_X(32) PSB_X(48) PSB_X(64) PSB_X(96) PSB_X(128)
  PSB_X(256)
#undef PSB_X
  return cudaErrorInvalidValue;
}

template cudaError_t launch_split_plane<float>(const PlaneWork<float>*, int, int, const float2*, const float2*,
                                               cudaStream_t);
template cudaError_t launch_split_plane<double>(const PlaneWork<double>*, int, int, const double2*, const double2*,
                                                cudaStream_t);
template cudaError_t launch_split_pencil<float>(const PencilWork<float>*, int, int, int, const float2*, cudaStream_t);
template cudaError_t launch_split_pencil<double>(const PencilWork<double>*, int, int, int, const double2*,
                                                 cudaStream_t);

}  // namespace psb
