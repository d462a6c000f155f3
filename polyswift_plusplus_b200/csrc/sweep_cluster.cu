// Grids with a one-launch sweep (sweep_cluster.cuh) and its dispatch.
#include "sweep_cluster.cuh"

namespace psb {

bool sweep_cluster_supported(int nx, int ny, int nz) {
  const int f = (nz == 1);
#define PSB_X(NX, NY, NZ, CL) \
  if (nx == NX && (f ? (NY == 1 && ny == NZ) : (ny == NY && nz == NZ))) return true;
  PSB_SWEEP_GRIDS(PSB_X)
#undef PSB_X
  return false;
}

template <typename T, bool DST>
static cudaError_t launch_any(const SweepWork<T>* w, int nw, int nx, int ny, int nz, const c2_t<T>* tx,
                                 const c2_t<T>* ty, const c2_t<T>* tz, cudaStream_t st) {
  const int f = (nz == 1);
#define PSB_X(NX, NY, NZ, CL) \
  if (nx == NX && (f ? (NY == 1 && ny == NZ) : (ny == NY && nz == NZ))) \
    return launch_sweep_cluster_t<T, NX, NY, NZ, CL, DST>(w, nw, tx, f ? tz : ty, f ? ty : tz, st);
  PSB_SWEEP_GRIDS(PSB_X)
#undef PSB_X
  return cudaErrorInvalidValue;
}
template <typename T>
cudaError_t launch_sweep_cluster(const SweepWork<T>* w, int nw, int nx, int ny, int nz, const c2_t<T>* tx,
                                 const c2_t<T>* ty, const c2_t<T>* tz, cudaStream_t st) {
  return launch_any<T, false>(w, nw, nx, ny, nz, tx, ty, tz, st);
}
cudaError_t launch_sweep_cluster_to(const SweepWork<double>* w, int nw, int nx, int ny, int nz, const double2* tx,
                                    const double2* ty, const double2* tz, cudaStream_t st) {
  return launch_any<double, true>(w, nw, nx, ny, nz, tx, ty, tz, st);
}
template cudaError_t launch_sweep_cluster<float>(const SweepWork<float>*, int, int, int, int, const float2*,
                                                 const float2*, const float2*, cudaStream_t);
template cudaError_t launch_sweep_cluster<double>(const SweepWork<double>*, int, int, int, int, const double2*,
                                                  const double2*, const double2*, cudaStream_t);

cudaError_t sweep_cluster_set_polls(uint32_t polls) {
  return cudaMemcpyToSymbol(c_sweep_wait_polls, &polls, sizeof(polls));
}

}  // namespace psb
