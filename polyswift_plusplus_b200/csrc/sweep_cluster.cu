// Grids with a one-launch sweep (sweep_cluster.cuh) and its dispatch.
#include "../../include/pswift.h"
#include "sweep_cluster.cuh"

namespace psb {

template <typename T, bool DST> static bool fits_any(int nx, int ny, int nz) {
  const int f = (nz == 1);
#define PSB_X(NX, NY, NZ, CL) \
  if (nx == NX && (f ? (NY == 1 && ny == NZ) : (ny == NY && nz == NZ))) return sweep_cluster_fits_t<T, NX, NY, NZ, CL, DST>();
  PSB_SWEEP_GRIDS(PSB_X)
#undef PSB_X
  return false;
}
template <typename T> bool sweep_cluster_fits(int nx, int ny, int nz) { return fits_any<T, false>(nx, ny, nz); }
bool sweep_cluster_to_fits(int nx, int ny, int nz) { return fits_any<double, true>(nx, ny, nz); }
template bool sweep_cluster_fits<float>(int, int, int);
template bool sweep_cluster_fits<double>(int, int, int);

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

extern "C" int ps_gpu_one_launch(const int n[3], int precision) {
  if (!n) return 0;
  return precision == PS_PREC_MIXED ? psb::sweep_cluster_fits<float>(n[0], n[1], n[2])
                                    : psb::sweep_cluster_fits<double>(n[0], n[1], n[2]);
}
