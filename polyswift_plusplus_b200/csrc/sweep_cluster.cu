// Grids with a one-launch sweep (sweep_cluster.cuh) and its dispatch.
#include "sweep_cluster.cuh"

namespace psb {

// (nx, ny, nz, CTAs of the cluster), a film nx x ny x 1 as (nx, 1, ny).  One plane
// or a few rows per CTA, as many CTAs as a cluster may have: us per step of both
// sweeps, FP64 (FP32), against the step passes' two launches:
//   16^3 1.8, eight CTAs 1.9 (4.6)     24^3 3.7 (2.8), eight CTAs 4.6 (3.3), passes 5.7
//   32^3 4.6 (3.2), passes 5.5 (5.0)   film 128^2 3.9, eight CTAs 4.5, passes 6.4
//   film 64^2 2.3, passes 4.9
// 48^3 has too much work for 16 SMs per sweep: FP32 9.0 against 7.3.
#define PSB_SWEEP_GRIDS(X)                                        \
  X(16, 16, 16, 16) X(24, 24, 24, 12) X(32, 32, 32, 16)           \
  X(16, 1, 16, 2) X(32, 1, 32, 4) X(64, 1, 64, 8) X(128, 1, 128, 16)

bool sweep_cluster_supported(int nx, int ny, int nz) {
  const int f = (nz == 1);
#define PSB_X(NX, NY, NZ, CL) \
  if (nx == NX && (f ? (NY == 1 && ny == NZ) : (ny == NY && nz == NZ))) return true;
  PSB_SWEEP_GRIDS(PSB_X)
#undef PSB_X
  return false;
}

template <typename T>
cudaError_t launch_sweep_cluster(const SweepWork<T>* w, int nw, int nx, int ny, int nz, const c2_t<T>* tx,
                                 const c2_t<T>* ty, const c2_t<T>* tz, cudaStream_t st) {
  const int f = (nz == 1);
#define PSB_X(NX, NY, NZ, CL) \
  if (nx == NX && (f ? (NY == 1 && ny == NZ) : (ny == NY && nz == NZ))) \
    return launch_sweep_cluster_t<T, NX, NY, NZ, CL>(w, nw, tx, f ? tz : ty, f ? ty : tz, st);
  PSB_SWEEP_GRIDS(PSB_X)
#undef PSB_X
  return cudaErrorInvalidValue;
}
template cudaError_t launch_sweep_cluster<float>(const SweepWork<float>*, int, int, int, int, const float2*,
                                                 const float2*, const float2*, cudaStream_t);
template cudaError_t launch_sweep_cluster<double>(const SweepWork<double>*, int, int, int, int, const double2*,
                                                  const double2*, const double2*, cudaStream_t);

cudaError_t sweep_cluster_set_polls(uint32_t polls) {
  return cudaMemcpyToSymbol(c_sweep_wait_polls, &polls, sizeof(polls));
}

}  // namespace psb
