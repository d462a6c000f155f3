// Grids with a one-launch sweep (sweep_cluster.cuh) and its dispatch.
#include "sweep_cluster.cuh"

namespace psb {

// (nx, ny, nz, CTAs of the cluster), a film nx x ny x 1 as (nx, 1, ny).  One plane
// or a few rows per CTA, as many CTAs as a cluster may have: us per step of both
// sweeps, FP64 (FP32), against the step passes' two launches:
//   8^3 1.3 (1.4), 12^3 1.7 (1.6)      passes 5.6 and 6.3 (7.0)
//   16^3 1.8, eight CTAs 1.9           passes 4.6
//   24^3 3.7 (2.8), eight CTAs 4.6 (3.3), passes 5.7
//   32^3 4.6 (3.2), passes 5.5 (5.0)
//   films, eight rows a CTA: 24^2 1.6 (1.5), passes 10 (12); 48^2 2.1 (1.9), 11 (13);
//   64^2 2.3, 4.9; 96^2 3.5 (2.6), 16 (19); 128^2 3.9, eight CTAs 4.5, passes 6.4
// 48^3 has too much work for 16 SMs per sweep: FP32 9.0 against 7.3.
#define PSB_SWEEP_GRIDS(X)                                        \
  X(8, 8, 8, 8) X(12, 12, 12, 12) X(16, 16, 16, 16)               \
  X(24, 24, 24, 12) X(32, 32, 32, 16) X(16, 1, 16, 2)             \
  X(24, 1, 24, 3) X(32, 1, 32, 4) X(48, 1, 48, 6)                 \
  X(64, 1, 64, 8) X(96, 1, 96, 12) X(128, 1, 128, 16)

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
