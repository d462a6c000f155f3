// Adjoint steps in the step plane pass: descriptors shared by adjoint.cu and
// step_plane.cuh.
#pragma once

#include <cuda_runtime.h>

#include "../../include/pswift.h"
#include "kernels.h"

namespace psb {

struct SrcEntry {
  const double* gphi;
  const double* partner;
  double coef;  // without the 1/Q factor
};

// The real-space part of the adjoint of one propagator step s -> s + 1:
//   mu_s = wf G(wf lam_{s+1});  dL/dw -= ds/2 (lam_{s+1} q_{s+1} + q_s mu_s);
//   lam_s = mu_s + the explicit sources of slice s.
// The fused pass takes the two products slice by slice instead of step by step:
// q_s mu_s for step s's block (gwb) and q_s lam_s for step s - 1's (gwb2), so that
// it reads neither lam_{s+1} nor q_{s+1}.
struct AdjPoint {
  const double* q_s;
  double* gwb;       // dL/dw of step s's block (the fused pass at a sweep's end: nullptr)
  double* gwb2;      // of step s - 1's (nullptr: none)
  double* lam_out;   // nullptr: lambda_s is not needed (s = 0)
  double half_ds, half_ds2;
  // the separate pointwise kernel only
  const double* mu;
  const double* lam_next;
  const double* q_next;
  const double* w;
  double* dsw_part;  // partials of the explicit ds derivative, one per CTA
  int n_src;
  SrcEntry src[2];
  const double* q_partner;  // Q source partner (nullptr: none at this slice)
  const double* extra;      // lambda of a sweep's end: junction contributions (nullptr: none)
  const double* psi;        // charged block: the exponent is w + facz psi (nullptr: w alone)
  double facz;
};

struct AdjArgs {
  const AdjPoint* points;  // by work (blockIdx.y); read for works in an adjoint mode
  const double* q;         // Q
  const double* gq;        // dL/dQ
  double n;                // grid points
};
struct AdjGlobals {
  double inv_q, gq_n;
};

// Plane pass modes beside FIRST, MID and LAST: INIT makes lambda of a sweep's end
// from its sources and starts the transform of wf lambda; MID finishes mu, makes the
// next lambda and starts its transform; LAST only finishes.
enum { MODE_ADJ_INIT = 3, MODE_ADJ_MID = 4, MODE_ADJ_LAST = 5 };

// The fused adjoint steps exist for square planes of the step plane pass.
bool adj_step_supported(int ny, int nz);
cudaError_t launch_step_plane_adj(const PlaneWork<double>* d_works, int nworks, int nx, int ny, const double2* tw_y,
                                  const double2* tw_z, const AdjArgs& adj, cudaStream_t st);
// x pass of an adjoint step on the compact layout: U and V forward, the stress
// partials of sum conj(U) V K k_d^2 (d = 0, 1, 2: part[d * stride + CTA]), then
// U <- IFFT(K U).
struct AdjXWork {
  double2* u;
  const double2* v;
  const double* kx;
  const double* kyzc;
  double* part;
};
int adj_x_tiles(int nx, int inner);  // CTAs of the pass
cudaError_t launch_adj_x(const AdjXWork* d_works, int nworks, int nx, int ny, int nz, double dx, double dy, double dz, int stride,
                         const double2* tw, cudaStream_t st);

}  // namespace psb
