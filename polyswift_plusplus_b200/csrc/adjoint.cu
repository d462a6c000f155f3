// Adjoint of the propagator sweeps of one linear block copolymer (FP64).
//
// Forward:  q_{s+1} = wf_s * G_s(wf_s * q_s) along the chain (sweep 0, from
// block 0's free head) and q+ the same way from the other end (sweep 1);
// phi_f = (1/Q) sum_blocks densfac ds_b sum_n c_n q_n q+_{M-n} with the
// reference's quadrature weights (pspolymer/PsBlock.cpp:256-380) and
// Q = <q_head q+_end> of block 0 (pspolymer/PsBlock.cpp:205-237).  wf_s =
// exp(-ds_b w_f/2) and G_s = IFFT exp(-ds_b b^2 k^2) FFT / N for the block b
// of step s, as in pspolymer/PsFlexPseudoSpec.cpp:158-293.
//
// Backward, for a loss L(phi, ln Q): G is a real symmetric convolution, so the
// transpose of a step is the step itself and the adjoint of each sweep is one
// more sweep run backwards with sources from the quadrature:
//   lam_s = wf_s G_s(wf_s lam_{s+1}) + dL/dq_s (explicit),
//   dL/dw_f      += -ds_b/2 (lam_{s+1} q_{s+1} + q_s mu_s),   mu_s = wf G(wf lam_{s+1}),
//   dL/dL_d      += (2 ds_b b^2 / L_d) R_d,   R_d = (1/N) sum_k conj(U) V K k_d^2,
//   dL/d(ds_b)   += -b^2 sum_d R_d - 1/2 <w_f, lam_{s+1} q_{s+1} + q_s mu_s>,
// with U = FFT(wf lam_{s+1}), V = FFT(wf q_s), plus the explicit ds factor of
// the quadrature weights.  L_d are the box lengths n_d * cell_d.
//
// Storage: the slices of both sweeps are checkpointed every C contour steps
// (C = 1: full storage; C ~ sqrt(M): square-root checkpointing).  Segment j of
// sweep 0 covers n in [jC, min((j+1)C, M)]; the matching part of sweep 1
// (m = M - n) starts at a checkpoint placed at m = M - min((j+1)C, M), so both
// halves of a segment are recomputed from one checkpoint each into two
// C-slice buffers (the checkpoint is the first slice), and the recomputed slices
// equal the stored ones bit for bit.
//
// Up to nx = 96 the two adjoint sweeps advance together, sweep 0's through segments
// J - 1, J - 2, ... and sweep 1's through 0, 1, ...: both segments are recomputed by
// the same launches into two sets of buffers, and so are the quadrature's, two at a
// time.  A launch has a sweep's nx planes to work on, so at 64^3 one sweep leaves
// half the chip idle: forward and backward of 128 steps, one sweep's adjoint at a
// time and both, ms: 16^3 4.9 and 3.2, 32^3 6.9 and 4.3, 64^3 9.9 and 7.8, 96^3 26.1
// and 23.5.  At 128^3 (49.8 and 49.3) the second set of buffers is not worth its
// memory.  On grids with a one-launch sweep (sweep_cluster.cuh) the forward and every
// recomputation is one launch: 16^3 3.2 -> 2.3, 32^3 4.3 -> 3.8.
//
// Branched (tree) chains keep every slice of every sweep (no checkpoints): the
// forward is the engine's own sweeps with junction products, and the adjoint
// sweeps run in reverse dependency order.  A sweep that starts at a junction,
// q_0 = prod_j q^(j)_end, hands its lam_0 back to each arriving sweep's end:
// lam^(j)_end += lam_0 prod_{j' != j} q^(j')_end, before that sweep's adjoint
// starts.
//
// On square planes of extents 16 to 128 an adjoint step is two launches
// (adjoint.cuh, adj_step.cu): the plane pass finishes mu, does the pointwise update
// and starts the transforms of the next wf lambda and wf q; the x pass forms the
// stress sums and U's way back.  Elsewhere the passes are separate.
//
// Every launch and descriptor is fixed at creation; reductions use a fixed
// grid and are summed on the host in a fixed order, so results are
// deterministic.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <functional>
#include <string>
#include <vector>

#include "adjoint.cuh"
#include "engine_state.h"

namespace psb {

constexpr int kAdjRB = 296;
constexpr int kAdjRT = 256;

struct AccumEntry {
  double* dst;
  const double* x;
  const double* y;
  double coef;
};

// lam_out[j] += lam0 * prod_{i != j} q_in[i] for the sweeps arriving at a
// junction (the adjoint of the junction product).
struct JunctionAdj {
  const double* lam0;
  int n;
  const double* q_in[PS_MAX_JOINS];
  double* lam_out[PS_MAX_JOINS];
};

struct BlockFieldMap {
  int nb, nf;
  int field[PS_MAX_BLOCKS];
};

__device__ __forceinline__ double adj_block_sum(double v, double* sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = kAdjRT / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  const double r = sh[0];
  __syncthreads();
  return r;
}

#define ADJ_LOOP(r, N) \
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < (N); r += (long long)gridDim.x * blockDim.x)

// dst += coef x y over the entries.  A block's entries follow one another, so that its
// sum stays in a register (read and written back for every entry it was 29 us for the
// 13 slice pairs of a 64^3 segment).
__global__ void adj_accum_kernel(const AccumEntry* __restrict__ e, int ne, long long N) {
  ADJ_LOOP(r, N) {
    double* dst = e[0].dst;
    double acc = dst[r];
#pragma unroll 4
    for (int i = 0; i < ne; ++i) {
      const AccumEntry a = e[i];
      if (a.dst != dst) {  // the next block
        dst[r] = acc;
        dst = a.dst;
        acc = dst[r];
      }
      acc += a.coef * __ldg(a.x + r) * __ldg(a.y + r);
    }
    dst[r] = acc;
  }
}

__global__ void adj_normalize_kernel(double* __restrict__ P, double* __restrict__ phi, BlockFieldMap m,
                                     long long N, const DevScalars* __restrict__ sc) {
  const double inv_q = 1.0 / sc->q[0];
  ADJ_LOOP(r, N) {
    double acc[PS_MAX_FIELDS] = {0.0, 0.0, 0.0, 0.0};
    for (int b = 0; b < m.nb; ++b) {
      const double v = P[(size_t)b * N + r] * inv_q;
      P[(size_t)b * N + r] = v;
      acc[m.field[b]] += v;
    }
    for (int f = 0; f < m.nf; ++f) phi[(size_t)f * N + r] = acc[f];
  }
}

__global__ void adj_dot_kernel(const double* __restrict__ a, const double* __restrict__ b, long long n,
                               double* __restrict__ part) {
  __shared__ double sh[kAdjRT];
  double acc = 0.0;
  ADJ_LOOP(r, n) acc += a[r] * b[r];
  acc = adj_block_sum(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// sum (w + facz psi) g
__global__ void adj_dotw_kernel(const double* __restrict__ w, const double* __restrict__ psi, double facz,
                                const double* __restrict__ g, long long n, double* __restrict__ part) {
  __shared__ double sh[kAdjRT];
  double acc = 0.0;
  ADJ_LOOP(r, n) acc += (psi ? w[r] + facz * psi[r] : w[r]) * g[r];
  acc = adj_block_sum(acc, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// dL/dQ = g_lnQ / Q - (1/Q) sum_f <g_phi_f, phi_f>  (phi carries 1/Q).
__global__ void adj_gq_kernel(const double* __restrict__ part, double g_lnq, const DevScalars* __restrict__ sc,
                              double* __restrict__ gq) {
  __shared__ double sh[kAdjRT];
  double acc = 0.0;
  for (int i = threadIdx.x; i < kAdjRB; i += blockDim.x) acc += part[i];
  acc = adj_block_sum(acc, sh);
  if (threadIdx.x == 0) {
    const double q = sc->q[0];
    *gq = g_lnq / q - acc / q;
  }
}

// out[row] = the sum of row's `stride` partials, in a fixed order.
__global__ void adj_rows_kernel(const double* __restrict__ part, int stride, double* __restrict__ out) {
  __shared__ double sh[kAdjRT];
  double acc = 0.0;
  for (int i = threadIdx.x; i < stride; i += blockDim.x) acc += part[(size_t)blockIdx.x * stride + i];
  acc = adj_block_sum(acc, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = acc;
}

__global__ void adj_kmul_kernel(double2* __restrict__ spec, const double* __restrict__ kx,
                                const double* __restrict__ kyz, int nx, int inner) {
  const long long n = (long long)nx * inner;
  ADJ_LOOP(i, n) {
    const int x = (int)(i / inner);
    const int c = (int)(i - (long long)x * inner);
    const double f = kx[x] * kyz[c];
    const double2 v = spec[i];
    spec[i] = make_double2(v.x * f, v.y * f);
  }
}

__device__ __forceinline__ double adj_kcomp(int i, int n, double dx) {
  const double n2 = (double)n / 2.0;
  const double nk = n2 - fabs((double)i - n2);
  return 2.0 * 3.14159265358979323846 * nk / ((double)n * dx);
}

// R_d = sum over the half spectrum (weight 2 off the kz = 0 / nz/2 planes) of
// Re(conj(U) V) * kx*kyz * k_d^2; kx carries 1/N.
__global__ void adj_stress_kernel(const double2* __restrict__ U, const double2* __restrict__ V,
                                  const double* __restrict__ kx, const double* __restrict__ kyz, int nx,
                                  int ny, int nz, double dx, double dy, double dz, int stride,
                                  double* __restrict__ part) {
  __shared__ double sh[kAdjRT];
  const int nzh = nz / 2 + 1;
  const long long n = (long long)nx * ny * nzh;
  double a0 = 0.0, a1 = 0.0, a2 = 0.0;
  ADJ_LOOP(i, n) {
    const int x = (int)(i / ((long long)ny * nzh));
    const int rem = (int)(i - (long long)x * ny * nzh);
    const int y = rem / nzh;
    const int kz = rem - y * nzh;
    const double mult = (kz == 0 || (2 * kz == nz)) ? 1.0 : 2.0;
    const double2 u = U[i], v = V[i];
    const double t = mult * (u.x * v.x + u.y * v.y) * kx[x] * kyz[rem];
    const double k0 = adj_kcomp(x, nx, dx), k1 = adj_kcomp(y, ny, dy), k2 = adj_kcomp(kz, nz, dz);
    a0 += t * k0 * k0;
    a1 += t * k1 * k1;
    a2 += t * k2 * k2;
  }
  a0 = adj_block_sum(a0, sh);
  a1 = adj_block_sum(a1, sh);
  a2 = adj_block_sum(a2, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = a0;
    part[stride + blockIdx.x] = a1;
    part[2 * stride + blockIdx.x] = a2;
  }
}

__global__ void adj_init_kernel(const AdjPoint* __restrict__ pp, long long N, const DevScalars* __restrict__ sc,
                                const double* __restrict__ gq) {
  const AdjPoint p = *pp;
  const double inv_q = 1.0 / sc->q[0];
  const double gqn = p.q_partner ? (*gq) / (double)N : 0.0;
  ADJ_LOOP(r, N) {
    double s = 0.0;
    for (int i = 0; i < p.n_src; ++i) s += p.src[i].coef * p.src[i].gphi[r] * p.src[i].partner[r];
    double l = inv_q * s;
    if (p.q_partner) l += gqn * p.q_partner[r];
    if (p.extra) l += p.extra[r];
    p.lam_out[r] = l;
  }
}

__global__ void adj_axpy_kernel(double* __restrict__ dst, const double* __restrict__ x, double coef, long long N) {
  ADJ_LOOP(r, N) dst[r] += coef * x[r];
}

__global__ void adj_junction_kernel(const JunctionAdj* __restrict__ jp, long long N) {
  const JunctionAdj j = *jp;
  ADJ_LOOP(r, N) {
    const double l = j.lam0[r];
    for (int i = 0; i < j.n; ++i) {
      double v = l;
      for (int k = 0; k < j.n; ++k)
        if (k != i) v *= j.q_in[k][r];
      j.lam_out[i][r] += v;
    }
  }
}

__global__ void adj_point_kernel(const AdjPoint* __restrict__ pp, long long N, const DevScalars* __restrict__ sc,
                                 const double* __restrict__ gq) {
  __shared__ double sh[kAdjRT];
  const AdjPoint p = *pp;
  const double inv_q = 1.0 / sc->q[0];
  const double gqn = p.q_partner ? (*gq) / (double)N : 0.0;
  double acc = 0.0;
  ADJ_LOOP(r, N) {
    const double t = p.lam_next[r] * p.q_next[r] + p.q_s[r] * p.mu[r];
    p.gwb[r] += -p.half_ds * t;
    const double x = p.psi ? p.w[r] + p.facz * p.psi[r] : p.w[r];
    acc += x * (-0.5 * t);
    if (p.lam_out) {
      double s = 0.0;
      for (int i = 0; i < p.n_src; ++i) s += p.src[i].coef * p.src[i].gphi[r] * p.src[i].partner[r];
      double l = p.mu[r] + inv_q * s;
      if (p.q_partner) l += gqn * p.q_partner[r];
      p.lam_out[r] = l;
    }
  }
  acc = adj_block_sum(acc, sh);
  if (threadIdx.x == 0) p.dsw_part[blockIdx.x] = acc;
}

__global__ void adj_sum_blocks_kernel(const double* __restrict__ gwb, BlockFieldMap m, long long N,
                                      double* __restrict__ gw) {
  ADJ_LOOP(r, N) {
    double acc[PS_MAX_FIELDS] = {0.0, 0.0, 0.0, 0.0};
    for (int b = 0; b < m.nb; ++b) acc[m.field[b]] += gwb[(size_t)b * N + r];
    for (int f = 0; f < m.nf; ++f) gw[(size_t)f * N + r] = acc[f];
  }
}

// Quadrature weight of local slice n of a block with `steps` steps, without ds
// (PsBlock::setCalcQQTIntegral: extended Simpson with 0.33333, trapezoid on the
// last interval when the point count is even).
static std::vector<double> quad_weights(int steps) {
  const int num = steps + 1;
  const int npts = num - 1;
  const bool even = (num % 2) == 0;
  const int numstail = even ? npts - 3 : npts - 2;
  std::vector<double> c(num, 0.0);
  for (int n = 0; n <= numstail; n += 2) {
    c[n] += 0.33333;
    c[n + 1] += 4.0 * 0.33333;
    c[n + 2] += 0.33333;
  }
  if (even) {
    c[num - 2] += 0.5;
    c[num - 1] += 0.5;
  }
  return c;
}

}  // namespace psb

using Op = std::function<cudaError_t(cudaStream_t)>;

struct ps_adj {
  ps_handle* h = nullptr;
  std::string err;
  int ip = 0;  // the polymer of the configuration this adjoint differentiates
  int M = 0, C = 1, J = 0, nb = 0, nf = 0;
  long long N = 0;
  int n0 = 0;  // sweep-0 index of block 0's head slice (Q = <q_n0 q+_{M-n0}>)
  std::vector<int> blk[2];
  std::vector<int> seg_a, seg_b;
  std::vector<std::vector<std::pair<int, double>>> quad;  // per n: (block, densfac ds c)
  double* ck[2] = {nullptr, nullptr};
  double* endq[2] = {nullptr, nullptr};
  double* seg[2][2] = {};       // [set][sweep]: slices 1 .. C of a recomputed segment
  double* lam[4] = {};          // two of each adjoint lane
  double* mu = nullptr;
  double2* spec[4] = {};   // U and V of the adjoint steps of each lane
  double2* rspec[4] = {};  // the recomputed sweeps' (U stays across segments)
  bool pair = false;       // the adjoints of both sweeps run in the same launches (two lanes)
  double* P = nullptr;
  double* gwb = nullptr;
  double* gphi = nullptr;
  double* gq = nullptr;
  // rows of `stride` partials: four per adjoint step (stress x, y, z, explicit ds),
  // two per block (E, and w . dL/dw of the fused steps), one for <g_phi, phi>; summed by rows into d_sum, read to h_sum
  double* part = nullptr;
  double* d_sum = nullptr;
  double* h_sum = nullptr;
  int stride = 0;
  size_t rows = 0;
  std::vector<int> slot_block;
  psb::SweepWork<double>* d_sw = nullptr;  // one-launch sweeps
  double** d_dst = nullptr;                // their slices' places
  std::vector<psb::SweepWork<double>> h_sw;
  std::vector<double*> h_dst;
  std::vector<size_t> sw_dst;              // by work: its part of h_dst
  psb::AdjXWork* d_ax = nullptr;
  std::vector<psb::AdjXWork> h_ax;
  psb::PlaneWork<double>* d_pw = nullptr;
  psb::PencilWork<double>* d_xw = nullptr;
  psb::AccumEntry* d_acc = nullptr;
  psb::AdjPoint* d_pt = nullptr;
  std::vector<psb::PlaneWork<double>> h_pw;
  std::vector<psb::PencilWork<double>> h_xw;
  std::vector<psb::AccumEntry> h_acc;
  std::vector<psb::AdjPoint> h_pt;
  std::vector<Op> fwd, bwd;
  // branched chains: the polymer's executed sweeps (h->sweeps indices, in
  // dependency order), the steps' blocks, junction accumulators, descriptors
  bool tree = false;
  std::vector<int> tsw;
  std::vector<std::vector<int>> tblk;
  std::vector<double*> jacc;
  std::vector<psb::JunctionAdj> h_jn;
  psb::JunctionAdj* d_jn = nullptr;
  size_t storage_bytes = 0;
  size_t E_row = 0, W_row = 0, gq_row = 0;  // rows of part
  double* row(size_t r) const { return part + r * (size_t)stride; }
  bool have_forward = false;
  bool have_backward = false;
};

namespace psb {

#define PA_CUDA(a, call)                                                 \
  do {                                                                   \
    cudaError_t e_ = (call);                                             \
    if (e_ != cudaSuccess) {                                             \
      (a)->err = std::string(#call) + ": " + cudaGetErrorString(e_);     \
      return PS_GPU_ERR;                                                 \
    }                                                                    \
  } while (0)

static thread_local std::string g_adj_err;

// Program builder: descriptors go to host tables (uploaded once), ops refer to
// them by offset.
struct Builder {
  ps_adj* a;
  ps_handle* h;
  int nx, ny, nz, nzh;
  bool fused;
  bool step;  // the sweeps run the step plane pass and the register x pass (compact layout)
  bool adj;   // ... and the adjoint steps their fused forms
  bool one;   // a sweep is one launch (sweep_cluster.cuh)
  Builder(ps_adj* a_, ps_handle* h_) : a(a_), h(h_), nx(h_->n[0]), ny(h_->n[1]), nz(h_->n[2]), nzh(h_->nzh) {
    fused = plane_fused_supported(8, ny, nz);
    step = step_plane_supported(ny, nz);
    adj = adj_step_supported(ny, nz);
    one = sweep_cluster_to_fits(nx, ny, nz);
  }

  const double* wf(int b) const {
    const BlockMap& bm = h->blocks[a->ip][b];
    for (size_t i = 0; i < h->wfac_keys.size(); ++i) {
      const WfacKey& k = h->wfac_keys[i];
      if (k.field == bm.field && k.ds == bm.ds && k.charge_field == bm.charge_field &&
          (bm.charge_field < 0 || k.facz == bm.facz))
        return h->bd.wfac[i];
    }
    return nullptr;
  }
  int ktab(int b) const {
    const BlockMap& bm = h->blocks[a->ip][b];
    for (size_t i = 0; i < h->ktab_keys.size(); ++i)
      if (h->ktab_keys[i].first == bm.ds && h->ktab_keys[i].second == bm.bseg) return (int)i;
    return 0;
  }
  size_t plane(const PlaneWork<double>& w) {
    a->h_pw.push_back(w);
    return a->h_pw.size() - 1;
  }
  size_t pencil(const PencilWork<double>& w) {
    a->h_xw.push_back(w);
    return a->h_xw.size() - 1;
  }
  PlaneWork<double> pw(int mode, const double* src, double2* spec, const double* win, const double* wout,
                       double* store) {
    PlaneWork<double> w;
    memset(&w, 0, sizeof(w));
    w.mode = mode;
    w.src = src;
    w.spec = spec;
    w.wfac_in = win;
    w.wfac_out = wout;
    w.store = store;
    w.status = &h->d_sc->error_flags;
    return w;
  }
  PencilWork<double> xw(double2* spec, int b) {
    PencilWork<double> x;
    memset(&x, 0, sizeof(x));
    x.spec = spec;
    if (b >= 0) {
      x.kx = h->bd.kx[ktab(b)];
      x.kyz = h->bd.kyz[ktab(b)];
      x.kyzc = h->bd.kyzc[ktab(b)];
    }
    return x;
  }
  // Real-space plane pass (rows + y pencils on grids without the fused design):
  // MODE_FIRST / MID end with the forward y-z transform; MID / LAST start with
  // the inverse one.
  void real_pass(std::vector<Op>& ops, size_t pw0, int n, size_t yx0, int mode) {
    ps_adj* A = a;
    const int nx_ = nx, ny_ = ny, nz_ = nz, nzh_ = nzh;
    ps_handle* H = h;
    if (fused) {
      ops.push_back([=](cudaStream_t st) {
        return launch_plane<double>(A->d_pw + pw0, n, nx_, ny_, nz_, H->bd.tw_y, H->bd.tw_zh, H->bd.tw_z, st);
      });
      return;
    }
    if (mode != MODE_FIRST && ny > 1)
      ops.push_back([=](cudaStream_t st) {
        return launch_pencil<double>(A->d_xw + yx0, n, PENCIL_INV, ny_, nx_, nzh_, H->bd.tw_y, nx_, ny_, nz_, st);
      });
    ops.push_back([=](cudaStream_t st) {
      return launch_rows<double>(A->d_pw + pw0, n, nx_ * ny_, nz_, H->bd.tw_zh, H->bd.tw_z, st);
    });
    if (mode != MODE_LAST && ny > 1)
      ops.push_back([=](cudaStream_t st) {
        return launch_pencil<double>(A->d_xw + yx0, n, PENCIL_FWD, ny_, nx_, nzh_, H->bd.tw_y, nx_, ny_, nz_, st);
      });
  }
  void x_pass(std::vector<Op>& ops, size_t x0, int n, int mode) {
    ps_adj* A = a;
    const int nx_ = nx, ny_ = ny, nz_ = nz, inner = ny * nzh;
    ps_handle* H = h;
    ops.push_back([=](cudaStream_t st) {
      return launch_pencil<double>(A->d_xw + x0, n, mode, nx_, 1, inner, H->bd.tw_x, nx_, ny_, nz_, st);
    });
  }
  void step_pass(std::vector<Op>& ops, size_t p0, int n) {
    ps_adj* A = a;
    ps_handle* H = h;
    const int nx_ = nx, ny_ = ny, nz_ = nz;
    ops.push_back([=](cudaStream_t st) {
      return launch_step_plane<double>(A->d_pw + p0, n, nx_, ny_, nz_, false, H->bd.tw_y, H->bd.tw_z, st);
    });
  }
  // Fused adjoint steps: the plane pass of lambda works in adjoint modes (with their
  // points) and, beside them, starts of FFT(wf q) for the next steps; the x pass of
  // steps of the given blocks (stress sums of the slot, U <- IFFT(K U)).
  struct LamWork {
    int mode, lane;
    AdjPoint p;
    const double *win, *wout;
  };
  struct QWork {
    int lane;
    const double *q, *wq;
  };
  struct XWork {
    int lane, block, slot;
  };
  void lambda_pass(std::vector<Op>& ops, const std::vector<LamWork>& lam, const std::vector<QWork>& qs) {
    const size_t p0 = a->h_pw.size(), pi = a->h_pt.size();
    const int n = (int)(lam.size() + qs.size());
    for (const LamWork& l : lam) {
      plane(pw(l.mode, nullptr, a->spec[2 * l.lane], l.win, l.wout, nullptr));
      a->h_pt.push_back(l.p);
    }
    for (const QWork& q : qs) plane(pw(MODE_FIRST, q.q, a->spec[2 * q.lane + 1], nullptr, q.wq, nullptr));
    if (lam.empty()) {
      step_pass(ops, p0, n);
      return;
    }
    ps_adj* A = a;
    ps_handle* H = h;
    const int nx_ = nx, ny_ = ny;
    ops.push_back([=](cudaStream_t st) {
      const AdjArgs args{A->d_pt + pi, &H->d_sc->q[0], A->gq, (double)A->N};
      return launch_step_plane_adj(A->d_pw + p0, n, nx_, ny_, H->bd.tw_y, H->bd.tw_z, args, st);
    });
  }
  void stress_x(std::vector<Op>& ops, const std::vector<XWork>& xs) {
    const size_t xi = a->h_ax.size();
    for (const XWork& w : xs) {
      AdjXWork x;
      x.u = a->spec[2 * w.lane];
      x.v = a->spec[2 * w.lane + 1];
      x.kx = h->bd.kx[ktab(w.block)];
      x.kyzc = h->bd.kyzc[ktab(w.block)];
      x.part = a->row((size_t)w.slot * 4);
      a->h_ax.push_back(x);
    }
    ps_adj* A = a;
    ps_handle* H = h;
    const int nx_ = nx, ny_ = ny, nz_ = nz, n = (int)xs.size();
    ops.push_back([=](cudaStream_t st) {
      return launch_adj_x(A->d_ax + xi, n, nx_, ny_, nz_, H->cfg.cell[0], H->cfg.cell[1], H->cfg.cell[2], A->stride,
                          H->bd.tw_x, st);
    });
  }
  // Every run in one launch.
  struct Run;
  bool one_launch(std::vector<Op>& ops, const std::vector<Run>& runs);

  // Lockstep sweeps.  Sweep i runs steps s0 .. s0 + len - 1 of sweep sig from slice
  // src (nullptr: ones); store(k) gives the destination of its slice k (nullptr: not
  // stored).
  struct Run {
    int sig, s0, len;
    const double* src;
    std::function<double*(int)> store;
  };
  void sweeps(std::vector<Op>& ops, const std::vector<Run>& runs) {
    if (one && one_launch(ops, runs)) return;
    int top = 0;
    for (const Run& r : runs) top = std::max(top, r.len);
    for (int k = 0; k <= top; ++k) {
      const size_t p0 = a->h_pw.size(), y0 = a->h_xw.size();
      int n = 0;
      int mode = MODE_MID;  // of the separate passes, whose runs have one length
      for (size_t i = 0; i < runs.size(); ++i) {
        const Run& r = runs[i];
        if (k > r.len) continue;
        const std::vector<int>& bl = a->blk[r.sig];
        mode = (k == 0) ? MODE_FIRST : (k == r.len ? MODE_LAST : MODE_MID);
        const double* win = (k > 0) ? wf(bl[r.s0 + k - 1]) : nullptr;
        const double* wout = (k < r.len) ? wf(bl[r.s0 + k]) : nullptr;
        plane(pw(mode, k == 0 ? r.src : nullptr, a->rspec[i], win, wout, r.store(k)));
        pencil(xw(a->rspec[i], -1));
        ++n;
      }
      if (step) step_pass(ops, p0, n);
      else real_pass(ops, p0, n, y0, mode);
      const size_t x0 = a->h_xw.size();
      int nx_works = 0;
      for (size_t i = 0; i < runs.size(); ++i)
        if (k < runs[i].len) {
          pencil(xw(a->rspec[i], a->blk[runs[i].sig][runs[i].s0 + k]));
          ++nx_works;
        }
      if (nx_works == 0) continue;
      if (step) {
        ps_adj* A = a;
        ps_handle* H = h;
        const int nx_ = nx, inner = ny * nzh;
        // The plane pass behind it starts early (early_path in sweeps.cuh).  Forward and
        // backward of 100 steps, ms, without and with: 16 x 24^2 2.78 -> 2.64, 48^3 4.10 -> 3.99,
        // 64 x 48^2 4.64 -> 4.47, 64^3 5.74 -> 5.59, 64 x 96 x 48 15.27 -> 15.05, 96^3 18.08 ->
        // 17.87; of 14 grids and two checkpoint intervals in this range one lost 2%
        // (32 x 48^2 3.48 -> 3.56, at full storage 2.34 -> 2.28), the others 0 to 6% less.
        const bool early = nx <= 96 && a->N <= 96LL * 96 * 96;
        ops.push_back([=](cudaStream_t st) {
          return launch_step_pencil<double>(A->d_xw + x0, nx_works, nx_, inner, true, early, H->bd.tw_x, st);
        });
      } else {
        x_pass(ops, x0, nx_works, PENCIL_KINV);
      }
    }
  }
};

bool Builder::one_launch(std::vector<Op>& ops, const std::vector<Run>& runs) {
  std::vector<SweepWork<double>> ws;
  for (const Run& r : runs) {
    SweepWork<double> w;
    memset(&w, 0, sizeof(w));
    w.src = r.src;
    w.status = &h->d_sc->error_flags;
    w.total = r.len;
    const std::vector<int>& bl = a->blk[r.sig];
    int g = 0;
    for (int k = 0; k < r.len; ++k) {
      const int b = bl[r.s0 + k];
      if (k > 0 && b != bl[r.s0 + k - 1] && ++g == kSweepSegs) return false;
      w.seg[g].wfac = wf(b);
      w.seg[g].kx = h->bd.kx[ktab(b)];
      w.seg[g].kyzc = h->bd.kyzc[ktab(b)];
      w.seg[g].end = k + 1;
    }
    ws.push_back(w);
  }
  const size_t w0 = a->h_sw.size();
  const int n = (int)ws.size();
  for (int i = 0; i < n; ++i) {
    a->sw_dst.push_back(a->h_dst.size());
    a->h_sw.push_back(ws[i]);
    for (int k = 0; k <= runs[i].len; ++k) a->h_dst.push_back(runs[i].store(k));
  }
  ps_adj* A = a;
  ps_handle* H = h;
  const int nx_ = nx, ny_ = ny, nz_ = nz;
  ops.push_back([=](cudaStream_t st) {
    return launch_sweep_cluster_to(A->d_sw + w0, n, nx_, ny_, nz_, H->bd.tw_x, H->bd.tw_y, H->bd.tw_z, st);
  });
  return true;
}

// Slice idx of sweep sig while segment j is resident in buffer set `set` (its first
// slice is the checkpoint).
static double* slice_ptr(ps_adj* a, int sig, int idx, int j, int set) {
  const long long N = a->N;
  if (a->C == 1) {
    if (idx == a->M) return a->endq[sig];
    return a->ck[sig] + (size_t)(sig == 0 ? idx : a->M - 1 - idx) * N;
  }
  const int at = idx - (sig == 0 ? a->seg_a[j] : a->M - a->seg_b[j]);
  return at == 0 ? a->ck[sig] + (size_t)j * N : a->seg[set][sig] + (size_t)(at - 1) * N;
}

// Segment js[set] of both sweeps into buffer set `set`, for n sets.
static void recompute(Builder& B, std::vector<Op>& ops, const int* js, int n) {
  ps_adj* a = B.a;
  if (a->C == 1) return;
  std::vector<Builder::Run> runs;
  for (int set = 0; set < n; ++set)
    for (int sig = 0; sig < 2; ++sig) {
      const int j = js[set];
      double* const to = a->seg[set][sig];
      const long long N = a->N;
      runs.push_back({sig, sig == 0 ? a->seg_a[j] : a->M - a->seg_b[j], a->seg_b[j] - a->seg_a[j],
                      a->ck[sig] + (size_t)j * N,
                      [to, N](int k) { return k == 0 ? nullptr : to + (size_t)(k - 1) * N; }});
    }
  B.sweeps(ops, runs);
}

// Sources of slice idx of sweep sig: every quadrature pair it belongs to, and Q.
static void fill_sources(ps_adj* a, AdjPoint& p, int sig, int idx, int j, int set) {
  const int n = (sig == 0) ? idx : a->M - idx;
  p.n_src = 0;
  for (auto& e : a->quad[n]) {
    const int f = a->h->blocks[a->ip][e.first].field;
    SrcEntry s;
    s.gphi = a->gphi + (size_t)f * a->N;
    s.partner = slice_ptr(a, 1 - sig, a->M - idx, j, set);
    s.coef = e.second;
    p.src[p.n_src++] = s;
  }
  const int qslice = (sig == 0) ? a->n0 : a->M - a->n0;
  p.q_partner = (idx == qslice) ? slice_ptr(a, 1 - sig, a->M - idx, j, set) : nullptr;
}

// One adjoint step through block b: mu = wf G(wf lam_next), the stress
// partials of (U, V) = (FFT(wf lam_next), FFT(wf q_s)), dL/dw of the step and,
// when lam_out is set, lam_s = mu + the explicit sources of slice s (in `src`).
static AdjPoint step_point(Builder& B, int b, int slot, const double* q_s, const double* q_next,
                           const double* lam_next, double* lam_out, const AdjPoint& src, int b2 = -1, int lane = 0) {
  ps_adj* a = B.a;
  ps_handle* h = B.h;
  const BlockMap& bm = h->blocks[a->ip][b];
  AdjPoint p = src;
  if (b2 >= 0) {
    p.gwb2 = a->gwb + (size_t)(lane * a->nb + b2) * a->N;
    p.half_ds2 = 0.5 * h->blocks[a->ip][b2].ds;
  }
  p.mu = a->mu;
  p.lam_next = lam_next;
  p.q_s = q_s;
  p.q_next = q_next;
  p.w = h->d_w + (size_t)bm.field * a->N;
  p.gwb = a->gwb + (size_t)(lane * a->nb + b) * a->N;
  p.lam_out = lam_out;
  p.dsw_part = a->row((size_t)slot * 4 + 3);
  p.half_ds = 0.5 * bm.ds;
  p.extra = nullptr;
  p.psi = (bm.charge_field >= 0) ? h->d_psi + (size_t)bm.charge_field * a->N : nullptr;
  p.facz = bm.facz;
  return p;
}

static void adjoint_step_p(Builder& B, std::vector<Op>& ops, int b, const double* q_s, const double* q_next,
                           const double* lam_next, double* lam_out, const AdjPoint& src) {
  ps_adj* a = B.a;
  ps_handle* h = B.h;
  const double* wfb = B.wf(b);
  const int slot = (int)a->slot_block.size();
  a->slot_block.push_back(b);
  // U = FFT(wf lam_{s+1}) in spec[0], V = FFT(wf q_s) in spec[1]
  const size_t p0 = B.plane(B.pw(MODE_FIRST, lam_next, a->spec[0], nullptr, wfb, nullptr));
  B.plane(B.pw(MODE_FIRST, q_s, a->spec[1], nullptr, wfb, nullptr));
  const size_t y0 = B.pencil(B.xw(a->spec[0], -1));
  B.pencil(B.xw(a->spec[1], -1));
  B.real_pass(ops, p0, 2, y0, MODE_FIRST);
  const size_t x0 = B.pencil(B.xw(a->spec[0], -1));
  B.pencil(B.xw(a->spec[1], -1));
  B.x_pass(ops, x0, 2, PENCIL_FWD);
  const int kt = B.ktab(b);
  const int nx = B.nx, ny = B.ny, nz = B.nz;
  const double dx = h->cfg.cell[0], dy = h->cfg.cell[1], dz = h->cfg.cell[2];
  double* const part = a->row((size_t)slot * 4);
  const int stride = a->stride;
  ops.push_back([=](cudaStream_t st) {
    adj_stress_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->spec[0], a->spec[1], h->bd.kx[kt], h->bd.kyz[kt], nx, ny,
                                                   nz, dx, dy, dz, stride, part);
    return cudaGetLastError();
  });
  const int inner = ny * B.nzh;
  ops.push_back([=](cudaStream_t st) {
    adj_kmul_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->spec[0], h->bd.kx[kt], h->bd.kyz[kt], nx, inner);
    return cudaGetLastError();
  });
  const size_t x1 = B.pencil(B.xw(a->spec[0], -1));
  B.x_pass(ops, x1, 1, PENCIL_INV);
  const size_t p1 = B.plane(B.pw(MODE_LAST, nullptr, a->spec[0], wfb, nullptr, a->mu));
  const size_t y1 = B.pencil(B.xw(a->spec[0], -1));
  B.real_pass(ops, p1, 1, y1, MODE_LAST);
  const AdjPoint p = step_point(B, b, slot, q_s, q_next, lam_next, lam_out, src);
  a->h_pt.push_back(p);
  const size_t pi = a->h_pt.size() - 1;
  const long long N = a->N;
  ops.push_back([=](cudaStream_t st) {
    adj_point_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_pt + pi, N, h->d_sc, a->gq);
    return cudaGetLastError();
  });
}

static void adjoint_step(Builder& B, std::vector<Op>& ops, int sig, int s, int j, int cur) {
  ps_adj* a = B.a;
  AdjPoint src;
  memset(&src, 0, sizeof(src));
  if (s >= 1) fill_sources(a, src, sig, s, j, 0);
  adjoint_step_p(B, ops, a->blk[sig][s], slice_ptr(a, sig, s, j, 0), slice_ptr(a, sig, s + 1, j, 0), a->lam[cur],
                 (s >= 1) ? a->lam[1 - cur] : nullptr, src);
}

// The adjoint steps hi - 1 .. lo of sweep sig while segment j is resident in `set`.
struct SegRun {
  int sig, j, set, lo, hi;
  bool first;  // lambda starts here (the sweep's end); at later segments only q's transform is missing
};

// The runs' steps, fused: one plane pass and one x pass a step for all of them.  Run i
// is lane i; cur[i] says which of the lane's two lambda buffers is current.
static void adjoint_segments(Builder& B, std::vector<Op>& ops, const std::vector<SegRun>& runs, int* cur) {
  ps_adj* a = B.a;
  std::vector<Builder::LamWork> lam;
  std::vector<Builder::QWork> qs;
  std::vector<Builder::XWork> xs;
  int top = 0;
  for (size_t i = 0; i < runs.size(); ++i) {
    const SegRun& r = runs[i];
    const int lane = (int)i;
    const int b = a->blk[r.sig][r.hi - 1];
    top = std::max(top, r.hi - r.lo);
    if (r.first) {
      AdjPoint p;
      memset(&p, 0, sizeof(p));
      p.lam_out = a->lam[2 * lane + cur[i]];
      p.q_s = slice_ptr(a, r.sig, r.hi, r.j, r.set);
      p.gwb2 = a->gwb + (size_t)(lane * a->nb + b) * a->N;
      p.half_ds2 = 0.5 * B.h->blocks[a->ip][b].ds;
      fill_sources(a, p, r.sig, r.hi, r.j, r.set);
      lam.push_back({MODE_ADJ_INIT, lane, p, nullptr, B.wf(b)});
    }
    qs.push_back({lane, slice_ptr(a, r.sig, r.hi - 1, r.j, r.set), B.wf(b)});
  }
  B.lambda_pass(ops, lam, qs);
  for (int k = 1; k <= top; ++k) {
    lam.clear();
    qs.clear();
    xs.clear();
    for (size_t i = 0; i < runs.size(); ++i) {
      const SegRun& r = runs[i];
      const int s = r.hi - k, lane = (int)i;
      if (s < r.lo) continue;
      const std::vector<int>& bl = a->blk[r.sig];
      const int slot = r.sig * a->M + (a->M - 1 - s);
      a->slot_block[slot] = bl[s];
      xs.push_back({lane, bl[s], slot});
      AdjPoint src;
      memset(&src, 0, sizeof(src));
      if (s >= 1) fill_sources(a, src, r.sig, s, r.j, r.set);
      double* const* const l = a->lam + 2 * lane;
      const AdjPoint p =
          step_point(B, bl[s], slot, slice_ptr(a, r.sig, s, r.j, r.set), slice_ptr(a, r.sig, s + 1, r.j, r.set),
                     l[cur[i]], (s >= 1) ? l[1 - cur[i]] : nullptr, src, s >= 1 ? bl[s - 1] : -1, lane);
      const double* wn = (s >= 1) ? B.wf(bl[s - 1]) : nullptr;
      lam.push_back({s >= 1 ? MODE_ADJ_MID : MODE_ADJ_LAST, lane, p, B.wf(bl[s]), wn});
      if (s > r.lo) qs.push_back({lane, slice_ptr(a, r.sig, s - 1, r.j, r.set), wn});
      cur[i] = 1 - cur[i];
    }
    B.stress_x(ops, xs);
    B.lambda_pass(ops, lam, qs);
  }
}

static void adjoint_init(ps_adj* a, std::vector<Op>& ops, int sig, int j, int cur) {
  AdjPoint p;
  memset(&p, 0, sizeof(p));
  p.lam_out = a->lam[cur];
  fill_sources(a, p, sig, a->M, j, 0);
  a->h_pt.push_back(p);
  const size_t pi = a->h_pt.size() - 1;
  const long long N = a->N;
  ps_handle* h = a->h;
  ops.push_back([=](cudaStream_t st) {
    adj_init_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_pt + pi, N, h->d_sc, a->gq);
    return cudaGetLastError();
  });
}

template <typename T>
static int adj_upload(ps_adj* a, T** dst, const std::vector<T>& v) {
  PA_CUDA(a, cudaMalloc((void**)dst, sizeof(T) * std::max<size_t>(v.size(), 1)));
  if (!v.empty()) PA_CUDA(a, cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return PS_OK;
}

static BlockFieldMap field_map(ps_adj* a) {
  BlockFieldMap fm;
  memset(&fm, 0, sizeof(fm));
  fm.nb = a->nb;
  fm.nf = a->nf;
  for (int b = 0; b < a->nb; ++b) fm.field[b] = a->h->blocks[a->ip][b].field;
  return fm;
}


static void push_dotw(Builder& B, std::vector<Op>& ops) {
  if (!B.adj) return;
  ps_adj* a = B.a;
  ps_handle* h = B.h;
  const long long N = a->N;
  for (int b = 0; b < a->nb; ++b) {
    const BlockMap& bm = h->blocks[a->ip][b];
    const double* w = h->d_w + (size_t)bm.field * N;
    const double* psi = (bm.charge_field >= 0) ? h->d_psi + (size_t)bm.charge_field * N : nullptr;
    const double facz = bm.facz;
    ops.push_back([=](cudaStream_t st) {
      adj_dotw_kernel<<<kAdjRB, kAdjRT, 0, st>>>(w, psi, facz, a->gwb + (size_t)b * N, N, a->row(a->W_row + b));
      return cudaGetLastError();
    });
  }
}

// Partials of `steps` adjoint steps.
static int alloc_partials(ps_adj* a, size_t steps) {
  ps_handle* h = a->h;
  a->stride = std::max(std::max(kAdjRB, h->n[0]), adj_x_tiles(h->n[0], h->n[1] * h->nzh));
  a->E_row = steps * 4;
  a->W_row = a->E_row + (size_t)a->nb;
  a->gq_row = a->W_row + (size_t)a->nb;
  a->rows = a->gq_row + 1;
  const size_t n = a->rows * (size_t)a->stride;
  PA_CUDA(a, cudaMalloc((void**)&a->part, sizeof(double) * n));
  PA_CUDA(a, cudaMemset(a->part, 0, sizeof(double) * n));
  PA_CUDA(a, cudaMalloc((void**)&a->d_sum, sizeof(double) * a->rows));
  PA_CUDA(a, cudaMallocHost((void**)&a->h_sum, sizeof(double) * a->rows));
  return PS_OK;
}

// Branched chain (see the header): every slice stored by the engine's sweeps.
static int tree_build(ps_adj* a, int ec) {
  ps_handle* h = a->h;
  const int ip = ec;  // the engine's (expanded) polymer index
  a->tree = true;
  a->C = 1;
  a->J = 0;
  a->N = h->N;
  a->nf = h->nf;
  a->nb = (int)h->blocks[ip].size();
  const long long N = a->N;
  std::vector<int> pos(h->sweeps.size(), -1);  // h->sweeps index -> position in tsw
  for (int e : h->exec)
    if (h->sweeps[e].polymer == ip) {
      pos[e] = (int)a->tsw.size();
      a->tsw.push_back(e);
    }
  const int ns = (int)a->tsw.size();
  auto S = [h](int sweep, int idx) -> double* {
    return h->bd.slices[h->sweeps[sweep].storage] + (size_t)idx * h->N;
  };
  int steps_total = 0;
  size_t slice_count = 0;
  a->tblk.resize(ns);
  for (int t = 0; t < ns; ++t) {
    const Sweep& sw = h->sweeps[a->tsw[t]];
    a->tblk[t].assign(sw.total, 0);
    for (const Seg& g : sw.segs)
      for (int k = 0; k < g.steps; ++k) a->tblk[t][g.off + k] = g.block;
    steps_total += sw.total;
    slice_count += (size_t)sw.total + 1;
  }
  a->M = 0;
  for (int b = 0; b < a->nb; ++b) a->M += h->blocks[ip][b].steps;
  // explicit sources per (sweep position, slice): quadrature pairs and Q
  struct Src {
    int block;
    double coef;
    int psweep, pidx;
  };
  std::vector<std::vector<std::vector<Src>>> src(ns);
  for (int t = 0; t < ns; ++t) src[t].resize(h->sweeps[a->tsw[t]].total + 1);
  const double densfac = h->chain_dwt[ip] * h->chain_vf[ip] / h->alpha[ip];
  for (int b = 0; b < a->nb; ++b) {
    const BlockMap& bm = h->blocks[ip][b];
    const std::vector<double> c = quad_weights(bm.steps);
    for (int n = 0; n <= bm.steps; ++n) {
      const double coef = densfac * bm.ds * c[n];
      const int hi = bm.off_head + n, ti = bm.off_tail + bm.steps - n;
      src[pos[bm.sweep_head]][hi].push_back({b, coef, bm.sweep_tail, ti});
      src[pos[bm.sweep_tail]][ti].push_back({b, coef, bm.sweep_head, hi});
      AccumEntry ae;
      ae.dst = a->P + (size_t)b * N;
      ae.x = S(bm.sweep_head, hi);
      ae.y = S(bm.sweep_tail, ti);
      ae.coef = coef;
      a->h_acc.push_back(ae);
    }
  }
  for (auto& v : src)
    for (auto& e : v)
      if (e.size() > 2) {
        a->err = "more than two quadrature pairs on one contour slice";
        return PS_INPUT_ERR;
      }
  const BlockMap& b0 = h->blocks[ip][0];
  const int qh_sw = b0.sweep_head, qh_i = b0.off_head;
  const int qt_sw = b0.sweep_tail, qt_i = b0.off_tail + b0.steps;
  auto fill = [&](AdjPoint& p, int t, int i) {
    p.n_src = 0;
    for (const Src& e : src[t][i]) {
      SrcEntry se;
      se.gphi = a->gphi + (size_t)h->blocks[ip][e.block].field * N;
      se.partner = S(e.psweep, e.pidx);
      se.coef = e.coef;
      p.src[p.n_src++] = se;
    }
    const int sw = a->tsw[t];
    p.q_partner = (sw == qh_sw && i == qh_i) ? S(qt_sw, qt_i) : (sw == qt_sw && i == qt_i) ? S(qh_sw, qh_i) : nullptr;
  };
  // junction accumulators: one per sweep whose end feeds a junction
  a->jacc.assign(ns, nullptr);
  const size_t NB = sizeof(double) * (size_t)N;
  PA_CUDA(a, cudaSetDevice(h->dev));
  for (int t = 0; t < ns; ++t)
    for (auto& in : h->sweeps[a->tsw[t]].jin) {
      const int u = pos[in.first];
      if (u < 0 || in.second != h->sweeps[in.first].total) {
        a->err = "junction input is not the end of one of this polymer's sweeps";
        return PS_INPUT_ERR;
      }
      if (!a->jacc[u]) PA_CUDA(a, cudaMalloc((void**)&a->jacc[u], NB));
    }
  for (int sg = 0; sg < 2; ++sg) {
    PA_CUDA(a, cudaMalloc((void**)&a->lam[sg], NB));
    PA_CUDA(a, cudaMalloc((void**)&a->spec[sg], sizeof(double2) * (size_t)h->n[0] * h->n[1] * h->nzh));
  }
  a->storage_bytes = NB * slice_count;
  PA_CUDA(a, cudaMalloc((void**)&a->mu, NB));
  PA_CUDA(a, cudaMalloc((void**)&a->gwb, NB * a->nb));
  PA_CUDA(a, cudaMalloc((void**)&a->gphi, NB * a->nf));
  PA_CUDA(a, cudaMemset(a->gphi, 0, NB * a->nf));
  PA_CUDA(a, cudaMalloc((void**)&a->gq, sizeof(double)));
  {
    int rp = alloc_partials(a, (size_t)steps_total);
    if (rp) return rp;
  }
  // a->P was sized before the accumulation entries pointed at it
  Builder B(a, h);
  const BlockFieldMap fm = field_map(a);

  // ---- forward: the engine's sweeps (every slice stored), Q, quadrature
  a->fwd.push_back([h](cudaStream_t) {
    long long nl = 0;
    return engine_sweeps(h, &nl, VARIANT_FUSE_Z | VARIANT_FUSE_K) == PS_OK ? cudaSuccess : cudaErrorLaunchFailure;
  });
  {
    const double* qx = S(qh_sw, qh_i);
    const double* qy = S(qt_sw, qt_i);
    a->fwd.push_back([=](cudaStream_t st) {
      BigQSet<double> set;
      set.n = 1;
      set.a[0] = qx;
      set.b[0] = qy;
      return launch_big_q<double>(set, N, h->d_qpart, h->d_count, h->d_sc, st);
    });
    a->fwd.push_back([=](cudaStream_t st) { return cudaMemsetAsync(a->P, 0, sizeof(double) * N * a->nb, st); });
    const int ne = (int)a->h_acc.size();
    a->fwd.push_back([=](cudaStream_t st) {
      adj_accum_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_acc, ne, N);
      return cudaGetLastError();
    });
    a->fwd.push_back([=](cudaStream_t st) {
      adj_normalize_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->P, h->d_phi, fm, N, h->d_sc);
      return cudaGetLastError();
    });
  }
  // ---- backward (bwd[0]: the <g_phi, phi> reduction, as for linear chains)
  {
    const long long nfN = (long long)a->nf * N;
    a->bwd.push_back([=](cudaStream_t st) {
      adj_dot_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->gphi, h->d_phi, nfN, a->row(a->gq_row));
      return cudaGetLastError();
    });
    for (int b = 0; b < a->nb; ++b) {
      const int f = h->blocks[ip][b].field;
      a->bwd.push_back([=](cudaStream_t st) {
        adj_dot_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->gphi + (size_t)f * N, a->P + (size_t)b * N, N,
                                                  a->row(a->E_row + b));
        return cudaGetLastError();
      });
    }
    a->bwd.push_back([=](cudaStream_t st) { return cudaMemsetAsync(a->gwb, 0, sizeof(double) * N * a->nb, st); });
    for (int t = 0; t < ns; ++t)
      if (a->jacc[t]) {
        double* jb = a->jacc[t];
        a->bwd.push_back([=](cudaStream_t st) { return cudaMemsetAsync(jb, 0, NB, st); });
      }
    for (int t = ns - 1; t >= 0; --t) {
      const int sw = a->tsw[t];
      const Sweep& swp = h->sweeps[sw];
      const int T = swp.total;
      const bool junction = !swp.jin.empty();
      int cur = 0;
      if (B.adj) {
        // fused steps; every slice is stored, so q's transform always goes along
        const std::vector<int>& bl = a->tblk[t];
        AdjPoint p0;
        memset(&p0, 0, sizeof(p0));
        p0.lam_out = a->lam[cur];
        p0.q_s = S(sw, T);
        p0.gwb2 = a->gwb + (size_t)bl[T - 1] * N;
        p0.half_ds2 = 0.5 * h->blocks[ip][bl[T - 1]].ds;
        fill(p0, t, T);
        p0.extra = a->jacc[t];
        B.lambda_pass(a->bwd, {{MODE_ADJ_INIT, 0, p0, nullptr, B.wf(bl[T - 1])}}, {{0, S(sw, T - 1), B.wf(bl[T - 1])}});
        for (int st_ = T - 1; st_ >= 0; --st_) {
          const int slot = (int)a->slot_block.size();
          a->slot_block.push_back(bl[st_]);
          B.stress_x(a->bwd, {{0, bl[st_], slot}});
          AdjPoint src_;
          memset(&src_, 0, sizeof(src_));
          const bool out = (st_ >= 1) || junction;
          if (out) fill(src_, t, st_);
          const AdjPoint p = step_point(B, bl[st_], slot, S(sw, st_), S(sw, st_ + 1), a->lam[cur],
                                        out ? a->lam[1 - cur] : nullptr, src_, st_ >= 1 ? bl[st_ - 1] : -1);
          const double* wn = (st_ >= 1) ? B.wf(bl[st_ - 1]) : nullptr;
          std::vector<Builder::QWork> q;
          if (st_ >= 1) q.push_back({0, S(sw, st_ - 1), wn});
          B.lambda_pass(a->bwd, {{st_ >= 1 ? MODE_ADJ_MID : MODE_ADJ_LAST, 0, p, B.wf(bl[st_]), wn}}, q);
          if (out) cur = 1 - cur;
        }
      } else {
        AdjPoint p;
        memset(&p, 0, sizeof(p));
        p.lam_out = a->lam[cur];
        fill(p, t, T);
        p.extra = a->jacc[t];
        a->h_pt.push_back(p);
        const size_t pi = a->h_pt.size() - 1;
        a->bwd.push_back([=](cudaStream_t st) {
          adj_init_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_pt + pi, N, h->d_sc, a->gq);
          return cudaGetLastError();
        });
      }
      for (int st_ = T - 1; st_ >= 0 && !B.adj; --st_) {
        AdjPoint p;
        memset(&p, 0, sizeof(p));
        const bool out = (st_ >= 1) || junction;
        if (out) fill(p, t, st_);
        adjoint_step_p(B, a->bwd, a->tblk[t][st_], S(sw, st_), S(sw, st_ + 1), a->lam[cur],
                       out ? a->lam[1 - cur] : nullptr, p);
        if (out) cur = 1 - cur;
      }
      if (junction) {
        JunctionAdj jn;
        memset(&jn, 0, sizeof(jn));
        jn.lam0 = a->lam[cur];
        jn.n = (int)swp.jin.size();
        for (int i = 0; i < jn.n; ++i) {
          jn.q_in[i] = S(swp.jin[i].first, swp.jin[i].second);
          jn.lam_out[i] = a->jacc[pos[swp.jin[i].first]];
        }
        a->h_jn.push_back(jn);
        const size_t ji = a->h_jn.size() - 1;
        a->bwd.push_back([=](cudaStream_t st) {
          adj_junction_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_jn + ji, N);
          return cudaGetLastError();
        });
      }
    }
  }
  push_dotw(B, a->bwd);
  int r2 = adj_upload(a, &a->d_pw, a->h_pw);
  if (!r2) r2 = adj_upload(a, &a->d_xw, a->h_xw);
  if (!r2) r2 = adj_upload(a, &a->d_acc, a->h_acc);
  if (!r2) r2 = adj_upload(a, &a->d_pt, a->h_pt);
  if (!r2) r2 = adj_upload(a, &a->d_ax, a->h_ax);
  if (!r2) r2 = adj_upload(a, &a->d_jn, a->h_jn);
  return r2;
}

// polymer: the caller's polymer of cfg to differentiate (its phi contribution
// and ln Q), chain: its quadrature chain (0 unless polyDisperseBCP); single:
// the configuration must be a one-polymer melt (ps_adj_create).
static int adj_build(ps_adj* a, const ps_config* cfg, int polymer, int chain, bool single, int checkpoint) {
  if (cfg->precision != PS_PREC_FP64) {
    a->err = "the adjoint runs in FP64 (precision must be PS_PREC_FP64)";
    return PS_ATTRIB_ERR;
  }
  if (polymer < 0 || polymer >= cfg->n_polymers) {
    a->err = "polymer index out of range";
    return PS_ATTRIB_ERR;
  }
  if (single && (cfg->n_polymers != 1 || cfg->n_solvents != 0)) {
    a->err = "ps_adj_create takes one polymer and no solvent (ps_adj_create_polymer takes a blend)";
    return PS_INPUT_ERR;
  }
  a->h = new ps_handle();
  a->h->no_slices = true;
  a->h->no_alias = true;  // mirror-symmetric chains: both sweeps run and are differentiated
  int rc = engine_create(a->h, cfg);
  if (rc) {
    a->err = a->h->err;
    return rc;
  }
  ps_handle* h = a->h;
  if (chain < 0 || chain >= h->user_ng[polymer]) {
    a->err = "chain index out of range (a polyDisperseBCP polymer has n_g chains, any other one)";
    return PS_ATTRIB_ERR;
  }
  const int ec = h->user_first[polymer] + chain;  // the engine's (expanded) polymer index
  a->ip = ec;
  std::vector<int> own;  // this chain's sweeps
  for (int k = 0; k < (int)h->sweeps.size(); ++k)
    if (h->sweeps[k].polymer == ec) own.push_back(k);
  bool linear = (own.size() == 2);
  for (int k : own) linear = linear && h->sweeps[k].jin.empty();
  if (!linear) {
    // a branched chain: rebuild the engine with slice storage
    engine_free(a->h);
    delete a->h;
    a->h = new ps_handle();
    a->h->no_slices = false;
    rc = engine_create(a->h, cfg);
    if (rc) {
      a->err = a->h->err;
      return rc;
    }
    PA_CUDA(a, cudaMalloc((void**)&a->P, sizeof(double) * (size_t)a->h->N * a->h->blocks[ec].size()));
    return tree_build(a, ec);
  }
  const Sweep& s0 = h->sweeps[own[0]];
  const Sweep& s1 = h->sweeps[own[1]];
  if (s0.storage < 0 || s1.storage < 0 || s0.storage == s1.storage) {
    a->err = "the adjoint needs two executed sweeps";
    return PS_INPUT_ERR;
  }
  a->M = s0.total;
  a->N = h->N;
  a->nf = h->nf;
  a->nb = (int)h->blocks[a->ip].size();
  const int M = a->M;
  for (int sg = 0; sg < 2; ++sg) {
    const Sweep& sw = sg ? s1 : s0;
    a->blk[sg].assign(M, 0);
    for (const Seg& g : sw.segs)
      for (int k = 0; k < g.steps; ++k) a->blk[sg][g.off + k] = g.block;
  }
  // quadrature pairs in sweep-0 indexing: (q_n, q+_{M-n})
  a->quad.assign(M + 1, {});
  const double densfac = h->chain_dwt[ec] * h->chain_vf[ec] / h->alpha[ec];
  for (int b = 0; b < a->nb; ++b) {
    const BlockMap& bm = h->blocks[a->ip][b];
    const std::vector<double> c = quad_weights(bm.steps);
    const bool head0 = (h->sweeps[bm.sweep_head].storage == s0.storage);
    const int o = head0 ? bm.off_head : M - bm.off_head - bm.steps;  // block start in sweep 0
    for (int n = o; n <= o + bm.steps; ++n) {
      const int loc = head0 ? n - o : o + bm.steps - n;
      a->quad[n].push_back({b, densfac * bm.ds * c[loc]});
    }
  }
  for (auto& v : a->quad)
    if (v.size() > 2) {
      a->err = "more than two quadrature pairs on one contour slice";
      return PS_INPUT_ERR;
    }
  {
    const BlockMap& b0 = h->blocks[a->ip][0];
    const bool head0 = (h->sweeps[b0.sweep_head].storage == s0.storage);
    a->n0 = head0 ? b0.off_head : M - b0.off_head;
    if (a->n0 != 0 && a->n0 != M) {
      a->err = "the adjoint needs block 0 to start at a free chain end";
      return PS_INPUT_ERR;
    }
  }
  // checkpoints
  int C = checkpoint;
  if (C <= 0) C = std::max(1, (int)ceil(sqrt((double)M)));
  if (C > M) C = M;
  a->C = C;
  for (int s = 0; s < M; s += C) {
    a->seg_a.push_back(s);
    a->seg_b.push_back(std::min(s + C, M));
  }
  a->J = (int)a->seg_a.size();
  const size_t NB = sizeof(double) * (size_t)a->N;
  const size_t nspec = (size_t)h->n[0] * h->n[1] * h->nzh;
  PA_CUDA(a, cudaSetDevice(h->dev));
  Builder B(a, h);
  a->pair = B.adj && h->n[0] <= 96;  // see the header
  const int lanes = a->pair ? 2 : 1;
  const int sets = C == 1 ? 0 : lanes;
  for (int sg = 0; sg < 2; ++sg) {
    PA_CUDA(a, cudaMalloc((void**)&a->ck[sg], NB * a->J));
    for (int set = 0; set < sets; ++set) PA_CUDA(a, cudaMalloc((void**)&a->seg[set][sg], NB * C));
    // the last slices are needed for Q alone: in checkpointed runs they pass through a segment buffer
    if (C == 1) PA_CUDA(a, cudaMalloc((void**)&a->endq[sg], NB));
    else a->endq[sg] = a->seg[0][sg];
  }
  for (int i = 0; i < 2 * lanes; ++i) {
    PA_CUDA(a, cudaMalloc((void**)&a->lam[i], NB));
    PA_CUDA(a, cudaMalloc((void**)&a->spec[i], sizeof(double2) * nspec));
    PA_CUDA(a, cudaMalloc((void**)&a->rspec[i], sizeof(double2) * nspec));
  }
  a->storage_bytes = NB * (2 * (size_t)a->J + (C > 1 ? 2 * (size_t)sets * C : 2));
  PA_CUDA(a, cudaMalloc((void**)&a->mu, NB));
  PA_CUDA(a, cudaMalloc((void**)&a->P, NB * a->nb));
  PA_CUDA(a, cudaMalloc((void**)&a->gwb, NB * a->nb * lanes));
  PA_CUDA(a, cudaMalloc((void**)&a->gphi, NB * a->nf));
  PA_CUDA(a, cudaMemset(a->gphi, 0, NB * a->nf));
  PA_CUDA(a, cudaMalloc((void**)&a->gq, sizeof(double)));
  {
    int rp = alloc_partials(a, (size_t)2 * M);
    if (rp) return rp;
  }

  const BlockFieldMap fm = field_map(a);
  const long long N = a->N;
  if (B.adj) a->slot_block.assign(2 * (size_t)M, 0);

  // ---- forward: both sweeps in lockstep, checkpoints and end slices stored
  {
    std::vector<Builder::Run> runs;
    for (int i = 0; i < 2; ++i)
      runs.push_back({i, 0, M, nullptr, [a, M, i](int k) -> double* {
                        if (k == M) return a->endq[i];
                        for (int j = 0; j < a->J; ++j) {
                          const int pos = (i == 0) ? a->seg_a[j] : M - a->seg_b[j];
                          if (pos == k) return a->ck[i] + (size_t)j * a->N;
                        }
                        return nullptr;
                      }});
    B.sweeps(a->fwd, runs);
    // Q = <q_n0 q+_{M-n0}>
    const double* qx = (a->n0 == 0) ? a->ck[0] : a->endq[0];
    const double* qy = (a->n0 == 0) ? a->endq[1] : a->ck[1] + (size_t)(a->J - 1) * N;
    a->fwd.push_back([=](cudaStream_t st) {
      BigQSet<double> set;
      set.n = 1;
      set.a[0] = qx;
      set.b[0] = qy;
      return launch_big_q<double>(set, N, h->d_qpart, h->d_count, h->d_sc, st);
    });
    // quadrature, segment by segment
    a->fwd.push_back([=](cudaStream_t st) { return cudaMemsetAsync(a->P, 0, sizeof(double) * N * a->nb, st); });
    size_t e0 = 0;
    const int group = C == 1 ? a->J : lanes;  // segments resident together
    for (int j0 = 0; j0 < a->J; j0 += group) {
      const int n = std::min(group, a->J - j0);
      const int js[2] = {j0, j0 + 1};
      recompute(B, a->fwd, js, n);
      for (int j = j0; j < j0 + n; ++j) {
        const int nend = (j == a->J - 1) ? a->seg_b[j] : a->seg_b[j] - 1;
        for (int n_ = a->seg_a[j]; n_ <= nend; ++n_)
          for (auto& e : a->quad[n_]) {
            AccumEntry ae;
            ae.dst = a->P + (size_t)e.first * N;
            ae.x = slice_ptr(a, 0, n_, j, j - j0);
            ae.y = slice_ptr(a, 1, M - n_, j, j - j0);
            ae.coef = e.second;
            a->h_acc.push_back(ae);
          }
      }
      const int ne = (int)(a->h_acc.size() - e0);
      const size_t off = e0;
      a->fwd.push_back([=](cudaStream_t st) {
        adj_accum_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->d_acc + off, ne, N);
        return cudaGetLastError();
      });
      e0 = a->h_acc.size();
    }
    a->fwd.push_back([=](cudaStream_t st) {
      adj_normalize_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->P, h->d_phi, fm, N, h->d_sc);
      return cudaGetLastError();
    });
  }
  // ---- backward.  bwd[0] is the <g_phi, phi> reduction; ps_adj_backward
  // launches the dL/dQ kernel right after it, before any source is read.
  {
    const long long nfN = (long long)a->nf * N;
    a->bwd.push_back([=](cudaStream_t st) {
      adj_dot_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->gphi, h->d_phi, nfN, a->row(a->gq_row));
      return cudaGetLastError();
    });
    for (int b = 0; b < a->nb; ++b) {
      const int f = h->blocks[a->ip][b].field;
      a->bwd.push_back([=](cudaStream_t st) {
        adj_dot_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->gphi + (size_t)f * N, a->P + (size_t)b * N, N,
                                                  a->row(a->E_row + b));
        return cudaGetLastError();
      });
    }
    a->bwd.push_back(
        [=](cudaStream_t st) { return cudaMemsetAsync(a->gwb, 0, sizeof(double) * N * a->nb * lanes, st); });
    // sweep 0: lambda from n = M down, segments last to first; sweep 1: lambda+ from
    // m = M down, segments first to last
    int cur[2] = {0, 0};
    auto seg_run = [&](int sig, int j, int set, bool first) {
      return SegRun{sig, j, set, sig == 0 ? a->seg_a[j] : M - a->seg_b[j], sig == 0 ? a->seg_b[j] : M - a->seg_a[j],
                    first};
    };
    if (B.adj && C == 1) {  // every slice is resident
      const SegRun all[2] = {{0, 0, 0, 0, M, true}, {1, 0, 0, 0, M, true}};
      if (a->pair) {
        adjoint_segments(B, a->bwd, {all[0], all[1]}, cur);
      } else {
        for (int sig = 0; sig < 2; ++sig) {
          cur[0] = 0;
          adjoint_segments(B, a->bwd, {all[sig]}, cur);
        }
      }
    } else if (a->pair) {
      for (int t = 0; t < a->J; ++t) {
        const int js[2] = {a->J - 1 - t, t};
        const int n = js[0] == js[1] ? 1 : 2;
        recompute(B, a->bwd, js, n);
        adjoint_segments(B, a->bwd, {seg_run(0, js[0], 0, t == 0), seg_run(1, js[1], n - 1, t == 0)}, cur);
      }
    } else {
      for (int sig = 0; sig < 2; ++sig) {
        cur[0] = 0;
        for (int t = 0; t < a->J; ++t) {
          const int j = sig == 0 ? a->J - 1 - t : t;
          recompute(B, a->bwd, &j, 1);
          const SegRun run = seg_run(sig, j, 0, t == 0);
          if (B.adj) {
            adjoint_segments(B, a->bwd, {run}, cur);
            continue;
          }
          if (t == 0) adjoint_init(a, a->bwd, sig, j, cur[0]);
          for (int s = run.hi - 1; s >= run.lo; --s) {
            adjoint_step(B, a->bwd, sig, s, j, cur[0]);
            cur[0] = 1 - cur[0];
          }
        }
      }
    }
    if (a->pair)  // the lanes' sums
      a->bwd.push_back([=](cudaStream_t st) {
        adj_axpy_kernel<<<kAdjRB, kAdjRT, 0, st>>>(a->gwb, a->gwb + (size_t)a->nb * N, 1.0, N * a->nb);
        return cudaGetLastError();
      });
  }
  push_dotw(B, a->bwd);
  int r2 = adj_upload(a, &a->d_pw, a->h_pw);
  if (!r2) r2 = adj_upload(a, &a->d_xw, a->h_xw);
  if (!r2) r2 = adj_upload(a, &a->d_acc, a->h_acc);
  if (!r2) r2 = adj_upload(a, &a->d_pt, a->h_pt);
  if (!r2) r2 = adj_upload(a, &a->d_ax, a->h_ax);
  if (!r2) r2 = adj_upload(a, &a->d_dst, a->h_dst);
  for (size_t i = 0; i < a->h_sw.size(); ++i) a->h_sw[i].dst = a->d_dst + a->sw_dst[i];
  if (!r2) r2 = adj_upload(a, &a->d_sw, a->h_sw);
  return r2;
}

static void adj_free(ps_adj* a) {
  if (a->h) {
    cudaSetDevice(a->h->dev);
    if (a->h->st) cudaStreamSynchronize(a->h->st);
  }
  auto f = [](void* p) { if (p) cudaFree(p); };
  for (int sg = 0; sg < 2; ++sg) {
    f(a->ck[sg]);
    if (a->C == 1) f(a->endq[sg]);
    for (int set = 0; set < 2; ++set) f(a->seg[set][sg]);
  }
  for (int i = 0; i < 4; ++i) {
    f(a->lam[i]);
    f(a->spec[i]);
    f(a->rspec[i]);
  }
  f(a->mu);
  f(a->P);
  f(a->gwb);
  f(a->gphi);
  f(a->gq);
  f(a->part);
  f(a->d_sum);
  f(a->d_ax);
  f(a->d_sw);
  f(a->d_dst);
  if (a->h_sum) cudaFreeHost(a->h_sum);
  f(a->d_pw);
  f(a->d_xw);
  f(a->d_acc);
  f(a->d_pt);
  f(a->d_jn);
  for (auto p : a->jacc) f(p);
  if (a->h) {
    engine_free(a->h);
    delete a->h;
  }
}

static int run_ops(ps_adj* a, const std::vector<Op>& ops, size_t from) {
  for (size_t i = from; i < ops.size(); ++i) PA_CUDA(a, ops[i](a->h->st));
  return PS_OK;
}

}  // namespace psb

using namespace psb;

extern "C" {

static int adj_create(const ps_config* cfg, int polymer, int chain, bool single, int checkpoint_interval,
                      ps_adj** out) {
  if (!cfg || !out) {
    g_adj_err = "null argument";
    return PS_ATTRIB_ERR;
  }
  *out = nullptr;
  ps_adj* a = new ps_adj();
  int rc = adj_build(a, cfg, polymer, chain, single, checkpoint_interval);
  if (rc) {
    g_adj_err = a->err;
    adj_free(a);
    delete a;
    cudaGetLastError();  // clear a failed allocation's last-error state
    return rc;
  }
  *out = a;
  return PS_OK;
}

int ps_adj_create(const ps_config* cfg, int checkpoint_interval, ps_adj** out) {
  return adj_create(cfg, 0, 0, true, checkpoint_interval, out);
}

int ps_adj_create_polymer(const ps_config* cfg, int polymer, int chain, int checkpoint_interval,
                          ps_adj** out) {
  return adj_create(cfg, polymer, chain, false, checkpoint_interval, out);
}

int ps_adj_set_potential(ps_adj* a, const double* psi) {
  if (!a || !a->h || !psi) return PS_ATTRIB_ERR;
  ps_handle* h = a->h;
  if (h->nq == 0) {
    a->err = "the configuration has no chargeDens field";
    return PS_ATTRIB_ERR;
  }
  PA_CUDA(a, cudaSetDevice(h->dev));
  PA_CUDA(a, cudaMemcpyAsync(h->d_psi, psi, sizeof(double) * (size_t)h->nq * a->N, cudaMemcpyDeviceToDevice,
                             h->st));
  a->have_forward = false;
  return PS_OK;
}

int ps_adj_potential_grad(ps_adj* a, double* g_psi) {
  if (!a || !a->h || !g_psi) return PS_ATTRIB_ERR;
  ps_handle* h = a->h;
  if (h->nq == 0) {
    a->err = "the configuration has no chargeDens field";
    return PS_ATTRIB_ERR;
  }
  if (!a->have_backward) {
    a->err = "ps_adj_potential_grad needs a ps_adj_backward first";
    return PS_ATTRIB_ERR;
  }
  const long long N = a->N;
  PA_CUDA(a, cudaSetDevice(h->dev));
  PA_CUDA(a, cudaMemsetAsync(g_psi, 0, sizeof(double) * (size_t)h->nq * N, h->st));
  // psi enters a charged block's exponent as facz psi next to w: dL/dpsi = facz dL/dw of the block
  for (int b = 0; b < a->nb; ++b) {
    const BlockMap& bm = h->blocks[a->ip][b];
    if (bm.charge_field < 0) continue;
    adj_axpy_kernel<<<kAdjRB, kAdjRT, 0, h->st>>>(g_psi + (size_t)bm.charge_field * N, a->gwb + (size_t)b * N,
                                                  bm.facz, N);
    PA_CUDA(a, cudaGetLastError());
  }
  PA_CUDA(a, cudaStreamSynchronize(h->st));
  return PS_OK;
}

int ps_adj_species(const ps_adj* a, double* f_weight, double* length_ratio, double* dens_avg) {
  if (!a || !a->h) return PS_ATTRIB_ERR;
  const ps_handle* h = a->h;
  if (f_weight) *f_weight = h->chain_dwt[a->ip] * h->chain_vf[a->ip];
  if (length_ratio) *length_ratio = h->alpha[a->ip];
  if (dens_avg)
    for (int i = 0; i < h->nf; ++i) dens_avg[i] = h->fm.dens_avg[i];
  return PS_OK;
}

int ps_adj_destroy(ps_adj* a) {
  if (!a) return PS_OK;
  adj_free(a);
  delete a;
  return PS_OK;
}

const char* ps_adj_last_error(const ps_adj* a) { return a ? a->err.c_str() : g_adj_err.c_str(); }

int ps_adj_info(const ps_adj* a, int* contour_steps, int* checkpoint_interval, size_t* slice_bytes) {
  if (!a) return PS_ATTRIB_ERR;
  if (contour_steps) *contour_steps = a->M;
  if (checkpoint_interval) *checkpoint_interval = a->C;
  if (slice_bytes) *slice_bytes = a->storage_bytes;
  return PS_OK;
}

int ps_adj_forward(ps_adj* a, const double* w, double* phi, double* log_q) {
  if (!a || !w) return PS_ATTRIB_ERR;
  ps_handle* h = a->h;
  const size_t nfN = (size_t)a->nf * a->N;
  a->have_forward = a->have_backward = false;  // until this one is complete
  PA_CUDA(a, cudaSetDevice(h->dev));
  PA_CUDA(a, cudaMemcpyAsync(h->d_w, w, sizeof(double) * nfN, cudaMemcpyDeviceToDevice, h->st));
  PA_CUDA(a, cudaMemsetAsync(&h->d_sc->error_flags, 0, sizeof(int), h->st));
  long long nl = 0;
  int rc = engine_pre(h, &nl);
  if (rc) {
    a->err = h->err;
    return rc;
  }
  rc = run_ops(a, a->fwd, 0);
  if (rc) return rc;
  if (phi) PA_CUDA(a, cudaMemcpyAsync(phi, h->d_phi, sizeof(double) * nfN, cudaMemcpyDeviceToDevice, h->st));
  rc = engine_check_scalars(h);
  if (rc) {
    a->err = h->err;
    return rc;
  }
  if (log_q) *log_q = h->h_sc->log_q[0];
  a->have_forward = true;
  return PS_OK;
}

int ps_adj_backward(ps_adj* a, const double* g_phi, double g_log_q, double* g_w, double* g_box,
                    double* g_ds) {
  if (!a || !g_phi || !g_w) return PS_ATTRIB_ERR;
  if (!a->have_forward) {
    a->err = "ps_adj_backward needs a ps_adj_forward first";
    return PS_ATTRIB_ERR;
  }
  ps_handle* h = a->h;
  const long long N = a->N;
  a->have_backward = false;
  PA_CUDA(a, cudaSetDevice(h->dev));
  // a wait that ran out in an earlier backward pass says nothing about this one
  PA_CUDA(a, cudaMemsetAsync(&h->d_sc->error_flags, 0, sizeof(int), h->st));
  PA_CUDA(a, cudaMemcpyAsync(a->gphi, g_phi, sizeof(double) * (size_t)a->nf * N, cudaMemcpyDeviceToDevice,
                             h->st));
  PA_CUDA(a, a->bwd[0](h->st));
  adj_gq_kernel<<<1, kAdjRT, 0, h->st>>>(a->row(a->gq_row), g_log_q, h->d_sc, a->gq);
  PA_CUDA(a, cudaGetLastError());
  int rc = run_ops(a, a->bwd, 1);
  if (rc) return rc;
  adj_sum_blocks_kernel<<<kAdjRB, kAdjRT, 0, h->st>>>(a->gwb, field_map(a), N, g_w);
  PA_CUDA(a, cudaGetLastError());
  adj_rows_kernel<<<(unsigned)a->rows, kAdjRT, 0, h->st>>>(a->part, a->stride, a->d_sum);
  PA_CUDA(a, cudaGetLastError());
  PA_CUDA(a, cudaMemcpyAsync(a->h_sum, a->d_sum, sizeof(double) * a->rows, cudaMemcpyDeviceToHost, h->st));
  PA_CUDA(a, cudaMemcpyAsync(&h->h_sc->error_flags, &h->d_sc->error_flags, sizeof(int), cudaMemcpyDeviceToHost,
                             h->st));
  PA_CUDA(a, cudaStreamSynchronize(h->st));
  if (h->h_sc->error_flags & 4) {
    a->err = "an exchange of a recomputed sweep did not complete within the wait limit";
    return PS_GPU_ERR;
  }
  // host sums in a fixed order
  double gbox[3] = {0.0, 0.0, 0.0};
  std::vector<double> gds(a->nb, 0.0);
  const double L[3] = {h->n[0] * h->cfg.cell[0], h->n[1] * h->cfg.cell[1], h->n[2] * h->cfg.cell[2]};
  for (size_t slot = 0; slot < a->slot_block.size(); ++slot) {
    const int b = a->slot_block[slot];
    const BlockMap& bm = h->blocks[a->ip][b];
    const double* R = a->h_sum + slot * 4;
    const double b2 = bm.bseg * bm.bseg;
    for (int d = 0; d < 3; ++d) gbox[d] += 2.0 * bm.ds * b2 / L[d] * R[d];
    gds[b] += -b2 * (R[0] + R[1] + R[2]) + R[3];
  }
  // the fused steps' explicit ds derivative: sum over the block's steps of -1/2 (w, t)
  // with dL/dw = sum of -ds/2 t
  for (int b = 0; b < a->nb; ++b)
    gds[b] += (a->h_sum[a->E_row + b] + a->h_sum[a->W_row + b]) / h->blocks[a->ip][b].ds;
  if (g_box)
    for (int d = 0; d < 3; ++d) g_box[d] = gbox[d];
  if (g_ds)
    for (int b = 0; b < a->nb; ++b) g_ds[b] = gds[b];
  a->have_backward = true;
  return PS_OK;
}

void* ps_adj_stream(const ps_adj* a) { return (a && a->h) ? (void*)a->h->st : nullptr; }

}  // extern "C"
