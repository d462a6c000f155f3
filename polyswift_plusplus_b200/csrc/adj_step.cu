// Fused adjoint steps (adjoint.cuh): the plane pass in the adjoint modes and the x
// pass with the stress sums.
//
// What was slow: an adjoint step was seven launches (two forward planes, two x
// passes, the stress sums, the k^2 multiply, the inverse passes and the pointwise
// update), each reading and writing whole spectra or fields.  Now it is two: the x pass
// keeps U and V in registers between their forward transforms, the stress sums and U's
// way back, and the plane pass turns mu into the next lambda and starts its transform
// (and that of wf q) in the same pass.
//
// At 64^3: 33 -> 13 us a step; forward and backward of 128 steps 18.6 -> 9.9 ms (half of
// it the sweeps and their recomputation from checkpoints), 7.6 with the adjoints of both
// sweeps in the same launches.  A step is bound by the latency of its two launches.
// Replaying the passes as graphs changed nothing: submitting them is not the limit.
// Neither is one plane CTA of 240 registers per SM: with 128 (two) 7.6 to 7.9 ms.
#include "step_plane.cuh"

namespace psb {

template <int N>
static cudaError_t launch_adj_plane(const PlaneWork<double>* w, int nw, int nx, const double2* ty, const double2* tz,
                                    const AdjArgs& adj, cudaStream_t st) {
  using P = StepPlane<double, N, N>;
  auto kern = step_plane_kernel<double, N, N, true, false>;
  static unsigned attr_mask = 0;
  cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
  if (e != cudaSuccess) return e;
  return launch_sweep_kernel(kern, dim3(nx, nw), dim3(P::TH), P::SMEM, st, w, ty, tz, adj);
}

bool adj_step_supported(int ny, int nz) { return ny == nz && step_plane_supported(ny, nz); }

cudaError_t launch_step_plane_adj(const PlaneWork<double>* w, int nw, int nx, int ny, const double2* ty,
                                  const double2* tz, const AdjArgs& adj, cudaStream_t st) {
  switch (ny) {
    case 16: return launch_adj_plane<16>(w, nw, nx, ty, tz, adj, st);
    case 24: return launch_adj_plane<24>(w, nw, nx, ty, tz, adj, st);
    case 32: return launch_adj_plane<32>(w, nw, nx, ty, tz, adj, st);
    case 48: return launch_adj_plane<48>(w, nw, nx, ty, tz, adj, st);
    case 64: return launch_adj_plane<64>(w, nw, nx, ty, tz, adj, st);
    case 96: return launch_adj_plane<96>(w, nw, nx, ty, tz, adj, st);
    case 128: return launch_adj_plane<128>(w, nw, nx, ty, tz, adj, st);
  }
  return cudaErrorInvalidValue;
}

template <int L> struct AdjX {
  static constexpr int G = (L >= 256) ? 16 : (L >= 16 ? 8 : (L >= 8 ? 4 : (L >= 4 ? 2 : 1)));
  static constexpr int R = L / G, U = (R + G - 1) / G;
  static constexpr int TK = (G == 1) ? 32 : (L >= 128 ? 8 : 16), TH = TK * G;
  static constexpr size_t SMEM = sizeof(double2) * (2 * (size_t)L * TK + L) + sizeof(double) * (L + 3 * 32);
};

__device__ __forceinline__ double adj_x_kcomp(int i, int n, double dx) {
  const double n2 = (double)n / 2.0;
  const double nk = n2 - fabs((double)i - n2);
  return 2.0 * 3.14159265358979323846 * nk / ((double)n * dx);
}

template <int L>
__global__ void __launch_bounds__(AdjX<L>::TH)
    adj_x_kernel(const AdjXWork* __restrict__ work, int ny, int nz, double dx, double dy, double dz, int stride,
                 const double2* __restrict__ tw) {
  using P = AdjX<L>;
  constexpr int G = P::G, R = P::R, U = P::U, TK = P::TK, TH = P::TH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double2* bu = reinterpret_cast<double2*>(smem_raw);
  double2* bv = bu + L * TK;
  double2* s_tw = bv + L * TK;
  double* s_k2 = reinterpret_cast<double*>(s_tw + L);  // k_x^2
  double* s_sum = s_k2 + L;
  const AdjXWork w = work[blockIdx.y];
  const int tid = threadIdx.x;
  const int cc = tid % TK, j = tid / TK;
  const int hz = nz / 2, inner = ny * (hz + 1);
  const int c = blockIdx.x * TK + cc;
  const bool in = c < inner;
  for (int i = tid; i < L; i += TH) {
    s_tw[i] = tw[i];
    const double k = adj_x_kcomp(i, L, dx);
    s_k2[i] = k * k;
  }
  pdl_wait();
  double2* const ub = w.u + c;
  const double2* const vb = w.v + c;
  double2 a[R], b[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    a[r] = in ? __ldcg(ub + (size_t)(j + G * r) * inner) : double2{0.0, 0.0};
    b[r] = in ? __ldcg(vb + (size_t)(j + G * r) * inner) : double2{0.0, 0.0};
  }
  Dft<R, false, double2>::run(a);
  Dft<R, false, double2>::run(b);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    bu[(j * R + r) * TK + cc] = a[r];
    bv[(j * R + r) * TK + cc] = b[r];
  }
  __syncthreads();
  const double fyz = in ? __ldg(w.kyzc + c) : 0.0;
  double s0 = 0.0, s1 = 0.0;  // sums of t k_x^2 and of t over this thread's wave numbers
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int jp = j + u * G;
    if (R % G == 0 || jp < R) {
      double2 p[G], q[G];
#pragma unroll
      for (int r = 0; r < G; ++r) {
        p[r] = bu[(r * R + jp) * TK + cc];
        q[r] = bv[(r * R + jp) * TK + cc];
      }
#pragma unroll
      for (int r = 1; r < G; ++r) {
        p[r] = cmul(p[r], s_tw[r * jp]);
        q[r] = cmul(q[r], s_tw[r * jp]);
      }
      Dft<G, false, double2>::run(p);
      Dft<G, false, double2>::run(q);
#pragma unroll
      for (int r = 0; r < G; ++r) {
        const double f = __ldg(w.kx + jp + R * r) * fyz;
        const double t = (p[r].x * q[r].x + p[r].y * q[r].y) * f;
        s0 += t * s_k2[jp + R * r];
        s1 += t;
        p[r] = double2{p[r].x * f, p[r].y * f};
      }
      Dft<G, true, double2>::run(p);
#pragma unroll
      for (int r = 0; r < G; ++r) bu[(r * R + jp) * TK + cc] = p[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = bu[(j * R + r) * TK + cc];
#pragma unroll
  for (int r = 1; r < R; ++r) a[r] = cmulc(a[r], s_tw[r * j]);
  Dft<R, true, double2>::run(a);
  if (in) {
#pragma unroll
    for (int r = 0; r < R; ++r) __stcg(ub + (size_t)(j + G * r) * inner, a[r]);
  }
  // The spectra and kyzc carry 2 x 2 x 1/2 of conj(U) V K; wave numbers off the
  // kz = 0 and nz/2 planes stand for their mirror images too.
  const int ky = (c < ny * hz) ? c / hz : c - ny * hz;
  const int kz = (c < ny * hz) ? c - ky * hz : hz;
  const double mult = 0.5 * ((kz == 0 || kz == hz) ? 1.0 : 2.0);
  const double k1 = adj_x_kcomp(ky, ny, dy), k2 = adj_x_kcomp(kz, nz, dz);
  double r3[3] = {mult * s0, mult * s1 * k1 * k1, mult * s1 * k2 * k2};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) r3[d] += __shfl_xor_sync(0xffffffffu, r3[d], off);
    if ((tid & 31) == 0) s_sum[d * 32 + (tid >> 5)] = r3[d];
  }
  __syncthreads();
  if (tid < 3) {
    double s = 0.0;
    for (int i = 0; i < TH / 32; ++i) s += s_sum[tid * 32 + i];
    w.part[(size_t)tid * stride + blockIdx.x] = s;
  }
}

template <int L>
static cudaError_t launch_adj_x_t(const AdjXWork* w, int nw, int ny, int nz, double dx, double dy, double dz, int stride,
                                  const double2* tw, cudaStream_t st) {
  using P = AdjX<L>;
  auto kern = adj_x_kernel<L>;
  static unsigned attr_mask = 0;
  cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
  if (e != cudaSuccess) return e;
  const int inner = ny * (nz / 2 + 1);
  return launch_sweep_kernel(kern, dim3((inner + P::TK - 1) / P::TK, nw), dim3(P::TH), P::SMEM, st, w, ny, nz, dx, dy, dz,
                             stride, tw);
}

#define PSB_ADJ_X(X) X(1) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(256)

int adj_x_tiles(int nx, int inner) {
#define PSB_X(L) \
  if (nx == L) return (inner + AdjX<L>::TK - 1) / AdjX<L>::TK;
  PSB_ADJ_X(PSB_X)
#undef PSB_X
  return 0;
}

cudaError_t launch_adj_x(const AdjXWork* w, int nw, int nx, int ny, int nz, double dx, double dy, double dz, int stride,
                         const double2* tw, cudaStream_t st) {
#define PSB_X(L) \
  if (nx == L) return launch_adj_x_t<L>(w, nw, ny, nz, dx, dy, dz, stride, tw, st);
  PSB_ADJ_X(PSB_X)
#undef PSB_X
  return cudaErrorInvalidValue;
}

}  // namespace psb
