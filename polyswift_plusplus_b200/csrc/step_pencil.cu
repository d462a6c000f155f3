// x pass of a propagator step in registers (VARIANT_FUSE_K): forward x FFT,
// multiply by exp(-ds b^2 k^2) / N, inverse x FFT.
//
// The pass it replaces for the sweeps (pencil_kernel) took the tile through
// shared memory six times (load, two forward passes, two inverse passes,
// store).  Here thread (c, j) loads the L / G elements x = j + G r of column c
// straight into its radix-(L / G) butterfly, the elements are exchanged once, the
// radix-G butterflies, the k^2 multiply and the first inverse butterflies work
// on the same registers, and after a second exchange the result goes straight
// back to memory: two exchanges, two barriers.  A tile is 16 adjacent columns
// (128-byte segments in FP32, 256 in FP64).  With the plane pass unchanged, a step
// of both sweeps at 128^3 went from 31.3 to 26.6 us (FP32) and from 53.9 to 44.8
// (FP64); the pass itself takes 6.9 and 12.5 us there for 17 and 34 MB each way,
// bound by the latency of its loads in one wave of CTAs.
#include "step_common.cuh"

namespace psb {

template <typename T, int L> struct PencilG {
  static constexpr int G = (L >= 256) ? 16 : (L >= 16 ? 8 : (L >= 8 ? 4 : (L >= 4 ? 2 : 1)));
  static constexpr int R = L / G, U = (R + G - 1) / G;
  // a warp at least; at L = 256 in FP64 half the columns, for 48 KB of shared memory
  static constexpr int TK = (G == 1) ? 32 : (L >= 256 && sizeof(T) == 8 ? 8 : 16);
  static constexpr int TH = TK * G;
  static_assert(R * G == L && TH >= 32, "pencil groups");
};

// EARLY: see early_path in sweeps.cuh (a template argument: as a run-time one it cost up to
// 4% of an FP32 step at 48^3).
template <typename T, int L, bool EARLY>
__global__ void __launch_bounds__((PencilG<T, L>::TH))
    step_pencil_kernel(const PencilWork<T>* __restrict__ works, int inner, int compact,
                       const c2_t<T>* __restrict__ tw) {
  using P = PencilG<T, L>;
  using C = c2_t<T>;
  constexpr int G = P::G, R = P::R, U = P::U, TK = P::TK, TH = P::TH;
  __shared__ C buf[L * TK];
  __shared__ C s_tw[L];
  __shared__ T s_kx[L];
  const PencilWork<T> w = works[blockIdx.y];
  const int tid = threadIdx.x;
  const int cc = tid % TK, j = tid / TK;
  const int c = blockIdx.x * TK + cc;
  const bool in = c < inner;
  C* const base = w.spec + c;
  const bool dc0 = w.dc_total && blockIdx.x == 0;  // mean-mode carry: see PlaneWork
  for (int i = tid; i < L; i += TH) {
    s_tw[i] = tw[i];
    s_kx[i] = __ldg(w.kx + i);
  }
  const T fyz = in ? __ldg((compact ? w.kyzc : w.kyz) + c) : T(0);
  pdl_wait();  // before any read or write of the spectrum
  if constexpr (EARLY) pdl_trigger();
  C v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = in ? __ldcg(base + (size_t)(j + G * r) * inner) : C{T(0), T(0)};
  DcFinish<T> dcf;
  if (dc0 && tid < 32) dcf.load(w);
  Dft<R, false, C>::run(v);
  C* const col = buf + cc;
#pragma unroll
  for (int r = 0; r < R; ++r) col[(j * R + r) * TK] = v[r];
  if (dc0 && tid < 32) dcf.finish(w);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int jp = j + u * G;
    if (R % G == 0 || jp < R) {
      C b[G];
#pragma unroll
      for (int r = 0; r < G; ++r) b[r] = col[(r * R + jp) * TK];
#pragma unroll
      for (int r = 1; r < G; ++r) b[r] = cmul(b[r], s_tw[r * jp]);
      Dft<G, false, C>::run(b);
#pragma unroll
      for (int r = 0; r < G; ++r) {
        const T f = s_kx[jp + R * r] * fyz;
        b[r] = C{b[r].x * f, b[r].y * f};
      }
      if (dc0 && c == 0 && jp == 0) b[0] = C{T(0), T(0)};
      Dft<G, true, C>::run(b);
#pragma unroll
      for (int r = 0; r < G; ++r) col[(r * R + jp) * TK] = b[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = col[(j * R + r) * TK];
#pragma unroll
  for (int r = 1; r < R; ++r) v[r] = cmulc(v[r], s_tw[r * j]);
  Dft<R, true, C>::run(v);
  if (in) {
#pragma unroll
    for (int r = 0; r < R; ++r) __stcg(base + (size_t)(j + G * r) * inner, v[r]);
  }
}

template <typename T, int L>
static cudaError_t launch_step_pencil_t(const PencilWork<T>* d_works, int nworks, int inner, bool compact, bool early,
                                        const c2_t<T>* tw, cudaStream_t st) {
  using P = PencilG<T, L>;
  return launch_sweep_kernel(early ? step_pencil_kernel<T, L, true> : step_pencil_kernel<T, L, false>,
                             dim3((inner + P::TK - 1) / P::TK, nworks), dim3(P::TH), 0, st, d_works, inner,
                             compact ? 1 : 0, tw);
}

template <typename T>
cudaError_t launch_step_pencil(const PencilWork<T>* w, int nw, int L, int inner, bool compact, bool early,
                               const c2_t<T>* tw, cudaStream_t st) {
  switch (L) {
    case 1: return launch_step_pencil_t<T, 1>(w, nw, inner, compact, early, tw, st);
    case 4: return launch_step_pencil_t<T, 4>(w, nw, inner, compact, early, tw, st);
    case 8: return launch_step_pencil_t<T, 8>(w, nw, inner, compact, early, tw, st);
    case 12: return launch_step_pencil_t<T, 12>(w, nw, inner, compact, early, tw, st);
    case 16: return launch_step_pencil_t<T, 16>(w, nw, inner, compact, early, tw, st);
    case 24: return launch_step_pencil_t<T, 24>(w, nw, inner, compact, early, tw, st);
    case 32: return launch_step_pencil_t<T, 32>(w, nw, inner, compact, early, tw, st);
    case 48: return launch_step_pencil_t<T, 48>(w, nw, inner, compact, early, tw, st);
    case 64: return launch_step_pencil_t<T, 64>(w, nw, inner, compact, early, tw, st);
    case 96: return launch_step_pencil_t<T, 96>(w, nw, inner, compact, early, tw, st);
    case 128: return launch_step_pencil_t<T, 128>(w, nw, inner, compact, early, tw, st);
    case 256: return launch_step_pencil_t<T, 256>(w, nw, inner, compact, early, tw, st);
  }
  return cudaErrorInvalidValue;
}
template cudaError_t launch_step_pencil<float>(const PencilWork<float>*, int, int, int, bool, bool, const float2*,
                                               cudaStream_t);
template cudaError_t launch_step_pencil<double>(const PencilWork<double>*, int, int, int, bool, bool, const double2*,
                                                cudaStream_t);

}  // namespace psb
