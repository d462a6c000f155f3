// Pieces shared by the sweep kernels (prop_kernels.cu, step_plane.cuh,
// step_pencil.cu): the FP64 mean-mode carry, the c2r / r2c pairing of one
// element, and the launch with programmatic stream serialisation.
#pragma once

#include <stdlib.h>

#include "fft_smem.cuh"
#include "kernels.h"

namespace psb {

// ---------------------------------------------------------------------------
// Mean-mode carry (see PlaneWork in kernels.h).
// ---------------------------------------------------------------------------
// Per-warp FP64 sums of the forward input, summed into one CTA partial.
static __shared__ double s_dc_warp[32];
// The mean-mode value of the inverse transform rounded to T; written by
// thread 0 after pdl_wait(), read after the barriers that precede the inverse
// step (kept in shared memory, not in registers, through the FFT passes).  What
// the rounding drops comes back through the next step's mean (dc_err).
static __shared__ __align__(16) double s_dc_hilo[2];

template <typename T>
__device__ __forceinline__ void dc_hilo_store(const double* dc_in) {
  if (threadIdx.x == 0 && dc_in) reinterpret_cast<T*>(s_dc_hilo)[0] = T(*dc_in);
}

// x + mean-mode value
template <typename T>
__device__ __forceinline__ c2_t<T> dc_add2(c2_t<T> x) {
  const T m = reinterpret_cast<const T*>(s_dc_hilo)[0];
  return cadd(x, c2_t<T>{m, m});
}
template <typename T>
__device__ __forceinline__ T dc_add(T x) {
  return x + reinterpret_cast<const T*>(s_dc_hilo)[0];
}

// Every thread of the CTA calls this (CTA-uniform): lane 0 keeps its warp's sum.
__device__ __forceinline__ void dc_warp_sum(double v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) s_dc_warp[threadIdx.x >> 5] = v;
}

// After a __syncthreads() that follows dc_warp_sum: thread 0 stores the CTA's
// partial (warps in order) and CTA 0 the number of partials.  The pointers are
// read from the descriptor here, not kept in registers through the kernel.
template <typename T>
__device__ __forceinline__ void dc_cta_store(const PlaneWork<T>* wp) {
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) s += s_dc_warp[i];
    double* out = reinterpret_cast<double*>(
        __ldg(reinterpret_cast<const unsigned long long*>(&wp->dc_out)));
    out[blockIdx.x] = s;
    if (blockIdx.x == 0) {
      double* cnt = reinterpret_cast<double*>(
          __ldg(reinterpret_cast<const unsigned long long*>(&wp->dc_count)));
      *cnt = (double)gridDim.x;
    }
  }
}

// Spectral pass side: one warp sums the plane pass's partials in a fixed order
// (lane l takes slots l, l + 32, ...; then a butterfly) and stores the mean.
// load() issues the count and the first kDcMinSlots slots (before the count is
// known) so that they travel with the tile loads; finish() sums them.
template <typename T> struct DcFinish {
  double cnt;
  double v[kDcMinSlots / 32];
  __device__ __forceinline__ void load(const PencilWork<T>& w) {
    const int lane = threadIdx.x & 31;
    cnt = *w.dc_count;
#pragma unroll
    for (int k = 0; k < kDcMinSlots / 32; ++k) v[k] = w.dc_parts[lane + 32 * k];
  }
  __device__ __forceinline__ void finish(const PencilWork<T>& w) const {
    const int lane = threadIdx.x & 31;
    const int n = (int)cnt;
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kDcMinSlots / 32; ++k)
      if (lane + 32 * k < n) s += v[k];
    for (int i = kDcMinSlots + lane; i < n; i += 32) s += w.dc_parts[i];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) {
      // error feedback: add what the previous step's rounding to T dropped
      const double m = s * w.dc_scale + (w.dc_first ? 0.0 : *w.dc_err);
      *w.dc_total = m;
      *w.dc_err = m - (double)T(m);
    }
  }
};

// One element of the c2r pre-processing and of the r2c post-processing, from
// the element and its mirror image (k with h - k of the same row).
template <typename C>
__device__ __forceinline__ C c2r_pre_one(C a, C b, C w) {
  // C'[k] = (A[k] + conj(A[h-k])) + i conj(W^k) (A[k] - conj(A[h-k]))
  const C ep = {a.x + b.x, a.y - b.y};
  const C dm = {a.x - b.x, a.y + b.y};
  const C op = cmulc(dm, w);
  return {ep.x - op.y, ep.y + op.x};
}

template <typename C>
__device__ __forceinline__ C r2c_post_one(C c, C d, C w) {
  // E = (C[k] + conj(C[km]))/2, O = -i (C[k] - conj(C[km]))/2, A[k] = E + W^k O
  using S = decltype(c.x);
  const C E = {S(0.5) * (c.x + d.x), S(0.5) * (c.y - d.y)};
  const C O = {S(0.5) * (c.y + d.y), S(0.5) * (d.x - c.x)};
  return cadd(E, cmul(w, O));
}

// Opt in to large dynamic shared memory once per (kernel, device).
template <typename K>
static cudaError_t ensure_smem_attr(K kern, size_t smem, unsigned* done_mask) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned bit = 1u << (dev & 31);
  if (*done_mask & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) *done_mask |= bit;
  return e;
}

// Sweep kernels are launched with programmatic stream serialisation (they call
// pdl_wait() before touching data another kernel wrote), unless PSB_PDL=0.
static bool pdl_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("PSB_PDL");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on != 0;
}

template <typename... K, typename... Args>
static cudaError_t launch_sweep_kernel(void (*kern)(K...), dim3 grid, dim3 block, size_t smem,
                                       cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_enabled() ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace psb
