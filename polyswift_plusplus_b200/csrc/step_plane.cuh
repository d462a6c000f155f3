// Plane pass of a propagator step with group-local FFTs (VARIANT_FUSE_Z).
//
// What bounded the pass it replaces (plane_kernel): a chain of eleven CTA-wide
// barrier pairs per plane, one for every butterfly pass, packing loop and
// pre-/post-processing step, with every warp of the CTA in the same phase
// (shared-memory loads, arithmetic, stores) at the same time: a third of the
// issue slots used.  Here an FFT of length L = R G is held by G threads with R
// elements each and exchanges its elements once, so only its own threads need
// to meet: a y column belongs to a few warps (a named barrier), a z row to lanes
// of one warp (__syncwarp).  The CTA meets twice per plane: rows complete,
// columns complete.
//
// Two real rows y and y + ny/2 make one complex row, so that a plane is ny/2
// rows of nz complex values: the z transforms need no c2r / r2c twiddles, and
// separating the two rows costs additions only, done in registers between the
// y and z parts on column c and its mirror image nz - c, which belong to the
// same threads.  The first y butterflies read global memory directly and the
// last ones write it.
//
//   y part    thread (c, j), c < nz/2: ky = j + G r from global memory (16 adjacent
//             columns: 128-byte segments) -> radix R -> exchange -> radix G ->
//             columns c and nz - c of the packed rows
//   z part    thread (row, j): radix R, exchange, radix G, the real-space step in
//             registers, radix G, exchange, radix R
//   y part    columns c and nz - c -> radix G, exchange, radix R -> global memory
//
// Both sweeps of a diblock, one propagator step each, with the x pass of
// step_pencil.cu (B200, us; the fastest earlier variant first): 128^3 FP32 30.6 ->
// 23.8, FP64 59.0 -> 44.4; 96^3 27.0 -> 14.2, 34.6 -> 20.9; 64^3 12.0 -> 7.2, 14.1 ->
// 9.2; 48^3 11.7 -> 5.5, 11.9 -> 7.2; 32^3 6.5 -> 4.5, 6.7 -> 4.6; less with early starts
// (early_path in sweeps.cuh).  64 x 96 x 48 (a blend, three sweeps; it had a row pass
// and two y pencil passes): 28 -> 10.
// What bounds it now: at 128^2 the shared-memory and L1 data path (66% busy, 13.4 k
// wavefronts a plane) with one wave of CTAs that load, compute and store at the
// same time; at 64^2 and below the latency of one plane's chain.
//
// Spectrum layout (compact): plane x holds [ky][kz < nz/2] and then the nz/2
// (Nyquist) column, so that rows of 16 columns are aligned segments.  The real
// kz = 0 and Nyquist columns share one complex y transform (a_0 + i a_h).  The
// values are twice those of the transform (the separation's factor 1/2 is left
// to the k^2 table kyzc: exact, and four multiplies fewer per pair).
#pragma once

#include "adjoint.cuh"
#include "step_common.cuh"

namespace psb {

// Threads of a y FFT of length L (an even number), L / G elements each.  G does
// not have to divide L / G: with fewer than G radix-G butterflies some lanes
// idle there.
template <int L> struct GroupOf { static constexpr int v = (L >= 256) ? 16 : (L >= 16 ? 8 : 4); };
// Threads of a z row: lanes of one warp, and whole warps over the PR rows.
template <int PR, int L> struct RowGroup { static constexpr int v = (L >= 48 || L == 24 || PR % 8 != 0) ? 8 : 4; };
constexpr int kStepExtents[] = {16, 24, 32, 48, 64, 96, 128};

template <typename T, int NY, int NZ> struct StepPlane {
  static constexpr int H = NZ / 2, PR = NY / 2;
  static constexpr int GY = GroupOf<NY>::v, RY = NY / GY, UY = (RY + GY - 1) / GY;
  static constexpr int GZ = RowGroup<PR, NZ>::v, RZ = NZ / GZ, UZ = (RZ + GZ - 1) / GZ;
  // FP32: exchange slots in pairs (16-byte accesses), an odd number of 16-byte
  // units per thread; the rows of a half-warp 8 slots apart modulo 16
  static constexpr bool V2 = sizeof(T) == 4 && RZ % 2 == 0;
  static constexpr int PA = V2 ? ((RZ / 2) % 2 ? RZ : RZ + 2) : RZ + 1;
  static constexpr int S0 = GZ * PA;
  static constexpr int S = (sizeof(T) == 4) ? S0 + ((24 - S0 % 16) % 16) : S0;
  static constexpr int TH = H * GY;
  // columns of a y group: 128-byte segments where the row length allows
  static constexpr int CW = (sizeof(T) == 4) ? 16 : 8;
  static constexpr int CG = (H % CW == 0) ? CW : ((H % 8 == 0) ? 8 : H);
  static constexpr int NG = H / CG;
  static constexpr int TASKS = PR * GZ;
  // positions whose Boltzmann factors are loaded together: FP32 with two
  // positions per butterfly has registers for two (128^2: 17.7 us for 256 planes,
  // 18.1 with one and 19.3 with four), the others for four (64^2 FP64: 5.8 us
  // for 128 planes, 6.0 with one; 128^2 FP64: 40.0, 42.3)
  static constexpr int CH = (sizeof(T) == 4 && UZ == 2 && GZ == 8) ? 2 : 4;
  static constexpr size_t SMEM = sizeof(c2_t<T>) * ((size_t)PR * S + 2 * NY + 2 * NZ);
  // registers: FP32 64 and FP64 128 a thread
  static constexpr int BY_REG = 65536 / (TH * (sizeof(T) == 4 ? 64 : 128));
  static constexpr int BY_SMEM = (int)((size_t)224 * 1024 / (SMEM + 1024));
  static constexpr int MINB0 = BY_REG < BY_SMEM ? BY_REG : BY_SMEM;
  static constexpr int MINB = MINB0 < 1 ? 1 : (MINB0 > 16 ? 16 : MINB0);
  static constexpr bool CAN_EARLY = sizeof(T) == 4 && NY >= 96 && NZ >= 96;
  static_assert(TH % 32 == 0 && TH <= 1024 && TASKS % 32 == 0 && UZ <= 2, "step plane layout");
  static_assert(NG == 1 || ((CG * GY) % 32 == 0 && NG <= 15), "step plane groups");
  static_assert(S >= NZ && RY * GY == NY && RZ * GZ == NZ && GY % 2 == 0, "step plane layout");
};

// The threads of one y group (id 1..15), or the CTA when it is one group.
template <int NG, int THREADS> __device__ __forceinline__ void group_sync(int g) {
  if constexpr (NG == 1) __syncthreads();
  else if constexpr (THREADS == 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(THREADS) : "memory");
}

// U adjacent reals.
template <typename T, int U> struct Reals;
template <> struct Reals<float, 1> { using type = float; };
template <> struct Reals<double, 1> { using type = double; };
template <> struct Reals<float, 2> { using type = float2; };
template <> struct Reals<double, 2> { using type = double2; };

template <typename T, int U> struct RealRun {
  T v[U];
  __device__ __forceinline__ void ones() {
#pragma unroll
    for (int i = 0; i < U; ++i) v[i] = T(1);
  }
  __device__ __forceinline__ void load(const T* p) {
    using V = typename Reals<T, U>::type;
    const V x = __ldg(reinterpret_cast<const V*>(p));
#pragma unroll
    for (int i = 0; i < U; ++i) v[i] = reinterpret_cast<const T*>(&x)[i];
  }
  __device__ __forceinline__ void load_plain(const T* p) {
    using V = typename Reals<T, U>::type;
    const V x = *reinterpret_cast<const V*>(p);
#pragma unroll
    for (int i = 0; i < U; ++i) v[i] = reinterpret_cast<const T*>(&x)[i];
  }
  __device__ __forceinline__ void store(T* p) const {
    using V = typename Reals<T, U>::type;
    V x;
#pragma unroll
    for (int i = 0; i < U; ++i) reinterpret_cast<T*>(&x)[i] = v[i];
    *reinterpret_cast<V*>(p) = x;
  }
};

// The real-space part of an adjoint step (adjoint.cuh) at M runs of U adjacent
// points.  load() fetches every stream before any is used (one run at a time the
// pass was a chain of L2 latencies: 30 us at 64^3); apply() turns mu (has_mu) into
// the next lambda, in x.
template <int U, int M> struct AdjRuns {
  using Run = RealRun<double, U>;
  Run q[M], gp[M], pt[M], gw[M];
  __device__ __forceinline__ void fetch(Run (&r)[M], const double* base, const size_t (&at)[M]) {
#pragma unroll
    for (int m = 0; m < M; ++m) r[m].load(base + at[m]);
  }
  __device__ __forceinline__ void load(const AdjPoint& p, const size_t (&at)[M]) {
    fetch(q, p.q_s, at);
    if (p.lam_out && p.n_src > 0) {
      fetch(gp, p.src[0].gphi, at);
      fetch(pt, p.src[0].partner, at);
    }
    const double* g = p.gwb ? p.gwb : p.gwb2;
#pragma unroll
    for (int m = 0; m < M; ++m) gw[m].load_plain(g + at[m]);
  }
  __device__ __forceinline__ void apply(const AdjPoint& p, const AdjGlobals& g, const size_t (&at)[M], bool has_mu,
                                        Run (&x)[M]) {
    const bool lam = p.lam_out != nullptr, src = lam && p.n_src > 0;
    Run l[M];
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (!has_mu) x[m].v[u] = 0.0;
        l[m].v[u] = src ? x[m].v[u] + (g.inv_q * p.src[0].coef) * (gp[m].v[u] * pt[m].v[u]) : x[m].v[u];
      }
    if (lam) {
      for (int i = 1; i < p.n_src; ++i) {  // a block joint: two quadrature pairs
        fetch(gp, p.src[i].gphi, at);
        fetch(pt, p.src[i].partner, at);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int u = 0; u < U; ++u) l[m].v[u] += (g.inv_q * p.src[i].coef) * (gp[m].v[u] * pt[m].v[u]);
      }
      if (p.q_partner) {
        fetch(gp, p.q_partner, at);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int u = 0; u < U; ++u) l[m].v[u] += g.gq_n * gp[m].v[u];
      }
      if (p.extra) {
        fetch(gp, p.extra, at);
#pragma unroll
        for (int m = 0; m < M; ++m)
#pragma unroll
          for (int u = 0; u < U; ++u) l[m].v[u] += gp[m].v[u];
      }
#pragma unroll
      for (int m = 0; m < M; ++m) l[m].store(p.lam_out + at[m]);
    }
    const bool one = (p.gwb == p.gwb2);
    if (p.gwb) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int u = 0; u < U; ++u)
          gw[m].v[u] -= p.half_ds * q[m].v[u] * (one ? x[m].v[u] + l[m].v[u] : x[m].v[u]);
        gw[m].store(p.gwb + at[m]);
      }
    }
    if (p.gwb2 && !one) {
      if (p.gwb) {
#pragma unroll
        for (int m = 0; m < M; ++m) gw[m].load_plain(p.gwb2 + at[m]);
      }
#pragma unroll
      for (int m = 0; m < M; ++m) {
#pragma unroll
        for (int u = 0; u < U; ++u) gw[m].v[u] -= p.half_ds2 * q[m].v[u] * l[m].v[u];
        gw[m].store(p.gwb2 + at[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < M; ++m) x[m] = l[m];
  }
};

// ADJ (FP64): works in the adjoint modes of adjoint.cuh beside FIRST ones.
// EARLY: the x pass behind it may be placed before this pass has ended (early_path in
// sweeps.cuh).
template <typename T, int NY, int NZ, bool ADJ, bool EARLY>
__global__ void __launch_bounds__((StepPlane<T, NY, NZ>::TH), (ADJ ? 1 : StepPlane<T, NY, NZ>::MINB))
    step_plane_kernel(const PlaneWork<T>* __restrict__ works, const c2_t<T>* __restrict__ tw_y,
                      const c2_t<T>* __restrict__ tw_z, AdjArgs adj) {
  using P = StepPlane<T, NY, NZ>;
  using C = c2_t<T>;
  constexpr int H = P::H, PR = P::PR, S = P::S, TH = P::TH, CG = P::CG, PA = P::PA;
  constexpr int GY = P::GY, RY = P::RY, UY = P::UY, GZ = P::GZ, RZ = P::RZ, UZ = P::UZ;
  constexpr int GH = GY / 2, CH = (ADJ && UZ == 2) ? 1 : P::CH;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  C* s_nyq = buf + PR * S;  // column 0 on its way out, to separate the Nyquist column
  C* s_tw_y = s_nyq + NY;
  C* s_twb = s_tw_y + NY;  // exp(-2 pi i r j / nz) as [r][j] for the radix-GZ passes
  C* s_twf = s_twb + NZ;   // ... and for the radix-RZ ones: consecutive lanes, consecutive banks

  const PlaneWork<T> w = works[blockIdx.y];
  const int tid = threadIdx.x;
  const int g = tid / (CG * GY);
  const int tg = tid - g * (CG * GY);
  const int c = g * CG + tg % CG;
  const int j = tg / CG;
  // the mirror column; columns 0 and nz/2 are their own and go together
  const int mc = (c == 0) ? H : NZ - c;
  C* const spec = w.spec + (size_t)blockIdx.x * (NY * (H + 1)) + c;
  const size_t roff = (size_t)blockIdx.x * (NY * NZ);
  const bool adj_on = ADJ && w.mode >= MODE_ADJ_INIT;
  const bool inverse = w.mode != MODE_FIRST && !(ADJ && w.mode == MODE_ADJ_INIT);
  const bool forward = w.mode != MODE_LAST && !(ADJ && w.mode == MODE_ADJ_LAST);
  const bool dc_sum = forward && (w.dc_out != nullptr);

  for (int i = tid; i < NY; i += TH) s_tw_y[i] = tw_y[i];
  for (int i = tid; i < NZ; i += TH) {
    s_twb[i] = tw_z[(i / RZ) * (i % RZ)];
    s_twf[i] = tw_z[(i / GZ) * (i % GZ)];
  }
  __syncthreads();  // the groups below read tables that other groups wrote
  pdl_wait();       // before any read of the spectrum, src or wfac, and any write

  // exchange slot d of column c: row d % (ny/2) of column c, or of its mirror
  C* const slot_j = buf + (j % GH) * RY * S + (j < GH ? c : mc);  // slots j RY + r
  if (inverse) {
    dc_hilo_store<T>(w.dc_in);  // used after the barriers below
    C v[RY];
#pragma unroll
    for (int r = 0; r < RY; ++r) v[r] = __ldcg(spec + (j + GY * r) * H);
    if (c == 0) {  // column 0 carries a_0 + i a_h
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        const C b = __ldcg(spec + NY * H + (j + GY * r));
        v[r] = C{v[r].x - b.y, v[r].y + b.x};
      }
    }
    Dft<RY, true, C>::run(v);
#pragma unroll
    for (int r = 0; r < RY; ++r) slot_j[r * S] = v[r];
    group_sync<P::NG, CG * GY>(g);
#pragma unroll
    for (int u = 0; u < UY; ++u) {
      const int jp = j + u * GY;
      if (RY % GY == 0 || jp < RY) {
        C b[GY];
        C* const row = buf + jp * S;
#pragma unroll
        for (int r = 0; r < GH; ++r) {
          b[r] = row[r * RY * S + c];
          b[r + GH] = row[r * RY * S + mc];
        }
#pragma unroll
        for (int r = 1; r < GY; ++r) b[r] = cmulc(b[r], s_tw_y[r * jp]);
        Dft<GY, true, C>::run(b);
        // rows y = jp + RY r (a) and y + ny/2 (a2): column c of the packed row is
        // a + i a2, its mirror conj(a) + i conj(a2)
#pragma unroll
        for (int r = 0; r < GH; ++r) {
          const C a = b[r], a2 = b[r + GH];
          row[r * RY * S + c] = (c == 0) ? C{a.x, a2.x} : C{a.x - a2.y, a.y + a2.x};
          row[r * RY * S + mc] = (c == 0) ? C{a.y, a2.y} : C{a.x + a2.y, a2.x - a.y};
        }
      }
    }
    __syncthreads();  // every row complete
  }

  if constexpr (EARLY) pdl_trigger();
  // z rows: inverse, real-space step, forward
  T acc = T(0);
  const AdjPoint* const point = ADJ ? adj.points + blockIdx.y : nullptr;
  AdjGlobals globals{0.0, 0.0};
  if constexpr (ADJ) {
    if (adj_on) {
      globals.inv_q = 1.0 / *adj.q;
      globals.gq_n = *adj.gq / adj.n;
    }
  }
#pragma unroll 1
  for (int task = tid; task < P::TASKS; task += TH) {
    const int b = task / GZ, jz = task % GZ;
    const int j0 = jz * UZ;  // this thread's radix-GZ butterflies j0 .. j0 + UZ - 1
    C* const row = buf + b * S;
    const size_t ra = roff + (size_t)b * NZ + j0;  // the pair's first real row, z = j0
    const bool on = (RZ % GZ == 0) || j0 < RZ;
    C q[UZ][GZ];
    // the Boltzmann factors (FIRST: the initial q) of CH positions at a time: the
    // first ones are loaded ahead of the exchange, the next while the previous
    // ones are used
    const T* const lead = inverse ? w.wfac_in : w.src;
    const bool lead_on = on && lead;
    RealRun<T, UZ> f[2][CH], f2[2][CH];
    auto load_lead = [&](int s, int r0) {
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        f[s][i].ones();
        f2[s][i].ones();
        if (lead_on) {
          f[s][i].load(lead + ra + RZ * (r0 + i));
          f2[s][i].load(lead + ra + (size_t)PR * NZ + RZ * (r0 + i));
        }
      }
    };
    load_lead(0, 0);
    // ADJ: the pointwise streams, where registers allow one chunk ahead
    constexpr bool AHEAD = ADJ && UZ == 1;
    AdjRuns<UZ, ADJ ? 2 * CH : 1> runs[AHEAD ? 2 : 1];
    auto adj_load = [&](int i, int r0) {
      if constexpr (ADJ) {
        size_t at[2 * CH];
#pragma unroll
        for (int k = 0; k < CH; ++k) {
          at[2 * k] = ra + RZ * (r0 + k);
          at[2 * k + 1] = at[2 * k] + (size_t)PR * NZ;
        }
        runs[i].load(*point, at);
      }
    };
    if constexpr (AHEAD) {
      if (adj_on && on) adj_load(0, 0);
    }
    if (inverse) {
      C v[RZ];
#pragma unroll
      for (int r = 0; r < RZ; ++r) v[r] = row[jz + GZ * r];
      __syncwarp();
      Dft<RZ, true, C>::run(v);
      if constexpr (P::V2) {
#pragma unroll
        for (int r = 0; r < RZ; r += 2)
          *reinterpret_cast<float4*>(row + jz * PA + r) = make_float4(v[r].x, v[r].y, v[r + 1].x, v[r + 1].y);
      } else {
#pragma unroll
        for (int r = 0; r < RZ; ++r) row[jz * PA + r] = v[r];
      }
      __syncwarp();
      if (on) {
#pragma unroll
        for (int r = 0; r < GZ; ++r) {
          if constexpr (P::V2 && UZ == 2) {
            const float4 x = *reinterpret_cast<const float4*>(row + r * PA + j0);
            q[0][r] = C{x.x, x.y};
            q[UZ - 1][r] = C{x.z, x.w};
          } else {
#pragma unroll
            for (int u = 0; u < UZ; ++u) q[u][r] = row[r * PA + j0 + u];
          }
        }
#pragma unroll
        for (int u = 0; u < UZ; ++u) {
#pragma unroll
          for (int r = 1; r < GZ; ++r) q[u][r] = cmulc(q[u][r], s_twb[r * RZ + j0 + u]);
          Dft<GZ, true, C>::run(q[u]);
        }
      }
    } else {
#pragma unroll
      for (int u = 0; u < UZ; ++u)
#pragma unroll
        for (int r = 0; r < GZ; ++r) q[u][r] = C{T(1), T(1)};
    }
    if (on) {
      const bool same = (w.wfac_in == w.wfac_out) && inverse;
      const bool dc_in = inverse && w.dc_in;
#pragma unroll
      for (int r0 = 0; r0 < GZ; r0 += CH) {
        const int s = (r0 / CH) & 1;
        if (r0 + CH < GZ) load_lead(s ^ 1, r0 + CH);
RealRun<T, UZ> xs[2 * CH];  // the rows' values at the chunk's positions
        size_t at[2 * CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) {
          const int r = r0 + i;
          at[2 * i] = ra + RZ * r;
          at[2 * i + 1] = at[2 * i] + (size_t)PR * NZ;
#pragma unroll
          for (int u = 0; u < UZ; ++u) {
            const C a = dc_in ? dc_add2<T>(q[u][r]) : q[u][r];
            xs[2 * i].v[u] = a.x * f[s][i].v[u];
            xs[2 * i + 1].v[u] = a.y * f2[s][i].v[u];
          }
        }
        if constexpr (ADJ) {
          if (adj_on) {
            if (AHEAD && r0 + CH < GZ) adj_load((r0 / CH + 1) & 1, r0 + CH);
            if (!AHEAD) adj_load(0, r0);
            runs[AHEAD ? (r0 / CH) & 1 : 0].apply(*point, globals, at, inverse, xs);
          }
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) {
          const int r = r0 + i;
          if (w.store) {
            xs[2 * i].store(w.store + at[2 * i]);
            xs[2 * i + 1].store(w.store + at[2 * i + 1]);
          }
          if (!same) {
            f[s][i].ones();
            f2[s][i].ones();
            if (w.wfac_out && forward) {
              f[s][i].load(w.wfac_out + at[2 * i]);
              f2[s][i].load(w.wfac_out + at[2 * i + 1]);
            }
          }
#pragma unroll
          for (int u = 0; u < UZ; ++u) q[u][r] = C{xs[2 * i].v[u] * f[s][i].v[u], xs[2 * i + 1].v[u] * f2[s][i].v[u]};
        }
      }
      if (forward) {
#pragma unroll
        for (int u = 0; u < UZ; ++u) {
          Dft<GZ, false, C>::run(q[u]);
          acc += q[u][0].x + q[u][0].y;  // the sum of this butterfly's inputs (mean-mode carry)
        }
#pragma unroll
        for (int r = 0; r < GZ; ++r) {
          if constexpr (P::V2 && UZ == 2) {
            *reinterpret_cast<float4*>(row + r * PA + j0) =
                make_float4(q[0][r].x, q[0][r].y, q[UZ - 1][r].x, q[UZ - 1][r].y);
          } else {
#pragma unroll
            for (int u = 0; u < UZ; ++u) row[r * PA + j0 + u] = q[u][r];
          }
        }
      }
    }
    if (!forward) continue;
    __syncwarp();
    C v[RZ];
    if constexpr (P::V2) {
#pragma unroll
      for (int r = 0; r < RZ; r += 2) {
        const float4 x = *reinterpret_cast<const float4*>(row + jz * PA + r);
        v[r] = C{x.x, x.y};
        v[r + 1] = C{x.z, x.w};
      }
    } else {
#pragma unroll
      for (int r = 0; r < RZ; ++r) v[r] = row[jz * PA + r];
    }
#pragma unroll
    for (int r = 1; r < RZ; ++r) v[r] = cmul(v[r], s_twf[r * GZ + jz]);
    Dft<RZ, false, C>::run(v);
    __syncwarp();
#pragma unroll
    for (int r = 0; r < RZ; ++r) row[jz + GZ * r] = v[r];
  }
  if (!forward) return;  // uniform over the CTA
  if (dc_sum) dc_warp_sum((double)acc);
  __syncthreads();  // every column complete

#pragma unroll
  for (int u = 0; u < UY; ++u) {
    const int jp = j + u * GY;
    if (RY % GY == 0 || jp < RY) {
      C b[GY];
      C* const row = buf + jp * S;
      // twice the two rows' transforms: a = z + conj(z'), a2 = -i (z - conj(z'))
      // (column 0: the real columns 0 and nz/2 as they are, for x_0 + i x_h)
#pragma unroll
      for (int r = 0; r < GH; ++r) {
        const C z = row[r * RY * S + c], m = row[r * RY * S + mc];
        b[r] = (c == 0) ? C{z.x, m.x} : C{z.x + m.x, z.y - m.y};
        b[r + GH] = (c == 0) ? C{z.y, m.y} : C{z.y + m.y, m.x - z.x};
      }
      Dft<GY, false, C>::run(b);
#pragma unroll
      for (int r = 0; r < GH; ++r) {
        row[r * RY * S + c] = b[r];
        row[r * RY * S + mc] = b[r + GH];
      }
    }
  }
  group_sync<P::NG, CG * GY>(g);
  C v[RY];
#pragma unroll
  for (int r = 0; r < RY; ++r) v[r] = slot_j[r * S];
#pragma unroll
  for (int r = 1; r < RY; ++r) v[r] = cmul(v[r], s_tw_y[r * j]);
  Dft<RY, false, C>::run(v);
  if (g == 0) {
    // column 0 holds the transform of x_0 + i x_h: split it by Hermitian
    // symmetry (twice the two transforms, as everywhere)
    if (c == 0) {
#pragma unroll
      for (int r = 0; r < RY; ++r) s_nyq[j + GY * r] = v[r];
    }
    group_sync<P::NG, CG * GY>(g);
    if (c == 0) {
#pragma unroll
      for (int r = 0; r < RY; ++r) {
        const int k = j + GY * r;
        const C d = s_nyq[(NY - k) % NY];
        const C a = v[r];
        v[r] = C{a.x + d.x, a.y - d.y};
        __stcg(spec + NY * H + k, C{a.y + d.y, d.x - a.x});
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RY; ++r) __stcg(spec + (j + GY * r) * H, v[r]);
  if (dc_sum) dc_cta_store(works + blockIdx.y);
}

template <typename T, int NY, int NZ>
cudaError_t launch_step_plane_t(const PlaneWork<T>* d_works, int nworks, int nx, bool early, const c2_t<T>* tw_y,
                                const c2_t<T>* tw_z, cudaStream_t st) {
  using P = StepPlane<T, NY, NZ>;
  if constexpr (P::CAN_EARLY) {
    if (early) {
      auto kern = step_plane_kernel<T, NY, NZ, false, true>;
      static unsigned attr_mask = 0;
      cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
      if (e != cudaSuccess) return e;
      return launch_sweep_kernel(kern, dim3(nx, nworks), dim3(P::TH), P::SMEM, st, d_works, tw_y, tw_z, AdjArgs{});
    }
  }
  auto kern = step_plane_kernel<T, NY, NZ, false, false>;
  static unsigned attr_mask = 0;
  cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
  if (e != cudaSuccess) return e;
  return launch_sweep_kernel(kern, dim3(nx, nworks), dim3(P::TH), P::SMEM, st, d_works, tw_y, tw_z, AdjArgs{});
}

// Planes of NY rows, for every nz of kStepExtents (one translation unit per NY).
template <typename T, int NY>
cudaError_t launch_step_plane_ny(const PlaneWork<T>* w, int nw, int nx, int nz, bool early, const c2_t<T>* ty,
                                 const c2_t<T>* tz, cudaStream_t st) {
  switch (nz) {
    case 16: return launch_step_plane_t<T, NY, 16>(w, nw, nx, early, ty, tz, st);
    case 24: return launch_step_plane_t<T, NY, 24>(w, nw, nx, early, ty, tz, st);
    case 32: return launch_step_plane_t<T, NY, 32>(w, nw, nx, early, ty, tz, st);
    case 48: return launch_step_plane_t<T, NY, 48>(w, nw, nx, early, ty, tz, st);
    case 64: return launch_step_plane_t<T, NY, 64>(w, nw, nx, early, ty, tz, st);
    case 96: return launch_step_plane_t<T, NY, 96>(w, nw, nx, early, ty, tz, st);
    case 128: return launch_step_plane_t<T, NY, 128>(w, nw, nx, early, ty, tz, st);
  }
  return cudaErrorInvalidValue;
}
#define PSB_STEP_PLANE_NY(PREFIX, NY)                                                                             \
  PREFIX template cudaError_t launch_step_plane_ny<float, NY>(const PlaneWork<float>*, int, int, int, bool,       \
                                                              const float2*, const float2*, cudaStream_t);        \
  PREFIX template cudaError_t launch_step_plane_ny<double, NY>(const PlaneWork<double>*, int, int, int, bool,     \
                                                               const double2*, const double2*, cudaStream_t);

}  // namespace psb
