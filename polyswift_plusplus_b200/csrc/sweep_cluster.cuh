// A whole propagator sweep in one launch, for grids whose half spectrum fits the
// shared memory of one thread-block cluster.
//
// What bounded small grids: two launches a step, each a chain of loads, exchanges
// and stores of a few microseconds on a few CTAs (32^3: 5.5 us a step for 0.3 us of
// arithmetic).  Here a cluster of CL CTAs runs every step of one sweep and keeps
// the spectrum in shared memory: CTA m owns the planes x in [m PX, (m + 1) PX) for
// the y and z transforms and the real-space step, and COLS (ky, kz) columns for the
// x transforms.  The last y butterflies write straight into the column owners'
// shared memory and the last x butterflies into the plane owners' (asynchronous
// stores counted on the owner's mbarrier): nothing but the propagator slices goes to global memory, and
// the Boltzmann factors stay in registers while the sweep stays in a block.
//
// The passes are those of step_plane.cuh (packed row pairs, group-local exchanges)
// and step_pencil.cu.  A film (ny = 1) pairs its rows along x and has no y part.
#pragma once

#include "step_plane.cuh"
#include "tma.cuh"

namespace psb {

__device__ __forceinline__ uint32_t cl_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// This CTA's shared-memory address of p, in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cl_addr(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
// Asynchronous stores into another CTA's shared memory; their bytes count on
// that CTA's mbarrier.  A release (cluster barrier, fence) instead of the count
// would also wait for the slices on their way to global memory: 30% of the time of
// a first version.
__device__ __forceinline__ void cl_store(uint32_t addr, uint32_t bar, float2 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "f"(v.x), "f"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t addr, uint32_t bar, double2 v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "d"(v.x), "d"(v.y), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t addr, uint32_t bar, double v) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}
// A plain store of 1; a cluster barrier makes it visible.
__device__ __forceinline__ void cl_store_flag(uint32_t addr) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(1) : "memory");
}
// Bounded wait for a phase whose data other CTAs of the cluster wrote.
__device__ __forceinline__ bool cl_wait(uint64_t* bar, uint32_t parity, uint32_t polls) {
  for (uint32_t i = 0; i < polls; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// The threads of one plane.
template <bool CTA, int THREADS> __device__ __forceinline__ void plane_sync(int pl) {
  if constexpr (CTA) __syncthreads();
  else asm volatile("bar.sync %0, %1;" ::"r"(pl + 1), "n"(THREADS) : "memory");
}

template <typename T, int NX, int NY, int NZ, int CL_> struct SweepCl {
  static constexpr int CL = CL_, H = NZ / 2;
  static constexpr bool FILM = (NY == 1);
  static constexpr int PX = NX / CL;                    // planes (film: rows) of a CTA
  static constexpr int PR = FILM ? PX / 2 : NY / 2;     // packed rows of a plane (film: of the CTA)
  static constexpr int NP = FILM ? 1 : PX;              // plane buffers
  // four threads a column leave no lane idle at ny = 16 and 32 (32^3 FP64: 4.60 us a
  // step, 4.84 with eight)
  static constexpr int GY = (NY == 16 || NY == 32) ? 4 : GroupOf<NY>::v, RY = FILM ? 1 : NY / GY, UY = (RY + GY - 1) / GY;
  static constexpr int GZ = (NZ < 16) ? 4 : RowGroup<PR, NZ>::v, RZ = NZ / GZ, UZ = (RZ + GZ - 1) / GZ;
  static constexpr int GX = (NX >= 64) ? 16 : 4, RX = NX / GX, UX = (RX + GX - 1) / GX;
  static constexpr bool V2 = sizeof(T) == 4 && RZ % 2 == 0;
  static constexpr int PA = V2 ? ((RZ / 2) % 2 ? RZ : RZ + 2) : RZ + 1;
  static constexpr int S0 = GZ * PA;
  static constexpr int S = (sizeof(T) == 4) ? S0 + ((24 - S0 % 16) % 16) : S0;
  static constexpr int NCOL = NY * (H + 1);
  // CTA m owns the columns from col0(m) to col0(m + 1), the last one also what is left
  // over (a film's Nyquist column), and none owns nothing: what a CTA sends from its
  // columns is what keeps the others from running into the next step while it is still
  // in this one (see bar_a and bar_b below).
  static constexpr int EACH = NCOL / CL, COLS = NCOL - EACH * (CL - 1);  // COLS: at most
  static constexpr __host__ __device__ int col0(int m) { return m < CL ? m * EACH : NCOL; }
  static constexpr __host__ __device__ int owner(int col) {
    return (COLS == EACH || col < EACH * CL) ? col / EACH : CL - 1;
  }
  // threads of a plane's z rows and of a plane: whole warps.  At nz < 16 the last
  // warp has lanes without a row (they take PRB - PR spare rows of the buffer along)
  // or without a column.
  static constexpr int ROWT = (PR * GZ + 31) / 32 * 32, PRB = ROWT / GZ;
  static constexpr int COLT = FILM ? 0 : (H * GY + 31) / 32 * 32;
  static constexpr int PTH = COLT > ROWT ? COLT : ROWT;
  static constexpr int TH0 = NP * PTH, THX = COLS * GX;
  static constexpr int TH1 = TH0 > THX ? TH0 : THX;
  static constexpr int TH = (TH1 + 31) / 32 * 32;
  static constexpr int BUF = NP * PRB * S, AIN = PX * NCOL, BIN = NX * COLS;
  static constexpr size_t SMEM =
      sizeof(c2_t<T>) * ((size_t)BUF + AIN + 2 * BIN + NP * NY + NX + NX / 2 + NY + NZ) +
      sizeof(double) * (CL * (TH / 32) + 1) + 2 * sizeof(uint64_t) + sizeof(int);
  static_assert(PX * CL == NX && TH <= 1024 && PRB * GZ == ROWT && (!FILM || PRB == PR), "cluster sweep layout");
  static_assert(S >= NZ && RZ * GZ == NZ && RX * GX == NX && (FILM || RY * GY == NY) && UZ <= 2, "cluster sweep layout");
  static_assert(NP <= 15 && (!FILM || PX % 2 == 0) && CL * 2 <= TH, "cluster sweep layout");
  // the bytes of two phases are within an mbarrier's transaction count
  static_assert(2 * (sizeof(c2_t<T>) * (AIN > BIN ? AIN : BIN) + sizeof(double) * CL * (TH / 32)) < (1u << 20),
                "cluster sweep phases");
  static_assert(EACH >= 1 && COLS <= EACH + 1, "every CTA owns columns, as many as the others or one more");
};

// The grids that have one: (nx, ny, nz, CTAs of the cluster), a film nx x ny x 1 as
// (nx, 1, ny).  One plane or a few rows per CTA, as many CTAs as a cluster may have: us
// per step of both sweeps, FP64 (FP32), against the step passes' two launches:
//   8^3 1.3 (1.4), 12^3 1.7 (1.6)      passes 5.6 and 6.3 (7.0)
//   16^3 1.8 (1.8), eight CTAs 1.9     passes 4.6
//   24^3 3.6 (2.7), eight CTAs 4.6 (3.3), passes 5.7
//   32^3 4.5 (3.2), passes 5.5 (5.0)
//   films, eight rows a CTA: 24^2 1.6 (1.6), passes 10 (12); 48^2 2.1 (1.9), 11 (13);
//   64^2 2.2 (1.9), 4.9; 96^2 3.6 (2.7), 16 (19); 128^2 3.8 (3.1), eight CTAs 4.5, passes 6.4
// 48^3 has too much work for 16 SMs per sweep: FP32 9.0 against 7.3.
#define PSB_SWEEP_GRIDS(X)                                        \
  X(8, 8, 8, 8) X(12, 12, 12, 12) X(16, 16, 16, 16)               \
  X(24, 24, 24, 12) X(32, 32, 32, 16) X(16, 1, 16, 2)             \
  X(24, 1, 24, 3) X(32, 1, 32, 4) X(48, 1, 48, 6)                 \
  X(64, 1, 64, 8) X(96, 1, 96, 12) X(128, 1, 128, 16)

// Poll limit of the waits below (see ps_gpu_set_bulk_wait_limit).
static __constant__ uint32_t c_sweep_wait_polls = kMaxPolls;

// DST: the slices' places come from w.dst (1% of a step at 16^3 as a run-time choice).
template <typename T, int NX, int NY, int NZ, int CL_, bool DST>
__global__ void __launch_bounds__((SweepCl<T, NX, NY, NZ, CL_>::TH), 1)
    sweep_cluster_kernel(const SweepWork<T>* __restrict__ works, const c2_t<T>* __restrict__ tw_x,
                         const c2_t<T>* __restrict__ tw_y, const c2_t<T>* __restrict__ tw_z) {
  using P = SweepCl<T, NX, NY, NZ, CL_>;
  using C = c2_t<T>;
  constexpr int CL = P::CL, H = P::H, PX = P::PX, PR = P::PR, NP = P::NP, S = P::S, PA = P::PA, TH = P::TH;
  constexpr int GY = P::GY, RY = P::RY, UY = P::UY, GZ = P::GZ, RZ = P::RZ, UZ = P::UZ;
  constexpr int GX = P::GX, RX = P::RX, UX = P::UX, NCOL = P::NCOL, COLS = P::COLS, PTH = P::PTH;
  constexpr bool FILM = P::FILM;
  constexpr int W = TH / 32;
  constexpr int GH = GY / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);  // packed rows of the planes
  C* a_in = buf + P::BUF;                   // [plane][column]: from the x part
  C* b_in = a_in + P::AIN;                  // [x][column]: from the y (film: z) part
  C* b_ex = b_in + P::BIN;                  // exchange of the x part
  C* s_nyq = b_ex + P::BIN;
  C* s_tw_x = s_nyq + NP * NY;
  C* s_tw_y = s_tw_x + NX;
  C* s_tw_z = s_tw_y + NY;
  T* s_kx = reinterpret_cast<T*>(s_tw_z + NZ);              // x factors of the current block (NX / 2 complex of room)
  double* s_part = reinterpret_cast<double*>(s_tw_z + NZ + NX / 2);  // every warp's sum of the forward input, by CTA
  double* s_mean = s_part + CL * W;                         // the mean-mode value of the inverse
  uint64_t* bar_a = reinterpret_cast<uint64_t*>(s_mean + 1);  // a_in written
  uint64_t* bar_b = bar_a + 1;                                // b_in (and s_part) written
  int* s_stop = reinterpret_cast<int*>(bar_b + 1);            // a wait ran out in this cluster

  const SweepWork<T>& w = works[blockIdx.y];
  const int tid = threadIdx.x;
  const uint32_t me = cl_rank();
  const int x0 = (int)me * PX;
  for (int i = tid; i < NX; i += TH) s_tw_x[i] = tw_x[i];
  for (int i = tid; i < NY; i += TH) s_tw_y[i] = tw_y[i];
  for (int i = tid; i < NZ; i += TH) s_tw_z[i] = tw_z[i];
  const int total = w.total;
  const bool dc = w.dc != 0;

  // y part: plane pl, column c, butterfly j (film: none)
  const int pl = tid / PTH, tp = tid - pl * PTH;
  const bool in_plane = pl < NP;
  const int c = FILM ? 0 : tp % H, j = FILM ? 0 : tp / H;
  const bool in_y = (PTH == H * GY) || j < GY;
  const int mc = (c == 0) ? H : NZ - c;
  C* const pbuf = buf + (in_plane ? pl : 0) * (P::PRB * S);
  // z part: row b of the plane's packed rows
  const bool in_row = in_plane && tp < P::ROWT;
  const int b = tp / GZ, jz = tp % GZ, j0 = jz * UZ;
  const bool on = in_row && (P::PRB == PR || b < PR) && ((RZ % GZ == 0) || j0 < RZ);
  C* const row = pbuf + b * S;
  // the pair's real rows in memory: y and y + ny/2 of plane x0 + pl (film: x and x + PX/2)
  const size_t ra = (FILM ? (size_t)(x0 + b) * NZ : ((size_t)(x0 + pl) * NY + b) * NZ) + j0;
  constexpr size_t RB = (size_t)PR * NZ;
  // x part: column cc of this CTA, butterfly jx
  const int cc = tid % COLS, jx = tid / COLS;
  const int gcols0 = P::col0((int)me);
  const int my_cols = P::col0((int)me + 1) - gcols0;
  const int gc = gcols0 + cc;
  const bool in_col = jx < GX && cc < my_cols;

  int seg = 0, seg_end = w.seg[0].end;
  T* const slices = w.slices;
  const double dc_scale = w.dc_scale;
  T fyz = T(0);  // this column's k^2 factor in the current block; the x factors are in s_kx
  auto load_ktab = [&](int i) {
    if (in_col) fyz = __ldg(w.seg[i].kyzc + gc);
    for (int x = tid; x < NX; x += TH) s_kx[x] = __ldg(w.seg[i].kx + x);
  };
  RealRun<T, UZ> f[GZ], f2[GZ];  // Boltzmann factors of the current block
  auto load_factors = [&](const T* p) {
#pragma unroll
    for (int r = 0; r < GZ; ++r) {
      f[r].ones();
      f2[r].ones();
      if (on && p) {
        f[r].load(p + ra + RZ * r);
        f2[r].load(p + ra + RB + RZ * r);
      }
    }
  };
  double dc_err = 0.0;
  // A phase of bar_a or bar_b completes when thread 0 has armed it and every byte has
  // arrived.  Phases cannot overlap: a CTA sends its part of bar_b's next phase after its
  // bar_a has the columns of every CTA, which each sends after its own bar_b phase (and
  // after its warps have read s_part); and its part of bar_a's next phase after its bar_b
  // has rows of every CTA, which each sends after its own bar_a phase.
  const uint32_t bytes_a = (uint32_t)(P::AIN * sizeof(C));
  const uint32_t bytes_b = (uint32_t)(NX * my_cols * sizeof(C)) + (dc ? (uint32_t)(CL * W * sizeof(double)) : 0u);
  if (tid == 0) {
    *s_stop = 0;
    mbar_init(bar_a, 1);
    mbar_init(bar_b, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(bar_a, bytes_a);
    mbar_arrive_expect_tx(bar_b, bytes_b);
  }
  // A wait that runs out sets the error flag and stops its CTA before it sends anything
  // from its columns.  The bar_a phases that lack them stay incomplete, so that the other
  // CTAs' waits run out too: within a step nobody sends, and no barrier counts more than the
  // bytes of two phases (were a CTA to go on for the rest of the sweep, 60 steps at 32^3
  // would pass what an mbarrier can count).
  const uint32_t polls = c_sweep_wait_polls;
  bool failed = false;
  auto wait = [&](uint64_t* bar, uint32_t phase, uint32_t bytes, bool rearm) {
    if (failed) return;
    if (!cl_wait(bar, phase & 1u, polls)) {
      failed = true;
      *reinterpret_cast<volatile int*>(s_stop) = 1;  // waits come before a step's first CTA barrier in the x part
      if (w.status) atomicOr(w.status, 4);
    } else if (rearm && tid == 0) {
      mbar_arrive_expect_tx(bar, bytes);
    }
  };
  cl_sync();  // every CTA of the cluster runs, its barriers are armed and the tables are written
  pdl_wait();
  load_factors(w.seg[0].wfac);
  load_ktab(0);

  for (int k = 0; k <= total; ++k) {
    T* slice = nullptr;
    if constexpr (DST) slice = w.dst[k];
    // ---- y inverse -------------------------------------------------------
    if (k > 0) wait(bar_a, (uint32_t)(k - 1), bytes_a, k < total);
    if (!FILM && k > 0) {
      if (in_plane) {
        if (in_y) {
          const C* const src = a_in + pl * NCOL + c;
          C v[RY];
#pragma unroll
          for (int r = 0; r < RY; ++r) v[r] = src[(j + GY * r) * H];
          if (c == 0) {
#pragma unroll
            for (int r = 0; r < RY; ++r) {
              const C n = src[NY * H + (j + GY * r)];
              v[r] = C{v[r].x - n.y, v[r].y + n.x};
            }
          }
          Dft<RY, true, C>::run(v);
          C* const slot_j = pbuf + (j % GH) * RY * S + (j < GH ? c : mc);
#pragma unroll
          for (int r = 0; r < RY; ++r) slot_j[r * S] = v[r];
        }
        plane_sync<TH == PTH, PTH>(pl);
#pragma unroll
        for (int u = 0; u < UY; ++u) {
          const int jp = j + u * GY;
          if (in_y && (RY % GY == 0 || jp < RY)) {
            C q[GY];
            C* const r0 = pbuf + jp * S;
#pragma unroll
            for (int r = 0; r < GH; ++r) {
              q[r] = r0[r * RY * S + c];
              q[r + GH] = r0[r * RY * S + mc];
            }
#pragma unroll
            for (int r = 1; r < GY; ++r) q[r] = cmulc(q[r], s_tw_y[r * jp]);
            Dft<GY, true, C>::run(q);
#pragma unroll
            for (int r = 0; r < GH; ++r) {
              const C a = q[r], a2 = q[r + GH];
              r0[r * RY * S + c] = (c == 0) ? C{a.x, a2.x} : C{a.x - a2.y, a.y + a2.x};
              r0[r * RY * S + mc] = (c == 0) ? C{a.y, a2.y} : C{a.x + a2.y, a2.x - a.y};
            }
          }
        }
        plane_sync<TH == PTH, PTH>(pl);  // the plane's rows complete
      }
    }
    // ---- z inverse, real-space step, z forward ----------------------------
    T acc = T(0);
    if (in_row) {
      C q[UZ][GZ];
      if (k > 0) {
        C v[RZ];
        if constexpr (FILM) {
          // columns of the two rows: z = a + i a2, mirror conj(a) + i conj(a2)
          const C* const a1 = a_in + b * NCOL;
          const C* const a2 = a1 + PR * NCOL;
#pragma unroll
          for (int r = 0; r < RZ; ++r) {
            const int kz = jz + GZ * r;
            const int m = (kz <= H) ? kz : NZ - kz;
            const C p = a1[m], s = a2[m];
            v[r] = (kz <= H) ? C{p.x - s.y, p.y + s.x} : C{p.x + s.y, s.x - p.y};
          }
        } else {
#pragma unroll
          for (int r = 0; r < RZ; ++r) v[r] = row[jz + GZ * r];
          __syncwarp();
        }
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
          const T m = dc ? T(*s_mean) : T(0);
#pragma unroll
          for (int u = 0; u < UZ; ++u) {
#pragma unroll
            for (int r = 1; r < GZ; ++r) q[u][r] = cmulc(q[u][r], s_tw_z[r * (j0 + u)]);
            Dft<GZ, true, C>::run(q[u]);
            if (dc) {
#pragma unroll
              for (int r = 0; r < GZ; ++r) q[u][r] = C{q[u][r].x + m, q[u][r].y + m};
            }
          }
#pragma unroll
          for (int r = 0; r < GZ; ++r)
#pragma unroll
            for (int u = 0; u < UZ; ++u) q[u][r] = C{q[u][r].x * f[r].v[u], q[u][r].y * f2[r].v[u]};
        }
      } else {
#pragma unroll
        for (int r = 0; r < GZ; ++r) {
          RealRun<T, UZ> x, x2;
          x.ones();
          x2.ones();
          if (on && w.src) {
            x.load(w.src + ra + RZ * r);
            x2.load(w.src + ra + RB + RZ * r);
          }
#pragma unroll
          for (int u = 0; u < UZ; ++u) q[u][r] = C{x.v[u], x2.v[u]};
        }
      }
      if (on && (!DST || slice)) {
        T* const st = (DST ? slice : slices + (size_t)k * ((size_t)NX * NY * NZ)) + ra;
#pragma unroll
        for (int r = 0; r < GZ; ++r) {
          RealRun<T, UZ> x, x2;
#pragma unroll
          for (int u = 0; u < UZ; ++u) {
            x.v[u] = q[u][r].x;
            x2.v[u] = q[u][r].y;
          }
          x.store(st + RZ * r);
          x2.store(st + RB + RZ * r);
        }
      }
      if (k < total) {
        if (k == seg_end) load_factors(w.seg[seg + 1].wfac);
        if (on) {
#pragma unroll
          for (int u = 0; u < UZ; ++u) {
#pragma unroll
            for (int r = 0; r < GZ; ++r) q[u][r] = C{q[u][r].x * f[r].v[u], q[u][r].y * f2[r].v[u]};
            Dft<GZ, false, C>::run(q[u]);
            acc += q[u][0].x + q[u][0].y;
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
        for (int r = 1; r < RZ; ++r) v[r] = cmul(v[r], s_tw_z[r * jz]);
        Dft<RZ, false, C>::run(v);
        __syncwarp();
#pragma unroll
        for (int r = 0; r < RZ; ++r) row[jz + GZ * r] = v[r];
      }
    }
    if (k == total) break;  // uniform over the cluster (bar_b keeps an armed phase: never waited for)
    if (k == seg_end) {  // the next block
      seg_end = w.seg[++seg].end;
      load_ktab(seg);  // read after the x part's first barrier, last read before this step's
    }
    if (dc) {  // this warp's sum, to every CTA
      double v = (double)acc;
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      if ((tid & 31) < CL) cl_store(cl_addr(s_part + me * W + (tid >> 5), tid & 31), cl_addr(bar_b, tid & 31), v);
    }

    // ---- y forward, into the column owners' shared memory -----------------
    if constexpr (!FILM) {
      if (in_plane) {
        plane_sync<TH == PTH, PTH>(pl);  // the plane's columns complete
#pragma unroll
        for (int u = 0; u < UY; ++u) {
          const int jp = j + u * GY;
          if (in_y && (RY % GY == 0 || jp < RY)) {
            C q[GY];
            C* const r0 = pbuf + jp * S;
#pragma unroll
            for (int r = 0; r < GH; ++r) {
              const C z = r0[r * RY * S + c], m = r0[r * RY * S + mc];
              q[r] = (c == 0) ? C{z.x, m.x} : C{z.x + m.x, z.y - m.y};
              q[r + GH] = (c == 0) ? C{z.y, m.y} : C{z.y + m.y, m.x - z.x};
            }
            Dft<GY, false, C>::run(q);
#pragma unroll
            for (int r = 0; r < GH; ++r) {
              r0[r * RY * S + c] = q[r];
              r0[r * RY * S + mc] = q[r + GH];
            }
          }
        }
        plane_sync<TH == PTH, PTH>(pl);
        C v[RY];
        C* const ny = s_nyq + pl * NY;
        if (in_y) {
          const C* const slot_j = pbuf + (j % GH) * RY * S + (j < GH ? c : mc);
#pragma unroll
          for (int r = 0; r < RY; ++r) v[r] = slot_j[r * S];
#pragma unroll
          for (int r = 1; r < RY; ++r) v[r] = cmul(v[r], s_tw_y[r * j]);
          Dft<RY, false, C>::run(v);
          // column 0: separate the Nyquist column (c = 0 threads of all j meet)
          if (c == 0) {
#pragma unroll
            for (int r = 0; r < RY; ++r) ny[j + GY * r] = v[r];
          }
        }
        plane_sync<TH == PTH, PTH>(pl);
        if (in_y) {
          const int x = x0 + pl;
          if (c == 0) {
#pragma unroll
            for (int r = 0; r < RY; ++r) {
              const int ky = j + GY * r;
              const C d = ny[(NY - ky) % NY], a = v[r];
              v[r] = C{a.x + d.x, a.y - d.y};
              const int col = NY * H + ky, to = P::owner(col);
              cl_store(cl_addr(b_in + x * COLS + col - P::col0(to), to), cl_addr(bar_b, to), C{a.y + d.y, d.x - a.x});
            }
          }
#pragma unroll
          for (int r = 0; r < RY; ++r) {
            const int col = (j + GY * r) * H + c, to = P::owner(col);
            cl_store(cl_addr(b_in + x * COLS + col - P::col0(to), to), cl_addr(bar_b, to), v[r]);
          }
        }
      }
    } else {
      __syncthreads();  // rows complete (each row's lanes are one warp's; the unpacking crosses warps)
      for (int e = tid; e < PR * (H + 1); e += TH) {
        const int rb = e / (H + 1), kz = e - rb * (H + 1);
        const C z = buf[rb * S + kz], m = buf[rb * S + (kz == 0 || kz == H ? kz : NZ - kz)];
        const int to = P::owner(kz);
        C* const at = b_in + (x0 + rb) * COLS + kz - P::col0(to);
        const uint32_t bb = cl_addr(bar_b, to);
        cl_store(cl_addr(at, to), bb, C{z.x + m.x, z.y - m.y});
        cl_store(cl_addr(at + PR * COLS, to), bb, C{z.y + m.y, m.x - z.x});
      }
    }

    // ---- x part ----------------------------------------------------------
    wait(bar_b, (uint32_t)k, bytes_b, true);  // every column complete
    if (dc && tid >= TH - 32) {
      // the same sum in the same order on every CTA; what the rounding to T drops
      // comes back in the next step (PlaneWork in kernels.h)
      double s = 0.0;
      for (int i = tid & 31; i < CL * W; i += 32) s += s_part[i];
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      const double m = s * dc_scale + dc_err;
      if (tid == TH - 1) *s_mean = m;
      dc_err = m - (double)T(m);
    }
    if (in_col) {
      C v[RX];
      C* const ex = b_ex + cc;
#pragma unroll
      for (int r = 0; r < RX; ++r) v[r] = b_in[(jx + GX * r) * COLS + cc];
      Dft<RX, false, C>::run(v);
#pragma unroll
      for (int r = 0; r < RX; ++r) ex[(jx * RX + r) * COLS] = v[r];
    }
    __syncthreads();
    const int stop = *reinterpret_cast<volatile int*>(s_stop);  // between two barriers: the same for every thread
    if (in_col) {
      C* const ex = b_ex + cc;
#pragma unroll
      for (int u = 0; u < UX; ++u) {
        const int jp = jx + u * GX;
        if (RX % GX == 0 || jp < RX) {
          C q[GX];
#pragma unroll
          for (int r = 0; r < GX; ++r) q[r] = ex[(r * RX + jp) * COLS];
#pragma unroll
          for (int r = 1; r < GX; ++r) q[r] = cmul(q[r], s_tw_x[r * jp]);
          Dft<GX, false, C>::run(q);
#pragma unroll
          for (int r = 0; r < GX; ++r) {
            const T s = s_kx[jp + RX * r] * fyz;
            q[r] = C{q[r].x * s, q[r].y * s};
          }
          if (dc && gc == 0 && jp == 0) q[0] = C{T(0), T(0)};
          Dft<GX, true, C>::run(q);
#pragma unroll
          for (int r = 0; r < GX; ++r) ex[(r * RX + jp) * COLS] = q[r];
        }
      }
    }
    __syncthreads();
    if (stop) break;
    if (in_col) {
      const C* const ex = b_ex + cc;
      C v[RX];
#pragma unroll
      for (int r = 0; r < RX; ++r) v[r] = ex[(jx * RX + r) * COLS];
#pragma unroll
      for (int r = 1; r < RX; ++r) v[r] = cmulc(v[r], s_tw_x[r * jx]);
      Dft<RX, true, C>::run(v);
#pragma unroll
      for (int r = 0; r < RX; ++r) {
        const int x = jx + GX * r;
        cl_store(cl_addr(a_in + (x % PX) * NCOL + gc, x / PX), cl_addr(bar_a, x / PX), v[r]);
      }
    }
  }
  // No CTA leaves while another may still write to it.  After a wait that ran out, stores
  // may be on their way that nothing waits for: every CTA stays 200,000 cycles (about 100
  // us; a store between two SMs takes about one) after the last one has sent its last.
  __syncthreads();
  if (*s_stop && tid < CL) cl_store_flag(cl_addr(s_stop, tid));
  cl_sync();
  if (*s_stop) {
    for (const long long t0 = clock64(); clock64() - t0 < 200000;) __nanosleep(1000);
    cl_sync();
  }
}

template <typename T, int NX, int NY, int NZ, int CL, bool DST> struct SweepClLaunch {
  using P = SweepCl<T, NX, NY, NZ, CL>;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  static auto kernel() { return sweep_cluster_kernel<T, NX, NY, NZ, CL, DST>; }
  cudaError_t set(int nworks, cudaStream_t st) {
    static unsigned attr_mask = 0;
    cudaError_t e = ensure_smem_attr(kernel(), P::SMEM, &attr_mask);
    if (e != cudaSuccess) return e;
    if (CL > 8) {
      e = cudaFuncSetAttribute(kernel(), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
    }
    cfg.gridDim = dim3(CL, nworks);
    cfg.blockDim = dim3(P::TH);
    cfg.dynamicSmemBytes = P::SMEM;
    cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaSuccess;
  }
};

template <typename T, int NX, int NY, int NZ, int CL, bool DST>
cudaError_t launch_sweep_cluster_t(const SweepWork<T>* d_works, int nworks, const c2_t<T>* tx, const c2_t<T>* ty,
                                   const c2_t<T>* tz, cudaStream_t st) {
  SweepClLaunch<T, NX, NY, NZ, CL, DST> l;
  cudaError_t e = l.set(nworks, st);
  if (e != cudaSuccess) return e;
  return cudaLaunchKernelEx(&l.cfg, l.kernel(), d_works, tx, ty, tz);
}

// The device can place a cluster of this kernel: a part of it (a partition, a share given
// to the process) may have no 16 SMs that can form one.
template <typename T, int NX, int NY, int NZ, int CL, bool DST> bool sweep_cluster_fits_t() {
  SweepClLaunch<T, NX, NY, NZ, CL, DST> l;
  int clusters = 0;
  cudaError_t e = l.set(1, nullptr);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, l.kernel(), &l.cfg);
  if (e != cudaSuccess) cudaGetLastError();  // not this caller's error: the sweeps take the step passes
  return e == cudaSuccess && clusters > 0;
}

}  // namespace psb
