// Propagator step with the y transform split between the two passes, for y-z planes
// that one CTA cannot hold (256 x 256).
//
// y = j + J r and ky = k1 + 16 k2 (r, k1 < 16; j, k2 < J = ny / 16).  The plane pass
// does the z transforms and, in registers, the radix-16 part over r <-> k1 of JC of
// the J row classes j: a CTA needs 16 JC rows of a plane, not the plane.  The x pass
// does the radix-J part over j <-> k2 together with the x transform of all columns
// (k1, kz).  Both passes are chains of five register butterflies with four
// shared-memory exchanges; nothing crosses CTAs.  (The pass it replaces, one plane
// on a cluster of eight CTAs, sent the plane through distributed shared memory twice
// and ran three-pass transforms: 147 us of 179 for a 256^3 sweep step.)
//
// Spectrum layout: [x][k1][kz / KB][j][kz % KB], KB complex values of 32 bytes: the x
// pass reads J KB consecutive values per x, the plane pass JC KB.  The last kz block
// holds the nz/2 column and padding.  Packed row pairs, the doubled transform and
// the halved k^2 table kyzc are those of step_plane.cuh; the real columns 0 and nz/2
// share a radix-16 transform and are separated in registers (over r they are real
// sequences of their own).
#pragma once

#include "step_common.cuh"
#include "step_plane.cuh"
#include "tma.cuh"

namespace psb {

template <typename T> struct SplitKB { static constexpr int v = 32 / (2 * (int)sizeof(T)); };
constexpr int kSplitR = 16;
template <int NY> struct SplitJ { static constexpr int v = NY / kSplitR; };

template <typename T, int NY, int NZ> struct SplitPlane {
  static constexpr int H = NZ / 2, J = SplitJ<NY>::v, KB = SplitKB<T>::v;
  static constexpr int JC = sizeof(T) == 4 ? 4 : 2;  // row classes of a CTA
  static constexpr int NKB = H / KB + 1;
  static constexpr int PR = (kSplitR / 2) * JC;
  static constexpr int TH = H * JC;
  static constexpr int GZ = (NZ >= 256) ? 16 : 8, RZ = NZ / GZ, UZ = (RZ + GZ - 1) / GZ;
  static constexpr bool V2 = sizeof(T) == 4 && RZ % 2 == 0;
  static constexpr int PA = V2 ? ((RZ / 2) % 2 ? RZ : RZ + 2) : RZ + 1;
  // the JC rows of a warp's columns fall into different banks
  static constexpr int S0 = GZ * PA;
  static constexpr int BM = sizeof(T) == 4 ? 16 : 8, BW = sizeof(T) == 4 ? 4 : 4;
  static constexpr int S = S0 + ((BM + BW - S0 % BM) % BM);
  static constexpr int TASKS = PR * GZ;
  static constexpr size_t SMEM = sizeof(c2_t<T>) * ((size_t)PR * S + NY + 2 * NZ);
  static constexpr int MINB = 65536 / (TH * (sizeof(T) == 4 ? 64 : 128));
  static constexpr int CH = sizeof(T) == 4 ? 4 : 2;
  static_assert(S >= NZ && S % 2 == 0 && J % JC == 0 && H % KB == 0 && TASKS % 32 == 0 && UZ <= 2, "split plane layout");
};

template <typename T, int NY, int NZ>
__global__ void __launch_bounds__((SplitPlane<T, NY, NZ>::TH), (SplitPlane<T, NY, NZ>::MINB))
    split_plane_kernel(const PlaneWork<T>* __restrict__ works, const c2_t<T>* __restrict__ tw_y,
                       const c2_t<T>* __restrict__ tw_z) {
  using P = SplitPlane<T, NY, NZ>;
  using C = c2_t<T>;
  constexpr int H = P::H, J = P::J, JC = P::JC, KB = P::KB, NKB = P::NKB, S = P::S, TH = P::TH, PA = P::PA;
  constexpr int GZ = P::GZ, RZ = P::RZ, UZ = P::UZ, CH = P::CH, R = kSplitR, RH = R / 2;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  C* s_tw_y = buf + P::PR * S;
  C* s_twb = s_tw_y + NY;  // exp(-2 pi i r j / nz) as [r][j] for the radix-GZ passes
  C* s_twf = s_twb + NZ;   // ... and for the radix-RZ ones: consecutive lanes, consecutive banks
  const PlaneWork<T> w = works[blockIdx.y];
  const int tid = threadIdx.x;
  const int x = blockIdx.x / (J / JC);
  const int jb = (blockIdx.x - x * (J / JC)) * JC;
  const int jl = (tid / KB) % JC;
  const int c = (tid / (KB * JC)) * KB + tid % KB;
  const int mc = (c == 0) ? H : NZ - c;
  const int j = jb + jl;
  // element (k1, c): + k1 NKB J KB; the nz/2 column: block H / KB, first of its KB
  C* const spec = w.spec + (size_t)x * (R * NKB * J * KB) + (c / KB) * (J * KB) + j * KB + c % KB;
  constexpr int K1 = NKB * J * KB;
  constexpr int NYQ = (H / KB) * (J * KB);
  const bool inverse = w.mode != MODE_FIRST, forward = w.mode != MODE_LAST;
  const bool dc_sum = forward && (w.dc_out != nullptr);
  for (int i = tid; i < NY; i += TH) s_tw_y[i] = tw_y[i];
  for (int i = tid; i < NZ; i += TH) {
    s_twb[i] = tw_z[(i / RZ) * (i % RZ)];
    s_twf[i] = tw_z[(i / GZ) * (i % GZ)];
  }
  __syncthreads();
  pdl_wait();  // before any read of the spectrum, src or wfac, and any write

  if (inverse) {
    dc_hilo_store<T>(w.dc_in);
    C v[R];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = __ldcg(spec + k * K1);
    if (c == 0) {
#pragma unroll
      for (int k = 0; k < R; ++k) {
        const C n = __ldcg(spec + NYQ + k * K1);
        v[k] = C{v[k].x - n.y, v[k].y + n.x};
      }
    }
#pragma unroll
    for (int k = 1; k < R; ++k) v[k] = cmulc(v[k], s_tw_y[k * j]);
    Dft<R, true, C>::run(v);
    // rows y = j + J r (a) and y + ny/2 (a2) in packed row r JC + jl
#pragma unroll
    for (int r = 0; r < RH; ++r) {
      const C a = v[r], a2 = v[r + RH];
      C* const row = buf + (r * JC + jl) * S;
      row[c] = (c == 0) ? C{a.x, a2.x} : C{a.x - a2.y, a.y + a2.x};
      row[mc] = (c == 0) ? C{a.y, a2.y} : C{a.x + a2.y, a2.x - a.y};
    }
    __syncthreads();  // every row complete
  }

  T acc = T(0);
#pragma unroll 1
  for (int task = tid; task < P::TASKS; task += TH) {
    const int b = task / GZ, jz = task % GZ, j0 = jz * UZ;
    C* const row = buf + b * S;
    const int y = jb + b % JC + J * (b / JC);
    const size_t ra = ((size_t)x * NY + y) * NZ + j0;
    constexpr size_t RB = (size_t)(NY / 2) * NZ;
    C q[UZ][GZ];
    const T* const lead = inverse ? w.wfac_in : w.src;
    RealRun<T, UZ> f[2][CH], f2[2][CH];
    auto load_lead = [&](int s, int r0) {
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        f[s][i].ones();
        f2[s][i].ones();
        if (lead) {
          f[s][i].load(lead + ra + RZ * (r0 + i));
          f2[s][i].load(lead + ra + RB + RZ * (r0 + i));
        }
      }
    };
    load_lead(0, 0);
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
#pragma unroll
      for (int r = 0; r < GZ; ++r) {
        if constexpr (P::V2 && UZ == 2) {
          const float4 t = *reinterpret_cast<const float4*>(row + r * PA + j0);
          q[0][r] = C{t.x, t.y};
          q[UZ - 1][r] = C{t.z, t.w};
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
    } else {
#pragma unroll
      for (int u = 0; u < UZ; ++u)
#pragma unroll
        for (int r = 0; r < GZ; ++r) q[u][r] = C{T(1), T(1)};
    }
    const bool same = (w.wfac_in == w.wfac_out) && inverse;
    const bool dc_in = inverse && w.dc_in;
#pragma unroll
    for (int r0 = 0; r0 < GZ; r0 += CH) {
      const int s = (r0 / CH) & 1;
      if (r0 + CH < GZ) load_lead(s ^ 1, r0 + CH);
#pragma unroll
      for (int i = 0; i < CH; ++i) {
        const int r = r0 + i;
        const size_t at = ra + RZ * r, at2 = at + RB;
        RealRun<T, UZ> v, v2;
#pragma unroll
        for (int u = 0; u < UZ; ++u) {
          const C a = dc_in ? dc_add2<T>(q[u][r]) : q[u][r];
          v.v[u] = a.x * f[s][i].v[u];
          v2.v[u] = a.y * f2[s][i].v[u];
        }
        if (w.store) {
          v.store(w.store + at);
          v2.store(w.store + at2);
        }
        if (!same) {
          f[s][i].ones();
          f2[s][i].ones();
          if (w.wfac_out && forward) {
            f[s][i].load(w.wfac_out + at);
            f2[s][i].load(w.wfac_out + at2);
          }
        }
#pragma unroll
        for (int u = 0; u < UZ; ++u) q[u][r] = C{v.v[u] * f[s][i].v[u], v2.v[u] * f2[s][i].v[u]};
      }
    }
    if (!forward) continue;
#pragma unroll
    for (int u = 0; u < UZ; ++u) {
      Dft<GZ, false, C>::run(q[u]);
      acc += q[u][0].x + q[u][0].y;  // mean-mode carry
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
    __syncwarp();
    C v[RZ];
    if constexpr (P::V2) {
#pragma unroll
      for (int r = 0; r < RZ; r += 2) {
        const float4 t = *reinterpret_cast<const float4*>(row + jz * PA + r);
        v[r] = C{t.x, t.y};
        v[r + 1] = C{t.z, t.w};
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

  C v[R];
#pragma unroll
  for (int r = 0; r < RH; ++r) {
    const C* const row = buf + (r * JC + jl) * S;
    const C z = row[c], m = row[mc];
    v[r] = (c == 0) ? C{z.x, m.x} : C{z.x + m.x, z.y - m.y};
    v[r + RH] = (c == 0) ? C{z.y, m.y} : C{z.y + m.y, m.x - z.x};
  }
  Dft<R, false, C>::run(v);
  if (c == 0) {
    // x_0 + i x_h: twice the two real sequences' transforms
    C a[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const C p = v[k], d = v[(R - k) % R];
      a[k] = C{p.x + d.x, p.y - d.y};
      C n = C{p.y + d.y, d.x - p.x};
      if (k > 0) n = cmul(n, s_tw_y[k * j]);
      __stcg(spec + NYQ + k * K1, n);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = a[k];
  }
  __stcg(spec, v[0]);
#pragma unroll
  for (int k = 1; k < R; ++k) __stcg(spec + k * K1, cmul(v[k], s_tw_y[k * j]));
  if (dc_sum) dc_cta_store(works + blockIdx.y);
}

// The x pass: tile (k1, kz block), every x and every j.
template <typename T, int NX, int NY> struct SplitPencil {
  static constexpr int J = SplitJ<NY>::v, KB = SplitKB<T>::v, COLS = J * KB;
  static constexpr int G = (NX >= 256) ? 16 : (NX >= 16 ? 8 : (NX >= 8 ? 4 : (NX >= 4 ? 2 : 1)));
  static constexpr int R = NX / G, U = (R + G - 1) / G;
  static constexpr int YT = NX * KB, XT = COLS * G;
  static constexpr int TH0 = YT > XT ? YT : XT;
  static constexpr int TH = TH0 < 64 ? 64 : (TH0 + 31) / 32 * 32;
  // the x rows of a half-warp (FP64: quarter-warp) of the y part in different banks
  static constexpr int SC = COLS + KB;
  static constexpr size_t SMEM = sizeof(c2_t<T>) * ((size_t)NX * SC + NX) + sizeof(uint64_t) + sizeof(T) * NX;
  static_assert(TH <= 1024, "split pencil layout");
};

template <typename T, int NX, int NY>
__global__ void __launch_bounds__((SplitPencil<T, NX, NY>::TH))
    split_pencil_kernel(const PencilWork<T>* __restrict__ works, int nz, const c2_t<T>* __restrict__ tw_x) {
  using P = SplitPencil<T, NX, NY>;
  using C = c2_t<T>;
  constexpr int J = P::J, KB = P::KB, COLS = P::COLS, G = P::G, R = P::R, U = P::U, TH = P::TH, SC = P::SC;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* buf = reinterpret_cast<C*>(smem_raw);
  C* s_tw = buf + NX * SC;
  uint64_t* bar = reinterpret_cast<uint64_t*>(s_tw + NX);
  T* s_kx = reinterpret_cast<T*>(bar + 1);
  const PencilWork<T> w = works[blockIdx.y];
  const int tid = threadIdx.x;
  const int hz = nz / 2, nkb = hz / KB + 1;
  const int k1 = blockIdx.x / nkb, kb = blockIdx.x - k1 * nkb;
  const bool dc0 = w.dc_total && blockIdx.x == 0;  // mean-mode carry: see PlaneWork
  for (int i = tid; i < NX; i += TH) {
    s_tw[i] = tw_x[i];
    s_kx[i] = __ldg(w.kx + i);
  }
  // y part: (x, kz)
  const int yx = tid / KB, ykz = tid % KB;
  // x part: column col = k2 KB + kz, butterfly jx
  const int col = tid % COLS, jx = tid / COLS;
  const bool in_x = jx < G;
  const int kz = kb * KB + col % KB, ky = k1 + kSplitR * (col / KB);
  // every x's J KB values are contiguous: bulk copies into the padded rows
  constexpr uint32_t ROWB = (uint32_t)(COLS * sizeof(C));
  C* const rows = w.spec + ((size_t)k1 * nkb + kb) * COLS;
  const size_t xs = (size_t)kSplitR * nkb * COLS;
  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(bar, NX * ROWB);
  }
  __syncthreads();
  pdl_wait();  // before any read or write of the spectrum
  for (int x = tid; x < NX; x += TH) bulk_g2s(buf + x * SC, rows + x * xs, ROWB, bar);
  C v[J > R ? J : R];
  const T fyz = (in_x && kz <= hz) ? __ldg(w.kyzc + (kz < hz ? ky * hz + kz : NY * hz + ky)) : T(0);
  DcFinish<T> dcf;
  if (dc0 && tid < 32) dcf.load(w);
  if (dc0 && tid < 32) dcf.finish(w);
  const int ok = __syncthreads_and(mbar_wait_bounded(bar, 0) ? 1 : 0);
  if (!ok) {  // flag it, give the copies in flight one more bounded wait, and leave
    if (tid == 0) {
      if (w.status) atomicOr(w.status, 4);
      mbar_wait_bounded(bar, 0);
    }
    return;
  }
  if (yx < NX) {
#pragma unroll
    for (int j = 0; j < J; ++j) v[j] = buf[yx * SC + j * KB + ykz];
    Dft<J, false, C>::run(v);
#pragma unroll
    for (int k = 0; k < J; ++k) buf[yx * SC + k * KB + ykz] = v[k];
  }
  __syncthreads();
  // x part, every pass in place: thread jx has rows jx + G r in the radix-R passes and
  // rows r + G jp in the radix-G ones
  if constexpr (G > 1) {
    if (in_x) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = buf[(jx + G * r) * SC + col];
      Dft<R, false, C>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[(jx + G * r) * SC + col] = v[r];
    }
    __syncthreads();
    if (in_x) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int jp = jx + u * G;
        if (R % G == 0 || jp < R) {
          C b[G];
#pragma unroll
          for (int r = 0; r < G; ++r) b[r] = buf[(r + G * jp) * SC + col];
#pragma unroll
          for (int r = 1; r < G; ++r) b[r] = cmul(b[r], s_tw[r * jp]);
          Dft<G, false, C>::run(b);
#pragma unroll
          for (int r = 0; r < G; ++r) {
            const T f = s_kx[jp + R * r] * fyz;
            b[r] = C{b[r].x * f, b[r].y * f};
          }
          if (dc0 && col == 0 && jp == 0) b[0] = C{T(0), T(0)};
          Dft<G, true, C>::run(b);
#pragma unroll
          for (int r = 0; r < G; ++r) buf[(r + G * jp) * SC + col] = b[r];
        }
      }
    }
    __syncthreads();
    if (in_x) {
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = buf[(jx + G * r) * SC + col];
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmulc(v[r], s_tw[r * jx]);
      Dft<R, true, C>::run(v);
#pragma unroll
      for (int r = 0; r < R; ++r) buf[(jx + G * r) * SC + col] = v[r];
    }
  } else if (in_x) {
    const T f = s_kx[0] * fyz;
    const C t = buf[col];
    buf[col] = (dc0 && col == 0) ? C{T(0), T(0)} : C{t.x * f, t.y * f};
  }
  __syncthreads();
  if (yx < NX) {
#pragma unroll
    for (int k = 0; k < J; ++k) v[k] = buf[yx * SC + k * KB + ykz];
    Dft<J, true, C>::run(v);
#pragma unroll
    for (int j = 0; j < J; ++j) buf[yx * SC + j * KB + ykz] = v[j];
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (tid < NX) {
    for (int x = tid; x < NX; x += TH) bulk_s2g(rows + x * xs, buf + x * SC, ROWB);
    bulk_commit();
    bulk_wait_read_all();
  }
}

template <typename T, int NY, int NZ>
cudaError_t launch_split_plane_t(const PlaneWork<T>* w, int nw, int nx, const c2_t<T>* ty, const c2_t<T>* tz,
                                 cudaStream_t st) {
  using P = SplitPlane<T, NY, NZ>;
  auto kern = split_plane_kernel<T, NY, NZ>;
  static unsigned attr_mask = 0;
  cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
  if (e != cudaSuccess) return e;
  return launch_sweep_kernel(kern, dim3(nx * (P::J / P::JC), nw), dim3(P::TH), P::SMEM, st, w, ty, tz);
}

template <typename T, int NX, int NY>
cudaError_t launch_split_pencil_t(const PencilWork<T>* w, int nw, int nz, const c2_t<T>* tx, cudaStream_t st) {
  using P = SplitPencil<T, NX, NY>;
  auto kern = split_pencil_kernel<T, NX, NY>;
  static unsigned attr_mask = 0;
  cudaError_t e = ensure_smem_attr(kern, P::SMEM, &attr_mask);
  if (e != cudaSuccess) return e;
  return launch_sweep_kernel(kern, dim3(kSplitR * (nz / 2 / P::KB + 1), nw), dim3(P::TH), P::SMEM, st, w, nz, tx);
}

}  // namespace psb
