// Plane pass (pass B) for planes that one CTA can hold at the full doubled y length: N0 x 2 N1 values
// in shared memory, no cluster.
//
//   rows     2 N1-point FFT of every image row (upper half zero)   -> P[z][ky]
//   columns  2 N0-point FFT along z (upper half zero), x T, inverse, keeping z < N0
//   rows     inverse 2 N1-point FFT, keeping y < N1, straight to the spill
//
// The parity split (plane_yz_kernel) halves a plane between two CTAs, which pays for planes that do
// not fit one; it moves each row into shared memory first, twiddles half of the frequencies
// and adds the halves through distributed shared memory behind cluster barriers.  Here the zero
// padding is pruned inside the transforms, a plane is loaded and stored once, and two block
// barriers remain.  Bound: the shared-memory pipe (the exchanges: 8.2 K of the cycles of a 64 x 64
// plane).  Measured, 128 kx planes of 1 / 16 slots, us, parity split -> this form: 64 x 64 15.0 / 171
// -> 9.8 / 99.6; 32 x 32 7.1 / 41 -> 3.9 / 24; 16 x 16 5.3 / 24 -> 3.1 / 11; 64 x 128 28 / 364 -> 18 /
// 261; 128 x 64 26 / 315 -> 18 / 252; 32 x 128 20 / 260 -> 10 / 99; 8 x 128 12 / 147 -> 4.9 / 26.
#pragma once

#include "common.cuh"
#include "fft.cuh"
#include "toeplitz_kernels.cuh"

namespace hb {

template <int N0, int N1, int THREADS_>
struct PlaneFullCfg {
  static constexpr int M0 = 2 * N0, M1 = 2 * N1, THREADS = THREADS_;
  static constexpr int SR = TeamCfg<M1>::S, ER = TeamCfg<M1>::E, SZ = TeamCfg<M0>::S, EZ = TeamCfg<M0>::E;
  static constexpr int NTR = THREADS / SR, NTZ = THREADS / SZ;
  static constexpr int LDP = M1 + 1;
  static constexpr int TBR = team_buf_stride<M1>(), TBZ = team_buf_stride<M0>();
  static constexpr int XBUF = (NTR * TBR > NTZ * TBZ) ? NTR * TBR : NTZ * TBZ;
  static constexpr int SMEM_F2 = N0 * LDP + XBUF + M1 + M0;  // plane, exchange, tables
};

template <int N0, int N1, int THREADS_>
__global__ void __launch_bounds__(THREADS_) plane_full_kernel(PassArgs a) {
  chained_kernel_begin();
  using C = PlaneFullCfg<N0, N1, THREADS_>;
  constexpr int M0 = C::M0, M1 = C::M1, LDP = C::LDP;
  constexpr int SR = C::SR, ER = C::ER, SZ = C::SZ, EZ = C::EZ, NTR = C::NTR, NTZ = C::NTZ;
  extern __shared__ float2 smem[];
  float2* P = smem;                 // [N0][LDP]
  float2* xbuf = P + N0 * LDP;
  float2* tw_r = xbuf + C::XBUF;    // [M1]
  float2* tw_z = tw_r + M1;         // [M0]
  const int slot = blockIdx.x, kx = blockIdx.y;
  const int sys = a.slot_sys[slot];
  if (a.active && !a.active[sys]) return;
  const int M2 = 2 * a.N2;
  const SpillPlane<N1> g(a.spill, slot, kx, N0, M2);
  // 16-byte pairs (y, y + SR) of the spill rows, see SpillPlane
  constexpr bool kPair = SpillPlane<N1>::YT == 2 * SR && ER % 4 == 0;

  const int team_r = threadIdx.x / SR, tr = threadIdx.x % SR;
  const int row0 = row_of_team<SR, NTR, N0>(team_r);
  auto load_row = [&](int z, float2* v) {
#pragma unroll
    for (int e = 0; e < ER / 2; e += kPair ? 2 : 1) {
      if constexpr (kPair) g.pair(z, tr + SR * e, v[e], v[e + 1]);
      else v[e] = g.at(z, tr + SR * e);
    }
  };
  constexpr int LPR = (N0 + NTR - 1) / NTR;
  float2 nv[ER / 2];  // the next row, loaded ahead of its use
  load_row(row0 < N0 ? row0 : 0, nv);
  const TableOffsets to = table_offsets(N0, N1, a.N2);
  for (int i = threadIdx.x; i < M1; i += C::THREADS) tw_r[i] = a.tables[to.circ + (i % SR) * (i / SR)];
  for (int i = threadIdx.x; i < M0; i += C::THREADS) tw_z[i] = a.tables[to.z + i];
  __syncthreads();

  // stage 1
  {
    float2* buf = xbuf + team_r * C::TBR;
#pragma unroll
    for (int it = 0; it < LPR; ++it) {
      const int z = row0 + it * NTR;
      float2 v[ER];
#pragma unroll
      for (int e = 0; e < ER / 2; ++e) v[e] = nv[e];
      if (it + 1 < LPR) load_row(z + NTR < N0 ? z + NTR : 0, nv);
      team_fft_din_to_dout<M1, -1, true>(v, tr, buf, tw_r);
      if (N0 % NTR == 0 || z < N0) {
#pragma unroll
        for (int r = 0; r < ER; ++r) P[z * LDP + dout_index<M1>(tr, r)] = v[r];
      }
    }
  }
  __syncthreads();

  // stage 2: column ky at packed column (ky & 1, ky >> 1)
  {
    const int team = threadIdx.x / SZ, t = threadIdx.x % SZ;
    float2* buf = xbuf + team * C::TBZ;
    const float* T = a.sys_diag[sys] + (long long)kx * M1 * M0;
    constexpr int LPZ = (M1 + NTZ - 1) / NTZ;
    const int col0 = row_of_team<SZ, NTZ, M1>(team);
    auto tcol = [&](int ky) { return T + ((long long)(ky & 1) * N1 + (ky >> 1)) * M0; };
    float2 twz[EZ];
    load_lane_twiddles<M0>(twz, tw_z, t);
    float tnext[EZ];
    load_tcol<EZ, SZ>(tnext, tcol(col0 < M1 ? col0 : 0), t);
#pragma unroll 2
    for (int it = 0; it < LPZ; ++it) {
      const int col = col0 + it * NTZ;
      const bool ok = M1 % NTZ == 0 || col < M1;
      const int cc = ok ? col : 0;
      float tv[EZ];
#pragma unroll
      for (int r = 0; r < EZ; ++r) tv[r] = tnext[r];
      float2 v[EZ];
#pragma unroll
      for (int e = 0; e < EZ / 2; ++e) v[e] = P[din_index<M0>(t, e) * LDP + cc];
      team_fft_din_to_dout_r<M0, -1, true>(v, t, buf, twz);
#pragma unroll
      for (int r = 0; r < EZ; ++r) v[r] = cscale(v[r], tv[r]);
      if (it + 1 < LPZ) load_tcol<EZ, SZ>(tnext, tcol(col + NTZ < M1 ? col + NTZ : 0), t);
      team_fft_dout_to_din_r<M0, 1, true>(v, t, buf, twz);
      if (ok) {
#pragma unroll
        for (int e = 0; e < EZ / 2; ++e) P[din_index<M0>(t, e) * LDP + col] = v[e];
      }
    }
  }
  __syncthreads();

  // stage 3
  {
    float2* buf = xbuf + team_r * C::TBR;
#pragma unroll 2
    for (int it = 0; it < LPR; ++it) {
      const int z = row0 + it * NTR;
      const bool ok = N0 % NTR == 0 || z < N0;
      const int zc = ok ? z : 0;
      float2 v[ER];
#pragma unroll
      for (int r = 0; r < ER; ++r) v[r] = P[zc * LDP + dout_index<M1>(tr, r)];
      team_fft_dout_to_din<M1, 1, true>(v, tr, buf, tw_r);
      if (ok) {
#pragma unroll
        for (int e = 0; e < ER / 2; e += kPair ? 2 : 1) {
          if constexpr (kPair) g.put_pair(z, tr + SR * e, v[e], v[e + 1]);
          else g.at(z, tr + SR * e) = v[e];
        }
      }
    }
  }
}

}  // namespace hb
