// Plane pass (pass B) for square planes of side N = 32 K with odd K: K = 3 (96) and K = 5 (160).
//
// The doubled grid has M = 2 N = 64 K points per axis, so both axes split by frequency residue
// mod K into 64-point transforms, the engine's best case (8 lanes x 8 registers, one
// exchange).  A cluster of K CTAs owns one (z, y) plane and CTA q takes ky = K k + q:
//   rows     X_q[k] = FFT_64( w_M^(y' q) sum_m a[y' + 64 m] e^(-2 pi i m q / K) )[k]
//   columns  for every residue r of kz (|r| <= K / 2) the same fold along z, FFT_64, x T[K k + r],
//            inverse FFT_64, and w_M^(-z' r) (...) is added to z' + 64 m with e^(+2 pi i m r / K)
//   inverse rows, then out[y' + 64 m] = sum_q e^(+2 pi i m q / K) w_M^(-y' q) R_q[y'] across the
//            cluster (distributed shared memory),
// with y', z' < 64 and m < K / 2 (the last m is half: the image ends at 32 K).  Every
// factor e^(2 pi i m r / K) is a compile-time constant.
//
// Bound: the shared-memory pipe (73 % of its peak in ncu at N = 160; issue 53 %), as the mod-4
// plane pass.  A CTA holds N x 64 of the plane and its exchange buffers: 107 KB at N = 160, two CTAs
// of 256 threads per SM; 63 KB at N = 96, three of 128 (256 threads: 1714 us).  The parity split it
// replaces transformed 96- to 320-point lines with 24 or 40 registers per lane, which left one
// small CTA per SM.  Measured: 40 slots of 160 x 160 x 128 4.73 ms against 13.75 ms, 60 slots of 96^3
// 1.66 ms against 3.38 ms.  On the way (160): residues 0 .. K - 1 one by one 5.63 ms, constants as
// FMAs 5.50 ms, +-R pairs (twiddles read once per pair, shared folds) 4.92 ms, column order without
// bank conflicts 4.73 ms; 128 threads 5.62 ms.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "fft.cuh"
#include "toeplitz_kernels.cuh"

namespace hb {

template <int K, int THREADS_>
struct PlaneOddCfg {
  static_assert(K == 3 || K == 5, "odd plane split");
  static constexpr int N = 32 * K, M = 64 * K, L = 64, S = 8, E = 8;
  static constexpr int THREADS = THREADS_, NTEAMS = THREADS / S;
  static constexpr int HM = K / 2;        // whole 64-blocks of an image line; half a block more
  static constexpr int NA = HM * E + E / 2;  // registers of a lane's share of an image line
  static constexpr int LDP = L + 1;
  static constexpr int TBUF = team_buf_stride<L>();
  static constexpr int SMEM_F2 = N * LDP + NTEAMS * TBUF + L + M;  // share, exchange, tables: 64-point, circle
  static_assert(N % NTEAMS == 0 && L % NTEAMS == 0, "teams tile the rows and columns");
};

// acc + a * e^(DIR 2 pi i P / K): one packed and two scalar FMAs
template <int K, int P, int DIR>
__device__ __forceinline__ float2 fma_root(float2 a, float2 acc) {
  constexpr int p = P % K;
  if constexpr (p == 0) return cadd(acc, a);
  constexpr float c = (float)ct_cos(kTwoPi * p / K), s = (float)(DIR * ct_sin(kTwoPi * p / K));
  const float2 v = __ffma2_rn(make_float2(c, c), a, acc);
  return make_float2(fmaf(-s, a.y, v.x), fmaf(s, a.x, v.y));
}
// v[e] = sum_m e^(-2 pi i m R / K) a[m * 8 + e]: the fold of one residue (m = K / 2 only for e < 4)
template <int K, int R>
__device__ __forceinline__ void odd_fold(const float2* a, float2* v) {
  constexpr int HM = K / 2;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    v[e] = a[e];
    if constexpr (HM == 2) v[e] = fma_root<K, R, -1>(a[8 + e], v[e]);
    if (e < 4) v[e] = fma_root<K, HM * R, -1>(a[HM * 8 + e], v[e]);
  }
}
// Diagonal of one column at kz = K (t + 8 j) + R mod M, j < 8 (-K < R < K).  The packed column holds
// kz = (t' + 8 c) + 8 K k2 at float4 (2 c + k2 / 4) * 8 + t' (column_kz), so with t' + 8 c = K t + R the
// eight values are two 16-byte loads; for R < 0 lane 0 has t' + 8 c = 8 K + R and k2 = j - 1 mod 8.
template <int K, int R>
__device__ __forceinline__ void odd_load_t(float* tv, const float* col, int t) {
  const bool turn = R < 0 && t == 0;
  const int i = K * t + R + (turn ? 8 * K : 0);
  const float4* src = reinterpret_cast<const float4*>(col) + (i / 8) * 16 + i % 8;
  const float4 a = __ldg(src), b = __ldg(src + 8);
  tv[0] = turn ? b.w : a.x; tv[1] = turn ? a.x : a.y; tv[2] = turn ? a.y : a.z; tv[3] = turn ? a.z : a.w;
  tv[4] = turn ? a.w : b.x; tv[5] = turn ? b.x : b.y; tv[6] = turn ? b.y : b.z; tv[7] = turn ? b.z : b.w;
}

// v <- inverse FFT_64( T x FFT_64(v) )
__device__ __forceinline__ void odd_filter(float2* v, const float* tv, int t, float2* buf, const float2* twr) {
  team_fft_din_to_dout_r<64, -1, false>(v, t, buf, twr);
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = cscale(v[j], tv[j]);
  team_fft_dout_to_din_r<64, 1, false>(v, t, buf, twr);
}

// Residues +R and -R of a column, and then those above: the two folds share the sums of real and of
// imaginary multiples, and the twiddles of -R are the conjugates of those of R.
//   tp: the diagonal of residue +R;  P: the column
template <int K, int R>
__device__ __forceinline__ void odd_pair(float2* acc, const float* tp, const float2* P, const float* col, int t,
                                         float2* buf, const float2* twr, const float2* circ) {
  constexpr int HM = K / 2, M = 64 * K, LDP = PlaneOddCfg<K, 128>::LDP;
  static_assert(63 * HM < M, "the circle table is indexed without a wrap");
  float tm[8], tn[8];
  odd_load_t<K, -R>(tm, col, t);  // the diagonal is fetched one residue ahead of its use
  float2 vp[8], vm[8], w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    float2 s = P[(t + 8 * e) * LDP], d = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 1; m <= HM; ++m) {
      if (m == HM && e >= 4) continue;
      const float c = (float)ct_cos(kTwoPi * ((m * R) % K) / K), sn = (float)ct_sin(kTwoPi * ((m * R) % K) / K);
      const float2 x = P[(t + 8 * e + 64 * m) * LDP];
      s = __ffma2_rn(make_float2(c, c), x, s);
      d = __ffma2_rn(make_float2(sn, sn), x, d);
    }
    w[e] = circ[(t + 8 * e) * R];
    vp[e] = cmul(make_float2(s.x + d.y, s.y - d.x), w[e]);   // (s - i d) w
    vm[e] = cmulc(make_float2(s.x - d.y, s.y + d.x), w[e]);  // (s + i d) conj(w)
  }
  odd_filter(vp, tp, t, buf, twr);
  if constexpr (R < HM) odd_load_t<K, R + 1>(tn, col, t);
  odd_filter(vm, tm, t, buf, twr);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float2 up = cmulc(vp[e], w[e]), um = cmul(vm[e], w[e]);
    const float2 p = cadd(up, um), q = csub(up, um);
    acc[e] = cadd(acc[e], p);
#pragma unroll
    for (int m = 1; m <= HM; ++m) {
      if (m == HM && e >= 4) continue;
      const float c = (float)ct_cos(kTwoPi * ((m * R) % K) / K), sn = (float)ct_sin(kTwoPi * ((m * R) % K) / K);
      const float2 v = __ffma2_rn(make_float2(c, c), p, acc[m * 8 + e]);
      acc[m * 8 + e] = make_float2(fmaf(-sn, q.y, v.x), fmaf(sn, q.x, v.y));
    }
  }
  if constexpr (R < HM) odd_pair<K, R + 1>(acc, tn, P, col, t, buf, twr, circ);
}

template <int K, int THREADS_>
__global__ void __cluster_dims__(K, 1, 1) __launch_bounds__(THREADS_, THREADS_ == 128 ? 4 : 2) plane_odd_kernel(PassArgs a) {
  namespace cg = cooperative_groups;
  using C = PlaneOddCfg<K, THREADS_>;
  constexpr int N = C::N, M = C::M, L = C::L, LDP = C::LDP, HM = C::HM, NT = C::NTEAMS;
  extern __shared__ float2 smem[];
  float2* P = smem;                  // [N][LDP]: this CTA's share of the plane
  float2* xbuf = P + N * LDP;
  float2* tw = xbuf + NT * C::TBUF;  // [64] 64-point team table
  float2* circ = tw + L;             // [M] exp(-2 pi i k / M)

  cg::cluster_group cluster = cg::this_cluster();
  const int q = (int)cluster.block_rank();  // ky mod K
  const int slot = blockIdx.y;
  const int kx = blockIdx.z;
  const int sys = a.slot_sys[slot];
  if (a.active && !a.active[sys]) return;  // uniform for the whole cluster
  const int M2 = 2 * a.N2;

  const float2* circ_g = a.tables + table_offsets(N, N, a.N2).circ;
  for (int i = threadIdx.x; i < M; i += C::THREADS) circ[i] = circ_g[i];
  for (int i = threadIdx.x; i < L; i += C::THREADS) tw[i] = circ_g[(i % 8) * (i / 8) * K];
  __syncthreads();

  const SpillPlane<N> g(a.spill, slot, kx, N, M2);
  {
    // warm L2 with the plane of the cluster a.prefetch_ahead clusters later (a hint only)
    const long long cl = (long long)blockIdx.z * gridDim.y + blockIdx.y + a.prefetch_ahead;
    if (a.prefetch_ahead > 0 && cl < (long long)gridDim.y * gridDim.z) {
      const SpillPlane<N> nxt(a.spill, (int)(cl % gridDim.y), (int)(cl / gridDim.y), N, M2);
      prefetch_plane_rows_l2<C::THREADS>(nxt, q * 32, 32);
    }
  }
  const int team = threadIdx.x / 8, t = threadIdx.x % 8;
  const int tr = row_of_team<8, NT, N>(team);
  float2* buf = xbuf + team * C::TBUF;

  // stage 1: rows; the rank is a compile-time constant inside
  with_rank<K>(q, [&](auto rank) {
    constexpr int q = decltype(rank)::value;
    float2 twr[8], cw[8];
    load_lane_twiddles<L>(twr, tw, t);
#pragma unroll
    for (int e = 0; e < 8; ++e) cw[e] = circ[(t + 8 * e) * q];
    float2 nv[C::NA];  // the next row's values, loaded while the current one is transformed
    auto load_row = [&](int z) {
#pragma unroll
      for (int i = 0; i < C::NA; i += 2) g.pair(z, t + 8 * (i % 8) + 64 * (i / 8), nv[i], nv[i + 1]);
    };
    load_row(tr);
#pragma unroll 1
    for (int z = tr; z < N; z += NT) {
      float2 v[8];
      odd_fold<K, q>(nv, v);
      if constexpr (q > 0) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = cmul(v[e], cw[e]);
      }
      if (z + NT < N) load_row(z + NT);
      team_fft_din_to_dout_r<L, -1, false>(v, t, buf, twr);
#pragma unroll
      for (int r = 0; r < 8; ++r) P[z * LDP + dout_index<L>(t, r)] = v[r];
    }
  });
  __syncthreads();

  // stage 2: the CTA's 64 columns, residue 0 and then the pairs +-R (the column is read again for each
  // pair: holding it would cost 40 registers at K = 5)
  float2 twr[8];
  load_lane_twiddles<L>(twr, tw, t);
#pragma unroll 1
  for (int col = row_of_team<8, NT, L>(team); col < L; col += NT) {  // half-warp mates 8 columns apart: other banks
    const int ky = K * col + q;
    const float* T = a.sys_diag[sys] + (((long long)kx * 2 + (ky & 1)) * N + (ky >> 1)) * M;
    float t0[8], t1[8];
    odd_load_t<K, 0>(t0, T, t);
    float2 acc[C::NA], v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      v[e] = P[(t + 8 * e) * LDP + col];
#pragma unroll
      for (int m = 1; m <= HM; ++m)
        if (m < HM || e < 4) v[e] = cadd(v[e], P[(t + 8 * e + 64 * m) * LDP + col]);
    }
    odd_load_t<K, 1>(t1, T, t);
    odd_filter(v, t0, t, buf, twr);
#pragma unroll
    for (int i = 0; i < C::NA; ++i) acc[i] = v[i % 8];
    odd_pair<K, 1>(acc, t1, P + col, T, t, buf, twr, circ);
#pragma unroll
    for (int i = 0; i < C::NA; ++i) P[(t + 8 * (i % 8) + 64 * (i / 8)) * LDP + col] = acc[i];
  }
  __syncthreads();

  // stage 3: rows, 64-point inverse FFT in place: P[z][y'] = R_q[z][y']
  {
#pragma unroll 2
    for (int z = tr; z < N; z += NT) {
      float2 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) v[r] = P[z * LDP + dout_index<L>(t, r)];
      team_fft_dout_to_din_r<L, 1, false>(v, t, buf, twr);
#pragma unroll
      for (int e = 0; e < 8; ++e) P[z * LDP + t + 8 * e] = v[e];
    }
  }
  cluster.sync();  // every R_q is complete

  // stage 4: CTA q writes rows [32 q, 32 q + 32)
  {
    const float2* R[K];
#pragma unroll
    for (int qq = 0; qq < K; ++qq) R[qq] = cluster.map_shared_rank(P, qq);
    static_assert(C::THREADS % L == 0 && (32 * L) % C::THREADS == 0, "a thread keeps its y through the loop");
    const int y = threadIdx.x % L;
    float2 cy[K];  // w_M^(y qq)
#pragma unroll
    for (int qq = 1; qq < K; ++qq) cy[qq] = circ[y * qq];
#pragma unroll
    for (int j = 0; j < 32 * L / C::THREADS; ++j) {
      const int z = q * 32 + threadIdx.x / L + j * (C::THREADS / L);
      float2 u[K];
      u[0] = R[0][z * LDP + y];
#pragma unroll
      for (int qq = 1; qq < K; ++qq) u[qq] = cmulc(R[qq][z * LDP + y], cy[qq]);
      Dft<K, 1>::run(u);
#pragma unroll
      for (int m = 0; m < HM; ++m) g.at(z, y + L * m) = u[m];
      if (y < 32) g.at(z, y + L * HM) = u[HM];
    }
  }
  // keep this CTA's shared memory alive until the partners have read it (see plane_mod_kernel)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory");
}

}  // namespace hb
