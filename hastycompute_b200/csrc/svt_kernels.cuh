// Block singular-value thresholding (the locally-low-rank proximal step): restates
// hasty::svt::svt_soft / svt_hard on extracted blocks (lib/op/svt.cpp:60-168, block
// extraction :11-58 and insertion :170-240, the block loops of Random3DBlocksSVT and
// Normal3DBlocksSVT :268-490).
//
// x is [d0][d1][S0][S1][S2] complex64.  A block with corner (c0, c1, c2) and shape
// b0 x b1 x b2 is the matrix M [R = d1*b0*b1*b2][d0] (row = (d1 index, voxel in the block,
// row-major), column = d0 index), as extract_block(..., flatten_split 0, transpose) forms
// it.  With M = U S V^H: soft f(s) = max(s - thresh, 0), hard keeps the `rank` largest s,
// and the block is replaced by U f(S) V^H = M W,  W = V diag(f(s)/s) V^H  (0 where s = 0).
// One CTA of 128 threads per block, columns padded to a multiple of four:
//   1. G = M^H M in FP64: rows are staged in shared memory in single precision and converted as a
//      thread reads them; every thread accumulates one 4 x 4 tile of G over its share of the rows (its
//      group's) in registers, and the groups' sums are added up;
//   2. G is diagonalised by Jacobi rotations (FP64), G = V diag(lambda) V^H, s = sqrt(lambda): a round
//      rotates the n / 2 disjoint pairs of a round-robin tournament at once, each 2 x 2 block of
//      A' = J^H A J by one thread, so a round takes two barriers;
//   3. W, then every row is replaced by (row) W in FP32, in place.
// Blocks of one launch must not overlap (the host launches overlapping sets in waves).
//
// Bound: the three parts take about equal shares (of 2.65 ms, measured by leaving each out: Gram 0.97,
// rotations 0.73, rows 0.92); the floors are FP64 issue 0.5 + 0.3 ms, FP32 issue 0.4 ms and two reads
// and a write of the data 0.8 ms, with the shared-memory pipe (4 bytes per lane and cycle, broadcast
// or not) next.  Measured, 3375 blocks of 2560 x 20: 2.65 ms against 10.03 ms when one warp made the
// rotations one after the other and every thread computed single entries of G; 32 columns 5.64
// against 19.5 ms, 8 columns 0.74 against 2.53 ms.  On the way: rotations of a round in parallel
// 3.26 ms, staging ahead without divisions 2.93 ms, single-precision staging and unpaired W 2.65 ms,
// rows last to first 2.51 ms, the real products of W summed apart (a sum of 40 terms in one chain
// rounds worse than the 20 complex products it stands for) 2.65 ms.  G by FP64 mma.sync m8n8k4 straight from global memory: 3.26 ms; At
// 20 columns 96 registers for five CTAs per SM 3.65 ms, 168 for three 2.87 ms; the bound of 128 holds for every
// column count, and from 21 columns on it spills 100 to 412 bytes a thread (other bounds were not measured there).
#pragma once

#include "common.cuh"

namespace hb {

constexpr int kSvtMaxCols = 32;  // d0 <= 32
constexpr int kSvtThreads = 128;
constexpr int kSvtChunk = 64;    // rows staged per Gram step
constexpr int kSvtMaxSweeps = 15;

struct SvtArgs {
  float2* x;
  int d0, d1, S0, S1, S2;
  int b0, b1, b2;
  const int* corners;  // [nblocks][3]
  int soft;            // 1: soft threshold, 0: hard (keep `rank`)
  float thresh;
  int rank;
};

// Walks the rows of a block's matrix in steps of a fixed number of rows, keeping the row's element
// offset in x: mixed-radix addition instead of divisions.
struct SvtRow {
  int i0, i1, i2;       // voxel in the block
  int s0, s1, s2;       // the step's digits
  long long off;
  long long step, w2, w1, w0;  // offset of a step; corrections when i2, i1, i0 wrap
  __device__ __forceinline__ SvtRow(const SvtArgs& a, int c0, int c1, int c2, int row, int stride) {
    const long long p1 = a.S2, p0 = p1 * a.S1, pd = p0 * a.S0;
    i2 = row % a.b2;
    i1 = (row / a.b2) % a.b1;
    i0 = (row / (a.b2 * a.b1)) % a.b0;
    off = (long long)(row / (a.b2 * a.b1 * a.b0)) * pd + (c0 + i0) * p0 + (c1 + i1) * p1 + c2 + i2;
    s2 = stride % a.b2;
    s1 = (stride / a.b2) % a.b1;
    s0 = (stride / (a.b2 * a.b1)) % a.b0;
    step = (long long)(stride / (a.b2 * a.b1 * a.b0)) * pd + s0 * p0 + s1 * p1 + s2;
    w2 = p1 - a.b2;
    w1 = p0 - a.b1 * p1;
    w0 = pd - a.b0 * p0;
  }
  __device__ __forceinline__ void next(const SvtArgs& a) {
    off += step;
    i2 += s2;
    i1 += s1;
    i0 += s0;
    if (i2 >= a.b2) { i2 -= a.b2; ++i1; off += w2; }
    if (i1 >= a.b1) { i1 -= a.b1; ++i0; off += w1; }
    if (i0 >= a.b0) { i0 -= a.b0; off += w0; }
  }
  __device__ __forceinline__ void prev(const SvtArgs& a) {
    off -= step;
    i2 -= s2;
    i1 -= s1;
    i0 -= s0;
    if (i2 < 0) { i2 += a.b2; --i1; off -= w2; }
    if (i1 < 0) { i1 += a.b1; --i0; off -= w1; }
    if (i0 < 0) { i0 += a.b0; off -= w0; }
  }
};

// NT: columns in tiles of four, NT = ceil(d0 / 4).  Dynamic shared memory: A and V [NC][NC + 1] doubles
// (complex), then the staged rows [kSvtChunk][NC + 1], whose space later holds W.
template <int NT>
struct SvtCfg {
  static constexpr int NC = 4 * NT;
  static constexpr int LD = NC + 1;                      // odd pitch in 16-byte units: rows on distinct banks
  static constexpr int TILES = NT * (NT + 1) / 2;        // upper-triangle tiles of G
  // Row groups.  Up to 12 columns there are so many (128, 40, 20) that they are added up by shuffles within a
  // warp before the warps' sums go to shared memory one after the other, and a warp holds whole groups: one
  // group after the other took 20 us of a block of 4 columns (512 blocks of 8 rows x 4 columns 31 us, now 11; 18
  // with one warp making the rotations; 64 blocks of 2560 x 4 62 -> 43, x 8 106 -> 99, x 12 170 -> 169).  From 13
  // columns on whole groups would leave a warp's lanes idle, and there are 12 sums or fewer.
  static constexpr bool SHUFFLE = NT <= 3;
  static constexpr int WARP_GROUPS = 32 / TILES;  // SHUFFLE: groups in a warp
  static constexpr int GROUPS = SHUFFLE ? kSvtThreads / 32 * WARP_GROUPS : kSvtThreads / TILES;
  static constexpr int RLD = NC + 2;                     // pitch of the staged rows
  static constexpr size_t SMEM = (size_t)2 * NC * LD * sizeof(double2) + (size_t)kSvtChunk * RLD * sizeof(float2);
  static_assert(kSvtChunk * RLD >= NC * NC, "W takes the place of the staged rows");
};

__device__ __forceinline__ double svt_block_sum(double v, double* red) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  __syncthreads();
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = v;
  __syncthreads();
  double s = 0.0;
  for (int w = 0; w < kSvtThreads / 32; ++w) s += red[w];
  return s;
}

template <int NT>
__global__ void __launch_bounds__(kSvtThreads, 4) svt_blocks_kernel(SvtArgs a) {
  using C = SvtCfg<NT>;
  constexpr int NC = C::NC, LD = C::LD;
  extern __shared__ __align__(16) double2 svt_smem[];
  double2* A = svt_smem;           // [NC][LD]
  double2* V = A + NC * LD;        // [NC][LD]
  float2* rows = reinterpret_cast<float2*>(V + NC * LD);  // [kSvtChunk][RLD]
  float2* W = rows;                                       // [NC][NC]
  __shared__ double wdiag[kSvtMaxCols], red[kSvtThreads / 32];
  // rotations of the current and the next round: columns p < q, c, s e
  __shared__ int2 rot_pq[2][kSvtMaxCols / 2];
  __shared__ double rot_c[2][kSvtMaxCols / 2];
  __shared__ double2 rot_s[2][kSvtMaxCols / 2];
  const int n = a.d0, tid = threadIdx.x;
  const int c0 = a.corners[3 * blockIdx.x], c1 = a.corners[3 * blockIdx.x + 1], c2 = a.corners[3 * blockIdx.x + 2];
  // a block that does not fit inside the image is left untouched (the host validates corners)
  if (c0 < 0 || c1 < 0 || c2 < 0 || c0 + a.b0 > a.S0 || c1 + a.b1 > a.S1 || c2 + a.b2 > a.S2) return;
  const int R = a.d1 * a.b0 * a.b1 * a.b2;
  const long long col_stride = (long long)a.d1 * a.S0 * a.S1 * a.S2;

  // 1. Gram matrix: thread (tile, group) accumulates G[4 ti + i][4 tj + j] over rows group, group + GROUPS, ...
  const int wgroup = tid % 32 / C::TILES;  // SHUFFLE: the group's number in its warp
  const int tile = (C::SHUFFLE ? tid % 32 : tid) % C::TILES;
  const int group = !C::SHUFFLE ? tid / C::TILES : wgroup < C::WARP_GROUPS ? tid / 32 * C::WARP_GROUPS + wgroup : C::GROUPS;
  int ti = 0, tj = tile;
  while (tj >= NT - ti) {
    tj -= NT - ti;
    ++ti;
  }
  tj += ti;
  double2 g[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) g[i][j] = make_double2(0.0, 0.0);
  // staging: consecutive threads take consecutive rows of one column, two column groups; the next
  // chunk's values are loaded while the current one is used
  constexpr int STEP = kSvtThreads / kSvtChunk, NV = NC / STEP;
  const int srow = tid % kSvtChunk, scol = tid / kSvtChunk;
  float2 v[NV];
  SvtRow stage(a, c0, c1, c2, srow, kSvtChunk);
  auto load = [&](int r0) {
    const bool in = r0 + srow < R;
    const float2* src = a.x + stage.off + scol * col_stride;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = in && scol + STEP * k < n ? src[STEP * k * col_stride] : make_float2(0.f, 0.f);
    stage.next(a);
  };
  load(0);
#pragma unroll 1
  for (int r0 = 0; r0 < R; r0 += kSvtChunk) {
    const int nr = (R - r0) < kSvtChunk ? (R - r0) : kSvtChunk;
    __syncthreads();  // the previous rows have been used
#pragma unroll
    for (int k = 0; k < NV; ++k) rows[srow * C::RLD + scol + STEP * k] = v[k];
    __syncthreads();
    if (r0 + kSvtChunk < R) load(r0 + kSvtChunk);
    if (group < C::GROUPS) {
#pragma unroll 1
      for (int r = group; r < nr; r += C::GROUPS) {
        // shared memory delivers 4 bytes per lane and cycle, broadcast or not, so the rows stay in single
        // precision there
        const float4* u = reinterpret_cast<const float4*>(rows + r * C::RLD + 4 * ti);
        const float4* w = reinterpret_cast<const float4*>(rows + r * C::RLD + 4 * tj);
        double2 ui[4];
        float2 wf[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float4 p = u[i], q = w[i];
          ui[2 * i] = make_double2((double)p.x, (double)p.y);
          ui[2 * i + 1] = make_double2((double)p.z, (double)p.w);
          wf[2 * i] = make_float2(q.x, q.y);
          wf[2 * i + 1] = make_float2(q.z, q.w);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double2 wj = make_double2((double)wf[j].x, (double)wf[j].y);
#pragma unroll
          for (int i = 0; i < 4; ++i) {  // conj(u_i) w_j
            g[i][j].x = fma(ui[i].x, wj.x, fma(ui[i].y, wj.y, g[i][j].x));
            g[i][j].y = fma(ui[i].x, wj.y, fma(-ui[i].y, wj.x, g[i][j].y));
          }
        }
      }
    }
  }
  for (int i = tid; i < NC * LD; i += kSvtThreads) V[i] = make_double2(i / LD == i % LD ? 1.0 : 0.0, 0.0);
  // the groups add up in a fixed order
  if constexpr (C::SHUFFLE) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      if (d >= C::WARP_GROUPS) continue;
      const bool add = wgroup < d && wgroup + d < C::WARP_GROUPS;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double x = __shfl_down_sync(0xffffffffu, g[i][j].x, d * C::TILES);
          const double y = __shfl_down_sync(0xffffffffu, g[i][j].y, d * C::TILES);
          if (add) g[i][j] = make_double2(g[i][j].x + x, g[i][j].y + y);
        }
    }
  }
  constexpr int SUMS = C::SHUFFLE ? kSvtThreads / 32 : C::GROUPS;
  const int sum = !C::SHUFFLE ? group : wgroup == 0 ? tid / 32 : SUMS;  // this thread's, if it has one
#pragma unroll 1
  for (int k = 0; k < SUMS; ++k) {
    if (sum == k) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          double2* at = A + (4 * ti + i) * LD + 4 * tj + j;
          *at = k == 0 ? g[i][j] : make_double2(at->x + g[i][j].x, at->y + g[i][j].y);
        }
    }
    __syncthreads();
  }

  // 2. Jacobi rotations of the upper triangle of G (A).  m: n rounded up to even; a padding index
  // has a zero row and column.  This thread's block of A (pairs bi < bj) and parts of V (pair, row):
  const int m = (n + 1) & ~1, np = m / 2;
  int bi = 0, bj = tid;  // tid counts the pairs of pairs (bi, bj), bi < bj
  while (bi < np && bj >= np - 1 - bi) {
    bj -= np - 1 - bi;
    ++bi;
  }
  bj = bi < np ? bj + bi + 1 : bi;
  constexpr int kVTasks = (NC / 2 * NC + kSvtThreads - 33) / (kSvtThreads - 32);
  int vtask[kVTasks];
#pragma unroll
  for (int t = 0; t < kVTasks; ++t) {
    const int i = tid - 32 + t * (kSvtThreads - 32);
    vtask[t] = tid >= 32 && i < np * n ? (i / n) | (i % n) << 5 : -1;
  }
  // rotations of a round into buffer `to`, and what they make of the diagonal blocks (threads < np)
  auto rotations = [&](int round, int to) {
    if (tid >= np) return;
    // round-robin tournament: m - 1 stays, the others turn
    int p = tid == 0 ? m - 1 : round + tid, q = round - tid;
    if (tid > 0 && p >= m - 1) p -= m - 1;
    if (q < 0) q += m - 1;
    if (p > q) {
      const int h = p;
      p = q;
      q = h;
    }
    const double2 apq = A[p * LD + q];
    const double app = A[p * LD + p].x, aqq = A[q * LD + q].x;
    const double mag2 = apq.x * apq.x + apq.y * apq.y;
    double c = 1.0, f = 0.0;  // s e = f apq
    if (mag2 > 1e-300) {
      // t = sign(d) |apq| / (|d| + sqrt(d^2 + |apq|^2)), d = (aqq - app) / 2; c = 1 / sqrt(1 + t^2)
      const double d = 0.5 * (aqq - app), h = fabs(d) + sqrt(d * d + mag2);
      const double te = (d < 0.0 ? -1.0 : 1.0) / h;  // t e = te apq
      c = rsqrt(1.0 + te * te * mag2);
      f = c * te;
      A[p * LD + p].x = app - te * mag2;  // t |apq| = te |apq|^2
      A[q * LD + q].x = aqq + te * mag2;
      A[p * LD + q] = make_double2(0.0, 0.0);
    }
    rot_pq[to][tid] = make_int2(p, q);
    rot_c[to][tid] = c;
    rot_s[to][tid] = make_double2(f * apq.x, f * apq.y);
  };
  auto sum2 = [&](bool diagonal) {  // sum of |A|^2 over the full matrix, with or without its diagonal
    double part = 0.0;
    for (int i = tid; i < NC * NC; i += kSvtThreads) {
      const int p = i / NC, q = i % NC;
      if (p < q || (diagonal && p == q)) {
        const double2 v = A[p * LD + q];
        part += (p < q ? 2.0 : 1.0) * (v.x * v.x + v.y * v.y);
      }
    }
    return svt_block_sum(part, red);
  };
  const double fro = sum2(true);
#pragma unroll 1
  for (int sweep = 0; sweep < kSvtMaxSweeps; ++sweep) {
    if (!(sum2(false) > 1e-30 * fro)) break;  // uniform across the block
    rotations(0, 0);
    __syncthreads();
#pragma unroll 1
    for (int round = 0; round < m - 1; ++round) {
      const int cur = round & 1;
      // new_p = c col_p - conj(se) col_q, new_q = se col_p + c col_q (columns; rows with se conjugated)
      if (bi < bj) {
        const int2 I = rot_pq[cur][bi], J = rot_pq[cur][bj];
        const double ci = rot_c[cur][bi], cj = rot_c[cur][bj];
        const double2 si = rot_s[cur][bi], sj = rot_s[cur][bj];
        auto get = [&](int r, int c) {
          const double2 v = A[r < c ? r * LD + c : c * LD + r];
          return make_double2(v.x, r < c ? v.y : -v.y);
        };
        const double2 pp = get(I.x, J.x), pq = get(I.x, J.y), qp = get(I.y, J.x), qq = get(I.y, J.y);
        auto left = [&](double2 u, double2 v) {
          return make_double2(cj * u.x - (sj.x * v.x + sj.y * v.y), cj * u.y - (sj.x * v.y - sj.y * v.x));
        };
        auto right = [&](double2 u, double2 v) {
          return make_double2(sj.x * u.x - sj.y * u.y + cj * v.x, sj.x * u.y + sj.y * u.x + cj * v.y);
        };
        const double2 tpp = left(pp, pq), tpq = right(pp, pq), tqp = left(qp, qq), tqq = right(qp, qq);
        auto top = [&](double2 u, double2 v) {
          return make_double2(ci * u.x - (si.x * v.x - si.y * v.y), ci * u.y - (si.x * v.y + si.y * v.x));
        };
        auto low = [&](double2 u, double2 v) {
          return make_double2(si.x * u.x + si.y * u.y + ci * v.x, si.x * u.y - si.y * u.x + ci * v.y);
        };
        auto put = [&](int r, int c, double2 v) {  // only the upper triangle is kept
          A[r < c ? r * LD + c : c * LD + r] = r < c ? v : make_double2(v.x, -v.y);
        };
        put(I.x, J.x, top(tpp, tqp));
        put(I.y, J.x, low(tpp, tqp));
        put(I.x, J.y, top(tpq, tqq));
        put(I.y, J.y, low(tpq, tqq));
      }
      __syncthreads();
      // the next round's rotations (warp 0) beside this round's update of V (the other warps)
      if (tid < 32) {
        if (round + 1 < m - 1) rotations(round + 1, cur ^ 1);
      } else {
#pragma unroll
        for (int t = 0; t < kVTasks; ++t) {
          if (vtask[t] < 0) break;
          const int b = vtask[t] & 31, k = vtask[t] >> 5;
          const int2 J = rot_pq[cur][b];
          const double c = rot_c[cur][b];
          const double2 se = rot_s[cur][b], u = V[k * LD + J.x], v = V[k * LD + J.y];
          V[k * LD + J.x] = make_double2(c * u.x - (se.x * v.x + se.y * v.y), c * u.y - (se.x * v.y - se.y * v.x));
          V[k * LD + J.y] = make_double2(se.x * u.x - se.y * u.y + c * v.x, se.x * u.y + se.y * u.x + c * v.y);
        }
      }
      __syncthreads();
    }
  }
  // 3a. thresholded weights f(s)/s per eigenvalue
  if (tid < n) {
    const double ev = A[tid * LD + tid].x;
    const double sv = sqrt(ev > 0.0 ? ev : 0.0);
    double w = 0.0;
    if (a.soft) {
      w = sv > (double)a.thresh ? (sv - (double)a.thresh) / sv : 0.0;
    } else {
      int larger = 0;  // rank of this eigenvalue (ties broken by index)
      for (int j = 0; j < n; ++j) {
        const double lj = A[j * LD + j].x;
        larger += (lj > ev || (lj == ev && j < tid)) ? 1 : 0;
      }
      w = larger < a.rank ? 1.0 : 0.0;
    }
    wdiag[tid] = w;
  }
  __syncthreads();
  // 3b. W = V diag(w) V^H (zero in the padding)
  for (int i = tid; i < NC * NC; i += kSvtThreads) {
    const int r = i / NC, c = i % NC;
    double sx = 0.0, sy = 0.0;
    if (r < n && c < n) {
      for (int j = 0; j < n; ++j) {
        const double2 vr = V[r * LD + j], vc = V[c * LD + j];  // V[r][j] w_j conj(V[c][j])
        sx += wdiag[j] * (vr.x * vc.x + vr.y * vc.y);
        sy += wdiag[j] * (vr.y * vc.x - vr.x * vc.y);
      }
    }
    W[i] = make_float2((float)sx, (float)sy);
  }
  __syncthreads();
  // 3c. rows <- rows W, in place, last rows first (the end of the block is still in L2 from the
  // Gram pass); a thread takes two rows, side by side in FP32x2 pairs
  const int last = tid + (R - 1) / (2 * kSvtThreads) * (2 * kSvtThreads) + kSvtThreads;
  SvtRow it(a, c0, c1, c2, last, kSvtThreads);
#pragma unroll 1
  for (int r = last - kSvtThreads; r >= 0; r -= 2 * kSvtThreads) {
    const bool one = r < R, two = r + kSvtThreads < R;
    const long long off1 = it.off;
    it.prev(a);
    const long long off0 = it.off;
    it.prev(a);
    if (!one) continue;
    float2* row0 = a.x + off0;
    float2* row1 = two ? a.x + off1 : row0;
    float2 vx[NC], vy[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const float2 u = c < n ? row0[c * col_stride] : make_float2(0.f, 0.f);
      const float2 v = c < n ? row1[c * col_stride] : make_float2(0.f, 0.f);
      vx[c] = make_float2(u.x, v.x);
      vy[c] = make_float2(u.y, v.y);
    }
#pragma unroll 1
    for (int c = 0; c < n; ++c) {
      // the four real products in chains of their own: half the length, so the rounding of a plain sum
      float2 xx = make_float2(0.f, 0.f), yy = xx, xy = xx, yx = xx;
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const float2 w = W[j * NC + c];
        const float2 wx = make_float2(w.x, w.x), wy = make_float2(w.y, w.y);
        xx = __ffma2_rn(vx[j], wx, xx);
        yy = __ffma2_rn(vy[j], wy, yy);
        xy = __ffma2_rn(vx[j], wy, xy);
        yx = __ffma2_rn(vy[j], wx, yx);
      }
      const float2 ox = csub(xx, yy), oy = cadd(xy, yx);
      row0[c * col_stride] = make_float2(ox.x, oy.x);
      if (two) row1[c * col_stride] = make_float2(ox.y, oy.y);
    }
  }
}

// ADMM vector steps around the CG x-update and the SVT z-update (scaled form, constraint
// x = z; lib/op/opalgs.cpp:103-111, lib/mri/batch_sense.ixx:302-431):
//   stage 0: b = b0 + (rho/2) (z - u)    (right-hand side of (A^H A + rho/2 I) x = b)
//   stage 1: z = x + u                   (input of the proximal step, thresholded in place)
//   stage 2: u = u + x - z               (dual update)
__global__ void admm_vectors_kernel(long long n, int stage, const float2* x, float2* z, float2* u, const float2* b0,
                                    float2* b, float rho) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (stage == 0) {
    b[i] = cadd(b0[i], cscale(csub(z[i], u[i]), 0.5f * rho));
  } else if (stage == 1) {
    z[i] = cadd(x[i], u[i]);
  } else {
    u[i] = cadd(u[i], csub(x[i], z[i]));
  }
}

}  // namespace hb
