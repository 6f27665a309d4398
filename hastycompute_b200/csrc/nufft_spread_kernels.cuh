// Type-1 spreading without a zeroed grid and, but for crowded tiles, without atomics: one warp owns
// a tile of grid cells, holds its sums for all transforms of the group in registers, and
// visits the samples that reach the tile.
//
// The plan sorts its samples into bins (nufft_bin_*), so the samples near a tile are a few
// contiguous runs of the sorted array.  A warp loads 128 candidates at a time, collects those
// whose kernel support meets the tile, and per batch of 32 collected samples evaluates the
// kernel at the tile's coordinates of each axis (4 + 4 + 8 values for a 4 x 4 x 8 tile, zero
// outside the support) and accumulates weight x value into every cell.  A tile that few
// samples reach is written once.  Near the centre of a radial trajectory thousands do: the plan
// cuts the candidates of such a tile into pieces of at most `cap`, which add into cells
// zeroed beforehand (nufft_zero_tiles_kernel).
//
// Bound: the FP32 pipe, 59 % of its cycles busy in ncu (an FP32x2 FMA takes it for two), issue 56 % (5.6 M
// visits of 32 packed FMAs + about 50 other instructions), at the 15 warps per SM that are there on average
// of the 20 that fit: one-warp CTAs come and go, and the phases of a batch (collecting, weights, visits) of a
// warp depend on one another.  The reduction form it replaces issued W^3 vector reductions per sample and
// transform.  Measured at W = 7, 512 k radial samples on a 256^3 grid:
// 8 transforms 751 us + 24 us (gathering the values) + 9 us (zeroing) against 2145 + 172 us,
// 4: 484 us, 1: 307 us against 916 us.  Choices, 8 transforms: one warp per CTA (two: 1192 us, a
// CTA waits for its slower warp; four: 1140 us), 96 registers (128: 825 us), long pieces first
// (in tile order: 821 us), values gathered into sorted order first (read from the caller's rows:
// 1018 us).  Tile: 4 x 4 x 8 gives each lane 64 accumulators for 8 transforms; a
// sample visits 10.9 tiles at W = 7, where a quarter of the weights are inside its support.
#pragma once

#include "common.cuh"
#include "nufft_kernels.cuh"

namespace hb {

// Cells and transforms of a lane: x = l % 8, then the y group and the half of the transforms.
// A visit reads the lane's weights and transform values from shared memory, which delivers 4 bytes
// per lane and cycle whether or not the lanes share an address.  In 3-D with eight transforms
// each half of the warp therefore takes four of them on two y (cells z = 0..3 x 2 y): 15 cycles of
// reads a visit instead of 22 for all of them on one y (751 us against 775 us for 512 k samples on a
// 256^3 grid, 525 against 546 for 128^3).  Elsewhere a lane holds one y (in 2-D four) and all
// transforms: the added products undo it with four transforms (485 us against 537) and in 2-D
// (28.2 us against 30.4 for 128 x 128 modes x 8).
template <int DIM, int NB>
struct SpreadLane {
  static constexpr int HALVES = DIM == 3 && NB == 8 ? 2 : 1, TL = NB / HALVES;  // transforms of a lane
  static constexpr int YC = HALVES, R = 4 * YC;                                // y in 3-D, cells
  static constexpr int YG = 4 / HALVES;                                        // y groups
};
template <int DIM>
struct SpreadTile {
  static constexpr int T0 = DIM == 3 ? 4 : 1, T1 = DIM == 3 ? 4 : 16, T2 = 8;
  static constexpr int NW = (DIM == 3 ? T0 : 0) + T1 + T2;  // kernel values per sample
};
constexpr int kSpreadBatch = 32;  // samples whose kernel values are evaluated together
constexpr int kSpreadChunk = 4;   // candidates a lane loads at once
constexpr int kSpreadList = kSpreadBatch - 1 + 32 * kSpreadChunk;

// One piece of a tile's work: candidates [begin, end) in the tile's run order; origin = its first
// cell, x | y << 10 | z << 20; split = the tile has several pieces.
struct SpreadItem {
  int origin, begin, end, split;
};
template <int DIM>
__device__ __forceinline__ int tile_origin(const NufftGeom& g, int tile) {
  using T = SpreadTile<DIM>;
  const int t2 = g.n[2] / T::T2, t1 = (g.n[1] + T::T1 - 1) / T::T1;
  return (tile % t2) * T::T2 | ((tile / t2) % t1) * T::T1 << 10 | (tile / (t2 * t1)) * T::T0 << 20;
}

// The sample runs of a tile: bins (z, y, x-range) in unwrapped numbering, in z, y, x order; the
// x-range of a bin row is one run per period of the grid that it meets.  A kernel reaches at
// most a quarter of the grid past either end (n >= 2w), so periods are -1, 0 or 1 and need no
// division.
template <int DIM>
struct TileRuns {
  static constexpr int LB0 = DIM == 3 ? 2 : 0, LB1 = DIM == 3 ? 2 : 3, LB2 = 3;  // log2 cells per bin (nufft_bins)
  int o[3];           // first cell of the tile
  int b0, b1, b2;     // first (unwrapped) bin per axis
  int m1, count;      // bins along y; runs
  int e2;             // last (unwrapped) x bin
  int p2, nx;         // first period of x, periods
  float im1;
  __device__ __forceinline__ static int period(int b, int nb) { return b < 0 ? -1 : (b >= nb ? 1 : 0); }
  __device__ __forceinline__ TileRuns(const NufftGeom& g, int origin) {
    using T = SpreadTile<DIM>;
    o[2] = origin & 1023;
    o[1] = (origin >> 10) & 1023;
    o[0] = origin >> 20;
    // a sample at u reaches cells (u - w/2, u + w/2): u in (first - w/2, last + w/2)
    const int h = (g.w + 1) / 2;
    int m0 = 1;
    b0 = 0;
    if (DIM == 3) {
      b0 = (o[0] - h) >> LB0;
      m0 = ((o[0] + T::T0 - 1 + h) >> LB0) - b0 + 1;
    }
    b1 = (o[1] - h) >> LB1;
    m1 = ((min(o[1] + T::T1, g.n[1]) - 1 + h) >> LB1) - b1 + 1;
    b2 = (o[2] - h) >> LB2;
    e2 = (o[2] + T::T2 - 1 + h) >> LB2;
    p2 = period(b2, g.nb[2]);
    nx = period(e2, g.nb[2]) - p2 + 1;
    count = m0 * m1 * nx;
    im1 = 1.f / (float)m1;
  }
  // run r: samples [s, s + len), periods (q0, q1, q2) of its bins; returns len
  __device__ __forceinline__ int run(const NufftGeom& g, const int* start, int r, int* s, int* q0, int* q1, int* q2) const {
    const int row = nx == 1 ? r : nx == 2 ? r >> 1 : (int)(((float)r + 0.5f) * (1.f / 3.f));
    const int ix = r - row * nx, iz = (int)(((float)row + 0.5f) * im1), iy = row - iz * m1;  // exact: small integers
    *q0 = DIM == 3 ? period(b0 + iz, g.nb[0]) : 0;
    *q1 = period(b1 + iy, g.nb[1]);
    *q2 = p2 + ix;
    const int lo = max(b2, *q2 * g.nb[2]) - *q2 * g.nb[2], hi = min(e2, (*q2 + 1) * g.nb[2] - 1) - *q2 * g.nb[2];
    const int at = ((b0 + iz - *q0 * g.nb[0]) * g.nb[1] + (b1 + iy - *q1 * g.nb[1])) * g.nb[2];
    *s = start[at + lo];
    return start[at + hi + 1] - *s;
  }
};

// ---- plan time: candidates per tile and the number of pieces, then the list of pieces.  The
// pieces of split tiles come first: they are the long ones, and a kernel that ends with
// them waits for a few warps (the centre of the grid is the last tile in z, y, x order). ----
struct SpreadCounts {
  int items, split_tiles, split_items, single_items;
};
__device__ __forceinline__ int spread_pieces(int candidates, int cap) {
  return candidates > cap ? (candidates + cap - 1) / cap : 1;
}
template <int DIM>
__global__ void __launch_bounds__(256)
nufft_tile_count_kernel(NufftGeom g, const int* start, int ntiles, int cap, int* candidates, SpreadCounts* n) {
  const int tile = blockIdx.x * blockDim.x + threadIdx.x;
  int pieces = 0;
  if (tile < ntiles) {
    const TileRuns<DIM> tr(g, tile_origin<DIM>(g, tile));
    int tot = 0, s, q0, q1, q2;
    for (int r = 0; r < tr.count; ++r) tot += tr.run(g, start, r, &s, &q0, &q1, &q2);
    candidates[tile] = tot;
    pieces = spread_pieces(tot, cap);
  }
  pieces = __reduce_add_sync(0xffffffffu, pieces);
  if (threadIdx.x % 32 == 0) atomicAdd(&n->items, pieces);
}
template <int DIM>
__global__ void __launch_bounds__(256)
nufft_tile_items_kernel(NufftGeom g, int ntiles, int cap, const int* candidates, SpreadItem* items, int* split_tiles,
                        SpreadCounts* n) {
  const int tile = blockIdx.x * blockDim.x + threadIdx.x;
  if (tile >= ntiles) return;
  const int tot = candidates[tile], pieces = spread_pieces(tot, cap), origin = tile_origin<DIM>(g, tile);
  if (pieces == 1) {
    items[n->items - 1 - atomicAdd(&n->single_items, 1)] = {origin, 0, tot, 0};
    return;
  }
  const int at = atomicAdd(&n->split_items, pieces);
  for (int i = 0; i < pieces; ++i) items[at + i] = {origin, i * cap, min(tot, (i + 1) * cap), 1};
  split_tiles[atomicAdd(&n->split_tiles, 1)] = origin;
}

// ---- per call ----
// Zeroes the cells of a tile that several pieces add into.
template <int DIM, int THREADS>
__device__ __forceinline__ void zero_tile(const NufftGeom& g, int origin, int lgnb, float2* grid) {
  using T = SpreadTile<DIM>;
  const int o0 = origin >> 20, o1 = (origin >> 10) & 1023, o2 = origin & 1023;
  for (int i = threadIdx.x; i < T::T0 * T::T1 * (T::T2 << lgnb); i += THREADS) {
    const int q = i % (T::T2 << lgnb), y = (i / (T::T2 << lgnb)) % T::T1, z = i / ((T::T2 << lgnb) * T::T1);
    if (o1 + y < g.n[1])
      grid[((((long long)(o0 + z) * g.n[1] + o1 + y) * g.n[2] + o2) << lgnb) + q] = make_float2(0.f, 0.f);
  }
}
template <int DIM>
__global__ void __launch_bounds__(128) nufft_zero_tiles_kernel(NufftGeom g, const int* split_tiles, int lgnb, float2* grid) {
  chained_kernel_begin();
  zero_tile<DIM, 128>(g, split_tiles[blockIdx.x], lgnb, grid + nufft_side(g, blockIdx.y, 1 << lgnb));
}

// vals[side][i][b] = the value of sorted sample i for transform side * NB + b (zero from nact on), so that a tile
// reads a sample's NB values as one contiguous run: gathered straight from the caller's
// [transform][sample] rows, every visit of a sample (about 11 of them at W = 7) touched NB
// separate cache lines.  CTAs from `gather_ctas` on zero a split tile each: a launch of their own costs
// 2 us, which a type 1 of one 160 x 160 slice with 150 k samples (45 us) had lost against spreading by reductions.
template <int DIM, bool SIDES>
__global__ void __launch_bounds__(256) nufft_gather_values_kernel(NufftGeom g, const float4* pts,
                                                                  const __grid_constant__ SpreadSource src, int lgnb,
                                                                  int nact, float csgn, float2* vals,
                                                                  unsigned gather_ctas, const int* split_tiles,
                                                                  float2* grid) {
  chained_kernel_begin();
  const int side = side_index<SIDES>();
  if (blockIdx.x >= gather_ctas) {
    zero_tile<DIM, 256>(g, split_tiles[blockIdx.x - gather_ctas], lgnb, grid + nufft_side(g, side, 1 << lgnb));
    return;
  }
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int b = (side << lgnb) + (int)(id & ((1 << lgnb) - 1));
  const long long i = id >> lgnb;
  if (i >= g.K) return;
  vals[(side * g.K << lgnb) + id] = b < nact ? spread_value(src, b, __float_as_int(pts[i].w), csgn) : make_float2(0.f, 0.f);
}

__device__ __forceinline__ void store_cell8(float2* p, const float2* v) {  // four float2, one 32-byte store
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0].x), "f"(v[0].y), "f"(v[1].x),
               "f"(v[1].y), "f"(v[2].x), "f"(v[2].y), "f"(v[3].x), "f"(v[3].y)
               : "memory");
}
__device__ __forceinline__ void red_add4(float2* p, float2 a, float2 b) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y) : "memory");
}

template <int DIM, int NB, bool SIDES>
__global__ void __launch_bounds__(32, NB < 4 ? 28 : NB == 4 ? 24 : DIM == 3 ? 20 : 16)
nufft_spread_tiles_kernel(NufftGeom g, const float4* pts, const int* start, const SpreadItem* items,
                          const float2* vals, float2* grid) {
  chained_kernel_begin();
  using T = SpreadTile<DIM>;
  constexpr int NW = T::NW, WX = NW - T::T2;  // x values last
  __shared__ float4 list[kSpreadList];  // position relative to the tile's first cell, sorted index
  __shared__ __align__(16) float w_s[kSpreadBatch][NW];
  __shared__ __align__(16) float2 c_s[kSpreadBatch][NB];
  const int lane = threadIdx.x;
  const int side = side_index<SIDES>();
  vals += side * g.K * NB;
  grid += nufft_side(g, side, NB);
  const SpreadItem it = items[blockIdx.x];
  const TileRuns<DIM> tr(g, it.origin);

  using Q = SpreadLane<DIM, NB>;
  constexpr int R = Q::R, TL = Q::TL, YC = Q::YC;
  const int yg = (lane / 8) % Q::YG, tb = TL * (lane / (8 * Q::YG));  // y group, first transform
  float2 acc[R][TL];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int b = 0; b < TL; ++b) acc[r][b] = make_float2(0.f, 0.f);
  const float hw = 0.5f * (float)g.w, inv_hw = 1.f / hw;

  // kernel values: lane l evaluates cell coordinate l % 16 of every other sample: in 3-D z 0-3, y 0-3,
  // x 0-7, in 2-D y 0-15
  const int wi = lane % 16;
  const int wax = DIM == 3 ? (wi < 4 ? 0 : wi < 8 ? 1 : 2) : 1;
  const float wm = (float)(DIM == 3 ? (wi < 4 ? wi : wi < 8 ? wi - 4 : wi - 8) : wi);
  const int nruns = tr.count;
  int listed = 0;               // collected samples
  int rb = -32, pos = 0;        // runs [rb, rb + 32) are loaded, one per lane; candidates before them
  int total = 0, k0 = 0, k_end = 0;  // their candidates; next candidate, end of the piece among them
  int incl = 0, first = 0;      // lane's run: candidates up to its end, its first sample - candidates before it
  float f0 = 0.f, f1 = 0.f, f2 = 0.f;  // unwrapped tile origin seen by the lane's run
  bool more = true;
#pragma unroll 1
  for (;;) {
    // collect at least a batch of samples, up to 128 candidates at a time
#pragma unroll 1
    while (listed < kSpreadBatch && more) {
      if (k0 >= k_end) {  // next 32 runs
        rb += 32;
        pos += total;
        more = rb < nruns && pos < it.end;
        if (!more) break;
        int s = 0, len = 0, q0 = 0, q1 = 0, q2 = 0;
        if (rb + lane < nruns) len = tr.run(g, start, rb + lane, &s, &q0, &q1, &q2);
        incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane >= d) incl += v;
        }
        first = s + len - incl;
        total = __shfl_sync(0xffffffffu, incl, 31);
        f0 = (float)(tr.o[0] - q0 * g.n[0]);
        f1 = (float)(tr.o[1] - q1 * g.n[1]);
        f2 = (float)(tr.o[2] - q2 * g.n[2]);
        k_end = min(total, it.end - pos);
        k0 = max(0, it.begin - pos);
        if (k0 >= k_end) continue;
      }
      float4 p[kSpreadChunk];
      int run[kSpreadChunk], at[kSpreadChunk];
#pragma unroll
      for (int c = 0; c < kSpreadChunk; ++c) {
        // the run of candidate k: the first whose inclusive count exceeds k
        const int k = k0 + 32 * c + lane;
        int r = 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
          const int v = __shfl_sync(0xffffffffu, incl, r + d - 1);
          if (v <= k) r += d;
        }
        run[c] = r;
        const int si = __shfl_sync(0xffffffffu, first, r);
        at[c] = k < k_end ? si + k : 0;
        p[c] = pts[at[c]];
      }
#pragma unroll
      for (int c = 0; c < kSpreadChunk; ++c) {
        const float o0 = __shfl_sync(0xffffffffu, f0, run[c]), o1 = __shfl_sync(0xffffffffu, f1, run[c]),
                    o2 = __shfl_sync(0xffffffffu, f2, run[c]);
        const float d0 = p[c].x - o0, d1 = p[c].y - o1, d2 = p[c].z - o2;
        const bool in = k0 + 32 * c + lane < k_end && (DIM < 3 || (d0 > -hw && d0 < (float)(T::T0 - 1) + hw)) &&
                        d1 > -hw && d1 < (float)(T::T1 - 1) + hw && d2 > -hw && d2 < (float)(T::T2 - 1) + hw;
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in) list[listed + __popc(mask & ((1u << lane) - 1u))] = make_float4(d0, d1, d2, __int_as_float(at[c]));
        listed += __popc(mask);
      }
      k0 += 32 * kSpreadChunk;
    }
    const int n = min(listed, kSpreadBatch);
    if (n == 0) break;
    // the batch is taken from the end of the list, so nothing has to move
    listed -= n;
    const float4* pt = list + listed;
    __syncwarp();

    // transform values (first: their latency hides behind the weights; entries past n repeat the
    // last) and kernel values of the batch
    constexpr int EC = 32 / NB;  // entries per round of value loads
    float2 cv[kSpreadBatch / EC];
#pragma unroll
    for (int k = 0; k < kSpreadBatch / EC; ++k)
      cv[k] = vals[(long long)__float_as_int(pt[min(k * EC + lane / NB, n - 1)].w) * NB + lane % NB];
    {
      const float* pe = reinterpret_cast<const float*>(pt) + wax;
#pragma unroll 4
      for (int e = lane / 16; e < n; e += 2) w_s[e][lane % 16] = es_kernel(wm - pe[4 * e], g.beta, inv_hw);
      if (DIM == 2) {  // the eight x values
#pragma unroll 4
        for (int e = lane / 8; e < n; e += 4)
          w_s[e][WX + lane % 8] = es_kernel((float)(lane % 8) - reinterpret_cast<const float*>(pt + e)[2], g.beta, inv_hw);
      }
    }
#pragma unroll
    for (int k = 0; k < kSpreadBatch / EC; ++k) (&c_s[0][0])[k * 32 + lane] = cv[k];
    __syncwarp();

#pragma unroll 2
    for (int e = 0; e < n; ++e) {
      const float* w = w_s[e];
      const float wx = w[WX + lane % 8];
      float wr[R];  // weights of the lane's cells: z major in 3-D
      if constexpr (DIM == 3) {
        const float4 wz = *reinterpret_cast<const float4*>(w);
        float wyx[YC];
        if constexpr (YC == 2) {
          const float2 wy = *reinterpret_cast<const float2*>(w + T::T0 + 2 * yg);
          wyx[0] = wy.x * wx;
          wyx[1] = wy.y * wx;
        } else {
          wyx[0] = w[T::T0 + yg] * wx;
        }
#pragma unroll
        for (int y = 0; y < YC; ++y) {
          wr[y] = wz.x * wyx[y];
          wr[YC + y] = wz.y * wyx[y];
          wr[2 * YC + y] = wz.z * wyx[y];
          wr[3 * YC + y] = wz.w * wyx[y];
        }
      } else {
        const float4 wy = *reinterpret_cast<const float4*>(w + R * yg);
        wr[0] = wy.x * wx;
        wr[1] = wy.y * wx;
        wr[2] = wy.z * wx;
        wr[3] = wy.w * wx;
      }
      float2 cv2[TL];
      if constexpr (TL >= 2) {
#pragma unroll
        for (int b = 0; b < TL; b += 2) {
          const float4 q = *reinterpret_cast<const float4*>(&c_s[e][tb + b]);
          cv2[b] = make_float2(q.x, q.y);
          cv2[b + 1] = make_float2(q.z, q.w);
        }
      } else {
        cv2[0] = c_s[e][0];
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float2 wv = make_float2(wr[r], wr[r]);
#pragma unroll
        for (int b = 0; b < TL; ++b) acc[r][b] = __ffma2_rn(wv, cv2[b], acc[r][b]);
      }
    }
    __syncwarp();
  }

#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int z = tr.o[0] + (DIM == 3 ? r / YC : 0), y = tr.o[1] + (DIM == 3 ? YC * yg + r % YC : R * yg + r);
    if (DIM == 2 && y >= g.n[1]) continue;
    float2* p = grid + (((long long)z * g.n[1] + y) * g.n[2] + tr.o[2] + lane % 8) * NB + tb;
    if (it.split) {
      if constexpr (TL == 1) red_add(p, acc[r][0]);
      else
#pragma unroll
        for (int b = 0; b < TL; b += 2) red_add4(p + b, acc[r][b], acc[r][b + 1]);
    } else {
      if constexpr (TL == 1) p[0] = acc[r][0];
      else if constexpr (TL == 2) *reinterpret_cast<float4*>(p) = make_float4(acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y);
      else
#pragma unroll
        for (int b = 0; b < TL; b += 4) store_cell8(p + b, &acc[r][b]);
    }
  }
}

}  // namespace hb
