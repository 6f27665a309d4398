// Non-uniform FFT (types 1 and 2) on sm_100a: the gridding method with the
// "exponential of semicircle" kernel of Barnett, Magland and af Klinteberg (SIAM J. Sci.
// Comput. 41, 2019), the method of the finufft/cufinufft libraries that the reference
// calls (hasty::fft::CUDANufft, lib/fft/nufft.cpp:540-767).
//
// Conventions (those of the reference's plans): coordinates [3][K] float32, row a pairs
// with image axis a (nufft.cpp:192-197), any real value, 2*pi periodic; modes are
// centred, k_a = i_a - floor(N_a/2) for array index i_a < N_a;
//   type 1:  f[k] = sum_j c_j exp(isign * i * k . x_j)
//   type 2:  c_j  = sum_k f[k] exp(isign * i * k . x_j)
// Fine grid n_a = 2 N_a (upsampling 2).  Kernel width w from the tolerance,
// phi(z) = exp(beta * (sqrt(1 - (2z/w)^2) - 1)) for |z| < w/2 (z in fine-grid cells),
// beta = 2.30 w.  Type 1 = spread c_j * phi(g - u_j) onto the fine grid (u_j = x_j n/(2pi)),
// FFT with sign isign, divide by phi_hat(k) and crop; type 2 = the transpose.
//
// Samples are bucketed by fine-grid bin once per plan (counting sort into an array of grid
// positions), so that spreading (nufft_spread_kernels.cuh) finds the samples near a tile and
// interpolation walks the grid with locality.  The order of a bin's samples comes from
// atomics, so type 1 is not bitwise reproducible across plans, as the reference's cufinufft
// is not.
#pragma once

#include "common.cuh"

namespace hb {

constexpr int kNufftMaxBatch = 32;  // largest maxbatch of a plan
constexpr int kNufftGroup = 8;      // transforms interleaved in one grid
struct CoilMaps {  // coil-map pointers by value
  const float2* s[kNufftMaxBatch];
};
constexpr float kNufftInvTwoPi = 0.159154943091895336f;

// A plan of dimension d < 3 keeps the 3-axis layout with its leading 3 - d axes
// degenerate (N = n = 1, one bin, coordinates 0, no spreading along them, correction 1).
struct NufftGeom {
  int N[3];          // modes per axis
  int n[3];          // fine grid per axis (2 N; 1 on a degenerate axis)
  int bin[3];        // cells per bin: (4, 4, 8) for spreading by tiles, (8, 8, 8) without; (1, 8, 8) in 2-D, (1, 1, 8) in 1-D
  int nb[3];         // bins per axis
  int w;             // kernel width (cells)
  float beta;        // kernel shape
  long long K;       // samples
  int dim;           // 1, 2 or 3 transformed axes (the trailing ones)
};
// Kernels on several grids of NB transforms side by side (SIDES) take the grid's number, the side, from
// blockIdx.y; its cells start at nufft_side.  The form for one grid has no trace of it: the address
// arithmetic alone cost the 3-D kernels 0.7 % (forward 128^3 x 16 coils 2333 -> 2351 us).
template <bool SIDES>
__device__ __forceinline__ int side_index() {
  if constexpr (SIDES) return blockIdx.y;
  else return 0;
}
__device__ __forceinline__ long long nufft_side(const NufftGeom& g, int side, int NB) {
  return (long long)side * g.n[0] * g.n[1] * g.n[2] * NB;
}

__device__ __forceinline__ float nufft_grid_pos(float x, int n) {
  float u = x * kNufftInvTwoPi * (float)n;
  u -= (float)n * floorf(u / (float)n);
  return u < (float)n ? u : 0.f;  // rounding may land exactly on n
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Square root of s in [1e-30, 1] without a branch, so that a lane's evaluations overlap: Newton's (Heron's)
// iteration for r^2 = s, r <- r - (r^2 - s) / (2 r), made once from r = s y with y in the place of 1 / r.  y, the
// approximate reciprocal root, is within 2^-22.9 (PTX ISA, rsqrt.approx.f32), so the start is within 2^-22.2;
// the iteration squares that, the residual is exact to an fma's rounding, and the result is within
// 0.5 + 2^-18 ulp of the root.
__device__ __forceinline__ float es_root(float s) {
  const float y = rsqrt_approx(s), r = s * y;
  return fmaf(0.5f * y, fmaf(-r, r, s), r);
}
__device__ __forceinline__ float es_kernel(float z, float beta, float inv_hw) {
  const float t = z * inv_hw;
  const float s = 1.f - t * t;
  const float e = expf(beta * (es_root(fmaxf(s, 1e-30f)) - 1.f));  // s = 0 is kept off the reciprocal
  return s > 0.f ? e : 0.f;
}
// phi[i] = the kernel of width w at z[i], root[i] = es_root(s[i]) (tests)
__global__ void __launch_bounds__(256) nufft_kernel_values_kernel(int w, float beta, const float* z, const float* s, float* phi,
                                                                  float* root, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  phi[i] = es_kernel(z[i], beta, 1.f / (0.5f * (float)w));
  root[i] = es_root(s[i]);
}

// First cell and the W kernel values of one axis.
template <int W>
__device__ __forceinline__ int nufft_axis_weights(float u, float beta, float* wt) {
  const float hw = 0.5f * (float)W;
  const int i0 = (int)ceilf(u - hw);
  const float inv_hw = 1.f / hw;
#pragma unroll
  for (int m = 0; m < W; ++m) wt[m] = es_kernel((float)(i0 + m) - u, beta, inv_hw);
  return i0;
}

__device__ __forceinline__ int wrap(int i, int n) { return i < 0 ? i + n : (i >= n ? i - n : i); }

// *p += v as one vector reduction (no value returned, so the issuing warp does not wait)
__device__ __forceinline__ void red_add(float2* p, float2 v) {
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y) : "memory");
}

// The values to spread: transform b of sample j is c[b * c_ld + j] (1 when c is null), times w[j].
struct SpreadSource {
  const float2* c;
  long long c_ld;
  const float* w;  // nullable
};
__device__ __forceinline__ float2 spread_value(const SpreadSource& src, int b, int j, float csgn) {
  float2 v = src.c ? src.c[b * src.c_ld + j] : make_float2(1.f, 0.f);
  if (src.w) v = cscale(v, src.w[j]);
  v.y *= csgn;
  return v;
}

// ---- binning (once per plan): coords [dim][K] pair with the trailing axes ----
__device__ __forceinline__ float nufft_coord_pos(const NufftGeom& g, const float* coords, int a, long long j) {
  return a < 3 - g.dim ? 0.f : nufft_grid_pos(coords[(a - (3 - g.dim)) * g.K + j], g.n[a]);
}
// bin of every sample and its rank within the bin
__global__ void nufft_bin_count_kernel(NufftGeom g, const float* coords, int2* bin_rank, int* bin_count) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.K) return;
  int bin = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const int bi = (int)nufft_coord_pos(g, coords, a, j) / g.bin[a];
    bin = bin * g.nb[a] + (bi < g.nb[a] ? bi : g.nb[a] - 1);
  }
  bin_rank[j] = make_int2(bin, atomicAdd(&bin_count[bin], 1));
}

// Exclusive prefix sum of n ints: per block of 4096 (block totals to `sums`), a one-block scan
// of the totals, and their addition; out[n] = total.  (A single CTA took 524 us for the
// 262144 bins of a 512^3 grid; this form takes 3 launches of a few us.)
constexpr int kScanBlock = 4096;
__device__ __forceinline__ int block_scan_exclusive(int s, int* part) {  // 1024 threads; part[1024]
  part[threadIdx.x] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int v = threadIdx.x >= d ? part[threadIdx.x - d] : 0;
    __syncthreads();
    part[threadIdx.x] += v;
    __syncthreads();
  }
  return part[threadIdx.x] - s;
}
__global__ void __launch_bounds__(1024) nufft_scan_block_kernel(const int* in, int* out, int* sums, int n) {
  __shared__ int part[1024];
  const int lo = blockIdx.x * kScanBlock + threadIdx.x * 4;
  int v[4], s = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = lo + i < n ? in[lo + i] : 0;
    s += v[i];
  }
  int run = block_scan_exclusive(s, part);
  if (threadIdx.x == 1023) sums[blockIdx.x] = run + s;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (lo + i < n) out[lo + i] = run;
    run += v[i];
  }
}
__global__ void __launch_bounds__(1024) nufft_scan_sums_kernel(int* sums, int nblocks) {  // in place
  __shared__ int part[1024];
  const int per = (nblocks + 1023) / 1024;
  const int lo = threadIdx.x * per, hi = (lo + per) < nblocks ? (lo + per) : nblocks;
  int s = 0;
  for (int i = lo; i < hi; ++i) s += sums[i];
  int run = block_scan_exclusive(s, part);
  for (int i = lo; i < hi; ++i) {
    const int v = sums[i];
    sums[i] = run;
    run += v;
  }
}
__global__ void __launch_bounds__(1024) nufft_scan_add_kernel(const int* in, int* out, const int* sums, int n) {
  const int lo = blockIdx.x * kScanBlock + threadIdx.x * 4, add = sums[blockIdx.x];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (lo + i < n) {
      out[lo + i] += add;
      if (lo + i == n - 1) out[n] = out[n - 1] + in[n - 1];
    }
}

// pts[position] = (u0, u1, u2, sample number), in bin order
__global__ void nufft_bin_scatter_kernel(NufftGeom g, const float* coords, const int2* bin_rank, const int* start,
                                         float4* pts) {
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.K) return;
  const int2 br = bin_rank[j];
  pts[start[br.x] + br.y] = make_float4(nufft_coord_pos(g, coords, 0, j), nufft_coord_pos(g, coords, 1, j),
                                        nufft_coord_pos(g, coords, 2, j), __int_as_float((int)j));
}

// Kernel weights of an axis at position u, or the single weight 1 at cell 0 on a degenerate axis
template <int W, int WA>
__device__ __forceinline__ int nufft_axis(const NufftGeom& g, float u, float* wt) {
  if constexpr (WA == 1) {
    wt[0] = 1.f;
    return 0;
  } else {
    return nufft_axis_weights<W>(u, g.beta, wt);
  }
}

// ---- type 1 by vector reductions into a zeroed grid.  Used where the tile form
// (nufft_spread_kernels.cuh) is not: 1-D plans (a sample has only W cells, fewer than a tile's tests
// would cost) and the point-spread function.  There thousands of equal terms meet at the centre of a
// trajectory, and their sum in single precision rounds by its order: by tiles, single entries of a 128^3
// diagonal move by 2e-3 of its rms.  Whether they move towards the FP64 diagonal (hb_diag_build) entry by
// entry has not been measured (in the L2 norm they do: 3.6e-6 from it, the reductions 1.5e-5); until then the
// diagonals stay what they were. ----
// 1-D, grid [n2][NB], NB = 1 << lgnb: one thread per (sample, transform), transform fastest; blockIdx.y = side
template <int W>
__global__ void __launch_bounds__(256) nufft_spread_line_kernel(NufftGeom g, const float4* pts, const float2* vals,
                                                                int lgnb, float2* grid) {
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long i = id >> lgnb;
  if (i >= g.K) return;
  const float2 v = vals[((long long)blockIdx.y * g.K << lgnb) + id];
  grid += nufft_side(g, blockIdx.y, 1 << lgnb);
  float w[W];
  const int i2 = nufft_axis_weights<W>(pts[i].z, g.beta, w);
#pragma unroll
  for (int m = 0; m < W; ++m) red_add(grid + (wrap(i2 + m, g.n[2]) << lgnb) + (id & ((1 << lgnb) - 1)), cscale(v, w[m]));
}
// 3-D, one transform: one thread per sample.  (Eight lanes per sample, each the cells of one x, take 409
// against 1300 us for 512 k samples on 512^3, but add in another order: see above; single entries of the
// diagonal move by 1e-3 of its rms.)
template <int W>
__global__ void __launch_bounds__(256) nufft_spread_reductions_kernel(NufftGeom g, const float4* pts, const float2* vals,
                                                                      float2* grid) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= g.K) return;
  const float2 cj = vals[i];
  const float4 p = pts[i];
  float w0[W], w1[W], w2[W];
  const int i0 = nufft_axis_weights<W>(p.x, g.beta, w0);
  const int i1 = nufft_axis_weights<W>(p.y, g.beta, w1);
  const int i2 = nufft_axis_weights<W>(p.z, g.beta, w2);
  int x2[W];
#pragma unroll
  for (int m = 0; m < W; ++m) x2[m] = wrap(i2 + m, g.n[2]);
#pragma unroll 1
  for (int a = 0; a < W; ++a) {
    const float2 ca = cscale(cj, w0[a]);
    float2* Ga = grid + (long long)wrap(i0 + a, g.n[0]) * g.n[1] * g.n[2];
#pragma unroll
    for (int b = 0; b < W; ++b) {
      const float2 cab = cscale(ca, w1[b]);
      float2* Gab = Ga + (long long)wrap(i1 + b, g.n[1]) * g.n[2];
#pragma unroll
      for (int m = 0; m < W; ++m) red_add(Gab + x2[m], cscale(cab, w2[m]));
    }
  }
}

// Where interpolated values go: to the caller's rows c[b * c_ld + j], or (c null) through the
// k-space step of the SENSE normal operator, v = (v - y_b[j]) * w[j] (the reference's
// mid-appliers; y and w nullable), to vals[side][i][NB] in sorted order, where spreading reads them.
struct InterpDest {
  float2* c;
  long long c_ld;
  const float2* y[kNufftMaxBatch];
  const float* w;
  float2* vals;
  float vsgn;  // -1 conjugates vals
};

// Stores transform b's value at sample j, which is vals[at].
__device__ __forceinline__ void interp_store(const InterpDest& dst, int b, int nact, long long at, int j, float2 v,
                                             float csgn) {
  if (b >= nact) {
    if (!dst.c) dst.vals[at] = make_float2(0.f, 0.f);
    return;
  }
  v.y *= csgn;
  if (dst.c) {
    dst.c[b * dst.c_ld + j] = v;
    return;
  }
  if (dst.y[b]) v = csub(v, dst.y[b][j]);
  if (dst.w) v = cscale(v, dst.w[j]);
  v.y *= dst.vsgn;
  dst.vals[at] = v;
}

// ---- type 2 of 1-D and 2-D plans: one thread per (sample, transform), transform fastest, blockIdx.y = side;
// csgn = -1 conjugates the result.  In 2-D a sample has W rows, too few to pay for a group of lanes per sample
// (8 transforms, W = 6, 51 k samples: 16 us against 20-26 us). ----
template <int W, int DIM>
__global__ void __launch_bounds__(256) nufft_interp_points_kernel(NufftGeom g, const float4* pts, const float2* grid,
                                                                  int lgnb, int nact, float csgn,
                                                                  const __grid_constant__ InterpDest dst) {
  chained_kernel_begin();
  constexpr int W1 = DIM == 2 ? W : 1;
  const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int bt = (int)(id & ((1 << lgnb) - 1));
  const long long i = id >> lgnb;
  if (i >= g.K) return;
  grid += nufft_side(g, blockIdx.y, 1 << lgnb);
  const float4 p = pts[i];
  float w1[W1], w2[W];
  const int i1 = nufft_axis<W, W1>(g, p.y, w1);
  const int i2 = nufft_axis<W, W>(g, p.z, w2);
  int x2[W];
#pragma unroll
  for (int m = 0; m < W; ++m) x2[m] = (wrap(i2 + m, g.n[2]) << lgnb) + bt;
  float2 acc = make_float2(0.f, 0.f);
#pragma unroll
  for (int b = 0; b < W1; ++b) {
    const float2* row = grid + ((long long)wrap(i1 + b, g.n[1]) * g.n[2] << lgnb);
    float2 s = make_float2(0.f, 0.f);
#pragma unroll
    for (int m = 0; m < W; ++m) {
      const float2 v = row[x2[m]];
      s.x = fmaf(w2[m], v.x, s.x);
      s.y = fmaf(w2[m], v.y, s.y);
    }
    acc.x = fmaf(w1[b], s.x, acc.x);
    acc.y = fmaf(w1[b], s.y, acc.y);
  }
  interp_store(dst, (blockIdx.y << lgnb) + bt, nact, ((long long)blockIdx.y * g.K << lgnb) + id, __float_as_int(p.w), acc,
               csgn);
}

template <int V>
__device__ __forceinline__ void load_cells(const float2* p, float2* v) {  // V float2 as one load
  if constexpr (V == 4) {
    asm("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[2].x), "=f"(v[2].y), "=f"(v[3].x), "=f"(v[3].y)
        : "l"(p));
  } else if constexpr (V == 2) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = make_float2(q.x, q.y);
    v[1] = make_float2(q.z, q.w);
  } else {
    v[0] = *p;
  }
}

// ---- type 2 of a 3-D plan: a group of XL x PL lanes per sample (two to eight samples per warp).  A load
// of the group reads one row of W cells x NB transforms, a contiguous run of the interleaved grid:
// lane = (cell x, part of the cell), up to 32 bytes per lane.  Every lane sums its x over the
// sample's rows (first y, then z), multiplies by its x weight once, and the group's lanes are added up
// at the end.  Neighbours in the sorted order run at the same time, so most rows are in L1.
//
// Bound: latency and the L1 data path together.  A request is served 128 bytes a cycle when its lines are
// aligned, and half of that when every quarter of it straddles two lines; at W = 7 and 8 transforms ncu
// has that path busy 68 % of the cycles (the reads alone would take 0.35 ms of 0.66), a third of the sectors
// missing L1, and the 24 warps per SM that 80 registers allow waiting for loads for 15 of 21 cycles.
// From W = 11 on (tolerances below 1e-9) groups of 4 and 8 spill up to 148 bytes a thread, still
// faster than the form with one thread per value: 64^3 modes, 40 k samples, 8 transforms W = 13 518 us against
// 1231, W = 16 749 against 1814.  Measured, 512 k radial samples on 256^3, one
// thread per (sample, transform) -> this form: 8 transforms, W = 7 1175 -> 663 us, W = 6 665 -> 506 us,
// W = 5 614 -> 360 us, W = 4 328 -> 139 us; 4 transforms, W = 7 609 -> 356 us; 1 transform 253 -> 129 us.
// One warp per sample with 16-byte loads: 738 us (1081 us without the aligned window). ----
constexpr int kInterpWarps = 8;
template <int W, int NB>
struct InterpCfg {
  static constexpr int V = NB < 4 ? NB : 4;                // transforms per lane
  static constexpr int PL = NB / V;                        // lanes per cell
  static constexpr int XL = W <= 4 ? 4 : 8;                // cells per row and load
  static constexpr int XS = (W + XL - 1) / XL;             // loads per row
  static constexpr int LANES = XL * PL, SL = 32 / LANES;   // lanes per sample, samples per warp
  // the load's window starts at a multiple of XA cells (a 128-byte line of 8 transforms is 2 cells, of 4
  // transforms 4) where it is wide enough to reach over the row from there
  static constexpr int LINE = NB == 8 ? 2 : NB == 4 ? 4 : 1, XA = XS * XL >= W + LINE - 1 ? LINE : 1;
  static constexpr int ROUNDS = 4;                         // samples per group
  static constexpr int PER_CTA = kInterpWarps * SL * ROUNDS;
};
template <int W, int NB, bool SIDES>
__global__ void __launch_bounds__(32 * kInterpWarps, W <= 5 && NB > 1 ? 4 : 3)
nufft_interp_rows_kernel(NufftGeom g, const float4* pts, const float2* grid, int nact, float csgn,
                         const __grid_constant__ InterpDest dst) {
  chained_kernel_begin();
  using C = InterpCfg<W, NB>;
  constexpr int V = C::V, PL = C::PL, XL = C::XL, XS = C::XS, SL = C::SL;
  __shared__ float w_s[kInterpWarps][SL][3 * W];  // z, y, x weights of the warp's samples
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int p = lane % PL, xl = (lane / PL) % XL, sl = lane / C::LANES;
  const float hw = 0.5f * (float)W, inv_hw = 1.f / hw;
  const unsigned rowlen = (unsigned)g.n[2] * NB, planelen = (unsigned)g.n[1] * rowlen;
  const int side = side_index<SIDES>();
  grid += nufft_side(g, side, NB);
  const long long base = (long long)blockIdx.x * C::PER_CTA + warp * SL;
#pragma unroll 1
  for (int k = 0; k < C::ROUNDS; ++k) {
    const long long w0 = base + k * (kInterpWarps * SL);  // the warp's first sample
    if (w0 >= g.K) break;
    const long long i = w0 + sl < g.K ? w0 + sl : g.K - 1;
    const float4 pt = pts[i];
    const int c0 = (int)ceilf(pt.x - hw), c1 = (int)ceilf(pt.y - hw), c2 = (int)ceilf(pt.z - hw);
    __syncwarp();  // the previous weights have been read
#pragma unroll
    for (int m = lane % C::LANES; m < 3 * W; m += C::LANES) {
      const int ax = m / W, t = m - ax * W;
      const float u = ax == 0 ? pt.x : ax == 1 ? pt.y : pt.z;
      const int c = ax == 0 ? c0 : ax == 1 ? c1 : c2;
      w_s[warp][sl][m] = es_kernel((float)(c + t) - u, g.beta, inv_hw);
    }
    __syncwarp();
    const float* wt = w_s[warp][sl];
    unsigned yo[W], xo[XS];
    float2 wy[W];
    bool xok[XS];
#pragma unroll
    for (int b = 0; b < W; ++b) {
      wy[b] = make_float2(wt[W + b], wt[W + b]);
      yo[b] = (unsigned)wrap(c1 + b, g.n[1]) * rowlen;
    }
    const int x0 = (c2 & ~(C::XA - 1)) - c2 + xl;
#pragma unroll
    for (int c = 0; c < XS; ++c) {
      const int x = x0 + c * XL;
      xok[c] = x >= 0 && x < W;
      xo[c] = (unsigned)wrap(c2 + (xok[c] ? x : 0), g.n[2]) * NB + V * p;
    }
    float2 acc[XS][V];
#pragma unroll
    for (int c = 0; c < XS; ++c)
#pragma unroll
      for (int v = 0; v < V; ++v) acc[c][v] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int a = 0; a < W; ++a) {
      const unsigned zo = (unsigned)wrap(c0 + a, g.n[0]) * planelen;
      float2 s[XS][V];
#pragma unroll
      for (int c = 0; c < XS; ++c)
#pragma unroll
        for (int v = 0; v < V; ++v) s[c][v] = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < XS; ++c)
        if (xok[c]) {
#pragma unroll
          for (int b = 0; b < W; ++b) {
            float2 q[V];
            load_cells<V>(grid + (zo + yo[b] + xo[c]), q);  // fewer than 2^32 values in a grid
#pragma unroll
            for (int v = 0; v < V; ++v) s[c][v] = __ffma2_rn(wy[b], q[v], s[c][v]);
          }
        }
      const float2 wz = make_float2(wt[a], wt[a]);
#pragma unroll
      for (int c = 0; c < XS; ++c)
#pragma unroll
        for (int v = 0; v < V; ++v) acc[c][v] = __ffma2_rn(wz, s[c][v], acc[c][v]);
    }
    float2 r[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      r[v] = make_float2(0.f, 0.f);
#pragma unroll
      for (int c = 0; c < XS; ++c)
        if (xok[c]) {
          const float w = wt[2 * W + x0 + c * XL];
          r[v] = __ffma2_rn(make_float2(w, w), acc[c][v], r[v]);
        }
    }
    // add up the group's lanes; while a lane has several transforms, each half keeps half of them
    int b = V * p, d = C::LANES / 2;
#pragma unroll
    for (int h = V / 2; h >= 1; h /= 2, d /= 2) {
      const bool hi = lane & d;
#pragma unroll
      for (int v = 0; v < h; ++v) {
        const float2 give = hi ? r[v] : r[v + h], keep = hi ? r[v + h] : r[v];
        r[v] = cadd(keep, make_float2(__shfl_xor_sync(0xffffffffu, give.x, d), __shfl_xor_sync(0xffffffffu, give.y, d)));
      }
      b += hi ? h : 0;
    }
    // The halving above has left every transform to LANES / V neighbouring lanes (one lane each for four
    // transforms and four cells a load); the first of them (PL = 2: of both parts) stores.
    constexpr int same = C::LANES / V;
    static_assert(same >= 1 && same * V == C::LANES, "a group holds every transform");
#pragma unroll
    for (; d >= PL; d /= 2)
      r[0] = cadd(r[0], make_float2(__shfl_xor_sync(0xffffffffu, r[0].x, d), __shfl_xor_sync(0xffffffffu, r[0].y, d)));
    if (lane % same < PL && w0 + sl < g.K) 
      interp_store(dst, side * NB + b, nact, (side * g.K + i) * NB + b, __float_as_int(pt.w), r[0], csgn);
  }
}

// ---- tables (once per plan): corr = 1/phi_hat per axis [N0 | N1 | N2], team twiddles of n0, n1, n2 ----
// phi_hat(k) = integral over |z| < w/2 of phi(z) cos(2 pi k z / n), by 64-point Gauss-Legendre quadrature on
// [0, w/2] (the integrand is even); relative error below 1e-11 for the widths of tolerances <= 1e-4.
// In FP64 on the device: on the host the 64 x (N0 + N1 + N2) exponentials and cosines took 3 ms for a 256^3 plan.
constexpr int kGaussNodes = 64;
struct GaussLegendre {
  double x[kGaussNodes], w[kGaussNodes];
};
__global__ void __launch_bounds__(256) nufft_corr_kernel(NufftGeom g, double beta, const __grid_constant__ GaussLegendre gl,
                                                         float* corr) {
  const int id = blockIdx.x * blockDim.x + threadIdx.x;
  if (id >= g.N[0] + g.N[1] + g.N[2]) return;
  const int a = id < g.N[0] ? 0 : id < g.N[0] + g.N[1] ? 1 : 2;
  if (a < 3 - g.dim) {
    corr[id] = 1.f;
    return;
  }
  const int i = id - (a > 0 ? g.N[0] : 0) - (a > 1 ? g.N[1] : 0);
  const int k = i - g.N[a] / 2, n = g.n[a];
  const double hw = 0.5 * g.w;
  double acc = 0.0;
  for (int j = 0; j < kGaussNodes; ++j) {
    const double z = 0.5 * hw * (gl.x[j] + 1.0);
    const double t = z / hw, s = 1.0 - t * t;
    const double phi = s > 0.0 ? exp(beta * (sqrt(s) - 1.0)) : 0.0;
    acc += gl.w[j] * phi * cos(2.0 * 3.14159265358979323846 * k * z / n);
  }
  corr[id] = (float)(1.0 / (hw * acc));  // 2 x (hw / 2) x the sum
}

}  // namespace hb
