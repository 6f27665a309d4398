// The NUFFT's fine-grid transforms: one kernel per axis on a grid whose transforms
// (coils) are interleaved, with the zero padding, the crop, the kernel correction and the
// coil maps folded into the passes.
//
// Grid layout of a group of NB = 1, 2, 4 or 8 transforms: [n0][n1][n2][NB] complex64.  A
// cell's NB values are neighbours, so spreading and interpolation move 8 * NB contiguous
// bytes per cell instead of NB scattered 8-byte ones, and every axis, the contiguous one
// included, is transformed as columns of a [L][16] tile.
//
// Only the N_a = n_a / 2 central modes of an axis are wanted (type 1) or non-zero (type 2):
// grid cells [0, N_a/2) and [n_a - N_a/2, n_a), the "kept" cells.  The passes run in the order
// that lets each one skip what the next does not read:
//   type 1:  z (all columns; kept z stored) -> y (kept z; kept y stored) -> x + modes
//   type 2:  modes + x (kept z, y) -> y (kept z, kept y loaded) -> z (kept z loaded)
// so no pass reads or writes padding, nothing is zeroed first, and the grid crosses HBM
// about 2.6 times per transform instead of 7.3 (memset, three full in-place passes, and
// a separate mode pass; coil expansion and combination were two more kernels).
//
// All passes compute the forward transform; the caller conjugates what enters and leaves the
// chain for the other sign.
//
// Bound: HBM (each pass reads and writes its share of the grid once).  One CTA owns a tile
// of L rows x 16 columns (128-byte rows), staged by 16-byte asynchronous copies; the FFT's
// exchange reuses the tile, so a CTA needs 128 L bytes + twiddles (34 KB at L = 256) and
// several CTAs per SM overlap their copies with each other's arithmetic.  Measured at 128^3
// modes x 16 transforms: 1000 us for the three passes with the coil combination (type 1, 5.9 TB/s
// in the two axis passes) against 3210 us of memset, in-place passes, mode pass and combination
// on separate grids; type 2 1060 us against 3200 us.
#pragma once

#include "bulk.cuh"
#include "common.cuh"
#include "fft.cuh"
#include "nufft_kernels.cuh"

namespace hb {

template <int L>
struct TilePassCfg {
  static constexpr int E = TeamCfg<L>::E, S = TeamCfg<L>::S;
  static constexpr int XT = 16;            // tile columns (float2)
  static constexpr int THREADS = XT * S;   // one team per column
  static constexpr int SMEM = L * XT + L;  // float2 slots: tile + twiddles
  static_assert(E % 4 == 0, "the kept quarters are whole register groups");
  static_assert((S & (S - 1)) == 0, "the exchange XORs lane numbers");
};

// Column c of row r sits at r * 16 + (c ^ 2 (r % 8)): the 16-byte pairs of a row are permuted by
// the row number (a pair stays whole, so it can be copied and read as 16 bytes), and a
// half-warp that reads 8 consecutive rows x 2 adjacent columns touches all 32 banks once.
__device__ __forceinline__ int tile_at(int r, int c) { return r * 16 + (c ^ ((r & 7) << 1)); }

// Lane -> (column, lane of the team): the two columns of a pair alternate between lanes, see tile_at.
template <int S>
__device__ __forceinline__ void tile_team(int* col, int* t) {
  const int w = threadIdx.x / 32, l = threadIdx.x % 32;
  *t = (l >> 1) % S;
  *col = w * (32 / S) + 2 * (l / (2 * S)) + (l & 1);
}

// Forward L-point FFT of tile column `col`, natural order in and out, in place; rows
// outside the kept quarters are taken as zero when PAD.  The exchange XORs the lane with the
// row as team_fft_dout_to_din_xor does, inside the team's own column, so teams need no
// barrier among themselves.
template <int L, bool PAD>
__device__ __forceinline__ void tile_fft(float2* tile, int col, int t, const float2* tws) {
  constexpr int E = TeamCfg<L>::E, S = TeamCfg<L>::S;
  float2 v[E];
#pragma unroll
  for (int e = 0; e < E; ++e)
    v[e] = (PAD && e >= E / 4 && e < 3 * E / 4) ? make_float2(0.f, 0.f) : tile[tile_at(t + S * e, col)];
  Dft<E, -1>::run(v);
  __syncwarp();  // the team has read its column
#pragma unroll
  for (int k1 = 0; k1 < E; ++k1) tile[tile_at(k1 * S + (t ^ (k1 % S)), col)] = cmul(v[k1], tws[k1 * S + t]);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < E / S; ++c) {
    float2 u[S];
#pragma unroll
    for (int j = 0; j < S; ++j) u[j] = tile[tile_at((t + S * c) * S + (j ^ t), col)];
    Dft<S, -1>::run(u);
#pragma unroll
    for (int k2 = 0; k2 < S; ++k2) v[c * S + k2] = u[k2];
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < E; ++r) tile[tile_at(dout_index<L>(t, r), col)] = v[r];
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Grid cell of kept index i of an axis (N modes on n cells): [0, N/2) and [n - N/2, n).
__device__ __forceinline__ int kept_cell(int i, int N, int n) { return i < N - N / 2 ? i : i + (n - N); }

// Transform along a strided axis, in place: row r of column q lies at base + r * row_stride + q,
// q < ncols contiguous, base = grid + kept_cell(blockIdx.y) * outer_stride.  PAD: only kept
// rows are loaded (type 2); otherwise only kept rows are stored (type 1).
template <int L, bool PAD>
__global__ void __launch_bounds__(TilePassCfg<L>::THREADS)
nufft_axis_pass_kernel(float2* grid, long long row_stride, int ncols, int outer_N, int outer_n, long long outer_stride,
                       const float2* tw) {
  chained_kernel_begin();
  using C = TilePassCfg<L>;
  extern __shared__ __align__(128) float2 smem[];
  float2* tile = smem;
  float2* tws = tile + L * C::XT;
  const int q0 = blockIdx.x * C::XT;
  float2* base = grid + kept_cell(blockIdx.y, outer_N, outer_n) * outer_stride + q0;
  const int npair = (ncols - q0) < C::XT ? (ncols - q0) / 2 : C::XT / 2;  // ncols is even
  constexpr int ROWS_IN = PAD ? L / 2 : L, ROWS_OUT = PAD ? L : L / 2;
  for (int i = threadIdx.x; i < ROWS_IN * 8; i += C::THREADS) {
    const int k = i / 8, u = i % 8;
    const int r = PAD ? (k < L / 4 ? k : k + L / 2) : k;
    if (u < npair) cp_async16(&tile[tile_at(r, 2 * u)], base + r * row_stride + 2 * u);
  }
  cp_async_commit();
  for (int i = threadIdx.x; i < L; i += C::THREADS) tws[i] = tw[i];
  cp_async_wait<0>();
  __syncthreads();
  int col, t;
  tile_team<C::S>(&col, &t);
  tile_fft<L, PAD>(tile, col, t, tws);  // columns past ncols transform leftovers that are not stored
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS_OUT * 8; i += C::THREADS) {
    const int k = i / 8, u = i % 8;
    const int r = PAD ? k : (k < L / 4 ? k : k + L / 2);
    if (u < npair)
      *reinterpret_cast<float4*>(base + r * row_stride + 2 * u) = *reinterpret_cast<const float4*>(&tile[tile_at(r, 2 * u)]);
  }
}

// Mode side of a group of transforms: either plain mode arrays (transform b at f + b * f_ld),
// or the SENSE operators' coil-weighted images: coil b's modes are maps.s[b] * x (type 2), and
// out = add + sum_b conj(maps.s[b]) * modes_b (type 1).
struct NufftModeOp {
  float2* f;         // plain modes (read by type 2, written by type 1); null selects the coil form
  long long f_ld;
  float circulant;   // nonzero: type 1 writes circulant order (offset d at d mod N) times this factor
  const float2* x;   // coil form, type 2: the image
  float2* out;       // coil form, type 1: the combined image
  const float2* add;  // coil form, type 1: what the sum starts from (null: zero; may be out)
  CoilMaps maps;
};

// One CTA transforms 16 >> lgnb x-lines of NB = 1 << lgnb transforms: tile column = line * NB + b.
// A side has transforms side * NB + b; nact exist in all, the others are zero and are not stored.
// sgn = -1 conjugates the modes.

// Grid offset (cells) and y, z correction of the CTA's lines, once per CTA: 64-bit products and a division
// per element cost more than the transform.
__device__ __forceinline__ void mode_lines(const NufftGeom& g, int line0, int nl, const float* corr, long long* cell,
                                           float* scale) {
  if ((int)threadIdx.x < nl) {
    const int line = min(line0 + (int)threadIdx.x, g.N[0] * g.N[1] - 1);
    const int i0 = line / g.N[1], i1 = line - i0 * g.N[1];
    const int k0 = i0 - g.N[0] / 2, k1 = i1 - g.N[1] / 2;
    const int c0 = k0 < 0 ? k0 + g.n[0] : k0, c1 = k1 < 0 ? k1 + g.n[1] : k1;
    cell[threadIdx.x] = ((long long)c0 * g.n[1] + c1) * g.n[2];
    scale[threadIdx.x] = corr[i0] * corr[g.N[0] + i1];
  }
}

// type 2: grid lines = FFT along x of the corrected modes, at the kept (z, y) rows
template <int L, bool SIDES>
__global__ void __launch_bounds__(TilePassCfg<L>::THREADS)
nufft_modes_to_grid_kernel(NufftGeom g, const __grid_constant__ NufftModeOp op, int lgnb, int nact, float sgn, const float* corr,
                           const float2* tw, float2* grid) {
  chained_kernel_begin();
  using C = TilePassCfg<L>;
  constexpr int N2 = L / 2;
  extern __shared__ __align__(128) float2 smem[];
  float2* tile = smem;
  float2* tws = tile + L * C::XT;
  const int nb = 1 << lgnb, nl = C::XT >> lgnb;
  const int nlines = g.N[0] * g.N[1], line0 = blockIdx.x * nl;
  const float* corr2 = corr + g.N[0] + g.N[1];
  __shared__ long long cell_s[C::XT];
  __shared__ float scale_s[C::XT];
  mode_lines(g, line0, nl, corr, cell_s, scale_s);
  for (int i = threadIdx.x; i < L; i += C::THREADS) tws[i] = tw[i];
  // all loads of a thread first (E / 2 columns' modes), then the tile
  constexpr int LD = C::XT * N2 / C::THREADS;
  static_assert(LD * C::THREADS == C::XT * N2, "whole rounds");
  float2 v[LD], w[LD];
#pragma unroll
  for (int k = 0; k < LD; ++k) {
    const int i = threadIdx.x + k * C::THREADS, i2 = i % N2, col = i / N2;
    const int line = line0 + (col >> lgnb), b = (side_index<SIDES>() << lgnb) + (col & (nb - 1));
    v[k] = w[k] = make_float2(0.f, 0.f);
    if (line < nlines && b < nact) {
      const long long m = (long long)line * N2 + i2;
      v[k] = op.f ? op.f[b * op.f_ld + m] : op.x[m];
      if (!op.f) w[k] = op.maps.s[b][m];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < LD; ++k) {
    const int i = threadIdx.x + k * C::THREADS, i2 = i % N2, col = i / N2;
    float2 u = cscale(op.f ? v[k] : cmul(v[k], w[k]), scale_s[col >> lgnb] * corr2[i2]);
    u.y *= sgn;
    tile[tile_at(i2 < N2 / 2 ? i2 + L - N2 / 2 : i2 - N2 / 2, col)] = u;
  }
  __syncthreads();
  int col, t;
  tile_team<C::S>(&col, &t);
  tile_fft<L, true>(tile, col, t, tws);
  __syncthreads();
  grid += nufft_side(g, side_index<SIDES>(), nb);
  auto row_base = [&](int lc) { return grid + (cell_s[lc] << lgnb); };  // grid line of the CTA's mode line
  if (lgnb == 0) {
    for (int i = threadIdx.x; i < C::XT * L; i += C::THREADS) {
      const int r = i % L, c = i / L;
      if (line0 + c < nlines) row_base(c)[r] = tile[tile_at(r, c)];
    }
  } else {
    const int lgp = lgnb - 1;  // 16-byte pairs per cell
    for (int i = threadIdx.x; i < 8 * L; i += C::THREADS) {
      const int r = (i >> lgp) % L, lc = (i >> lgp) / L, p = i & ((1 << lgp) - 1);
      if (line0 + lc < nlines)
        *reinterpret_cast<float4*>(row_base(lc) + (r << lgnb) + 2 * p) =
            *reinterpret_cast<const float4*>(&tile[tile_at(r, (lc << lgnb) + 2 * p)]);
    }
  }
}

// type 1: modes = correction x FFT along x of the grid lines at the kept (z, y) rows (coil form: one side a
// launch, the sum runs through all coils)
template <int L, bool SIDES>
__global__ void __launch_bounds__(TilePassCfg<L>::THREADS)
nufft_grid_to_modes_kernel(NufftGeom g, const __grid_constant__ NufftModeOp op, int lgnb, int nact, float sgn, const float* corr,
                           const float2* tw, const float2* grid) {
  chained_kernel_begin();
  using C = TilePassCfg<L>;
  constexpr int N2 = L / 2;
  extern __shared__ __align__(128) float2 smem[];
  float2* tile = smem;
  float2* tws = tile + L * C::XT;
  const int nb = 1 << lgnb, nl = C::XT >> lgnb;
  const int nlines = g.N[0] * g.N[1], line0 = blockIdx.x * nl;
  const float* corr2 = corr + g.N[0] + g.N[1];
  __shared__ long long cell_s[C::XT];
  __shared__ float scale_s[C::XT];
  mode_lines(g, line0, nl, corr, cell_s, scale_s);
  __syncthreads();
  grid += nufft_side(g, side_index<SIDES>(), nb);
  auto row_base = [&](int lc) { return grid + (cell_s[lc] << lgnb); };
  if (lgnb == 0) {
    for (int i = threadIdx.x; i < C::XT * L; i += C::THREADS) {
      const int r = i % L, c = i / L;
      if (line0 + c < nlines) cp_async8(&tile[tile_at(r, c)], row_base(c) + r);
    }
  } else {
    const int lgp = lgnb - 1;
    for (int i = threadIdx.x; i < 8 * L; i += C::THREADS) {
      const int r = (i >> lgp) % L, lc = (i >> lgp) / L, p = i & ((1 << lgp) - 1);
      if (line0 + lc < nlines)
        cp_async16(&tile[tile_at(r, (lc << lgnb) + 2 * p)], row_base(lc) + (r << lgnb) + 2 * p);
    }
  }
  cp_async_commit();
  for (int i = threadIdx.x; i < L; i += C::THREADS) tws[i] = tw[i];
  cp_async_wait<0>();
  __syncthreads();
  int col, t;
  tile_team<C::S>(&col, &t);
  tile_fft<L, false>(tile, col, t, tws);  // columns past nlines transform leftovers that are not stored
  __syncthreads();
  const int per = op.f ? C::XT : nl;  // plain: one output per column; coil form: one per line
  for (int i = threadIdx.x; i < per * N2; i += C::THREADS) {
    const int i2 = i % N2, c = i / N2;
    const int lc = op.f ? c >> lgnb : c, line = line0 + lc;
    if (line >= nlines) continue;
    const int r = i2 < N2 / 2 ? i2 + L - N2 / 2 : i2 - N2 / 2;
    const float s = scale_s[lc] * corr2[i2];
    const long long m = (long long)line * N2 + i2;
    if (op.f) {
      const int b = (side_index<SIDES>() << lgnb) + (c & (nb - 1));
      if (b >= nact) continue;
      float2 v = cscale(tile[tile_at(r, c)], s);
      v.y *= sgn;
      if (op.circulant != 0.f) {
        const int i0 = line / g.N[1], i1 = line % g.N[1];
        const int j0 = (i0 + g.N[0] / 2) % g.N[0], j1 = (i1 + g.N[1] / 2) % g.N[1], j2 = (i2 + N2 / 2) % N2;
        op.f[((long long)j0 * g.N[1] + j1) * N2 + j2] = cscale(v, op.circulant);
      } else {
        op.f[b * op.f_ld + m] = v;
      }
    } else {
      float2 acc = op.add ? op.add[m] : make_float2(0.f, 0.f);
      float2 w[kNufftGroup];
#pragma unroll
      for (int b = 0; b < kNufftGroup; ++b)
        if (b < nact) w[b] = op.maps.s[b][m];
#pragma unroll
      for (int b = 0; b < kNufftGroup; ++b)
        if (b < nact) {
          float2 v = cscale(tile[tile_at(r, (lc << lgnb) + b)], s);
          v.y *= sgn;
          acc = cadd(acc, cmulc(v, w[b]));
        }
      op.out[m] = acc;
    }
  }
}

}  // namespace hb
