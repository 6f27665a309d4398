// C ABI of the NUFFT (types 1 and 2) and the SENSE forward/adjoint around it
// (include/hasty_b200.h, section "Non-uniform FFT").  Replaces the cufinufft plans of
// hasty::fft::CUDANufft (lib/fft/nufft.cpp:540-767, declared nufft.ixx:108-160), the
// coil loops of the SENSE operators that use them (lib/mri/sense.ixx:426-497) and the
// NUFFT construction of the Toeplitz diagonal (build_diagonal_base, nufft.cpp:932-971).
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <vector>

#include "../../include/hasty_b200.h"
#include "fft3_launch.cuh"
#include "nufft_kernels.cuh"
#include "nufft_pass_kernels.cuh"
#include "nufft_spread_kernels.cuh"
#include "runtime.cuh"

using namespace hb;
using hb::fftl::fft3_grid;
using hb::fftl::team_length;
using hb::fftl::team_tables_device;

struct hb_nufft {
  int device;
  NufftGeom g;
  int group;                // transforms interleaved in one grid: 1, 2, 4 or 8
  int sides;                // grids side by side (1, or up to 4 of 8 transforms in small plans)
  void* mem = nullptr;        // one allocation (null: in the creator's workspace): the arrays below up to image
  float4* pts = nullptr;      // [K] grid positions and sample numbers in bin order
  int* start = nullptr;       // [bins + 1] first position of every bin
  float* corr = nullptr;      // [N0 | N1 | N2] 1 / phi_hat
  float2* tw = nullptr;       // team twiddle tables of n0, n1, n2 (offsets 0, n0, n0 + n1)
  float2* grid = nullptr;     // [sides][n0][n1][n2][group]
  float2* vals = nullptr;     // [sides][K][group] values to spread, in sorted order
  float2* image = nullptr;    // [modes] sum of the coils so far of a call with several groups
  // spreading (2-D and 3-D): pieces of tile work and the tiles cut into several
  void* items_mem = nullptr;
  SpreadItem* items = nullptr;
  int* split_tiles = nullptr;
  int nitems = 0, nsplit = 0;
};

namespace {

// Kernel width for a requested tolerance (upsampling 2): w = ceil(log10(1/tol)) + 1.
int width_for_tol(double tol) {
  int w = (int)std::ceil(std::log10(1.0 / tol)) + 1;
  return w < 2 ? 2 : (w > 16 ? 16 : w);
}

// Gauss-Legendre nodes and weights on [-1, 1] (Newton iteration on the Legendre
// polynomial, the textbook method), computed once.
const GaussLegendre& gauss_legendre() {
  static const GaussLegendre gl = [] {
    GaussLegendre r;
    const int n = kGaussNodes;
    for (int i = 0; i < n; ++i) {
      double z = std::cos(M_PI * (i + 0.75) / (n + 0.5)), dp = 1.0;
      for (int it = 0; it < 100; ++it) {
        double p0 = 1.0, p1 = z;  // P_0, P_1
        for (int k = 2; k <= n; ++k) {
          const double p2 = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
          p0 = p1;
          p1 = p2;
        }
        dp = n * (z * p1 - p0) / (z * z - 1.0);  // P_n'(z)
        const double dz = p1 / dp;
        z -= dz;
        if (std::fabs(dz) < 1e-16) break;
      }
      r.x[i] = z;
      r.w[i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
    return r;
  }();
  return gl;
}

// Plans whose calls are bound by their launches: 1-D, 2-D, and 3-D of up to 16^3 modes.  (A larger 3-D grid
// keeps the GPU busy with 8 transforms.)
bool small_plan(const NufftGeom& g) { return g.dim < 3 || (long long)g.n[0] * g.n[1] * g.n[2] <= 32768; }

// Transforms of one set of launches: nact <= nz * NB, NB = 1 << lgnb interleaved in each of nz grids.
// Sizes that are not a power of two are padded, except 5 in 3-D, which runs as 4 + 1 (padding it to 8 moves
// 1.6 times the bytes); at 3, 6 and 7, and in small plans, a second set of launches costs more than the
// padding (type 1 of 5 transforms, 8^3 modes and 1 k samples: 22 us padded, 36 us as 4 + 1).
// Beyond 8 transforms small plans run several grids in one set of launches: type 1 of 16 transforms, 64 x 64
// modes and 3 k samples, tol 1e-3, 22 us against 40 us one grid after the other; 32 of 64 modes and 300 samples
// 17 against 44 us.  The last grid may be padded, too: always from 5 transforms on, which would be padded on
// their own as well, and below that where the padding is less work than another set of launches.  9
// transforms, 160 x 160 modes, type 1: 52 us padded and 64 us on its own at 30 k samples, 147 and 131 us at
// 150 k; 12: 147 and 147 us at 150 k.
struct Group {
  int nact, lgnb, nz;
};
Group next_group(const hb_nufft* p, int64_t left) {
  if (left > p->group && p->sides > 1) {
    const int64_t full = left / p->group < p->sides ? left / p->group : p->sides, rem = left - full * p->group;
    const int64_t cells = (int64_t)p->g.n[0] * p->g.n[1] * p->g.n[2];
    const bool pad = full < p->sides && rem > 0 &&
                     (rem > 4 || (p->g.K + cells / 8) * (p->group - rem) <= (int64_t)1 << 19);
    const int64_t nz = full + (pad ? 1 : 0), n = nz * p->group;
    return {(int)(left < n ? left : n), 3, (int)nz};
  }
  int n = (int)(left < p->group ? left : p->group);
  if (n == 5 && !small_plan(p->g)) n = 4;
  return {n, n > 4 ? 3 : n > 2 ? 2 : n - 1, 1};
}

template <int W>
cudaError_t spread_reductions_w(const hb_nufft* p, Group q, cudaStream_t st) {
  LaunchScope ls(HB_KERNEL_NUFFT, st);
  if (p->g.dim == 3) {  // one transform
    nufft_spread_reductions_kernel<W><<<(unsigned)((p->g.K + 255) / 256), 256, 0, st>>>(p->g, p->pts, p->vals, p->grid);
  } else {
    const dim3 grid((unsigned)(((p->g.K << q.lgnb) + 255) / 256), q.nz);
    nufft_spread_line_kernel<W><<<grid, 256, 0, st>>>(p->g, p->pts, p->vals, q.lgnb, p->grid);
  }
  return cudaGetLastError();
}
template <int W>
cudaError_t interp_w(const hb_nufft* p, const InterpDest& dst, Group q, float csgn, cudaStream_t st) {
  LaunchScope ls(HB_KERNEL_NUFFT, st);
  if (p->g.dim < 3) {
    const dim3 grid((unsigned)(((p->g.K << q.lgnb) + 255) / 256), q.nz);
    return launch_chained(p->g.dim == 2 ? nufft_interp_points_kernel<W, 2> : nufft_interp_points_kernel<W, 1>, grid, 256, 0, st,
                          p->g, p->pts, p->grid, q.lgnb, q.nact, csgn, dst);
  }
  auto go = [&](auto kernel, int per_cta) {
    const dim3 grid((unsigned)((p->g.K + per_cta - 1) / per_cta), q.nz);
    return launch_chained(kernel, grid, 32 * kInterpWarps, 0, st, p->g, p->pts, p->grid, q.nact, csgn, dst);
  };
  if (q.nz > 1) return go(nufft_interp_rows_kernel<W, 8, true>, InterpCfg<W, 8>::PER_CTA);
  if (q.lgnb == 3) return go(nufft_interp_rows_kernel<W, 8, false>, InterpCfg<W, 8>::PER_CTA);
  if (q.lgnb == 2) return go(nufft_interp_rows_kernel<W, 4, false>, InterpCfg<W, 4>::PER_CTA);
  if (q.lgnb == 1) return go(nufft_interp_rows_kernel<W, 2, false>, InterpCfg<W, 2>::PER_CTA);
  return go(nufft_interp_rows_kernel<W, 1, false>, InterpCfg<W, 1>::PER_CTA);
}

// p->vals = the values to spread, and zeros in the split tiles
template <int DIM>
cudaError_t gather_dim(const hb_nufft* p, const SpreadSource& src, Group q, float csgn, cudaStream_t st) {
  const unsigned ctas = (unsigned)(((p->g.K << q.lgnb) + 255) / 256);
  LaunchScope ls(HB_KERNEL_NUFFT, st);
  return launch_chained(q.nz > 1 ? nufft_gather_values_kernel<DIM, true> : nufft_gather_values_kernel<DIM, false>,
                        dim3(ctas + p->nsplit, q.nz), 256, 0, st, p->g, p->pts, src, q.lgnb, q.nact, csgn, p->vals, ctas,
                        p->split_tiles, p->grid);
}
cudaError_t gather_values(const hb_nufft* p, const SpreadSource& src, Group q, float csgn, cudaStream_t st) {
  return p->g.dim == 3 ? gather_dim<3>(p, src, q, csgn, st) : gather_dim<2>(p, src, q, csgn, st);
}
// Zeros in the split tiles, where interpolation has written p->vals
cudaError_t zero_tiles(const hb_nufft* p, Group q, cudaStream_t st) {
  if (p->nsplit == 0) return cudaSuccess;
  LaunchScope ls(HB_KERNEL_NUFFT, st);
  return launch_chained(p->g.dim == 3 ? nufft_zero_tiles_kernel<3> : nufft_zero_tiles_kernel<2>, dim3(p->nsplit, q.nz), 128, 0,
                        st, p->g, p->split_tiles, q.lgnb, p->grid);
}

template <int DIM>
cudaError_t spread_tiles(const hb_nufft* p, Group q, cudaStream_t st) {
  LaunchScope ls(HB_KERNEL_NUFFT, st);
  auto go = [&](auto kernel) {
    return launch_chained(kernel, dim3(p->nitems, q.nz), 32, 0, st, p->g, p->pts, p->start, p->items, p->vals, p->grid);
  };
  if (q.nz > 1) return go(nufft_spread_tiles_kernel<DIM, 8, true>);
  if (q.lgnb == 3) return go(nufft_spread_tiles_kernel<DIM, 8, false>);
  if (q.lgnb == 2) return go(nufft_spread_tiles_kernel<DIM, 4, false>);
  if (q.lgnb == 1) return go(nufft_spread_tiles_kernel<DIM, 2, false>);
  return go(nufft_spread_tiles_kernel<DIM, 1, false>);
}

#define HB_W_DISPATCH(FN, ...)                                                                      \
  switch (p->g.w) {                                                                                 \
    case 2: return FN<2>(__VA_ARGS__);   case 3: return FN<3>(__VA_ARGS__);                          \
    case 4: return FN<4>(__VA_ARGS__);   case 5: return FN<5>(__VA_ARGS__);                          \
    case 6: return FN<6>(__VA_ARGS__);   case 7: return FN<7>(__VA_ARGS__);                          \
    case 8: return FN<8>(__VA_ARGS__);   case 9: return FN<9>(__VA_ARGS__);                          \
    case 10: return FN<10>(__VA_ARGS__); case 11: return FN<11>(__VA_ARGS__);                        \
    case 12: return FN<12>(__VA_ARGS__); case 13: return FN<13>(__VA_ARGS__);                        \
    case 14: return FN<14>(__VA_ARGS__); case 15: return FN<15>(__VA_ARGS__);                        \
    case 16: return FN<16>(__VA_ARGS__);                                                             \
    default: return cudaErrorInvalidValue;                                                           \
  }

cudaError_t spread_reductions(const hb_nufft* p, Group q, cudaStream_t st) {
  HB_W_DISPATCH(spread_reductions_w, p, q, st)
}
cudaError_t interp(const hb_nufft* p, const InterpDest& dst, Group q, float csgn, cudaStream_t st) {
  HB_W_DISPATCH(interp_w, p, dst, q, csgn, st)
}

long long nmodes(const hb_nufft* p) { return (long long)p->g.N[0] * p->g.N[1] * p->g.N[2]; }
long long nfine(const hb_nufft* p) { return (long long)p->g.n[0] * p->g.n[1] * p->g.n[2]; }

// ---- fine-grid passes (nufft_pass_kernels.cuh); axis twiddles at tw + {0, n0, n0 + n1} ----
template <int L, bool PAD>
cudaError_t axis_pass_l(const hb_nufft* p, int axis, Group q, cudaStream_t st) {
  using C = TilePassCfg<L>;
  constexpr size_t smem = C::SMEM * sizeof(float2);
  cudaError_t e = hb::fftl::allow_smem<nufft_axis_pass_kernel<L, PAD>>(smem);
  if (e != cudaSuccess) return e;
  const NufftGeom& g = p->g;
  const long long side = nfine(p) << q.lgnb;
  if (axis == 0) {  // z: every (y, x) column of every side
    const long long ncols = (long long)g.n[1] * g.n[2] << q.lgnb;
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    return launch_chained(nufft_axis_pass_kernel<L, PAD>, dim3((unsigned)((ncols + 15) / 16), q.nz), C::THREADS, smem, st,
                          p->grid, ncols, (int)ncols, q.nz, q.nz, side, p->tw);
  }
  // y: the kept z planes; in 2-D every side is one plane
  const int ncols = g.n[2] << q.lgnb, planes = g.N[0] > 1 ? 1 : q.nz;
  for (int s = 0; s < q.nz; s += planes) {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    e = launch_chained(nufft_axis_pass_kernel<L, PAD>, dim3((ncols + 15) / 16, g.N[0] * planes), C::THREADS, smem, st,
                       p->grid + s * side, ncols, ncols, g.N[0] * planes, g.n[0] * planes, (long long)ncols * L,
                       p->tw + g.n[0]);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
// to_grid: modes -> grid (type 2), else grid -> modes (type 1); the grids from `side` on
template <int L, bool SIDES>
cudaError_t mode_pass_l(const hb_nufft* p, const NufftModeOp& op, Group q, int side, float sgn, bool to_grid, cudaStream_t st) {
  using C = TilePassCfg<L>;
  constexpr size_t smem = C::SMEM * sizeof(float2);
  const NufftGeom& g = p->g;
  const int nl = 16 >> q.lgnb;
  const dim3 grid((unsigned)((g.N[0] * g.N[1] + nl - 1) / nl), q.nz);
  float2* cells = p->grid + ((side * nfine(p)) << q.lgnb);
  const float2* tw = p->tw + g.n[0] + g.n[1];
  cudaError_t e;
  if (to_grid) {
    if ((e = hb::fftl::allow_smem<nufft_modes_to_grid_kernel<L, SIDES>>(smem)) != cudaSuccess) return e;
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    return launch_chained(nufft_modes_to_grid_kernel<L, SIDES>, grid, C::THREADS, smem, st, g, op, q.lgnb, q.nact, sgn, p->corr,
                          tw, cells);
  } else {
    if ((e = hb::fftl::allow_smem<nufft_grid_to_modes_kernel<L, SIDES>>(smem)) != cudaSuccess) return e;
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    return launch_chained(nufft_grid_to_modes_kernel<L, SIDES>, grid, C::THREADS, smem, st, g, op, q.lgnb, q.nact, sgn, p->corr,
                          tw, cells);
  }
}

#define HB_L_DISPATCH(n, CALL)                                                        \
  switch (n) {                                                                        \
    case 8: { constexpr int L = 8; return CALL; }     case 16: { constexpr int L = 16; return CALL; }   \
    case 32: { constexpr int L = 32; return CALL; }   case 64: { constexpr int L = 64; return CALL; }   \
    case 128: { constexpr int L = 128; return CALL; } case 256: { constexpr int L = 256; return CALL; } \
    case 512: { constexpr int L = 512; return CALL; } case 96: { constexpr int L = 96; return CALL; }   \
    case 160: { constexpr int L = 160; return CALL; } case 192: { constexpr int L = 192; return CALL; } \
    case 320: { constexpr int L = 320; return CALL; }                                 \
    default: return cudaErrorInvalidValue;                                            \
  }
cudaError_t axis_pass(const hb_nufft* p, int axis, bool pad, Group q, cudaStream_t st) {
  if (p->g.n[axis] == 1) return cudaSuccess;  // a degenerate axis of a 1-D or 2-D plan
  HB_L_DISPATCH(p->g.n[axis], (pad ? axis_pass_l<L, true>(p, axis, q, st) : axis_pass_l<L, false>(p, axis, q, st)))
}
cudaError_t mode_pass(const hb_nufft* p, const NufftModeOp& op, Group q, int side, float sgn, bool to_grid, cudaStream_t st) {
  HB_L_DISPATCH(p->g.n[2], (q.nz > 1 ? mode_pass_l<L, true>(p, op, q, side, sgn, to_grid, st)
                                    : mode_pass_l<L, false>(p, op, q, side, sgn, to_grid, st)))
}

// The passes transform forward; the other sign conjugates what enters and leaves the chain.
float conj_sign(int isign) { return isign > 0 ? -1.f : 1.f; }

// The whole grids = the spread values p->vals; the split tiles are zeroed
cudaError_t spread(const hb_nufft* p, Group q, cudaStream_t st) {
  if (p->nitems > 0) return p->g.dim == 3 ? spread_tiles<3>(p, q, st) : spread_tiles<2>(p, q, st);
  cudaError_t e = cudaMemsetAsync(p->grid, 0, ((size_t)nfine(p) << q.lgnb) * q.nz * sizeof(float2), st);
  return e != cudaSuccess ? e : spread_reductions(p, q, st);
}

// One group of transforms: p->vals (already conjugated for isign) -> grid, transformed along z and y
int type1_grid(const hb_nufft* p, Group q, cudaStream_t st) {
  HB_CUDA(spread(p, q, st));
  HB_CUDA(axis_pass(p, 0, false, q, st));
  HB_CUDA(axis_pass(p, 1, false, q, st));
  return HB_OK;
}
// One group of transforms: samples (src) -> modes (op, plain)
int type1_group(const hb_nufft* p, const SpreadSource& src, const NufftModeOp& op, Group q, int isign, cudaStream_t st) {
  HB_CUDA(gather_values(p, src, q, conj_sign(isign), st));
  if (int r = type1_grid(p, q, st)) return r;
  HB_CUDA(mode_pass(p, op, q, 0, conj_sign(isign), false, st));
  return HB_OK;
}

// One group of transforms: modes (op) -> samples (dst)
int type2_group(const hb_nufft* p, const NufftModeOp& op, const InterpDest& dst, Group q, int isign, cudaStream_t st) {
  const float sgn = conj_sign(isign);
  HB_CUDA(mode_pass(p, op, q, 0, sgn, true, st));
  HB_CUDA(axis_pass(p, 1, true, q, st));
  HB_CUDA(axis_pass(p, 0, true, q, st));
  HB_CUDA(interp(p, dst, q, sgn, st));
  return HB_OK;
}
InterpDest rows_dest(float2* c, long long c_ld) {
  InterpDest d{};
  d.c = c;
  d.c_ld = c_ld;
  return d;
}

NufftModeOp plain_modes(const float2* f, long long f_ld) {
  NufftModeOp op{};
  op.f = const_cast<float2*>(f);
  op.f_ld = f_ld;
  return op;
}
// Coil form of the mode side for coils [b0, b0 + n)
NufftModeOp coil_modes(const void* smaps, const int64_t* coils, int64_t b0, int n, long long nm) {
  NufftModeOp op{};
  for (int b = 0; b < n; ++b) op.maps.s[b] = (const float2*)smaps + coils[b0 + b] * nm;
  return op;
}
// Last step of the type 1 of coils [b0, b0 + q.nact) of ncoil (isign +1): grid lines -> their part of the
// coil sum, one grid after the other.  `out` is written with the last coils only, so that it may be one
// of the call's inputs (the normal operator in place): every group has read them by then.  The sum up to
// there is kept in the plan.
int coil_combine(const hb_nufft* p, const void* smaps, const int64_t* coils, int64_t b0, Group q, int64_t ncoil,
                 void* out, int accumulate, cudaStream_t st) {
  for (int side = 0; side < q.nz; ++side) {
    const int first = side << q.lgnb, n = q.nact - first < 1 << q.lgnb ? q.nact - first : 1 << q.lgnb;
    NufftModeOp op = coil_modes(smaps, coils, b0 + first, n, nmodes(p));
    op.add = b0 + first > 0 ? p->image : accumulate ? (const float2*)out : nullptr;
    op.out = b0 + first + n < ncoil ? p->image : (float2*)out;
    HB_CUDA(mode_pass(p, op, {n, q.lgnb, 1}, side, conj_sign(+1), false, st));
  }
  return HB_OK;
}

void free_plan(hb_nufft* p) {
  if (!p) return;
  cudaFree(p->mem);
  cudaFree(p->items_mem);
  delete p;
}

// hb_nufft_create; tiles = false leaves out the tile work lists (spread by reductions only).  With
// `external` the plan's arrays and the temporaries of the sort are taken from that arena, which
// outlives the plan, and nothing waits for the stream; a dry arena (base null) measures them and
// creates nothing.
int create_plan(hb_nufft** out, int64_t nz, int64_t ny, int64_t nx, const float* coords, int64_t nsamples, double tol,
                int maxbatch, int device, void* stream, bool tiles, Arena* external = nullptr) {
  if (!out) return fail(HB_ERR_INVALID, "hb_nufft_create: null output");
  *out = nullptr;
  const bool dry = external && !external->base;
  if ((!coords && !dry) || nsamples < 1 || nsamples > (int64_t)0x7fffffff)
    return fail(HB_ERR_INVALID, "hb_nufft_create: need coords and 1 <= nsamples < 2^31");
  if (!(tol > 0.0 && tol < 1.0)) return fail(HB_ERR_INVALID, "hb_nufft_create: tol must be in (0, 1)");
  if (maxbatch < 1 || maxbatch > kNufftMaxBatch)
    return fail(HB_ERR_INVALID, "hb_nufft_create: maxbatch must be in [1, " + std::to_string(kNufftMaxBatch) + "]");
  const int64_t Nv[3] = {nz, ny, nx};
  NufftGeom g{};
  g.w = width_for_tol(tol);
  g.beta = (float)(2.30 * g.w);
  g.K = nsamples;
  // nz = 1: a 2-D plan over (ny, nx); nz = ny = 1: a 1-D plan over nx (coords [dim][K])
  g.dim = nz != 1 ? 3 : (ny != 1 ? 2 : 1);
  for (int a = 0; a < 3; ++a) {
    if (a < 3 - g.dim) {  // degenerate leading axis
      g.N[a] = g.n[a] = g.nb[a] = g.bin[a] = 1;
      continue;
    }
    int E = 0, S = 0;
    const int64_t n = 2 * Nv[a];
    if (Nv[a] < 1 || n > 512 || !team_length((int)n, &E, &S) || n < 2 * g.w)
      return fail(HB_ERR_UNSUPPORTED, "hb_nufft_create: mode count " + std::to_string(Nv[a]) +
                                          " unsupported (2N must be one of 8,16,32,64,128,256,512,96,160,192,320 "
                                          "and >= 2w)");
    g.N[a] = (int)Nv[a];
    g.n[a] = (int)n;
    g.bin[a] = g.dim == 3 && a < 2 && tiles ? 4 : 8;  // every fine-grid length is a multiple of 8
    g.nb[a] = g.n[a] / g.bin[a];
  }
  // A tile's candidates are counted in 32 bits, and on a grid smaller than its neighbourhood it meets a bin
  // once per period.
  if (tiles && g.dim > 1) {
    long long most = nsamples;
    for (int a = 3 - g.dim; a < 3; ++a) {
      const int T = g.dim == 3 ? (a < 2 ? SpreadTile<3>::T0 : SpreadTile<3>::T2) : a == 1 ? SpreadTile<2>::T1 : SpreadTile<2>::T2;
      const int h = (g.w + 1) / 2, met = ((T < g.n[a] ? T : g.n[a]) - 1 + h) / g.bin[a] + (h + g.bin[a] - 1) / g.bin[a] + 1;
      most *= (met + g.nb[a] - 1) / g.nb[a];
    }
    if (most > 0x7fffffffLL - 4096)
      return fail(HB_ERR_UNSUPPORTED, "hb_nufft_create: too many samples for a grid of " + std::to_string(g.n[0]) + " x " +
                                          std::to_string(g.n[1]) + " x " + std::to_string(g.n[2]) + " cells");
  }
  DeviceGuard dg(device);
  if (!dg.ok) return fail(HB_ERR_CUDA, "hb_nufft_create: cannot select device");
  cudaStream_t st = (cudaStream_t)stream;
  hb_nufft* p = new hb_nufft();
  p->device = device;
  p->g = g;
  p->group = maxbatch > 4 ? 8 : maxbatch > 2 ? 4 : maxbatch;
  const int nbins = g.nb[0] * g.nb[1] * g.nb[2];
  const long long vol = (long long)g.n[0] * g.n[1] * g.n[2];
  p->sides = small_plan(g) ? (maxbatch + kNufftGroup - 1) / kNufftGroup : 1;
  const int ntiles = !tiles       ? 0
                     : g.dim == 3 ? (g.n[0] / SpreadTile<3>::T0) * (g.n[1] / SpreadTile<3>::T1) * (g.n[2] / SpreadTile<3>::T2)
                     : g.dim == 2 ? ((g.n[1] + SpreadTile<2>::T1 - 1) / SpreadTile<2>::T1) * (g.n[2] / SpreadTile<2>::T2)
                                  : 0;
  void* tmp = nullptr;
  auto bail = [&](cudaError_t e, const char* what) {
    cudaFree(tmp);
    free_plan(p);
    return fail(HB_ERR_CUDA, std::string("hb_nufft_create: ") + what + ": " + cudaGetErrorString(e));
  };
  // one allocation for the plan's arrays, one for the temporaries of the sort (a cudaMalloc
  // and its cudaFree cost as much as the kernels between them)
  auto carve = [&](Arena& ar) {
    p->pts = ar.take<float4>(nsamples);
    p->start = ar.take<int>(nbins + 1);
    p->corr = ar.take<float>(g.N[0] + g.N[1] + g.N[2]);
    p->tw = ar.take<float2>(g.n[0] + g.n[1] + g.n[2]);
    p->grid = ar.take<float2>((size_t)p->sides * p->group * vol);
    p->vals = ar.take<float2>((size_t)p->sides * p->group * nsamples);
    if (!external) p->image = ar.take<float2>((size_t)g.N[0] * g.N[1] * g.N[2]);
  };
  int2* bin_rank;
  int *counts, *sums, *candidates;
  SpreadCounts* nwork;
  auto carve_tmp = [&](Arena& ar) {
    bin_rank = ar.take<int2>(nsamples);
    counts = ar.take<int>(nbins);
    sums = ar.take<int>((nbins + kScanBlock - 1) / kScanBlock);
    candidates = ar.take<int>(ntiles);
    nwork = ar.take<SpreadCounts>(1);
  };
  cudaError_t e;
  if (external) {
    carve(*external);
    carve_tmp(*external);
    if (dry) {
      delete p;
      return HB_OK;
    }
  } else {
    Arena size(nullptr), size_tmp(nullptr);
    carve(size);
    carve_tmp(size_tmp);
    if ((e = cudaMalloc(&p->mem, size.off)) != cudaSuccess) return bail(e, "plan arrays and fine grid");
    if ((e = cudaMalloc(&tmp, size_tmp.off)) != cudaSuccess) return bail(e, "sort temporaries");
    Arena ar(p->mem), ar_tmp(tmp);
    carve(ar);
    carve_tmp(ar_tmp);
  }

  // counting sort of the samples by bin
  const unsigned blocks = (unsigned)((nsamples + 255) / 256);
  if ((e = cudaMemsetAsync(counts, 0, nbins * sizeof(int), st)) != cudaSuccess) return bail(e, "memset");
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_bin_count_kernel<<<blocks, 256, 0, st>>>(g, coords, bin_rank, counts);
  }
  const unsigned sb = (unsigned)((nbins + kScanBlock - 1) / kScanBlock);
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_scan_block_kernel<<<sb, 1024, 0, st>>>(counts, p->start, sums, nbins);
  }
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_scan_sums_kernel<<<1, 1024, 0, st>>>(sums, (int)sb);
  }
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_scan_add_kernel<<<sb, 1024, 0, st>>>(counts, p->start, sums, nbins);
  }
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_bin_scatter_kernel<<<blocks, 256, 0, st>>>(g, coords, bin_rank, p->start, p->pts);
  }
  // Spreading: cut the tiles' candidates into pieces of at most `cap`, about 32 pieces per SM
  // sub-partition over the whole plan (a sample is a candidate of up to 27 tiles of 4 x 4 x 8 or 6
  // of 16 x 8).  Measured, 8 transforms: 64^3 modes with 524 k radial samples 632 / 555 / 542 /
  // 551 us at cap 128 / 256 / 512 / 1024 (a piece re-adds its tile; one of 1024 is the tail), 201 x
  // 256 samples on 128^2 modes 37 / 28 / 29 / 40 us at 32 / 64 / 128 / 256.
  const long long per_sample = g.dim == 3 ? 27 : 6;
  const long long want = nsamples * per_sample / (148 * 4 * 32);
  const int cap = (int)(want < 64 ? 64 : want > 512 ? 512 : want);
  const unsigned tb = (unsigned)((ntiles + 255) / 256);
  if (ntiles > 0) {
    if ((e = cudaMemsetAsync(nwork, 0, sizeof(SpreadCounts), st)) != cudaSuccess) return bail(e, "memset");
    {
      LaunchScope ls(HB_KERNEL_NUFFT, st);
      if (g.dim == 3) nufft_tile_count_kernel<3><<<tb, 256, 0, st>>>(g, p->start, ntiles, cap, candidates, nwork);
      else nufft_tile_count_kernel<2><<<tb, 256, 0, st>>>(g, p->start, ntiles, cap, candidates, nwork);
    }
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return bail(e, "binning");

  // tables: 1/phi_hat per axis and the team twiddles of each fine-grid length
  {
    LaunchScope ls(HB_KERNEL_NUFFT, st);
    nufft_corr_kernel<<<(g.N[0] + g.N[1] + g.N[2] + 255) / 256, 256, 0, st>>>(g, 2.30 * g.w, gauss_legendre(), p->corr);
  }
  if ((e = team_tables_device(g.n, p->tw, st, HB_KERNEL_NUFFT)) != cudaSuccess) return bail(e, "tables");
  if (ntiles > 0) {
    if ((e = cudaMemcpyAsync(&p->nitems, &nwork->items, sizeof(int), cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
      return bail(e, "binning");
    // at most every piece beyond the first of its tile belongs to a split tile
    const int most_split = p->nitems - ntiles;
    if ((e = cudaMalloc(&p->items_mem, p->nitems * sizeof(SpreadItem) + most_split * sizeof(int) + 16)) != cudaSuccess)
      return bail(e, "spread items");
    p->items = (SpreadItem*)p->items_mem;
    p->split_tiles = (int*)(p->items + p->nitems);
    {
      LaunchScope ls(HB_KERNEL_NUFFT, st);
      if (g.dim == 3)
        nufft_tile_items_kernel<3><<<tb, 256, 0, st>>>(g, ntiles, cap, candidates, p->items, p->split_tiles, nwork);
      else
        nufft_tile_items_kernel<2><<<tb, 256, 0, st>>>(g, ntiles, cap, candidates, p->items, p->split_tiles, nwork);
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return bail(e, "spread items");
    if ((e = cudaMemcpyAsync(&p->nsplit, &nwork->split_tiles, sizeof(int), cudaMemcpyDeviceToHost, st)) != cudaSuccess)
      return bail(e, "spread items");
  }
  if (!external && (e = cudaStreamSynchronize(st)) != cudaSuccess) return bail(e, "binning");
  cudaFree(tmp);
  *out = p;
  return HB_OK;
}

}  // namespace

namespace hb {

// The NUFFT plan of the point-spread function on an M grid, in `ar` (measured only when ar is dry)
static int psf_plan(hb_nufft** np, const int* M, const float* coords, int64_t nsamples, double tol, int device,
                    cudaStream_t st, Arena& ar) {
  // type 1 over the grid's modes: sum_j exp(+i c_j . d), d in [-M/2, M/2)
  return create_plan(np, M[0], M[1], M[2], coords, nsamples, tol, 1, device, st, false, &ar);
}

static int psf_in(const int* M, const float* coords, int64_t nsamples, double tol, const float* weights, int device,
                  float2* out, cudaStream_t st, Arena& ar) {
  const long long vol = (long long)M[0] * M[1] * M[2];
  hb_nufft* np = nullptr;
  if (int r = psf_plan(&np, M, coords, nsamples, tol, device, st, ar)) return r;
  NufftModeOp op = plain_modes(out, vol);
  op.circulant = (float)(1.0 / (double)vol);
  const int rc = type1_group(np, {nullptr, 0, weights}, op, {1, 0, 1}, +1, st);
  free_plan(np);  // host state only: its arrays are the arena's
  return rc;
}

int nufft_psf_circulant(const int* M, const float* coords, int64_t nsamples, double tol, const float* weights,
                        int device, float2* out, cudaStream_t st) {
  Arena size(nullptr);
  hb_nufft* none = nullptr;
  if (int r = psf_plan(&none, M, nullptr, nsamples, tol, device, st, size)) return r;
  void* mem = nullptr;
  HB_CUDA(cudaMalloc(&mem, size.off));
  Arena ar(mem);
  int rc = psf_in(M, coords, nsamples, tol, weights, device, out, st, ar);
  const cudaError_t e = cudaStreamSynchronize(st);
  if (rc == HB_OK && e != cudaSuccess) rc = fail(HB_ERR_CUDA, std::string("psf: ") + cudaGetErrorString(e));
  cudaFree(mem);
  return rc;
}

}  // namespace hb

extern "C" {

int hb_nufft_create(hb_nufft** out, int64_t nz, int64_t ny, int64_t nx, const float* coords, int64_t nsamples,
                    double tol, int maxbatch, int device, void* stream) {
  return create_plan(out, nz, ny, nx, coords, nsamples, tol, maxbatch, device, stream, true);
}
int hb_nufft_destroy(hb_nufft* plan) {
  if (!plan) return HB_OK;
  DeviceGuard dg(plan->device);
  free_plan(plan);
  return HB_OK;
}

int hb_nufft_width(const hb_nufft* plan) { return plan ? plan->g.w : -1; }

int hb_nufft_kernel_values(const hb_nufft* plan, const float* z, const float* s, float* phi, float* root, int64_t n,
                           void* stream) {
  if (!plan || !z || !s || !phi || !root || n < 1 || n > (int64_t)0x7fffffff)
    return fail(HB_ERR_INVALID, "hb_nufft_kernel_values: null argument or n out of range");
  DeviceGuard dg(plan->device);
  LaunchScope ls(HB_KERNEL_NUFFT, (cudaStream_t)stream);
  nufft_kernel_values_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(plan->g.w, plan->g.beta, z, s, phi,
                                                                                       root, n);
  HB_CUDA(cudaGetLastError());
  return HB_OK;
}

int hb_nufft_type1(const hb_nufft* plan, const void* c, void* f, int64_t ntransf, int isign, void* stream) {
  if (!plan || !c || !f || ntransf < 0 || (isign != 1 && isign != -1))
    return fail(HB_ERR_INVALID, "hb_nufft_type1: null argument, negative ntransf or isign not +-1");
  DeviceGuard dg(plan->device);
  const long long K = plan->g.K, nm = nmodes(plan);
  for (int64_t t0 = 0; t0 < ntransf;) {
    const Group q = next_group(plan, ntransf - t0);
    if (int r = type1_group(plan, {(const float2*)c + t0 * K, K, nullptr}, plain_modes((const float2*)f + t0 * nm, nm), q,
                            isign, (cudaStream_t)stream))
      return r;
    t0 += q.nact;
  }
  return HB_OK;
}

int hb_nufft_type2(const hb_nufft* plan, const void* f, void* c, int64_t ntransf, int isign, void* stream) {
  if (!plan || !c || !f || ntransf < 0 || (isign != 1 && isign != -1))
    return fail(HB_ERR_INVALID, "hb_nufft_type2: null argument, negative ntransf or isign not +-1");
  DeviceGuard dg(plan->device);
  const long long K = plan->g.K, nm = nmodes(plan);
  for (int64_t t0 = 0; t0 < ntransf;) {
    const Group q = next_group(plan, ntransf - t0);
    if (int r = type2_group(plan, plain_modes((const float2*)f + t0 * nm, nm), rows_dest((float2*)c + t0 * K, K), q,
                            isign, (cudaStream_t)stream))
      return r;
    t0 += q.nact;
  }
  return HB_OK;
}

int hb_sense_adjoint_nufft(const hb_nufft* plan, const void* kdata, const void* smaps, const int64_t* coils,
                           int64_t ncoil, const float* weights, void* out, int accumulate, void* stream) {
  if (!plan || !kdata || !smaps || !out || ncoil < 0 || (ncoil > 0 && !coils))
    return fail(HB_ERR_INVALID, "hb_sense_adjoint_nufft: null argument or negative ncoil");
  for (int64_t b = 0; b < ncoil; ++b)
    if (coils[b] < 0) return fail(HB_ERR_INVALID, "hb_sense_adjoint_nufft: negative coil index");
  DeviceGuard dg(plan->device);
  cudaStream_t st = (cudaStream_t)stream;
  const long long K = plan->g.K, nm = nmodes(plan);
  if (ncoil == 0 && !accumulate) HB_CUDA(cudaMemsetAsync(out, 0, nm * sizeof(float2), st));
  for (int64_t b0 = 0; b0 < ncoil;) {
    const Group q = next_group(plan, ncoil - b0);
    HB_CUDA(gather_values(plan, {(const float2*)kdata + b0 * K, K, weights}, q, conj_sign(+1), st));
    if (int r = type1_grid(plan, q, st)) return r;
    if (int r = coil_combine(plan, smaps, coils, b0, q, ncoil, out, accumulate, st)) return r;
    b0 += q.nact;
  }
  return HB_OK;
}

int hb_sense_forward_nufft(const hb_nufft* plan, const void* x, const void* smaps, const int64_t* coils,
                           int64_t ncoil, void* kdata, void* stream) {
  if (!plan || !x || !smaps || !kdata || ncoil < 0 || (ncoil > 0 && !coils))
    return fail(HB_ERR_INVALID, "hb_sense_forward_nufft: null argument or negative ncoil");
  for (int64_t b = 0; b < ncoil; ++b)
    if (coils[b] < 0) return fail(HB_ERR_INVALID, "hb_sense_forward_nufft: negative coil index");
  DeviceGuard dg(plan->device);
  cudaStream_t st = (cudaStream_t)stream;
  const long long K = plan->g.K, nm = nmodes(plan);
  for (int64_t b0 = 0; b0 < ncoil;) {
    const Group q = next_group(plan, ncoil - b0);
    const int nb = q.nact;
    NufftModeOp op = coil_modes(smaps, coils, b0, nb, nm);
    op.x = (const float2*)x;
    if (int r = type2_group(plan, op, rows_dest((float2*)kdata + b0 * K, K), q, -1, st)) return r;
    b0 += nb;
  }
  return HB_OK;
}

int hb_sense_normal_nufft(const hb_nufft* plan, const void* x, const void* smaps, const int64_t* coils, int64_t ncoil,
                          const void* kdata, const float* weights, void* out, int accumulate, void* stream) {
  if (!plan || !x || !smaps || !out || ncoil < 0 || (ncoil > 0 && !coils))
    return fail(HB_ERR_INVALID, "hb_sense_normal_nufft: null argument or negative ncoil");
  for (int64_t b = 0; b < ncoil; ++b)
    if (coils[b] < 0) return fail(HB_ERR_INVALID, "hb_sense_normal_nufft: negative coil index");
  DeviceGuard dg(plan->device);
  cudaStream_t st = (cudaStream_t)stream;
  const long long K = plan->g.K, nm = nmodes(plan);
  if (ncoil == 0 && !accumulate) HB_CUDA(cudaMemsetAsync(out, 0, nm * sizeof(float2), st));
  for (int64_t b0 = 0; b0 < ncoil;) {
    const Group q = next_group(plan, ncoil - b0);
    const int nb = q.nact;
    InterpDest mid{};
    for (int b = 0; b < nb; ++b) mid.y[b] = kdata ? (const float2*)kdata + coils[b0 + b] * K : nullptr;
    mid.w = weights;
    mid.vals = plan->vals;
    mid.vsgn = conj_sign(+1);
    NufftModeOp op = coil_modes(smaps, coils, b0, nb, nm);
    op.x = (const float2*)x;
    if (int r = type2_group(plan, op, mid, q, -1, st)) return r;
    HB_CUDA(zero_tiles(plan, q, st));
    if (int r = type1_grid(plan, q, st)) return r;
    if (int r = coil_combine(plan, smaps, coils, b0, q, ncoil, out, accumulate, st)) return r;
    b0 += nb;
  }
  return HB_OK;
}

// Scratch of a diagonal build: twiddles, T (unless the caller's array takes it) and the NUFFT plan.
// Returns an error code; with a dry arena it only measures.
static int diag_scratch(const hb_plan* plan, int64_t nsamples, double tol, bool own_T, cudaStream_t st, Arena& ar,
                        float2** tw, float2** T) {
  int N[3], dev = 0;
  plan_geometry(plan, N, &dev);
  const int M[3] = {2 * N[0], 2 * N[1], 2 * N[2]};
  *tw = ar.take<float2>(M[0] + M[1] + M[2]);
  if (own_T) *T = ar.take<float2>((size_t)M[0] * M[1] * M[2]);
  if (ar.base) return HB_OK;
  hb_nufft* none = nullptr;
  return psf_plan(&none, M, nullptr, nsamples, tol, dev, st, ar);
}

size_t hb_diag_build_nufft_workspace_bytes(const hb_plan* plan, int64_t nsamples, double tol) {
  if (!plan || nsamples < 1) return 0;
  Arena size(nullptr);
  float2 *tw = nullptr, *T = nullptr;
  return diag_scratch(plan, nsamples, tol, true, nullptr, size, &tw, &T) == HB_OK ? size.off + 256 : 0;
}

int hb_diag_build_nufft_ws(const hb_plan* plan, const float* coords, int64_t nsamples, double tol, const float* weights,
                           float* packed, void* T_complex, void* ws, size_t ws_bytes, void* stream) {
  if (!plan || !coords || nsamples < 1) return fail(HB_ERR_INVALID, "hb_diag_build_nufft: null plan or no samples");
  if (!packed && !T_complex) return fail(HB_ERR_INVALID, "hb_diag_build_nufft: no output requested");
  int N[3], dev = 0;
  plan_geometry(plan, N, &dev);
  DeviceGuard dg(dev);
  cudaStream_t st = (cudaStream_t)stream;
  const int M[3] = {2 * N[0], 2 * N[1], 2 * N[2]};
  float2 *tw = nullptr, *T = (float2*)T_complex;  // T goes straight to the caller's array when that is wanted
  Arena size(nullptr);
  if (int r = diag_scratch(plan, nsamples, tol, !T_complex, st, size, &tw, &T)) return r;
  if (!ws || ws_bytes < size.off) return fail(HB_ERR_WORKSPACE, "hb_diag_build_nufft: workspace too small");
  if (((uintptr_t)ws & 255u) != 0) return fail(HB_ERR_INVALID, "hb_diag_build_nufft: workspace not 256-byte aligned");
  Arena ar(ws);
  T = (float2*)T_complex;
  if (int r = diag_scratch(plan, nsamples, tol, !T_complex, st, ar, &tw, &T)) return r;
  HB_CUDA(team_tables_device(M, tw, st, HB_KERNEL_DIAG));
  // PSF in circulant layout on the 2x grid, then T = FFT(PSF)
  if (int r = psf_in(M, coords, nsamples, tol, weights, dev, T, st, ar)) return r;
  HB_CUDA(fft3_grid<-1>(M[0], M[1], M[2], tw, T, 1, st));
  return packed ? hb_diag_pack(plan, T, packed, stream) : HB_OK;
}

int hb_diag_build_nufft(const hb_plan* plan, const float* coords, int64_t nsamples, double tol, const float* weights,
                        float* packed, void* T_complex, void* stream) {
  if (!plan || !coords || nsamples < 1) return fail(HB_ERR_INVALID, "hb_diag_build_nufft: null plan or no samples");
  if (!packed && !T_complex) return fail(HB_ERR_INVALID, "hb_diag_build_nufft: no output requested");
  int N[3], dev = 0;
  plan_geometry(plan, N, &dev);
  DeviceGuard dg(dev);
  cudaStream_t st = (cudaStream_t)stream;
  float2 *tw = nullptr, *T = nullptr;
  Arena size(nullptr);
  if (int r = diag_scratch(plan, nsamples, tol, !T_complex, st, size, &tw, &T)) return r;
  void* mem = nullptr;
  HB_CUDA(cudaMalloc(&mem, size.off));
  int rc = hb_diag_build_nufft_ws(plan, coords, nsamples, tol, weights, packed, T_complex, mem, size.off, stream);
  const cudaError_t e = cudaStreamSynchronize(st);
  if (rc == HB_OK && e != cudaSuccess)
    rc = fail(HB_ERR_CUDA, std::string("hb_diag_build_nufft: ") + cudaGetErrorString(e));
  cudaFree(mem);
  return rc;
}

}  // extern "C"
