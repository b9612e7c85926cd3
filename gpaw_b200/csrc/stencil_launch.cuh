// stencil_launch.cuh -- host-side tile selection and template dispatch for the
// stencil kernels.  Included by one translation unit per element type so the
// instantiations compile in parallel.
#pragma once

#include <algorithm>
#include <type_traits>

#include "internal.h"
#include "march_split.h"
#include "stencil.cuh"
#include "stencil_dirs.cuh"
#include "stencil_flex.cuh"
#include "stencil_line.cuh"
#include "stencil_pair.cuh"
#include "stencil_split.cuh"
#include "stencil_tma.cuh"
#include "stencil_tmasplit.cuh"

namespace gfd {

// Tile shapes (BZ x TY threads, VY rows per thread; TILE_* in internal.h).
// Wide tiles for grids whose fastest axis fills a warp, narrow ones for the
// small coarse multigrid levels.

inline int pick_tile(const gfd_operator* op) {
  if (op->R > 2) return TILE_WIDE;
  if (op->n[2] <= 8) return TILE_NARROW;
  if (op->n[2] <= 16) return TILE_MID;
  return TILE_WIDE;
}

struct TileDims {
  int BZ, BY, NT;
};
inline TileDims tile_dims(int tile) {
  switch (tile) {
    case TILE_NARROW: return {8, 8, 64};
    case TILE_MID: return {16, 16, 128};
    case TILE_SHORT: return {32, 8, 128};
    case TILE_SPLIT: return {32, 4 * GFD_SPLIT_VY, 128};
    case TILE_48: return {kTile48Z, 8, 4 * kTile48Z};
    case TILE_48R: return {kTile48Z, 16, 4 * kTile48Z};
    default: return {32, 16, 128};
  }
}

constexpr int kStages = 4;

// Grids up to direct_max_points() (all bands) use the one-thread-per-point
// kernel: the marching kernel's plane pipeline only pays off on larger grids.
inline bool use_direct(const gfd_operator* op, int64_t nin) {
  return (long long)op->n[0] * op->n[1] * op->n[2] * nin <= direct_max_points();
}
inline int direct_blocks(long long total) {
  long long b = (total + 255) / 256;
  long long cap = 8LL * num_sms();
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}

// Raise a kernel's dynamic shared-memory limit when it needs more than 48 KB.
template <class F>
int raise_smem_limit(F* kern, size_t bytes, const char* what) {
  if (bytes <= 48 * 1024) return GFD_OK;
  return check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)bytes),
                    what);
}

struct LaunchGeom {
  dim3 grid;
  int nxc, x_chunk;
  int64_t bands_per_launch;
};

// The target in CTAs per SM that a launch is split by: a plan's (cps), the
// environment's, four for kernels whose CTAs per SM are not known (resident 0),
// else none, the rounds are counted.
inline int split_target(int cps, int resident) {
  if (cps > 0) return cps;
  return resident > 0 && !march_ctas_given() ? 0 : march_ctas_per_sm();
}

// resident: CTAs per SM of the kernel where known; cps: a launch plan's target.
inline LaunchGeom star_geom(const gfd_operator* op, int tile, int64_t nin, int R, int cps = 0,
                            int resident = 0) {
  TileDims td = tile_dims(tile);
  LaunchGeom g;
  int gx = (op->n[2] + td.BZ - 1) / td.BZ;
  int gy = (op->n[1] + td.BY - 1) / td.BY;
  int64_t tiles = (int64_t)gx * gy * std::max<int64_t>(nin, 1);
  const int nxc =
      march_chunks(op->n[0], R, tiles, resident, num_sms(), split_target(cps, resident));
  g.x_chunk = (op->n[0] + nxc - 1) / nxc;
  g.nxc = (op->n[0] + g.x_chunk - 1) / g.x_chunk;
  g.bands_per_launch = std::max<int64_t>(1, 65535 / g.nxc);
  g.grid = dim3(gx, gy, 1);
  return g;
}

// CTAs per SM of star_kernel's real tiles up to radius 3, from their registers
// (bytes: size of a value); 0 for the others.  A residual's figure depends on the
// radius alone: partials_count() does not know the type.
inline int real_resident(const gfd_operator* op, int tile, int mode, int bytes) {
  if (op->R > 3) return 0;
  if (tile == TILE_48R) return 3;
  if (tile != TILE_WIDE) return 0;
  if (mode == OP_RESIDUAL) return op->R == 2 ? 3 : 4;
  if (bytes == 4) return op->R == 3 ? 4 : 5;
  if (op->R == 1) return mode == OP_APPLY ? 5 : 4;
  return op->R == 2 && mode == OP_APPLY ? 4 : 3;
}

// The real 48-column tile where its launch takes less time than the wide one's:
// a CTA of its full SM steps once in 1.18 us (float32 0.80) against 0.76 (0.68),
// fitted as in march_split.h.
inline bool tile48r_pays(const gfd_operator* op, int mode, int bytes, int64_t nin) {
  auto steps = [&](int tile) {
    const TileDims td = tile_dims(tile);
    const int64_t tiles =
        (int64_t)((op->n[1] + td.BY - 1) / td.BY) * ((op->n[2] + td.BZ - 1) / td.BZ) * nin;
    return march_split(op->n[0], op->R, tiles, real_resident(op, tile, mode, bytes), num_sms())
        .steps;
  };
  return steps(TILE_48R) * (bytes == 4 ? 0.80 : 1.18) < steps(TILE_WIDE) * (bytes == 4 ? 0.68 : 0.76);
}

template <class S>
void fill_phases(Phases<S>& P, const double* ph) {
  for (int c = 0; c < 3; c++)
    for (int d = 0; d < 2; d++) {
      P.ph[c][d].re = ph ? S(ph[4 * c + 2 * d]) : S(1);
      P.ph[c][d].im = ph ? S(ph[4 * c + 2 * d + 1]) : S(0);
    }
}

template <class V, int R, int BZ, int TY, int VY, int MODE, bool LOW = false, int S = kStages>
int star_go(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
            const StarParams<typename vt<V>::S>& base, const LaunchGeom& g, double* partials,
            cudaStream_t s) {
  constexpr size_t smem = star_smem_bytes<BZ, TY, VY, R, S, V, MODE>();
  auto kern = star_kernel<V, R, BZ, TY, VY, S, MODE, LOW>;
  int st = raise_smem_limit(kern, smem, "cudaFuncSetAttribute(star_kernel)");
  if (st) return st;
  StarParams<typename vt<V>::S> p = base;
  const long long band = (long long)op->n[0] * op->n[1] * op->n[2];
  for (int64_t b0 = 0; b0 < nin; b0 += g.bands_per_launch) {
    int64_t nb = std::min<int64_t>(g.bands_per_launch, nin - b0);
    dim3 grid(g.grid.x, g.grid.y, (unsigned)(nb * g.nxc));
    p.partials = partials ? partials + b0 * g.nxc * g.grid.x * g.grid.y : nullptr;
    launch_k(kern, grid, BZ * TY, smem, s, in + b0 * band, out + b0 * band,
                                     rho ? rho + b0 * band : nullptr, p);
  }
  return check_launch("star_kernel");
}

// Wide tile: 32 columns x 16 rows; 4 rows per thread for 8-byte and
// smaller values, 2 rows per thread where 4 would exceed the register file
// (16-byte values or radius > 3).
// Complex Jacobi / residual sweeps (the band preconditioner) are built for
// radii up to 3 only, which keeps the number of kernels in check.
constexpr int kMaxComplexRelaxR = 3;

// The short tile exists for complex128 apply (and apply with a potential)
// up to radius 4 (beyond, its 2R + 1 partial sums per row do not fit the
// registers of three CTAs per SM): the built-in choice at radius 4 where the
// 48-column tile below does not apply, and up to radius 3 where c128_tile()
// prices it lowest.  On the 512-band 96^3 Laplace (one box) it measured 3730
// GB/s at four CTAs of 128 threads per SM, against 3120 for the 32 x 16 tile,
// 3100 for the lane-pair kernel and 3270 for its TMA-staged form; three CTAs
// per SM with up to 170 registers took it to 3934.
constexpr int kMaxShortR = 4;
template <class V, int R, int MODE>
constexpr bool has_short_tile() {
  return sizeof(V) >= 16 && (MODE == MODE_APPLY || MODE == MODE_POTENTIAL) && R <= kMaxShortR;
}
// The 48-column tile: complex bands (complex128 and complex64), the same
// launches, where axis 2 is a multiple of 48: complex64's built-in choice, and
// complex128's as for the short tile.
template <class V, int R, int MODE>
constexpr bool has_tile48() {
  return vt<V>::NC == 2 && (MODE == MODE_APPLY || MODE == MODE_POTENTIAL) && R <= kMaxShortR;
}
// 48 x 4 threads with 2 rows each, two CTAs per SM.  On the 512-band 96^3
// Laplace the 48-column tile measured
// 4010-4099 GB/s against 3730-3826 for the short tile at 4 CTAs per SM
// (3934 at 3)
// (apply with a potential: 3610-3750 against 3260-3380).  A 96-column tile
// measured slower at every thread shape tried (2110-3570 GB/s): one CTA per
// SM, or registers short of its 2R + 1 partial sums per row.

// The wide tile of 8-byte values in the form of 2R sums and 128 registers, four
// CTAs per SM, where the form of 2R + 1 sums leaves room for two or three:
// complex64 from radius 2 (radius 3: 0.65 to 0.9 of its time in 110 launches of
// more than two CTAs per SM, 1.0 to 1.1 in 29 smaller ones, which fit the SMs
// in either form and keep the 2R + 1 sums), and the float64 residual of radius 3
// (176 registers).  The float64 apply, apply with a potential and Jacobi sweep
// keep the 2R + 1 sums, three CTAs per SM at radius 3: per CTA and plane both
// forms take the same time on a full chip (0.25 us), and on grids that do not
// fill it the form of 2R sums took 9% longer (23 launches).
template <class V, int R, int MODE>
constexpr bool wide_low() {
  return sizeof(V) == 8 && ((vt<V>::NC == 2 && (R == 2 || R == 3)) ||
                            (vt<V>::NC == 1 && R == 3 && MODE == MODE_RESIDUAL));
}
template <class V, int R, int MODE>
constexpr bool wide_both() {
  return wide_low<V, R, MODE>() && vt<V>::NC == 2 && R == 3;
}

template <class V, int R, int MODE>
int star_wide(const gfd_operator* op, int tile, const V* in, V* out, const V* rho, int64_t nin,
              const StarParams<typename vt<V>::S>& p, const LaunchGeom& g, double* partials,
              cudaStream_t s) {
  if constexpr (has_short_tile<V, R, MODE>()) {
    if (tile == TILE_SHORT)
      return star_go<V, R, 32, 4, 2, MODE>(op, in, out, rho, nin, p, g, partials, s);
  }
  if constexpr (has_tile48<V, R, MODE>()) {
    if (tile == TILE_48)
      return star_go<V, R, kTile48Z, 4, 2, MODE>(op, in, out, rho, nin, p, g, partials, s);
  }
  if constexpr (vt<V>::NC == 1 && R == 3 && MODE != MODE_RESIDUAL) {
    if (tile == TILE_48R)
      return star_go<V, R, kTile48Z, 4, 4, MODE, true>(op, in, out, rho, nin, p, g, partials, s);
  }
  if constexpr (sizeof(V) >= 16 || R > 3) {
    return star_go<V, R, 32, 8, 2, MODE>(op, in, out, rho, nin, p, g, partials, s);
  } else {
    if constexpr (wide_low<V, R, MODE>()) {
      const int64_t ctas = (int64_t)g.grid.x * g.grid.y * g.nxc * nin;
      if (!wide_both<V, R, MODE>() || ctas > 2 * num_sms())
        return star_go<V, R, 32, 4, 4, MODE, true>(op, in, out, rho, nin, p, g, partials, s);
    }
    if constexpr (!wide_low<V, R, MODE>() || wide_both<V, R, MODE>())
      return star_go<V, R, 32, 4, 4, MODE>(op, in, out, rho, nin, p, g, partials, s);
  }
  return set_error(GFD_EUNSUPPORTED, "star stencil form");  // not reached
}

template <class V, int MODE>
int star_dispatch(const gfd_operator* op, int tile, const V* in, V* out, const V* rho, int64_t nin,
                  const StarParams<typename vt<V>::S>& p, const LaunchGeom& g, double* partials,
                  cudaStream_t s) {
#define GFD_STAR_SMALL(RR)                                                                   \
  case RR:                                                                                   \
    if (tile == TILE_NARROW)                                                                 \
      return star_go<V, RR, 8, 8, 1, MODE>(op, in, out, rho, nin, p, g, partials, s);        \
    if (tile == TILE_MID)                                                                    \
      return star_go<V, RR, 16, 8, 2, MODE>(op, in, out, rho, nin, p, g, partials, s);       \
    return star_wide<V, RR, MODE>(op, tile, in, out, rho, nin, p, g, partials, s);
#define GFD_STAR_WIDE(RR)                                                                    \
  case RR:                                                                                   \
    if constexpr (RR > kMaxComplexRelaxR && vt<V>::NC == 2 && MODE != MODE_APPLY &&          \
                  MODE != MODE_POTENTIAL)                                                    \
      return set_error(GFD_EUNSUPPORTED, "complex Jacobi/residual sweeps need radius <= 3"); \
    else                                                                                     \
      return star_wide<V, RR, MODE>(op, tile, in, out, rho, nin, p, g, partials, s);
  switch (op->R) {
    GFD_STAR_SMALL(1)
    GFD_STAR_SMALL(2)
    GFD_STAR_WIDE(3)
    GFD_STAR_WIDE(4)
    GFD_STAR_WIDE(5)
    GFD_STAR_WIDE(6)
  }
#undef GFD_STAR_SMALL
#undef GFD_STAR_WIDE
  return set_error(GFD_EUNSUPPORTED, "star stencil radius out of range");
}

// ---------------------------------------------------------------------------
// Complex bands with the real and imaginary parts on lane pairs
// (stencil_split.cuh): 32 x 16 tile, 4 rows x 2 columns per lane, four
// pipeline stages (three with a staged source term), three CTAs per SM.
// ---------------------------------------------------------------------------
constexpr int kSplitVY = GFD_SPLIT_VY, kSplitWY = 4;

// GFD_SPLIT=0 in the environment keeps complex bands on star_kernel (for
// comparisons); the lane-pair kernel is the default.

template <class V>
inline bool split_eligible(const gfd_operator* op) {
  return vt<V>::NC == 2 && op->R >= 1 && op->R <= kSplitMaxR && split_enabled();
}

template <class V, int R, int MODE>
int split_go(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
             const StarParams<typename vt<V>::S>& p, const LaunchGeom& g, cudaStream_t s) {
  constexpr bool RHO = MODE == MODE_JACOBI || MODE == MODE_RESIDUAL;
  constexpr int S = RHO ? 3 : 4;
  constexpr size_t smem = split_smem_bytes<V, R, kSplitVY, kSplitWY, S, MODE>();
  auto kern = star_split_kernel<V, R, kSplitVY, kSplitWY, S, MODE>;
  int st = raise_smem_limit(kern, smem, "cudaFuncSetAttribute(star_split_kernel)");
  if (st) return st;
  if ((st = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                            int(cudaSharedmemCarveoutMaxShared)),
                       "cudaFuncSetAttribute(carveout)")))
    return st;
  const long long band = (long long)op->n[0] * op->n[1] * op->n[2];
  for (int64_t b0 = 0; b0 < nin; b0 += g.bands_per_launch) {
    int64_t nb = std::min<int64_t>(g.bands_per_launch, nin - b0);
    dim3 grid(g.grid.x, g.grid.y, (unsigned)(nb * g.nxc));
    launch_k(kern, grid, 32 * kSplitWY, smem, s, in + b0 * band, out + b0 * band,
             rho ? rho + b0 * band : nullptr, p);
  }
  return check_launch("star_split_kernel");
}

template <class V, int MODE>
int split_dispatch(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
                   const StarParams<typename vt<V>::S>& p, const LaunchGeom& g, cudaStream_t s) {
  if constexpr (vt<V>::NC == 2) {
    switch (op->R) {
      case 1: return split_go<V, 1, MODE>(op, in, out, rho, nin, p, g, s);
      case 2: return split_go<V, 2, MODE>(op, in, out, rho, nin, p, g, s);
      case 3: return split_go<V, 3, MODE>(op, in, out, rho, nin, p, g, s);
    }
  }
  return set_error(GFD_EUNSUPPORTED, "lane-pair stencil: complex bands, radius <= 3");
}

// ---------------------------------------------------------------------------
// complex128 bands on full-row tiles staged by TMA, real and imaginary parts
// on lane pairs (stencil_tmasplit.cuh).  Takes grids up to 128 columns
// (32 ng, ng <= kTsMaxNG) whose rows tile evenly along a periodic axis 1, and
// a potential only on an even number of columns (its rows must start on a
// 16-byte boundary).
// ---------------------------------------------------------------------------
}  // namespace gfd
GFD_DECLARE_TS_ENTRY(1)
GFD_DECLARE_TS_ENTRY(2)
GFD_DECLARE_TS_ENTRY(3)
GFD_DECLARE_TS_ENTRY(4)
namespace gfd {

inline int ts_ng(const gfd_operator* op) { return (op->n[2] + 31) / 32; }

template <class V>
inline bool ts_eligible(const gfd_operator* op, int mode, const void* in, const void* rho) {
  if constexpr (!std::is_same_v<V, cplx<double>>) {
    return false;
  } else {
    if (!tmasplit_enabled() || op->R < 1 || op->R > kSplitMaxR) return false;
    if (ts_ng(op) > kTsMaxNG) return false;
    if (op->per[1] && op->n[1] % kTsBY) return false;
    if (mode == OP_POTENTIAL && (op->n[2] & 1)) return false;
    auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return aligned(in) && (!rho || aligned(rho));
  }
}

inline int ts_dispatch(const gfd_operator* op, int kmode, const cplx<double>* in,
                       cplx<double>* out, const cplx<double>* rho, const void* pot, int64_t nin,
                       const StarParams<double>& p, int cps, cudaStream_t s) {
  switch (ts_ng(op)) {
    case 1: return ts_launch_1(op, kmode, in, out, rho, pot, nin, p, cps, s);
    case 2: return ts_launch_2(op, kmode, in, out, rho, pot, nin, p, cps, s);
    case 3: return ts_launch_3(op, kmode, in, out, rho, pot, nin, p, cps, s);
    case 4: return ts_launch_4(op, kmode, in, out, rho, pot, nin, p, cps, s);
  }
  return set_error(GFD_EUNSUPPORTED, "TMA lane-pair stencil: at most 128 columns");
}

// ---------------------------------------------------------------------------
// TMA-fed kernel (stencil_tma.cuh): complex128 apply on grids whose plane
// holds whole 16 x 32 tiles along periodic axes (zero-boundary axes may end
// in a partial tile: the loads fill zeros past the edge).
// ---------------------------------------------------------------------------
constexpr int kTmaVY = 2, kTmaG = 8, kTmaBY = kTmaVY * kTmaG, kTmaStages = 8;

// Defined in operator.cu.
bool star_tma_enabled();
int* star_error_flag();
int encode_tma_maps(TmaMaps* maps, const void* base, const gfd_operator* op, int64_t nb, int R,
                    int by);

inline bool tma_eligible(const gfd_operator* op, const void* in) {
  if (!star_tma_enabled() || op->R < 1 || op->R > 3) return false;
  if (op->n[2] < kTmaBZ || op->n[1] < kTmaBY) return false;
  if (op->per[2] && op->n[2] % kTmaBZ) return false;
  if (op->per[1] && op->n[1] % kTmaBY) return false;
  return (reinterpret_cast<uintptr_t>(in) & 15) == 0;
}

template <int R>
int star_tma_go(const gfd_operator* op, const cplx<double>* in, cplx<double>* out, int64_t nin,
                const StarParams<double>& base, const LaunchGeom& g, cudaStream_t s) {
  constexpr size_t smem = star_tma_smem_bytes<R, kTmaBY, kTmaStages>();
  auto kern = star_tma_kernel<R, kTmaVY, kTmaG, kTmaStages>;
  int st = raise_smem_limit(kern, smem, "cudaFuncSetAttribute(star_tma_kernel)");
  if (st) return st;
  // Two CTAs per SM need the largest shared-memory carveout.
  if ((st = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                                            int(cudaSharedmemCarveoutMaxShared)),
                       "cudaFuncSetAttribute(carveout)")))
    return st;
  int* err = star_error_flag();
  if (!err) return GFD_ECUDA;
  TmaMaps maps;
  if ((st = encode_tma_maps(&maps, in, op, nin, R, kTmaBY))) return st;
  const long long band = (long long)op->n[0] * op->n[1] * op->n[2];
  for (int64_t b0 = 0; b0 < nin; b0 += g.bands_per_launch) {
    int64_t nb = std::min<int64_t>(g.bands_per_launch, nin - b0);
    dim3 grid(g.grid.x, g.grid.y, (unsigned)(nb * g.nxc));
    launch_k(kern, grid, 32 * kTmaG, smem, s, out + b0 * band, base, maps, (int)b0, err);
  }
  return check_launch("star_tma_kernel");
}

inline int star_tma_dispatch(const gfd_operator* op, const cplx<double>* in, cplx<double>* out,
                             int64_t nin, const StarParams<double>& p, const LaunchGeom& g,
                             cudaStream_t s) {
  switch (op->R) {
    case 1: return star_tma_go<1>(op, in, out, nin, p, g, s);
    case 2: return star_tma_go<2>(op, in, out, nin, p, g, s);
    case 3: return star_tma_go<3>(op, in, out, nin, p, g, s);
  }
  return set_error(GFD_EUNSUPPORTED, "TMA stencil radius out of range");
}

template <class V, int R, int MODE>
int direct_go(const gfd_operator* op, const V* in, V* out, const V* rho,
              const StarParams<typename vt<V>::S>& p, int64_t nin, cudaStream_t s) {
  // fewer than 2^31 points per launch
  const int64_t most = std::max<int64_t>(1, 2000000000LL / p.band);
  for (int64_t b0 = 0; b0 < nin; b0 += most) {
    const int total = int(std::min<int64_t>(most, nin - b0) * p.band);
    launch_k(star_direct_kernel<V, R, MODE>, direct_blocks(total), 256, 0, s, in + b0 * p.band,
             out + b0 * p.band, rho ? rho + b0 * p.band : nullptr, p, total);
  }
  return check_launch("star_direct_kernel");
}

template <class V, int MODE>
int direct_dispatch(const gfd_operator* op, const V* in, V* out, const V* rho,
                    const StarParams<typename vt<V>::S>& p, int64_t nin, cudaStream_t s) {
  constexpr bool RELAX = MODE != MODE_APPLY && MODE != MODE_POTENTIAL;
  switch (op->R) {
    case 1: return direct_go<V, 1, MODE>(op, in, out, rho, p, nin, s);
    case 2: return direct_go<V, 2, MODE>(op, in, out, rho, p, nin, s);
    case 3: return direct_go<V, 3, MODE>(op, in, out, rho, p, nin, s);
  }
  if constexpr (vt<V>::NC == 2 && RELAX) {
    return set_error(GFD_EUNSUPPORTED, "complex Jacobi/residual sweeps need radius <= 3");
  } else {
    switch (op->R) {
      case 4: return direct_go<V, 4, MODE>(op, in, out, rho, p, nin, s);
      case 5: return direct_go<V, 5, MODE>(op, in, out, rho, p, nin, s);
      case 6: return direct_go<V, 6, MODE>(op, in, out, rho, p, nin, s);
    }
    return set_error(GFD_EUNSUPPORTED, "star stencil radius out of range");
  }
}

// Stencil parameters of a star operator for one mode (weights in the
// element precision S; Jacobi folds (1 - w) phi into the centre weight, see
// star_kernel, and the negated sweep flips the sign of w / c0, exactly).
template <class S>
void star_params(const gfd_operator* op, int mode, double w, const double* phase_cd,
                 StarParams<S>& p) {
  p = StarParams<S>{};
  p.n0 = op->n[0]; p.n1 = op->n[1]; p.n2 = op->n[2];
  p.per0 = op->per[0]; p.per1 = op->per[1]; p.per2 = op->per[2];
  p.band = (long long)op->n[0] * op->n[1] * op->n[2];
  p.c0 = S(op->c0);
  for (int i = 0; i < 2 * kMaxR + 1; i++) {
    p.cx[i] = S(op->cx[i]);
    p.cy[i] = S(op->cy[i]);
    p.cz[i] = S(op->cz[i]);
  }
  if (mode == OP_JACOBI || mode == OP_JACOBI_NEG) {
    p.c0 = S(-(1.0 - w) * op->c0 / w);
    p.wc = S(w / op->c0);
    if (mode == OP_JACOBI_NEG) p.wc = -p.wc;
  }
  fill_phases(p.P, phase_cd);
  p.fix_yz = 0;
  if (phase_cd)
    for (int c = 1; c < 3; c++)
      for (int d = 0; d < 2; d++)
        if (op->per[c] && (phase_cd[4 * c + 2 * d] != 1.0 || phase_cd[4 * c + 2 * d + 1] != 0.0))
          p.fix_yz = 1;
}

// ---------------------------------------------------------------------------
// complex128 bands up to radius 3: star_flex_kernel and star_pair_kernel.
// ---------------------------------------------------------------------------
// Axis-0 chunks and launches of a tiling with gx x gy tiles per plane.
template <class F>
int march_launches(const gfd_operator* op, int gx, int gy, int64_t nin, int cps, int resident,
                   StarParams<double>& p, F launch) {
  const int64_t tiles = (int64_t)gx * gy * nin;
  const int nxc =
      march_chunks(op->n[0], op->R, tiles, resident, num_sms(), split_target(cps, resident));
  p.x_chunk = (op->n[0] + nxc - 1) / nxc;
  p.nxc = (op->n[0] + p.x_chunk - 1) / p.x_chunk;
  const int64_t per_launch = std::max<int64_t>(1, 65535 / p.nxc);
  for (int64_t b0 = 0; b0 < nin; b0 += per_launch) {
    const int64_t nb = std::min<int64_t>(per_launch, nin - b0);
    launch(dim3(gx, gy, (unsigned)(nb * p.nxc)), b0 * p.band);
  }
  return GFD_OK;
}

// Time of one plane step of a CTA with its SM full, in microseconds, and the
// CTAs that an SM holds (registers).  Fitted to 27000 timed launches of the four
// kernels (grids of 24 to 144 points a side, 1 to 64 bands, every axis-0 split,
// zero and periodic boundaries; 7 to 10% rms) with march_split.h's rounds.  A
// potential adds 11% to each.
struct StepCost {
  double us;
  int resident;
};
inline double flex_step_us(const FlexTile& t, int R) {
  // a staged row costs as much as 20 staged cells
  return 0.155 + 0.00075 * flex_cells(t, R) + 0.0157 * (t.ty * kFlexVY + 2 * R);
}
inline StepCost c128_fixed_cost(int tile, int R) {
  const double us = tile == TILE_48 ? 0.45 + 0.11 * R : 0.28 + 0.184 * R;
  const int resident = tile == TILE_48 ? 2 : 3;
  if (R > 1) return {us, resident};
  return {us * (resident + 1) / resident, resident + 1};
}
// Bloch phases of axes 1 and 2 cost the pair kernel 63%, the others 39 to 47%.
inline StepCost pair_cost(bool phases) { return {phases ? 1.30 : 1.11, 3}; }

// The tile with the least time per plane.  Measured for 108^3 R = 3, 64 bands:
// (36, 6) 692 us, (36, 7) 725, (54, 4) 796; 90 x 100: (50, 5) 430, (26, 9) and
// (34, 7) slower; 96^2: (32, 8) 928, (48, 5) 989, (48, 4) 1006.
inline FlexTile flex_tile(const gfd_operator* op, int mode) {
  const int n1 = op->n[1], n2 = op->n[2], R = op->R;
  // Two CTAs in 196 KB, so that 60 KB stay with L1: tiles past that took 18 to
  // 24% longer than their cost (20 launches).
  const size_t most_smem = 97 * 1024 - (mode == OP_APPLY ? 0 : mode == OP_POTENTIAL ? 16 : 32) * 1024;
  FlexTile best = {std::min(n2, 8), 1};
  double cost = 0.0;
  int last = 0;
  for (int gx = (n2 + kFlexBZ - 1) / kFlexBZ; gx <= n2; gx++) {
    FlexTile t;
    t.bz = (n2 + gx - 1) / gx;
    if (t.bz == last) continue;
    last = t.bz;
    if (t.bz < 16 && cost > 0.0) break;
    const int most = std::min(kFlexNT / t.bz, (n1 + kFlexVY - 1) / kFlexVY);
    for (t.ty = 1; t.ty <= most; t.ty++) {
      if (flex_cells(t, R) > kFlexCPT * kFlexNT ||
          size_t(kFlexStages) * (t.ty * kFlexVY + 2 * R) * (kFlexBZ + 2 * R) * 16 > most_smem)
        break;
      const double tiles = double((n2 + t.bz - 1) / t.bz) *
                           ((n1 + t.ty * kFlexVY - 1) / (t.ty * kFlexVY));
      const double c = tiles * flex_step_us(t, R);
      if (cost == 0.0 || c < cost) {
        cost = c;
        best = t;
      }
    }
  }
  return best;
}
inline PairTile pair_tile(const gfd_operator* op) {
  // 32 columns by 12 rows; fewer where the grid is smaller
  const int gx = (op->n[2] + kPairBZ - 1) / kPairBZ;
  PairTile t;
  t.bz = ((op->n[2] + gx - 1) / gx + 1) / 2 * 2;
  t.ty = std::min(4, (op->n[1] + kPairVY - 1) / kPairVY);
  return t;
}
// Points of the padded plane of a tile.
inline long long padded(int n1, int n2, int by, int bz) {
  return (long long)((n1 + by - 1) / by * by) * ((n2 + bz - 1) / bz * bz);
}
// Built-in choice for complex128 up to radius 3 past the one-thread-per-point
// size (`fixed`: the fixed-side tile that would be taken; phases: Bloch phases on
// axes 1 or 2).
// Applies: the kernel whose launch takes the least time by the costs above, the
// fixed-side tile unless another saves 3%.  498 launches, one B200, times
// against the fixed-side tiles and four CTAs per SM for all: 0.87 in the
// geometric mean, 1.00 at the 90th percentile; with flex or pair tiles for every
// grid, whatever the bands, 0.98 and 1.23.
// Jacobi and residual sweeps: flex where the fixed tile pads the plane 8% more
// (Jacobi 104^2 2623 GB/s against 1929, but 2619 against 2685 on 96^2).
inline int c128_tile(const gfd_operator* op, int mode, int fixed, int64_t nin, bool phases) {
  const int n1 = op->n[1], n2 = op->n[2];
  const FlexTile f = flex_tile(op, mode);
  if (mode == OP_APPLY || mode == OP_POTENTIAL) {
    int tile = fixed;
    double cost = 0.0;
    auto consider = [&](int cand, int by, int bz, const StepCost& c) {
      const int64_t tiles = (int64_t)((n1 + by - 1) / by) * ((n2 + bz - 1) / bz) * nin;
      const double t = march_split(op->n[0], op->R, tiles, c.resident, num_sms()).steps * c.us;
      if (cost == 0.0 || t < cost) {
        tile = cand;
        cost = cost == 0.0 ? 0.97 * t : t;
      }
    };
    const TileDims td = tile_dims(fixed);
    consider(fixed, td.BY, td.BZ, c128_fixed_cost(fixed, op->R));
    consider(TILE_FLEX, f.ty * kFlexVY, f.bz, {flex_step_us(f, op->R), 2});
    if (mode == OP_APPLY && op->R == kPairR) {
      const PairTile t = pair_tile(op);
      consider(TILE_PAIR, t.ty * kPairVY, t.bz, pair_cost(phases));
    }
    if (fixed == TILE_48) consider(TILE_SHORT, 8, kShortTileZ, c128_fixed_cost(TILE_SHORT, op->R));
    return tile;
  }
  const TileDims td = tile_dims(fixed);
  return padded(n1, n2, td.BY, td.BZ) * 100 > padded(n1, n2, f.ty * kFlexVY, f.bz) * 108
             ? TILE_FLEX
             : fixed;
}

inline int pair_launch(const gfd_operator* op, const cplx<double>* in, cplx<double>* out,
                       int64_t nin, StarParams<double> p, int cps, cudaStream_t s) {
  const PairTile t = pair_tile(op);
  const int gx = (op->n[2] + t.bz - 1) / t.bz;
  const int gy = (op->n[1] + t.ty * kPairVY - 1) / (t.ty * kPairVY);
  const size_t smem = pair_smem_bytes(t.ty);
  int st = raise_smem_limit(star_pair_kernel, smem, "cudaFuncSetAttribute(star_pair_kernel)");
  if (st) return st;
  march_launches(op, gx, gy, nin, cps, 3, p, [&](dim3 grid, long long off) {
    launch_k(star_pair_kernel, grid, kPairNT, smem, s, in + off, out + off, p, t);
  });
  return check_launch("star_pair_kernel");
}

template <int R, int MODE>
int flex_go(const gfd_operator* op, int mode, const cplx<double>* in, cplx<double>* out,
            const cplx<double>* rho, int64_t nin, StarParams<double> p, int cps, cudaStream_t s) {
  const FlexTile t = flex_tile(op, mode);
  const int gx = (op->n[2] + t.bz - 1) / t.bz;
  const int gy = (op->n[1] + t.ty * kFlexVY - 1) / (t.ty * kFlexVY);
  auto kern = star_flex_kernel<R, MODE>;
  const size_t smem = flex_smem_bytes<R, MODE>(t);
  int st = raise_smem_limit(kern, smem, "cudaFuncSetAttribute(star_flex_kernel)");
  if (st) return st;
  march_launches(op, gx, gy, nin, cps, 2, p, [&](dim3 grid, long long off) {
    launch_k(kern, grid, kFlexNT, smem, s, in + off, out + off, rho ? rho + off : nullptr, p, t);
  });
  return check_launch("star_flex_kernel");
}
template <int MODE>
int flex_dispatch(const gfd_operator* op, int mode, const cplx<double>* in, cplx<double>* out,
                  const cplx<double>* rho, int64_t nin, const StarParams<double>& p, int cps,
                  cudaStream_t s) {
  switch (op->R) {
    case 1: return flex_go<1, MODE>(op, mode, in, out, rho, nin, p, cps, s);
    case 2: return flex_go<2, MODE>(op, mode, in, out, rho, nin, p, cps, s);
    case 3: return flex_go<3, MODE>(op, mode, in, out, rho, nin, p, cps, s);
  }
  return set_error(GFD_EUNSUPPORTED, "flex stencil: radius <= 3");
}

// ---------------------------------------------------------------------------
// Stencils along one axis (stencil_line.cuh), for applies past the
// one-thread-per-point limit.
// ---------------------------------------------------------------------------
template <class V, int R>
int line_go(const gfd_operator* op, int axis, const V* in, V* out, int64_t nin,
            LineParams<typename vt<V>::S>& p, cudaStream_t s) {
  const int n0 = op->n[0], n1 = op->n[1], n2 = op->n[2];
  p.n = op->n[axis];
  p.per = op->per[axis];
  if (axis == 2) {
    const int rows = std::max(1, 256 / n2);
    p.inner = (long long)n0 * n1 * nin;
    p.outer = 1;
    // up to 40 KB of staged rows, so several blocks share an SM
    const size_t row_b = size_t(rows) * (n2 + 2 * R) * sizeof(V);
    const int passes = (int)std::max<size_t>(1, std::min<size_t>(kLinePasses, 40 * 1024 / row_b));
    const long long blocks = (p.inner + (long long)rows * passes - 1) / ((long long)rows * passes);
    if (blocks > 0x7fffffffLL) return set_error(GFD_EUNSUPPORTED, "too many rows");
    launch_k(line_row_kernel<V, R>, dim3((unsigned)blocks), rows * n2, passes * row_b, s, in, out,
             p, rows, passes);
    return check_launch("line_row_kernel");
  }
  p.inner = axis == 0 ? (long long)n1 * n2 : n2;
  p.outer = axis == 0 ? nin : nin * n0;
  // Whole lines per thread once that fills the chip a few times over; below,
  // chunks of at least 4 (2R) outputs, whose 2R extra values come from L2, and
  // down to 2R outputs where the chip would not be full once.
  const long long threads = p.inner * p.outer, fill = 2048LL * num_sms();
  const int maxc = std::max(1, p.n / (8 * R)), most = std::max(1, p.n / std::max(4, 2 * R));
  p.nch = (int)std::min<long long>(maxc, std::max<long long>(1, 4 * fill / threads));
  if (threads * p.nch < fill)
    p.nch = (int)std::min<long long>(most, (fill + threads - 1) / threads);
  p.chunk = (p.n + p.nch - 1) / p.nch;
  p.nch = (p.n + p.chunk - 1) / p.chunk;
  const long long blocks = (threads + 255) / 256;
  if (blocks > 0x7fffffffLL) return set_error(GFD_EUNSUPPORTED, "too many lines");
  launch_k(line_march_kernel<V, R>, dim3((unsigned)blocks, (unsigned)p.nch), 256, 0, s, in, out, p);
  return check_launch("line_march_kernel");
}

template <class V>
int line_dispatch(const gfd_operator* op, int axis, const V* in, V* out, int64_t nin,
                  const double* phase_cd, cudaStream_t s) {
  using S = typename vt<V>::S;
  LineParams<S> p{};
  const double* w = axis == 0 ? op->cx : axis == 1 ? op->cy : op->cz;
  for (int i = 0; i < 2 * kMaxR + 1; i++) p.w[i] = S(w[i]);
  p.w[kMaxR] = S(op->c0);
  for (int d = 0; d < 2; d++)
    p.ph[d] = {S(phase_cd ? phase_cd[4 * axis + 2 * d] : 1.0),
               S(phase_cd ? phase_cd[4 * axis + 2 * d + 1] : 0.0)};
  switch (op->R) {
    case 1: return line_go<V, 1>(op, axis, in, out, nin, p, s);
    case 2: return line_go<V, 2>(op, axis, in, out, nin, p, s);
    case 3: return line_go<V, 3>(op, axis, in, out, nin, p, s);
    case 4: return line_go<V, 4>(op, axis, in, out, nin, p, s);
    case 5: return line_go<V, 5>(op, axis, in, out, nin, p, s);
    case 6: return line_go<V, 6>(op, axis, in, out, nin, p, s);
  }
  return set_error(GFD_EUNSUPPORTED, "star stencil radius out of range");
}

template <class V>
int launch_star_typed(const gfd_operator* op, int mode, const void* in, void* out, const void* rho,
                      int64_t nin, const double* phase_cd, double w, double* partials,
                      cudaStream_t s) {
  using S = typename vt<V>::S;
  StarParams<S> p;
  star_params(op, mode, w, phase_cd, p);
  const V* vin = static_cast<const V*>(in);
  V* vout = static_cast<V*>(out);
  const V* vrho = static_cast<const V*>(rho);
  const bool relax_mode = mode == OP_JACOBI || mode == OP_JACOBI_NEG || mode == OP_RESIDUAL;
  if constexpr (vt<V>::NC == 2) {
    if (relax_mode && op->R > kMaxComplexRelaxR)
      return set_error(GFD_EUNSUPPORTED, "complex Jacobi/residual sweeps need radius <= 3");
  }
  if (mode == OP_POTENTIAL) p.pot = rho;  // the potential travels as the source argument
  TunePlan plan;
  const bool tuned =
      mode != OP_RESIDUAL && tune_lookup(star_tune_key(op, dtype_of<V>(), mode, nin), &plan);
  if (tuned ? plan.path == PLAN_DIRECT : use_direct(op, nin)) {
    p.partials = partials;
    if (mode == OP_POTENTIAL)
      return direct_dispatch<V, MODE_POTENTIAL>(op, vin, vout, nullptr, p, nin, s);
    if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
      return direct_dispatch<V, MODE_JACOBI>(op, vin, vout, vrho, p, nin, s);
    if (mode == OP_RESIDUAL)
      return direct_dispatch<V, MODE_RESIDUAL>(op, vin, vout, vrho, p, nin, s);
    return direct_dispatch<V, MODE_APPLY>(op, vin, vout, nullptr, p, nin, s);
  }
  if (mode == OP_APPLY) {
    const int axis = line_apply_axis(op, (int)sizeof(V), nin);
    if (axis >= 0) return line_dispatch<V>(op, axis, vin, vout, nin, phase_cd, s);
  }
  if constexpr (std::is_same_v<V, cplx<double>>) {
    if (!tuned && mode == OP_APPLY && tma_eligible(op, in)) {
      LaunchGeom g = star_geom(op, TILE_WIDE, nin, op->R);
      p.nxc = g.nxc;
      p.x_chunk = g.x_chunk;
      return star_tma_dispatch(op, vin, vout, nin, p, g, s);
    }
  }
  // Built-in choices: the wide tile (narrow ones for short rows of radius 1 and
  // 2); complex applies the short or the 48-column tile, complex128 up to radius
  // 3 by c128_tile(); real bands of radius 3 the 48-column tile where it pays.
  // The lane-pair tiles come from plans only.  A plan's tile that a launch does
  // not have falls back to the built-in choice, so the geometry always matches
  // the kernel launched.
  int tile = pick_tile(op);
  const bool split = split_eligible<V>(op);
  const bool tsplit = ts_eligible<V>(op, mode, in, rho);
  const bool shortok =
      sizeof(V) >= 16 && (mode == OP_APPLY || mode == OP_POTENTIAL) && op->R <= kMaxShortR;
  const bool t48ok = vt<V>::NC == 2 && (mode == OP_APPLY || mode == OP_POTENTIAL) &&
                     op->R <= kMaxShortR && tile48_eligible(op);
  if (shortok && tile == TILE_WIDE) tile = tile48_eligible(op) ? TILE_48 : TILE_SHORT;
  // complex64 (512-band 96^3 Laplace): 2970-2990 GB/s against 2905-2918 for
  // the 32 x 16 tile
  if (t48ok && !shortok && tile == TILE_WIDE) tile = TILE_48;
  const bool flexok = sizeof(V) >= 16 && op->R <= kFlexR;
  const bool pairok = sizeof(V) >= 16 && op->R == kPairR && mode == OP_APPLY;
  if (flexok && (tile == TILE_WIDE || tile == TILE_SHORT || tile == TILE_48))
    tile = c128_tile(op, mode, tile, nin, p.fix_yz != 0);
  // real bands: 16 of 47^3 17.7 us against 21.1 us (two 32-column tiles)
  const bool t48rok = vt<V>::NC == 1 && mode != OP_RESIDUAL && tile48r_eligible(op);
  if (t48rok && tile == TILE_WIDE && tile48r_pays(op, mode, (int)sizeof(V), nin)) tile = TILE_48R;
  if (tuned) {
    if (plan.tile == TILE_PAIR)
      tile = pairok ? TILE_PAIR : tile;
    else if (plan.tile == TILE_FLEX)
      tile = flexok ? TILE_FLEX : tile;
    else if (plan.tile == TILE_48R)
      tile = t48rok ? TILE_48R : tile;
    else if (plan.tile == TILE_SHORT)
      tile = shortok ? TILE_SHORT : tile;
    else if (plan.tile == TILE_48)
      tile = t48ok ? TILE_48 : tile;
    else if (plan.tile == TILE_TMASPLIT)
      tile = tsplit ? TILE_TMASPLIT : tile;
    else if (plan.tile == TILE_SPLIT)
      tile = split ? TILE_SPLIT : tile;
    else if (op->R <= 2 || plan.tile == TILE_WIDE)
      tile = plan.tile;
  }
  if constexpr (std::is_same_v<V, cplx<double>>) {
    if (tile == TILE_TMASPLIT) {
      const int cps = tuned ? plan.cps : 0;
      if (mode == OP_POTENTIAL)
        return ts_dispatch(op, MODE_POTENTIAL, vin, vout, nullptr, rho, nin, p, cps, s);
      if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
        return ts_dispatch(op, MODE_JACOBI, vin, vout, vrho, nullptr, nin, p, cps, s);
      if (mode == OP_RESIDUAL)
        return ts_dispatch(op, MODE_RESIDUAL, vin, vout, vrho, nullptr, nin, p, cps, s);
      return ts_dispatch(op, MODE_APPLY, vin, vout, nullptr, nullptr, nin, p, cps, s);
    }
  }
  if constexpr (std::is_same_v<V, cplx<double>>) {
    const int cps = tuned ? plan.cps : 0;
    if (tile == TILE_PAIR) return pair_launch(op, vin, vout, nin, p, cps, s);
    if (tile == TILE_FLEX) {
      if (mode == OP_POTENTIAL)
        return flex_dispatch<MODE_POTENTIAL>(op, mode, vin, vout, nullptr, nin, p, cps, s);
      if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
        return flex_dispatch<MODE_JACOBI>(op, mode, vin, vout, vrho, nin, p, cps, s);
      if (mode == OP_RESIDUAL)
        return flex_dispatch<MODE_RESIDUAL>(op, mode, vin, vout, vrho, nin, p, cps, s);
      return flex_dispatch<MODE_APPLY>(op, mode, vin, vout, nullptr, nin, p, cps, s);
    }
  }
  int resident = 0;
  if (vt<V>::NC == 1) resident = real_resident(op, tile, mode, (int)sizeof(V));
  if (flexok && (tile == TILE_SHORT || tile == TILE_48))
    resident = c128_fixed_cost(tile, op->R).resident;
  LaunchGeom g = star_geom(op, tile, nin, op->R, tuned ? plan.cps : 0, resident);
  p.nxc = g.nxc;
  p.x_chunk = g.x_chunk;
  if (tile == TILE_SPLIT) {
    if (mode == OP_POTENTIAL)
      return split_dispatch<V, MODE_POTENTIAL>(op, vin, vout, nullptr, nin, p, g, s);
    if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
      return split_dispatch<V, MODE_JACOBI>(op, vin, vout, vrho, nin, p, g, s);
    if (mode == OP_RESIDUAL)
      return split_dispatch<V, MODE_RESIDUAL>(op, vin, vout, vrho, nin, p, g, s);
    return split_dispatch<V, MODE_APPLY>(op, vin, vout, nullptr, nin, p, g, s);
  }
  if (mode == OP_POTENTIAL)
    return star_dispatch<V, MODE_POTENTIAL>(op, tile, vin, vout, nullptr, nin, p, g, nullptr, s);
  if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
    return star_dispatch<V, MODE_JACOBI>(op, tile, vin, vout, vrho, nin, p, g, nullptr, s);
  if (mode == OP_RESIDUAL)
    return star_dispatch<V, MODE_RESIDUAL>(op, tile, vin, vout, vrho, nin, p, g, partials, s);
  return star_dispatch<V, MODE_APPLY>(op, tile, vin, vout, nullptr, nin, p, g, nullptr, s);
}

// ---------------------------------------------------------------------------
// Lattice-direction stencils (stencil_dirs.cuh): 256 threads, 2 rows each, two
// CTAs per SM; tile sides fit the grid (bz columns up to 48, the rows that the
// threads and 110 KB of staged 16-byte cells allow).
// ---------------------------------------------------------------------------
constexpr int kDirNT = 256, kDirVY = 2, kDirBZ = 48, kDirCPT = 5, kDirStages = 4;
constexpr size_t kDirSmem = 110 * 1024;

inline bool dirs_eligible(const gfd_operator* op, int mode) {
  return op->dirs && op->mp <= (mode == OP_APPLY ? kDirMaxR : 3);
}

struct DirGeom {
  int bz, ty, gx, gy, nxc, x_chunk;
  int64_t bands_per_launch;
};
// CTAs per SM of dirs_kernel, from its registers.  As for real_resident, a
// residual's figure does not depend on the type.
template <class V>
int dirs_resident(int R, int mode) {
  if (mode == OP_RESIDUAL) return 2;
  if (sizeof(V) == 16) return R == 1 ? 3 : 2;
  if (sizeof(V) == 4) return R <= 3 ? 4 : 3;
  if (vt<V>::NC == 2) return R <= 2 ? 3 : 2;
  if (mode != OP_APPLY) return R == 1 ? 3 : 2;
  return R == 1 ? 4 : R <= 3 ? 3 : 2;
}

inline DirGeom dirs_geom(const gfd_operator* op, int resident, int64_t nin) {
  const int R = op->mp;
  DirGeom g;
  g.gx = (op->n[2] + kDirBZ - 1) / kDirBZ;
  g.bz = (op->n[2] + g.gx - 1) / g.gx;
  auto fits = [&](int ty) {
    const int rows = ty * kDirVY + 2 * R;
    return (g.bz + 2 * R) * rows <= kDirCPT * kDirNT &&
           size_t(kDirStages) * rows * (kDirBZ + 2 * R) * 16 <= kDirSmem;
  };
  int ty = kDirNT / g.bz;
  while (ty > 1 && !fits(ty)) ty--;
  g.gy = (op->n[1] + ty * kDirVY - 1) / (ty * kDirVY);
  const int rows = (op->n[1] + g.gy - 1) / g.gy;
  g.ty = (rows + kDirVY - 1) / kDirVY;
  g.gy = (op->n[1] + g.ty * kDirVY - 1) / (g.ty * kDirVY);
  const int64_t tiles = (int64_t)g.gx * g.gy * std::max<int64_t>(nin, 1);
  const int nxc =
      march_chunks(op->n[0], R, tiles, resident, num_sms(), split_target(0, resident));
  g.x_chunk = (op->n[0] + nxc - 1) / nxc;
  g.nxc = (op->n[0] + g.x_chunk - 1) / g.x_chunk;
  g.bands_per_launch = std::max<int64_t>(1, 65535 / g.nxc);
  return g;
}

template <class S>
void dirs_params(const gfd_operator* op, int mode, double w, const double* phase_cd,
                 const DirGeom& g, DirParams<S>& p) {
  p = DirParams<S>{};
  p.n0 = op->n[0]; p.n1 = op->n[1]; p.n2 = op->n[2];
  p.per0 = op->per[0]; p.per1 = op->per[1]; p.per2 = op->per[2];
  p.band = (long long)op->n[0] * op->n[1] * op->n[2];
  p.bz = g.bz; p.ty = g.ty; p.x_chunk = g.x_chunk; p.nxc = g.nxc;
  const bool jacobi = mode == OP_JACOBI || mode == OP_JACOBI_NEG;
  double wx[2 * kDirMaxR + 1] = {0}, wh[8][kDirMaxR][3] = {};
  for (int c = 0; c < op->ncoefs; c++) {
    const int dx = op->off[3 * c], dy = op->off[3 * c + 1], dz = op->off[3 * c + 2];
    double x = op->coefs[c];
    // (1 - w) phi folded into the diagonal, as in star_kernel
    if (jacobi && c == 0) x = -(1.0 - w) * x / w;
    if (dy == 0 && dz == 0) {
      wx[kDirMaxR + dx] += x;
      p.xmask |= dx == 0 ? 1u : dx > 0 ? 2u : 4u;
      continue;
    }
    const int k = std::max(std::abs(dy), std::abs(dz));
    int h = 0;
    while (half_a(h) * k != dy || half_b(h) * k != dz) ++h;
    const int i = dx == 0 ? 0 : (dx > 0 ? 1 : 2);
    wh[h][k - 1][i] += x;
    p.mask |= 1u << (3 * h + i);
  }
  for (int i = 0; i < 2 * kDirMaxR + 1; i++) p.wx[i] = S(wx[i]);
  for (int h = 0; h < 8; h++)
    for (int k = 0; k < kDirMaxR; k++)
      for (int i = 0; i < 3; i++) p.w[h][k][i] = S(wh[h][k][i]);
  if (jacobi) {
    p.wc = S(w / op->coefs[0]);
    if (mode == OP_JACOBI_NEG) p.wc = -p.wc;
  }
  fill_phases(p.P, phase_cd);
  if (phase_cd)
    for (int c = 1; c < 3; c++)
      for (int d = 0; d < 2; d++)
        if (op->per[c] && (phase_cd[4 * c + 2 * d] != 1.0 || phase_cd[4 * c + 2 * d + 1] != 0.0))
          p.fix_yz = 1;
}

template <class V, int R, int MODE, bool FULL>
int dirs_launch(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
                DirParams<typename vt<V>::S>& p, const DirGeom& g, double* partials,
                cudaStream_t s) {
  auto kern = dirs_kernel<V, R, kDirVY, kDirNT, 2, kDirBZ, kDirCPT, kDirStages, MODE, FULL>;
  const size_t smem = dirs_smem_bytes<V, R, kDirVY, kDirNT, kDirBZ, kDirStages>(g.ty);
  int st = raise_smem_limit(kern, smem, "cudaFuncSetAttribute(dirs_kernel)");
  if (st) return st;
  for (int64_t b0 = 0; b0 < nin; b0 += g.bands_per_launch) {
    const int64_t nb = std::min<int64_t>(g.bands_per_launch, nin - b0);
    p.partials = partials ? partials + b0 * g.nxc * g.gx * g.gy : nullptr;
    launch_k(kern, dim3(g.gx, g.gy, (unsigned)(nb * g.nxc)), kDirNT, smem, s, in + b0 * p.band,
             out + b0 * p.band, rho ? rho + b0 * p.band : nullptr, p);
  }
  return check_launch("dirs_kernel");
}

template <class V, int R, int MODE>
int dirs_go(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
            DirParams<typename vt<V>::S>& p, const DirGeom& g, double* partials,
            cudaStream_t s) {
  if constexpr (sizeof(V) == 16 || (sizeof(V) == 8 && vt<V>::NC == 1)) {
    if (p.xmask == 7u) return dirs_launch<V, R, MODE, true>(op, in, out, rho, nin, p, g, partials, s);
  }
  return dirs_launch<V, R, MODE, false>(op, in, out, rho, nin, p, g, partials, s);
}

template <class V, int MODE>
int dirs_dispatch(const gfd_operator* op, int mode, const V* in, V* out, const V* rho,
                  int64_t nin, const double* phase_cd, double w, double* partials,
                  cudaStream_t s) {
  const DirGeom g = dirs_geom(op, dirs_resident<V>(op->mp, mode), nin);
  DirParams<typename vt<V>::S> p;
  dirs_params(op, mode, w, phase_cd, g, p);
  switch (op->mp) {
    case 1: return dirs_go<V, 1, MODE>(op, in, out, rho, nin, p, g, partials, s);
    case 2: return dirs_go<V, 2, MODE>(op, in, out, rho, nin, p, g, partials, s);
    case 3: return dirs_go<V, 3, MODE>(op, in, out, rho, nin, p, g, partials, s);
    case 4:
      if constexpr (MODE == MODE_APPLY)
        return dirs_go<V, 4, MODE>(op, in, out, rho, nin, p, g, partials, s);
  }
  return set_error(GFD_EUNSUPPORTED, "direction stencil radius out of range");
}

template <class V, int MODE>
int general_go(const gfd_operator* op, const V* in, V* out, const V* rho, int64_t nin,
               GenParams<typename vt<V>::S>& p, double* partials, cudaStream_t s) {
  constexpr int BZ = 32, TY = 4, VY = 2, BY = TY * VY;
  const int mp = std::max(op->mp, 0);
  const int gx = (op->n[2] + BZ - 1) / BZ, gy = (op->n[1] + BY - 1) / BY;
  gfd_operator tmp = *op;
  tmp.scratch = nullptr;  // geometry only
  LaunchGeom g = star_geom(op, TILE_WIDE, nin, std::max(mp, 1));
  g.grid = dim3(gx, gy, 1);
  p.nxc = g.nxc;
  p.x_chunk = g.x_chunk;
  size_t smem = (size_t)(2 * mp + 1) * (BY + 2 * mp) * (BZ + 2 * mp) * sizeof(V);
  if (smem > 227 * 1024) return set_error(GFD_EUNSUPPORTED, "stencil range too large");
  cudaError_t e = cudaFuncSetAttribute(general_kernel<V, BZ, TY, VY, MODE>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(general_kernel)");
  const long long band = (long long)op->n[0] * op->n[1] * op->n[2];
  for (int64_t b0 = 0; b0 < nin; b0 += g.bands_per_launch) {
    int64_t nb = std::min<int64_t>(g.bands_per_launch, nin - b0);
    dim3 grid(gx, gy, (unsigned)(nb * g.nxc));
    p.partials = partials ? partials + b0 * g.nxc * gx * gy : nullptr;
    launch_k(general_kernel<V, BZ, TY, VY, MODE>, grid, BZ * TY, smem, s, 
        in + b0 * band, out + b0 * band, rho ? rho + b0 * band : nullptr, p, mp);
  }
  return check_launch("general_kernel");
}

template <class V>
int launch_general_typed(const gfd_operator* op, int mode, const void* in, void* out,
                         const void* rho, int64_t nin, const double* phase_cd, double w,
                         double* partials, cudaStream_t s) {
  using S = typename vt<V>::S;
  if (op->ncoefs > kMaxCoefs) return set_error(GFD_EUNSUPPORTED, "too many stencil coefficients");
  if (dirs_eligible(op, mode)) {
    const V* a = static_cast<const V*>(in);
    V* b = static_cast<V*>(out);
    const V* r = static_cast<const V*>(rho);
    if (mode == OP_APPLY)
      return dirs_dispatch<V, MODE_APPLY>(op, mode, a, b, nullptr, nin, phase_cd, w, nullptr, s);
    if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
      return dirs_dispatch<V, MODE_JACOBI>(op, mode, a, b, r, nin, phase_cd, w, nullptr, s);
    if (mode == OP_RESIDUAL)
      return dirs_dispatch<V, MODE_RESIDUAL>(op, mode, a, b, r, nin, phase_cd, w, partials, s);
  }
  GenParams<S> p{};
  p.n0 = op->n[0]; p.n1 = op->n[1]; p.n2 = op->n[2];
  p.per0 = op->per[0]; p.per1 = op->per[1]; p.per2 = op->per[2];
  p.band = (long long)op->n[0] * op->n[1] * op->n[2];
  p.ncoefs = op->ncoefs;
  for (int c = 0; c < op->ncoefs; c++) {
    p.coefs[c] = S(op->coefs[c]);
    for (int a = 0; a < 3; a++) p.off[c][a] = (signed char)op->off[3 * c + a];
  }
  p.w = S(w);
  p.sign = mode == OP_JACOBI_NEG ? S(-1) : S(1);
  fill_phases(p.P, phase_cd);
  const V* vin = static_cast<const V*>(in);
  V* vout = static_cast<V*>(out);
  const V* vrho = static_cast<const V*>(rho);
  if (mode == OP_JACOBI || mode == OP_JACOBI_NEG)
    return general_go<V, MODE_JACOBI>(op, vin, vout, vrho, nin, p, nullptr, s);
  if (mode == OP_RESIDUAL)
    return general_go<V, MODE_RESIDUAL>(op, vin, vout, vrho, nin, p, partials, s);
  if (mode != OP_APPLY) return set_error(GFD_EUNSUPPORTED, "mode not available for this stencil");
  return general_go<V, MODE_APPLY>(op, vin, vout, nullptr, nin, p, nullptr, s);
}

inline int64_t partials_count(const gfd_operator* op, int64_t nin) {
  if (op->star && use_direct(op, nin))
    return direct_blocks((long long)op->n[0] * op->n[1] * op->n[2] * nin);
  if (op->star) {
    int tile = pick_tile(op);
    TileDims td = tile_dims(tile);
    LaunchGeom g = star_geom(op, tile, nin, op->R, 0,
                             real_resident(op, tile, OP_RESIDUAL, 8));
    int gx = (op->n[2] + td.BZ - 1) / td.BZ, gy = (op->n[1] + td.BY - 1) / td.BY;
    return (int64_t)gx * gy * g.nxc * nin;
  }
  if (dirs_eligible(op, OP_RESIDUAL)) {
    const DirGeom g = dirs_geom(op, dirs_resident<double>(op->mp, OP_RESIDUAL), nin);
    return (int64_t)g.gx * g.gy * g.nxc * nin;
  }
  const int BZ = 32, BY = 8;
  LaunchGeom g = star_geom(op, TILE_WIDE, nin, std::max(op->mp, 1));
  int gx = (op->n[2] + BZ - 1) / BZ, gy = (op->n[1] + BY - 1) / BY;
  return (int64_t)gx * gy * g.nxc * nin;
}

// Stencil parameters of a Gauss-Seidel colour pass (any offset set).
template <class S>
void gs_params(const gfd_operator* op, GenParams<S>& p) {
  p = GenParams<S>{};
  p.n0 = op->n[0]; p.n1 = op->n[1]; p.n2 = op->n[2];
  p.per0 = op->per[0]; p.per1 = op->per[1]; p.per2 = op->per[2];
  p.band = (long long)op->n[0] * op->n[1] * op->n[2];
  p.ncoefs = op->ncoefs;
  for (int c = 0; c < op->ncoefs; c++) {
    p.coefs[c] = S(op->coefs[c]);
    for (int a = 0; a < 3; a++) p.off[c][a] = (signed char)op->off[3 * c + a];
  }
}

// The same for an axis-aligned stencil (gs_star_point_at).
template <class S>
void gs_star_params(const gfd_operator* op, StarParams<S>& p) {
  star_params(op, OP_APPLY, 0.0, nullptr, p);
  p.wc = S(1) / p.c0;
}

// Gauss-Seidel sweeps: one launch per colour, R = 0 for offset tables.
template <class V, int R, class P>
int gs_sweeps(const gfd_operator* op, V* phi, const V* rho, int nsweeps, V* frozen, int ncolor,
              const P& p, cudaStream_t s) {
  const long long n = p.band;
  const bool any_per = op->per[0] || op->per[1] || op->per[2];
  const long long nq = (long long)op->n[0] * op->n[1] * gs_row_slots(op->n[2], ncolor);
  int blocks = (int)std::min<long long>((nq + 255) / 256, 148LL * 16);
  for (int sw = 0; sw < nsweeps; sw++) {
    if (any_per) {
      cudaError_t e = cudaMemcpyAsync(frozen, phi, n * sizeof(V), cudaMemcpyDeviceToDevice, s);
      if (e != cudaSuccess) return check_cuda(e, "cudaMemcpyAsync(frozen)");
    }
    V* fr = any_per ? frozen : phi;
    for (int c = 0; c < ncolor; c++) {
      if constexpr (R == 0)
        launch_k(color_gs_kernel<V>, blocks, 256, 0, s, phi, rho, fr, p, ncolor, c);
      else
        launch_k(color_gs_star_kernel<V, R>, blocks, 256, 0, s, phi, rho, fr, p, ncolor, c);
    }
  }
  return check_launch("color_gs_kernel");
}

// The same on a colour-split copy in the scratch grid, from kGsSplitPoints
// points of a zero-boundary grid up.
constexpr long long kGsSplitPoints = 40000;
inline bool gs_split_pays(const gfd_operator* op, int ncolor) {
  return op->full_star && !op->per[0] && !op->per[1] && !op->per[2] && (op->R == 2 || op->R == 3) &&
         ncolor == op->R + 1 &&
         (long long)op->n[0] * op->n[1] * op->n[2] >= kGsSplitPoints;
}
template <class V, int R>
int gs_split_sweeps(const gfd_operator* op, V* phi, const V* rho, int nsweeps, V* copy,
                    const StarParams<typename vt<V>::S>& p, cudaStream_t s) {
  const int n = (int)p.band, NC = R + 1;
  const int nq = p.n0 * p.n1 * gs_row_slots(p.n2, NC);
  const int cap = 16 * num_sms();
  const int nb = std::min((n + 255) / 256, cap), qb = std::min((nq + 255) / 256, cap);
  launch_k(gs_split_kernel<V, R + 1>, nb, 256, 0, s, phi, copy, p.n2, n, 1);
  for (int sw = 0; sw < nsweeps; sw++)
    for (int c = 0; c < NC; c++)
      launch_k(color_gs_split_kernel<V, R>, qb, 256, 0, s, copy, rho, p, c);
  launch_k(gs_split_kernel<V, R + 1>, nb, 256, 0, s, phi, copy, p.n2, n, 0);
  return check_launch("color_gs_split_kernel");
}

template <class V>
int gs_typed(const gfd_operator* op, V* phi, const V* rho, int nsweeps, V* frozen, int ncolor,
             cudaStream_t s) {
  using S = typename vt<V>::S;
  // The star form multiplies all 6 R weights; an operator that lacks some keeps
  // the offset table, which touches only the neighbours that there are.
  if (op->full_star) {
    StarParams<S> p;
    gs_star_params(op, p);
    if (frozen && nsweeps > 0 && gs_split_pays(op, ncolor))
      return op->R == 2 ? gs_split_sweeps<V, 2>(op, phi, rho, nsweeps, frozen, p, s)
                        : gs_split_sweeps<V, 3>(op, phi, rho, nsweeps, frozen, p, s);
    switch (op->R) {
      case 1: return gs_sweeps<V, 1>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
      case 2: return gs_sweeps<V, 2>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
      case 3: return gs_sweeps<V, 3>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
      case 4: return gs_sweeps<V, 4>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
      case 5: return gs_sweeps<V, 5>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
      case 6: return gs_sweeps<V, 6>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
    }
  }
  GenParams<S> p;
  gs_params(op, p);
  return gs_sweeps<V, 0>(op, phi, rho, nsweeps, frozen, ncolor, p, s);
}

}  // namespace gfd

// One of these per element type, defined in stencil_<type>.cu.
#define GFD_DECLARE_STENCIL_ENTRY(NAME)                                                        \
  namespace gfd {                                                                             \
  int star_##NAME(const gfd_operator*, int, const void*, void*, const void*, int64_t,          \
                  const double*, double, double*, cudaStream_t);                              \
  int general_##NAME(const gfd_operator*, int, const void*, void*, const void*, int64_t,       \
                     const double*, double, double*, cudaStream_t);                           \
  }
