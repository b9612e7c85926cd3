// stencil_dirs.cuh -- stencils whose offsets are the multiples k d, all of
// k = 1 .. R, of lattice directions d (every component -1, 0 or 1; 13 and their
// opposites): the Laplacians of non-orthogonal cells
// (gpaw/fd_operators.py:231-282) and the Mehrstellen pair.
//
// A CTA marches a tile along axis 0 as star_kernel does; planes arrive with
// their full halo (corners included) in a cp.async ring.  On an incoming plane
// a point's taps sit at its own position and at k (a, b) for the eight in-plane
// half directions (a, b); the value at k (a, b) belongs to the outputs 0, +k or
// -k planes away, whose 2R + 1 partial sums stay in registers.  A value is
// therefore read from shared memory once for up to three taps (fcc, R = 3: 19
// reads for 37 taps), weights come from the parameter block, and which half
// directions exist at all is decided by uniform branches on a mask.  The kernel
// over an offset table this replaces (general_kernel, kept for all other offset
// sets) looked up offset, weight and plane slot per tap.  96 complex128 bands of
// a 48^3 fcc cell, nn = 3: 1157 us with general_kernel, 195 us (1750 GB/s) here;
// 53 us of memory time, the 19 16-byte shared reads per point bound it.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace gfd {

constexpr int kDirMaxR = 4;
// In-plane half directions (a, b): (1, 0), (0, 1), (1, 1), (1, -1), each
// followed by its opposite.
__host__ __device__ constexpr int half_a(int h) {
  return (h >> 1) == 1 ? 0 : ((h & 1) ? -1 : 1);
}
__host__ __device__ constexpr int half_b(int h) {
  return ((h >> 1) == 0 ? 0 : (h >> 1) == 3 ? -1 : 1) * ((h & 1) ? -1 : 1);
}

template <class S>
struct DirParams {
  int n0, n1, n2;
  int per0, per1, per2;
  int x_chunk, nxc;
  int bz, ty;          // tile: bz columns by ty * VY rows
  long long band;
  // Weights: centre column wx[kDirMaxR + dx] (dx planes away; dx = 0 the
  // centre), and for half direction h at distance k: w[h][k - 1][0] in the
  // plane, [1] and [2] for offsets (+k, k a, k b) and (-k, k a, k b).
  S wx[2 * kDirMaxR + 1];
  S w[8][kDirMaxR][3];
  unsigned mask;       // bit 3 h + i: weights w[h][.][i] exist
  unsigned xmask;      // bit 0: the centre's weight exists, 1: those of
                       // +1 .. +R planes, 2: of -1 .. -R planes
  S wc;                // MODE_JACOBI: +-w / diagonal
  int fix_yz;
  Phases<S> P;
  double* partials;
};

template <class V, int R, int VY, int NT, int BZMAX, int S>
size_t dirs_smem_bytes(int ty) {
  return size_t(S) * (ty * VY + 2 * R) * (BZMAX + 2 * R) * sizeof(V);
}

// FULL: the operator has the centre's weight and the whole axis-0 column.  The
// other form takes a value without a weight as zero (zero times an infinity is
// not), by selects: they cost complex128 5 to 30% by their registers, float64 up
// to 3%, the other types nothing; a branch around the column cost 3 to 12%.
template <class V, int R, int VY, int NT, int MINB, int BZMAX, int CPT, int S, int MODE, bool FULL>
__global__ void __launch_bounds__(NT, MINB)
dirs_kernel(const V* __restrict__ in, V* __restrict__ out, const V* __restrict__ rho,
            const DirParams<typename vt<V>::S> p) {
  pdl_enter();
  constexpr int Q = 2 * R + 1, PITCH = BZMAX + 2 * R;
  constexpr int CB = int(sizeof(V));
  constexpr bool RHO = MODE == MODE_JACOBI || MODE == MODE_RESIDUAL;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double red[NT / 32];
  const int BY = p.ty * VY, SY = BY + 2 * R, SZ = p.bz + 2 * R;
  const int stage = SY * PITCH;

  const int t = threadIdx.x, ty = t / p.bz, tz = t - ty * p.bz;
  const int z0 = blockIdx.x * p.bz, y0 = blockIdx.y * BY;
  const int bnd = blockIdx.z / p.nxc, xc = blockIdx.z % p.nxc;
  const int x0 = xc * p.x_chunk, x1 = min(p.n0, x0 + p.x_chunk);
  const int pbeg = x0 - R, pend = x1 + R;
  const int plane = p.n1 * p.n2;
  const size_t plane_b = size_t(plane) * CB;
  const char* inb = reinterpret_cast<const char*>(in + bnd * p.band);

  unsigned csrc[CPT], cdst[CPT];
  unsigned clive = 0, cphase = 0;
  const int cells = SY * SZ;
#pragma unroll
  for (int i = 0; i < CPT; i++) {
    const int c = t + i * NT;
    csrc[i] = cdst[i] = 0;
    if (c < cells) {
      const int sy = c / SZ, sz = c - sy * SZ;
      int ysd, zsd;
      const int ys = wrap_axis(y0 - R + sy, p.n1, p.per1, ysd);
      const int zs = wrap_axis(z0 - R + sz, p.n2, p.per2, zsd);
      cdst[i] = unsigned(sy * PITCH + sz) * CB;
      if (ys >= 0 && zs >= 0) {
        csrc[i] = unsigned(ys * p.n2 + zs) * CB;
        clive |= 1u << i;
        if (ysd >= 0 || zsd >= 0) cphase |= 1u << i;
      } else {
        // A zero point: cleared in every stage once, never copied.
#pragma unroll
        for (int s = 0; s < S; s++)
          *reinterpret_cast<V*>(smem_raw + size_t(s) * stage * CB + cdst[i]) = vzero<V>();
      }
    }
  }
  const bool fix = vt<V>::NC == 2 && p.fix_yz && cphase != 0;
  const bool live = ty < p.ty && z0 + tz < p.n2;
  const int y = y0 + ty * VY;
  const unsigned own0 = unsigned(y * p.n2 + z0 + tz);
  const unsigned smem0 = smem_addr(smem_raw);

  int ist = 0;
  auto issue = [&](int P) {
    int side;
    const int xs = P < pend ? wrap_plane(P, p.n0, p.per0, side) : -1;
    if (xs >= 0) {
      const char* src = inb + size_t(xs) * plane_b;
      const unsigned sb = smem0 + unsigned(ist * stage) * CB;
#pragma unroll
      for (int i = 0; i < CPT; i++)
        if (clive >> i & 1u)
          asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(sb + cdst[i]),
                       "l"(src + csrc[i]), "n"(CB)
                       : "memory");
    }
    cp_async_commit();
    ist = ist + 1 == S ? 0 : ist + 1;
  };
#pragma unroll
  for (int k = 0; k < S - 1; k++) issue(pbeg + k);

  V acc[VY][Q];  // acc[j][i]: output plane pl - R + i
#pragma unroll
  for (int j = 0; j < VY; j++)
#pragma unroll
    for (int i = 0; i < Q; i++) acc[j][i] = vzero<V>();
  double sumsq = 0.0;
  const unsigned wbase = unsigned((ty * VY + R) * PITCH + R + tz) * CB;
  int st = 0;

  for (int pl = pbeg; pl < pend; ++pl) {
    cp_async_wait<S - 2>();
    int xside;
    const int xs = wrap_plane(pl, p.n0, p.per0, xside);
    if constexpr (vt<V>::NC == 2) {
      // Bloch phases of the cells this thread copied: in the plane, and on a
      // wrapped plane the axis-0 phase of every cell.
      if (xs >= 0 && (fix || xside >= 0)) {
#pragma unroll
        for (int i = 0; i < CPT; i++) {
          if (!(clive >> i & 1u)) continue;
          V* cell = reinterpret_cast<V*>(smem_raw + size_t(st * stage) * CB + cdst[i]);
          V v = *cell;
          if (xside >= 0) v = phase_mul(phase_of(p.P, 0, xside), v);
          if (fix && (cphase >> i & 1u)) {
            const int c = t + i * NT, sy = c / SZ, sz = c - sy * SZ;
            int ysd, zsd;
            wrap_axis(y0 - R + sy, p.n1, p.per1, ysd);
            wrap_axis(z0 - R + sz, p.n2, p.per2, zsd);
            if (ysd >= 0) v = phase_mul(phase_of(p.P, 1, ysd), v);
            if (zsd >= 0) v = phase_mul(phase_of(p.P, 2, zsd), v);
          }
          *cell = v;
        }
      }
    }
    __syncthreads();
    issue(pl + S - 1);

    const int q = pl - R;  // the output this plane completes
    V src[VY];
    if constexpr (RHO) {
      if (q >= x0 && q < x1 && live) {
        const V* rp = rho + bnd * p.band + (long long)q * plane + own0;
#pragma unroll
        for (int j = 0; j < VY; j++)
          if (y + j < p.n1) src[j] = ldro(rp + j * p.n2);
      }
    }
    if (live && xs >= 0) {
      const unsigned char* wp = smem_raw + size_t(st * stage) * CB + wbase;
      auto at = [&](int j, int dy, int dz) -> V {
        return *reinterpret_cast<const V*>(wp + ((j + dy) * PITCH + dz) * CB);
      };
#pragma unroll
      for (int j = 0; j < VY; j++) {
        const V v = at(j, 0, 0);
        const V own = value_or_zero(FULL || (p.xmask & 1u), v);
        const V up = value_or_zero(FULL || (p.xmask & 2u), v);
        const V down = value_or_zero(FULL || (p.xmask & 4u), v);
#pragma unroll
        for (int dx = -R; dx <= R; dx++)
          madd(acc[j][R - dx], p.wx[kDirMaxR + dx], dx == 0 ? own : dx > 0 ? up : down);
      }
#pragma unroll
      for (int h = 0; h < 8; h++) {
        const unsigned m = p.mask >> (3 * h) & 7u;
        if (!m) continue;
        V v[R][VY];
#pragma unroll
        for (int k = 1; k <= R; k++)
#pragma unroll
          for (int j = 0; j < VY; j++) v[k - 1][j] = at(j, k * half_a(h), k * half_b(h));
        if (m & 1u) {
#pragma unroll
          for (int k = 1; k <= R; k++)
#pragma unroll
            for (int j = 0; j < VY; j++) madd(acc[j][R], p.w[h][k - 1][0], v[k - 1][j]);
        }
        if (m & 2u) {
#pragma unroll
          for (int k = 1; k <= R; k++)
#pragma unroll
            for (int j = 0; j < VY; j++) madd(acc[j][R - k], p.w[h][k - 1][1], v[k - 1][j]);
        }
        if (m & 4u) {
#pragma unroll
          for (int k = 1; k <= R; k++)
#pragma unroll
            for (int j = 0; j < VY; j++) madd(acc[j][R + k], p.w[h][k - 1][2], v[k - 1][j]);
        }
      }
    }

    if (q >= x0 && q < x1 && live) {
      V* op = out + bnd * p.band + (long long)q * plane + own0;
#pragma unroll
      for (int j = 0; j < VY; j++) {
        if (y + j >= p.n1) continue;
        V o = acc[j][0];
        if constexpr (MODE == MODE_JACOBI) o = vmul(p.wc, vsub(src[j], o));
        if constexpr (MODE == MODE_RESIDUAL) {
          o = vsub(o, src[j]);
          if constexpr (vt<V>::NC == 1) sumsq += sq(o);
        }
        stcs(op + j * p.n2, o);
      }
    }
#pragma unroll
    for (int j = 0; j < VY; j++) {
#pragma unroll
      for (int i = 0; i + 1 < Q; i++) acc[j][i] = acc[j][i + 1];
      acc[j][Q - 1] = vzero<V>();
    }
    st = st + 1 == S ? 0 : st + 1;
  }
  cp_async_wait<0>();

  if constexpr (MODE == MODE_RESIDUAL) {
    if (p.partials) {
      const double sblk = block_sum<NT>(sumsq, red);
      if (t == 0) {
        const long long cta = (long long)blockIdx.z * gridDim.y * gridDim.x +
                              (long long)blockIdx.y * gridDim.x + blockIdx.x;
        p.partials[cta] = sblk;
      }
    }
  }
}

}  // namespace gfd
