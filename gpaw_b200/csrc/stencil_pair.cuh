// stencil_pair.cuh -- axis-aligned stencils of complex128 bands, two adjacent
// columns per lane pair.
//
// The same computation as star_kernel (stencil.cuh): a CTA owns a tile of rows
// by columns and marches along axis 0, planes arrive in a cp.async ring, and
// each output keeps 2R partial sums in registers.  Shared-memory reads bound
// star_kernel (89% of its rate): a thread of one column and two rows reads ten
// 16-byte values per point at R = 3.  Here
//
//  * the real and imaginary parts of a column pair sit on neighbouring lanes,
//    so a lane's values are 8 bytes and six outputs (3 rows by 2 columns) fit
//    its registers at 12 warps per SM: a window of 2R + 2 cells serves both
//    columns, a column of cells three rows, six reads per point;
//  * a staged row is kept in two halves, even columns then odd ones, so the
//    windows of neighbouring lanes are consecutive words at compile-time
//    offsets;
//  * tile sides are run-time values (an even number of columns up to 32, rows
//    in threes), so a grid of 95 points is not padded further;
//  * cells outside a zero-boundary axis are cleared once and never copied,
//    planes outside it are skipped.
//
// Plain applies of radius 3 only: 256 bands of 96^3, one B200, 4424 GB/s against
// 3949 for star_kernel's 48-column tile and 3906 for star_flex_kernel; two rows
// per lane (128 registers, 16 warps) 3728, four spill.  Radius 1, the Jacobi
// sweep and the apply with a potential were not faster (5493 against 5998 GB/s,
// 433 against 360 us, 3668 against 3639 GB/s).  At 64 bands the L1 pipe runs at
// 73% (star_kernel 90%, flex 84%) with 11 warps per SM.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace gfd {

constexpr int kPairR = 3;        // radius
constexpr int kPairVY = 3;       // rows per lane
constexpr int kPairNT = 128;     // threads, three CTAs per SM
constexpr int kPairBZ = 32;      // largest number of columns
constexpr int kPairCPT = 6;      // staged cells per thread
constexpr int kPairStages = 4;

// Tile of a launch: bz columns (even), ty lane rows of kPairVY rows.
struct PairTile {
  int bz, ty;
};

// Row layout in 16-byte cells: even columns from 0, odd ones from HALF on, half
// a 128-byte segment past a segment start, so the two runs that one warp
// writes land in different banks.
constexpr int pair_half() {
  int h = kPairBZ / 2 + kPairR;
  while (h % 8 != 4) ++h;
  return h;
}
constexpr int pair_pitch() { return pair_half() + kPairBZ / 2 + kPairR; }
inline size_t pair_smem_bytes(int ty) {
  return size_t(kPairStages) * (ty * kPairVY + 2 * kPairR) * pair_pitch() * 16;
}

static __global__ void __launch_bounds__(kPairNT, 3)
star_pair_kernel(const cplx<double>* __restrict__ in, cplx<double>* __restrict__ out,
                 const StarParams<double> p, const PairTile tl) {
  pdl_enter();
  using V = cplx<double>;
  constexpr int R = kPairR, VY = kPairVY, NT = kPairNT, S = kPairStages, CPT = kPairCPT;
  constexpr int Q = 2 * R, W = 2 * R + 2, CB = 16;
  constexpr int HALF = pair_half(), PITCH = pair_pitch();

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int BY = tl.ty * VY, SY = BY + 2 * R, SZ = tl.bz + 2 * R;
  const int stage = SY * PITCH;                                     // cells

  const int t = threadIdx.x;
  const int ty = t / tl.bz, lz = t - ty * tl.bz;  // bz lanes carry bz / 2 column pairs
  const int zp = lz >> 1, comp = lz & 1;
  const bool live = ty < tl.ty;
  const unsigned pair_mask = 3u << (t & 30);
  const int z0 = blockIdx.x * tl.bz, y0 = blockIdx.y * BY;
  const int bnd = blockIdx.z / p.nxc, xc = blockIdx.z % p.nxc;
  const int x0 = xc * p.x_chunk;
  const int x1 = min(p.n0, x0 + p.x_chunk);
  const V* inb = in + bnd * p.band;
  V* outb = out + bnd * p.band;
  const int pbeg = x0 - R, pend = x1 + R;
  const int plane = p.n1 * p.n2;

  // Cells this thread copies: byte offset in the plane and in the stage.
  unsigned csrc[CPT], cdst[CPT];
  unsigned clive = 0, cphase = 0;
  int ccode = 0;  // wrap sides, 4 bits per cell
  const int cells = SY * SZ;
#pragma unroll
  for (int i = 0; i < CPT; i++) {
    const int c = t + i * NT;
    csrc[i] = 0;
    cdst[i] = 0;
    if (c < cells) {
      const int sy = c / SZ, sz = c - sy * SZ;
      int ysd, zsd;
      const int ys = wrap_axis(y0 - R + sy, p.n1, p.per1, ysd);
      const int zs = wrap_axis(z0 - R + sz, p.n2, p.per2, zsd);
      cdst[i] = unsigned(sy * PITCH + (sz & 1) * HALF + (sz >> 1)) * CB;
      if (ys >= 0 && zs >= 0) {
        csrc[i] = unsigned(ys * p.n2 + zs) * CB;
        clive |= 1u << i;
        if (ysd >= 0 || zsd >= 0) cphase |= 1u << i;
        ccode |= ((ysd + 1) | ((zsd + 1) << 2)) << (4 * i);
      } else {
#pragma unroll
        for (int s = 0; s < S; s++)
          *reinterpret_cast<V*>(smem_raw + size_t(s) * stage * CB + cdst[i]) = vzero<V>();
      }
    }
  }
  const bool fix = p.fix_yz && cphase != 0;
  const int y = y0 + ty * VY, z = z0 + 2 * zp;  // first own point
  bool yin[VY];
#pragma unroll
  for (int j = 0; j < VY; j++) yin[j] = live && y + j < p.n1;
  const unsigned own0 = unsigned(y * p.n2 + z);
  const bool zin = z + comp < p.n2;  // the column this lane copies for and stores

  const unsigned smem0 = smem_addr(smem_raw);
  const size_t plane_b = size_t(plane) * CB;
  const char* inb_c = reinterpret_cast<const char*>(inb);

  int ist = 0;  // stage of the next plane to issue
  auto issue = [&](int P) {
    if (P < pend) {
      int xside;
      const int xs = wrap_plane(P, p.n0, p.per0, xside);
      if (xs >= 0) {
        const char* src = inb_c + size_t(xs) * plane_b;
        const unsigned sb = smem0 + unsigned(ist * stage) * CB;
#pragma unroll
        for (int i = 0; i < CPT; i++)
          if (clive >> i & 1u)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sb + cdst[i]),
                         "l"(src + csrc[i])
                         : "memory");
      }
    }
    cp_async_commit();
    ist = ist + 1 == S ? 0 : ist + 1;
  };

#pragma unroll
  for (int k = 0; k < S - 1; k++) issue(pbeg + k);

  double acc[VY][2][Q];
#pragma unroll
  for (int j = 0; j < VY; j++)
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int q = 0; q < Q; q++) acc[j][c][q] = 0.0;
  char* out_c = reinterpret_cast<char*>(outb);
  // Window origin: row ty * VY (the first row's halo row 0), window position 0;
  // position k sits at (k & 1) * HALF + k / 2.
  const unsigned wbase = unsigned(ty * VY * PITCH + zp) * CB + unsigned(comp) * 8u;
  int st = 0;

  for (int base = pbeg; base < pend; base += Q) {
#pragma unroll
    for (int u = 0; u < Q; ++u) {
      const int pl = base + u;
      if (pl < pend) {
        cp_async_wait<S - 2>();
        if (fix) {
#pragma unroll
          for (int i = 0; i < CPT; i++) {
            if (!(cphase >> i & 1u)) continue;
            const int ys = ((ccode >> (4 * i)) & 3) - 1, zs = ((ccode >> (4 * i + 2)) & 3) - 1;
            V* cell = reinterpret_cast<V*>(smem_raw + size_t(st * stage) * CB + cdst[i]);
            V v = *cell;
            if (ys >= 0) v = phase_mul(phase_of(p.P, 1, ys), v);
            if (zs >= 0) v = phase_mul(phase_of(p.P, 2, zs), v);
            *cell = v;
          }
        }
        __syncthreads();
        issue(pl + S - 1);

        int xside;
        const int xs = wrap_plane(pl, p.n0, p.per0, xside);
        double own[VY][2];
#pragma unroll
        for (int j = 0; j < VY; j++) own[j][0] = own[j][1] = 0.0;
        if (live && xs >= 0) {
          const unsigned char* wp = smem_raw + size_t(st * stage) * CB + wbase;
          auto at = [&](int row, int k) -> double {  // row from -R, window position k
            return *reinterpret_cast<const double*>(
                wp + ((row + R) * PITCH + (k & 1) * HALF + (k >> 1)) * CB);
          };
          if (pl >= x0 && pl < x1) {
#pragma unroll
            for (int r = -R; r < VY + R; r++) {
              double v[2];
              if (r >= 0 && r < VY) {
                double w[W];
#pragma unroll
                for (int k = 0; k < W; k++) w[k] = at(r, k);
#pragma unroll
                for (int c = 0; c < 2; c++) {
                  v[c] = own[r][c] = w[R + c];
                  madd(acc[r][c][u], p.c0, v[c]);
                }
#pragma unroll
                for (int k = 1; k <= R; k++)
#pragma unroll
                  for (int c = 0; c < 2; c++) {
                    madd(acc[r][c][u], p.cz[kMaxR - k], w[R + c - k]);
                    madd(acc[r][c][u], p.cz[kMaxR + k], w[R + c + k]);
                  }
              } else {
                v[0] = at(r, R);
                v[1] = at(r, R + 1);
              }
#pragma unroll
              for (int j = 0; j < VY; j++)
                if (r != j && r - j <= R && j - r <= R) {
#pragma unroll
                  for (int c = 0; c < 2; c++) madd(acc[j][c][u], p.cy[kMaxR + r - j], v[c]);
                }
            }
          } else {
#pragma unroll
            for (int j = 0; j < VY; j++) {
              own[j][0] = at(j, R);
              own[j][1] = at(j, R + 1);
            }
          }
          if (xside >= 0) {
            // (pr re - pi im, pr im + pi re) over the two lanes
            const cplx<double> ph = phase_of(p.P, 0, xside);
#pragma unroll
            for (int j = 0; j < VY; j++)
#pragma unroll
              for (int c = 0; c < 2; c++) {
                const double other = __shfl_xor_sync(pair_mask, own[j][c], 1);
                own[j][c] = fma(ph.re, own[j][c], (comp ? ph.im : -ph.im) * other);
              }
          }
#pragma unroll
          for (int k = 1; k <= R; k++)
#pragma unroll
            for (int j = 0; j < VY; j++)
#pragma unroll
              for (int c = 0; c < 2; c++) {
                madd(acc[j][c][(u - k + 2 * Q) % Q], p.cx[kMaxR + k], own[j][c]);
                if (k < R) madd(acc[j][c][(u + k) % Q], p.cx[kMaxR - k], own[j][c]);
              }
        }

        const int q = pl - R;
        const int qs = (u + R) % Q;  // slot of output pl - R, then of output pl + R
        if (q >= x0 && q < x1) {
          char* dstp = out_c + size_t(q) * plane_b + size_t(own0) * CB;
#pragma unroll
          for (int j = 0; j < VY; j++) {
            const double o[2] = {acc[j][0][qs], acc[j][1][qs]};
            // Each lane stores one whole column: the re lane column z, the im
            // lane column z + 1.
            const double got = __shfl_xor_sync(pair_mask, comp ? o[0] : o[1], 1);
            const V full = comp ? V{got, o[1]} : V{o[0], got};
            if (yin[j] && zin) stcs(reinterpret_cast<V*>(dstp + size_t(j) * p.n2 * CB) + comp, full);
          }
        }
#pragma unroll
        for (int j = 0; j < VY; j++)
#pragma unroll
          for (int c = 0; c < 2; c++) acc[j][c][qs] = vmul(p.cx[kMaxR - R], own[j][c]);
        st = st + 1 == S ? 0 : st + 1;
      }
    }
  }
  cp_async_wait<0>();
}

}  // namespace gfd
