// stencil_flex.cuh -- axis-aligned stencils of complex128 bands on tiles whose
// sides fit the grid.
//
// star_kernel's tiles have compile-time sides, so a grid of 100 columns is
// padded to 128 (32-column tiles) or 144 (48): a quarter of the reads and
// sums are thrown away.  Here a CTA of 256 threads takes any bz <= 64 columns by
// ty * 2 rows that the threads allow (100 columns: 2 x 50); the row pitch in
// shared memory stays a compile-time constant, so the 2 + 2R column cells and 2R
// row cells of a thread are reads at fixed offsets.  Two rows per thread hold 4R
// complex partial sums: 128 registers, 16 warps per SM.  Cells outside a
// zero-boundary axis are cleared once and never copied; planes outside it are
// skipped.  The order of the sums is star_kernel's.  84 x 90 x 100, 16 bands:
// 120 us, the L1 pipe at 83%, short-scoreboard stalls 3.1 per issue: shared
// reads and their latency bound it.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace gfd {

constexpr int kFlexR = 3, kFlexVY = 2, kFlexNT = 256, kFlexBZ = 64, kFlexCPT = 4, kFlexStages = 4;

struct FlexTile {
  int bz, ty;
};
inline int flex_cells(const FlexTile& t, int R) {
  return (t.bz + 2 * R) * (t.ty * kFlexVY + 2 * R);
}
template <int R, int MODE>
size_t flex_smem_bytes(const FlexTile& t) {
  constexpr bool RHO = MODE == MODE_JACOBI || MODE == MODE_RESIDUAL;
  const size_t slots = size_t(kFlexStages) * kFlexVY * kFlexNT;
  return size_t(kFlexStages) * (t.ty * kFlexVY + 2 * R) * (kFlexBZ + 2 * R) * 16 +
         (RHO ? slots * 16 : 0) + (MODE == MODE_POTENTIAL ? slots * 8 : 0);
}

template <int R, int MODE>
__global__ void __launch_bounds__(kFlexNT, 2)
star_flex_kernel(const cplx<double>* __restrict__ in, cplx<double>* __restrict__ out,
                 const cplx<double>* __restrict__ rho, const StarParams<double> p,
                 const FlexTile tl) {
  pdl_enter();
  using V = cplx<double>;
  constexpr int VY = kFlexVY, NT = kFlexNT, S = kFlexStages, CPT = kFlexCPT;
  constexpr int Q = 2 * R, PITCH = kFlexBZ + 2 * R, CB = 16;
  constexpr bool RHO = MODE == MODE_JACOBI || MODE == MODE_RESIDUAL;
  constexpr bool POT = MODE == MODE_POTENTIAL;

  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int BY = tl.ty * VY, SZ = tl.bz + 2 * R;
  const unsigned stage_b = unsigned((BY + 2 * R) * PITCH) * CB;
  unsigned char* extra = smem_raw + size_t(S) * stage_b;  // [S][VY][NT] source terms

  const int t = threadIdx.x, ty = t / tl.bz, tz = t - ty * tl.bz;
  const int z0 = blockIdx.x * tl.bz, y0 = blockIdx.y * BY;
  const int bnd = blockIdx.z / p.nxc, xc = blockIdx.z % p.nxc;
  const int x0 = xc * p.x_chunk;
  const int x1 = min(p.n0, x0 + p.x_chunk);
  const int pbeg = x0 - R, pend = x1 + R;
  const int plane = p.n1 * p.n2;
  const size_t plane_b = size_t(plane) * CB;
  const char* inb_c = reinterpret_cast<const char*>(in + bnd * p.band);

  unsigned csrc[CPT], cdst[CPT];
  unsigned clive = 0, cphase = 0;
  int ccode = 0;  // wrap sides, 4 bits per cell
  const int cells = (BY + 2 * R) * SZ;
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
        ccode |= ((ysd + 1) | ((zsd + 1) << 2)) << (4 * i);
      } else {
#pragma unroll
        for (int s = 0; s < S; s++)
          *reinterpret_cast<V*>(smem_raw + size_t(s) * stage_b + cdst[i]) = vzero<V>();
      }
    }
  }
  const bool fix = p.fix_yz && cphase != 0;
  const bool live = ty < tl.ty && z0 + tz < p.n2;
  const int y = y0 + ty * VY;
  bool yin[VY];
#pragma unroll
  for (int j = 0; j < VY; j++) yin[j] = live && y + j < p.n1;
  const unsigned own0 = unsigned(y * p.n2 + z0 + tz);
  const unsigned smem0 = smem_addr(smem_raw), esmem0 = smem_addr(extra);

  int ist = 0;
  auto issue = [&](int P) {
    if (P < pend) {
      int xside;
      const int xs = wrap_plane(P, p.n0, p.per0, xside);
      if (xs >= 0) {
        const char* src = inb_c + size_t(xs) * plane_b;
        const unsigned sb = smem0 + unsigned(ist) * stage_b;
#pragma unroll
        for (int i = 0; i < CPT; i++)
          if (clive >> i & 1u)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(sb + cdst[i]),
                         "l"(src + csrc[i])
                         : "memory");
      }
      if constexpr (RHO) {
        const int q = P - R;
        if (q >= x0 && q < x1) {
          const V* rs = rho + bnd * p.band + size_t(q) * plane + own0;
#pragma unroll
          for (int j = 0; j < VY; j++)
            if (yin[j])
              asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(
                               esmem0 + unsigned((ist * VY + j) * NT + t) * 16u),
                           "l"(rs + j * p.n2)
                           : "memory");
        }
      }
      if constexpr (POT) {
        if (P >= x0 && P < x1) {
          const double* vs = static_cast<const double*>(p.pot) + size_t(P) * plane + own0;
#pragma unroll
          for (int j = 0; j < VY; j++)
            if (yin[j])
              asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                               esmem0 + unsigned((ist * VY + j) * NT + t) * 8u),
                           "l"(vs + j * p.n2)
                           : "memory");
        }
      }
    }
    cp_async_commit();
    ist = ist + 1 == S ? 0 : ist + 1;
  };
#pragma unroll
  for (int k = 0; k < S - 1; k++) issue(pbeg + k);

  V acc[VY][Q];
#pragma unroll
  for (int j = 0; j < VY; j++)
#pragma unroll
    for (int q = 0; q < Q; q++) acc[j][q] = vzero<V>();
  char* out_c = reinterpret_cast<char*>(out + bnd * p.band);
  const unsigned wbase = unsigned(ty * VY * PITCH + R + tz) * CB;
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
            V* cell = reinterpret_cast<V*>(smem_raw + size_t(unsigned(st) * stage_b) + cdst[i]);
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
        V own[VY];
#pragma unroll
        for (int j = 0; j < VY; j++) own[j] = vzero<V>();
        if (live && xs >= 0) {
          const V* colp =
              reinterpret_cast<const V*>(smem_raw + size_t(unsigned(st) * stage_b) + wbase);
          if (pl >= x0 && pl < x1) {
            V col[VY + 2 * R];
#pragma unroll
            for (int m = 0; m < VY + 2 * R; m++) col[m] = colp[m * PITCH];
#pragma unroll
            for (int j = 0; j < VY; j++) {
              own[j] = col[R + j];
              const V* row = colp + (R + j) * PITCH;
              double cc = p.c0;
              if constexpr (POT)
                cc += reinterpret_cast<const double*>(extra)[(st * VY + j) * NT + t];
              V sy = vmul(cc, col[R + j]);
              V sz = vzero<V>();
#pragma unroll
              for (int k = 1; k <= R; k++) {
                madd(sy, p.cy[kMaxR - k], col[R + j - k]);
                madd(sz, p.cz[kMaxR - k], row[-k]);
                madd(sy, p.cy[kMaxR + k], col[R + j + k]);
                madd(sz, p.cz[kMaxR + k], row[k]);
              }
              acc[j][u] = vadd(acc[j][u], vadd(sy, sz));
            }
          } else {
#pragma unroll
            for (int j = 0; j < VY; j++) own[j] = colp[(R + j) * PITCH];
          }
          if (xside >= 0) {
#pragma unroll
            for (int j = 0; j < VY; j++) own[j] = phase_mul(phase_of(p.P, 0, xside), own[j]);
          }
#pragma unroll
          for (int j = 0; j < VY; j++) {
#pragma unroll
            for (int k = 1; k <= R; k++)
              madd(acc[j][(u - k + 2 * Q) % Q], p.cx[kMaxR + k], own[j]);
#pragma unroll
            for (int k = 1; k < R; k++) madd(acc[j][(u + k) % Q], p.cx[kMaxR - k], own[j]);
          }
        }

        const int q = pl - R;
        const int qs = (u + R) % Q;  // slot of output pl - R, then of output pl + R
        if (q >= x0 && q < x1) {
          char* dstp = out_c + size_t(q) * plane_b + size_t(own0) * CB;
#pragma unroll
          for (int j = 0; j < VY; j++) {
            if (!yin[j]) continue;
            V o = acc[j][qs];
            if constexpr (RHO) {
              const V rv = reinterpret_cast<const V*>(extra)[(st * VY + j) * NT + t];
              if constexpr (MODE == MODE_JACOBI) o = vmul(p.wc, vsub(rv, o));
              else o = vsub(o, rv);
            }
            stcs(reinterpret_cast<V*>(dstp + size_t(j) * p.n2 * CB), o);
          }
        }
#pragma unroll
        for (int j = 0; j < VY; j++) acc[j][qs] = vmul(p.cx[kMaxR - R], own[j]);
        st = st + 1 == S ? 0 : st + 1;
      }
    }
  }
  cp_async_wait<0>();
}

}  // namespace gfd
