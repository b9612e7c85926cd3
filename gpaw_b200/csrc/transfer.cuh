// transfer.cuh -- multigrid restriction and interpolation for sm_100a.
//
// The reference (c/bmgs/restrict.c, c/bmgs/interpolate.c, driven by
// c/transformers.c:54-123) fills a halo-padded copy of each band and then
// runs three transposing 1-D passes (axis 2, axis 1, axis 0) through scratch
// buffers: about four reads and four writes of the array.  Here one kernel
// does all three passes:
//   * a CTA owns a tile of output points in (axis 1, axis 2) and marches
//     along axis 0;
//   * each input plane (with its halo, mapped in-kernel: zero, periodic, or
//     periodic times the Bloch phase) is staged in shared memory, the axis-2
//     pass and then the axis-1 pass run there (the reference's pass order,
//     so the arithmetic matches term by term);
//   * the axis-0 pass works on 2-D results in registers: a queue of the last
//     planes' (interpolation) or the sums of the coarse planes under way
//     (restriction).
// HBM traffic is one read of the input and one write of the output.
//
// Weights: Lagrange weights for K = 2*nn taps (c/bmgs/restrict.c:37-57,
// c/bmgs/interpolate.c:46-59).
#pragma once

#include "common.cuh"
#include "internal.h"

namespace gfd {

template <int NN, class S>
__host__ __device__ __forceinline__ S lagw(int m) {
  if (NN == 1) return S(0.5);
  if (NN == 2) return m == 0 ? S(0.5625) : S(-0.0625);
  if (NN == 3) return m == 0 ? S(0.58593750) : (m == 1 ? S(-0.09765625) : S(0.01171875));
  return m == 0 ? S(0.59814453125)
                : (m == 1 ? S(-0.11962890625) : (m == 2 ? S(0.02392578125) : S(-0.00244140625)));
}

// Restriction tap around a[0] with stride st (in elements of V):
// 0.5 * (a0 + w1 (a[+1] + a[-1]) + w2 (a[+3] + a[-3]) + ...)
template <int NN, class V, class Get>
__device__ __forceinline__ V rst_tap(Get get) {
  using S = typename vt<V>::S;
  V x = get(0);
#pragma unroll
  for (int k = 0; k < NN; k++) x = vadd(x, vmul(lagw<NN, S>(k), vadd(get(2 * k + 1), get(-(2 * k + 1)))));
  return vmul(S(0.5), x);
}

// Interpolated value between a[0] and a[1]:
// w0 (a[0] + a[1]) + w1 (a[-1] + a[2]) + ...
template <int NN, class V, class Get>
__device__ __forceinline__ V ip_tap(Get get) {
  using S = typename vt<V>::S;
  V x = vmul(lagw<NN, S>(0), vadd(get(0), get(1)));
#pragma unroll
  for (int m = 1; m < NN; m++) x = vadd(x, vmul(lagw<NN, S>(m), vadd(get(-m), get(1 + m))));
  return x;
}

template <class S>
struct TrParams {
  int ni0, ni1, ni2;   // input points per axis
  int no0, no1, no2;   // output points per axis
  int lo0, lo1, lo2;   // low-side padding of the input (pad[c][0])
  int sk0, sk1, sk2;   // interpolation: skip[c][0]
  int per0, per1, per2;
  int x_chunk, nxc;    // output planes per CTA along axis 0, chunk count
  long long band_in, band_out;
  Phases<S> P;
  // Restriction only: when seed != nullptr, also write seed = seed_scale *
  // out (same layout as out).  A weighted-Jacobi sweep from a zero guess
  // gives exactly (w / c0) rho, so a multigrid level's first sweep comes
  // out of the restriction that produces its rho.
  void* seed;
  S seed_scale;
  // Factor on the transferred value (1, or -1 for the negated transfers of
  // the band preconditioner; multiplying by -1 is exact).
  S out_scale;
  // Interpolation only: when total != nullptr the factor is target / *total
  // instead (a device scalar that an earlier kernel on the stream wrote).
  const double* total;
  double target;
};
template <class S>
__device__ __forceinline__ S out_factor(const TrParams<S>& p) {
  return p.total ? S(p.target / *p.total) : p.out_scale;
}

// Transfer parameters of a transformer (host side).
template <class S>
void tr_params(const gfd_transformer* tr, const double* ph, void* seed, double seed_scale,
               double out_scale, TrParams<S>& p) {
  p = TrParams<S>{};
  p.ni0 = tr->nin[0]; p.ni1 = tr->nin[1]; p.ni2 = tr->nin[2];
  p.no0 = tr->nout[0]; p.no1 = tr->nout[1]; p.no2 = tr->nout[2];
  p.lo0 = tr->pad[0][0]; p.lo1 = tr->pad[1][0]; p.lo2 = tr->pad[2][0];
  p.sk0 = tr->skip[0][0]; p.sk1 = tr->skip[1][0]; p.sk2 = tr->skip[2][0];
  p.per0 = tr->per[0]; p.per1 = tr->per[1]; p.per2 = tr->per[2];
  p.band_in = (long long)tr->nin[0] * tr->nin[1] * tr->nin[2];
  p.band_out = (long long)tr->nout[0] * tr->nout[1] * tr->nout[2];
  for (int c = 0; c < 3; c++)
    for (int d = 0; d < 2; d++) {
      p.P.ph[c][d].re = ph ? S(ph[4 * c + 2 * d]) : S(1);
      p.P.ph[c][d].im = ph ? S(ph[4 * c + 2 * d + 1]) : S(0);
    }
  p.seed = seed;
  p.seed_scale = S(seed_scale);
  p.out_scale = S(out_scale);
}

// Pack an in-plane source offset and its wrap sides; -1 = zero point.
__device__ __forceinline__ int pack_src(int ys, int zs, int n2, int ysd, int zsd) {
  if (ys < 0 || zs < 0) return -1;
  return ((ys * n2 + zs) << 4) | ((ysd + 1) | ((zsd + 1) << 2));
}

template <class V, class S>
__device__ __forceinline__ V apply_phases(V v, int code, int xside, const Phases<S>& P) {
  if constexpr (vt<V>::NC == 2) {
    if (xside >= 0) v = phase_mul(phase_of(P, 0, xside), v);
    int ys = (code & 3) - 1, zs = ((code >> 2) & 3) - 1;
    if (ys >= 0) v = phase_mul(phase_of(P, 1, ys), v);
    if (zs >= 0) v = phase_mul(phase_of(P, 2, zs), v);
  }
  return v;
}

// Staged fine rows of the restriction kernel (RZ cells) are stored with
// their even positions first and their odd ones from HALF on.  HALF sits
// half a 128-byte segment past a segment start (E / 2 elements mod E), so
// the even and odd runs that one shared-memory wavefront writes land in
// different banks.
template <class V, int RZ>
constexpr int rst_half() {
  constexpr int E = 128 / int(sizeof(V));
  int h = (RZ + 1) / 2;
  while (h % E != E / 2) ++h;
  return h;
}
template <class V, int RZ>
constexpr int rst_pitch() {
  return rst_half<V, RZ>() + RZ / 2;
}

// Types up to 8 bytes: each thread restricts two neighbouring coarse
// columns at once, and a staged fine row is kept in four phases (position
// mod 4), phase q at q * QS + position / 4.  The 2nn + 1 taps of the pair
// (even positions) and its two centres (odd ones) are then consecutive
// words across lanes: 2nn + 3 loads per pair instead of 2 (2nn + 1).  QS is
// E / 4 past a 128-byte segment start (E / 4 elements mod E), so the four
// phase runs one wavefront writes use each bank at most twice.
template <class V, int RZ>
constexpr int rst_quad() {
  constexpr int E = 128 / int(sizeof(V));
  int q = (RZ + 3) / 4;
  while (q % E != E / 4) ++q;
  return q;
}
template <class V>
constexpr bool rst_pairs() {
  return sizeof(V) <= 8;
}
// Shared-memory row pitch of a staged fine row (elements).
template <class V, int RZ>
constexpr int rst_row_pitch() {
  if constexpr (rst_pairs<V>()) return 4 * rst_quad<V, RZ>();
  else return rst_pitch<V, RZ>();
}

template <class V>
struct alignas(2 * sizeof(V)) VPair {
  V a, b;
};

// ---------------------------------------------------------------------------
// Restriction: coarse index i on an axis takes the fine padded point
// (K-1) + 2i (c/bmgs/restrict.c:65-69), i.e. fine array index
// 2i + (2nn-1) - lo.
// ---------------------------------------------------------------------------
template <class V, int NN, int BZC, int TYC, int VYC>
__global__ void __launch_bounds__(BZC * TYC)
restrict_kernel(const V* __restrict__ in, V* __restrict__ out,
                const TrParams<typename vt<V>::S> p) {
  pdl_enter();
  using S = typename vt<V>::S;
  constexpr int NT = BZC * TYC, BYC = TYC * VYC;
  constexpr int W = 2 * NN - 1;           // wing of one restriction tap
  constexpr int RY = 2 * BYC - 1 + 2 * W;
  constexpr int RZ = 2 * BZC - 1 + 2 * W;
  constexpr int CELLS = RY * RZ;
  constexpr int CC = (CELLS + NT - 1) / NT;
  // Each staged fine row holds its even positions first, then its odd ones:
  // the axis-2 taps of neighbouring coarse points are then consecutive
  // words (a stride-2 read would hit every bank twice).
  constexpr bool PAIRS = rst_pairs<V>();
  constexpr int HALF = rst_half<V, RZ>(), QS = rst_quad<V, RZ>();
  constexpr int RZP = rst_row_pitch<V, RZ>(), STG = RY * RZP;
  static_assert(!PAIRS || BZC % 2 == 0, "coarse columns come in pairs");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* F = reinterpret_cast<V*>(smem_raw);          // [2][RY][RZP], rows in phases
  V* T = F + 2 * STG;                             // [2][RY][BZC]

  const int t = threadIdx.x, tz = t % BZC, ty = t / BZC;
  const int Z0 = blockIdx.x * BZC, Y0 = blockIdx.y * BYC;
  const int bnd = blockIdx.z / p.nxc, xc = blockIdx.z % p.nxc;
  const int X0 = xc * p.x_chunk, X1 = min(p.no0, X0 + p.x_chunk);
  const long long plane_in = (long long)p.ni1 * p.ni2;
  const long long plane_out = (long long)p.no1 * p.no2;
  const V* inb = in + bnd * p.band_in;
  V* outb = out + bnd * p.band_out;
  const int fy0 = 2 * Y0 - p.lo1, fz0 = 2 * Z0 - p.lo2;

  int src[CC];
  int dpos[CC];  // stage position of cell t + i * NT
#pragma unroll
  for (int i = 0; i < CC; i++) {
    int c = t + i * NT;
    src[i] = -1;
    dpos[i] = 0;
    if (c < CELLS) {
      int sy = c / RZ, sz = c % RZ;
      if constexpr (PAIRS) dpos[i] = sy * RZP + (sz & 3) * QS + (sz >> 2);
      else dpos[i] = sy * RZP + ((sz & 1) ? HALF + (sz >> 1) : (sz >> 1));
      int ysd, zsd;
      int ys = wrap_axis(fy0 + sy, p.ni1, p.per1, ysd);
      int zs = wrap_axis(fz0 + sz, p.ni2, p.per2, zsd);
      src[i] = pack_src(ys, zs, p.ni2, ysd, zsd);
    }
  }

  const int fbeg = 2 * X0 + W - p.lo0 - W;
  const int fend = 2 * (X1 - 1) + W - p.lo0 + W + 1;

  V rv[CC];
  auto load = [&](int f) {
    int xside;
    int xs = (f < fend) ? wrap_axis(f, p.ni0, p.per0, xside) : -1;
#pragma unroll
    for (int i = 0; i < CC; i++) {
      V v = vzero<V>();
      if (xs >= 0 && src[i] >= 0) {
        v = ldro(inb + xs * plane_in + (src[i] >> 4));
        v = apply_phases<V, S>(v, src[i] & 15, xside, p.P);
      }
      rv[i] = v;
    }
  };

  load(fbeg);
  // The in-plane values of fine plane f at this thread's coarse points: stage
  // the plane, axis-2 pass, axis-1 pass.
  auto in_plane = [&](int f, V (&v)[VYC]) {
    V* Fb = F + (f & 1) * STG;
    V* Tb = T + (f & 1) * RY * BZC;
#pragma unroll
    for (int i = 0; i < CC; i++)
      if (t + i * NT < CELLS) Fb[dpos[i]] = rv[i];
    load(f + 1);
    __syncthreads();
    if constexpr (PAIRS) {
      // axis-2 pass, columns cz = 2m and 2m + 1 of every staged row: their
      // taps are fine positions 4m + 2j (j = 0 .. 2nn; j = 0 .. 2nn - 1 for
      // cz = 2m, 1 .. 2nn for 2m + 1), their centres 4m + W and 4m + W + 2.
      for (int c = t; c < RY * (BZC / 2); c += NT) {
        const int sy = c / (BZC / 2), m = c % (BZC / 2);
        const V* row = Fb + sy * RZP + m;
        V tap[2 * NN + 1];
#pragma unroll
        for (int j = 0; j <= 2 * NN; j++) tap[j] = row[((2 * j) & 3) * QS + (j >> 1)];
        const V c0 = row[(W & 3) * QS + (W >> 2)];
        const V c1 = row[((W + 2) & 3) * QS + ((W + 2) >> 2)];
        VPair<V> r;
        r.a = rst_tap<NN, V>([&](int o) { return o == 0 ? c0 : tap[(o + W) >> 1]; });
        r.b = rst_tap<NN, V>([&](int o) { return o == 0 ? c1 : tap[((o + W) >> 1) + 1]; });
        *reinterpret_cast<VPair<V>*>(Tb + sy * BZC + 2 * m) = r;
      }
    } else {
      // axis-2 pass: Tb[sy][cz] for every staged row; fine position
      // 2 cz + W + o sits at (W + o) & 1 ? HALF : 0, + cz + (W + o) / 2.
      for (int c = t; c < RY * BZC; c += NT) {
        const int sy = c / BZC, cz = c % BZC;
        const V* row = Fb + sy * RZP + cz;
        Tb[c] = rst_tap<NN, V>([&](int o) { return row[((W + o) & 1 ? HALF : 0) + ((W + o) >> 1)]; });
      }
    }
    __syncthreads();
    if constexpr (VYC == 2) {
      // axis-1 pass, adjacent coarse rows 2 ty and 2 ty + 1: as for the column
      // pairs, 2nn + 3 reads instead of 2 (2nn + 1)
      const V* col = Tb + 4 * ty * BZC + tz;
      V tap[2 * NN + 1];
#pragma unroll
      for (int m = 0; m <= 2 * NN; m++) tap[m] = col[2 * m * BZC];
      const V c0 = col[W * BZC], c1 = col[(W + 2) * BZC];
      v[0] = rst_tap<NN, V>([&](int o) { return o == 0 ? c0 : tap[(o + W) >> 1]; });
      v[1] = rst_tap<NN, V>([&](int o) { return o == 0 ? c1 : tap[((o + W) >> 1) + 1]; });
    } else {
      static_assert(VYC == 1, "one or two coarse rows per thread");
      const V* col = Tb + (2 * ty + W) * BZC + tz;
      v[0] = rst_tap<NN, V>([&](int o) { return col[o * BZC]; });
    }
  };

  // axis-0 pass: fine planes 2h and 2h + 1 past fbeg.  The first is an odd
  // neighbour of coarse planes X0 + h - m, m = 0 .. W, whose sums stay in
  // registers (s[.][m]); the second is the centre of X0 + h - (nn - 1).
  V s[VYC][W + 1];
#pragma unroll
  for (int j = 0; j < VYC; j++)
#pragma unroll
    for (int m = 0; m <= W; m++) s[j][m] = vzero<V>();
  const int last = X1 - X0 + W - 1;
  for (int h = 0; h <= last; h++) {
    V v[VYC];
    in_plane(fbeg + 2 * h, v);
#pragma unroll
    for (int j = 0; j < VYC; j++) {
#pragma unroll
      for (int m = W; m > 0; m--) s[j][m] = s[j][m - 1];
      s[j][0] = vzero<V>();
#pragma unroll
      for (int m = 0; m <= W; m++) {
        const int d = 2 * m - W, k = ((d < 0 ? -d : d) - 1) / 2;
        madd(s[j][m], lagw<NN, S>(k), v[j]);
      }
    }
    const int X = X0 + h - W;
    if (X >= X0) {
#pragma unroll
      for (int j = 0; j < VYC; j++) {
        const int y = Y0 + ty * VYC + j, z = Z0 + tz;
        if (y < p.no1 && z < p.no2) {
          V r = vmul(S(0.5), s[j][W]);
          if (p.out_scale != S(1)) r = vmul(p.out_scale, r);
          const long long o = X * plane_out + (long long)y * p.no2 + z;
          stcs(outb + o, r);
          if (p.seed) stcs(static_cast<V*>(p.seed) + (outb - out) + o, vmul(p.seed_scale, r));
        }
      }
    }
    if (h < last) {
      in_plane(fbeg + 2 * h + 1, v);
#pragma unroll
      for (int j = 0; j < VYC; j++) s[j][NN - 1] = vadd(s[j][NN - 1], v[j]);
    }
  }
}

// ---------------------------------------------------------------------------
// Interpolation: fine index f on an axis has g = f + skip[c][0]; g = 2i is a
// copy of coarse padded point (nn-1) + i, g = 2i + 1 the K-tap value between
// (nn-1) + i and (nn-1) + i + 1 (c/bmgs/interpolate.c:19-66).  Coarse array
// index of step i: c(i) = i + nn - 1 - lo.
// ---------------------------------------------------------------------------
// SUB: out = base - interpolated value (the multigrid correction
// phi -= interpolate(e), in place when base == out).
// TOTAL: the factor comes from p.total (the renormalised density; a form of its
// own: carried in a register by all, it cost complex64 nn = 2 12%).
template <class V, int NN, int BZF, int TYF, int VYF, bool SUB, bool TOTAL>
__global__ void __launch_bounds__(BZF * TYF)
interp_kernel(const V* __restrict__ in, V* out, const V* base,
              const TrParams<typename vt<V>::S> p) {
  pdl_enter();
  using S = typename vt<V>::S;
  constexpr int NT = BZF * TYF, BYF = TYF * VYF;
  constexpr int CY = BYF / 2 + 2 * NN, CZ = BZF / 2 + 2 * NN;
  constexpr int CELLS = CY * CZ;
  constexpr int CC = (CELLS + NT - 1) / NT;
  constexpr int QL = 2 * NN;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* C = reinterpret_cast<V*>(smem_raw);  // [2][CY][CZ]
  V* T = C + 2 * CELLS;                   // [2][CY][BZF]

  const int t = threadIdx.x, tz = t % BZF, ty = t / BZF;
  const int Z0 = blockIdx.x * BZF, Y0 = blockIdx.y * BYF;
  const int bnd = blockIdx.z / p.nxc, xc = blockIdx.z % p.nxc;
  const int X0 = xc * p.x_chunk, X1 = min(p.no0, X0 + p.x_chunk);
  const long long plane_in = (long long)p.ni1 * p.ni2;
  const long long plane_out = (long long)p.no1 * p.no2;
  [[maybe_unused]] const S factor = TOTAL ? out_factor(p) : S(1);
  const V* inb = in + bnd * p.band_in;
  V* outb = out + bnd * p.band_out;
  const V* baseb = SUB ? base + bnd * p.band_out : nullptr;
  const int iy0 = (Y0 + p.sk1) >> 1, iz0 = (Z0 + p.sk2) >> 1;
  const int cy0 = iy0 - p.lo1, cz0 = iz0 - p.lo2;  // coarse origin of the tile

  int src[CC];
#pragma unroll
  for (int i = 0; i < CC; i++) {
    int c = t + i * NT;
    src[i] = -1;
    if (c < CELLS) {
      int sy = c / CZ, sz = c % CZ;
      int ysd, zsd;
      int ys = wrap_axis(cy0 + sy, p.ni1, p.per1, ysd);
      int zs = wrap_axis(cz0 + sz, p.ni2, p.per2, zsd);
      src[i] = pack_src(ys, zs, p.ni2, ysd, zsd);
    }
  }

  const int ia = (X0 + p.sk0) >> 1, ib = (X1 - 1 + p.sk0) >> 1;
  const int cbeg = ia - p.lo0;                    // c(ia) - (nn-1)
  const int cend = ib + NN - 1 - p.lo0 + NN + 1;  // one past c(ib) + nn

  V rv[CC];
  auto load = [&](int c) {
    int xside;
    int xs = (c < cend) ? wrap_axis(c, p.ni0, p.per0, xside) : -1;
#pragma unroll
    for (int i = 0; i < CC; i++) {
      V v = vzero<V>();
      if (xs >= 0 && src[i] >= 0) {
        v = ldro(inb + xs * plane_in + (src[i] >> 4));
        v = apply_phases<V, S>(v, src[i] & 15, xside, p.P);
      }
      rv[i] = v;
    }
  };

  V q[VYF][QL];
#pragma unroll
  for (int j = 0; j < VYF; j++)
#pragma unroll
    for (int k = 0; k < QL; k++) q[j][k] = vzero<V>();

  // One barrier per coarse plane: plane c + 1 is staged (into the other
  // buffer) while plane c's axis-2 results are being written, and both C
  // and T are double-buffered, so every read of a buffer is separated from
  // the next write into it by a barrier.
  load(cbeg);
#pragma unroll
  for (int i = 0; i < CC; i++)
    if (t + i * NT < CELLS) C[(cbeg & 1) * CELLS + t + i * NT] = rv[i];
  load(cbeg + 1);
  __syncthreads();
  for (int c = cbeg; c < cend; ++c) {
    const V* Cb = C + (c & 1) * CELLS;
    V* Tb = T + (c & 1) * CY * BZF;
    // axis-2 pass: every staged coarse row to this tile's fine columns, two
    // adjacent fine columns per thread (one even, one odd, whatever the
    // skip), so every lane does one copy and one K-tap value.
    static_assert(BZF % 2 == 0, "fine columns come in pairs");
    for (int e = t; e < CY * (BZF / 2); e += NT) {
      const int sy = e / (BZF / 2), fz = 2 * (e % (BZF / 2));
      const int g = Z0 + fz + p.sk2;
      const int odd0 = g & 1;  // the same for every pair of the tile
      const int ge = g + odd0, go = g + 1 - odd0;  // the pair's even and odd g
      const V* rowe = Cb + sy * CZ + ((ge >> 1) - iz0 + NN - 1);
      const V* rowo = Cb + sy * CZ + ((go >> 1) - iz0 + NN - 1);
      V* out = Tb + sy * BZF + fz;
      out[odd0] = rowe[0];
      out[1 - odd0] = ip_tap<NN, V>([&](int o) { return rowo[o]; });
    }
    if (c + 1 < cend) {
      V* Cn = C + ((c + 1) & 1) * CELLS;
#pragma unroll
      for (int i = 0; i < CC; i++)
        if (t + i * NT < CELLS) Cn[t + i * NT] = rv[i];
      load(c + 2);
    }
    __syncthreads();
    // axis-1 pass for this thread's fine points
#pragma unroll
    for (int j = 0; j < VYF; j++) {
      const int g = Y0 + ty + j * TYF + p.sk1;
      const int cl = (g >> 1) - iy0 + NN - 1;
      const V* col = Tb + cl * BZF + tz;
      V v = (g & 1) ? ip_tap<NN, V>([&](int o) { return col[o * BZF]; }) : col[0];
#pragma unroll
      for (int k = 0; k + 1 < QL; k++) q[j][k] = q[j][k + 1];
      q[j][QL - 1] = v;
    }
    // axis-0 pass: step i with c(i) + nn == c emits fine g = 2i and 2i + 1
    const int i = c - 2 * NN + 1 + p.lo0;
    if (c - cbeg >= QL - 1 && i >= ia && i <= ib) {
#pragma unroll
      for (int par = 0; par < 2; par++) {
        const int X = 2 * i + par - p.sk0;
        if (X < X0 || X >= X1) continue;
#pragma unroll
        for (int j = 0; j < VYF; j++) {
          const int y = Y0 + ty + j * TYF, z = Z0 + tz;
          if (y < p.no1 && z < p.no2) {
            V v = par ? ip_tap<NN, V>([&](int o) { return q[j][NN - 1 + o]; }) : q[j][NN - 1];
            const long long o = X * plane_out + (long long)y * p.no2 + z;
            if constexpr (TOTAL) v = vmul(factor, v);
            else if (p.out_scale != S(1)) v = vmul(p.out_scale, v);
            if constexpr (SUB) v = vsub(baseb[o], v);
            stcs(outb + o, v);
          }
        }
      }
    }
  }
}

// Input position u of an axis: element offset (always inside the band) in
// units of the axis stride, whether it holds a value, and its wrap side.
struct TrTap {
  int off;
  int side;
  bool ok;
};
__device__ __forceinline__ TrTap tr_map(int u, int n, int per, int stride) {
  TrTap t;
  t.off = map_axis(u, n, per, t.side, t.ok) * stride;
  return t;
}

// A value where even, the K-tap value of `get` where odd; both are computed
// for nn = 1 (a select, so no lane waits for another's path), the wider taps
// branch.
template <int NN, class V, class Get>
__device__ __forceinline__ V ip_along(int odd, Get get) {
  if constexpr (NN == 1) {
    const V a = get(0), m = ip_tap<NN, V>([&](int o) { return o == 0 ? a : get(odd); });
    V r;
    if constexpr (vt<V>::NC == 2) r = {odd ? m.re : a.re, odd ? m.im : a.im};
    else r = odd ? m : a;
    return r;
  } else {
    return odd ? ip_tap<NN, V>(get) : get(0);
  }
}

// ---------------------------------------------------------------------------
// Two-tap restriction (nn = 1: the multigrid V-cycle, the band preconditioner)
// on large grids.  With three taps per axis a point needs so few neighbours
// that staging them in shared memory costs more than reading them through L1
// (the staged kernel's two barriers per plane and its one plane of prefetch
// kept it at a fifth of the memory rate: 493 us for 32 complex128 bands of
// 96^3): a thread owns one output column and marches along axis 0, carrying
// the in-plane value of the plane that two outputs share.  Per coarse plane it
// makes the in-plane values of two fine planes from 18 independent loads (2.25
// per fine point).  Registers are held to 6 (complex128) or 8 blocks of 128
// threads per SM: with all 18 values in flight per thread (138 registers, one
// block of 256) the same case took 227 us.
// ---------------------------------------------------------------------------
constexpr int kTwoTapNT = 128;
template <class V>
__global__ void __launch_bounds__(kTwoTapNT, sizeof(V) >= 16 ? 6 : 8)
restrict1_kernel(const V* __restrict__ in, V* __restrict__ out,
                 const TrParams<typename vt<V>::S> p) {
  pdl_enter();
  using S = typename vt<V>::S;
  const int plane_out = p.no1 * p.no2, g = blockIdx.x * kTwoTapNT + threadIdx.x;
  if (g >= plane_out) return;
  const int Y = g / p.no2, Z = g - Y * p.no2;
  const int bnd = blockIdx.y / p.nxc, xc = blockIdx.y % p.nxc;
  const int X0 = xc * p.x_chunk, X1 = min(p.no0, X0 + p.x_chunk);
  const V* inb = in + bnd * p.band_in;
  V* outb = out + bnd * p.band_out;
  TrTap ty[3], tz[3];
  bool ok = true, side = false;
#pragma unroll
  for (int k = 0; k < 3; k++) {
    ty[k] = tr_map(2 * Y + k - p.lo1, p.ni1, p.per1, p.ni2);
    tz[k] = tr_map(2 * Z + k - p.lo2, p.ni2, p.per2, 1);
    ok = ok && ty[k].ok && tz[k].ok;
    side = side || ty[k].side >= 0 || tz[k].side >= 0;
  }
  const long long plane_in = (long long)p.ni1 * p.ni2;
  // In-plane value of fine plane f (axis 2 innermost, as the reference).
  auto value = [&](int f) -> V {
    int xs;
    const int x = wrap_plane(f, p.ni0, p.per0, xs);
    if (x < 0) return vzero<V>();
    const V* a = inb + x * plane_in;
    V v[3][3];
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int k = 0; k < 3; k++) v[i][k] = ldro(a + (ty[i].off + tz[k].off));
    if (!ok) {
#pragma unroll
      for (int i = 0; i < 3; i++)
#pragma unroll
        for (int k = 0; k < 3; k++) v[i][k] = value_or_zero(ty[i].ok && tz[k].ok, v[i][k]);
    }
    if constexpr (vt<V>::NC == 2) {
      if (xs >= 0 || side) {
#pragma unroll
        for (int i = 0; i < 3; i++)
#pragma unroll
          for (int k = 0; k < 3; k++) {
            if (xs >= 0) v[i][k] = phase_mul(phase_of(p.P, 0, xs), v[i][k]);
            v[i][k] = side_phase(p.P, 1, ty[i].side, v[i][k]);
            v[i][k] = side_phase(p.P, 2, tz[k].side, v[i][k]);
          }
      }
    }
    return rst_tap<1, V>([&](int oy) {
      return rst_tap<1, V>([&](int oz) { return v[oy + 1][oz + 1]; });
    });
  };
  V prev = value(2 * X0 - p.lo0);
  for (int X = X0; X < X1; X++) {
    const V c = value(2 * X + 1 - p.lo0), next = value(2 * X + 2 - p.lo0);
    V v = rst_tap<1, V>([&](int o) { return o == 0 ? c : (o < 0 ? prev : next); });
    prev = next;
    if (p.out_scale != S(1)) v = vmul(p.out_scale, v);
    const long long o = (long long)X * plane_out + g;
    stcs(outb + o, v);
    if (p.seed) stcs(static_cast<V*>(p.seed) + bnd * p.band_out + o, vmul(p.seed_scale, v));
  }
}

// ---------------------------------------------------------------------------
// Direct forms for small grids (coarse multigrid levels): one thread per
// output point, the three 1-D passes nested in registers in the reference's
// order (axis 2 innermost, then axis 1, then axis 0), neighbours read through
// the L1 cache.  The marching kernels above pay a memory round trip per plane,
// which dominates on grids of a few thousand points.
// ---------------------------------------------------------------------------
template <class LD, class V, class S>
__device__ __forceinline__ V tr_fetch(const V* base, const TrTap& x, const TrTap& y,
                                      const TrTap& z, const TrParams<S>& p) {
  V v = value_or_zero(x.ok && y.ok && z.ok, LD::ld(base + (x.off + y.off + z.off)));
  if constexpr (vt<V>::NC == 2) {
    v = side_phase(p.P, 0, x.side, v);
    v = side_phase(p.P, 1, y.side, v);
    v = side_phase(p.P, 2, z.side, v);
  }
  return v;
}

// rst_tap with the pairs in a loop (not unrolled): the outer axes of the
// wider transfers, whose (2nn + 1)^3 taps would otherwise all be expanded.
template <int NN, class V, class Get>
__device__ __forceinline__ V rst_tap_loop(Get get) {
  using S = typename vt<V>::S;
  if constexpr (NN == 1) {
    return rst_tap<NN, V>(get);
  } else {
    V x = get(0);
#pragma unroll 1
    for (int k = 0; k < NN; k++)
      x = vadd(x, vmul(lagw<NN, S>(k), vadd(get(2 * k + 1), get(-(2 * k + 1)))));
    return vmul(S(0.5), x);
  }
}

// One restricted point at output coordinates (X, Y, Z) of a band (base:
// the band's input), times out_scale; LD is the load policy (common.cuh).
// The axis-2 taps (all 27 taps for nn = 1) are loaded without branches, so
// they are in flight together.
template <class V, int NN, class LD>
__device__ __forceinline__ V restrict_point_at(const V* __restrict__ base, int X, int Y, int Z,
                                               const TrParams<typename vt<V>::S>& p) {
  constexpr int W = 2 * NN - 1;
  // fine centre of each axis: 2i + (2nn-1) - lo
  const int fx = 2 * X + W - p.lo0, fy = 2 * Y + W - p.lo1, fz = 2 * Z + W - p.lo2;
  TrTap tz[2 * NN + 1];  // slot (o + W) / 2 for the odd offsets, 2nn the centre
#pragma unroll
  for (int j = 0; j < 2 * NN; j++) tz[j] = tr_map(fz - W + 2 * j, p.ni2, p.per2, 1);
  tz[2 * NN] = tr_map(fz, p.ni2, p.per2, 1);
  if constexpr (NN == 1) {
    // The loads first (see star_point_at): all 27, or the nine of one plane at a
    // time where 27 values need too many registers (complex128: 166, one block of
    // 256 per SM).
    TrTap ty[3];
#pragma unroll
    for (int k = 0; k < 3; k++) ty[k] = tr_map(fy + k - 1, p.ni1, p.per1, p.ni2);
    auto plane = [&](int ox) -> V {
      const TrTap tx = tr_map(fx + ox, p.ni0, p.per0, p.ni1 * p.ni2);
      V c[3][3];
#pragma unroll
      for (int j = 0; j < 3; j++)
#pragma unroll
        for (int k = 0; k < 3; k++) c[j][k] = tr_fetch<LD>(base, tx, ty[j], tz[k == 1 ? 2 : k >> 1], p);
      return rst_tap<1, V>([&](int oy) {
        return rst_tap<1, V>([&](int oz) { return c[oy + 1][oz + 1]; });
      });
    };
    V below = vzero<V>(), own = vzero<V>(), above = vzero<V>();
    if constexpr (sizeof(V) >= 16) {
#pragma unroll 1
      for (int i = -1; i <= 1; i++) {
        const V v = plane(i);
        if (i < 0) below = v;
        else if (i == 0) own = v;
        else above = v;
      }
    } else {
      below = plane(-1);
      own = plane(0);
      above = plane(1);
    }
    V r = rst_tap<1, V>([&](int o) { return o == 0 ? own : o < 0 ? below : above; });
    if (p.out_scale != typename vt<V>::S(1)) r = vmul(p.out_scale, r);
    return r;
  }
  V v = rst_tap_loop<NN, V>([&](int ox) {
    const TrTap tx = tr_map(fx + ox, p.ni0, p.per0, p.ni1 * p.ni2);
    return rst_tap_loop<NN, V>([&](int oy) {
      const TrTap ty = tr_map(fy + oy, p.ni1, p.per1, p.ni2);
      return rst_tap<NN, V>([&](int oz) {
        return tr_fetch<LD>(base, tx, ty, tz[oz == 0 ? 2 * NN : (oz + W) >> 1], p);
      });
    });
  });
  if (p.out_scale != typename vt<V>::S(1)) v = vmul(p.out_scale, v);
  return v;
}

// Output coordinates of flat index g over all output bands (32-bit arithmetic:
// fewer than 2^31 points per launch) and its band.
template <class S>
__device__ __forceinline__ int tr_split(const TrParams<S>& p, int g, int total, int& X, int& Y,
                                        int& Z, int& rem) {
  const int band = int(p.band_out);
  const int b = total == band ? 0 : g / band;
  rem = g - b * band;
  const int row = rem / p.no2;
  Z = rem - row * p.no2;
  X = row / p.no1;
  Y = row - X * p.no1;
  return b;
}

// One interpolated point at output coordinates (X, Y, Z), times osc
// (SUB: *bo, the base value at that point, minus it).  For nn = 1 the eight
// corner loads are independent (an even axis reads its one point twice).
template <class V, int NN, bool SUB, class LD>
__device__ __forceinline__ V interp_point_at(const V* __restrict__ base, const V* bo, int X, int Y,
                                             int Z, const TrParams<typename vt<V>::S>& p,
                                             typename vt<V>::S osc) {
  // g = f + skip[c][0]; even g: coarse point c(i) = i + nn - 1 - lo, odd: between c(i), c(i)+1
  const int gx = X + p.sk0, gy = Y + p.sk1, gz = Z + p.sk2;
  const int cx = (gx >> 1) + NN - 1 - p.lo0, cy = (gy >> 1) + NN - 1 - p.lo1,
            cz = (gz >> 1) + NN - 1 - p.lo2;
  V b = vzero<V>();
  // bo may be the output itself (in-place correction): a plain load.
  if constexpr (SUB) b = *bo;
  V v = ip_along<NN, V>(gx & 1, [&](int ox) {
    const TrTap tx = tr_map(cx + ox, p.ni0, p.per0, p.ni1 * p.ni2);
    return ip_along<NN, V>(gy & 1, [&](int oy) {
      const TrTap ty = tr_map(cy + oy, p.ni1, p.per1, p.ni2);
      return ip_along<NN, V>(gz & 1, [&](int oz) {
        return tr_fetch<LD>(base, tx, ty, tr_map(cz + oz, p.ni2, p.per2, 1), p);
      });
    });
  });
  if (osc != typename vt<V>::S(1)) v = vmul(osc, v);
  if constexpr (SUB) v = vsub(b, v);
  return v;
}

template <class V, int NN>
__global__ void __launch_bounds__(256)
restrict_direct_kernel(const V* __restrict__ in, V* __restrict__ out,
                       const TrParams<typename vt<V>::S> p, int total) {
  pdl_enter();
  for (long long g = blockIdx.x * 256 + threadIdx.x; g < total; g += gridDim.x * 256) {
    int X, Y, Z, rem;
    const long long b = tr_split(p, int(g), total, X, Y, Z, rem);
    const V v = restrict_point_at<V, NN, LoadRO>(in + b * p.band_in, X, Y, Z, p);
    out[g] = v;
    if (p.seed) static_cast<V*>(p.seed)[g] = vmul(p.seed_scale, v);
  }
}

template <class V, int NN, bool SUB>
__global__ void __launch_bounds__(256)
interp_direct_kernel(const V* __restrict__ in, V* out, const V* base_out,
                     const TrParams<typename vt<V>::S> p, int total) {
  pdl_enter();
  const auto osc = out_factor(p);
  for (long long g = blockIdx.x * 256 + threadIdx.x; g < total; g += gridDim.x * 256) {
    int X, Y, Z, rem;
    const long long b = tr_split(p, int(g), total, X, Y, Z, rem);
    out[g] = interp_point_at<V, NN, SUB, LoadRO>(in + b * p.band_in, SUB ? base_out + g : nullptr,
                                                 X, Y, Z, p, osc);
  }
}

}  // namespace gfd
