// stencil_line.cuh -- stencils along a single axis (Gradient on orthorhombic
// cells, gpaw/fd_operators.py:123-144): out[g] = c0 a[g] + sum_k c_k a[g + k e].
//
// Run through star_kernel such an operator stages the halos of all three axes
// and multiplies by 4R zero weights.  Here only the operator's own axis is
// touched:
//
//  * axes 0 and 1 (line_march_kernel): a thread marches along the axis at a
//    fixed position of the contiguous rest, keeping the last 2R values in
//    registers, several new values loaded at a time: one load and one store
//    per point, both coalesced.
//  * axis 2 (line_row_kernel): a block stages whole rows with their wrapped or
//    zero ends in shared memory; rows past 1024 points stay with star_kernel.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace gfd {

// Values loaded at a time (8: 171 us against 157, 200 against 180).
constexpr int kLineBlock = 4;

template <class S>
struct LineParams {
  int n;             // points along the axis
  int per;
  long long inner;   // contiguous points per step of the axis (axis 2: rows)
  long long outer;   // independent lines' outer count (axis 2: 1)
  int chunk, nch;    // axes 0 and 1: outputs per thread and chunks per line
  S w[2 * kMaxR + 1];  // weight of offset k at kMaxR + k, the centre included
  cplx<S> ph[2];     // Bloch phases of the axis (high halo, low halo)
};

// The centre's term; nothing (not zero times the value) where it has no weight.
template <class V, class S>
__device__ __forceinline__ V centre(const LineParams<S>& p, const V& v) {
  return value_or_zero(p.w[kMaxR] != S(0), vmul(p.w[kMaxR], v));
}

template <class V, int R>
__global__ void __launch_bounds__(256)
line_march_kernel(const V* __restrict__ in, V* __restrict__ out,
                  const LineParams<typename vt<V>::S> p) {
  pdl_enter();
  constexpr int B = kLineBlock, W = B + 2 * R;
  const long long g = blockIdx.x * 256LL + threadIdx.x, lines = p.inner * p.outer;
  if (g >= lines) return;
  // Lanes run over the lines as they lie in memory, past the end of one step of
  // the axis into the next: no lane idles where p.inner is not a multiple of 32.
  const long long o = lines <= 0x7fffffff ? int(g) / int(p.inner) : g / p.inner;
  const int c = blockIdx.y;
  const int x0 = c * p.chunk, x1 = min(p.n, x0 + p.chunk);
  const long long at = o * (p.n - 1) * p.inner + g;  // o whole lines and g - o inner
  const V* a = in + at;
  V* b = out + at;
  auto load = [&](int u) -> V {
    int side;
    const int j = wrap_plane(u, p.n, p.per, side);
    if (j < 0) return vzero<V>();
    V v = ldro(a + j * p.inner);
    if constexpr (vt<V>::NC == 2) {
      // not p.ph[side]: an index of the parameters copies them to local memory
      if (side >= 0) v = phase_mul(side == 1 ? p.ph[1] : p.ph[0], v);
    }
    return v;
  };
  V win[W];
#pragma unroll
  for (int k = 0; k < 2 * R; k++) win[k] = load(x0 - R + k);
  for (int x = x0; x < x1; x += B) {
#pragma unroll
    for (int k = 0; k < B; k++) win[2 * R + k] = x + R + k < x1 + R ? load(x + R + k) : vzero<V>();
#pragma unroll
    for (int j = 0; j < B; j++) {
      V s = centre(p, win[j + R]);
#pragma unroll
      for (int k = -R; k <= R; k++)
        if (k != 0) madd(s, p.w[kMaxR + k], win[j + R + k]);
      if (x + j < x1) stcs(b + (x + j) * p.inner, s);
    }
#pragma unroll
    for (int k = 0; k < 2 * R; k++) win[k] = win[k + B];
  }
}

// A block of rows x n threads takes `passes` groups of rows (n <= 1024): all
// their values are loaded first, then staged with the R wrapped (or zero)
// cells on either side, so the 2R + 1 neighbours are shared-memory reads at
// fixed offsets.  (Reading them through L1 took 175 instructions per point for
// the edges' index arithmetic: 298 us against 172 us for 64 complex64 bands of
// 120 x 64 x 80.)
constexpr int kLinePasses = 8;
template <class V, int R>
__global__ void __launch_bounds__(1024)
line_row_kernel(const V* __restrict__ in, V* __restrict__ out,
                const LineParams<typename vt<V>::S> p, int rows, int passes) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  V* tile = reinterpret_cast<V*>(smem_raw);  // [passes * rows][n + 2R]
  const int n = p.n, pitch = n + 2 * R;
  const int rz = threadIdx.x / n, z = threadIdx.x - rz * n;
  const long long r0 = (long long)blockIdx.x * rows * passes + rz;
  V v[kLinePasses];
#pragma unroll
  for (int q = 0; q < kLinePasses; q++) {
    const long long r = r0 + (long long)q * rows;
    v[q] = q < passes && r < p.inner ? ldro(in + r * n + z) : vzero<V>();
  }
#pragma unroll
  for (int q = 0; q < kLinePasses; q++) {
    if (q >= passes) break;
    V* row = tile + (q * rows + rz) * pitch;
    row[R + z] = v[q];
    if (p.per) {
      if (z >= n - R) row[z - (n - R)] = phase_mul(p.ph[1], v[q]);
      if (z < R) row[R + n + z] = phase_mul(p.ph[0], v[q]);
    } else {
      for (int h = z; h < R; h += n) row[h] = row[R + n + h] = vzero<V>();
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kLinePasses; q++) {
    if (q >= passes) break;
    const long long r = r0 + (long long)q * rows;
    if (r >= p.inner) break;
    const V* row = tile + (q * rows + rz) * pitch + R + z;
    V s = centre(p, row[0]);
#pragma unroll
    for (int k = -R; k <= R; k++)
      if (k != 0) madd(s, p.w[kMaxR + k], row[k]);
    stcs(out + r * n + z, s);
  }
}

}  // namespace gfd
