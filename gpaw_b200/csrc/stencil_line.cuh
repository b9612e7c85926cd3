// stencil_line.cuh -- stencils along a single axis (Gradient on orthorhombic
// cells, gpaw/fd_operators.py:123-144): out[g] = c0 a[g] + sum_k c_k a[g + k e].
//
// Run through star_kernel such an operator stages the halos of all three axes
// and multiplies by 4R zero weights.  Here only the operator's own axis is
// touched, without shared memory:
//
//  * axes 0 and 1 (line_march_kernel): a thread marches along the axis at a
//    fixed position of the contiguous rest, keeping the last 2R values in
//    registers, kLineBlock new values loaded at a time: one load and one store
//    per point, both coalesced.
//  * axis 2 (line_row_kernel): a thread keeps one column and walks over rows;
//    its 2R + 1 neighbours' offsets and wrap sides are worked out once and its
//    loads hit the same L1 lines as its neighbours'.
#pragma once

#include "common.cuh"
#include "stencil.cuh"

namespace gfd {

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

template <class V, int R>
__global__ void __launch_bounds__(256)
line_march_kernel(const V* __restrict__ in, V* __restrict__ out,
                  const LineParams<typename vt<V>::S> p) {
  pdl_enter();
  constexpr int B = kLineBlock, W = B + 2 * R;
  const long long i = blockIdx.x * 256LL + threadIdx.x;
  if (i >= p.inner) return;
  const int c = blockIdx.y;
  const int x0 = c * p.chunk, x1 = min(p.n, x0 + p.chunk);
  for (long long o = blockIdx.z; o < p.outer; o += gridDim.z) {
    const V* a = in + o * p.n * p.inner + i;
    V* b = out + o * p.n * p.inner + i;
    auto load = [&](int u) -> V {
      int side;
      const int j = wrap_plane(u, p.n, p.per, side);
      if (j < 0) return vzero<V>();
      V v = ldro(a + j * p.inner);
      if constexpr (vt<V>::NC == 2) {
        if (side >= 0) v = phase_mul(p.ph[side], v);
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
        V s = vmul(p.w[kMaxR], win[j + R]);
#pragma unroll
        for (int k = -R; k <= R; k++)
          if (k != 0) madd(s, p.w[kMaxR + k], win[j + R + k]);
        if (x + j < x1) stcs(b + (x + j) * p.inner, s);
      }
#pragma unroll
      for (int k = 0; k < 2 * R; k++) win[k] = win[k + B];
    }
  }
}

// blockDim.x threads = rows_per_pass rows of n columns (bz of them per block
// column when a row is longer than the block).
template <class V, int R>
__global__ void __launch_bounds__(256)
line_row_kernel(const V* __restrict__ in, V* __restrict__ out,
                const LineParams<typename vt<V>::S> p, int bz, int rows_per_pass, int passes) {
  pdl_enter();
  const int rz = threadIdx.x / bz, z = blockIdx.y * bz + threadIdx.x - rz * bz;
  if (rz >= rows_per_pass || z >= p.n) return;
  int off[2 * R + 1];  // neighbour column minus z
  unsigned ok = 0, low = 0, high = 0;
#pragma unroll
  for (int k = -R; k <= R; k++) {
    int side;
    bool in_range;
    off[k + R] = map_axis(z + k, p.n, p.per, side, in_range) - z;
    if (!in_range) off[k + R] = 0;
    ok |= unsigned(in_range) << (k + R);
    low |= unsigned(side == 1) << (k + R);
    high |= unsigned(side == 0) << (k + R);
  }
  const long long r0 = (long long)blockIdx.x * rows_per_pass * passes + rz;
#pragma unroll 2
  for (int q = 0; q < passes; q++) {
    const long long r = r0 + (long long)q * rows_per_pass;
    if (r >= p.inner) break;
    const V* a = in + r * p.n + z;
    V v[2 * R + 1];
#pragma unroll
    for (int k = 0; k <= 2 * R; k++) v[k] = ldro(a + off[k]);
    if (ok != (1u << (2 * R + 1)) - 1u) {
#pragma unroll
      for (int k = 0; k <= 2 * R; k++) v[k] = value_or_zero(ok >> k & 1u, v[k]);
    }
    if constexpr (vt<V>::NC == 2) {
      if (low | high) {
#pragma unroll
        for (int k = 0; k <= 2 * R; k++) {
          if (low >> k & 1u) v[k] = phase_mul(p.ph[1], v[k]);
          if (high >> k & 1u) v[k] = phase_mul(p.ph[0], v[k]);
        }
      }
    }
    V s = vmul(p.w[kMaxR], v[R]);
#pragma unroll
    for (int k = -R; k <= R; k++)
      if (k != 0) madd(s, p.w[kMaxR + k], v[R + k]);
    stcs(out + r * p.n + z, s);
  }
}

}  // namespace gfd
