// transfer_launch.cuh -- host-side tile selection and template dispatch for the
// transfer kernels.  Included by one translation unit per element type so the
// instantiations compile in parallel.
#pragma once

#include <algorithm>
#include <type_traits>

#include "internal.h"
#include "transfer.cuh"

namespace gfd {

template <class V, int NN>
int restrict_go(const gfd_transformer* tr, const V* in, V* out, int64_t nin,
                       TrParams<typename vt<V>::S>& p, int cps, cudaStream_t s) {
  // Two adjacent coarse rows per thread (16 per CTA) stage fewer halo rows per
  // output row and share axis-1 reads; complex128 keeps one, so two CTAs still
  // fit on an SM.  256 float64 bands of 224^3 -> 112^3, nn = 3: 3080 GB/s.
  // Other shapes, measured with the axis-0 queue this kernel had before (2800-2830
  // for this shape): 28 columns 2580; one coarse row per thread 2270; 32 rows
  // per CTA 2410; 4 rows per thread 2490 (253 registers); three CTAs per SM (80
  // registers, spills) 1740.
  constexpr int BZC = 32, TYC = 8, VYC = sizeof(V) >= 16 ? 1 : 2, BYC = TYC * VYC;
  constexpr int W = 2 * NN - 1;
  constexpr int RY = 2 * BYC - 1 + 2 * W, RZ = 2 * BZC - 1 + 2 * W;
  const size_t smem = (size_t)(2 * RY * rst_row_pitch<V, RZ>() + 2 * RY * BZC) * sizeof(V);
  const int gx = (tr->nout[2] + BZC - 1) / BZC, gy = (tr->nout[1] + BYC - 1) / BYC;
  const int64_t tiles = (int64_t)gx * gy * nin;
  const int64_t target = (int64_t)(cps > 0 ? cps : march_ctas_per_sm()) * num_sms();
  int maxc = std::max(1, tr->nout[0] / 2);
  int nxc = (int)std::min<int64_t>(maxc, std::max<int64_t>(1, (target + tiles - 1) / tiles));
  p.x_chunk = (tr->nout[0] + nxc - 1) / nxc;
  p.nxc = (tr->nout[0] + p.x_chunk - 1) / p.x_chunk;
  auto kern = restrict_kernel<V, NN, BZC, TYC, VYC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(restrict_kernel)");
  const int64_t per_launch = std::max<int64_t>(1, 65535 / p.nxc);
  for (int64_t b0 = 0; b0 < nin; b0 += per_launch) {
    int64_t nb = std::min<int64_t>(per_launch, nin - b0);
    dim3 grid(gx, gy, (unsigned)(nb * p.nxc));
    launch_k(kern, grid, BZC * TYC, smem, s, in + b0 * p.band_in, out + b0 * p.band_out, p);
  }
  return check_launch("restrict_kernel");
}

template <class V, int NN>
int interp_go(const gfd_transformer* tr, const V* in, V* out, const V* base, int64_t nin,
                     TrParams<typename vt<V>::S>& p, int cps, cudaStream_t s) {
  constexpr int BZF = 64, TYF = 4, VYF = 2, BYF = TYF * VYF;
  constexpr int CY = BYF / 2 + 2 * NN, CZ = BZF / 2 + 2 * NN;
  const size_t smem = (size_t)(2 * CY * CZ + 2 * CY * BZF) * sizeof(V);
  const int gx = (tr->nout[2] + BZF - 1) / BZF, gy = (tr->nout[1] + BYF - 1) / BYF;
  const int64_t tiles = (int64_t)gx * gy * nin;
  const int64_t target = (int64_t)(cps > 0 ? cps : march_ctas_per_sm()) * num_sms();
  int maxc = std::max(1, tr->nout[0] / 4);
  int nxc = (int)std::min<int64_t>(maxc, std::max<int64_t>(1, (target + tiles - 1) / tiles));
  p.x_chunk = (tr->nout[0] + nxc - 1) / nxc;
  p.nxc = (tr->nout[0] + p.x_chunk - 1) / p.x_chunk;
  auto kern = base ? interp_kernel<V, NN, BZF, TYF, VYF, true, false>
                   : interp_kernel<V, NN, BZF, TYF, VYF, false, false>;
  if (p.total) {
    if constexpr (std::is_same_v<V, double>) {
      if (base) return set_error(GFD_EINVAL, "a device factor is for plain interpolation");
      kern = interp_kernel<V, NN, BZF, TYF, VYF, false, true>;
    } else {
      return set_error(GFD_EINVAL, "a device factor is for float64");
    }
  }
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return check_cuda(e, "cudaFuncSetAttribute(interp_kernel)");
  const int64_t per_launch = std::max<int64_t>(1, 65535 / p.nxc);
  for (int64_t b0 = 0; b0 < nin; b0 += per_launch) {
    int64_t nb = std::min<int64_t>(per_launch, nin - b0);
    dim3 grid(gx, gy, (unsigned)(nb * p.nxc));
    launch_k(kern, grid, BZF * TYF, smem, s, in + b0 * p.band_in, out + b0 * p.band_out,
                                       base ? base + b0 * p.band_out : nullptr, p);
  }
  return check_launch("interp_kernel");
}

// Two-tap restriction past the one-thread-per-point limit: output planes in
// blocks of 128 columns, axis 0 cut into chunks of at least 4 output planes
// until about 16 blocks per SM are in flight.
template <class V>
int restrict1_go(const gfd_transformer* tr, const V* in, V* out, int64_t nin,
                 TrParams<typename vt<V>::S>& p, int cps, cudaStream_t s) {
  const int gx = (tr->nout[1] * tr->nout[2] + kTwoTapNT - 1) / kTwoTapNT;
  const int64_t tiles = (int64_t)gx * nin;
  const int64_t target = 4LL * (cps > 0 ? cps : march_ctas_per_sm()) * num_sms();
  const int maxc = std::max(1, tr->nout[0] / 4);
  const int nxc = (int)std::min<int64_t>(maxc, std::max<int64_t>(1, (target + tiles - 1) / tiles));
  p.x_chunk = (tr->nout[0] + nxc - 1) / nxc;
  p.nxc = (tr->nout[0] + p.x_chunk - 1) / p.x_chunk;
  const int64_t per_launch = std::max<int64_t>(1, 65535 / p.nxc);
  V* seed = static_cast<V*>(p.seed);
  for (int64_t b0 = 0; b0 < nin; b0 += per_launch) {
    const int64_t nb = std::min<int64_t>(per_launch, nin - b0);
    p.seed = seed ? seed + b0 * p.band_out : nullptr;
    launch_k(restrict1_kernel<V>, dim3(gx, (unsigned)(nb * p.nxc)), kTwoTapNT, 0, s,
             in + b0 * p.band_in, out + b0 * p.band_out, p);
  }
  return check_launch("restrict1_kernel");
}

// Outputs (all bands) up to direct_max_points() use the one-thread-per-point
// forms.
template <class V, int NN>
int transfer_direct_go(const gfd_transformer* tr, const V* in, V* out, const V* base, int64_t nin,
                       TrParams<typename vt<V>::S> p, cudaStream_t s) {
  const int64_t most = std::max<int64_t>(1, 2000000000LL / p.band_out);
  V* seed = static_cast<V*>(p.seed);
  for (int64_t b0 = 0; b0 < nin; b0 += most) {
    const int total = int(std::min<int64_t>(most, nin - b0) * p.band_out);
    const long long b = (total + 255) / 256, cap = 8LL * num_sms();
    const int blocks = int(b < 1 ? 1 : (b > cap ? cap : b));
    const V* a = in + b0 * p.band_in;
    V* o = out + b0 * p.band_out;
    p.seed = seed ? seed + b0 * p.band_out : nullptr;
    if (!tr->interpolate)
      launch_k(restrict_direct_kernel<V, NN>, blocks, 256, 0, s, a, o, p, total);
    else if (base)
      launch_k(interp_direct_kernel<V, NN, true>, blocks, 256, 0, s, a, o, base + b0 * p.band_out,
               p, total);
    else
      launch_k(interp_direct_kernel<V, NN, false>, blocks, 256, 0, s, a, o, (const V*)nullptr, p,
               total);
  }
  return check_launch("transfer_direct_kernel");
}

template <class V>
int tr_typed(const gfd_transformer* tr, const void* in, void* out, const void* base_v,
             int64_t nin, const double* ph, cudaStream_t s, void* seed, double seed_scale,
             double out_scale, const double* total, double target) {
  using S = typename vt<V>::S;
  TrParams<S> p;
  tr_params(tr, ph, seed, seed_scale, out_scale, p);
  p.total = total;
  p.target = target;
  if (seed && tr->interpolate) return set_error(GFD_EINVAL, "seeded form is for restriction only");
  const V* vin = static_cast<const V*>(in);
  V* vout = static_cast<V*>(out);
  const V* base = static_cast<const V*>(base_v);
  if (base && !tr->interpolate)
    return set_error(GFD_EINVAL, "subtracting form is for interpolation only");
  TunePlan plan;
  const bool tuned = tune_lookup(tr_tune_key(tr, dtype_of<V>(), nin), &plan);
  const int cps = tuned ? plan.cps : 0;
  // the one-thread-per-point forms index a band with 32 bits
  const bool small = p.band_in < 2000000000LL && p.band_out < 2000000000LL;
  if (small && (tuned ? plan.path == PLAN_DIRECT : p.band_out * nin <= direct_max_points())) {
    switch (tr->nn) {
      case 1: return transfer_direct_go<V, 1>(tr, vin, vout, base, nin, p, s);
      case 2: return transfer_direct_go<V, 2>(tr, vin, vout, base, nin, p, s);
      case 3: return transfer_direct_go<V, 3>(tr, vin, vout, base, nin, p, s);
      case 4: return transfer_direct_go<V, 4>(tr, vin, vout, base, nin, p, s);
    }
  }
  if (tr->interpolate) {
    switch (tr->nn) {
      case 1: return interp_go<V, 1>(tr, vin, vout, base, nin, p, cps, s);
      case 2: return interp_go<V, 2>(tr, vin, vout, base, nin, p, cps, s);
      case 3: return interp_go<V, 3>(tr, vin, vout, base, nin, p, cps, s);
      case 4: return interp_go<V, 4>(tr, vin, vout, base, nin, p, cps, s);
    }
  } else {
    if (base) return set_error(GFD_EINVAL, "subtracting form is for interpolation only");
    switch (tr->nn) {
      case 1: return restrict1_go<V>(tr, vin, vout, nin, p, cps, s);
      case 2: return restrict_go<V, 2>(tr, vin, vout, nin, p, cps, s);
      case 3: return restrict_go<V, 3>(tr, vin, vout, nin, p, cps, s);
      case 4: return restrict_go<V, 4>(tr, vin, vout, nin, p, cps, s);
    }
  }
  return set_error(GFD_EINVAL, "k must be 2, 4, 6 or 8");
}

}  // namespace gfd

// One of these per element type, defined in transfer_<type>.cu.
#define GFD_DECLARE_TRANSFER_ENTRY(NAME)                                                      \
  namespace gfd {                                                                             \
  int transfer_##NAME(const gfd_transformer*, const void*, void*, const void*, int64_t,       \
                      const double*, cudaStream_t, void*, double, double, const double*,      \
                      double);                                                                \
  }
