// transformer.cu -- gfd_transformer_*: the _gpaw.Transformer replacement
// (c/transformers.c:222-265 constructor, :127-185 apply).
#include <new>
#include <string>

#include "common.cuh"
#include "internal.h"
#include "transfer_launch.cuh"

GFD_DECLARE_TRANSFER_ENTRY(f64)
GFD_DECLARE_TRANSFER_ENTRY(f32)
GFD_DECLARE_TRANSFER_ENTRY(c128)
GFD_DECLARE_TRANSFER_ENTRY(c64)

namespace gfd {

int tr_launch_ex(const gfd_transformer* tr, int dtype, const void* in, void* out,
                 const void* base, int64_t nin, const double* phases, double out_scale,
                 void* seed, double seed_scale, cudaStream_t s, const double* total,
                 double target) {
  if (nin <= 0) return GFD_OK;
  switch (dtype) {
    case GFD_FLOAT64:
      return transfer_f64(tr, in, out, base, nin, phases, s, seed, seed_scale, out_scale, total,
                          target);
    case GFD_FLOAT32:
      return transfer_f32(tr, in, out, base, nin, phases, s, seed, seed_scale, out_scale, total,
                          target);
    case GFD_COMPLEX128:
      return transfer_c128(tr, in, out, base, nin, phases, s, seed, seed_scale, out_scale, total,
                          target);
    case GFD_COMPLEX64:
      return transfer_c64(tr, in, out, base, nin, phases, s, seed, seed_scale, out_scale, total,
                          target);
  }
  return set_error(GFD_EINVAL, "unknown dtype");
}

void lagrange_weights(int nn, double w[4]) {
  for (int k = 0; k < nn; k++)
    w[k] = nn == 1   ? lagw<1, double>(k)
           : nn == 2 ? lagw<2, double>(k)
           : nn == 3 ? lagw<3, double>(k)
                     : lagw<4, double>(k);
}

int tr_launch_sub(const gfd_transformer* tr, int dtype, const void* in, void* out,
                  const void* base, int64_t nin, const double* phases, cudaStream_t s) {
  return tr_launch_ex(tr, dtype, in, out, base, nin, phases, 1.0, nullptr, 0.0, s);
}

int tr_launch_seed(const gfd_transformer* tr, int dtype, const void* in, void* out, void* seed,
                   double seed_scale, cudaStream_t s) {
  return tr_launch_ex(tr, dtype, in, out, nullptr, 1, nullptr, 1.0, seed, seed_scale, s);
}

int tr_launch(const gfd_transformer* tr, int dtype, const void* in, void* out, int64_t nin,
              const double* phases, cudaStream_t s) {
  return tr_launch_sub(tr, dtype, in, out, nullptr, nin, phases, s);
}

}  // namespace gfd

using namespace gfd;

extern "C" int gfd_transformer_create(const int64_t size_in[3], const int64_t size_out[3], int k,
                                      const int64_t pad[6], const int64_t npad[6],
                                      const int64_t skip[6], const int64_t neighbors[6], int real,
                                      int interpolate, gfd_transformer** out) {
  if (!out) return set_error(GFD_EINVAL, "null output handle");
  *out = nullptr;
  if (!size_in || !size_out || !pad || !npad || !skip || !neighbors)
    return set_error(GFD_EINVAL, "null array argument");
  if (k != 2 && k != 4 && k != 6 && k != 8) return set_error(GFD_EINVAL, "k must be 2, 4, 6 or 8");
  gfd_transformer* tr = new (std::nothrow) gfd_transformer();
  if (!tr) return set_error(GFD_ENOMEM, "host allocation failed");
  tr->k = k;
  tr->nn = k / 2;
  tr->real = real ? 1 : 0;
  tr->interpolate = interpolate ? 1 : 0;
  for (int a = 0; a < 3; a++) {
    tr->nin[a] = (int)size_in[a];
    tr->nout[a] = (int)size_out[a];
    if (size_in[a] < 1 || size_out[a] < 1 || size_in[a] > (1 << 20) || size_out[a] > (1 << 20)) {
      delete tr;
      return set_error(GFD_EINVAL, "grid size out of range");
    }
    for (int d = 0; d < 2; d++) {
      if (pad[2 * a + d] < 0 || pad[2 * a + d] > 64 || skip[2 * a + d] < 0 || skip[2 * a + d] > 1) {
        delete tr;
        return set_error(GFD_EINVAL, "padding or skip out of range");
      }
      tr->pad[a][d] = (int)pad[2 * a + d];
      tr->skip[a][d] = interpolate ? (int)skip[2 * a + d] : 0;
    }
    int64_t lo = neighbors[2 * a], hi = neighbors[2 * a + 1];
    if (!((lo == 0 && hi == 0) || (lo == -1 && hi == -1))) {
      delete tr;
      return set_error(GFD_EUNSUPPORTED,
                       "neighbors must be 0 (periodic, this domain) or -1 (zero boundary); "
                       "domain decomposition is not provided");
    }
    tr->per[a] = lo == 0;
    if (tr->per[a] && (tr->pad[a][0] > tr->nin[a] || tr->pad[a][1] > tr->nin[a])) {
      delete tr;
      return set_error(GFD_EINVAL, "periodic axis has fewer points than the halo");
    }
    // Output size implied by the padding (c/bmgs/restrict.c:150-152,
    // c/bmgs/interpolate.c:158-167).
    int64_t s = size_in[a] + pad[2 * a] + pad[2 * a + 1];
    int64_t expect = interpolate
                         ? 2 * (s - (k - 1) + tr->skip[a][1]) - tr->skip[a][0] - tr->skip[a][1]
                         : (s - (2 * k - 3)) / 2;
    if (!interpolate && ((s - (2 * k - 3)) < 0 || (s - (2 * k - 3)) % 2)) expect = -1;
    if (expect != size_out[a]) {
      delete tr;
      return set_error(GFD_EINVAL, "size_out does not match size_in and the padding on axis " +
                                       std::to_string(a));
    }
  }
  *out = tr;
  return GFD_OK;
}

extern "C" int gfd_transformer_destroy(gfd_transformer* tr) {
  delete tr;
  return GFD_OK;
}

extern "C" int gfd_transformer_apply(gfd_transformer* tr, int dtype, const void* in, void* out,
                                     int64_t nin, const double* phases, void* stream) {
  if (!tr) return set_error(GFD_EINVAL, "null transformer");
  if (dtype < GFD_FLOAT64 || dtype > GFD_COMPLEX64) return set_error(GFD_EINVAL, "unknown dtype");
  if (tr->real != !dtype_is_complex(dtype))
    return set_error(GFD_EINVAL, tr->real ? "transformer was built for real arrays"
                                          : "transformer was built for complex arrays");
  if (nin < 0) return set_error(GFD_EINVAL, "negative band count");
  if (nin == 0) return GFD_OK;
  if (!in || !out) return set_error(GFD_EINVAL, "null array pointer");
  return tr_launch(tr, dtype, in, out, nin, phases, static_cast<cudaStream_t>(stream));
}
