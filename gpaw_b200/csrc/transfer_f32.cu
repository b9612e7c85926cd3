// Transfer kernels instantiated for one element type (float).
#include "transfer_launch.cuh"

namespace gfd {

int transfer_f32(const gfd_transformer* tr, const void* in, void* out, const void* base,
                int64_t nin, const double* ph, cudaStream_t s, void* seed, double seed_scale,
                double out_scale, const double* total, double target) {
  return tr_typed<float>(tr, in, out, base, nin, ph, s, seed, seed_scale, out_scale, total, target);
}

}  // namespace gfd
