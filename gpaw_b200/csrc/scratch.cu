// scratch.cu -- stream-ordered device scratch for the length of one call.
#include <mutex>

#include "common.cuh"
#include "internal.h"

namespace gfd {

// From a pool of the library's own on each device that keeps up to
// kScratchKeep bytes across synchronisations.  The default pool gives its
// memory back whenever the device runs idle, so a call of 40 us paid for
// mapping it again, about 400 us.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  cudaMemPool_t pool;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev]) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.handleTypes = cudaMemHandleTypeNone;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      cudaMemPool_t np = nullptr;
      if ((e = cudaMemPoolCreate(&np, &props)) != cudaSuccess) return e;
      uint64_t keep = kScratchKeep;
      e = cudaMemPoolSetAttribute(np, cudaMemPoolAttrReleaseThreshold, &keep);
      if (e != cudaSuccess) {
        cudaMemPoolDestroy(np);
        return e;
      }
      pools[dev] = np;
    }
    pool = pools[dev];
  }
  return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

}  // namespace gfd
