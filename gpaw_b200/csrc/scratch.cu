// scratch.cu -- stream-ordered device scratch for the length of one call.
#include <cuda.h>

#include <mutex>

#include "common.cuh"
#include "internal.h"

namespace gfd {

namespace {
// A driver function through the runtime, so the library needs no link-time
// dependency on libcuda.
void* driver_fn(const char* name) {
  void* f = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return f;
}
}  // namespace

// The id, not the handle, tells contexts apart: a primary context that was
// reset and bound again has its old handle and a new id.
unsigned long long context_id() {
  using GetCurrent = CUresult (*)(CUcontext*);
  using GetId = CUresult (*)(CUcontext, unsigned long long*);
  static const auto get_current = reinterpret_cast<GetCurrent>(driver_fn("cuCtxGetCurrent"));
  static const auto get_id = reinterpret_cast<GetId>(driver_fn("cuCtxGetId"));
  if (!get_current || !get_id) return 0;
  for (int attempt = 0; attempt < 2; attempt++) {
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) == CUDA_SUCCESS && ctx && get_id(ctx, &id) == CUDA_SUCCESS) return id;
    // None bound on this thread, or a reset one: bind the device's primary one.
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) break;
  }
  cudaGetLastError();
  return 0;
}

// From a pool of the library's own in each device's context that keeps up to
// kScratchKeep bytes across synchronisations.  The default pool gives its
// memory back whenever the device runs idle, so a call of 40 us paid for
// mapping it again, about 400 us.  A device reset takes the pool with it; the
// next call, in another context, makes a new one.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  static std::mutex mu;
  struct Pool {
    unsigned long long ctx = 0;
    cudaMemPool_t pool = nullptr;
  };
  static Pool pools[64];
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  const unsigned long long ctx = context_id();
  if (ctx == 0) return cudaErrorInvalidResourceHandle;
  cudaMemPool_t pool;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!pools[dev].pool || pools[dev].ctx != ctx) {
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
      pools[dev] = {ctx, np};
    }
    pool = pools[dev].pool;
  }
  return cudaMallocFromPoolAsync(p, bytes, pool, s);
}

}  // namespace gfd
