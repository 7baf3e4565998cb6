// scratch.cu -- device memory for the length of one call.
//
// cudaMalloc and cudaFree took 0.4-0.57 and 0.3-0.43 ms each on a B200 host (the
// free also waits for the device), which was most of the time of the calls that
// work on host buffers: a mesh's distance field, a snapshot's surface, the
// network's forward and gradient passes.  They now take their memory from one
// stream-ordered pool per device (2 us), which keeps at most kPoolKeep bytes
// that no call holds: the driver gives the rest back at the next
// synchronisation.  The pool orders reuse between streams and threads itself.
#include <cuda_runtime.h>

#include <mutex>

#include "host_internal.h"
#include "scratch.cuh"

namespace sphpc {

namespace {

constexpr size_t kPoolKeep = (size_t)64 << 20;
constexpr int kMaxDevices = 64;

// The pool of a device and the unique id of the context that it was made in (a
// cudaDeviceReset ends that context and the pool with it).
struct DevicePool {
  cudaMemPool_t pool = nullptr;
  unsigned long long ctx = 0;
};
std::mutex g_mu;
DevicePool g_pool[kMaxDevices];

// The current device's pool, or null (plain allocations then take its place).
cudaMemPool_t device_pool() {
  int dev = 0;
  unsigned long long ctx = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices ||
      cudaFree(nullptr) != cudaSuccess || !current_context_id(&ctx)) {
    cudaGetLastError();
    return nullptr;
  }
  std::lock_guard<std::mutex> lk(g_mu);
  DevicePool& d = g_pool[dev];
  if (d.pool && d.ctx == ctx) return d.pool;
  d = DevicePool{};
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  unsigned long long keep = kPoolKeep;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess ||
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  d.pool = pool;
  d.ctx = ctx;
  return pool;
}

}  // namespace

cudaError_t CallScratch::take(size_t bytes, cudaStream_t stream) {
  stream_ = stream;
  if (bytes == 0) bytes = 1;
  if (cudaMemPool_t pool = device_pool()) {
    if (cudaMallocFromPoolAsync(&p_, bytes, pool, stream) == cudaSuccess) {
      pooled_ = true;
      return cudaSuccess;
    }
    cudaGetLastError();
    p_ = nullptr;
  }
  return cudaMalloc(&p_, bytes);
}

CallScratch::~CallScratch() {
  if (!p_) return;
  if (pooled_) cudaFreeAsync(p_, stream_);
  else cudaFree(p_);
}

}  // namespace sphpc
