// hm_memory.cu -- the library's device memory: cudaMalloc for large blocks, a
// bounded pool per device for the small ones (hm_internal.h).
#include <mutex>

#include "hm_internal.h"

namespace hm {
namespace {

constexpr int kMaxDevices = 64;

struct DevicePool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the allocations of long-lived blocks
};
std::mutex g_mu;
DevicePool g_pools[kMaxDevices];

// The current device's pool, made on its first use.
cudaError_t device_pool(DevicePool** out, int* dev) {
  cudaError_t e = cudaGetDevice(dev);
  if (e != cudaSuccess) return e;
  if (*dev >= kMaxDevices) return cudaErrorInvalidDevice;
  DevicePool& P = g_pools[*dev];
  std::lock_guard<std::mutex> lock(g_mu);
  if (!P.pool) {
    cudaMemPoolProps pr{};
    pr.allocType = cudaMemAllocationTypePinned;
    pr.location.type = cudaMemLocationTypeDevice;
    pr.location.id = *dev;
    cudaMemPool_t pool = nullptr;
    if ((e = cudaMemPoolCreate(&pool, &pr)) != cudaSuccess) return e;
    unsigned long long keep = kPoolKeep;
    if ((e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess ||
        (e = cudaStreamCreateWithFlags(&P.stream, cudaStreamNonBlocking)) != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    P.pool = pool;
  }
  *out = &P;
  return cudaSuccess;
}

// Makes `dev` current for a scope (a block may be released while another
// device is).
struct OnDevice {
  int was = -1;
  explicit OnDevice(int dev) {
    int cur = dev;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != dev) {
      was = cur;
      cudaSetDevice(dev);
    }
  }
  ~OnDevice() {
    if (was >= 0) cudaSetDevice(was);
  }
};

// What the pool keeps goes back to the device.
cudaError_t give_back(DevicePool* P) {
  const cudaError_t e = cudaDeviceSynchronize();  // releases in flight count as kept only then
  return e != cudaSuccess ? e : cudaMemPoolTrimTo(P->pool, 0);
}

cudaError_t pool_alloc(DevicePool* P, void** p, size_t bytes, cudaStream_t s) {
  cudaError_t e = cudaMallocFromPoolAsync(p, bytes, P->pool, s);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back(P);
    e = cudaMallocFromPoolAsync(p, bytes, P->pool, s);
  }
  return e;
}

cudaError_t large_alloc(DevicePool* P, void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    give_back(P);
    e = cudaMalloc(p, bytes);
  }
  return e;
}

}  // namespace

cudaError_t dev_alloc(void** p, size_t bytes, int* dev) {
  DevicePool* P = nullptr;
  cudaError_t e = device_pool(&P, dev);
  if (e != cudaSuccess) return e;
  if (bytes >= kPoolMax) return large_alloc(P, p, bytes);
  if ((e = pool_alloc(P, p, bytes, P->stream)) != cudaSuccess) return e;
  // a block that another stream released may still be in use there: the
  // allocation completes on the pool's stream once it is not
  return cudaStreamSynchronize(P->stream);
}

cudaError_t dev_alloc_async(void** p, size_t bytes, cudaStream_t s, int* dev) {
  DevicePool* P = nullptr;
  const cudaError_t e = device_pool(&P, dev);
  if (e != cudaSuccess) return e;
  return bytes >= kPoolMax ? large_alloc(P, p, bytes) : pool_alloc(P, p, bytes, s);
}

void dev_free(void* p, size_t bytes, int dev) {
  if (bytes >= kPoolMax) {
    cudaFree(p);
    return;
  }
  OnDevice on(dev);
  cudaDeviceSynchronize();  // as cudaFree: the block may be in use on any stream
  cudaFreeAsync(p, g_pools[dev].stream);
}

void dev_free_async(void* p, size_t bytes, cudaStream_t s, int dev) {
  OnDevice on(dev);
  if (bytes >= kPoolMax)
    cudaFree(p);
  else
    cudaFreeAsync(p, s);
}

}  // namespace hm

extern "C" hm_status hm_release_memory(void) {
  using namespace hm;
  DevicePool* P = nullptr;
  int dev = 0;
  HM_CUDA(device_pool(&P, &dev));
  HM_CUDA(give_back(P));
  return HM_OK;
}
