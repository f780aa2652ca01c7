// hm_memory.cu -- the library's device memory: cudaMalloc for large blocks, a
// bounded pool per device for the small ones (hm_internal.h).
#include <chrono>
#include <mutex>
#include <vector>

#include "hm_internal.h"

namespace hm {
namespace {

constexpr int kMaxDevices = 64;

using Block = FreeTogether::Block;

struct DevicePool {
  cudaMemPool_t pool = nullptr;
  cudaStream_t stream = nullptr;  // orders the allocations of long-lived blocks
  std::vector<void*> tokens;      // see wait_device
  std::vector<Block> parked;      // released, but not yet known to be out of use
  std::chrono::steady_clock::time_point asked;  // dev_settle's last question, and what was idle then
  unsigned long long idle = 0;
};
std::mutex g_mu;
DevicePool g_pools[kMaxDevices];

// Lets this thread allocate and release while a stream is being captured, by
// itself or by another thread: neither touches what is captured.
struct WhileCapturing {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  WhileCapturing() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~WhileCapturing() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

constexpr size_t kToken = 256;

// The current device's pool, made on its first use.
cudaError_t device_pool(DevicePool** out, int* dev) {
  cudaError_t e = cudaGetDevice(dev);
  if (e != cudaSuccess) return e;
  if (*dev >= kMaxDevices) return cudaErrorInvalidDevice;
  DevicePool& P = g_pools[*dev];
  WhileCapturing guard;
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
    // two tokens: one stays while the other is released, so that the driver's
    // block that holds them stays mapped
    for (int i = 0; i < 2; ++i) {
      void* t = nullptr;
      if (cudaMalloc(&t, kToken) == cudaSuccess) P.tokens.push_back(t);
    }
    cudaGetLastError();
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

// Waits for the device's work on every stream, graphs in flight included, by
// releasing a small cudaMalloc block: cudaFree synchronises (30.0 ms behind a
// 30 ms kernel on a non-blocking stream) and may be called while streams are
// being captured.  cudaDeviceSynchronize may not: whichever thread captures and
// in whatever mode, it fails and invalidates that capture.  On an idle device
// 3.5 us, the next token included, against 1.5.
cudaError_t wait_device(DevicePool* P) {
  WhileCapturing guard;
  void* t = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!P->tokens.empty()) {
      t = P->tokens.back();
      P->tokens.pop_back();
    }
  }
  cudaError_t e = cudaSuccess;
  if (!t && (e = cudaMalloc(&t, kToken)) == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaMemPoolTrimTo(P->pool, 0);  // what is idle already
    e = cudaMalloc(&t, kToken);
  }
  if (e == cudaSuccess) e = cudaFree(t);
  if (e == cudaSuccess && cudaMalloc(&t, kToken) == cudaSuccess) {
    std::lock_guard<std::mutex> lock(g_mu);
    P->tokens.push_back(t);
  }
  cudaGetLastError();  // reported by e, or the next call makes its own token
  return e;
}

thread_local FreeTogether* t_together = nullptr;

// Blocks of long-lived buffers, after a wait: to the pool, or to the device.
void give_block(DevicePool* P, const Block& b) {
  WhileCapturing guard;
  const cudaError_t e = b.bytes >= kPoolMax ? cudaFree(b.p) : cudaFreeAsync(b.p, P->stream);
  if (e != cudaSuccess) {
    cudaGetLastError();  // not the caller's
    std::lock_guard<std::mutex> lock(g_mu);
    P->parked.push_back(b);
  }
}

// A wait, and what earlier waits that failed left behind with it.
cudaError_t wait_and_unpark(DevicePool* P) {
  std::vector<Block> parked;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    parked.swap(P->parked);
  }
  const cudaError_t e = wait_device(P);
  for (const Block& b : parked) {
    if (e == cudaSuccess) {
      give_block(P, b);
    } else {
      std::lock_guard<std::mutex> lock(g_mu);
      P->parked.push_back(b);
    }
  }
  return e;
}

// What the pool keeps goes back to the device.
cudaError_t give_back(DevicePool* P) {
  const cudaError_t e = wait_and_unpark(P);  // releases in flight count as kept only then
  if (e != cudaSuccess) return e;
  WhileCapturing guard;
  const cudaError_t sync = cudaStreamSynchronize(P->stream);
  return sync != cudaSuccess ? sync : cudaMemPoolTrimTo(P->pool, 0);
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
  WhileCapturing guard;
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

size_t dev_available() {
  DevicePool* P = nullptr;
  int dev = 0;
  size_t freeb = 0, total = 0;
  unsigned long long held = 0, used = 0;
  if (cudaMemGetInfo(&freeb, &total) != cudaSuccess || device_pool(&P, &dev) != cudaSuccess ||
      cudaMemPoolGetAttribute(P->pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
      cudaMemPoolGetAttribute(P->pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess)
    return freeb;
  return freeb + (held > used ? held - used : 0);
}

void dev_settle() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kMaxDevices) return;
  DevicePool* P = &g_pools[dev];
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!P->pool) return;  // nothing was allocated here yet
  }
  size_t freeb = 0, total = 0;
  unsigned long long held = 0, used = 0;
  WhileCapturing guard;
  if (cudaMemPoolGetAttribute(P->pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
      cudaMemPoolGetAttribute(P->pool, cudaMemPoolAttrUsedMemCurrent, &used) == cudaSuccess &&
      held > used + kPoolLow) {
    // cudaMemGetInfo takes 70 us, a small build 500: at most every 10 ms, or
    // when more has become idle
    const auto now = std::chrono::steady_clock::now();
    const unsigned long long idle = held - used;
    bool ask;
    {
      std::lock_guard<std::mutex> lock(g_mu);
      ask = idle > P->idle + (kPoolLow >> 2) || now - P->asked > std::chrono::milliseconds(10);
      if (ask) P->asked = now, P->idle = idle;
    }
    if (ask && cudaMemGetInfo(&freeb, &total) == cudaSuccess && freeb < kPoolRoom && give_back(P) == cudaSuccess) {
      std::lock_guard<std::mutex> lock(g_mu);
      P->idle = 0;
    }
  }
  cudaGetLastError();  // the entry point's own status stands
}

void dev_free(void* p, size_t bytes, int dev) {
  const Block b{p, bytes, dev};
  if (t_together) {
    t_together->blocks.push_back(b);
    return;
  }
  OnDevice on(dev);
  DevicePool* P = &g_pools[dev];
  // cudaFree waits by itself; a block of the pool may be in use on any stream
  if (bytes >= kPoolMax || wait_and_unpark(P) == cudaSuccess) {
    give_block(P, b);
    return;
  }
  std::lock_guard<std::mutex> lock(g_mu);
  P->parked.push_back(b);
}

FreeTogether::FreeTogether() : outer(t_together) { t_together = this; }

FreeTogether::~FreeTogether() {
  t_together = outer;
  if (outer) {
    outer->blocks.insert(outer->blocks.end(), blocks.begin(), blocks.end());
    return;
  }
  for (size_t i = 0; i < blocks.size();) {  // runs of blocks of one device
    const int dev = blocks[i].dev;
    OnDevice on(dev);
    DevicePool* P = &g_pools[dev];
    const cudaError_t e = wait_and_unpark(P);
    for (; i < blocks.size() && blocks[i].dev == dev; ++i) {
      if (e == cudaSuccess || blocks[i].bytes >= kPoolMax) {
        give_block(P, blocks[i]);
      } else {
        std::lock_guard<std::mutex> lock(g_mu);
        P->parked.push_back(blocks[i]);
      }
    }
  }
}

void dev_free_async(void* p, size_t bytes, cudaStream_t s, int dev) {
  if (bytes >= kPoolMax) {
    dev_free(p, bytes, dev);
    return;
  }
  OnDevice on(dev);
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
