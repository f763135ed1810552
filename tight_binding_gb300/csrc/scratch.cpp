// scratch.cpp — the library's pool of device memory for workspaces and small objects.
#include <cuda_runtime.h>

#include <mutex>

#include "tbk_internal.h"

namespace tbk {
namespace {

constexpr int kMaxDevices = 64;
std::mutex g_mu;
cudaMemPool_t g_pools[kMaxDevices] = {};
bool g_tried[kMaxDevices] = {};

int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) { cudaGetLastError(); return -1; }
  return dev < kMaxDevices ? dev : -1;
}

}  // namespace

// The current device's pool; null where there is none (DevBuf then uses cudaMalloc).
cudaMemPool_t scratch_pool() {
  const int dev = current_device();
  if (dev < 0) return nullptr;
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_tried[dev]) {
    g_tried[dev] = true;
    cudaMemPoolProps pp = {};
    pp.allocType = cudaMemAllocationTypePinned;
    pp.location.type = cudaMemLocationTypeDevice;
    pp.location.id = dev;
    if (cudaMemPoolCreate(&g_pools[dev], &pp) != cudaSuccess) {
      cudaGetLastError();
      g_pools[dev] = nullptr;
    } else {
      uint64_t keep = kScratchKeep;
      cudaMemPoolSetAttribute(g_pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
  }
  return g_pools[dev];
}

// Returns what the current device's pool keeps and nothing uses.
void scratch_trim() {
  const int dev = current_device();
  if (dev < 0) return;
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    pool = g_pools[dev];
  }
  if (!pool) return;
  cudaDeviceSynchronize();                 // frees still in flight
  cudaMemPoolTrimTo(pool, 0);
}

}  // namespace tbk
