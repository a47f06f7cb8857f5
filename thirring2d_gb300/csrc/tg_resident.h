// tg_resident.h -- how many blocks of a kernel the current device holds at once.
#pragma once

#include <cuda_runtime_api.h>

#include <map>
#include <mutex>
#include <tuple>

namespace tg {

// Blocks of `threads` threads and `smem` bytes of dynamic shared memory resident on
// the current device, whose limit for the kernel is raised to smem; 0 if it has no room
// for them.  Limit and count are the device's own and are kept for each device.
inline int resident_blocks(const void* kernel, int threads, int smem) {
  static std::mutex mu;
  static std::map<std::tuple<int, const void*, int, int>, int> cache;
  int dev = 0, sms = 0, per_sm = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_tuple(dev, kernel, threads, smem);
  const auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
  if ((smem > 0 && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm <= 0) {
    (void)cudaGetLastError();
    return 0;  // (not kept: the next call asks again)
  }
  cache.emplace(key, per_sm * sms);
  return per_sm * sms;
}

}  // namespace tg
