// Warp-per-item launches: item claiming on the device, grid sizes on the host.
#pragma once

#include <algorithm>
#include <mutex>
#include <set>

#include "ct_internal.cuh"

namespace ct {

__device__ __forceinline__ double dinf() { return __longlong_as_double(0x7ff0000000000000ll); }

__device__ __forceinline__ uint32_t global_warp() {
  return (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
}
__device__ __forceinline__ uint32_t total_warps() { return (gridDim.x * blockDim.x) >> 5; }

// Items of a warp-per-item launch.  A warp takes item global_warp() first;
// when the grid does not cover every item (a persistent launch), it then
// claims the items past the grid in order from a counter, so uneven items
// balance as they do with one warp per item.  Warp-collective.
template <typename F>
__device__ __forceinline__ void for_items(uint32_t count, uint32_t* claim, F item) {
  const uint32_t nw = total_warps();
  uint32_t w = global_warp();
  while (w < count) {
    item(w);
    __syncwarp();
    if (nw >= count) break;
    uint32_t k = 0;
    if (lane_id() == 0) k = atomicAdd(claim, 1u);
    w = nw + __shfl_sync(FULL, k, 0);
  }
}

__device__ __forceinline__ uint32_t read_error(const Counters* c) {
  return *reinterpret_cast<const volatile uint32_t*>(&c->error);
}
// Work-list count clamped to its capacity; 0 once an earlier kernel of the
// step flagged an error, so no kernel reads a record that was not written.
__device__ __forceinline__ uint32_t live_count(const LevelScratch& s, uint32_t count, uint32_t cap) {
  return read_error(s.ctr) ? 0u : min(count, cap);
}

// Blocks of a warp-per-item launch: one warp per item, or, for a launch that
// must not depend on the item count (persistent), at most the blocks that
// are resident at once, whose warps then loop over the items.
template <typename K>
uint32_t grid_for(K kernel, uint64_t warps, size_t smem, bool persistent) {
  uint32_t cap = 0;
  if (persistent) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, THREADS_PER_BLOCK, smem);
    cap = (uint32_t)std::max(1, sms) * (uint32_t)std::max(1, per);
  }
  return item_blocks(warps, cap);
}

// Raises a kernel's dynamic shared-memory limit once per device (kernels of
// one signature share this function).
template <typename K>
int allow_smem(K kernel, int bytes) {
  static std::mutex mu;
  static std::set<std::pair<int, const void*>> done;
  int dev = 0;
  CT_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (done.count({dev, (const void*)kernel})) return CT_OK;
  CT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  done.insert({dev, (const void*)kernel});
  return CT_OK;
}

}  // namespace ct
