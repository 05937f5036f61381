// A ring of TMA tile stages between one loading lane and WARPS consumer warps
// of a persistent CTA.  Each consumer warp waits for a stage and gives it back
// by itself, so no barrier holds the CTA's warps together: a warp that has
// stored its part of a tile starts the next one while others still compute.
#pragma once

#include "sm100_util.cuh"

namespace cct {

template <int STAGES, int WARPS>
struct TileRing {
  uint64_t full[STAGES], empty[STAGES];

  // One thread sets the barriers up; a __syncthreads of the caller follows.
  __device__ __forceinline__ void init() {
    if (threadIdx.x == 0) {
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(&full[s], 1);
        mbar_init(&empty[s], WARPS);
      }
      fence_barrier_init();
    }
  }
  // The loading lane: load(tile, stage, full barrier) issues a tile's copy.
  // If the consumers stop giving stages back (one of them timed out), the
  // copies in flight get a bounded chance to land before the lane leaves, so
  // that none outlives the CTA.
  template <typename Load>
  __device__ __forceinline__ void produce(int total, unsigned *err, Load load) {
    int j = 0;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < total; i += gridDim.x, ++j) {
      const int s = j % STAGES;
      if (j >= STAGES) {
        ok = mbar_wait(&empty[s], (uint32_t)((j / STAGES - 1) & 1), err);
        if (!ok) break;
        fence_proxy_async_smem();
      }
      load(i, s, &full[s]);
    }
    // the last copies land before this lane leaves
    for (int k = j < STAGES ? 0 : j - STAGES; k < j; ++k)
      mbar_wait(&full[k % STAGES], (uint32_t)((k / STAGES) & 1), err);
  }
  // Consumers, tile number j of the CTA; false on a timeout (the warp leaves).
  __device__ __forceinline__ bool wait_full(int j, unsigned *err) {
    return __all_sync(0xffffffffu, mbar_wait(&full[j % STAGES], (uint32_t)((j / STAGES) & 1), err));
  }
  __device__ __forceinline__ void release(int s) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive(&empty[s]);
  }
};

}  // namespace cct
