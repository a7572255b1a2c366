// Launch shapes of kernels with dynamic shared memory.
#pragma once
#include <cuda_runtime.h>

// Allow `fn` smem bytes of dynamic shared memory on the current device and return how many of its CTAs of
// `threads` threads the whole device holds at once (at least the number of SMs). (Remembering the answers was worth 3 us
// of a 32^3 call's 143: not worth state that outlives a device reset.)
inline int resident_ctas(const void *fn, int threads, size_t smem) {
  int dev = 0, per_sm = 1, nsm = 152;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return (per_sm > 0 ? per_sm : 1) * nsm;
}
