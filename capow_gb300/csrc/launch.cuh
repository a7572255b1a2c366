// Launch shapes of kernels with dynamic shared memory.
#pragma once
#include <cuda_runtime.h>

// Let `fn` take as much dynamic shared memory as a CTA can have (227 KB) beside `fixed` bytes for its own __shared__
// variables. Always the same limit, whatever the launch needs: the limit belongs to the function, and a launch that set it to
// its own need could have it lowered by another thread's launch for a smaller grid before it ran, and be refused.
constexpr int SMEM_CTA = 227 * 1024;
template <typename F>
inline void allow_smem(F *fn, int fixed = 0) {
  cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_CTA - fixed);
}

// Allow `fn` its dynamic shared memory on the current device and return how many of its CTAs of `threads` threads and smem
// bytes the whole device holds at once (at least the number of SMs). (Remembering the answers was worth 3 us
// of a 32^3 call's 143: not worth state that outlives a device reset.)
inline int resident_ctas(const void *fn, int threads, size_t smem, int fixed = 0) {
  int dev = 0, per_sm = 1, nsm = 152;
  allow_smem(fn, fixed);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return (per_sm > 0 ? per_sm : 1) * nsm;
}
