// Kernel launches of the operator and CG sequences.
//
// Consecutive kernels of a sequence are launched with programmatic stream
// serialization: the next kernel is set up while the previous one drains and
// starts, at the latest in pdl_wait(), when that has completed and its writes
// are visible.  Every kernel launched this way calls pdl_wait() before it
// reads or writes anything another kernel touches (active flags and scalars
// included), on every path, so completion stays transitive along the stream;
// a kernel launched without the attribute still waits for the whole sequence.
// fncB, called from C one after the other: one vector at n = 24 22.6 -> 11.7 us,
// three at n = 50 52 -> 39, ten at n = 60 197 -> 175 (complex64), two at n = 16 45.6 -> 31.0,
// four at n = 40 433 -> 419 (complex128).  (A call from Python has some 10 us of host
// time more: one vector at n = 24 takes 19.7, none of it waiting for the GPU.)
// No kernel triggers its successor early: CTAs placed while the previous kernel
// still runs are spread over the SMs by what is free at that moment, not
// evenly (complex128 CG of two vectors at n = 30: 10.1 ms with a trigger at
// the kernels' start, 5.9 without).
#pragma once

#include <cuda_runtime.h>

#include <atomic>

#include "fame_internal.h"

namespace fame {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Allows kernel K its dynamic shared memory, once per device.
template <auto K> cudaError_t allow_smem(size_t sm) {
  static std::atomic<unsigned long long> done{0};  // one bit per device
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
  if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return e;
}

// Launches K<<<grid, tb, sm, st>>>(args...) as a programmatic dependent of the
// previous kernel in st, in clusters of (1, CLUSTER, 1) CTAs.  sm is the same at
// every launch of K.
template <auto K, int CLUSTER = 1, class... A>
cudaError_t launch(dim3 grid, int tb, size_t sm, cudaStream_t st, A... args) {
  if (sm > 48 * 1024) {
    cudaError_t e = allow_smem<K>(sm);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(tb);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 1;
  at[1].val.clusterDim.y = CLUSTER;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CLUSTER > 1 ? 2 : 1;
  FAME_LAUNCHED(1);
  return cudaLaunchKernelEx(&cfg, K, args...);
}

}  // namespace fame
