// Kernel launches: back to back with the kernel before, with cluster dimensions, with more than 48 KB of shared memory.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>

namespace ody {

#ifdef __CUDACC__
template <class P>
__device__ __forceinline__ void opaque_pointer(P& p) { asm volatile("" : "+l"(p)); }

// First thing in a kernel that launch_kernel starts, before it reads or writes any global memory: its CTAs may already be
// resident while the kernel before it in the stream drains.  Waits until that kernel has finished and its writes are visible, then
// lets the next kernel of the stream come in as SMs run empty.  (In this order: when a kernel starts, everything before its direct
// predecessor is complete.)  What it saves is the gap between two kernels: a chain of products of 2048 x 1024 from K = 1024 took 11.9
// us each, this way 10.7; of 128 x 1024 from 1024 9.2 and 8.6.  A launch that waits for another GPU is not started like this.
// The pointers a kernel reads through, those inside its parameter structs among them, are passed along so that no load of read-only
// data, which the compiler may otherwise move across a fence, is formed before the wait.  (What TMA loads fetch needs none.)
template <class... P>
__device__ __forceinline__ void after_previous_kernel(P&... read) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  (opaque_pointer(read), ...);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

// Launch of a kernel that begins with after_previous_kernel; clusters of `cluster` CTAs along x.  Returns a cudaError_t.
template <class... P, class... A>
int launch_kernel(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, unsigned cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Opts `kernel` in to `bytes` of dynamic shared memory, once per device (the attribute belongs to a device's copy of it).
// `done` is the kernel's own bit set of devices.
template <class K>
int allow_smem(K* kernel, int bytes, std::atomic<uint64_t>& done) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  const uint64_t bit = dev < 64 ? 1ull << dev : 0;
  if (done.load(std::memory_order_acquire) & bit) return 0;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
  return (int)e;
}

}  // namespace ody
