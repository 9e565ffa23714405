// Programmatic dependent launch: a kernel of this library may be scheduled while its predecessor in the
// stream drains, so that its set-up (barriers, tensor memory, descriptors) and the launch itself are not
// paid between the two.
//
// Every kernel launched with launch_overlapped calls pdl_wait() in ALL its threads before its first
// access to global memory that another kernel may touch (reads AND writes): the wait returns when the
// predecessor has completed and its writes are visible.  A kernel that only calls
// pdl_launch_dependents() lets its successor in earlier; successors that were launched the ordinary way
// are ordered as ever.  Such a kernel takes its buffers as plain pointers: const __restrict__ and __ldg
// promise data that does not change while the kernel runs, but its predecessor may still be writing when
// it starts, and only the code's present order would keep such a load behind the wait.  (Loads that are to
// be in flight together are therefore written ahead of the stores.)  A kernel that waits for a peer GPU does not call it: its successor would hold SMs,
// shared memory and tensor memory for as long as the wait lasts.
#pragma once
#include <cuda_runtime.h>

namespace amem {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, const A&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) cudaGetLastError();
  return e;
}

}  // namespace amem
