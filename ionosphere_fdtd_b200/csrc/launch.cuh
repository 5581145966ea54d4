// Launches with programmatic dependence: a kernel launched by launch_after may be
// set up on an SM while the kernel before it on the stream drains there.  Such a
// kernel calls wait_previous, in every thread, before it reads or writes memory that
// an earlier launch may still write or read; the wait is for the whole of the kernel
// before, which in its turn waited for the one before it.  launch_next allows the
// following launch_after to begin; a plain launch or copy that follows still waits
// for the end of the kernel.  A kernel calls launch_next only when it holds all that it
// may have to wait for and that the following kernel could take first (tensor memory):
// what the following kernel holds, it holds until this one has ended.
#pragma once

#include <cuda_runtime.h>

namespace ifdtd {

__device__ __forceinline__ void launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kernel)(Params...), int blocks, int threads, size_t smem, cudaStream_t st,
                         const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace ifdtd
