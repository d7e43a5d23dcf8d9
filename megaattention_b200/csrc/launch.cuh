// Launches that may start while the kernel before them in the stream is on its way out.
//
// From the end of one kernel to the start of the next a stream waits 2-4 us, and the fused kernel sets
// up barriers and TMEM for another half.  With programmatic launches both run under the end of the
// kernel before: the CTAs start as soon as its CTAs have left (or said that they may), and
// wait_for_previous() holds them back before the first access to memory until that kernel is complete
// and all it wrote is visible.  Every kernel launched this way has to pass it, so that completion is
// handed on from kernel to kernel.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace ma {

__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel may start (it waits for this one's completion all the same).
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A pointer whose loads stay behind what is written above (the compiler may move loads through a
// const __restrict__ argument up, past an asm that clobbers memory too).
template <class T>
__device__ __forceinline__ T* from_here(T* p) {
  asm volatile("" : "+l"(p) :: "memory");
  return p;
}

template <class... P, class... A>
cudaError_t launch_behind(void (*kernel)(P...), int grid, int threads, size_t smem, cudaStream_t stream,
                          A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<A&&>(args)...);
  const cudaError_t last = cudaGetLastError();      // (reported here, not to the next caller)
  return e != cudaSuccess ? e : last;
}

}  // namespace ma
