// Overlapped launches: a kernel's launch may start while the kernel before it on the
// stream still runs its last CTAs (programmatic stream serialization).  A kernel lets its
// successor in (let_next_in; at its exit otherwise), reads what no kernel changes, and
// waits for its predecessor's completion (wait_for_previous) before it touches anything
// else: every thread that reads or writes global memory first, or by a barrier after one
// that has waited.  Every kernel launched this way waits, so that its own end is also the
// end of all before it.  What is read after the wait is read by ordinary loads: the
// read-only path (__ldg, const __restrict__) may be moved above it.
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void let_next_in() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Behind anything but a kernel it is an ordinary launch.
template <class K, class... A>
cudaError_t launch_overlapped(K kernel, dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
