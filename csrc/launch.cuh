// Programmatic dependent launch: the blocks of a kernel are placed as soon as the last block of the kernel before it in the stream has ended,
// without waiting for that kernel's completion to reach the front end and for its writes to be flushed; the kernel itself waits for those.  On a chain of
// dependent kernels this saves 2 us per launch (512 x 128 x 576 products 8.2 -> 6.3 us, 8192 x 576 x 1344 17.5 -> 15.3).  No kernel here
// releases its successor early (griddepcontrol.launch_dependents): that measured no better (6.1, 15.3 and, at 16384 x 576 x 2240, 40.4 against 38.0 us), and
// blocks waiting on an SM could hold the tensor memory that a block of the running kernel has yet to allocate.
#pragma once
#include <c10/cuda/CUDAException.h>
#include <cuda_runtime.h>

#include <utility>

namespace q38 {

// In every kernel that `launch` starts, before its first access to global memory: returns when the kernels before it in the stream are complete and their writes visible.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Returns the launch's error: for entry points that report one instead of throwing (a C++ exception must not cross a C boundary).
template <typename... P, typename... A>
cudaError_t try_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  C10_CUDA_CHECK(try_launch(kernel, grid, block, smem, stream, std::forward<A>(args)...));
}

}  // namespace q38
