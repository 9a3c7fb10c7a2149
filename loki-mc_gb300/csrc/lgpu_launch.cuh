// lgpu_launch.cuh - launches that overlap with the kernel before them.
#pragma once

#include <cuda_runtime.h>

namespace lgpu {

namespace {

// Kernels of one interval (or of one post-processing) follow one another with
// programmatic dependent launches: a kernel lets the next one's blocks start where its
// own leave room (next_may_start, at its beginning: every grid is resident at once or
// works off a list), and waits for the ones before it to have finished before it reads
// what they wrote (wait_for_previous). Both do nothing in an ordinary launch. A solve
// of 10,000 electrons took 11.8 ms without and 10.3 with them, two of 200,000 under AC
// 38.8 and 35.3.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// after_kernel: the last work on the stream is a kernel that calls next_may_start
// (else an ordinary launch)
template <class... Params, class... Args>
cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         bool after_kernel, const Args&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = after_kernel ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, args...);
}

}  // namespace

}  // namespace lgpu
