// Launches whose blocks start while the kernel before them in the stream
// ends (programmatic dependent launch).  Between two small dependent kernels
// the GPU idles ~2 us, half of it the launch of the second one's blocks.  A
// kernel launched by launch_dependent begins with dependent_begin, after at
// most what touches no memory that another kernel writes: it waits until the
// kernel before is complete and its writes are visible, so the order of a
// stream is kept.
//
// What an earlier kernel writes is read by ordinary loads: its pointers carry
// no __restrict__ where the kernel does not write through them, and no __ldg.
// The read-only path of those asks for data that stay unchanged for the
// kernel's whole life, which here begins before the earlier kernel's writes
// are visible.
//
// No kernel lets its successor start before its own end
// (griddepcontrol.launch_dependents): blocks that wait on an SM slowed the
// sweeps down.  Solves of the 32 x 32 cavity Newton: 229.9 ms without, 215.9
// ms so, 222.7 ms with early starts outside the sweeps, 228.5 ms everywhere.
#pragma once
#include <cuda_runtime.h>

namespace gb {

__device__ __forceinline__ void dependent_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
static cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                                    cudaStream_t st, A... args) {
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace gb
