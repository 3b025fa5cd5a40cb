// Launches that may begin while the previous kernel of the stream still runs
// (programmatic dependent launch). Every kernel launched through fz_launch_pdl
// calls pdl_begin before its first access to memory that earlier work of the
// stream may write or read (its inputs, outputs and scratch; tables are written
// at setup): it lets the next such kernel be brought onto the device once this
// one's last CTA has started, then waits until everything before it in the stream
// is complete and visible. What overlaps is the launch itself, the first CTAs'
// set-up and the first instruction fetches.
#pragma once
#include <cuda_runtime.h>

namespace fftz {
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
}  // namespace fftz

static inline int fz_launch_pdl(const void *fn, dim3 grid, dim3 block, void **args, size_t smem, void *stream) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = (cudaStream_t)stream;
  c.attrs = &at;
  c.numAttrs = 1;
  return (int)cudaLaunchKernelExC(&c, fn, args);
}
