// Kernel launches.
#pragma once
#include <cuda_runtime.h>

namespace tmc {

// Launches that overlap the end of the kernel before them (programmatic dependent launch).  A call is 12 to
// 90 short kernels; each costs 1.1 to 3 us between the one's end and the next one's start when the next is
// only set up then.  launch() lets it be set up while the one before runs: its blocks start as that one's
// leave, and wait in pdl_begin() until it is complete and its writes are visible.  So a kernel given to
// launch() calls pdl_begin() before it touches memory, and lets its own successor be set up there.
// 131x117x140 DMC with all outputs (87 kernels): 885 -> 721 us; 57x48x71 TMC with halfedges (18) 244 -> 208;
// 64^3 DMC (12) 150 -> 134; no difference on calls of milliseconds.
// Work that is not a kernel (copies, fills, event waits) still separates what is before it from what is
// after.  A wait in the stream holds back the launch itself, early or not: an event's, or one that the memory
// pool puts there when an allocation takes over what another stream freed (and nothing is touched before
// pdl_begin()).  Kernels behind the code's own event waits are launched plainly all the same.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
inline cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// Loads what an earlier kernel of the call wrote.  (Not __ldg: read-only loads may be moved ahead of
// pdl_begin().  It is for the field and for tables.)
template <typename T>
__device__ __forceinline__ T ld(const T* p) {
  return *p;
}

}  // namespace tmc
