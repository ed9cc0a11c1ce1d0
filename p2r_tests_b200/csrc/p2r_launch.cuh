// Kernel launches with programmatic dependent launch, shared by every kernel of the hot path.
//
// launch_pdl() lets a kernel be set up while the one before it on the stream still runs; the kernel
// begins with pdl_wait(), which returns when everything before it is complete and visible, so memory
// is accessed in the stream's order as before. No kernel releases its successor early
// (griddepcontrol.launch_dependents): the successor's CTAs would then be placed around the running
// ones and stay where they landed. 86060 tracks x 17 layers, 673 CTAs: 47.2 us without this launch,
// 45.5 with it, 54.1 with an early release. Other passes on one B200 before -> after: fused forward of
// 256 to 9600 tracks x 20 layers 20.5 -> 18.2 us, restart forward of 960000 tracks 41.3 -> 39.2 us,
// per-layer loop of 96000 tracks (40 launches) 287 -> 193 us.
#pragma once
#include <cuda_runtime.h>

namespace p2r {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kern)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &at;
  c.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&c, kern, (P)args...);
  if (e != cudaSuccess) cudaGetLastError();  // reported once: nothing stays pending
  return e;
}

}  // namespace p2r
