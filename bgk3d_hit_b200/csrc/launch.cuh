// Launches that overlap the end of the kernel before them in a stream.
#pragma once
#include <cuda_runtime.h>

namespace bgk {

// Consecutive steps overlap their launches: a step's blocks are scheduled while the
// last blocks of the step before still run (launch_step asks for it), and wait here
// until all of that step's stores can be seen. First statement of every kernel
// that launch_step launches. us per step without / with it on B200: FP64 32^3 4.1 /
// 3.2, 64^3 10.7 / 9.0, 128^3 98.6 / 95.9; FP16 32^3 4.1 / 2.2, 64^3 6.2 / 4.9, 128^3
// 28.7 / 26.0.
//
// Everything behind it is read with ordinary loads: no __ldg, no const __restrict__
// parameter. Its blocks are resident while the kernel before still writes, and
// ld.global.nc is defined only for data that nothing writes as long as the kernel
// that reads it runs; the wait above orders ordinary accesses and no others.
__device__ __forceinline__ void step_begin() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches a kernel that starts with step_begin; overlap: so that it may be scheduled
// beside the end of the kernel before it in the stream. Only on a context's own
// stream, where that kernel is one of these or an ordinary one: step_begin waits
// for the kernel before, and through its own for those before that.
template <class... P, class... A>
inline cudaError_t launch_after(bool overlap, void (*kern)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = overlap ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
template <class... P, class... A>
inline cudaError_t launch_step(void (*kern)(P...), dim3 grid, dim3 block, cudaStream_t st, A... args) {
  return launch_after(true, kern, grid, block, st, args...);
}

}  // namespace bgk
