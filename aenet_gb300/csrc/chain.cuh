// Launches of a pass that are set up while the one before still runs
// (programmatic stream serialisation): the kernel's first statement waits for
// that one, and so for all before it, so that only the launch itself overlaps.
// Every kernel launched by launch_next begins with wait_for_previous.  A pass of
// 4,000 atoms is seven dependent kernels of 7 to 15 us: mixed 86.4 -> 73.2 us;
// 2,765 atoms FP64 268 -> 253 us; 256 atoms mixed 50 -> 46 us.
#pragma once

__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
inline cudaError_t launch_next(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               A... args) {
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}
