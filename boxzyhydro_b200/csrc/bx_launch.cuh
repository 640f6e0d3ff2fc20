// Launches that start before the one ahead of them in the stream is through.
#pragma once

#include <cuda_runtime.h>

namespace bx {

// Programmatic dependent launch: a kernel launched with launch_after may start while
// the one before it in the stream still runs.  It reads and writes device memory only
// after grid_wait, which returns when that kernel has completed and its writes are
// visible; grid_release lets the next one start once every block has begun.  Every
// thread of every kernel of such a chain waits, so each is complete before the second
// one after it reads anything.  Both do nothing in an ordinary launch.
// A step of a small grid is three launches of 4-6 us each, about 0.6 us of them between
// two kernels: 512-cell tube 13.5 -> 12.1 us a step, stepped 4x196 tube 41 -> 38, 32^3
// 26.8 -> 25.0, 75^3 173 -> 171, closed 96^3 box (22 launches a step) 424 -> 396; on
// large grids the next launch's blocks fill the last wave (256^3 3.772 -> 3.755 ms).
__device__ __forceinline__ void grid_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_release() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Launch `fn`, with `after` as a programmatic dependent of the stream's last kernel.
template <class... P, class... Q>
inline cudaError_t launch_after(bool after, void (*fn)(P...), dim3 blocks, int threads,
                                size_t smem, cudaStream_t s, const Q&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = after ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, fn, P(args)...);
}

}  // namespace bx
