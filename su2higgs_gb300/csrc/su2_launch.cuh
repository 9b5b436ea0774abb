// su2_launch.cuh -- launches that start while the launch before them on the
// stream drains.  A sweep is a chain of dependent passes, and on a small
// lattice a pass is hardly longer than the gap between two launches.  With the
// programmatic attribute the next pass's launch is under way as soon as every
// block of the running pass has done its sites (dependents_go, before the
// counters and the block's end); its blocks wait (dependent_wait) until that
// pass has completed and its writes are visible.  Letting it start any earlier
// is worse: its blocks then fill the SMs that have room instead of all of them
// (48^3 adjoint sweep 543 us without, 634 us from the first instruction, 488 us
// from the end of the update; 16^3 438 / 409 / 393 us).
//
// Rules: a kernel launched by launch_dependent calls dependent_wait in every
// thread before it reads anything an earlier launch writes, or writes anything;
// and it reads such memory with plain loads, which the compiler cannot move
// above the wait (read-only-path loads it could).  A kernel launched normally
// passes through dependent_wait at once.
#pragma once

#include <cuda_runtime.h>

namespace su2 {

__device__ inline void dependent_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ inline void dependents_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline void launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace su2
