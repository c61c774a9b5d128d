// pdl.cuh -- chained launches of small kernels.
//
// A kernel launched by launch_chained may be scheduled once every block of
// the kernel before it on the stream has started; chain_enter, its first
// statement, then waits until that kernel has completed and its writes are
// visible.  What overlaps is the launch itself (about 1 us per kernel on the
// small grids, whose sub-step is a chain of some 13 kernels of 3-10 us), so
// the results and the order of all memory accesses are those of plain
// launches.  No kernel launched this way reads through a __restrict__ pointer
// to const, be it a parameter, a member of one, a local or a parameter of a
// function that it calls: such loads count as loads of constant memory and
// need not stay behind the wait.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace anel {

__device__ __forceinline__ void chain_enter() {
#if defined(__CUDA_ARCH__)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
#endif
}

// every kernel launched this way calls chain_enter first
template <class... P, class... A>
void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

}  // namespace anel
