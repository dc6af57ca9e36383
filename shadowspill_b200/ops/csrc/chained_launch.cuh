// Launches whose blocks may start before the kernel ahead of them in the stream has ended.
#pragma once
#include <cuda_runtime.h>

namespace ss {

// A kernel started by launch_chained may begin before the one ahead of it in the stream has ended. It sets
// up its barriers and TMEM, waits in chain_wait() until that kernel is complete and its writes are visible,
// and only then touches global memory; every thread of every block waits, so the end of a kernel implies the
// end of all before it. chain_release() lets the next kernel's blocks take what this one's leave free: it
// follows chain_wait() and, where there is TMEM, the allocation, so that no waiting block can hold columns
// that a block of this kernel still needs.
//
// Such a kernel's lifetime begins while the one ahead still writes, so nothing in global memory is read-only for
// it: no `const __restrict__` parameters, __ldg or other non-coherent loads, which also are not ordered behind
// the wait by the compiler.
//
// What it saves is the gap between two kernels, 2 to 3 us: a layer of 1,999 tokens and 2,048 channels, forward and
// backward, 1004 -> 955 us (41 launches), attention on 2,048 tokens with heads of 64 121 -> 112 us, a layer of 8,192
// tokens and 4,096 channels 1.4 %. Kernels that wait for other ranks are launched plainly and do not release, so
// nothing takes room beside them early; so are the expert banks' and the delta rule's, which were 5 % and 1 %
// slower chained.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
inline void launch_chained(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute chained[1];
  chained[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  chained[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = chained;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);   // the launchers return cudaGetLastError()
}

}  // namespace ss
