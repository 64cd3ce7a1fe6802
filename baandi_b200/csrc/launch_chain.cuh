// Kernels launched one behind the other on a stream with programmatic stream serialisation:
// a kernel's blocks may start while the previous kernel drains (its launch latency and the
// ramp of its first blocks then overlap the predecessor's tail), and chain_wait at the top
// of every such kernel holds them until the predecessor has finished and its writes are
// visible.  Every block calls it first, also where it returns at once: a kernel that could
// finish before its own predecessor would release its successor too early.
//
// A chained kernel lives while its predecessor still writes, so __restrict__ on one of its
// parameters is a promise that holds only for tables that no kernel writes (the compiler may
// read a const __restrict__ buffer through the non-coherent path, and may move any access
// through a __restrict__ pointer above the wait, which it takes not to touch it).  Buffers that
// kernels write stay without it; tests/test_launch_chain.py holds the list.  Measured (chained
// against plain launches): the Si2 Gamma apply's six kernels 40.3 -> 32.5 us, one Si8 k point's
// 88.1 -> 82.0 us, the Si64 field step's 24 286 -> 244 us, 308 launches of an Si216 eigenproblem
// 2 ms of 145 ms.
#pragma once
#include <cuda_runtime.h>

namespace bg {

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::);
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);  // errors surface in cudaGetLastError
}

}  // namespace bg
