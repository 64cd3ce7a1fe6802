// Kernels launched one behind the other on a stream with programmatic stream serialisation:
// the next kernel's launch work overlaps the end of the previous kernel, and chain_wait at the
// top of every such kernel holds its blocks until the predecessor has finished and its writes
// are visible.  Every block calls it first, also where it returns at
// once: a kernel that could finish before its own predecessor would release its successor too
// early.
//
// No kernel releases its successor before it ends.  Released at the top instead, the
// successor's blocks filled the SMs that the predecessor's last wave had left, unevenly, and ran
// with the L1 share of its shared-memory carve-out: eigenproblems of capacities 60 to 128 (the
// control kernel on matrices in global memory) ran 10 to 27 % longer than with plain launches,
// densities of 45^3 and 54^3 4 to 9 %, one apply of 28 columns on 54^3 5 %.  Plain, released at
// the top, as here (us): Si2 Gamma apply 39.0, 32.4, 30.0 (its six kernels), one Si8 k point of 24
// columns 88.1, 82.4, 75.7; 28 columns on 54^3 147, 154, 136; Si8 solve of 48 bands at one k point
// 9,360, 11,900, 9,160; density of 8 k points x 24 bands on 45^3 175, 190, 170; the Si64 field
// step's 24 kernels 283, 250, 244.
//
// A chained kernel may start before its predecessor's writes are visible, so __restrict__ on
// one of its parameters is a promise that holds only for tables that no kernel writes (the
// compiler may read a const __restrict__ buffer through the non-coherent path, and may move any
// access through a __restrict__ pointer above the wait, which it takes not to touch it).
// Buffers that kernels write stay without it; tests/test_launch_chain.py holds the list.
#pragma once
#include <cuda_runtime.h>

namespace bg {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

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
