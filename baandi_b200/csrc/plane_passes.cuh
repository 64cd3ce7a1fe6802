// Shared by the plane kernels of the compile-time lengths (hpsi_kernels.cu) and of the
// runtime plans (planes_rt.cu).
#pragma once
#include "fft_rt.cuh"
#include "hpsi.h"

namespace bg {

struct LineOffTable {
  const int* off;
  __device__ __forceinline__ int operator()(int l) const { return off[l]; }
};
struct LineOffCols {
  __device__ __forceinline__ int operator()(int l) const { return l; }
};

__device__ __forceinline__ void density_weights(const CallArgs& a, int gamma, const double* __restrict__ w, int unit,
                                                double* wa, double* wb) {
  if (gamma) {
    *wa = w[2 * unit];
    *wb = 2 * unit + 1 < a.cols ? w[2 * unit + 1] : 0.0;
  } else {
    *wa = *wb = w[unit];
  }
}

// Planes of any n0 x n1 (planes_rt.cu): the apply's passes and the band density's.
void launch_runtime_planes(const OpTables* tabs, const BoxGeo& g, const Batch& b, dim3 grid, size_t smem,
                           cudaStream_t s);
void launch_runtime_density(const OpTables* tabs, const BoxGeo& g, const Batch& b, int gamma, const double* w,
                            int wstride, int per_chunk, double* part, dim3 grid, size_t smem, cudaStream_t s);
int configure_runtime_planes(size_t plane_smem);

}  // namespace bg
