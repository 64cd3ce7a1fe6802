// Shared by the plane kernels of the tuned cubic lengths (hpsi_kernels.cu) and of the other
// lengths (planes_any.cu).
#pragma once
#include "hpsi.h"

namespace bg {

__device__ __forceinline__ void density_weights(const CallArgs& a, int gamma, const double* __restrict__ w, int unit,
                                                double* wa, double* wb) {
  if (gamma) {
    *wa = w[2 * unit];
    *wb = 2 * unit + 1 < a.cols ? w[2 * unit + 1] : 0.0;
  } else {
    *wa = *wb = w[unit];
  }
}

// Shared memory of a plane block that leaves room for a second one on the SM.
constexpr size_t kPlaneAnyPair = 113 * 1024;

// The most one block takes: the 227 KB a block may have, less its static part.
constexpr size_t kPlaneAnyMost = 226 * 1024;

// Whether both axes of the plane have a pass in fft_any.cuh and the plane fits.
bool plane_any_supported(const BoxGeo& g);
// x rows and columns per warp of the passes over nlines x rows.
void plane_lines_any(const BoxGeo& g, int nlines, int* yany, int* xper, int* dper);
void launch_planes_any(const OpTables* tabs, const BoxGeo& g, const Batch& b, dim3 grid, cudaStream_t s);
void launch_density_any(const OpTables* tabs, const BoxGeo& g, const Batch& b, int gamma, const double* w, int wstride,
                        int unit0, double* part, dim3 grid, cudaStream_t s);
int configure_planes_any();

}  // namespace bg
