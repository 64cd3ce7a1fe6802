// Plane passes of the apply and of the band density for any 2,3,5-smooth n0 x n1
// (runtime plans, fft_rt.cuh).
#include "plane_passes.cuh"

namespace bg {
namespace {

constexpr int kPlaneWarps = 8;

// The y lines of the x rows holding sticks, and the x lines of every column y.
__device__ __forceinline__ rt::Pass y_pass(const OpTables& t, const BoxGeo& g, double2* pl, const double2* tw1,
                                           const int* rows) {
  rt::Pass a{};
  a.base = rt::shared_addr(pl);
  a.tw = rt::shared_addr(tw1);
  a.rows = rt::shared_addr(rows);
  a.es = 1;
  a.n = g.n1;
  a.tab = t.line_stick;
  return a;
}
__device__ __forceinline__ rt::Pass x_pass(const OpTables& t, const BoxGeo& g, double2* pl, const double2* tw0) {
  rt::Pass a{};
  a.base = rt::shared_addr(pl);
  a.tw = rt::shared_addr(tw0);
  a.pitch = 1;
  a.es = g.pitch;
  a.n = g.n0;
  a.xb = t.xbits;
  return a;
}

// Planes of any n0 x n1 (runtime plans): the passes of k_planes_fast below with the stages
// of fft_rt.cuh.  y inverse on the x rows holding sticks, its first stage straight from the
// stick row; x inverse, x V(r), x forward on every column with the middle in registers;
// y forward, its last stage straight to the stick row.  Two 256-thread blocks per SM
// (radix-12 butterflies need about 120 registers).
__global__ void __launch_bounds__(32 * kPlaneWarps, 2) k_planes(const OpTables* __restrict__ tabs, const __grid_constant__ BoxGeo g,
                                                                const __grid_constant__ Batch b) {
  const OpTables& t = tabs[blockIdx.z];
  const CallArgs a = resolve(b.a[blockIdx.z]);
  const int unit = blockIdx.x, z = blockIdx.y;
  if (unit >= a.units) return;
  extern __shared__ double2 sm[];
  double2* tw0 = sm;
  double2* tw1 = tw0 + g.n0;
  double2* pl = tw1 + g.n1;
  int* rows = reinterpret_cast<int*>(pl + g.n0 * g.pitch);
  const int nx = t.nxact;
  for (int i = threadIdx.x; i < g.n0; i += blockDim.x) tw0[i] = g.tw0[i];
  for (int i = threadIdx.x; i < g.n1; i += blockDim.x) tw1[i] = g.tw1[i];
  for (int i = threadIdx.x; i < nx; i += blockDim.x) rows[i] = t.xact[i] * g.pitch;
  __syncthreads();
  rt::Pass y = y_pass(t, g, pl, tw1, rows);
  y.row = t.sbuf + ((int64_t)unit * g.n2 + z) * t.S;
  rt::Pass x = x_pass(t, g, pl, tw0);
  x.weight = (a.vt ? a.vt : t.vt) + (int64_t)z * g.vstride;
  x.wpitch = g.n0;
  fast::owned_block(nx, t.yper, &y.first, &y.count);
  if (y.count > 0) rt::lines<1, fast::kInGlobal, 0>(y, g.p1);
  __syncthreads();
  fast::owned_block(g.n1, g.xper, &x.first, &x.count);
  if (x.count > 0) rt::inverse_weight_forward(x, g.p0);
  __syncthreads();
  if (y.count > 0) rt::lines<-1, 0, fast::kOutGlobal>(y, g.p1);
}

// The same for planes of any n0 x n1 (runtime plans), adding into the slice in global memory.
__global__ void __launch_bounds__(32 * kPlaneWarps, 2) k_density_planes(const OpTables* __restrict__ tabs, const __grid_constant__ BoxGeo g,
                                                                    const __grid_constant__ Batch b, int gamma, const double* __restrict__ w,
                                                                    int wstride, int per_chunk,
                                                                    double* __restrict__ part) {
  const OpTables& t = tabs[blockIdx.z];
  const CallArgs& a = b.a[blockIdx.z];
  w += (int64_t)blockIdx.z * wstride;
  const int z = blockIdx.x, chunk = blockIdx.y + blockIdx.z * gridDim.y;
  const int u0 = blockIdx.y * per_chunk, u1 = min(a.units, u0 + per_chunk);
  extern __shared__ double2 sm[];
  double2* tw0 = sm;
  double2* tw1 = tw0 + g.n0;
  double2* pl = tw1 + g.n1;
  int* rows = reinterpret_cast<int*>(pl + g.n0 * g.pitch);
  const int nx = t.nxact;
  for (int i = threadIdx.x; i < g.n0; i += blockDim.x) tw0[i] = g.tw0[i];
  for (int i = threadIdx.x; i < g.n1; i += blockDim.x) tw1[i] = g.tw1[i];
  for (int i = threadIdx.x; i < nx; i += blockDim.x) rows[i] = t.xact[i] * g.pitch;
  const int pts = g.n0 * g.n1;
  double* acc = part + ((int64_t)chunk * g.n2 + z) * pts;
  if (u0 >= u1)
    for (int i = threadIdx.x; i < pts; i += blockDim.x) acc[i] = 0.0;
  __syncthreads();
  rt::Pass yp = y_pass(t, g, pl, tw1, rows), xp = x_pass(t, g, pl, tw0);
  fast::owned_block(nx, t.yper, &yp.first, &yp.count);
  fast::owned_block(g.n1, g.dper, &xp.first, &xp.count);
  for (int unit = u0; unit < u1; ++unit) {
    yp.row = t.sbuf + ((int64_t)unit * g.n2 + z) * t.S;
    if (yp.count > 0) rt::lines<1, fast::kInGlobal, 0>(yp, g.p1);
    __syncthreads();
    if (xp.count > 0) rt::lines<1, fast::kInMask, 0>(xp, g.p0);
    __syncthreads();
    double wa, wb;
    density_weights(a, gamma, w, unit, &wa, &wb);
    for (int i = threadIdx.x; i < pts; i += blockDim.x) {
      const int y = i / g.n0, x = i - y * g.n0;
      const double2 p = pl[x * g.pitch + y];
      double d = unit == u0 ? 0.0 : acc[i];
      d += wa * (p.x * p.x);
      d += wb * (p.y * p.y);
      acc[i] = d;
    }
    __syncthreads();
  }
}

}  // namespace

void launch_runtime_planes(const OpTables* tabs, const BoxGeo& g, const Batch& b, dim3 grid, size_t smem,
                           cudaStream_t s) {
  k_planes<<<grid, 32 * kPlaneWarps, smem, s>>>(tabs, g, b);
}

void launch_runtime_density(const OpTables* tabs, const BoxGeo& g, const Batch& b, int gamma, const double* w,
                            int wstride, int per_chunk, double* part, dim3 grid, size_t smem, cudaStream_t s) {
  k_density_planes<<<grid, 32 * kPlaneWarps, smem, s>>>(tabs, g, b, gamma, w, wstride, per_chunk, part);
}

int configure_runtime_planes(size_t plane_smem) {
  cudaError_t e =
      cudaFuncSetAttribute((const void*)k_planes, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plane_smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void*)k_density_planes, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)plane_smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void*)k_planes, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void*)k_density_planes, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  return e == cudaSuccess ? 0 : 1;
}

namespace {
// Lines per warp of a pass over nlines lines of `p` on `warps` warps: its first stage's rounds
// count a times, its last stage's b times (fast::balanced_lines).
int balanced(const FftPlan& p, int a, int b, int nlines, int warps) {
  if (p.nst == 0) return (nlines + warps - 1) / warps > 0 ? (nlines + warps - 1) / warps : 1;
  return fast::balanced_lines(fast::lines_per_round(p.n, p.radix[0]), fast::lines_per_round(p.n, p.radix[p.nst - 1]), a,
                              b, nlines, warps);
}
}  // namespace

int plane_lines_per_warp(const BoxGeo& g, int nlines, int warps) {
  if (g.n0 == g.n1 && g.n1 == g.n2) switch (g.n0) {
      case 25: return fast::balanced_lines<25, 1, 1>(nlines, warps);
      case 45: return fast::balanced_lines<45, 1, 1>(nlines, warps);
      case 54: return fast::balanced_lines<54, 1, 1>(nlines, warps);
      case 60: return fast::balanced_lines<60, 1, 1>(nlines, warps);
      case 72: return fast::balanced_lines<72, 1, 1>(nlines, warps);
      case 108: return fast::balanced_lines<108, 1, 1>(nlines, warps);
      default: break;
    }
  return balanced(g.p1, 1, 1, nlines, warps);
}

void plane_columns_per_warp(BoxGeo* g) {
  g->xper = balanced(g->p0, 2, 1, g->n1, kPlaneWarps);
  g->dper = balanced(g->p0, 1, 1, g->n1, kPlaneWarps);
}

}  // namespace bg
