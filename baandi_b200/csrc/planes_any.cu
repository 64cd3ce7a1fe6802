// Plane passes of the apply and of the band density for planes n0 x n1 of any two lengths of
// fft_any.cuh: the passes of k_planes_fast and k_density_planes_fast (hpsi_kernels.cu) with
// the two lengths chosen at run time.  The potential's plane is staged in shared memory
// (cp.async, behind the y pass) where it fits beside the plane.  Two blocks of eight warps
// per SM, or one of sixteen where the plane takes more than half the SM's shared memory: the
// radix-12 to -16 butterflies need 128 registers.  The planes of 111 columns on 45 x 60 x 36 take
// 147 us where the radix-2-to-5 runtime kernel (block barriers between four to six stages, the
// plane cleared and scattered first) took 596 us; an engine with the length read inside its
// stages took 470 us.
#include "launch_chain.cuh"
#include "plane_passes.cuh"

#include "fft_any.cuh"

namespace bg {
namespace {

// Warps of a block: 16 where only one block fits an SM, else 8 (two blocks).
size_t any_smem(const BoxGeo& g, bool vs) {
  const size_t pts = (size_t)g.n0 * g.n1;
  return sizeof(double2) * ((size_t)g.n0 + g.n1 + (size_t)g.n0 * g.pitch) + (vs ? sizeof(double) * ((pts + 1) / 2 * 2) : 0) +
         sizeof(int) * (size_t)g.n0;
}
int any_warps(const BoxGeo& g) { return any_smem(g, false) <= kPlaneAnyPair ? 8 : 16; }

// Shared memory of a block: twiddles of both axes, the plane, (the potential,) the rows' offsets.
__device__ __forceinline__ void setup(const OpTables& t, const BoxGeo& g, double2* sm, int* rows, fast::Pass* y,
                                      fast::Pass* x) {
  double2* tw0 = sm;
  double2* tw1 = tw0 + g.n0;
  double2* pl = tw1 + g.n1;
  for (int i = threadIdx.x; i < g.n0; i += blockDim.x) tw0[i] = g.tw0[i];
  for (int i = threadIdx.x; i < g.n1; i += blockDim.x) tw1[i] = g.tw1[i];
  for (int i = threadIdx.x; i < t.nxact; i += blockDim.x) rows[i] = t.xact[i] * g.pitch;
  if (threadIdx.x == 0) {
    *y = fast::Pass{fast::shared_addr(pl), fast::shared_addr(tw1), fast::shared_addr(rows), 0, 1, t.line_stick,
                    nullptr, nullptr, nullptr, 0};
    *x = fast::Pass{fast::shared_addr(pl), fast::shared_addr(tw0), 0u, 1, g.pitch, nullptr, nullptr, t.xbits, nullptr, 0};
  }
}

template <bool VS, int W>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : 1) k_planes_any(const OpTables* __restrict__ tabs,
                                                               const __grid_constant__ BoxGeo g,
                                                               const __grid_constant__ Batch b) {
  chain_wait();
  const OpTables& t = tabs[blockIdx.z];
  const CallArgs a = resolve(b.a[blockIdx.z]);
  const int unit = blockIdx.x, z = blockIdx.y;
  if (unit >= a.units) return;
  extern __shared__ __align__(16) double2 sm[];
  __shared__ fast::Pass y, x;
  const int pts = g.n0 * g.n1;
  double* vs = reinterpret_cast<double*>(sm + g.n0 + g.n1 + g.n0 * g.pitch);
  int* rows = reinterpret_cast<int*>(vs + (VS ? (pts + 1) / 2 * 2 : 0));
  const double* v = (a.vt ? a.vt : t.vt) + (int64_t)z * g.vstride;
  if (VS) {
    const unsigned dst = fast::shared_addr(vs);
    for (int i = threadIdx.x; i < pts / 2; i += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16u * i), "l"(v + 2 * i));
    if (threadIdx.x == 0 && (pts & 1)) vs[pts - 1] = v[pts - 1];
    asm volatile("cp.async.commit_group;\n" ::);
  }
  setup(t, g, sm, rows, &y, &x);
  if (threadIdx.x == 0) {
    y.row = t.sbuf + ((int64_t)unit * g.n2 + z) * t.S;
    x.weight = VS ? vs : v;
    x.wpitch = g.n0;
  }
  __syncthreads();
  int first, count;
  fast::owned_block(t.nxact, t.yany, &first, &count);
  fast::y_inverse_any(g.n1, &y, first, count);
  if (VS) asm volatile("cp.async.wait_all;\n" ::);
  __syncthreads();
  fast::owned_block(g.n1, g.xper, &first, &count);
  fast::x_weighted_any(g.n0, &x, first, count);
  __syncthreads();
  fast::owned_block(t.nxact, t.yany, &first, &count);
  fast::y_forward_any(g.n1, &y, first, count);
}

// One unit per (z plane, unit of the group, k point) block, as k_density_planes_fast.
template <int W>
__global__ void __launch_bounds__(32 * W, W == 8 ? 2 : 1)
    k_density_planes_any(const OpTables* __restrict__ tabs, const __grid_constant__ BoxGeo g,
                         const __grid_constant__ Batch b, int gamma, const double* w, int wstride,
                         int unit0, double* part) {
  chain_wait();
  const OpTables& t = tabs[blockIdx.z];
  const CallArgs& a = b.a[blockIdx.z];
  const int z = blockIdx.x, unit = unit0 + blockIdx.y;
  extern __shared__ __align__(16) double2 sm[];
  __shared__ fast::Pass y, x;
  double2* pl = sm + g.n0 + g.n1;
  int* rows = reinterpret_cast<int*>(pl + g.n0 * g.pitch);
  const int pts = g.n0 * g.n1;
  double* acc = part + ((int64_t)(blockIdx.y + blockIdx.z * gridDim.y) * g.n2 + z) * pts;
  if (unit >= a.units) {  // a k point with fewer units than the widest adds nothing
    for (int i = threadIdx.x; i < pts; i += blockDim.x) acc[i] = 0.0;
    return;
  }
  setup(t, g, sm, rows, &y, &x);
  if (threadIdx.x == 0) y.row = t.sbuf + ((int64_t)unit * g.n2 + z) * t.S;
  __syncthreads();
  int first, count;
  fast::owned_block(t.nxact, t.yany, &first, &count);
  fast::y_inverse_any(g.n1, &y, first, count);
  __syncthreads();
  fast::owned_block(g.n1, g.dper, &first, &count);
  fast::x_inverse_any(g.n0, &x, first, count);
  __syncthreads();
  double wa, wb;
  density_weights(a, gamma, w + (int64_t)blockIdx.z * wstride, unit, &wa, &wb);
  const float inv_n0 = 1.0f / (float)g.n0;
  for (int i = threadIdx.x; i < pts; i += blockDim.x) {
    const int yy = (int)(((float)i + 0.5f) * inv_n0), xx = i - yy * g.n0;  // i / n0, exact below 2^14
    const double2 p = pl[xx * g.pitch + yy];
    double d = wa * (p.x * p.x);
    d += wb * (p.y * p.y);
    acc[i] = d;
  }
}

}  // namespace

bool plane_any_supported(const BoxGeo& g) {
  return fast::any_length(g.n0) && fast::any_length(g.n1) && any_smem(g, false) <= kPlaneAnyMost;
}

void plane_lines_any(const BoxGeo& g, int nlines, int* yany, int* xper, int* dper) {
  const int warps = any_warps(g);
  *yany = fast::any_lines_per_warp(g.n1, 1, 1, nlines, warps);
  *xper = fast::any_lines_per_warp(g.n0, 2, 1, g.n1, warps);
  *dper = fast::any_lines_per_warp(g.n0, 1, 1, g.n1, warps);
}

void launch_planes_any(const OpTables* tabs, const BoxGeo& g, const Batch& b, dim3 grid, cudaStream_t s) {
  // the potential beside the plane where it costs no block
  if (any_warps(g) == 8) {
    if (any_smem(g, true) <= kPlaneAnyPair)
      launch_chained(k_planes_any<true, 8>, grid, 256, any_smem(g, true), s, tabs, g, b);
    else
      launch_chained(k_planes_any<false, 8>, grid, 256, any_smem(g, false), s, tabs, g, b);
  } else if (any_smem(g, true) <= kPlaneAnyMost) {
    launch_chained(k_planes_any<true, 16>, grid, 512, any_smem(g, true), s, tabs, g, b);
  } else {
    launch_chained(k_planes_any<false, 16>, grid, 512, any_smem(g, false), s, tabs, g, b);
  }
}

void launch_density_any(const OpTables* tabs, const BoxGeo& g, const Batch& b, int gamma, const double* w, int wstride,
                        int unit0, double* part, dim3 grid, cudaStream_t s) {
  if (any_warps(g) == 8)
    launch_chained(k_density_planes_any<8>, grid, 256, any_smem(g, false), s, tabs, g, b, gamma, w, wstride, unit0,
                   part);
  else
    launch_chained(k_density_planes_any<16>, grid, 512, any_smem(g, false), s, tabs, g, b, gamma, w, wstride, unit0,
                   part);
}

int configure_planes_any() {
  cudaError_t e = cudaSuccess;
  for (const void* f : {(const void*)k_planes_any<true, 8>, (const void*)k_planes_any<false, 8>,
                        (const void*)k_planes_any<true, 16>, (const void*)k_planes_any<false, 16>,
                        (const void*)k_density_planes_any<8>, (const void*)k_density_planes_any<16>}) {
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlaneAnyMost);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  }
  return e == cudaSuccess ? 0 : 1;
}

}  // namespace bg
