// Line passes of every 2,3,5-smooth length from 15 to 128 (but 125), selected at run time: one
// function per length and pass, called through a switch, so the index arithmetic inside is
// that of the compile-time plans of fft_fast.cuh.  The functions are not inlined: inlined into
// one kernel, the lengths' address and twiddle work is hoisted together and spills.  Their
// arguments sit in shared memory (a Pass per block), so a call costs a few instructions.
//
// Field grid of 72^3: 11 to 12 us per axis against 23.4 us with the runtime engine of fft_dev.cuh.
#pragma once
#include "fft_fast.cuh"

namespace bg {
namespace fast {

#define BG_ANY_LENGTHS(X)                                                                                        \
  X(15) X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48) X(50) X(54) X(60) X(64) X(72) X(75) \
  X(80) X(81) X(90) X(96) X(100) X(108) X(120) X(128)

__host__ __device__ constexpr bool any_length(int n) {
  switch (n) {
#define X(N) case N:
    BG_ANY_LENGTHS(X)
#undef X
    return true;
    default: return false;
  }
}

// Lines of a pass in shared memory: line l at base + rows[l] (rows given) or l pitch, elements
// es apart.  Shared-memory addresses are 32-bit.
struct Pass {
  unsigned base, tw, rows;  // double2*, const double2*, const int* (0: none)
  int pitch, es;
  const int* tab;           // stick of element e of line l at l N + e (StageIo)
  double2* row;             // the plane's stick row
  const unsigned* xb;       // element bits (StageIo)
  const double* weight;     // x pass: weight of element e of line l at l wpitch + e
  int wpitch;
};
template <class T>
__device__ __forceinline__ T* shared_at(unsigned a) {
  return static_cast<T*>(__cvta_shared_to_generic(a));
}
__device__ __forceinline__ unsigned shared_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

struct PassRows {
  const int* rows;
  __device__ __forceinline__ int operator()(int l) const { return rows[l]; }
};
struct PassPitch {
  int pitch;
  __device__ __forceinline__ int operator()(int l) const { return l * pitch; }
};
__device__ __forceinline__ StageIo<double2> pass_io(const Pass* a) {
  StageIo<double2> io;
  io.tab = a->tab;
  io.row = a->row;
  io.xb = a->xb;
  io.es = a->es;
  return io;
}

// y pass from the stick row (rows given, consecutive elements).
template <int N>
__device__ __noinline__ void y_inverse(const Pass* a, int first, int count) {
  double2* pl = shared_at<double2>(a->base);
  const double2* tw = shared_at<const double2>(a->tw);
  const PassRows off{shared_at<const int>(a->rows)};
  constexpr int R1 = Plan<N>::radix[0], R2 = Plan<N>::radix[1];
  stage<N, R1, 1, 1, 1, kInGlobal>(pl, first, count, off, tw, 0, pass_io(a));
  stage<N, R2, R1, 1, 1>(pl, first, count, off, tw, 0);
}
// y pass back to the stick row.
template <int N>
__device__ __noinline__ void y_forward(const Pass* a, int first, int count) {
  double2* pl = shared_at<double2>(a->base);
  const double2* tw = shared_at<const double2>(a->tw);
  const PassRows off{shared_at<const int>(a->rows)};
  constexpr int R1 = Plan<N>::radix[0], R2 = Plan<N>::radix[1];
  stage<N, R1, 1, -1, 1>(pl, first, count, off, tw, 0);
  stage<N, R2, R1, -1, 1, kOutGlobal>(pl, first, count, off, tw, 0, pass_io(a));
}
struct PassWeight {
  const double* w;
  int pitch;
  __device__ __forceinline__ double operator()(int line, int e) const { return w[line * pitch + e]; }
};
// x inverse, x weight, x forward (masked elements).
template <int N>
__device__ __noinline__ void x_weighted(const Pass* a, int first, int count) {
  double2* pl = shared_at<double2>(a->base);
  const double2* tw = shared_at<const double2>(a->tw);
  inverse_weight_forward<N, 0, true>(pl, first, count, PassPitch{a->pitch}, tw, PassWeight{a->weight, a->wpitch}, 0,
                                     pass_io(a));
}
// x inverse (masked inputs).
template <int N>
__device__ __noinline__ void x_inverse(const Pass* a, int first, int count) {
  double2* pl = shared_at<double2>(a->base);
  const double2* tw = shared_at<const double2>(a->tw);
  constexpr int R1 = Plan<N>::radix[0], R2 = Plan<N>::radix[1];
  stage<N, R1, 1, 1, 0, kInMask>(pl, first, count, PassPitch{a->pitch}, tw, 0, pass_io(a));
  stage<N, R2, R1, 1, 0>(pl, first, count, PassPitch{a->pitch}, tw, 0, pass_io(a));
}
// Whole lines of consecutive elements.
template <int N, int SIGN>
__device__ __noinline__ void whole_lines(unsigned base, unsigned tw, int pitch, int first, int count) {
  constexpr int R1 = Plan<N>::radix[0], R2 = Plan<N>::radix[1];
  double2* b = shared_at<double2>(base);
  const double2* t = shared_at<const double2>(tw);
  stage<N, R1, 1, SIGN, 1>(b, first, count, PassPitch{pitch}, t, 0);
  stage<N, R2, R1, SIGN, 1>(b, first, count, PassPitch{pitch}, t, 0);
}

#define BG_ANY_DISPATCH(NAME)                                                         \
  __device__ __forceinline__ void NAME##_any(int n, const Pass* a, int first, int count) { \
    if (count <= 0) return;                                                           \
    switch (n) { BG_ANY_LENGTHS(BG_ANY_CASE_##NAME) default: break; }                 \
  }
#define BG_ANY_CASE_y_inverse(N) case N: y_inverse<N>(a, first, count); break;
#define BG_ANY_CASE_y_forward(N) case N: y_forward<N>(a, first, count); break;
#define BG_ANY_CASE_x_weighted(N) case N: x_weighted<N>(a, first, count); break;
#define BG_ANY_CASE_x_inverse(N) case N: x_inverse<N>(a, first, count); break;
BG_ANY_DISPATCH(y_inverse)
BG_ANY_DISPATCH(y_forward)
BG_ANY_DISPATCH(x_weighted)
BG_ANY_DISPATCH(x_inverse)
#undef BG_ANY_CASE_y_inverse
#undef BG_ANY_CASE_y_forward
#undef BG_ANY_CASE_x_weighted
#undef BG_ANY_CASE_x_inverse
#undef BG_ANY_DISPATCH

// Rounds-balanced lines per warp (balanced_lines) of a pass of length n.
inline int any_lines_per_warp(int n, int a, int b, int nlines, int warps) {
  switch (n) {
#define X(N) \
  case N: return balanced_lines(lines_per_round(N, Plan<N>::radix[0]), lines_per_round(N, Plan<N>::radix[1]), a, b, nlines, warps);
    BG_ANY_LENGTHS(X)
#undef X
    default: return 1;
  }
}

}  // namespace fast

// Full transform of `nlines` lines (line l at base + l pitch, consecutive elements) by the
// whole block; begins and ends with __syncthreads.
template <int SIGN>
__device__ __forceinline__ void fft_block_lines(double2* base, int nlines, int pitch, const FftPlan& p,
                                                const double2* __restrict__ tw) {
  if (!fast::any_length(p.n)) {
    fft_lines<SIGN>(base, nlines, fast::PassPitch{pitch}, 1, p, tw);
    return;
  }
  __syncthreads();
  int first, count;
  fast::owned_lines(nlines, &first, &count);
  if (count > 0) {
    const unsigned b = fast::shared_addr(base), t = fast::shared_addr(tw);
    switch (p.n) {
#define X(N) case N: fast::whole_lines<N, SIGN>(b, t, pitch, first, count); break;
      BG_ANY_LENGTHS(X)
#undef X
      default: break;
    }
  }
  __syncthreads();
}

}  // namespace bg
