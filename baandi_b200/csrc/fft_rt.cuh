// Line FFTs of any 2,3,5-smooth length up to 128, FP64, radices chosen at run time.
//
// The stages are those of fft_fast.cuh (in-place Stockham decimation in time, a warp
// carrying its own block of lines through every stage with only __syncwarp between them),
// with the length, span and stride read from an FftPlan instead of being constants: the
// radix is the only template parameter, selected by a switch per stage.  Radices up to 12
// make every length but 75, 125 and 128 one or two stages (make_fft_plan), so a line
// crosses shared memory twice where radices 2 to 5 took three to five passes with a block
// barrier between them.
//
// Twiddles w^t of a butterfly are products of at most two table entries (w, w^2, w^4, w^8
// loaded from the length-N table in shared memory, the rest formed from them), so their
// error stays within two roundings.
//
// Sign convention (docs/physics-conventions.md:61-78 of the reference): SIGN = +1 is
// the unscaled inverse f(r) = sum_G f(G) e^{+iGr}; SIGN = -1 the forward transform
// (scaling by 1/N is applied by the caller).
#pragma once
#include "fft_fast.cuh"

namespace bg {
namespace rt {

using fast::kInGlobal;
using fast::kInMask;
using fast::kOutGlobal;
using fast::kOutMask;

// v[t] *= w^(t k step), t = 1 .. R-1 (conjugated for the forward sign).
template <int R, int SIGN>
__device__ __forceinline__ void twiddle(double2 (&v)[R], const double2* __restrict__ tw, int kstep) {
  double2 p[4];  // w, w^2, w^4, w^8
#pragma unroll
  for (int b = 0; b < 4; ++b)
    if ((1 << b) < R) {
      p[b] = tw[kstep << b];
      if (SIGN < 0) p[b].y = -p[b].y;
    }
#pragma unroll
  for (int t = 1; t < R; ++t) {
    // t = 3, 5, 6, 9, 10, 12: one product; 7 and 11: two
    double2 w = t & 8 ? p[3] : (t & 4 ? p[2] : (t & 2 ? p[1] : p[0]));
    const int top = t & 8 ? 8 : (t & 4 ? 4 : (t & 2 ? 2 : 1));
#pragma unroll
    for (int b = 2; b >= 0; --b)
      if ((t & (1 << b)) && (1 << b) < top) w = cmul(w, p[b]);
    v[t] = cmul(v[t], w);
  }
}

// Small-integer quotient a / d for a < 128 through the reciprocal of d.
__device__ __forceinline__ int quot(int a, float inv) { return (int)(((float)a + 0.5f) * inv); }

// Arguments of one stage over this warp's lines first .. first+count-1.  Lines start at
// base + l pitch (rows null) or base + rows[l]; es = element stride; ns = span of the
// earlier radices.  Shared-memory addresses are 32-bit, so that a call passes registers only.
struct Pass {
  unsigned base, tw, rows;  // double2*, double2*, const int* (0: none)
  int pitch, es, n, first, count;
  const int* tab;           // kInGlobal / kOutGlobal: stick of element e of line l at l n + e
  double2* row;
  const unsigned* xb;       // kInMask / kOutMask: element bits
  const double* weight;     // middle: weight of (line, element) at line wpitch + element
  int wpitch;
};
template <class T>
__device__ __forceinline__ T* shared_at(unsigned a) {
  return static_cast<T*>(__cvta_shared_to_generic(a));
}
__device__ __forceinline__ unsigned shared_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// A value the compiler cannot trace: what a stage computes from it stays inside its case of
// the radix switch (hoisted above the switch, the address and mask work of every radix
// together spills 20 KB a thread).
__device__ __forceinline__ void opaque(int& v) { asm volatile("" : "+r"(v)); }
__device__ __forceinline__ void opaque(unsigned& v) { asm volatile("" : "+r"(v)); }

// Stage (R, ns) of the lines of `a`; IO as in fast::stage.
template <int R, int SIGN, int IO>
__device__ __forceinline__ void stage(Pass a, int ns) {
  opaque(a.base);
  opaque(a.n);
  opaque(a.es);
  opaque(ns);
  double2* base = shared_at<double2>(a.base);
  const double2* tw = shared_at<const double2>(a.tw);
  const int* rows = shared_at<const int>(a.rows);
  const int n = a.n, span = n / R, es = a.es;
  const int lpr = 32 / span;
  const int lane = fast::lane_id();
  const int li = quot(lane, 1.0f / (float)span);
  const int j = lane - li * span;
  const bool lane_ok = li < lpr;
  const int k = j - quot(j, 1.0f / (float)ns) * ns;
  const int o = (j - k) * R + k;
  const int kstep = k * (span / ns);
  unsigned tin = 0u, tout = 0u;
  if constexpr ((IO & kInMask) != 0) {
#pragma unroll
    for (int t = 0; t < R; ++t) tin |= fast::xbit(a.xb, j + t * span) << t;
  }
  if constexpr ((IO & kOutMask) != 0) {
#pragma unroll
    for (int u = 0; u < R; ++u) tout |= fast::xbit(a.xb, o + u * ns) << u;
  }
  for (int r0 = 0; r0 < a.count; r0 += lpr) {
    double2 v[R];
    const bool act = lane_ok && r0 + li < a.count;
    const int line = a.first + r0 + li;
    double2* lp = base;
    if (act) {
      lp += a.rows ? rows[line] : line * a.pitch;
      if constexpr ((IO & kInGlobal) != 0) {
        int sidx[R];
#pragma unroll
        for (int t = 0; t < R; ++t) sidx[t] = __ldg(a.tab + line * n + j + t * span);
#pragma unroll
        for (int t = 0; t < R; ++t) v[t] = sidx[t] >= 0 ? a.row[sidx[t]] : make_double2(0.0, 0.0);
      } else {
#pragma unroll
        for (int t = 0; t < R; ++t)
          v[t] = ((IO & kInMask) == 0 || ((tin >> t) & 1u)) ? lp[(j + t * span) * es] : make_double2(0.0, 0.0);
      }
    }
    __syncwarp();
    if (act) {
      if (ns > 1) twiddle<R, SIGN>(v, tw, kstep);
      fast::Dft<R, SIGN, double2>::run(v);
      if constexpr ((IO & kOutGlobal) != 0) {
#pragma unroll
        for (int u = 0; u < R; ++u) {
          const int sx = __ldg(a.tab + line * n + o + u * ns);
          if (sx >= 0) a.row[sx] = v[u];
        }
      } else {
#pragma unroll
        for (int u = 0; u < R; ++u)
          if ((IO & kOutMask) == 0 || ((tout >> u) & 1u)) lp[(o + u * ns) * es] = v[u];
      }
    }
    __syncwarp();
  }
}

template <int SIGN, int IO>
__device__ __forceinline__ void stage_of(int radix, const Pass& a, int ns) {
  switch (radix) {
#define BG_RT(R) \
  case R: stage<R, SIGN, IO>(a, ns); break;
    BG_RT(2) BG_RT(3) BG_RT(4) BG_RT(5) BG_RT(6) BG_RT(8) BG_RT(9) BG_RT(10) BG_RT(12)
#undef BG_RT
    default: break;
  }
}

// Every stage of this warp's lines, first stage with IO bits FIRST, last with LAST
// (kInGlobal / kInMask and kOutGlobal); a one-stage plan does both.
template <int SIGN, int FIRST, int LAST>
__device__ __forceinline__ void lines(const Pass& a, const FftPlan& p) {
  if (p.nst == 0) {  // length 1: move the single elements
    double2* base = shared_at<double2>(a.base);
    const int* rows = shared_at<const int>(a.rows);
    for (int l = a.first + fast::lane_id(); l < a.first + a.count; l += 32) {
      double2* z = base + (a.rows ? rows[l] : l * a.pitch);
      const int sx = (FIRST | LAST) & (kInGlobal | kOutGlobal) ? __ldg(a.tab + l) : -1;
      if (FIRST & kInGlobal) *z = sx >= 0 ? a.row[sx] : make_double2(0.0, 0.0);
      if ((FIRST & kInMask) && !fast::xbit(a.xb, 0)) *z = make_double2(0.0, 0.0);
      if ((LAST & kOutGlobal) && sx >= 0) a.row[sx] = *z;
    }
    __syncwarp();
    return;
  }
  if (p.nst == 1) {
    stage_of<SIGN, FIRST | LAST>(p.radix[0], a, 1);
    return;
  }
  int ns = 1;
  for (int s = 0; s < p.nst; ++s) {
    const int r = p.radix[s];
    if (FIRST != 0 && s == 0)
      stage_of<SIGN, FIRST>(r, a, ns);
    else if (LAST != 0 && s + 1 == p.nst)
      stage_of<SIGN, LAST>(r, a, ns);
    else
      stage_of<SIGN, 0>(r, a, ns);
    ns *= r;
  }
}

// Middle of an x pass: the inverse's last stage (radix R, span n / R), times the weight of
// every element, and the first stage of a forward transform run with the plan reversed,
// whose butterflies take exactly the elements this one leaves.
template <int R, int IO>
__device__ __forceinline__ void middle(Pass a) {
  opaque(a.base);
  opaque(a.n);
  opaque(a.es);
  double2* base = shared_at<double2>(a.base);
  const double2* tw = shared_at<const double2>(a.tw);
  const int span = a.n / R, lpr = 32 / span, es = a.es;
  const int lane = fast::lane_id();
  const int li = quot(lane, 1.0f / (float)span);
  const int j = lane - li * span;
  const bool lane_ok = li < lpr;
  for (int r0 = 0; r0 < a.count; r0 += lpr) {
    double2 v[R];
    const bool act = lane_ok && r0 + li < a.count;
    const int line = a.first + r0 + li;
    double2* lp = base + line * a.pitch;
    if (act) {
#pragma unroll
      for (int t = 0; t < R; ++t)
        v[t] = ((IO & kInMask) == 0 || fast::xbit(a.xb, j + t * span)) ? lp[(j + t * span) * es]
                                                                         : make_double2(0.0, 0.0);
    }
    __syncwarp();
    if (act) {
      const double* w = a.weight + line * a.wpitch + j;
      double wt[R];
#pragma unroll
      for (int u = 0; u < R; ++u) wt[u] = __ldg(w + u * span);
      if (span > 1) twiddle<R, 1>(v, tw, j);
      fast::Dft<R, 1, double2>::run(v);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        v[u].x *= wt[u];
        v[u].y *= wt[u];
      }
      fast::Dft<R, -1, double2>::run(v);
#pragma unroll
      for (int u = 0; u < R; ++u) lp[(j * R + u) * es] = v[u];
    }
    __syncwarp();
  }
}

// Inverse transform, x weight, forward transform of this warp's lines.  Only the elements
// whose bit is set in a.xb are nonzero on input and wanted on output.
__device__ __forceinline__ void inverse_weight_forward(const Pass& a, const FftPlan& p) {
  if (p.nst == 0) {  // length 1: the weight alone
    double2* base = shared_at<double2>(a.base);
    for (int l = a.first + fast::lane_id(); l < a.first + a.count; l += 32) {
      const double w = __ldg(a.weight + l * a.wpitch);
      double2& z = base[l * a.pitch];
      z = make_double2(z.x * w, z.y * w);
    }
    __syncwarp();
    return;
  }
  const int last = p.nst - 1;
  int ns = 1;
  for (int s = 0; s < last; ++s) {
    if (s == 0)
      stage_of<1, kInMask>(p.radix[s], a, ns);
    else
      stage_of<1, 0>(p.radix[s], a, ns);
    ns *= p.radix[s];
  }
  switch (p.radix[last]) {
#define BG_RT(R)            \
  case R:                   \
    if (last == 0)          \
      middle<R, kInMask>(a); \
    else                    \
      middle<R, 0>(a);      \
    break;
    BG_RT(2) BG_RT(3) BG_RT(4) BG_RT(5) BG_RT(6) BG_RT(8) BG_RT(9) BG_RT(10) BG_RT(12)
#undef BG_RT
    default: break;
  }
  ns = p.radix[last];
  for (int s = last - 1; s >= 0; --s) {
    if (s == 0)
      stage_of<-1, kOutMask>(p.radix[s], a, ns);
    else
      stage_of<-1, 0>(p.radix[s], a, ns);
    ns *= p.radix[s];
  }
}

}  // namespace rt

// Full transform of `nlines` lines (line l at base + l pitch, consecutive elements) by the
// whole block; begins and ends with __syncthreads.
template <int SIGN>
__device__ __forceinline__ void fft_lines(double2* base, int nlines, int pitch, const FftPlan& p,
                                          const double2* __restrict__ tw) {
  __syncthreads();
  rt::Pass a{};
  fast::owned_lines(nlines, &a.first, &a.count);
  a.base = rt::shared_addr(base);
  a.tw = rt::shared_addr(tw);
  a.pitch = pitch;
  a.es = 1;
  a.n = p.n;
  if (a.count > 0) rt::lines<SIGN, 0, 0>(a, p);
  __syncthreads();
}

}  // namespace bg
