// Residue-number products on the int8 tensor cores (see gemm_rns.cuh for the scheme).
//
// Passes of one launch:
//   k_rns_scale_cols / _rows  power-of-two scale of every operand column or row (2-norm)
//   k_rns_balance             power-of-two balance of K (A B products that split A)
//   k_rns_split               integers, modulo the moduli, as int8 panels in MMA tile order
//   k_rns_mma                 the 2 kModuli int8 products; epilogue reduces to one byte
//   k_rns_join                Chinese remainder: bytes -> FP64, C (op)= result
//
// Panel layout: plane q (2 i + s: modulus i, sign s), row tile, K tile; a tile holds R rows
// x 64 K bytes in the canonical K-major layout without swizzle (16-byte K chunk c of row r
// at c R 16 + r 16), so a tile is one contiguous bulk copy.
#include "gemm_rns.cuh"

#include <algorithm>
#include <vector>

namespace bg {
namespace rns {
namespace {

constexpr int kSms = 148;
constexpr int kMaxDesc = 128;
constexpr int kStages = 6;
constexpr int kMmaThreads = 320;  // producer warp, MMA warp, eight epilogue warps
constexpr unsigned kMagic = 0x4B400000u;        // float 1.5 2^23: integers |x| < 2^22 sit in its low bits
constexpr float kMagicF = 12582912.0f;

// --------------------------------------------------------------------- moduli
// Largest pairwise coprime products of primes = 1 mod 4 (5 13 17 29 37 41 ...) up to 241.
constexpr int kP[kModuli] = {241, 233, 229, 221, 205, 197, 193, 181, 173, 157, 149, 137, 113, 109, 101, 97};
constexpr double kLog2M = 117.69;      // log2 of their product (checked below)
constexpr double kNormBits = 58.34;    // 2 kNormBits + 1 < kLog2M

struct Tables {
  int p[kModuli];
  float inv[kModuli];                // 1 / p
  int c16[kModuli];                  // 2^16 mod p, balanced
  unsigned wlo[kModuli], whi[kModuli];  // 256^j mod p, j = 0..7, as signed bytes
  unsigned rlo[kModuli], rhi[kModuli];  // r 256^j mod p
  int ca[kModuli], cb[kModuli];      // corrections of the 2^63 offset: -2^63 mod p, -r 2^63 mod p
  // CRT weights (M/p)^-1 / (2 p) and (M/p)^-1 / (2 r p) modulo 1 (real and imaginary part), each
  // as a multiple of 2^-36 within 1/2 of zero and the remainder
  double reh[kModuli], rel[kModuli], imh[kModuli], iml[kModuli];
  double mhi, mlo;                   // the product M of the moduli
};

constexpr int bal(int x, int p) {  // balanced residue
  int r = x % p;
  if (r < 0) r += p;
  return 2 * r > p ? r - p : r;
}
constexpr int inverse(int x, int p) {
  for (int y = 1; y < p; ++y)
    if ((x % p) * y % p == 1) return y;
  return 0;
}
constexpr int root(int p) {  // r^2 = -1 mod p
  for (int r = 2; r < p; ++r)
    if ((r * r + 1) % p == 0) return r;
  return 0;
}
constexpr int pow2(int e, int p) {
  int r = 1;
  for (int i = 0; i < e; ++i) r = r * 2 % p;
  return r;
}
// t / p modulo 1: the nearest multiple of 2^-36 (centred) and the remainder.
constexpr void weight(int t, int p, double* hi, double* lo) {
  const unsigned __int128 f = (((unsigned __int128)(unsigned)t) << 96) / (unsigned)p;
  const unsigned long long h = (unsigned long long)((f + (((unsigned __int128)1) << 59)) >> 60);
  const __int128 rest = (__int128)f - (__int128)(((unsigned __int128)h) << 60);
  const long long hc = h >= (1ull << 35) ? (long long)h - (1ll << 36) : (long long)h;
  *hi = (double)hc / 68719476736.0;                              // 2^-36
  *lo = (double)(long long)rest / 1152921504606846976.0 / 68719476736.0;  // 2^-60 2^-36
}
constexpr Tables make_tables() {
  Tables t{};
  unsigned __int128 m = 1;
  for (int i = 0; i < kModuli; ++i) m *= (unsigned)kP[i];
  t.mhi = (double)m;
  t.mlo = m >= (unsigned __int128)t.mhi ? (double)(m - (unsigned __int128)t.mhi)
                                        : -(double)((unsigned __int128)t.mhi - m);
  for (int i = 0; i < kModuli; ++i) {
    const int p = kP[i], r = root(p);
    t.p[i] = p;
    t.inv[i] = 1.0f / (float)p;
    t.c16[i] = bal(pow2(16, p), p);
    t.ca[i] = bal(-pow2(63, p), p);
    t.cb[i] = bal(-pow2(63, p) * r, p);
    for (int j = 0; j < 4; ++j) {
      t.wlo[i] |= ((unsigned)bal(pow2(8 * j, p), p) & 0xffu) << (8 * j);
      t.whi[i] |= ((unsigned)bal(pow2(8 * j + 32, p), p) & 0xffu) << (8 * j);
      t.rlo[i] |= ((unsigned)bal(pow2(8 * j, p) * r, p) & 0xffu) << (8 * j);
      t.rhi[i] |= ((unsigned)bal(pow2(8 * j + 32, p) * r, p) & 0xffu) << (8 * j);
    }
    int cof = 1;  // (M / p)^-1 mod p
    for (int j = 0; j < kModuli; ++j)
      if (j != i) cof = cof * (kP[j] % p) % p;
    cof = inverse(cof, p);
    const int re = cof * inverse(2, p) % p, im = cof * inverse(2 * r % p, p) % p;
    weight(re, p, &t.reh[i], &t.rel[i]);
    weight(im, p, &t.imh[i], &t.iml[i]);
  }
  return t;
}
constexpr Tables kTab = make_tables();
static_assert(kTab.mhi > 2.6806e35 && 2.0 * kNormBits + 1.0 < kLog2M, "2^117.69 = 2.6805e35 < product of the moduli");
__constant__ Tables c_tab = make_tables();

// --------------------------------------------------------------------- PTX
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// Shared-memory matrix descriptor: K-major, no swizzle, start/LBO/SBO in 16-byte units,
// descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor of kind::i8: int32 accumulator (bits 4-5 = 2), signed 8-bit A and B
// (bits 7-9, 10-12 = 1), both K-major, N / 8 at bits 17-22, M / 16 at bits 24-28.
__device__ __forceinline__ uint32_t idesc(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
}
__device__ __forceinline__ void mma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t"
      "}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(id), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile(
      "{\n\t"
      ".reg .b64 st;\n\t"
      "mbarrier.arrive.shared::cta.b64 st, [%0];\n\t"
      "}\n" ::"r"(mbar)
      : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes) {
  asm volatile(
      "{\n\t"
      ".reg .b64 st;\n\t"
      "mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t"
      "}\n" ::"r"(mbar),
      "r"(bytes)
      : "memory");
}
// Bounded wait; gives up early once another role of the block has.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, volatile int* failed, unsigned limit) {
  for (unsigned i = 0; i < limit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 255u) == 255u && *failed) return false;
  }
  return false;
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
__device__ __forceinline__ int dp4a_us(unsigned a, unsigned b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// --------------------------------------------------------------------- scales
// Power of two that brings a row of 2-norm sqrt(ssq) (largest part amax, n complex values)
// to at most 2^kNormBits; the inverse is NaN for a row holding a NaN or an infinity, so
// that every output it enters becomes NaN.  Rows whose squares over- or underflow take the
// bound amax sqrt(2 n).
__device__ __forceinline__ void scale_of(double ssq, double amax, double n, double* sc, double* inv) {
  if (isnan(ssq) || isinf(amax)) {
    *sc = 0.0;
    *inv = __longlong_as_double(0x7ff8000000000000LL);
    return;
  }
  if (amax == 0.0) {
    *sc = 1.0;
    *inv = 1.0;
    return;
  }
  const double lg = (ssq >= 1e-280 && ssq <= 1e300) ? 0.5 * log2(ssq) : log2(amax) + 0.5 * log2(2.0 * n);
  const double e = fmin(1000.0, fmax(-1000.0, floor(kNormBits - 1e-3 - lg)));
  *sc = ldexp(1.0, (int)e);
  *inv = ldexp(1.0, -(int)e);
}

struct Operand {  // element (row j, K index k): X[k sk + j sj] bal[k]
  const double2* X;
  int64_t sk, sj;
  int rows, K;
  const double* bal = nullptr;  // (BAL)
  template <bool BAL>
  __device__ __forceinline__ double2 balanced(double2 v, int k) const {
    if constexpr (BAL) {
      const double s = __ldg(bal + k);
      v.x *= s;
      v.y *= s;
    }
    return v;
  }
};
__device__ __forceinline__ Operand operand_of(const Desc& d, int mode, int which) {
  Operand o;
  o.K = d.K;
  if (which == 0) {
    o.X = d.A;
    o.rows = d.M;
    o.sk = mode == kTN ? 1 : d.lda;
    o.sj = mode == kTN ? d.lda : 1;
  } else {
    o.X = d.B;
    o.rows = d.N;
    o.sk = 1;
    o.sj = d.ldb;
  }
  return o;
}

// One block per row whose K run is contiguous (columns of A and B).
template <bool BAL>
__device__ __forceinline__ void scale_cols(const Operand& o, int j, double* sc, double* inv) {
  __shared__ double s_sum[8], s_max[8];
  const double2* x = o.X + (int64_t)j * o.sj;
  double ssq = 0.0, amax = 0.0;
#pragma unroll 4
  for (int k = threadIdx.x; k < o.K; k += 256) {
    const double2 v = o.template balanced<BAL>(__ldg(x + k), k);
    ssq = fma(v.x, v.x, fma(v.y, v.y, ssq));
    amax = fmax(amax, fmax(fabs(v.x), fabs(v.y)));
  }
  for (int off = 16; off > 0; off >>= 1) {
    ssq += __shfl_down_sync(0xffffffffu, ssq, off);
    amax = fmax(amax, __shfl_down_sync(0xffffffffu, amax, off));
  }
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = ssq;
    s_max[threadIdx.x >> 5] = amax;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) {
      ssq += s_sum[w];
      amax = fmax(amax, s_max[w]);
    }
    scale_of(ssq, amax, o.K, sc + j, inv + j);
  }
}
// d[k] = the largest of |B_kj| over the columns j, each relative to its column's norm (the power
// of two below it); dinv = 1 / d.  A D and D^-1 B have the product A B, but a row of A D counts
// its entries as the product does: coefficients of 1e-8 on large entries no longer set the
// quantum of the row's others.  32 K indices x 8 column slices per block.
__device__ __forceinline__ void balance(const Operand& o, const double* sc, double* d, double* dinv) {
  __shared__ double b_max[8][32];
  const int kl = threadIdx.x & 31, q = threadIdx.x >> 5, k = blockIdx.x * 32 + kl;
  double m = 0.0;
  if (k < o.K) {
#pragma unroll 8
    for (int j = q; j < o.rows; j += 8) {
      const double2 v = __ldg(o.X + k + (int64_t)j * o.sj);
      m = fmax(m, fmax(fabs(v.x), fabs(v.y)) * sc[j]);  // a row with a NaN or an infinity has scale 0: skipped
    }
  }
  b_max[q][kl] = m;
  __syncthreads();
  if (q == 0 && k < o.K) {
    for (int w = 1; w < 8; ++w) m = fmax(m, b_max[w][kl]);
    const int e = m >= 1.0 ? min(0, ilogb(m) - (int)kNormBits) : -(int)kNormBits;
    d[k] = ldexp(1.0, e);
    dinv[k] = ldexp(1.0, -e);
  }
}
// 64 rows x 4 K quarters per block, rows contiguous in memory (rows of A in A B).
template <bool BAL>
__device__ __forceinline__ void scale_rows(const Operand& o, int j0, double* sc, double* inv) {
  __shared__ double r_sum[4][64], r_max[4][64];
  const int jl = threadIdx.x & 63, q = threadIdx.x >> 6, j = j0 + jl;
  double ssq = 0.0, amax = 0.0;
  if (j < o.rows) {
    const double2* x = o.X + j;
#pragma unroll 8
    for (int k = q; k < o.K; k += 4) {
      const double2 v = o.template balanced<BAL>(__ldg(x + (int64_t)k * o.sk), k);
      ssq = fma(v.x, v.x, fma(v.y, v.y, ssq));
      amax = fmax(amax, fmax(fabs(v.x), fabs(v.y)));
    }
  }
  r_sum[q][jl] = ssq;
  r_max[q][jl] = amax;
  __syncthreads();
  if (q == 0 && j < o.rows) {
    for (int w = 1; w < 4; ++w) {
      ssq += r_sum[w][jl];
      amax = fmax(amax, r_max[w][jl]);
    }
    scale_of(ssq, amax, o.K, sc + j, inv + j);
  }
}

// --------------------------------------------------------------------- split
// A thread takes 8 consecutive K values of one panel row (two neighbouring threads share a
// 16-byte chunk): integers v = rint(x scale) with |v| < 2^59, their eight bytes (of
// v + 2^63) against the powers of 256 modulo p by dp4a (real part w, imaginary part r w),
// z+- = a +- r b, one rounded multiple of p taken off through a float, and one 8-byte store
// per plane.  Bound by these ~14 integer and float operations per value and modulus (0.59 of the
// copy rate; 64 registers with a small spill, for two 512-thread blocks per SM).
__device__ __forceinline__ unsigned pack4(const unsigned* b) {  // low bytes of four words
  return __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
}
template <bool BAL>
__device__ __forceinline__ void split_rows(const Operand& o, bool conj, int R, int rt, int rt_n, int ktc,
                                           const double* __restrict__ scale, unsigned char* panel) {
  const int r = threadIdx.x >> 1, h = threadIdx.x & 1;
  if (r >= R) return;
  const int j = rt * R + r;
  const int chunks = 4 * ((o.K + kTileK - 1) / kTileK);
  const double sc = j < o.rows ? scale[j] : 0.0;
  const size_t plane = (size_t)rt_n * ktc * ((size_t)R * kTileK);
  for (int q = blockIdx.x; q < chunks; q += gridDim.x) {
    const int k0 = 16 * q + 8 * h;
    double2 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      x[u] = make_double2(0.0, 0.0);
      if (j < o.rows && k0 + u < o.K)
        x[u] = o.template balanced<BAL>(__ldg(o.X + (int64_t)(k0 + u) * o.sk + (int64_t)j * o.sj), k0 + u);
    }
    unsigned al[8], ah[8], bl[8], bh[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const unsigned long long a = (unsigned long long)__double2ll_rn(x[u].x * sc) ^ (1ull << 63);
      const unsigned long long b = (unsigned long long)__double2ll_rn(x[u].y * sc) ^ (1ull << 63);
      al[u] = (unsigned)a;
      ah[u] = (unsigned)(a >> 32);
      bl[u] = (unsigned)b;
      bh[u] = (unsigned)(b >> 32);
    }
    unsigned char* dst =
        panel + ((size_t)rt * ktc + (q >> 2)) * ((size_t)R * kTileK) + ((size_t)(q & 3) * R + r) * 16 + 8 * h;
#pragma unroll 2
    for (int i = 0; i < kModuli; ++i) {
      const unsigned wlo = c_tab.wlo[i], whi = c_tab.whi[i], rlo = c_tab.rlo[i], rhi = c_tab.rhi[i];
      const int ca = c_tab.ca[i] + (int)kMagic, cb = c_tab.cb[i], p = c_tab.p[i];
      const float inv = c_tab.inv[i];
      unsigned bp[8], bm[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int a = dp4a_us(al[u], wlo, dp4a_us(ah[u], whi, ca));
        const int b = dp4a_us(bl[u], rlo, dp4a_us(bh[u], rhi, cb));
        const int xp = a + b, xm = a - b;
        const int qp = __float_as_int(fmaf(__int_as_float(xp) - kMagicF, inv, kMagicF));
        const int qm = __float_as_int(fmaf(__int_as_float(xm) - kMagicF, inv, kMagicF));
        bp[u] = (unsigned)(xp - qp * p);
        bm[u] = (unsigned)(xm - qm * p);
      }
      *reinterpret_cast<uint2*>(dst + (size_t)(2 * i + (conj ? 1 : 0)) * plane) = make_uint2(pack4(bp), pack4(bp + 4));
      *reinterpret_cast<uint2*>(dst + (size_t)(2 * i + (conj ? 0 : 1)) * plane) = make_uint2(pack4(bm), pack4(bm + 4));
    }
  }
}

// Geometry of a launch's workspace.
struct Geo {
  int ktc;          // K tiles of the launch's own panels
  int a_mt;         // A row tiles of the launch's own panels
  int trb, nt;      // B tile rows, B row tiles
  int ksplit;
  int mpad, n4;     // residue bytes: rows and groups of four columns per plane
  int max_m, max_n;
  size_t a_stride, b_stride, r_stride;  // bytes per descriptor (residues: all splits)
  size_t a_off, b_off, r_off, as_off, bs_off, total;  // byte offsets in the workspace
  int max_k;        // balance of K (kNN, A split with the launch): d and 1 / d per K index
  size_t bal_off;   // 0: none
};
__device__ __forceinline__ double* balance_of(const Geo& g, unsigned char* work, int z) {
  return reinterpret_cast<double*>(work + g.bal_off) + 2 * (size_t)z * g.max_k;
}

// BAL: with the balance of K (the second pass over B)
template <bool BAL>
__global__ void __launch_bounds__(256) k_rns_scale_cols(const Desc* __restrict__ descs, int mode, int which, Geo g,
                                                        unsigned char* work) {
  const Desc d = descs[blockIdx.y];
  if (d.M <= 0 || d.N <= 0 || d.K <= 0 || (which == 0 && d.a_panel)) return;
  Operand o = operand_of(d, mode, which);
  if ((int)blockIdx.x >= o.rows) return;
  if (BAL) o.bal = balance_of(g, work, blockIdx.y) + g.max_k;
  const int cap = which == 0 ? g.max_m : g.max_n;
  double* sc = reinterpret_cast<double*>(work + (which == 0 ? g.as_off : g.bs_off)) + 2 * (size_t)blockIdx.y * cap;
  scale_cols<BAL>(o, blockIdx.x, sc, sc + cap);
}
__global__ void __launch_bounds__(256) k_rns_scale_rows(const Desc* __restrict__ descs, int mode, Geo g,
                                                        unsigned char* work) {
  const Desc d = descs[blockIdx.y];
  if (d.M <= 0 || d.N <= 0 || d.K <= 0 || d.a_panel) return;
  Operand o = operand_of(d, mode, 0);
  if ((int)blockIdx.x * 64 >= o.rows) return;
  o.bal = balance_of(g, work, blockIdx.y);
  double* sc = reinterpret_cast<double*>(work + g.as_off) + 2 * (size_t)blockIdx.y * g.max_m;
  scale_rows<true>(o, blockIdx.x * 64, sc, sc + g.max_m);
}
__global__ void __launch_bounds__(256) k_rns_balance(const Desc* __restrict__ descs, int mode, Geo g,
                                                     unsigned char* work) {
  const Desc d = descs[blockIdx.y];
  if (d.M <= 0 || d.N <= 0 || d.K <= 0 || (int)blockIdx.x * 32 >= d.K) return;
  const double* sc = reinterpret_cast<const double*>(work + g.bs_off) + 2 * (size_t)blockIdx.y * g.max_n;
  double* bal = balance_of(g, work, blockIdx.y);
  balance(operand_of(d, mode, 1), sc, bal, bal + g.max_k);
}
__global__ void __launch_bounds__(256) k_rns_scale_args(Operand o, int by_rows, double* sc, double* inv) {
  if (by_rows)
    scale_rows<false>(o, blockIdx.x * 64, sc, inv);
  else
    scale_cols<false>(o, blockIdx.x, sc, inv);
}

template <bool BAL>
__global__ void __launch_bounds__(512, 2) k_rns_split(const Desc* __restrict__ descs, int mode, int which, Geo g,
                                                      unsigned char* work) {
  const Desc d = descs[blockIdx.z];
  if (d.M <= 0 || d.N <= 0 || d.K <= 0 || (which == 0 && d.a_panel)) return;
  Operand o = operand_of(d, mode, which);
  if (BAL) o.bal = balance_of(g, work, blockIdx.z) + (which == 0 ? 0 : g.max_k);
  const int R = which == 0 ? kTileM : g.trb, rt_n = which == 0 ? g.a_mt : g.nt;
  if ((int)blockIdx.y * R >= o.rows) return;
  const int cap = which == 0 ? g.max_m : g.max_n;
  const double* sc =
      reinterpret_cast<const double*>(work + (which == 0 ? g.as_off : g.bs_off)) + 2 * (size_t)blockIdx.z * cap;
  unsigned char* panel = work + (which == 0 ? g.a_off + blockIdx.z * g.a_stride : g.b_off + blockIdx.z * g.b_stride);
  split_rows<BAL>(o, which == 0 && mode == kTN, R, blockIdx.y, rt_n, g.ktc, sc, panel);
}
__global__ void __launch_bounds__(512, 2) k_rns_split_args(Operand o, int conj, int rt_n, int ktc,
                                                           const double* __restrict__ sc, unsigned char* panel) {
  split_rows<false>(o, conj != 0, kTileM, blockIdx.y, rt_n, ktc, sc, panel);
}

// --------------------------------------------------------------------- product
// The K-tile range of split y (the last splits may be empty).
__device__ __host__ __forceinline__ void split_range(int kt, int ksplit, int y, int* kb, int* ke) {
  const int chunk = (kt + ksplit - 1) / ksplit;
  *kb = min(kt, y * chunk);
  *ke = min(kt, *kb + chunk);
}

// A work item: 256 x trb outputs of one plane, K split and descriptor.
struct Item {
  int z, plane, split, mt, nt, kb, ke, halves;
};

__device__ __forceinline__ bool item_at(int idx, const int* prefix, int ndesc, const int* dm, const int* dn,
                                        const int* dk, int trb, int ksplit, int* zc, Item* it) {
  int z = *zc;
  while (z < ndesc && idx >= prefix[z + 1]) ++z;
  *zc = z;
  if (z >= ndesc) return false;
  const int mt2 = (dm[z] + 2 * kTileM - 1) / (2 * kTileM), nt = (dn[z] + trb - 1) / trb;
  int q = idx - prefix[z];
  it->z = z;
  it->nt = q % nt;
  q /= nt;
  it->mt = 2 * (q % mt2);
  q /= mt2;
  it->split = q % ksplit;
  it->plane = q / ksplit;
  split_range((dk[z] + kTileK - 1) / kTileK, ksplit, it->split, &it->kb, &it->ke);
  it->halves = dm[z] - it->mt * kTileM > kTileM ? 2 : 1;
  return true;
}

// 16 int32 accumulator columns of this warp's 32 tensor-memory lanes.
__device__ __forceinline__ void tmem_load(int (&x)[16], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]), "=r"(x[8]),
        "=r"(x[9]), "=r"(x[10]), "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
      : "r"(taddr));
}
// x modulo p as signed bytes, four columns per 32-bit store.  SHORT (|x| < 2^24): quotient
// from floor(x / 4) in a float's mantissa, remainder within 125 of zero; otherwise the high
// half is folded first (|y| < 2^22).
template <bool SHORT>
__device__ __forceinline__ void reduce_store(const int (&x)[16], int p, int c16, float inv, uint32_t* out, int mpad) {
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    unsigned b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int v = x[4 * w + e];
      const int y = SHORT ? (v >> 2) + (int)kMagic : (v >> 16) * c16 + (int)((unsigned)(v & 0xffff) | kMagic);
      const int q = __float_as_int(fmaf(__int_as_float(y) - kMagicF, inv, kMagicF));
      b[e] = (unsigned)((SHORT ? v : y) - q * p);
    }
    out[(size_t)w * mpad] = pack4(b);
  }
}

// Two roles feed eight epilogue warps: thread 0 streams the K tiles of its items through a
// ring of kStages stages with bulk copies and runs ahead into the next item; thread 32
// issues the MMAs (two 128-row halves share each B tile: 64 bytes of L2 traffic per SM and
// cycle at the full int8 rate, where a single 128-row tile would need 96); the epilogue
// warps reduce the int32 accumulators modulo p and store bytes.  With trb <= 128 the
// accumulator is double buffered in tensor memory.  Every wait is bounded (the roles' by
// `limit` tries); a role that gives up stops the block, which waits (bounded by kWaitLimit) for
// its own copies and MMAs, frees its tensor memory and sets the error word.  SHORT: K 121^2 < 2^24 (a cheaper
// reduction).  256 x 256 tiles measured 0.94 and 1.38 ms (kTN, kNN at Si216) where 256 x 128
// double-buffered ones took 1.55 and 1.74 ms; loading the next columns during the reduction
// took 0.94 and 1.38 to 0.87 and 1.07 ms.
template <bool SHORT>
__global__ void __launch_bounds__(kMmaThreads, 1)
    k_rns_mma(const Desc* __restrict__ descs, int ndesc, Geo g, unsigned char* work, int* err, unsigned limit) {
  extern __shared__ unsigned char dyn[];
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail, s_issued, s_consumed, s_done, s_bad;
  __shared__ int s_prefix[kMaxDesc + 1], s_m[kMaxDesc], s_n[kMaxDesc], s_k[kMaxDesc];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int trb = g.trb;
  const int nbuf = trb <= 128 ? 2 : 1;
  uint32_t acc_cols = 32;  // tensor-memory columns of one 128-row half
  while (acc_cols < (uint32_t)trb) acc_cols <<= 1;
  const uint32_t tcols = acc_cols * 2 * nbuf;
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(dyn) + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_addr(base);
  constexpr uint32_t abytes = kTileM * kTileK;
  const uint32_t bbytes = (uint32_t)trb * kTileK, sstage = 2 * abytes + bbytes;

  for (int z = tid; z < ndesc; z += kMmaThreads) {
    const Desc* d = descs + z;
    const bool live = d->M > 0 && d->N > 0 && d->K > 0;
    s_m[z] = live ? d->M : 0;
    s_n[z] = live ? d->N : 0;
    s_k[z] = live ? d->K : 0;
  }
  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(smem_addr(&full[s]), 1);
      mbar_init(smem_addr(&empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_addr(&tfull[b]), 1);
      mbar_init(smem_addr(&tempty[b]), 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = s_issued = s_consumed = s_done = s_bad = 0;
  }
  __syncthreads();
  if (tid == 0) {
    int n = 0;
    for (int z = 0; z < ndesc; ++z) {
      s_prefix[z] = n;
      if (s_m[z] > 0) {
        n += kPlanes * g.ksplit * ((s_m[z] + 2 * kTileM - 1) / (2 * kTileM)) * ((s_n[z] + trb - 1) / trb);
        if (!descs[z].a_panel && g.a_stride == 0) s_bad = 1;  // a launch for split A given a descriptor without
      }
    }
    s_prefix[ndesc] = n;
  }
  __syncthreads();
  if (s_bad) {
    if (tid == 0) atomicOr(err, kErrBit);
    return;
  }
  if (s_prefix[ndesc] <= (int)blockIdx.x) return;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&tmem_slot)),
                 "r"(tcols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  volatile int* failed = &s_fail;

  if (tid == 0) {  // producer
    int t = 0, zc = 0;
    Item it;
    for (int idx = blockIdx.x; item_at(idx, s_prefix, ndesc, s_m, s_n, s_k, trb, g.ksplit, &zc, &it) && !*failed;
         idx += gridDim.x) {
      const Desc* d = descs + it.z;
      const unsigned char* ap = d->a_panel;
      const int akt = ap ? d->a_kt : g.ktc, amt = ap ? (d->M + kTileM - 1) / kTileM : g.a_mt;
      if (!ap) ap = work + g.a_off + it.z * g.a_stride;
      const unsigned char* a0 = ap + (((size_t)it.plane * amt + it.mt) * akt + it.kb) * abytes;
      const unsigned char* a1 = a0 + (size_t)akt * abytes;
      const unsigned char* b0 =
          work + g.b_off + it.z * g.b_stride + (((size_t)it.plane * g.nt + it.nt) * g.ktc + it.kb) * bbytes;
      for (int k = 0; k < it.ke - it.kb; ++k, ++t) {
        const int s = t % kStages;
        if (t >= kStages && !mbar_wait(smem_addr(&empty[s]), (uint32_t)((t / kStages - 1) & 1), failed, limit)) {
          s_fail = 1;
          break;
        }
        const uint32_t sa = sbase + s * sstage, mb = smem_addr(&full[s]);
        mbar_expect_tx(mb, it.halves * abytes + bbytes);
        bulk_copy(sa, a0 + (size_t)k * abytes, abytes, mb);
        if (it.halves == 2) bulk_copy(sa + abytes, a1 + (size_t)k * abytes, abytes, mb);
        bulk_copy(sa + 2 * abytes, b0 + (size_t)k * bbytes, bbytes, mb);
      }
    }
    s_issued = t;
  } else if (tid == 32) {  // MMA issuer
    int t = 0, zc = 0, n = 0;
    Item it;
    bool ok = true;
    for (int idx = blockIdx.x; ok && item_at(idx, s_prefix, ndesc, s_m, s_n, s_k, trb, g.ksplit, &zc, &it);
         idx += gridDim.x) {
      if (it.ke <= it.kb) continue;
      const int buf = n % nbuf, use = n / nbuf;
      const int ncols = min(trb, s_n[it.z] - it.nt * trb);
      const uint32_t id = idesc((ncols + 15) / 16 * 16);
      if (use > 0 && !mbar_wait(smem_addr(&tempty[buf]), (uint32_t)((use - 1) & 1), failed, limit)) {
        s_fail = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + (uint32_t)buf * 2 * acc_cols;
      for (int k = 0; k < it.ke - it.kb; ++k, ++t) {
        const int s = t % kStages;
        if (!mbar_wait(smem_addr(&full[s]), (uint32_t)((t / kStages) & 1), failed, limit)) {
          s_fail = 1;
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t sa = sbase + s * sstage, sb = sa + 2 * abytes;
        const uint32_t achunk = kTileM * 16, bchunk = (uint32_t)trb * 16;
#pragma unroll
        for (int ks = 0; ks < kTileK / 32; ++ks) {
          const uint64_t bd = sdesc(sb + 2 * ks * bchunk, bchunk, 128);
          mma_i8(acc, sdesc(sa + 2 * ks * achunk, achunk, 128), bd, id, (k > 0 || ks > 0) ? 1u : 0u);
          if (it.halves == 2)
            mma_i8(acc + acc_cols, sdesc(sa + abytes + 2 * ks * achunk, achunk, 128), bd, id,
                   (k > 0 || ks > 0) ? 1u : 0u);
        }
        commit(smem_addr(&empty[s]));
      }
      if (!ok) break;
      commit(smem_addr(&tfull[buf]));
      ++n;
    }
    s_consumed = t;
    s_done = n;
  } else if (warp >= 2) {  // epilogue: warps 2-5 the first 128 rows, 6-9 the second
    const int half = (warp - 2) >> 2, quad = warp & 3;
    int zc = 0, n = 0;
    Item it;
    for (int idx = blockIdx.x; item_at(idx, s_prefix, ndesc, s_m, s_n, s_k, trb, g.ksplit, &zc, &it);
         idx += gridDim.x) {
      if (it.ke <= it.kb) continue;
      const int buf = n % nbuf, use = n / nbuf;
      ++n;
      bool ok = true;
      if (lane == 0) ok = mbar_wait(smem_addr(&tfull[buf]), (uint32_t)(use & 1), failed, limit);
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
      if (!ok) {
        if (lane == 0) s_fail = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (half < it.halves) {
        const int ncols = min(trb, s_n[it.z] - it.nt * trb);
        const int row = (it.mt + half) * kTileM + 32 * quad + lane;
        const int mod = it.plane >> 1;
        const int p = c_tab.p[mod], c16 = c_tab.c16[mod];
        const float inv = SHORT ? 4.0f * c_tab.inv[mod] : c_tab.inv[mod];
        uint32_t* out = reinterpret_cast<uint32_t*>(work + g.r_off + it.z * g.r_stride) +
                        (((size_t)it.split * kPlanes + it.plane) * g.n4 + (size_t)it.nt * (trb / 4)) * g.mpad + row;
        const uint32_t taddr = tmem + (uint32_t)(buf * 2 + half) * acc_cols + ((uint32_t)(32 * quad) << 16);
        // the next 16 columns are on their way while these are reduced; rows and columns
        // beyond M and N are padding that nothing reads
        int x[2][16];
        tmem_load(x[0], taddr);
        for (int n0 = 0; n0 < ncols; n0 += 32) {
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int nq = n0 + 16 * q;
            if (nq < ncols) {
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
              if (nq + 16 < ncols) tmem_load(x[q ^ 1], taddr + (uint32_t)(nq + 16));
              reduce_store<SHORT>(x[q], p, c16, inv, out, g.mpad);
              out += 4 * (size_t)g.mpad;
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_addr(&tempty[buf]));
    }
  }
  __syncthreads();
  if (s_fail) {
    // copies in flight land in the ring before the block ends; MMAs finish (their commits)
    __shared__ int s_none;
    if (tid == 0) {
      s_none = 0;
      for (int t = s_consumed; t < s_issued; ++t)
        mbar_wait(smem_addr(&full[t % kStages]), (uint32_t)((t / kStages) & 1), &s_none, kWaitLimit);
      if (s_consumed > 0) {
        const int t = s_consumed - 1;
        mbar_wait(smem_addr(&empty[t % kStages]), (uint32_t)((t / kStages) & 1), &s_none, kWaitLimit);
      }
      atomicOr(err, kErrBit);
    }
    __syncthreads();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tcols));
}

// --------------------------------------------------------------------- reconstruction
// One thread per row and four columns: for every modulus the sums z+ and z- over the K
// splits, real part (z+ + z-) and imaginary part (z+ - z-) times their CRT weights modulo
// 1.  The weights' high parts are multiples of 2^-36, so their sum is exact in FP64
// (|z| < 2^13, 16 terms) and its nearest integer comes off exactly; the low parts add
// 2^-74 of error, far below the operands' rounding.  The fraction times the moduli's
// product and the inverse scales is the output.  Six FP64 operations per modulus and
// complex output: a third of the time of 96-bit integer sums (IMAD.WIDE).
template <int MODE>
__global__ void __launch_bounds__(128) k_rns_join(const Desc* __restrict__ descs, Geo g,
                                                  const unsigned char* __restrict__ work) {
  const Desc d = descs[blockIdx.y];
  if (d.M <= 0 || d.N <= 0 || d.K <= 0) return;
  const int row_blocks = (d.M + 127) / 128, items = row_blocks * ((d.N + 3) / 4);
  int used = 1;
  if (MODE == kTN) {
    const int kt = (d.K + kTileK - 1) / kTileK, chunk = (kt + g.ksplit - 1) / g.ksplit;
    used = (kt + chunk - 1) / chunk;
  }
  const size_t plane = (size_t)g.n4 * g.mpad;
  // int -> double: the integer (biased to stay positive) in the low word of 2^52 + n
  const int bias = 256 * used;
  const double shift = 4503599627370496.0 + (double)bias;
  const double* ainv = d.a_panel ? d.a_inv
                                 : reinterpret_cast<const double*>(work + g.as_off) +
                                       2 * (size_t)blockIdx.y * g.max_m + g.max_m;
  const double* binv = reinterpret_cast<const double*>(work + g.bs_off) + 2 * (size_t)blockIdx.y * g.max_n + g.max_n;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int jc = item / row_blocks, row = (item - jc * row_blocks) * 128 + threadIdx.x;
    if (row >= d.M) continue;
    const uint32_t* r = reinterpret_cast<const uint32_t*>(work + g.r_off + blockIdx.y * g.r_stride) +
                        (size_t)jc * g.mpad + row;
    double reh[4], rel[4], imh[4], iml[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) reh[c] = rel[c] = imh[c] = iml[c] = 0.0;
#pragma unroll 4
    for (int i = 0; i < kModuli; ++i) {
      int zp[4], zm[4];
      if (MODE == kNN) {
        const uint32_t vp = __ldg(r + (size_t)(2 * i) * plane) ^ 0x80808080u;
        const uint32_t vm = __ldg(r + (size_t)(2 * i + 1) * plane) ^ 0x80808080u;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          zp[c] = (int)((vp >> (8 * c)) & 0xffu);
          zm[c] = (int)((vm >> (8 * c)) & 0xffu);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) zp[c] = zm[c] = 128 * used;
        for (int y = 0; y < used; ++y) {
          const uint32_t vp = __ldg(r + ((size_t)y * kPlanes + 2 * i) * plane);
          const uint32_t vm = __ldg(r + ((size_t)y * kPlanes + 2 * i + 1) * plane);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            zp[c] += (int)(signed char)(vp >> (8 * c));
            zm[c] += (int)(signed char)(vm >> (8 * c));
          }
        }
      }
      const double wrh = c_tab.reh[i], wrl = c_tab.rel[i], wih = c_tab.imh[i], wil = c_tab.iml[i];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const double sp = __hiloint2double(0x43300000, zp[c] + zm[c]) - shift;
        const double sm = __hiloint2double(0x43300000, zp[c] - zm[c] + bias) - shift;
        reh[c] = fma(sp, wrh, reh[c]);
        rel[c] = fma(sp, wrl, rel[c]);
        imh[c] = fma(sm, wih, imh[c]);
        iml[c] = fma(sm, wil, iml[c]);
      }
    }
    const double ai = ainv[row];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int j = 4 * jc + c;
      if (j >= d.N) break;
      const double fr = (reh[c] - rint(reh[c])) + rel[c], fi = (imh[c] - rint(imh[c])) + iml[c];
      // the smaller scale first: no overflow before the larger one (a NaN reaches the product)
      const double bj = binv[j], s1 = ai < bj ? ai : bj, s2 = ai < bj ? bj : ai;
      const double vr = fma(fr, c_tab.mlo, fr * c_tab.mhi) * s1 * s2;
      const double vi = fma(fi, c_tab.mlo, fi * c_tab.mhi) * s1 * s2;
      double2* out = d.C + row + (int64_t)j * d.ldc;
      if (d.op == kStore) {
        *out = make_double2(vr, vi);
      } else {
        const double2 old = *out;
        *out = d.op == kAdd ? make_double2(old.x + vr, old.y + vi) : make_double2(old.x - vr, old.y - vi);
      }
    }
  }
}

inline size_t round256(size_t b) { return (b + 255) / 256 * 256; }

// Splits of K: whole waves of the 148 persistent blocks, at least 16 K tiles each (K within
// the exact int32 range always).  Results do not depend on it.
int pick_ksplit(int mode, int ndesc, int max_m, int max_n, int max_k, int trb) {
  if (mode == kNN) return 1;
  const int64_t items = (int64_t)std::max(ndesc, 1) * kPlanes * ((max_m + 2 * kTileM - 1) / (2 * kTileM)) *
                        ((max_n + trb - 1) / trb);
  const int kt = k_tiles(max_k);
  const int lo = std::max(1, (max_k + kMaxK - 1) / kMaxK), hi = std::max(lo, std::min(16, kt / 16));
  int best = lo;
  double best_eff = 0.0;
  for (int ks = lo; ks <= hi; ++ks) {
    const int64_t n = items * ks, waves = (n + kSms - 1) / kSms;
    const double eff = (double)n / (double)(waves * kSms);
    if (eff > best_eff + 0.02) {
      best_eff = eff;
      best = ks;
    }
    if (eff >= 0.95) break;
  }
  return best;
}

Geo carve(int mode, int ndesc, int max_m, int max_n, int max_k, bool a_presplit, size_t limit = ~(size_t)0) {
  Geo g{};
  g.ktc = k_tiles(max_k);
  g.a_mt = m_tiles(max_m);
  g.nt = (max_n + kTileN - 1) / kTileN;
  g.trb = ((max_n + g.nt - 1) / g.nt + 15) / 16 * 16;
  g.max_m = max_m;
  g.max_n = max_n;
  g.mpad = g.a_mt * kTileM;
  g.n4 = g.nt * g.trb / 4;
  g.a_stride = a_presplit ? 0 : round256(a_panel_bytes(max_m, max_k));
  g.b_stride = round256((size_t)kPlanes * g.nt * g.ktc * g.trb * kTileK);
  size_t o = 0;
  g.a_off = o;
  o += ndesc * g.a_stride;
  g.b_off = o;
  o += ndesc * g.b_stride;
  g.as_off = o;
  o += round256(a_presplit ? 0 : (size_t)ndesc * 2 * max_m * sizeof(double));
  g.bs_off = o;
  o += round256((size_t)ndesc * 2 * max_n * sizeof(double));
  g.max_k = max_k;
  if (mode == kNN && !a_presplit) {
    g.bal_off = o;
    o += round256((size_t)ndesc * 2 * max_k * sizeof(double));
  }
  g.r_off = o;
  const int least = (max_k + kMaxK - 1) / kMaxK;
  for (g.ksplit = pick_ksplit(mode, ndesc, max_m, max_n, max_k, g.trb);; --g.ksplit) {
    g.r_stride = round256((size_t)g.ksplit * kPlanes * g.n4 * g.mpad * 4);
    g.total = o + ndesc * g.r_stride;
    if (g.total <= limit || g.ksplit <= least) break;
  }
  return g;
}

size_t mma_smem(int trb) { return (size_t)kStages * (2 * kTileM * kTileK + (size_t)trb * kTileK) + 1024; }

}  // namespace

size_t workspace_bytes(int mode, int ndesc, int max_m, int max_n, int max_k, bool a_presplit) {
  return carve(mode, ndesc, max_m, max_n, max_k, a_presplit).total;
}

cudaError_t prepare() {
  const int smem = (int)mma_smem(kTileN);
  cudaError_t e = cudaFuncSetAttribute((const void*)k_rns_mma<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute((const void*)k_rns_mma<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  return e;
}

int launch_product(int mode, const Desc* d_desc, int ndesc, int max_m, int max_n, int max_k, bool a_presplit,
                   void* work, size_t work_bytes, int* err, cudaStream_t s, unsigned wait_limit) {
  if (ndesc == 0 || max_m <= 0 || max_n <= 0 || max_k <= 0) return 0;
  const Geo g = carve(mode, ndesc, max_m, max_n, max_k, a_presplit, work_bytes);
  unsigned char* w = static_cast<unsigned char*>(work);
  int launches = 4;
  const unsigned chunks = (unsigned)(4 * g.ktc);
  auto split = [&](unsigned gx, int tiles, int threads, int which) {
    if (g.bal_off)
      k_rns_split<true><<<dim3(gx, tiles, ndesc), threads, 0, s>>>(d_desc, mode, which, g, w);
    else
      k_rns_split<false><<<dim3(gx, tiles, ndesc), threads, 0, s>>>(d_desc, mode, which, g, w);
  };
  if (g.bal_off) {
    k_rns_scale_cols<false><<<dim3(max_n, ndesc), 256, 0, s>>>(d_desc, mode, 1, g, w);
    k_rns_balance<<<dim3((max_k + 31) / 32, ndesc), 256, 0, s>>>(d_desc, mode, g, w);
    launches += 2;
  }
  if (!a_presplit) {
    if (mode == kTN)
      k_rns_scale_cols<false><<<dim3(max_m, ndesc), 256, 0, s>>>(d_desc, mode, 0, g, w);
    else
      k_rns_scale_rows<<<dim3((max_m + 63) / 64, ndesc), 256, 0, s>>>(d_desc, mode, g, w);
    const unsigned gx = std::max(1u, std::min(chunks, 148u * 16 / (unsigned)std::max(1, g.a_mt * ndesc) + 1));
    split(gx, g.a_mt, 2 * kTileM, 0);
    launches += 2;
  }
  if (g.bal_off)
    k_rns_scale_cols<true><<<dim3(max_n, ndesc), 256, 0, s>>>(d_desc, mode, 1, g, w);
  else
    k_rns_scale_cols<false><<<dim3(max_n, ndesc), 256, 0, s>>>(d_desc, mode, 1, g, w);
  {
    const unsigned gx = std::max(1u, std::min(chunks, 148u * 8 / (unsigned)std::max(1, g.nt * ndesc) + 1));
    split(gx, g.nt, 2 * g.trb, 1);
  }
  const int kper = (int)std::min<int64_t>(max_k, (int64_t)kTileK * ((g.ktc + g.ksplit - 1) / g.ksplit));
  if ((int64_t)kper * 121 * 121 < (1 << 24))
    k_rns_mma<true><<<kSms, kMmaThreads, mma_smem(g.trb), s>>>(d_desc, ndesc, g, w, err, wait_limit);
  else
    k_rns_mma<false><<<kSms, kMmaThreads, mma_smem(g.trb), s>>>(d_desc, ndesc, g, w, err, wait_limit);
  const int64_t blocks = (int64_t)((max_m + 127) / 128) * ((max_n + 3) / 4);
  const dim3 jg((unsigned)std::min<int64_t>(blocks, std::max(148, kSms * 24 / ndesc)), ndesc);
  if (mode == kTN)
    k_rns_join<kTN><<<jg, 128, 0, s>>>(d_desc, g, w);
  else
    k_rns_join<kNN><<<jg, 128, 0, s>>>(d_desc, g, w);
  return launches;
}

cudaError_t split_a(int mode, const double2* A, int64_t lda, int M, int K, unsigned char* panel, double* scale,
                    double* inv, cudaStream_t s) {
  if (M <= 0 || K <= 0) return cudaSuccess;
  Operand o;
  o.X = A;
  o.rows = M;
  o.K = K;
  o.sk = mode == kTN ? 1 : lda;
  o.sj = mode == kTN ? lda : 1;
  k_rns_scale_args<<<mode == kTN ? M : (M + 63) / 64, 256, 0, s>>>(o, mode == kTN ? 0 : 1, scale, inv);
  const int mt = m_tiles(M), kt = k_tiles(K);
  const unsigned gx = std::max(1u, std::min((unsigned)(4 * kt), 148u * 16 / (unsigned)mt + 1));
  k_rns_split_args<<<dim3(gx, mt), 2 * kTileM, 0, s>>>(o, mode == kTN ? 1 : 0, mt, kt, scale, panel);
  return cudaGetLastError();
}

}  // namespace rns
}  // namespace bg

// ------------------------------------------------------------------ test entries
#include "../../include/baandi_gpu_test.h"
#include "op_internal.h"

using namespace bg;

extern "C" int bg_test_residue_products(int32_t mode, int32_t count, const int64_t* shapes, const double* const* a,
                                        const int64_t* lda, const double* const* b, const int64_t* ldb,
                                        double* const* c, const int64_t* ldc, int32_t op, int32_t presplit,
                                        const int64_t* bounds, int64_t wait_limit) {
  using namespace bg::rns;
  if (count < 1 || count > kMaxDesc || !shapes || !a || !b || !c || !lda || !ldb || !ldc) return BG_EINVAL;
  int64_t top[3] = {0, 0, 0};
  for (int z = 0; z < count; ++z)
    for (int i = 0; i < 3; ++i) top[i] = std::max(top[i], shapes[3 * z + i]);
  std::vector<Desc> h(count);
  std::vector<DevBuf> panel(count), scale(count);
  DevBuf desc, err, work;
  auto alloc = [](DevBuf* x, size_t bytes) { return cudaMalloc(&x->p, bytes) == cudaSuccess; };
  size_t wb = 0;
  if (bounds)
    wb = workspace_bytes(mode, count, (int)bounds[0], (int)bounds[1], (int)bounds[2], presplit != 0);
  else
    wb = workspace_bytes(mode, count, (int)top[0], (int)top[1], (int)top[2], presplit != 0);
  if (prepare() != cudaSuccess || !alloc(&desc, sizeof(Desc) * count) || !alloc(&err, sizeof(int)) || !alloc(&work, wb))
    return BG_ENOMEM;
  for (int z = 0; z < count; ++z) {
    const int64_t m = shapes[3 * z], n = shapes[3 * z + 1], k = shapes[3 * z + 2];
    h[z] = Desc{reinterpret_cast<const double2*>(a[z]), reinterpret_cast<const double2*>(b[z]),
                reinterpret_cast<double2*>(c[z]), lda[z], ldb[z], ldc[z], (int)m, (int)n, (int)k, op};
    if (!presplit || m <= 0 || k <= 0) continue;
    if (!alloc(&scale[z], 2 * sizeof(double) * m) || !alloc(&panel[z], a_panel_bytes(m, k))) return BG_ENOMEM;
    double* s = static_cast<double*>(scale[z].p);
    if (split_a(mode, h[z].A, lda[z], (int)m, (int)k, static_cast<unsigned char*>(panel[z].p), s, s + m, nullptr) !=
        cudaSuccess)
      return BG_EDEVICE;
    h[z].a_panel = static_cast<const unsigned char*>(panel[z].p);
    h[z].a_inv = s + m;
    h[z].a_kt = k_tiles(k);
  }
  int word = 0;
  if (cudaMemset(err.p, 0, sizeof(int)) != cudaSuccess ||
      cudaMemcpy(desc.p, h.data(), sizeof(Desc) * count, cudaMemcpyHostToDevice) != cudaSuccess)
    return BG_EDEVICE;
  launch_product(mode, static_cast<Desc*>(desc.p), count, (int)top[0], (int)top[1], (int)top[2], presplit != 0, work.p,
                 wb, static_cast<int*>(err.p), nullptr, wait_limit < 0 ? kWaitLimit : (unsigned)wait_limit);
  if (cudaGetLastError() != cudaSuccess || cudaMemcpy(&word, err.p, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
    return BG_EDEVICE;
  return word ? BG_ETIMEOUT : BG_OK;
}

extern "C" int bg_test_residue_product(int32_t mode, int64_t m, int64_t n, int64_t k, const double* a, int64_t lda,
                                       const double* b, int64_t ldb, double* c, int64_t ldc, int32_t op,
                                       int32_t presplit) {
  const int64_t shape[3] = {m, n, k};
  return bg_test_residue_products(mode, 1, shape, &a, &lda, &b, &ldb, &c, &ldc, op, presplit, nullptr, -1);
}
