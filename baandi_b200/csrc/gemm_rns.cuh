// Complex FP64 products on the int8 tensor cores (tcgen05 kind::i8) by residue arithmetic.
//
//   kTN  C[M x N] (=, +=, -=) A^H B   A: K x M, B: K x N  (Gram products, projections)
//   kNN  C[M x N] (=, +=, -=) A B     A: M x K, B: K x N  (rotations, back-projection)
//
// tcgen05 has no FP64 kind and the FP64 units (DMMA and DFMA alike) stop at 37 TFLOP/s, so
// the large products are formed as exact integer products instead (the scheme of Ozaki,
// Uchino and Imamura, "Ozaki Scheme II", 2025, over a quadratic residue number system,
// Leung 1981):
//   1. every column of A^H B's operands (every row of A and column of B for A B) is scaled
//      by a power of two so that its 2-norm is at most 2^kNormBits, and rounded to integers
//      (|v| < 2^59);
//   2. the integers are taken modulo kModuli coprime moduli p <= 241 whose prime factors
//      are all 1 mod 4, so -1 has a square root r modulo p and the Gaussian integer a + ib
//      maps to the pair (a + r b, a - r b) mod p, on which a complex product acts component
//      by component: two int8 products per modulus instead of four;
//   3. tcgen05 forms the 2 kModuli int8 products with int32 accumulation, exact for the
//      K ranges used, and its epilogue reduces them modulo p to one byte;
//   4. the Chinese remainder theorem returns the integer of each output from its residues as
//      a fraction of the moduli's product (to 2^-74), which is scaled back to FP64.
// Cauchy-Schwarz bounds every output by the product of the two norms, 2^(2 kNormBits), below
// half the moduli's product, so no output can wrap.  The only rounding is that of step 1, of the
// fraction and of the final FP64 value.  Sums over K are exact; a different K split (it follows
// from the launch's products and workspace) gives other representatives of the same residues and
// with them other last bits of the fraction.
//
// The error is norm-wise: an output is off by about 2^-58 of its row's norm times its column's,
// where an FP64 GEMM is off by a few 2^-53 of sum |a_k| |b_k|.  Taken over a result this is the
// smaller one.  Against 80-bit sums (2-norm, random operands), here and for an FP64 GEMM: 864 x
// 480 x 80,725 A^H B 5.2e-16 and 7.7e-15 (2.0e-16 and 1.0e-14 with rows falling by e^12), 80,725 x
// 480 x 864 A B 1.0e-16 and 1.4e-15, 129 x 16 x 1,000 1.0e-16 and 3.7e-16.  An operand's entries
// below 2^-5 of their row's norm keep fewer than 53 bits, so an output far below the product of
// the norms can be less exact than an FP64 GEMM's: where a row and a column are graded against
// each other.  Rotations have such rows (steep tails of Ritz vectors beside slow tails of
// corrections, joined by small coefficients), so where A is split in the launch of an A B
// product, K is balanced first (k_rns_balance).  Steep and slow tails (e^-q2 and (1 + q2)^-2, q2 to
// 30), coefficients of 1e-8, largest error over sum |a_k| |b_k|: 7e-11 unbalanced, 2e-17 balanced,
// 3e-16 in an FP64 GEMM; with coefficients from 1e-9 to 0.1, column by column, the median relative
// error is 7e-15, 6e-16 and 3e-16, and entries 1e-12 below their row's largest stay less exact here
// (relative 2e-8 against 1e-13).  The balance costs 0.3 % of the Si216 eigenproblem (143.4 -> 143.8
// ms).  One more modulus (three more bits) made it 5 % slower and was not kept.
//
// Si216's projection (864 x 480 x 80,725, P split at build) takes 1.57 ms against the FP64 tiles'
// 9.62 ms: 0.11 ms scales and 0.49 ms residues of x (3.8 TB/s), 0.93 ms products (52 % of the
// int8 peak, bound by the tiles' L2 traffic, 40 bytes per SM and cycle), 0.03 ms
// reconstruction.  Its back-projection takes 1.79 against 8.69 ms: 1.12 ms products, 0.65 ms
// reconstruction (1.2 GB of residues read, y read and written).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "gemm_tc.cuh"

namespace bg {
namespace rns {

using tc::kAdd;
using tc::kNN;
using tc::kStore;
using tc::kSub;
using tc::kTN;

constexpr int kModuli = 16;
constexpr int kPlanes = 2 * kModuli;
constexpr int kTileM = 128;   // A rows per tile (MMA rows)
constexpr int kTileK = 64;    // K values per tile
constexpr int kTileN = 256;   // B rows per tile at most
constexpr int kMaxK = 131072; // int32 accumulation: K 121^2 < 2^31 per split
constexpr int kErrBit = 4;    // error-word bit of a bounded wait that gave up
constexpr unsigned kWaitLimit = 1u << 24;  // tries of a pipeline wait

// One product (device pointers; M = 0 marks an empty slot).
struct Desc {
  const double2* A;
  const double2* B;
  double2* C;
  int64_t lda, ldb, ldc;
  int M, N, K;
  int op;  // kStore, kAdd, kSub
  // A as panels of split_a (then A is not read), the K tiles of that split, 1 / scale of its rows
  const unsigned char* a_panel = nullptr;
  const double* a_inv = nullptr;
  int a_kt = 0;
};

inline int k_tiles(int64_t k) { return (int)((k + kTileK - 1) / kTileK); }
inline int m_tiles(int64_t m) { return (int)((m + kTileM - 1) / kTileM); }
// Panels of an A operand with M rows and depth K, and its scales (scale, 1 / scale per row).
inline size_t a_panel_bytes(int64_t m, int64_t k) {
  return (size_t)kPlanes * m_tiles(m) * k_tiles(k) * (size_t)(kTileM * kTileK);
}

// Whether a product of these dimensions runs faster here than on the FP64 tiles (28 and 31
// TFLOP/s for kTN and kNN).  With A split beforehand the fixed passes cost about 0.1 ms: 256 x
// 160 x 23,847 takes 0.19 ms (kTN and kNN) against 0.28 ms, 256 x 20 x 23,847 0.12 against
// 0.07 ms.  Splitting A costs 15 ps per element against the tiles' 0.29 ps per element and
// column of B, so it needs wide B: 320 x 160 x 23,847 takes 0.35 ms either way, 960 x 100 x
// 80,725 1.9 against 2.2 ms, 960 x 480 x 80,725 2.75 against 10.6 ms.
__host__ __device__ inline bool pays(int64_t m, int64_t n, int64_t k, bool a_presplit) {
  const double work = (double)m * (double)n * (double)k;
  return a_presplit ? m >= 64 && n >= 16 && k >= 64 && work >= 5.0e8 : m >= 96 && n >= 96 && k >= 96 && work >= 1.5e9;
}

// Workspace of one launch: panels and scales of every descriptor's operands (A's only when
// a_presplit is false) and the residue bytes of the outputs.
size_t workspace_bytes(int mode, int ndesc, int max_m, int max_n, int max_k, bool a_presplit);

// Launches over `ndesc` device descriptors: scales, residues, products, reconstruction.
// max_m, max_n, max_k bound every descriptor's dimensions; a_presplit: every non-empty
// descriptor names its A panels.  work: work_bytes at least workspace_bytes of these
// bounds or of larger ones (fewer K splits are used where the splits of the smaller
// product would need more).  err: device word, kErrBit set when a
// bounded wait gives up (after wait_limit tries).  Returns the number of launches.
int launch_product(int mode, const Desc* d_desc, int ndesc, int max_m, int max_n, int max_k, bool a_presplit,
                   void* work, size_t work_bytes, int* err, cudaStream_t s, unsigned wait_limit = kWaitLimit);

// Panels (a_panel_bytes(M, K)) and inverse scales (M doubles) of the A operand of a `mode`
// product (kTN: K x M, kNN: M x K, ld lda); scale: scratch of M doubles.
cudaError_t split_a(int mode, const double2* A, int64_t lda, int M, int K, unsigned char* panel, double* scale,
                    double* inv, cudaStream_t s);

// Kernel attributes (before the first launch, never inside a capture).
cudaError_t prepare();

}  // namespace rns
}  // namespace bg
