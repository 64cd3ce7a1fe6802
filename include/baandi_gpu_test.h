/* Entry points of libbaandi_b200 for its own tests: single stages, and conditions that a
 * calling program cannot bring about (a pipeline wait that gives up, short memory).  Not part
 * of the interface of baandi_gpu.h. */
#ifndef BAANDI_GPU_TEST_H
#define BAANDI_GPU_TEST_H

#include "baandi_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* One FP64 residue product of device matrices (column-major interleaved complex, as
 * bg_zgemm_bf16x3): c (op 0 =, 1 +=, 2 -=) a^H b (mode 0) or a b (mode 1).  presplit: a goes
 * through its residue panels first. */
int bg_test_residue_product(int32_t mode, int64_t m, int64_t n, int64_t k, const double* a, int64_t lda,
                            const double* b, int64_t ldb, double* c, int64_t ldc, int32_t op, int32_t presplit);

/* `count` products in one launch, shapes[3 z ..] = m, n, k of product z (0: an empty slot).
 * bounds (or NULL): m, n, k that the workspace is sized for, at least the largest of the
 * shapes.  wait_limit: tries of the pipeline's waits (negative: the library's own).  Returns
 * BG_ETIMEOUT when a wait gave up. */
int bg_test_residue_products(int32_t mode, int32_t count, const int64_t* shapes, const double* const* a,
                             const int64_t* lda, const double* const* b, const int64_t* ldb, double* const* c,
                             const int64_t* ldc, int32_t op, int32_t presplit, const int64_t* bounds,
                             int64_t wait_limit);

/* Bytes of the slices that a band density of the operator or the set (either may be NULL) forms
 * before it sums them; at least one unit's are formed. */
int bg_test_density_budget(bg_op* op, bg_kset* set, int64_t bytes);

/* Short memory: what the library takes for free device memory at most when it decides on buffers
 * that only make calls faster (negative: what the device says), and how many of the next
 * allocations of a batched Davidson solver fail. */
int bg_test_memory(bg_ctx* ctx, int64_t free_bytes, int32_t failures);

/* Whether the operator holds residue panels of its projectors, and whether the set's last solve
 * formed its large products as residue products (either output may be NULL). */
int bg_test_residue_state(const bg_op* op, const bg_kset* set, int32_t* panels, int32_t* products);

/* Set bits of the operator's device error word, as a kernel that met the error would. */
int bg_test_raise_error(bg_op* op, int32_t bits);

#ifdef __cplusplus
}
#endif
#endif
