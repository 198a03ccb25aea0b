/*
 * forge_gpu_selftest.h -- test hooks of libforge_gpu.so (not part of the drop-in boundary).
 *
 * Internal steps of the engine exposed for the test suite; no reference routine corresponds to
 * them and a host application has no use for them.
 */
#ifndef FORGE_GPU_SELFTEST_H
#define FORGE_GPU_SELFTEST_H

#include <stdint.h>

#include "forge_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* D = A B^T on the tcgen05 tensor cores with TF32 inputs and FP32 accumulation; A (batch x M x K),
 * B (batch x N x K), D (batch x M x N), all row-major fp32 host arrays. */
int forge_gpu_selftest_tc_gemm(int64_t M, int64_t N, int64_t K, int64_t batch, const float* A, const float* B,
                               float* D);

/* The same GEMM (batch 1) with a failure injected: the TMA producer issues only K block 0, so the
 * MMA issuer's wait for block 1 runs out after spin_limit polls (1..2^26); the kernel flags the
 * error, drains its copies and MMAs, frees its TMEM and returns.  Returns FORGE_ERR_TIMEOUT; the
 * context stays usable.  K must exceed 32. */
int forge_gpu_selftest_tc_gemm_timeout(int64_t M, int64_t N, int64_t K, int64_t spin_limit, const float* A,
                                       const float* B, float* D);

/* Host only: the small dense step of the window refinement.  G, S: n x n Hermitian (complex,
 * column-major, interleaved re/im doubles), n <= 32.  Returns theta (ascending) and M = L^{-H} U,
 * with S = L L^H and L^{-1} G L^{-H} = U diag(theta) U^H, so that G M = S M diag(theta) and
 * M^H S M = I.  Returns 1 if S is not positive definite. */
int forge_selftest_rr_small(int64_t n, const double* G, const double* S, double* theta, double* M);

/* Bytes that one launch of the eigenpair refinement and one of the sliced projectors may take (4 GB and 2 GB by
 * default), so that small cases run several; results do not depend on them. */
int forge_gpu_selftest_launch_bytes(forge_ctx* ctx, int64_t refinement, int64_t projectors);

/* The context's next `solves` FP64 eigen-solves and `projectors` batches of projectors report, once their work is
 * done, that a bounded wait gave up (FORGE_ERR_TIMEOUT); each is tried a second time. */
int forge_gpu_selftest_timeouts(forge_ctx* ctx, int64_t solves, int64_t projectors);

/* Numbers of eigenvalues <= x[q] of the tridiagonal (d, e), |T| <= 1, by the minors' Sturm counts of
 * the tridiagonal solver in FP64 and in FP32. */
int forge_gpu_selftest_sturm(int64_t n, const double* d, const double* e, int64_t nx, const double* x, int* c64,
                             int* c32);

/* The tridiagonal solver's division by FMAs against the compiler's on at least `count` pairs of random
 * operands over the exponents that it admits: out[0] pairs tried, out[1] different results, out[2]
 * results off by more than a unit in the last place. */
int forge_gpu_selftest_quot(int64_t seed, int64_t count, int64_t* out);

/* Host only: workspace of a batched eigen-solve.  out[0]: bytes; out[1], out[2]: K-split partial
 * products that a solve of this batch forms and the room for them; out[3], out[4]: the same of the
 * mixed solver's second split product (0 in FP64). */
int forge_selftest_eig_workspace(int64_t n, int64_t iu, int64_t batch, int mixed, int64_t* out);

#ifdef __cplusplus
}
#endif
#endif /* FORGE_GPU_SELFTEST_H */
