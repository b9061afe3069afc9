// Internal launchers shared by the operator entry points and the HOOI drivers.
// All pointers are device pointers; work is queued on ctx->stream.
#pragma once

#include "dt_core.cuh"
#include "dt_orth.cuh"

namespace dt {

// ---- dense FP64 kernels: dt_dense.cu --------------------------------------
// A dense tensor seen around mode n is a 3-way array X[l, i, b] with
// l < L = prod_{m<n} I_m (unit stride), i < I = I_n (stride L) and
// b < B = prod_{m>n} I_m (stride L*I).

// Y[l, j, b] = sum_i M(j, i) * X[l, i, b]   (Y is L x J x B), with
// M(j, i) = M[j*msj + i*msi]: (msj, msi) = (1, J) for a J x I col-major M,
// (I, 1) for the transpose of an I x J col-major factor U.  With `slot` (device
// memory) the kernel takes X's address from there, and X here only says how it
// is aligned: a captured launch then serves every X.
template <class TX>
void ttm_f64(dt_ctx *ctx, const TX *X, int64_t L, int64_t I, int64_t B, const double *M,
             int64_t msj, int64_t msi, int64_t J, double *Y, const void *const *slot = nullptr);

// C[i, j] = sum_{l,b} A[l, i, b] * Bt[l, j, b]   (C is IA x IB col-major).
void ttt_f64(dt_ctx *ctx, const double *A, const double *Bt, int64_t L, int64_t IA,
             int64_t IB, int64_t B, double *C);

// C(I x I) = A_(n) A_(n)^T (ttt_f64 of A with itself) with the split-K partial
// tiles in caller-provided device scratch; allocates nothing.  The number of
// splits is lowered to what fits; one split needs none.
void gram_f64_scratch(dt_ctx *ctx, const double *A, int64_t L, int64_t I, int64_t B, double *C,
                      double *scratch, int64_t scratch_doubles);

// out[0] = sum x[e]^2 (deterministic two-stage reduction).  dtype DT_F64/DT_F32.
void sumsq(dt_ctx *ctx, const void *x, int dtype, int64_t n, double *out);

// y[e] = (double) x[e]
void f32_to_f64(dt_ctx *ctx, const float *x, int64_t n, double *y);

// Column-major C(m x n) = op(A) op(B) (FP64, small and medium sizes).
void gemm_f64(dt_ctx *ctx, int transA, int transB, int64_t m, int64_t n, int64_t k,
              const double *A, int64_t lda, const double *B, int64_t ldb, double *C,
              int64_t ldc, double beta);

// ---- small dense linear algebra: dt_linalg.cu -----------------------------
// Householder QR (LAPACK dgeqrf/dorgqr reflector convention) of the m x n
// col-major A (m >= n).  Q (m x n) and optionally R (n x n).  work >= m*n+n.
void householder_qr(dt_ctx *ctx, const double *A, int64_t m, int64_t n, double *Q,
                    double *R, double *work);

// Orthonormal bases Q[b] of span(A[b]) for a batch of up to 16 matrices
// (CholeskyQR2 on the FP64 tensor-core path, Householder on breakdown or for
// large matrices), one CTA each.
void orth_batch(dt_ctx *ctx, int count, const double *const *A, double *const *Q,
                const int64_t *m, const int64_t *n);

// Orthonormal basis of span(S^iters L) for the n x n symmetric S and the n x r
// col-major L (in place); CholeskyQR with a Householder fallback.  work >= 3*n*r
// + r.  Sets *flag bit 2 when a fallback ran.  plain: round as the plain
// elimination does (for factors that are rounded to BF16 halves next).
void subspace_iter(dt_ctx *ctx, const double *S, int64_t n, double *L, int64_t r, int iters,
                   double *work, int *flag, bool plain = false);

// The same for `count` independent problems, side by side in one launch where
// the tiled kernel takes them (n <= 256, r <= 32).
void subspace_iter_batch(dt_ctx *ctx, int count, const double *const *S, const int64_t *n,
                         double *const *L, const int64_t *r, int iters, double *const *work,
                         int *flag);

// The cluster exchange of the subspace iteration, waiting for data that nobody
// sends: adds the number of threads that give up to *late, out of
// EXCHANGE_SELFTEST_THREADS.
constexpr int EXCHANGE_SELFTEST_THREADS = 512;
void exchange_selftest(dt_ctx *ctx, int *late, long long limit_cycles);

// LU inverse with partial pivoting (one CTA).  *flag = 1 on a zero pivot.
void lu_inverse(dt_ctx *ctx, const double *A, int64_t n, double *Ainv, double *work,
                int *flag);

// Modified Gram-Schmidt over the len1 rows of a len1 x len2 col-major A.
void orth2_rows(dt_ctx *ctx, double *A, int64_t len1, int64_t len2);

// The same in pieces, for r <= 32 and a caller that keeps the scratch (at
// least what orth_alloc takes, T of r x m and a flag, zeroed once) over many
// calls: orth_scratch lays it out for rows up to that r; the kernel that produces
// the r x m col-major A ends in gram_finish(s.f) (at most s.blocks CTAs of 256
// threads), and orth_finish makes the two products that follow, out(:, k)
// or, given `rows`, out(:, rows[k]); orth_check reads the flag back (one
// synchronisation) and fails on dependent rows.
struct OrthScratch {
    GramFinish f;
    double *T, *Linv2;
    int64_t blocks;
};
// The CTAs that a Gram over m columns keeps busy; any smaller number does too.
int64_t orth_blocks(const dt_ctx *ctx, int64_t m);
// Scratch for `blocks` CTAs, or as many as there is room for; returns how many
// (no room for one: fails with DT_ERR_NOMEM, or returns 0 when `may_fail`).
int64_t orth_alloc(dt_ctx *ctx, DevMem &mem, int r, int64_t blocks, bool may_fail = false);
OrthScratch orth_scratch(void *mem, double *T, int r, int64_t blocks, int *flag);
void orth_finish(dt_ctx *ctx, const double *A, int r, int64_t m, const OrthScratch &s, double *out,
                 const int32_t *rows);
void orth_check(dt_ctx *ctx, const int *flag);

}  // namespace dt
