// Small dense FP64 R x R kernels (eigendecomposition, pseudo-inverse).
#pragma once
#include "common.cuh"

namespace exafac {

size_t syev_smem_bytes(int R);
size_t syev_scratch_doubles(int R, int batch);

// Batched symmetric eigendecomposition / pseudo-inverse, one CTA per matrix
// (matrix b at A + b * a_stride, upper triangle read).  V, lam, pinv may be
// null.  vt_scratch: syev_scratch_doubles(R, batch) doubles.
int launch_syev(int R, const double* A, int64_t a_stride, int batch, double* V, double* lam, int64_t v_stride,
                double* pinv, double tol, double* vt_scratch, cudaStream_t stream);

// The same decomposition from an FP32 start refined in FP64 (the FP64 form's
// STS-CP sampling matrices).  scratch: syev_refine_doubles(R, batch) doubles.
size_t syev_refine_doubles(int R, int batch);
int launch_syev_refined(int R, const double* A, int64_t a_stride, int batch, double* V, double* lam, int64_t v_stride,
                        double* vt_scratch, double* scratch, cudaStream_t stream);

// Symmetric pseudo-inverse (eigenvalues <= tol dropped) of one matrix:
// Cholesky inverse when provably well conditioned, Jacobi otherwise.
// scr (chol_scratch_doubles(R) doubles, 32 < R): spread over many blocks; null:
// one CTA (for callers with vt_scratch only).
size_t chol_scratch_doubles(int R);
int launch_pinv(int R, const double* A, double* out, double tol, double* vt_scratch, cudaStream_t stream,
                double* scr = nullptr);

// The same followed by one Newton step X <- 2X - X A X (the refinement the
// mixed forms apply to the solve).
int launch_pinv_refined(int R, const double* A, double* out, double tol, double* vt_scratch, cudaStream_t stream,
                        double* scr);
// The leverage-score pseudo-inverse of the mixed forms (unit-diagonal Gram, R
// <= 32): sigma, ngram and the degenerate flag from the factor Gram, then the
// pseudo-inverse of ngram, the sweep in FP32 when its error bound allows, else
// the FP64 path, in one launch.
int launch_sigma_pinv_f32(int R, const double* ugram, double* sigma, double* ngram, int* degenerate, double* out,
                          double tol, double* vt_scratch, cudaStream_t stream);

// STS-CP computeM of the mixed forms from Cholesky factors: Phi (full and
// packed), E[N] and chain[k] *= Phi from chain[first] (Jacobi when not
// provably well conditioned; V, lam, vt its scratch), then E[k] for k = 1..
// N-1, k != n, from the pivoted Cholesky of chain[k].
int launch_sts_factors_chol(int N, int n, int R, double tol, double* chain, double* E, double* Phi, double* PhiP,
                            double* V, double* lam, double* vt, double* scr, cudaStream_t stream);

}  // namespace exafac
