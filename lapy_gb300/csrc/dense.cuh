// Batched small dense FP64 linear algebra for the Lanczos Ritz steps.
#pragma once
#include "common.cuh"

namespace lapy {

// Top-`want` eigenpairs (largest eigenvalues first) of `nmat` symmetric n_b x n_b
// matrices.  Matrix b lives at A + b*lda*lda (row-major, leading dimension lda,
// overwritten).  n_b = nsize[b] (device array) <= nmax <= lda.  Output: theta[b*want + i]
// (descending), S[b*lda*want + r*want + i] eigenvector i, row r (rows >= n_b zero).
// The tridiagonal form is reduced in double-float (about 2^-47 of the matrix
// norm a step) up to 384 rows and with FP64 reflectors above.  exact: its
// eigenvalues to FP64 accuracy; otherwise they may carry a further error of
// 2^-41 of the norm (the eigenvectors are those of the matrix either way: they
// come from inverse iteration at these shifts).
// Scratch `work` must hold sym_eig_work_doubles(lda, want) doubles per matrix.
size_t sym_eig_work_doubles(int lda, int want);
int sym_eig_top(int nmat, double* A, int lda, const int32_t* nsize, int nmax, int want, double* theta,
                double* S, double* work, const int32_t* active, bool exact, cudaStream_t stream);

}  // namespace lapy
