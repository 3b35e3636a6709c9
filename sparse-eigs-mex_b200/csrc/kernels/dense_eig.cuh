// A few eigenpairs of a dense symmetric matrix on the device: Householder
// reduction to tridiagonal form by one thread-block cluster, eigenvalues by
// bisection, and the reflectors applied to the tridiagonal's eigenvectors.
// With syev_host's inverse iteration between them this is the method of
// LAPACK's dsyevx (the reference's dense route is dsyev,
// src/speigs_core.c:405-428); the dense route uses it where the one-block
// Jacobi solver (krylov.cuh) is slower.
#pragma once

#include <cuda_runtime.h>

namespace spx {

constexpr int kDenseEigMin = 24;     // smaller orders: the Jacobi solver
constexpr int kDenseEigMax = 4096;   // the back-transformation's registers
constexpr int kDenseEigMaxK = 64;    // more vectors: the Jacobi solver

// The launchers return what the runtime says to the launch; after a refused
// one nothing has been written.

// D (n x n, full symmetric, kept) -> T = Q^T D Q: d[n], e[n-1], reflector k
// (I - beta[k] v v^T) in column k of V below the diagonal (n x n, ld n).
// work: n x n doubles, used when the matrix does not fit the cluster's shared
// memory (else may be null: see dense_tridiag_work).
bool dense_tridiag_work(int n);
cudaError_t launch_dense_tridiag(int n, const double *D, double *V, double *beta, double *d,
                                 double *e, double *work, cudaStream_t st);

// Eigenvalues of the tridiagonal (d, e): the 2k around zero (smallest) or the
// k lowest and k highest (else), val[2k] with their ascending positions in
// idx[2k]; -1 where there is none (2k > n).
cudaError_t launch_tri_bisect(int n, const double *d, const double *e, int k, bool smallest,
                              double *val, int *idx, cudaStream_t st);

// Z (n x nc, ld n) := Q Z
cudaError_t launch_apply_reflectors(int n, const double *V, const double *beta, double *Z, int nc,
                                    cudaStream_t st);

// Rayleigh quotients of the columns of X, accumulated in twice the working
// precision, and the squared residual norms ||D x - lambda x||^2 / ||x||^2
cudaError_t launch_rayleigh_dd(int n, const double *D, const double *X, int nc, double *lam,
                               double *res2, cudaStream_t st);

}  // namespace spx
