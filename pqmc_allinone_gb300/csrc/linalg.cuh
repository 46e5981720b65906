// linalg.cuh -- host launchers of the FP64 complex dense kernels (linalg.cu)
#pragma once
#include "common.cuh"

namespace pqmc {
// C = alpha*op(A)*op(B) + beta*C, ta/tb in {'N','C'}
int zgemm(cudaStream_t s, char ta, char tb, int m, int n, int k, cplx alpha, const cplx* A, int lda,
          const cplx* B, int ldb, cplx beta, cplx* C, int ldc);
// Householder QR, Q overwrites A (m x n), d = diag(R); work: m x m scratch (m
// n words are used, and n n more where m m has room for them); err: device
// word that takes PQMC_ERR_TIMEOUT if a wait inside ran out
int house_qr(cudaStream_t s, int m, int n, cplx* A, cplx* d, cplx* work, int* err);
// the same, also returning R (n x n upper triangle, column-major) and
// ln det Q (a phase) when R / lndet are not null
int house_qr_r(cudaStream_t s, int m, int n, cplx* A, cplx* d, cplx* R, cplx* lndet, cplx* work, int* err);
// LU with partial pivoting of A (n x n, destroyed) and A X = B solved in
// place on B (n x nrhs; nrhs may be 0).  diag: pivots in order, perm: their
// rows, info: device int (first zero pivot, 1-based, or 0), work: n x n scratch
int lu_solve(cudaStream_t s, int n, cplx* A, int nrhs, cplx* B, int ldb, cplx* diag, int* perm, int* info, cplx* work,
             int* err);
// log det A from lu_solve's pivots
int lu_logdet(cudaStream_t s, int n, const cplx* diag, const int* perm, cplx* out);
int herm_t(cudaStream_t s, int m, int n, const cplx* a, cplx* out);
int coop_grid(const void* fn, int threads, int want, size_t smem = 0);
}  // namespace pqmc
