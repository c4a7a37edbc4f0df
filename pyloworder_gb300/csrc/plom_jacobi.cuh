// One-sided Jacobi in shared memory (jacobi_cta.cu): interfaces for dense.cu.
#pragma once
#include "plom_common.cuh"

namespace plom {

// Whether n columns (per problem) fit the double-float form and its clusters
// can be resident on this device.
bool jacobi_cta_usable(int n, int cplx);
// SVD of `batch` n x n matrices on double-float rows (tol >= 1e-10): S, U, VH as
// jacobi_svd gives them.  trans (real): the rows of A are rotated instead of
// its columns.  At, Vt: batch x n x n (complex: 2n) FP64 scratch, nrm2: batch x n.
// V0 (one real problem, trans): A is B = A^T V0 and the rotations start from V0.
int jacobi_cta(const double* A, int n, int batch, int cplx, int trans, double tol, double* At,
               double* Vt, double* nrm2, unsigned long long* amax, double* S, double* U,
               double* VH, int* info, cudaStream_t st, const double* V0 = nullptr);
// FP32 sweeps over the rows of one real n x n matrix (jacobi_gram.cu): the
// rotation product V (n x n row-major, FP32) and the bits of max |a|.  plan_ok:
// by the size alone (workspace queries); usable: its CTAs can also be resident
// together on this device.
bool jacobi_gram_plan_ok(int n);
bool jacobi_gram_usable(int n);
int jacobi_gram_f32(const double* A, int n, float tol, float floor_rel, float tstop, float* V,
                    unsigned long long* amax, int* info, Arena& ws, cudaStream_t st);

}  // namespace plom
