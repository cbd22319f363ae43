// Batched complex128 GEMM on the FP64 tensor path (DMMA, mma.sync m8n8k4 f64).
//
//   C[b] = alpha * op(A[b]) * op(B[b]) + beta * C[b]        (row-major, C-ordered like nda views)
//   D[b] (+)= alpha * op(A[b]) * op(B[b])                     (optional second output)
//
// op(A) is A (stored m x k), A^T (stored k x m), optionally conjugated; either operand may be a
// real (float64) matrix, in which case the complex product needs only 2 (or 1) real DMMAs per
// k-step instead of 4.  This is the plain complex128 path of every dense product of the walker
// step (the reference routes these through nda -> cuBLAS / cuTENSOR, numerics/operations/
// product.hpp:125-323 and HamiltonianOperations/Real3IndexFactorization.hpp:321,384,571).
#pragma once

#include "common.cuh"

namespace afqmc {

struct GemmParams {
  int m, n, k;
  const void* A; long lda, strideA;
  const void* B; long ldb, strideB;
  c128* C; long ldc, strideC;
  c128 alpha, beta;
  c128* D; long ldd, strideD;  // optional second output (nullptr: none)
  bool d_store;                 // D = result (true) or D += result (false)
  int sym_m;                    // zgemm_sym_pairs only
};

// op codes for the C++ launcher
enum GemmTrans : int { GN = 0, GT = 1, GC = 2, GH = 3 };  // N, T, conj, conj-transpose

// Launch C = alpha*op(A)*op(B) + beta*C over `batch` problems on `stream`.
// a_real / b_real: the operand is float64 instead of complex128.
int zgemm(cudaStream_t stream, int batch, GemmTrans ta, bool a_real, GemmTrans tb, bool b_real,
          const GemmParams& p);

// C[w][(i, k)] = alpha * sum_n A[w][n] B[(i, k)][n] over all pairs of an M x M matrix (n = M*M,
// ldc >= M*M) for a real B with B[(i, k)] == B[(k, i)] bit for bit: the pairs are computed once
// per 8 x 8 block with block(i) <= block(k) and written to both places.  The same values as
// zgemm(stream, 1, GN, false, GT, true, p), bit for bit.
int zgemm_sym_pairs(cudaStream_t stream, int M, const GemmParams& p);

namespace zg {
constexpr int BK = 16;     // the kernel's K tile
constexpr int STAGES = 3;  // ... and how many of them a CTA's ring holds
// CTA shape of a launch: warps (8 output rows each), tn (8 output columns each), K split
struct Shape {
  int warps, tn, split;
};
}  // namespace zg

}  // namespace afqmc
