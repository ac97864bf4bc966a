// FP32 GEMMs on the CUDA cores (gemm.cu): activations times weights, and the
// A^T B reductions over rows that weight gradients are.
#pragma once
#include "common.cuh"
#include "dual.cuh"

namespace mlff {

// C[M][N] = A[M][K] B[K][N], row-major and contiguous (A's rows lda floats
// apart when lda is given), with an epilogue:
//   mode 0: C = acc + bias (bias may be NULL)
//   mode 1: the same, and C2 = silu(C)
//   mode 2: C = acc * silu'(Z), Z shaped like C
//   mode 3: C = acc, the sums starting from the bias
//   mode 4: C = silu of that
// M sizes the grid; with m_dev the kernel reads the row count there (M is
// then an upper bound).
int gemm_nn(int mode, const float* A, const float* B, const float* bias, float* C, float* C2, const float* Z,
            int64_t M, const int32_t* m_dev, int N, int K, const Status* st, cudaStream_t s, int lda = 0);

// C[M][N] = sum over rows r < rows of A[r][m] B[r][n] (row strides lda, ldb)
// and, when given, colsum[m] = sum_r A[r][m].  With A1 and B1 a second set of
// as many rows is added to C (not to colsum).  accumulate: added to C and
// colsum instead of written.  part: scratch of gemm_tn_floats(M, N) floats.
// Fixed-order sums: the same bits on every call of the same shape.
size_t gemm_tn_floats(int64_t M, int64_t N);
struct GemmRows {
    const float* A;
    const float* B;
    const float* A1 = nullptr;
    const float* B1 = nullptr;
};
int gemm_tn(const GemmRows& x, int lda, int ldb, int M, int N, int64_t rows, float* C, float* colsum,
            bool accumulate, float* part, const Status* st, cudaStream_t s);

}  // namespace mlff
