// Batched complex FP64 GEMM used by the plain (FP64) form of the walker step.
// C_b = alpha * op(A_b) * op(B_b) + beta * C_b for every batch entry b,
// column-major operands, op in {N, T, C}; A or B may be real (double).
// This is the B200 replacement for the reference's gmm_cpu/zgemm calls
// (common/tensorHao/source/tensor_2d_bl_cpu.cpp:61-75) and its zgemv
// (tensor_1d_bl_cpu.cpp:50-107), batched over the walker population.
#pragma once
#include "common.cuh"

enum { OP_N = 0, OP_T = 1, OP_C = 2 };
// operand storage kinds
enum { ST_Z64 = 0, ST_R64 = 1 };  // complex f64 | real f64

struct ZGemmArgs {
    int m = 0, n = 0, k = 0;
    int opA = OP_N, opB = OP_N;
    int a_real = 0, b_real = 0;   // operand stored as double instead of double2
    zd alpha = {1.0, 0.0}, beta = {0.0, 0.0};
    const void *A = nullptr; long long lda = 0, strideA = 0;
    const void *B = nullptr; long long ldb = 0, strideB = 0;
    zd *C = nullptr; long long ldc = 0, strideC = 0;
    int batch = 1;
    const int *mask = nullptr;     // skip batch b when mask[b] == 0
    const int *skip = nullptr;     // skip batch b when skip[b] != 0
    // symmetric product (m = n): only output tiles that meet the lower
    // triangle (row >= column) are computed; tiles above it are not written
    int lower = 0;
    // A symmetric (m = k) and C wanted only through sum_i x_i C_i with the
    // columns x of B, x^T A x: row block I takes its diagonal block of A once
    // and the blocks left of it twice, half the products.  Only A's entries
    // with row >= column and its 64 x 64 diagonal blocks are read.
    int quad = 0;
    // > 0: the batch entries are pieces of one contraction over ksum elements:
    // entry b takes the k from b k on (those that are left at the end; none: C_b =
    // 0), and strideA, strideB step by k of them.  With quad k is a multiple of 64.
    int ksum = 0;
    // A second product in the same launch and batch (parts = 2), of its own
    // sizes and at these element offsets from A, B and C: the two spins of
    // operators that do not mix them
    int parts = 1, m1 = 0, n1 = 0, k1 = 0;
    long long offA1 = 0, offB1 = 0, offC1 = 0;
    // op(B)'s rows scaled by these factors (k per batch entry, strideScale apart;
    // the second part's at offScale1): C = alpha op(A) diag(scale) B.  Both
    // operators N.  One tile then holds all rows of C (m <= 128), and C may be B.
    const zd *scaleB = nullptr;
    long long strideScale = 0, offScale1 = 0;
};

// Launches on `stream`; returns cudaGetLastError() (cudaErrorInvalidValue for an
// operator pair that no product of the engine has).
cudaError_t zgemm_batched(const ZGemmArgs &a, cudaStream_t stream);

// Pieces (1 to 8) of the contraction of `a` (batch 1) for which the product and
// the sum of the pieces take the least time: small outputs leave SMs idle.
int zgemm_pieces(const ZGemmArgs &a);
// `a` as that many pieces whose outputs are strideC apart; returns their number.
int zgemm_split(ZGemmArgs &a, int pieces, long long strideC);

// Whether scaleB is taken for a product of m rows.
inline bool zgemm_scaled_supported(int m) { return m <= 128; }

// Autotuner switch (process-wide) and the cached choice for a shape (-1: none).
void zgemm_set_autotune(int on);
int zgemm_tuned_choice(const ZGemmArgs &a);
