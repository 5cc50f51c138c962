// Tensor-core (tcgen05) complex GEMM of the mixed-precision path; see pw_umma.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace pwk {

// A K-major split-BF16 operand: `rows` rows of Kp BF16 values per piece
// (hi, lo, and optionally a third piece lo2): in blocks of 64 the real parts
// of 32 consecutive values, then their imaginary parts.  A product runs with three
// pieces (6 MMAs, ~2^-24) when both operands carry lo2, else with two
// (3 MMAs, ~2^-17).
struct UmmaOperand {
    __nv_bfloat16 *hi = nullptr;
    __nv_bfloat16 *lo = nullptr;
    __nv_bfloat16 *lo2 = nullptr;
    int64_t rows = 0;
    int Kp = 0;
};

int umma_kpad(int64_t K);                          // padded 2K (multiple of 64)
size_t umma_operand_bytes(int64_t rows, int64_t K);  // hi + lo bytes for `rows` rows (one piece: half)
// What a product of M x N complex values runs with.  splits > 0 overrides the
// split-K count; upper: the product is Hermitian and only tiles on or above the
// diagonal run (2: C is complex128).
struct UmmaPlan {
    int bn, S;         // tile width, parts of the sum
    int passes;        // kernels of umma_gemm with C given: 1 (C written directly), or 2
    size_t ws_bytes;   // the split sums, [S][N][M] complex (unused with 1 pass into C)
};
UmmaPlan umma_plan(int64_t M, int N, int Kp, int splits = 0, int upper = 0);

// Operand builders (CT = float2 or double2 input element).
//   tn:   m rows from Z (K x m)                for either operand of Z^H W
//   nn_a: M rows from Z = A^H, A (M x k)       for the first operand of A U
template <typename CT> cudaError_t umma_prep_tn(const void *Z, int64_t ld, int64_t K, int m, UmmaOperand &, cudaStream_t);
template <typename CT> cudaError_t umma_prep_nn_a(const void *A, int64_t lda, int64_t M, int k, UmmaOperand &, cudaStream_t);

// The operand of D P from the S split sums that umma_gemm with C == nullptr left
// in ws (P = betaNL' psi, nbeta x nb; D as CSR)
cudaError_t umma_dcsr_prep(const float *ws, int S, int nbeta, int nb, const int *rowptr, const int *col, const double *val,
                           UmmaOperand &, cudaStream_t);

// C (m x n complex of type CT, ldc) (+)= result; A.rows == m, B.rows == n; plan: of
// umma_plan(m, n, A.Kp, ..., upper).
// C == nullptr: the split sums stay in ws ([split][n][m] complex).
// err: device int set non-zero if a bounded wait in the kernel expired.
template <typename CT>
// upper: 1 = C is Hermitian and only C[i][j], i <= j, is formed and written,
// 2 = the other triangle is filled with its conjugate as well.
// lolo != 0 (two-piece operands from the same block, C = Z^H Z): add the
// lo*lo product, whose omission biases the diagonal |z|^2 low.
cudaError_t umma_gemm(const UmmaPlan &plan, const UmmaOperand &A, const UmmaOperand &B, int m, int n, void *C, int64_t ldc,
                      int accumulate, float *ws, int *err, cudaStream_t, int upper = 0, int lolo = 0);

}  // namespace pwk
