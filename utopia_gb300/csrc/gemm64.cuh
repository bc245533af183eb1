// FP64 matrix products, on the tensor cores or the FP64 pipes (gemm64.cu).
#pragma once
#include "internal.cuh"

namespace ugpu {

// parts of the product that are known to be zero or not wanted
enum Gemm64Flags : int {
    kGemmLower = 1,    // only tiles that reach the diagonal or below are computed
    kGemmKFromN = 2,   // op(B)(k, n) = 0 for k < n
    kGemmKFromM = 4,   // op(A)(m, k) = 0 for k < m
    kGemmKToN = 8,     // op(B)(k, n) = 0 for k > n
    kGemmKToM = 16,    // op(A)(m, k) = 0 for k > m
};

// C = op(A) op(B), negated and / or added to C; C row-major (M x N, leading dimension ldc) and apart from A and B.
// op(A)(m, k) = A[m a_row + k a_k], op(B)(k, n) = B[n b_row + k b_k]; of the two strides of an operand one is 1.
struct Gemm64 {
    int M = 0, N = 0, K = 0;
    const double *A = nullptr;
    int64_t a_row = 0, a_k = 0;
    const double *B = nullptr;
    int64_t b_row = 0, b_k = 0;
    bool negate = false, add = false;
    double *C = nullptr;
    int64_t ldc = 0;
    int flags = 0;
    bool fma = false;  // FP64 multiply-adds throughout: no split product
    int vec_a = 0, vec_b = 0;  // set by gemm64()
    long long spin = 0;        // likewise: clock cycles that a wait may take
    bool lose_commit = false;  // likewise, in a test: the first stage's MMAs never report their end
};
// scales: scratch of at least M + N 32-bit words, grown where it is smaller (stream-ordered use)
void gemm64(Context &c, const Gemm64 &g, Buffer &scales);

}  // namespace ugpu
