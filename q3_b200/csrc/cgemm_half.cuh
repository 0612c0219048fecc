// FP32 complex GEMMs with a packed A on FP16 tensor cores; see cgemm_half.cu.
#pragma once

#include "cgemm.cuh"

namespace q3b {
namespace half2x {

// An operand scaled by a power of two a row and split into two FP16 numbers a
// value, as the tiles of 128 rows x 64 K the kernel copies.  Rows are M of the
// product, K its reduction index.
struct PackedA {
    const unsigned char* tiles = nullptr;
    const int* exps = nullptr;  // power of two each row was scaled by
    int M = 0, K = 0;
    const int* balance = nullptr;  // exponents along K that were taken out of it, put into B (may be null)
};
constexpr int kLongestK = 65535 * 64;  // of a packed operand: one grid row per 64 of K
size_t packed_a_bytes(int M, int K);
size_t packed_a_exps(int M);  // ints
// kmajor: element (m, k) at A[m * lda + k] (the "C,N" operand); else at A[m + k * lda]
void pack_a(cudaStream_t st, int M, int K, const float2* A, long lda, bool kmajor, const int* balance,
            unsigned char* tiles, int* exps);

size_t workspace_bytes(bool conj_a, int M, int N, int K);
// C = alpha op(A) B + beta C; ws holds at least workspace_bytes(...)
void cgemm(cudaStream_t st, bool conj_a, int M, int N, int K, float2 alpha, const PackedA& A, const float2* B,
           long ldb, float2 beta, float2* C, long ldc, const GemmWorkspace& ws);

}  // namespace half2x
}  // namespace q3b
