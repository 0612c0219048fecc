// FP64 complex GEMMs on the integer tensor cores; see zgemm_mod.cu.
#pragma once

#include "cgemm.cuh"

namespace q3b {
namespace zmod {

constexpr int kLongestK = 257 * 16384;  // of a product (zmod_combine adds the bytes of 257 ranges)

// An operand scaled to integers and reduced modulo each modulus, as the tiles
// of 128 rows x 128 K the kernel copies, for operands used many times (a
// k-point's projectors).  Rows are M of the product, K its reduction index.
struct PackedA {
    const unsigned char* tiles = nullptr;
    const int* exps = nullptr;  // power of two each row was scaled by
    int M = 0, K = 0;
    const int* balance = nullptr;  // exponents along K that were taken out of it, put into B (may be null)
};
size_t packed_a_bytes(int M, int K);
size_t packed_a_exps(int M);  // ints
// kmajor: element (m, k) at A[m * lda + k] (the "C,N" operand); else at A[m + k * lda]
void pack_a(cudaStream_t st, int M, int K, const double2* A, long lda, bool kmajor, const int* balance,
            unsigned char* tiles, int* exps);

// The balance of the projectors (beta: npw x nproj, ld npw) along the projectors, for
// beta B', and along the plane waves, for beta^H psi: balance_ints of each.
size_t balance_ints(int lines);  // padded to whole K blocks
void balance_projectors(cudaStream_t st, int npw, int nproj, const double2* beta, int* along_proj, int* along_pw);

// whether the product is faster here than on the FP64 units
bool worth(bool conj_a, int M, int N, int K, bool packed);
size_t workspace_bytes(bool conj_a, int M, int N, int K, bool packed);

// C = alpha op(A) B + beta C as cgemm<double>; `pk` replaces A when given.
// ws holds at least workspace_bytes(...).
void zgemm(cudaStream_t st, bool conj_a, int M, int N, int K, double2 alpha, const double2* A, long lda,
           const PackedA* pk, const double2* B, long ldb, double2 beta, double2* C, long ldc,
           const GemmWorkspace& ws);

}  // namespace zmod
}  // namespace q3b
