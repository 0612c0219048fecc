// FP64 complex GEMMs on the integer tensor cores (tcgen05 kind::i8, sm_100a).
//
//   "C,N":  C = alpha A^H B + beta C    (A: K x M, lda; B: K x N, ldb)
//   "N,N":  C = alpha A B   + beta C    (A: M x K, lda; B: K x N, ldb)
//
// The 5th-generation tensor cores have no FP64, and the FP64 units take 4 K
// DFMAs per complex output.  Here the product is formed in integers, exactly,
// through its residues modulo 15 pairwise coprime numbers of at most 256 (the
// Chinese remainder form of the Ozaki scheme; Ozaki, Uchino, Imamura 2025):
//
//   1. Every row of op(A) and every column of B is scaled by a power of two so
//      that its 2-norm is at most 2^c and rounded to integers.  By Cauchy-
//      Schwarz the real and imaginary parts of every output are then below
//      2^(2c), and c = 58.39 is the largest for which 2^(2c) < P/2, P the
//      product of the moduli (2^117.8).
//   2. The integers are reduced modulo each modulus to bytes (pack_rows).
//   3. One u8 x u8 -> s32 product per modulus, exact: at most 16384 of K a
//      partial sum, so that the sum of two products stays below 2^31
//      (zmod_gemm).  Its epilogue reduces the sums to bytes again.
//   4. The output is (sum_i y_i c_i / m_i mod 1) P with c_i the inverse of P/m_i
//      modulo m_i: a sum of 80-bit fixed-point fractions, made signed, times
//      P and the two scales (zmod_combine).
//
// Error.  Only step 1 rounds, by at most half a unit in integers whose rows have
// norm 2^c, and step 4 once: an output differs from the exact product by about
// 0.6 2^-58.4 |a| |b| = 1.6e-18 |a| |b| (|a|, |b| the norms of its row and
// column), where K rounded DFMAs leave about 4e-17 |a| |b|.
//
// Balance.  DFMAs leave 1e-16 sum |a_k b_k| at the worst, whatever the scales along K;
// the norms count a_k and b_k by themselves.  Where the large entries of the one
// operand meet small ones of the other (projectors of unequal norms, whose D
// makes up for it; U^-1 of a basis of unequal norms), |a| |b| is far above the sum,
// so op(A) and B are first multiplied along K by 2^t_k and 2^-t_k, exactly:
//   N,N: t_k from the norms of B's rows;
//   projectors: from the norms of beta's columns for beta B', and of its rows, with
//     the columns balanced, for beta^H psi, once per k-point (balance_projectors).
// beta D beta^H psi of the 64-atom cell, relative 2-norm from the exact value, without
// the balance, with it, and on DFMAs: projector norms spread over 1e6, 1.7e-12, 1.6e-15
// and 3.7e-15; bands of high plane waves only, 1.9e-13, 3.4e-16 and 2.7e-15; as the cell
// has them, 1.7e-16, 2.0e-16 and 3.3e-15.  It cost 17 us of the 1.8 ms of H|psi> while the
// norms of a long row were formed by 256 threads, and nothing with 1024.
// Other C,N products are inner products of vectors, which need no more than
// 1.6e-18 of their norms.
//
// Rows or columns that hold an infinity or a NaN give NaN in all their outputs.
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "umma_pair.cuh"
#include "zgemm_mod.cuh"

namespace q3b {
namespace zmod {
namespace {

using namespace umma;

constexpr int NMOD = 15;
constexpr int kMod[NMOD] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};
constexpr int kNotFinite = -(1 << 30);  // exponent of a row that holds an infinity or a NaN
constexpr int kZeroLine = 1 << 29;      // of a line of zeros, where lines are balanced
constexpr int kBalanceSpan = 100;       // lines are balanced to within 2^100 of the largest

// ------------------------------------------------------------ modulus constants
constexpr unsigned pow256(int j, int m) {
    unsigned r = 1 % m;
    for (int i = 0; i < j; ++i) r = (r * 256u) % m;
    return r;
}
// four weights 256^(first + j) mod m, one a byte
constexpr unsigned weights(int m, int first) {
    unsigned w = 0;
    for (int j = 0; j < 4; ++j) w |= pow256(first + j, m) << (8 * j);
    return w;
}
// -2^63 mod m: takes back the offset that makes the integers unsigned
constexpr unsigned offset63(int m) {
    const unsigned r = (pow256(7, m) * 128u) % m;
    return (m - r) % m;
}
constexpr unsigned inv_up(int m) { return static_cast<unsigned>((0x100000000ull + m - 1) / m); }
// (P / m_i)^-1 modulo m_i
constexpr int cofactor_inverse(int i) {
    const int m = kMod[i];
    int r = 1 % m;
    for (int j = 0; j < NMOD; ++j)
        if (j != i) r = (r * kMod[j]) % m;
    for (int x = 1; x < m; ++x)
        if ((r * x) % m == 1) return x;
    return 0;
}
// 20-bit digit `d` (3: the highest) of floor(2^80 cofactor_inverse(i) / m_i)
constexpr unsigned fraction_digit_of(int i, int d) {
    unsigned long long rem = cofactor_inverse(i);
    unsigned digit = 0;
    for (int j = 3; j >= d; --j) {
        digit = static_cast<unsigned>((rem << 20) / kMod[i]);
        rem = (rem << 20) % kMod[i];
    }
    return digit;
}
// f(integral_constant<int, i>) for every modulus, so that constants are literals
template <typename F, int... I> __device__ __forceinline__ void each_mod(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <typename F> __device__ __forceinline__ void each_mod(F&& f) {
    each_mod(static_cast<F&&>(f), std::make_integer_sequence<int, NMOD>{});
}

// moduli for the GEMM's epilogue, which meets them in a run-time order
struct ModTable {
    unsigned m[NMOD];
    unsigned inv[NMOD];   // floor(2^32 / m)
};

double log2_product() {
    double s = 0.0;
    for (int m : kMod) s += std::log2(static_cast<double>(m));
    return s;
}
double scale_bits() { return 0.5 * (log2_product() - 1.0) - 1e-6; }

// ------------------------------------------------------------------ tiles
constexpr int BM = 128;               // complex rows a CTA holds of a pair's 256 (UMMA M = 256)
constexpr int BK = 128;               // K per stage: one 128-byte row of bytes
constexpr int A_TILE = 2 * BM * BK;   // real plane, imaginary plane
constexpr int STAGES = 4;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (EPI_WARPS + 2);
// TMEM: two buffers of at most 256 accumulator columns
// BC: complex columns a CTA holds of its pair's 2 BC (64, or 32 for narrow products)
template <int BC> struct Cols {
    static constexpr int b_tile = 3 * BC * BK;      // three planes, see pack_rows
    static constexpr int out_tile = BM * 2 * BC * 2;  // bytes of one modulus of a CTA's outputs
    static constexpr int smem = STAGES * (A_TILE + b_tile) + 1024;
    // D s32, A and B u8, K-major, M = 256, N = 4 BC
    static constexpr uint32_t instr = (2u << 4) | (static_cast<uint32_t>((4 * BC) >> 3) << 17) |
                                      (static_cast<uint32_t>((2 * BM) >> 4) << 24);
};
constexpr int kMaxK = 16384;          // of one partial sum: 2 * 255^2 * 16384 < 2^31
constexpr int kMaxSplits = 64;        // K ranges taken for the sake of a better share of work
constexpr int kMaxRanges = 257;       // K ranges at all: their bytes are added up in 16 bits
static_assert(kLongestK == kMaxRanges * kMaxK, "the longest product");
static_assert(255 * kMaxRanges <= 0xffff, "zmod_combine adds the ranges' bytes in 16 bits");

// --------------------------------------------------------- row scales
// exponent s with |row| 2^s <= 2^c from the row's sum of squares and largest
// magnitude; the sum of squares of very large or very small values leaves
// the range of doubles, and the bound |row| <= max sqrt(2 K) takes its place
__device__ __forceinline__ int row_exponent(double ss, double mx, int K, double c, int zero) {
    if (!(mx < INFINITY) || ss != ss) return kNotFinite;
    if (mx == 0.0) return zero;
    if (ss > 1e-280 && ss < 1e300) return static_cast<int>(floor(c - 0.5 * log2(ss)));
    int e;
    frexp(mx, &e);  // mx < 2^e; a denormal may have been rounded down to half
    return static_cast<int>(floor(c - e - 0.5 * log2(2.0 * K))) - (mx < 1e-300 ? 1 : 0);
}

__device__ __forceinline__ void take(double2 v, double& ss, double& mx) {
    ss += v.x * v.x + v.y * v.y;
    // a NaN fails the comparison, and stands in ss
    const double a = fabs(v.x), b = fabs(v.y);
    if (a > mx) mx = a;
    if (b > mx) mx = b;
}

__device__ __forceinline__ double pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }

// The operands along K (`balance`, may be null): op(A) and B times 2^(sign balance[k]),
// with opposite signs, which leaves the product as it is.
struct Balance {
    const int* exps;
    int sign;
    __device__ __forceinline__ int at(int k) const { return exps ? sign * exps[k] : 0; }
    // of 16 places from a multiple of 16 on (the array is padded with zeros to whole K blocks)
    __device__ __forceinline__ void get16(int k, int* e) const {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int4 v = exps ? *reinterpret_cast<const int4*>(exps + k + 4 * q) : make_int4(0, 0, 0, 0);
            e[4 * q] = sign * v.x;
            e[4 * q + 1] = sign * v.y;
            e[4 * q + 2] = sign * v.z;
            e[4 * q + 3] = sign * v.w;
        }
    }
};

// rows contiguous along K: one block of NT threads a row (kLongRow and above 1024, which takes
// the balance's extra reads in the time that 256 threads took without them)
constexpr int kLongRow = 4096;
template <int NT>
__global__ void __launch_bounds__(NT) exps_kmajor(int R, int K, const double2* __restrict__ X, long ld, double c,
                                                   Balance bal, int zero, int* exps) {
    chain_begin();
    const int r = blockIdx.x;
    double ss = 0.0, mx = 0.0;
    if (r < R) {
        const double2* x = X + (long)r * ld;
        for (int k = threadIdx.x; k < K; k += 4 * NT) {
            double2 v[4];
            double f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = k + NT * u < K;
                v[u] = ok ? x[k + NT * u] : make_double2(0.0, 0.0);
                f[u] = pow2(ok ? bal.at(k + NT * u) : 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) take(f[u] * v[u], ss, mx);
        }
    }
    __shared__ double s_ss[NT / 32], s_mx[NT / 32];
    for (int o = 16; o > 0; o >>= 1) {
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s_ss[threadIdx.x >> 5] = ss;
        s_mx[threadIdx.x >> 5] = mx;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NT / 32; ++w) {
            ss += s_ss[w];
            mx = fmax(mx, s_mx[w]);
        }
        exps[r] = r < R ? row_exponent(ss, mx, K, c, zero) : 0;
    }
}

// rows along the contiguous index: 32 rows a block, K dealt to W warps
template <int W>
__global__ void __launch_bounds__(32 * W) exps_mmajor(int R, int K, const double2* __restrict__ X, long ld, double c,
                                                   Balance bal, int zero, int* exps) {
    chain_begin();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int r = blockIdx.x * 32 + lane;
    double ss = 0.0, mx = 0.0;
    if (r < R) {
        for (int k = w; k < K; k += 4 * W) {
            double2 v[4];
            double f[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = k + W * u < K;
                v[u] = ok ? X[r + (long)(k + W * u) * ld] : make_double2(0.0, 0.0);
                f[u] = pow2(ok ? bal.at(k + W * u) : 0);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) take(f[u] * v[u], ss, mx);
        }
    }
    __shared__ double s_ss[W][32], s_mx[W][32];
    s_ss[w][lane] = ss;
    s_mx[w][lane] = mx;
    __syncthreads();
    if (w == 0) {
        for (int j = 1; j < W; ++j) {
            ss += s_ss[j][lane];
            mx = fmax(mx, s_mx[j][lane]);
        }
        exps[r] = r < R ? row_exponent(ss, mx, K, c, zero) : 0;
    }
}

// Exponents of lines (each with its norm's distance below 2^c) to those that bring
// the shorter lines up to the longest, times `sign`, with zeros up to `padded`.  One
// block.
__global__ void __launch_bounds__(1024) balance_lines(int n, int padded, int sign, int* exps) {
    chain_begin();
    __shared__ int s_least[32];
    int least = kZeroLine;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const int e = exps[i];
        if (e != kNotFinite) least = min(least, e);
    }
    least = __reduce_min_sync(0xffffffffu, least);
    if ((threadIdx.x & 31) == 0) s_least[threadIdx.x >> 5] = least;
    __syncthreads();
    for (int w = 0; w < 32; ++w) least = min(least, s_least[w]);
    for (int i = threadIdx.x; i < padded; i += 1024) {
        const int e = i < n ? exps[i] : kNotFinite;
        exps[i] = e == kNotFinite ? 0 : sign * (e == kZeroLine ? kBalanceSpan : min(e - least, kBalanceSpan));
    }
}

// ------------------------------------------------------------------ packing
// 32 rows x 128 K a block; a thread takes 16 consecutive K of one row and
// writes their residues as one 16-byte chunk per modulus and plane, in the
// 128-byte swizzle the tensor cores read.  Tiles: [tile of ROWS][kb][modulus]
// [plane][ROWS][128 bytes].  A's planes are re and im.  B has three, so that one
// product with Ar and one with Ai add up to both parts of the output:
//   N,N: -im, re, im   Ar [re | im] + Ai [-im | re] = [re | im] of A B
//   C,N: re, im, -re   Ar [re | im] + Ai [im | -re] = [re | im] of A^H B
// each pair of neighbouring planes being one operand.  The values pass through shared memory, so that
// both the reads (along the contiguous index) and the chunk stores (eight
// lanes a row) are coalesced.
constexpr int PACK_ROWS = 32;
constexpr int PACK_PITCH = 8 * 17 + 1;  // double2 per row: chunks of 16 + 1, odd in all
constexpr int PACK_SMEM = PACK_ROWS * PACK_PITCH * 16;

enum PackAs { kPackA, kPackB, kPackBConj };
template <bool KMAJOR, int ROWS, int AS>
__global__ void __launch_bounds__(256) pack_rows(int R, int K, const double2* __restrict__ X, long ld,
                                                 Balance bal, const int* __restrict__ exps, int nkb,
                                                 unsigned char* out) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char psm[];
    double2* s = reinterpret_cast<double2*>(psm);
    const int tid = threadIdx.x, kb = blockIdx.y, k0 = kb * BK, r0 = blockIdx.x * PACK_ROWS;
#pragma unroll 4
    for (int i = 0; i < PACK_ROWS * BK / 256; ++i) {
        const int idx = tid + i * 256;
        const int row = KMAJOR ? idx / BK : idx % PACK_ROWS;
        const int k = KMAJOR ? idx % BK : idx / PACK_ROWS;
        const int gr = r0 + row, gk = k0 + k;
        double2 v = make_double2(0.0, 0.0);
        if (gr < R && gk < K) v = KMAJOR ? X[(long)gr * ld + gk] : X[gr + (long)gk * ld];
        s[row * PACK_PITCH + (k >> 4) * 17 + (k & 15)] = v;
    }
    __syncthreads();
    const int row = tid >> 3, ch = tid & 7;
    const int gr = r0 + row;
    const int e = exps[gr];
    const int e1 = e == kNotFinite ? 0 : e / 2, e2 = e == kNotFinite ? 0 : e - e / 2;
    // in two steps, so that only the scaled value has to be in range
    const double f1 = pow2(e1);
    int along[16];
    bal.get16(k0 + 16 * ch, along);
    unsigned lo[2][16], hi[2][16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const double2 v = s[row * PACK_PITCH + ch * 17 + j];
        const double f2 = pow2(e2 + along[j]);
        // + 2^63 as an unsigned number; each modulus takes it back
        const unsigned long long a = static_cast<unsigned long long>(__double2ll_rn(v.x * f1 * f2)) ^ (1ull << 63);
        const unsigned long long b = static_cast<unsigned long long>(__double2ll_rn(v.y * f1 * f2)) ^ (1ull << 63);
        lo[0][j] = static_cast<unsigned>(a);
        hi[0][j] = static_cast<unsigned>(a >> 32);
        lo[1][j] = static_cast<unsigned>(b);
        hi[1][j] = static_cast<unsigned>(b >> 32);
    }
    const int tile = gr / ROWS, rr = gr % ROWS;
    constexpr int PLANE = ROWS * BK, TILE = (AS == kPackA ? 2 : 3) * PLANE;
    unsigned char* dst = out + ((size_t)tile * nkb + kb) * NMOD * TILE + rr * BK + ((ch ^ (rr & 7)) << 4);
    each_mod([&](auto I) {
        constexpr int i = decltype(I)::value, m = kMod[i];
        constexpr unsigned wl = weights(m, 0), wh = weights(m, 4), c0 = offset63(m), inv = inv_up(m);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            constexpr int negated = AS == kPackB ? 1 : AS == kPackBConj ? 0 : -1;  // part with a negative plane
            unsigned w[4], neg[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                unsigned b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (m == 256) {
                        b[j] = lo[p][4 * q + j];
                    } else {
                        // below 8 * 255 * 254 + 255: the quotient by umulhi is exact
                        const unsigned t = __dp4a(hi[p][4 * q + j], wh, __dp4a(lo[p][4 * q + j], wl, c0));
                        b[j] = t - __umulhi(t, inv) * m;
                    }
                }
                w[q] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
                // m - b in every byte, modulo m: m - 0 = m <= 255 is as good a residue as 0
                if (p == negated) {
                    if (m == 256) neg[q] = __vneg4(w[q]);
                    else neg[q] = m * 0x01010101u - w[q];
                }
            }
            unsigned char* at = dst + (size_t)i * TILE;
            *reinterpret_cast<uint4*>(at + (AS == kPackB ? p + 1 : p) * PLANE) = make_uint4(w[0], w[1], w[2], w[3]);
            if (p == negated)
                *reinterpret_cast<uint4*>(at + (AS == kPackB ? 0 : 2) * PLANE) = make_uint4(neg[0], neg[1], neg[2], neg[3]);
        }
    });
}

// ------------------------------------------------------------------ products
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t instr, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(instr), "r"(accumulate)
        : "memory");
}
// A pair of CTAs (one TPC) works on output tiles of 256 rows x 2 BC columns with
// cta_group::2 MMAs: each CTA holds 128 rows of A and BC columns of B in its
// shared memory, and its 128 rows of the accumulator, [re | im] of one half of
// the columns after the other, in TMEM.  A stage (128 of K) is 56 KB a CTA for
// 1024 clocks of the tensor pipe; with one-CTA tiles of 128 x 64 it was 48 KB for
// 512, and the kernel was bound by reading L2 (10 to 14 TB/s).
//
// One unit of work is a tile of one modulus over one range of K.  The pairs are
// persistent and take units round robin.  In each CTA a producer thread streams
// its operand tiles through a ring of four stages.  In the leader one thread
// issues the MMAs, into one of two TMEM buffers; in the other CTA that thread
// tells the leader of each full stage.  Eight warps a CTA empty the other
// buffer: the sums, reduced modulo m to bytes, [column / 8][row][8 x (re, im)].
// Neighbouring units share an operand tile: n runs fastest, then (N,N) the
// modulus and the row tile, or (C,N) the row tile, the modulus and the K range.
struct Units {
    int nt, mt, splits, kb_per;  // pair tiles along N and M, K ranges, K blocks a range
    int nkb;
    bool mod_inside;             // N,N order
};
__device__ __forceinline__ void unit_of(const Units& u, int i, int& n, int& m, int& mod, int& z) {
    n = i % u.nt;
    i /= u.nt;
    if (u.mod_inside) {
        mod = i % NMOD;
        i /= NMOD;
        m = i % u.mt;
    } else {
        m = i % u.mt;
        i /= u.mt;
        mod = i % NMOD;
        i /= NMOD;
        z = i;
        return;
    }
    z = i / u.mt;
}

template <bool CONJ_A, int BC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
zmod_gemm(Units un, int total, const unsigned char* __restrict__ A, const unsigned char* __restrict__ B,
          unsigned char* out, const __grid_constant__ ModTable tab, int* err) {
    chain_begin();
    constexpr int B_TILE = Cols<BC>::b_tile, STAGE = A_TILE + B_TILE;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[STAGES], peer_full[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2],
        done_bar;
    __shared__ uint32_t tmem_slot;
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&peer_full[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2 * EPI_WARPS);
        }
        mbar_init(&done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc_pair(&tmem_slot);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // both CTAs' barriers and TMEM are ready
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    if (warp == EPI_WARPS && lane == 0) {
        // ------------------------------------------------------------ producer
        int it = 0;
        bool ok = true;
        for (int i = pair; i < total && ok; i += pairs) {
            int n, m, mod, z;
            unit_of(un, i, n, m, mod, z);
            const int k1 = min(un.nkb, (z + 1) * un.kb_per);
            for (int kb = z * un.kb_per; kb < k1; ++kb, ++it) {
                const int s = it % STAGES;
                if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, err)) {
                    ok = false;
                    break;
                }
                unsigned char* st = smem + s * STAGE;
                mbar_arrive_tx(&full_bar[s], STAGE);
                bulk_copy_g2s(st, A + (((size_t)(2 * m + rank) * un.nkb + kb) * NMOD + mod) * A_TILE, A_TILE,
                              &full_bar[s]);
                bulk_copy_g2s(st + A_TILE, B + (((size_t)(2 * n + rank) * un.nkb + kb) * NMOD + mod) * B_TILE, B_TILE,
                              &full_bar[s]);
            }
        }
        if (!ok)  // leave no copy in flight
            for (int j = it > STAGES ? it - STAGES : 0; j < it; ++j)
                mbar_wait(&full_bar[j % STAGES], (j / STAGES) & 1, err, false);
    } else if (warp == EPI_WARPS + 1 && lane == 0 && rank == 0) {
        // ------------------------------------------------------------ MMA issuer
        int it = 0, ui = 0;
        bool ok = true;
        for (int i = pair; i < total && ok; i += pairs, ++ui) {
            int n, m, mod, z;
            unit_of(un, i, n, m, mod, z);
            const int buf = ui & 1;
            if (ui >= 2 && !mbar_wait(&acc_empty[buf], ((ui >> 1) - 1) & 1, err)) break;
            tc_fence_after();
            const uint32_t d = tmem + buf * 256;
            const int k1 = min(un.nkb, (z + 1) * un.kb_per);
            bool first = true;
            for (int kb = z * un.kb_per; kb < k1; ++kb, ++it) {
                const int s = it % STAGES;
                if (!mbar_wait(&full_bar[s], (it / STAGES) & 1, err) ||
                    !mbar_wait(&peer_full[s], (it / STAGES) & 1, err)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t a = smem_u32(smem + s * STAGE), b = a + A_TILE;
                // the operands that go with Ar and with Ai: planes 1, 2 and 0, 1 (N,N), or 0, 1 and 1, 2
                const uint32_t br = b + (CONJ_A ? 0 : BC * BK), bi = b + (CONJ_A ? BC * BK : 0);
#pragma unroll
                for (int ks = 0; ks < BK / 32; ++ks) {
                    mma_i8(d, smem_desc(a + ks * 32), smem_desc(br + ks * 32), Cols<BC>::instr, first ? 0u : 1u);
                    mma_i8(d, smem_desc(a + BM * BK + ks * 32), smem_desc(bi + ks * 32), Cols<BC>::instr, 1u);
                    first = false;
                }
                mma_commit_pair(&empty_bar[s]);
            }
            if (ok) mma_commit_pair(&acc_full[buf]);
        }
        mma_commit_pair(&done_bar);  // no MMA left running when the blocks end
        mbar_wait(&done_bar, 0, err, false);
    } else if (warp == EPI_WARPS + 1 && lane == 0) {
        // ------------------------------------------------------------ the other CTA's full stages
        int it = 0;
        bool ok = true;
        for (int i = pair; i < total && ok; i += pairs) {
            int n, m, mod, z;
            unit_of(un, i, n, m, mod, z);
            const int k1 = min(un.nkb, (z + 1) * un.kb_per);
            for (int kb = z * un.kb_per; kb < k1; ++kb, ++it) {
                const int s = it % STAGES;
                if (!mbar_wait(&full_bar[s], (it / STAGES) & 1, err)) {
                    ok = false;
                    break;
                }
                mbar_arrive_leader(&peer_full[s]);
            }
        }
        mbar_wait(&done_bar, 0, err, false);
    } else if (warp < EPI_WARPS) {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3, h = warp >> 2;  // TMEM lanes 32 q.., columns of half h
        const int row = q * 32 + lane;
        int ui = 0;
        for (int i = pair; i < total; i += pairs, ++ui) {
            int n, m, mod, z;
            unit_of(un, i, n, m, mod, z);
            const int buf = ui & 1;
            const bool have = mbar_wait(&acc_full[buf], (ui >> 1) & 1, err);
            if (!__all_sync(0xffffffffu, have)) break;
            tc_fence_after();
            const uint32_t t = tmem + buf * 256 + h * 2 * BC + (static_cast<uint32_t>(q * 32) << 16);
            const unsigned mm = tab.m[mod], inv = tab.inv[mod];
            uint4* o = reinterpret_cast<uint4*>(
                out + ((((size_t)z * NMOD + mod) * (2 * un.mt) + 2 * m + rank) * un.nt + n) * Cols<BC>::out_tile);
#pragma unroll
            for (int g = 0; g < BC / 8; ++g) {
                uint32_t re[8], im[8];
                tmem_ld8(t + g * 8, re);
                tmem_ld8(t + BC + g * 8, im);
                tmem_wait_ld();
                unsigned w[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    unsigned b[4];
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        // below 2^31; the quotient is short by one at most
                        const unsigned tr = re[2 * j + v], ti = im[2 * j + v];
                        const unsigned rr = tr - __umulhi(tr, inv) * mm, ri = ti - __umulhi(ti, inv) * mm;
                        b[2 * v] = min(rr, rr - mm);
                        b[2 * v + 1] = min(ri, ri - mm);
                    }
                    w[j] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
                }
                o[(h * (BC / 8) + g) * BM + row] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(&acc_empty[buf]);
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // no CTA leaves while the other may still read or signal it
    if (warp == 0) tmem_free_pair(tmem);
}

// ------------------------------------------------------------------ recombination
// `mt`: tiles of 128 rows.  A thread takes one row and four columns of a tile: eight real numbers, each a
// sum of y F_i modulo 1 over the moduli, F_i = c_i / m_i in 80-bit fixed point.
// The four 20-bit digits of F_i times y < 256 add up in 32 bits over the
// 15 moduli, so a term is four plain multiply-adds and the carries wait for the
// end (80 bits leave 2^-68 P, 2^-9 of what the rounding of the operands does).
// Sums over several K ranges are reduced below m first.
template <bool SPLIT, int BC>
__global__ void __launch_bounds__(256)
zmod_combine(int M, int N, int mt, int nt, int splits, const unsigned char* __restrict__ in,
             const int* __restrict__ ea, const int* __restrict__ eb, double product, double2 alpha, double2 beta,
             double2* C, long ldc) {
    chain_begin();
    constexpr int GROUPS = BC / 4, OUT_TILE = Cols<BC>::out_tile;  // groups of eight columns a tile
    const int row = threadIdx.x >> 1, half = threadIdx.x & 1, cg = blockIdx.x % GROUPS, n = blockIdx.x / GROUPS;
    const int m = blockIdx.y, gm = m * BM + row, gn0 = n * 2 * BC + cg * 8 + half * 4;
    if (gm >= M || gn0 >= N) return;
    unsigned d[4][8];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < 8; ++j) d[q][j] = 0;
    const size_t mstride = (size_t)mt * nt * OUT_TILE, zstride = NMOD * mstride;
    const unsigned char* src = in + ((size_t)m * nt + n) * OUT_TILE + (cg * BM + row) * 16 + half * 8;
    uint2 v[NMOD];
    if (!SPLIT) {
#pragma unroll
        for (int i = 0; i < NMOD; ++i) v[i] = __ldcs(reinterpret_cast<const uint2*>(src + i * mstride));
    }
    each_mod([&](auto I) {
        constexpr int i = decltype(I)::value;
        constexpr unsigned mod = kMod[i], inv = inv_up(kMod[i]);
        constexpr unsigned f0 = fraction_digit_of(i, 0), f1 = fraction_digit_of(i, 1), f2 = fraction_digit_of(i, 2),
                           f3 = fraction_digit_of(i, 3);
        unsigned y[8];
        if (SPLIT) {
            unsigned ev[2] = {0, 0}, od[2] = {0, 0};  // two 16-bit sums each
            for (int z = 0; z < splits; ++z) {
                const uint2 w = __ldcs(reinterpret_cast<const uint2*>(src + i * mstride + z * zstride));
                ev[0] += w.x & 0x00ff00ffu;
                od[0] += (w.x >> 8) & 0x00ff00ffu;
                ev[1] += w.y & 0x00ff00ffu;
                od[1] += (w.y >> 8) & 0x00ff00ffu;
            }
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const unsigned t[4] = {ev[q] & 0xffffu, od[q] & 0xffffu, ev[q] >> 16, od[q] >> 16};
#pragma unroll
                for (int j = 0; j < 4; ++j) y[4 * q + j] = t[j] - __umulhi(t[j], inv) * mod;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                y[j] = (v[i].x >> (8 * j)) & 0xffu;
                y[4 + j] = (v[i].y >> (8 * j)) & 0xffu;
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            d[0][j] += y[j] * f0;
            d[1][j] += y[j] * f1;
            d[2][j] += y[j] * f2;
            d[3][j] += y[j] * f3;
        }
    });
    const int e_row = ea[gm];
    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
    double2 old[4];
    if (use_beta) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            old[c] = gn0 + c < N ? C[gm + (long)(gn0 + c) * ldc] : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        if (gn0 + c >= N) break;
        const int e_col = eb[gn0 + c], e = -(e_row + e_col);
        const bool fine = e_row != kNotFinite && e_col != kNotFinite;
        double part[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int j = 2 * c + p;
            const unsigned long long low = d[0][j] + (static_cast<unsigned long long>(d[1][j]) << 20);
            const unsigned long long high = (low >> 40) + d[2][j] + (static_cast<unsigned long long>(d[3][j]) << 20);
            // the top 64 of the 80 bits, signed; then the last 16
            const long long top = static_cast<long long>((high << 24) | ((low >> 16) & 0xffffffull));
            const double f = fma(static_cast<double>(top), 65536.0, static_cast<double>(static_cast<unsigned>(low) & 0xffffu));
            const double x = f * product;
            part[p] = !fine ? NAN : e > -1000 && e < 1000 ? x * pow2(e) : scalbn(x, e);
        }
        double2 r = cmul(alpha, make_double2(part[0], part[1]));
        if (use_beta) r = r + cmul(beta, old[c]);
        C[gm + (long)(gn0 + c) * ldc] = r;
    }
}

// ------------------------------------------------------------------ host side
size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

// K ranges of a product with `tiles` pair tiles: the count with the least work
// for the busiest pair of SMs, in K blocks (a unit costs about two more for its
// start)
int choose_splits(long tiles, int nkb) {
    const int pairs = device_sms() / 2 > 0 ? device_sms() / 2 : 1;
    const int least = ceil_div((long)nkb * BK, kMaxK);
    int best = least;
    long best_cost = -1;
    for (int s = least; s <= kMaxSplits && s <= nkb; ++s) {
        const int per = ceil_div(nkb, s);
        const long units = tiles * NMOD * ceil_div(nkb, per);
        const long cost = ((units + pairs - 1) / pairs) * (per + 2);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = s;
        }
    }
    return best;
}

// tiles of 2 x 32 columns where 2 x 64 would be half empty
bool narrow(int N) { return N <= 64; }

struct Plan {
    int bc, mt, nt, nkb, splits, kb_per, panel;  // panel: pair tiles along M that a launch takes
    size_t b_bytes, a_bytes, out_bytes, exp_bytes, balance_bytes, total;
};

// the output bytes of one panel and the rows of A that are packed with it stay below this
constexpr size_t kPanelBytes = 640ull << 20;

Plan plan_of(bool conj_a, int M, int N, int K, bool packed) {
    Plan p;
    p.bc = narrow(N) ? 32 : 64;
    p.mt = ceil_div(M, 2 * BM);
    p.nt = ceil_div(N, 2 * p.bc);
    p.nkb = ceil_div(K, BK);
    const size_t b_tile = narrow(N) ? Cols<32>::b_tile : Cols<64>::b_tile;
    const size_t out_tile = narrow(N) ? Cols<32>::out_tile : Cols<64>::out_tile;
    const int s = conj_a ? choose_splits((long)p.mt * p.nt, p.nkb) : ceil_div((long)p.nkb * BK, kMaxK);
    p.kb_per = ceil_div(p.nkb, s);
    p.splits = ceil_div(p.nkb, p.kb_per);
    const size_t per = 2 * ((size_t)p.nt * NMOD * out_tile * p.splits + (packed ? 0 : (size_t)p.nkb * NMOD * A_TILE));
    p.panel = static_cast<int>(kPanelBytes / per);
    if (p.panel < 1) p.panel = 1;
    if (p.panel > p.mt) p.panel = p.mt;
    p.b_bytes = (size_t)p.nt * 2 * p.nkb * NMOD * b_tile;
    p.a_bytes = packed ? 0 : (size_t)p.panel * 2 * p.nkb * NMOD * A_TILE;
    p.out_bytes = (size_t)p.panel * 2 * p.nt * NMOD * out_tile * p.splits;
    p.exp_bytes = align256(((size_t)p.panel * 2 * BM + (size_t)p.nt * 2 * p.bc) * sizeof(int));
    p.balance_bytes = !conj_a && !packed ? align256(balance_ints(K) * sizeof(int)) : 0;
    p.total = p.b_bytes + p.a_bytes + p.out_bytes + p.exp_bytes + p.balance_bytes;
    return p;
}

template <typename F> void allow_smem(F* f, int bytes) {
    Q3B_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}
void set_limits() {
    static PerDeviceOnce once;
    once.run([] {
        allow_smem(zmod_gemm<true, 64>, Cols<64>::smem);
        allow_smem(zmod_gemm<false, 64>, Cols<64>::smem);
        allow_smem(zmod_gemm<true, 32>, Cols<32>::smem);
        allow_smem(zmod_gemm<false, 32>, Cols<32>::smem);
        allow_smem(pack_rows<true, BM, kPackA>, PACK_SMEM);
        allow_smem(pack_rows<false, BM, kPackA>, PACK_SMEM);
        allow_smem(pack_rows<true, 64, kPackB>, PACK_SMEM);
        allow_smem(pack_rows<true, 64, kPackBConj>, PACK_SMEM);
        allow_smem(pack_rows<true, 32, kPackB>, PACK_SMEM);
        allow_smem(pack_rows<true, 32, kPackBConj>, PACK_SMEM);
    });
}

// scales and residue tiles of R rows, padded to whole pair tiles (2 ROWS)
template <bool KMAJOR, int ROWS, int AS>
void pack_operand(cudaStream_t st, int R, int K, const double2* X, long ld, const int* balance, unsigned char* tiles,
                  int* exps) {
    const Balance bal{balance, AS == kPackA ? -1 : 1};
    const int padded = ceil_div(R, 2 * ROWS) * 2 * ROWS, nkb = ceil_div(K, BK);
    if (nkb > 65535) throw std::runtime_error("complex GEMM: operand too large to pack");
    if (KMAJOR && K >= kLongRow)
        launch_chained(exps_kmajor<1024>, padded, 1024, 0, st, R, K, X, ld, scale_bits(), bal, 0, exps);
    else if (KMAJOR) launch_chained(exps_kmajor<256>, padded, 256, 0, st, R, K, X, ld, scale_bits(), bal, 0, exps);
    else launch_chained(exps_mmajor<8>, padded / 32, 256, 0, st, R, K, X, ld, scale_bits(), bal, 0, exps);
    Q3B_LAUNCH_CHECK();
    launch_chained(pack_rows<KMAJOR, ROWS, AS>, dim3(padded / PACK_ROWS, nkb), 256, PACK_SMEM, st, R, K, X, ld, bal, exps, nkb, tiles);
    Q3B_LAUNCH_CHECK();
}
void pack_rows_of_a(cudaStream_t st, int M, int K, const double2* A, long lda, bool kmajor, const int* balance,
                    unsigned char* tiles, int* exps) {
    if (kmajor) pack_operand<true, BM, kPackA>(st, M, K, A, lda, balance, tiles, exps);
    else pack_operand<false, BM, kPackA>(st, M, K, A, lda, balance, tiles, exps);
}

template <bool CONJ_A, int BC>
void run_panel(cudaStream_t st, const Plan& p, int rows, int mt, int N, const unsigned char* a, const unsigned char* b,
               unsigned char* out, const int* ea, const int* eb, double product, double2 alpha, double2 beta,
               double2* C, long ldc, const ModTable& tab) {
    const long units = (long)mt * p.nt * NMOD * p.splits;
    if (units > 0x7fffffffL || 2 * mt > 65535) throw std::runtime_error("complex GEMM: too large");
    const Units un{p.nt, mt, p.splits, p.kb_per, p.nkb, !CONJ_A};
    const long pairs = device_sms() / 2 > 0 ? device_sms() / 2 : 1;
    const int grid = 2 * static_cast<int>(units < pairs ? units : pairs);
    launch_chained(zmod_gemm<CONJ_A, BC>, grid, THREADS, Cols<BC>::smem, st, un, (int)units, a, b, out, tab, tc::error_word());
    Q3B_LAUNCH_CHECK();
    const dim3 cgrid(p.nt * (BC / 4), 2 * mt);
    if (p.splits > 1)
        launch_chained(zmod_combine<true, BC>, cgrid, 256, 0, st, rows, N, 2 * mt, p.nt, p.splits, out, ea, eb, product, alpha,
                                                      beta, C, ldc);
    else
        launch_chained(zmod_combine<false, BC>, cgrid, 256, 0, st, rows, N, 2 * mt, p.nt, p.splits, out, ea, eb, product, alpha,
                                                       beta, C, ldc);
    Q3B_LAUNCH_CHECK();
}

ModTable mod_table() {
    ModTable t;
    for (int i = 0; i < NMOD; ++i) {
        const unsigned m = kMod[i];
        t.m[i] = m;
        t.inv[i] = static_cast<unsigned>(0x100000000ull / m);
    }
    return t;
}

}  // namespace

size_t packed_a_bytes(int M, int K) { return (size_t)ceil_div(M, 2 * BM) * 2 * ceil_div(K, BK) * NMOD * A_TILE; }
size_t packed_a_exps(int M) { return (size_t)ceil_div(M, 2 * BM) * 2 * BM; }

void pack_a(cudaStream_t st, int M, int K, const double2* A, long lda, bool kmajor, const int* balance,
            unsigned char* tiles, int* exps) {
    if (M <= 0 || K <= 0) return;
    set_limits();
    pack_rows_of_a(st, M, K, A, lda, kmajor, balance, tiles, exps);
}

size_t balance_ints(int lines) { return (size_t)ceil_div(lines, BK) * BK; }

void balance_projectors(cudaStream_t st, int npw, int nproj, const double2* beta, int* along_proj, int* along_pw) {
    if (npw <= 0 || nproj <= 0) return;
    launch_chained(exps_kmajor<256>, nproj, 256, 0, st, nproj, npw, beta, npw, scale_bits(), Balance{nullptr, 0}, kZeroLine,
                   along_proj);
    Q3B_LAUNCH_CHECK();
    launch_chained(balance_lines, 1, 1024, 0, st, nproj, (int)balance_ints(nproj), -1, along_proj);
    Q3B_LAUNCH_CHECK();
    launch_chained(exps_mmajor<8>, ceil_div(npw, 32), 256, 0, st, npw, nproj, beta, npw, scale_bits(),
                   Balance{along_proj, -1}, kZeroLine, along_pw);
    Q3B_LAUNCH_CHECK();
    launch_chained(balance_lines, 1, 1024, 0, st, npw, (int)balance_ints(npw), -1, along_pw);
    Q3B_LAUNCH_CHECK();
}

// Estimated times of both paths, from runs of q3b_gemm_residue and q3b_gemm on shapes
// of the 8- to 128-atom cells (B200, 1965 MHz): here 19 ps per packed entry, 60 ns per
// 128 x 64 tile and K block, 10 ps per output, and 40 us of launches; on the FP64 units
// as their own tiles are chosen.  Measured, here against there: 23847 x 256 x 512
// (N,N) 0.48 ms against 1.00, 512 x 256 x 23847 (C,N) 0.51 against 0.96,
// 1024 x 512 x 62669 (C,N) 3.5 against 10.2; the two meet near 23847 x 64 x 512 (N,N, 0.35
// against 0.30), 12000 x 128 x 256 (N,N, 0.145 against 0.158) and 256 x 128 x 12000 (C,N,
// 0.157 against 0.142).  With A packed before (the projectors), beta Q beta^H psi of 90
// bands of the 64-atom cell takes 0.37 ms against 1.14.
bool worth(bool conj_a, int M, int N, int K, bool packed) {
    if (M < 64 || N < 16 || K < 64 || K > kLongestK) return false;
    const double tiles = (double)ceil_div(M, 2 * BM) * (narrow(N) ? 2 : 4 * ceil_div(N, 128)) * ceil_div(K, BK);
    const double entries = (double)K * N + (packed ? 0.0 : (double)M * K);
    const double here = 40e-6 + 19e-12 * entries + 60e-9 * tiles + 10e-12 * (double)M * N;
    return here < fp64_units_seconds(conj_a, M, N, K);
}

size_t workspace_bytes(bool conj_a, int M, int N, int K, bool packed) {
    return plan_of(conj_a, M, N, K, packed).total;
}

void zgemm(cudaStream_t st, bool conj_a, int M, int N, int K, double2 alpha, const double2* A, long lda,
           const PackedA* pk, const double2* B, long ldb, double2 beta, double2* C, long ldc,
           const GemmWorkspace& ws) {
    if (M <= 0 || N <= 0) return;
    if (pk && (!pk->tiles || pk->M != M || pk->K != K))
        throw std::runtime_error("complex GEMM: packed operand of another shape");
    const Plan p = plan_of(conj_a, M, N, K, pk != nullptr);
    if (!ws.ptr || ws.bytes < p.total) throw std::runtime_error("complex GEMM: workspace too small");
    set_limits();
    unsigned char* w = static_cast<unsigned char*>(ws.ptr);
    unsigned char* bt = w;
    unsigned char* at = bt + p.b_bytes;
    unsigned char* out = at + p.a_bytes;
    int* eb = reinterpret_cast<int*>(out + p.out_bytes);
    int* ea_ws = eb + (size_t)p.nt * 2 * p.bc;
    long double prod = std::ldexp(1.0L, -80);
    for (int m : kMod) prod *= m;
    const double product = static_cast<double>(prod);
    const int* balance = pk ? pk->balance : nullptr;
    if (p.balance_bytes) {
        int* rows_of_b = reinterpret_cast<int*>(out + p.out_bytes + p.exp_bytes);
        launch_chained(exps_mmajor<32>, ceil_div(K, 32), 1024, 0, st, K, N, B, ldb, scale_bits(),
                       Balance{nullptr, 0}, kZeroLine, rows_of_b);
        Q3B_LAUNCH_CHECK();
        launch_chained(balance_lines, 1, 1024, 0, st, K, (int)balance_ints(K), 1, rows_of_b);
        Q3B_LAUNCH_CHECK();
        balance = rows_of_b;
    }
    if (p.bc == 64) {
        if (conj_a) pack_operand<true, 64, kPackBConj>(st, N, K, B, ldb, balance, bt, eb);
        else pack_operand<true, 64, kPackB>(st, N, K, B, ldb, balance, bt, eb);
    } else {
        if (conj_a) pack_operand<true, 32, kPackBConj>(st, N, K, B, ldb, balance, bt, eb);
        else pack_operand<true, 32, kPackB>(st, N, K, B, ldb, balance, bt, eb);
    }
    const ModTable tab = mod_table();
    for (int m0 = 0; m0 < p.mt; m0 += p.panel) {
        const int mt = p.mt - m0 < p.panel ? p.mt - m0 : p.panel;
        const long r0 = (long)m0 * 2 * BM;
        const int rows = static_cast<int>(M - r0 < (long)mt * 2 * BM ? M - r0 : (long)mt * 2 * BM);
        const unsigned char* a = pk ? pk->tiles + (size_t)m0 * 2 * p.nkb * NMOD * A_TILE : at;
        const int* ea = pk ? pk->exps + r0 : ea_ws;
        if (!pk) pack_rows_of_a(st, rows, K, conj_a ? A + r0 * lda : A + r0, lda, conj_a, balance, at, ea_ws);
        auto run = [&](auto conj) {
            constexpr bool CA = decltype(conj)::value;
            if (p.bc == 64)
                run_panel<CA, 64>(st, p, rows, mt, N, a, bt, out, ea, eb, product, alpha, beta, C + r0, ldc, tab);
            else run_panel<CA, 32>(st, p, rows, mt, N, a, bt, out, ea, eb, product, alpha, beta, C + r0, ldc, tab);
        };
        if (conj_a) run(std::true_type{});
        else run(std::false_type{});
    }
}

}  // namespace zmod
}  // namespace q3b
