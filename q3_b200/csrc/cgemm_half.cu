// FP32 complex GEMMs with a packed A operand on the FP16 tensor cores
// (tcgen05 kind::f16, sm_100a), for the projector products.
//
//   "C,N":  C = alpha A^H B + beta C    (A: K x M; B: K x N, ldb)
//   "N,N":  C = alpha A B   + beta C    (A: M x K; B: K x N, ldb)
//
// Every row of op(A) and column of B is scaled by a power of two so that its
// largest part lies in [2^13, 2^14), and every part is split into two FP16
// numbers, x = hi + lo with hi = rn(x), lo = rn(x - hi): 22 bits, what a split
// into two TF32 numbers keeps, for parts down to 2^-18 of the row's largest (lo
// stays normal), and an absolute 2^-39 of it below.  So that the large parts of the
// one operand do not meet the small ones of the other, beta and the bands are first
// balanced along K by powers of two (PackedA::balance).  A real product is
// hi*hi + hi*lo + lo*hi, accumulated in FP32 in TMEM, as in the TF32 kernel
// (cgemm_tc.cu) at twice the tensor rate and half the operand bytes.
//
// B is packed once a call into the image the stages take, where the TF32 kernel
// converts it again in every row tile (187 of them for beta B' of the 64-atom
// cell) and its producers, not the tensor pipe, set the pace.
//
// A pair of CTAs works on tiles of 256 rows x 2 BC columns (cta_group::2), each
// CTA holding 128 rows of A and BC columns of B; B has three planes per FP16
// number, so that one operand goes with Ar and one with Ai and both parts of
// the output add up in one accumulator (see zgemm_mod.cu, whose roles of warps,
// barriers and units this kernel shares).  Per 64 of K: 112 KB a CTA, 24 MMAs of
// 128 clocks.  At 256 bands of the 64-atom cell (512 projectors, 23847 plane
// waves) <beta|psi> takes 115 us against 146 on the TF32 kernel with its packed
// A, beta B' 87 against 154, and H|psi> is half as far from 64 bits (4e-7
// against 9e-7), the K ranges summed in TMEM being shorter.
#include <cuda_fp16.h>

#include <cmath>
#include <type_traits>

#include "cgemm_half.cuh"
#include "umma_pair.cuh"

namespace q3b {
namespace half2x {
namespace {

using namespace umma;

constexpr int BM = 128;              // complex rows a CTA holds of a pair's 256
constexpr int BK = 64;               // K per stage: one 128-byte row of FP16
static_assert(kLongestK == 65535 * BK, "a grid row per stage");
constexpr int ROW = 128;             // bytes
constexpr int A_TILE = 4 * BM * ROW;  // re hi, re lo, im hi, im lo
constexpr int STAGES = 2;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (EPI_WARPS + 2);
constexpr int kMaxSplits = 64;
constexpr int kTop = 14;             // scaled parts stay below 2^kTop
template <int BC> struct Cols {
    static constexpr int plane = BC * ROW;
    static constexpr int b_tile = 6 * plane;  // three planes of hi, three of lo
    static constexpr int smem = STAGES * (A_TILE + b_tile) + 1024;
    // D f32, A and B f16, K-major, M = 256, N = 4 BC
    static constexpr uint32_t instr = (1u << 4) | (static_cast<uint32_t>((4 * BC) >> 3) << 17) |
                                      (static_cast<uint32_t>((2 * BM) >> 4) << 24);
};

// ------------------------------------------------------------------ row scales
__device__ __forceinline__ int exponent_for(float mx) {
    if (!(mx > 0.f) || !(mx < INFINITY)) return 0;
    int e;
    frexpf(mx, &e);  // mx < 2^e
    return kTop - e;
}
__device__ __forceinline__ float larger(float mx, float2 v) { return fmaxf(mx, fmaxf(fabsf(v.x), fabsf(v.y))); }
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }

// The operands along K (PackedA::balance): A and B times 2^(sign balance[k]), with opposite
// signs.  Lines of A more than 2^60 below the largest are left 2^60 below it.
struct Balance {
    const int* exps;
    int sign;
    __device__ __forceinline__ int at(int k) const { return exps ? sign * max(exps[k], -60) : 0; }
    // of eight places from a multiple of eight on (the array is padded with zeros)
    __device__ __forceinline__ void get8(int k, int* e) const {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int4 v = exps ? *reinterpret_cast<const int4*>(exps + k + 4 * q) : make_int4(0, 0, 0, 0);
            e[4 * q] = sign * max(v.x, -60);
            e[4 * q + 1] = sign * max(v.y, -60);
            e[4 * q + 2] = sign * max(v.z, -60);
            e[4 * q + 3] = sign * max(v.w, -60);
        }
    }
};

// one block of NT threads a row, 1024 from kLongRow of K on
constexpr int kLongRow = 4096;
template <int NT>
__global__ void __launch_bounds__(NT) exps_kmajor(int R, int K, const float2* __restrict__ X, long ld, Balance bal,
                                                   int* exps) {
    chain_begin();
    const int r = blockIdx.x;
    float mx = 0.f;
    if (r < R) {
        const float2* x = X + (long)r * ld;
        for (int k = threadIdx.x; k < K; k += 8 * NT) {
            float2 v[8];
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool ok = k + NT * u < K;
                v[u] = ok ? x[k + NT * u] : make_float2(0.f, 0.f);
                f[u] = pow2f(ok ? bal.at(k + NT * u) : 0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) mx = larger(mx, f[u] * v[u]);
        }
    }
    __shared__ float s[NT / 32];
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < NT / 32; ++w) mx = fmaxf(mx, s[w]);
        exps[r] = exponent_for(mx);
    }
}

__global__ void __launch_bounds__(256) exps_mmajor(int R, int K, const float2* __restrict__ X, long ld, Balance bal,
                                                   int* exps) {
    chain_begin();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r = blockIdx.x * 32 + lane;
    float mx = 0.f;
    if (r < R) {
        for (int k = w; k < K; k += 8 * 8) {
            float2 v[8];
            float f[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const bool ok = k + 8 * u < K;
                v[u] = ok ? X[r + (long)(k + 8 * u) * ld] : make_float2(0.f, 0.f);
                f[u] = pow2f(ok ? bal.at(k + 8 * u) : 0);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) mx = larger(mx, f[u] * v[u]);
        }
    }
    __shared__ float s[8][32];
    s[w][lane] = mx;
    __syncthreads();
    if (w == 0) {
        for (int j = 1; j < 8; ++j) mx = fmaxf(mx, s[j][lane]);
        exps[r] = exponent_for(mx);
    }
}

// x 2^e without leaving the range on the way (|e| up to 163, and 60 along K)
__device__ __forceinline__ float scaled(float x, float f1, float f2) { return x * f1 * f2; }

// ------------------------------------------------------------------ packing
// 32 rows x 64 K a block; a thread takes eight consecutive K of one row and writes
// one 16-byte chunk per plane, in the 128-byte swizzle.  Tiles: [tile of ROWS]
// [kb][plane][ROWS][128 bytes]; the planes of A and B as the constants above say,
// B's three being -im, re, im (N,N) or re, im, -re (C,N).
enum PackAs { kPackA, kPackB, kPackBConj };
constexpr int PACK_ROWS = 32;
constexpr int PACK_PITCH = 8 * 9 + 1;  // float2 per row: chunks of 8 + 1, odd in all

template <bool KMAJOR, int ROWS, int AS>
__global__ void __launch_bounds__(256) pack_rows(int R, int K, const float2* __restrict__ X, long ld,
                                                 Balance bal, const int* __restrict__ exps, int nkb,
                                                 unsigned char* out) {
    chain_begin();
    __shared__ float2 s[PACK_ROWS * PACK_PITCH];
    const int tid = threadIdx.x, kb = blockIdx.y, k0 = kb * BK, r0 = blockIdx.x * PACK_ROWS;
    float2 in[PACK_ROWS * BK / 256];
#pragma unroll
    for (int i = 0; i < PACK_ROWS * BK / 256; ++i) {
        const int idx = tid + i * 256;
        const int gr = r0 + (KMAJOR ? idx / BK : idx % PACK_ROWS), gk = k0 + (KMAJOR ? idx % BK : idx / PACK_ROWS);
        in[i] = make_float2(0.f, 0.f);
        if (gr < R && gk < K) in[i] = KMAJOR ? X[(long)gr * ld + gk] : X[gr + (long)gk * ld];
    }
#pragma unroll
    for (int i = 0; i < PACK_ROWS * BK / 256; ++i) {
        const int idx = tid + i * 256;
        const int row = KMAJOR ? idx / BK : idx % PACK_ROWS, k = KMAJOR ? idx % BK : idx / PACK_ROWS;
        s[row * PACK_PITCH + (k >> 3) * 9 + (k & 7)] = in[i];
    }
    __syncthreads();
    const int row = tid >> 3, ch = tid & 7, gr = r0 + row, e = exps[gr];
    int along[8];
    bal.get8(k0 + 8 * ch, along);
    unsigned hi[2][4], lo[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 a = s[row * PACK_PITCH + ch * 9 + 2 * j], b = s[row * PACK_PITCH + ch * 9 + 2 * j + 1];
        const int ea = e + along[2 * j], eb = e + along[2 * j + 1];
        const float a1 = pow2f(ea / 2), a2 = pow2f(ea - ea / 2), b1 = pow2f(eb / 2), b2 = pow2f(eb - eb / 2);
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float x = scaled(p ? a.y : a.x, a1, a2), y = scaled(p ? b.y : b.x, b1, b2);
            const __half2 h = __floats2half2_rn(x, y);
            const float2 hf = __half22float2(h);
            const __half2 l = __floats2half2_rn(x - hf.x, y - hf.y);
            hi[p][j] = *reinterpret_cast<const unsigned*>(&h);
            lo[p][j] = *reinterpret_cast<const unsigned*>(&l);
        }
    }
    const int tile = gr / ROWS, rr = gr % ROWS;
    constexpr int PLANE = ROWS * ROW, PLANES = AS == kPackA ? 4 : 6;
    unsigned char* dst = out + ((size_t)tile * nkb + kb) * (PLANES * PLANE) + rr * ROW + ((ch ^ (rr & 7)) << 4);
    auto put = [&](int plane, const unsigned* v, unsigned flip) {
        *reinterpret_cast<uint4*>(dst + plane * PLANE) = make_uint4(v[0] ^ flip, v[1] ^ flip, v[2] ^ flip, v[3] ^ flip);
    };
    constexpr unsigned kMinus = 0x80008000u;
    if constexpr (AS == kPackA) {
        put(0, hi[0], 0);
        put(1, lo[0], 0);
        put(2, hi[1], 0);
        put(3, lo[1], 0);
    } else if constexpr (AS == kPackB) {
        put(0, hi[1], kMinus);
        put(1, hi[0], 0);
        put(2, hi[1], 0);
        put(3, lo[1], kMinus);
        put(4, lo[0], 0);
        put(5, lo[1], 0);
    } else {
        put(0, hi[0], 0);
        put(1, hi[1], 0);
        put(2, hi[0], kMinus);
        put(3, lo[0], 0);
        put(4, lo[1], 0);
        put(5, lo[0], kMinus);
    }
}

// ------------------------------------------------------------------ products
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t instr, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
        "l"(a), "l"(b), "r"(instr), "r"(accumulate)
        : "memory");
}

// units: tiles along N fastest, then M, then the K ranges
struct Units {
    int nt, mt, kb_per, nkb;
};
__device__ __forceinline__ void unit_of(const Units& u, int i, int& n, int& m, int& z) {
    n = i % u.nt;
    i /= u.nt;
    m = i % u.mt;
    z = i / u.mt;
}

template <bool CONJ_A, int BC>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
half_gemm(Units un, int total, int M, int N, const unsigned char* __restrict__ A, const unsigned char* __restrict__ B,
          const int* __restrict__ ea, const int* __restrict__ eb, float2 alpha, float2 beta, float2* C, long ldc,
          float2* part, int* err) {
    chain_begin();
    constexpr int B_TILE = Cols<BC>::b_tile, STAGE = A_TILE + B_TILE, PLANE = Cols<BC>::plane;
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
            int n, m, z;
            unit_of(un, i, n, m, z);
            const int k1 = min(un.nkb, (z + 1) * un.kb_per);
            for (int kb = z * un.kb_per; kb < k1; ++kb, ++it) {
                const int s = it % STAGES;
                if (it >= STAGES && !mbar_wait(&empty_bar[s], ((it / STAGES) - 1) & 1, err)) {
                    ok = false;
                    break;
                }
                unsigned char* st = smem + s * STAGE;
                mbar_arrive_tx(&full_bar[s], STAGE);
                bulk_copy_g2s(st, A + ((size_t)(2 * m + rank) * un.nkb + kb) * A_TILE, A_TILE, &full_bar[s]);
                bulk_copy_g2s(st + A_TILE, B + ((size_t)(2 * n + rank) * un.nkb + kb) * B_TILE, B_TILE, &full_bar[s]);
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
            int n, m, z;
            unit_of(un, i, n, m, z);
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
#pragma unroll
                for (int ks = 0; ks < BK / 16; ++ks) {
#pragma unroll
                    for (int t = 0; t < 6; ++t) {
                        const int im = t / 3, term = t % 3;  // hi*hi, hi*lo, lo*hi
                        const uint32_t ap = a + (2 * im + (term == 2 ? 1 : 0)) * (BM * ROW) + ks * 32;
                        // the planes that go with Ar: 1, 2 (N,N) or 0, 1 (C,N); with Ai: 0, 1 or 1, 2
                        const int plane = (CONJ_A ? im : 1 - im) + (term == 1 ? 3 : 0);
                        mma_f16(d, smem_desc(ap), smem_desc(b + plane * PLANE + ks * 32), Cols<BC>::instr,
                                first && t == 0 ? 0u : 1u);
                    }
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
            int n, m, z;
            unit_of(un, i, n, m, z);
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
        const bool use_beta = (beta.x != 0.f || beta.y != 0.f);
        int ui = 0;
        for (int i = pair; i < total; i += pairs, ++ui) {
            int n, m, z;
            unit_of(un, i, n, m, z);
            const int buf = ui & 1;
            const bool have = mbar_wait(&acc_full[buf], (ui >> 1) & 1, err);
            if (!__all_sync(0xffffffffu, have)) break;
            tc_fence_after();
            const uint32_t t = tmem + buf * 256 + h * 2 * BC + (static_cast<uint32_t>(q * 32) << 16);
            const int row = (2 * m + rank) * BM + q * 32 + lane, col0 = n * 2 * BC + h * BC;
            const int er = row < M ? ea[row] : 0;
#pragma unroll 1
            for (int g = 0; g < BC / 8; ++g) {
                __syncwarp();  // the loads below are the warp's
                uint32_t re[8], im[8];
                tmem_ld8(t + g * 8, re);
                tmem_ld8(t + BC + g * 8, im);
                tmem_wait_ld();
                if (row >= M) continue;
                const int c0 = col0 + g * 8;
                float2 old[8];
                if (use_beta && !part) {  // all the old values before the first is replaced
#pragma unroll
                    for (int j = 0; j < 8; ++j) old[j] = c0 + j < N ? C[row + (long)(c0 + j) * ldc] : make_float2(0.f, 0.f);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    if (c0 + j >= N) break;
                    const int e = -(er + eb[c0 + j]);
                    float2 v = make_float2(__uint_as_float(re[j]), __uint_as_float(im[j]));
                    if (e > -126 && e < 127) {
                        const float f = pow2f(e);
                        v.x *= f;
                        v.y *= f;
                    } else {
                        v.x = scalbnf(v.x, e);
                        v.y = scalbnf(v.y, e);
                    }
                    if (part) {
                        part[((size_t)z * N + c0 + j) * M + row] = v;
                    } else {
                        float2 r = cmul(alpha, v);
                        if (use_beta) r = r + cmul(beta, old[j]);
                        C[row + (long)(c0 + j) * ldc] = r;
                    }
                }
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

// C = alpha * sum_z part[z] + beta * C, the ranges in order
__global__ void sum_ranges(int M, int N, int ranges, const float2* __restrict__ part, float2 alpha, float2 beta,
                           float2* C, long ldc) {
    chain_begin();
    const long total = (long)M * N;
    const bool use_beta = (beta.x != 0.f || beta.y != 0.f);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const int m = static_cast<int>(i % M), n = static_cast<int>(i / M);
        float2 s = part[i];
#pragma unroll 4
        for (int z = 1; z < ranges; ++z) s = s + part[(long)z * total + i];
        float2 v = cmul(alpha, s);
        float2* c = C + m + (long)n * ldc;
        if (use_beta) v = v + cmul(beta, *c);
        *c = v;
    }
}

// ------------------------------------------------------------------ host side
size_t align256(size_t n) { return (n + 255) & ~size_t(255); }

struct Plan {
    int bc, mt, nt, nkb, splits, kb_per;
    size_t b_bytes, part_bytes, total;
};

// K ranges (C,N): the count with the least work for the busiest pair of SMs, a
// range costing about one K block to start
Plan plan_of(bool conj_a, int M, int N, int K) {
    Plan p;
    p.bc = N <= 64 ? 32 : 64;
    p.mt = ceil_div(M, 2 * BM);
    p.nt = ceil_div(N, 2 * p.bc);
    p.nkb = ceil_div(K, BK);
    const int pairs = device_sms() / 2 > 0 ? device_sms() / 2 : 1;
    int s = 1;
    if (conj_a) {
        long best = -1;
        for (int t = 1; t <= kMaxSplits && t <= p.nkb; ++t) {
            const int per = ceil_div(p.nkb, t);
            const long units = (long)p.mt * p.nt * ceil_div(p.nkb, per);
            const long cost = ((units + pairs - 1) / pairs) * (per + 1);
            if (best < 0 || cost < best) {
                best = cost;
                s = t;
            }
        }
    }
    p.kb_per = ceil_div(p.nkb, s);
    p.splits = ceil_div(p.nkb, p.kb_per);
    p.b_bytes = (size_t)p.nt * 2 * p.nkb * (p.bc == 64 ? Cols<64>::b_tile : Cols<32>::b_tile);
    p.part_bytes = p.splits > 1 ? align256((size_t)p.splits * M * N * sizeof(float2)) : 0;
    p.total = p.b_bytes + p.part_bytes + align256((size_t)p.nt * 2 * p.bc * sizeof(int));
    return p;
}

template <typename F> void allow_smem(F* f, int bytes) {
    Q3B_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}
void set_limits() {
    static PerDeviceOnce once;
    once.run([] {
        allow_smem(half_gemm<true, 64>, Cols<64>::smem);
        allow_smem(half_gemm<false, 64>, Cols<64>::smem);
        allow_smem(half_gemm<true, 32>, Cols<32>::smem);
        allow_smem(half_gemm<false, 32>, Cols<32>::smem);
    });
}

// scales and tiles of R rows, padded to whole pair tiles (2 ROWS)
template <bool KMAJOR, int ROWS, int AS>
void pack_operand(cudaStream_t st, int R, int K, const float2* X, long ld, const int* balance, unsigned char* tiles,
                  int* exps) {
    const Balance bal{balance, AS == kPackA ? -1 : 1};
    const int padded = ceil_div(R, 2 * ROWS) * 2 * ROWS, nkb = ceil_div(K, BK);
    if (K > kLongestK) throw std::runtime_error("tensor-core GEMM: operand too large to pack");
    if (KMAJOR && K >= kLongRow) launch_chained(exps_kmajor<1024>, padded, 1024, 0, st, R, K, X, ld, bal, exps);
    else if (KMAJOR) launch_chained(exps_kmajor<256>, padded, 256, 0, st, R, K, X, ld, bal, exps);
    else launch_chained(exps_mmajor, padded / 32, 256, 0, st, R, K, X, ld, bal, exps);
    Q3B_LAUNCH_CHECK();
    launch_chained(pack_rows<KMAJOR, ROWS, AS>, dim3(padded / PACK_ROWS, nkb), 256, 0, st, R, K, X, ld, bal, exps, nkb, tiles);
    Q3B_LAUNCH_CHECK();
}

template <bool CONJ_A, int BC>
void run(cudaStream_t st, const Plan& p, int M, int N, int K, float2 alpha, const PackedA& A, const float2* B, long ldb,
         float2 beta, float2* C, long ldc, unsigned char* bt, float2* part, int* eb) {
    pack_operand<true, BC, CONJ_A ? kPackBConj : kPackB>(st, N, K, B, ldb, A.balance, bt, eb);
    const long units = (long)p.mt * p.nt * p.splits, pairs = device_sms() / 2 > 0 ? device_sms() / 2 : 1;
    if (units > 0x7fffffffL) throw std::runtime_error("tensor-core GEMM: too large");
    const int grid = 2 * static_cast<int>(units < pairs ? units : pairs);
    launch_chained(half_gemm<CONJ_A, BC>, grid, THREADS, Cols<BC>::smem, st, Units{p.nt, p.mt, p.kb_per, p.nkb}, (int)units, M, N,
                                                                 A.tiles, bt, A.exps, eb, alpha, beta, C, ldc, part,
                                                                 tc::error_word());
    Q3B_LAUNCH_CHECK();
    if (part) {
        launch_chained(sum_ranges, stride_grid((long)M * N, 16), 256, 0, st, M, N, p.splits, part, alpha, beta, C, ldc);
        Q3B_LAUNCH_CHECK();
    }
}

}  // namespace

size_t packed_a_bytes(int M, int K) { return (size_t)ceil_div(M, 2 * BM) * 2 * ceil_div(K, BK) * A_TILE; }
size_t packed_a_exps(int M) { return (size_t)ceil_div(M, 2 * BM) * 2 * BM; }

void pack_a(cudaStream_t st, int M, int K, const float2* A, long lda, bool kmajor, const int* balance,
            unsigned char* tiles, int* exps) {
    if (M <= 0 || K <= 0) return;
    if (kmajor) pack_operand<true, BM, kPackA>(st, M, K, A, lda, balance, tiles, exps);
    else pack_operand<false, BM, kPackA>(st, M, K, A, lda, balance, tiles, exps);
}

size_t workspace_bytes(bool conj_a, int M, int N, int K) { return plan_of(conj_a, M, N, K).total; }

void cgemm(cudaStream_t st, bool conj_a, int M, int N, int K, float2 alpha, const PackedA& A, const float2* B,
           long ldb, float2 beta, float2* C, long ldc, const GemmWorkspace& ws) {
    if (M <= 0 || N <= 0) return;
    if (!A.tiles || A.M != M || A.K != K) throw std::runtime_error("tensor-core GEMM: packed A of another shape");
    const Plan p = plan_of(conj_a, M, N, K);
    if (!ws.ptr || ws.bytes < p.total) throw std::runtime_error("tensor-core GEMM: workspace too small");
    set_limits();
    unsigned char* bt = static_cast<unsigned char*>(ws.ptr);
    float2* part = p.splits > 1 ? reinterpret_cast<float2*>(bt + p.b_bytes) : nullptr;
    int* eb = reinterpret_cast<int*>(bt + p.b_bytes + p.part_bytes);
    auto go = [&](auto conj) {
        constexpr bool CA = decltype(conj)::value;
        if (p.bc == 64) run<CA, 64>(st, p, M, N, K, alpha, A, B, ldb, beta, C, ldc, bt, part, eb);
        else run<CA, 32>(st, p, M, N, K, alpha, A, B, ldb, beta, C, ldc, bt, part, eb);
    };
    if (conj_a) go(std::true_type{});
    else go(std::false_type{});
}

}  // namespace half2x
}  // namespace q3b
