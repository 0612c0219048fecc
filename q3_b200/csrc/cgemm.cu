#include <algorithm>
// Complex GEMMs on CUDA cores; see cgemm.cuh.
#include <cstdint>
#include <type_traits>

#include "cgemm.cuh"
#include "zgemm_mod.cuh"

namespace q3b {
namespace {

constexpr int kThreads = 256;
constexpr int kBK = 16;      // K per stage
constexpr int kStages = 4;
constexpr int kKP = kBK + 1;  // pitch of [m][k] and [n][k]

// one complex value, global -> shared (zeros where not valid)
template <typename T> __device__ __forceinline__ void cp_async(T* dst, const T* src, bool valid) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if constexpr (sizeof(T) == 16) {
        const int n = valid ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    } else {
        const int n = valid ? 8 : 0;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <typename R, int TM, int TN> struct PipeTile {
    static constexpr int bm = 16 * TM, bn = 16 * TN;
    static constexpr int a_pitch_n = bm + 4;  // [k][m]
    static constexpr int a_stage = kBK * a_pitch_n > bm * kKP ? kBK * a_pitch_n : bm * kKP;
    static constexpr int b_stage = bn * kKP;
    static constexpr size_t smem = (size_t)kStages * (a_stage + b_stage) * sizeof(cplx_t<R>);
};

// Products too small for the large tiles below: bm x bn tiles of C (32 x 16, 32 x 32
// or 64 x 64), TM x TN outputs a thread, K in four cp.async stages of 16, so that
// a block's K range is a few global latencies long.  With splits > 1 a block takes
// one range of K and leaves its sums in `part`; the last block of a tile to finish
// adds them in the order of the ranges (a fixed order, whichever block it is) and
// clears the tile's counter for the next product, so no second launch is needed.
// Bound: latency.  The 32 x 32 form it replaces staged 8 of K through registers
// and summed the splits in a kernel of its own: 96 x 48 x 3000 (C,N) took 25 us,
// 3000 x 48 x 96 (N,N) 19 us.
template <typename R, bool CONJ_A, int TM, int TN>
__global__ void __launch_bounds__(kThreads)
cgemm_pipe(int M, int N, int K, cplx_t<R> alpha, const cplx_t<R>* __restrict__ A, long lda,
           const cplx_t<R>* __restrict__ B, long ldb, cplx_t<R> beta, cplx_t<R>* C, long ldc, int kchunk,
           cplx_t<R>* part, unsigned* counters) {
    chain_begin();
    using T = cplx_t<R>;
    using S = PipeTile<R, TM, TN>;
    extern __shared__ __align__(16) unsigned char zsm[];
    __shared__ int s_last;
    T* As = reinterpret_cast<T*>(zsm);
    T* Bs = As + kStages * S::a_stage;
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    // N tiles run fastest: the blocks that share an A tile run together
    const int m0 = blockIdx.y * S::bm, n0 = blockIdx.x * S::bn;
    const int kbeg = blockIdx.z * kchunk, kend = min(K, kbeg + kchunk);
    const int nk = kend > kbeg ? (kend - kbeg + kBK - 1) / kBK : 0;

    auto fill = [&](int kb, int s) {
        const int k0 = kbeg + kb * kBK;
        T* as = As + s * S::a_stage;
        T* bs = Bs + s * S::b_stage;
#pragma unroll
        for (int r = 0; r < S::bm * kBK / kThreads; ++r) {
            const int idx = tid + r * kThreads;
            const int k = CONJ_A ? idx % kBK : idx / S::bm, m = CONJ_A ? idx / kBK : idx % S::bm;
            const int gk = k0 + k, gm = m0 + m;
            const bool ok = gk < kend && gm < M;
            cp_async(CONJ_A ? as + m * kKP + k : as + k * S::a_pitch_n + m,
                     ok ? (CONJ_A ? A + gk + (long)gm * lda : A + gm + (long)gk * lda) : A, ok);
        }
#pragma unroll
        for (int r = 0; r < S::bn * kBK / kThreads; ++r) {
            const int idx = tid + r * kThreads;
            const int k = idx % kBK, n = idx / kBK;
            const int gk = k0 + k, gn = n0 + n;
            const bool ok = gk < kend && gn < N;
            cp_async(bs + n * kKP + k, ok ? B + gk + (long)gn * ldb : B, ok);
        }
    };

    T acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = czero<T>();
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) {
        if (s < nk) fill(s, s);
        cp_commit();
    }
    for (int kb = 0; kb < nk; ++kb) {
        cp_wait<kStages - 2>();
        __syncthreads();  // stage kb is complete for everyone; stage kb - 1 is free
        const int nxt = kb + kStages - 1;
        if (nxt < nk) fill(nxt, nxt % kStages);
        cp_commit();
        const T* as = As + (kb % kStages) * S::a_stage;
        const T* bs = Bs + (kb % kStages) * S::b_stage;
#pragma unroll
        for (int kk = 0; kk < kBK; ++kk) {
            T a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const T v = CONJ_A ? as[(ty + 16 * i) * kKP + kk] : as[kk * S::a_pitch_n + ty + 16 * i];
                a[i] = CONJ_A ? conj2(v) : v;
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = bs[(tx + 16 * j) * kKP + kk];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) cfma(acc[i][j], a[i], b[j]);
        }
    }
    cp_wait<0>();

    if (gridDim.z > 1) {
        const int tile = blockIdx.y * gridDim.x + blockIdx.x, tiles = gridDim.x * gridDim.y;
        T* mine = part + ((size_t)blockIdx.z * tiles + tile) * (S::bm * S::bn) + tid;
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) __stcg(mine + (i * TN + j) * kThreads, acc[i][j]);
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(counters + tile, 1u) == gridDim.z - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        const T* first = part + (size_t)tile * (S::bm * S::bn) + tid;
        const size_t step = (size_t)tiles * (S::bm * S::bn);
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = czero<T>();
#pragma unroll 4
        for (int z = 0; z < (int)gridDim.z; ++z)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = acc[i][j] + __ldcg(first + z * step + (i * TN + j) * kThreads);
        if (tid == 0) counters[tile] = 0;
    }

    const bool use_beta = (beta.x != R(0) || beta.y != R(0));
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + 16 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + 16 * j;
            if (gn >= N) continue;
            T v = cmul(alpha, acc[i][j]);
            T* c = C + gm + (long)gn * ldc;
            if (use_beta) v = v + cmul(beta, *c);
            *c = v;
        }
    }
}

// ------------------------------------------------------------------ FP64, large tiles
// BM x 64 tiles of C (BM = 16 TM: 128 or 96), TM x 4 complex outputs per
// thread (outputs m = ty + 16 i, n = tx + 16 j), BK = 8 complex of K per stage, three stages filled by 16-byte
// cp.async copies (one complex each; out-of-range elements are zero-filled).
// Each shared-memory read of a stage feeds 128 DFMA per 24 doubles loaded.
// Shared-memory layouts (complex, padded so a warp's reads fall in distinct
// banks): A as [k][m] (pitch 132) when op(A) = A, as [m][k] (pitch 9) when
// op(A) = A^H; B as [n][k] (pitch 9).
namespace big {
constexpr int BM = 128, BN = 64, BK = 16, STAGES = 3, THREADS = 256;
constexpr int KP = BK + 1;         // [m][k] and [n][k]
template <int TM> struct Shape {   // BM = 16 TM rows of C per block
    static constexpr int bm = 16 * TM;
    static constexpr int a_pitch_n = bm + 4;  // [k][m]
    static constexpr int a_stage = (BK * a_pitch_n > bm * KP ? BK * a_pitch_n : bm * KP);  // complex
    static constexpr int b_stage = BN * KP;
    static constexpr size_t smem = (size_t)STAGES * (a_stage + b_stage) * sizeof(double2);
};

}  // namespace big

template <bool CONJ_A, int TM>
__global__ void __launch_bounds__(big::THREADS, 1)
zgemm_big(int M, int N, int K, double2 alpha, const double2* __restrict__ A, long lda,
          const double2* __restrict__ B, long ldb, double2 beta, double2* C, long ldc, int kchunk,
          double2* part) {
    chain_begin();
    using namespace big;
    constexpr int BM = Shape<TM>::bm, A_PITCH_N = Shape<TM>::a_pitch_n, A_STAGE = Shape<TM>::a_stage,
                  B_STAGE = Shape<TM>::b_stage;
    extern __shared__ __align__(16) unsigned char zsm[];
    double2* As = reinterpret_cast<double2*>(zsm);
    double2* Bs = As + STAGES * A_STAGE;
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int kbeg = blockIdx.z * kchunk;
    const int kend = min(K, kbeg + kchunk);
    const int nk = kend > kbeg ? (kend - kbeg + BK - 1) / BK : 0;

    // issue the copies of K block `kb` into stage `s`
    auto fill = [&](int kb, int s) {
        const int k0 = kbeg + kb * BK;
        double2* as = As + s * A_STAGE;
        double2* bs = Bs + s * B_STAGE;
        // A: BM x BK complex, TM / 2 per thread
#pragma unroll
        for (int r = 0; r < (BM * BK) / THREADS; ++r) {
            const int idx = tid + r * THREADS;
            if (CONJ_A) {  // A is K x M: each m holds BK consecutive k
                const int k = idx % BK, m = idx / BK;
                const int gk = k0 + k, gm = m0 + m;
                const bool ok = gk < kend && gm < M;
                cp_async(as + m * KP + k, ok ? A + gk + (long)gm * lda : A, ok);
            } else {       // A is M x K: each k holds BM consecutive m
                const int m = idx % BM, k = idx / BM;
                const int gk = k0 + k, gm = m0 + m;
                const bool ok = gk < kend && gm < M;
                cp_async(as + k * A_PITCH_N + m, ok ? A + gm + (long)gk * lda : A, ok);
            }
        }
        // B: BK x BN complex, 2 per thread; each n holds BK consecutive k
#pragma unroll
        for (int r = 0; r < (BN * BK) / THREADS; ++r) {
            const int idx = tid + r * THREADS;
            const int k = idx % BK, n = idx / BK;
            const int gk = k0 + k, gn = n0 + n;
            const bool ok = gk < kend && gn < N;
            cp_async(bs + n * KP + k, ok ? B + gk + (long)gn * ldb : B, ok);
        }
    };

    double2 acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = make_double2(0.0, 0.0);

#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < nk) fill(s, s);
        cp_commit();
    }
    for (int kb = 0; kb < nk; ++kb) {
        cp_wait<STAGES - 2>();
        __syncthreads();  // stage kb % STAGES is complete for everyone; stage (kb-1) % STAGES is free
        {
            const int nxt = kb + STAGES - 1;
            if (nxt < nk) fill(nxt, nxt % STAGES);
            cp_commit();
        }
        const double2* as = As + (kb % STAGES) * A_STAGE;
        const double2* bs = Bs + (kb % STAGES) * B_STAGE;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            double2 a[TM], b[4];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const double2 v = CONJ_A ? as[(ty + 16 * i) * KP + kk] : as[kk * A_PITCH_N + ty + 16 * i];
                a[i] = CONJ_A ? conj2(v) : v;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = bs[(tx + 16 * j) * KP + kk];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) cfma(acc[i][j], a[i], b[j]);
        }
    }
    cp_wait<0>();

    const bool use_beta = (beta.x != 0.0 || beta.y != 0.0);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + 16 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx + 16 * j;
            if (gn >= N) continue;
            if (part) {
                part[(long)blockIdx.z * M * N + (long)gn * M + gm] = acc[i][j];
            } else {
                double2 v = cmul(alpha, acc[i][j]);
                double2* c = C + gm + (long)gn * ldc;
                if (use_beta) v = v + cmul(beta, *c);
                *c = v;
            }
        }
    }
}

// DFMA rate probe: every thread runs 8 independent FMA chains of `iters` steps
// (2 flops each) on values that stay finite; the result is written so the
// chains are not optimised away.
__global__ void __launch_bounds__(256) dfma_probe(int iters, double seed, double* out) {
    double a[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = seed + 0.001 * (threadIdx.x + c);
    const double b = 0.999999, d = 1e-7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int c = 0; c < 8; ++c) a[c] = fma(a[c], b, d);
    }
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) s += a[c];
    if (s == 12345.678) out[blockIdx.x] = s;  // never true for these inputs; keeps the chains live
}

// C = alpha * sum_z part[z] + beta * C, the splits summed in index order
template <typename R>
__global__ void splitk_reduce(int M, int N, int splits, const cplx_t<R>* __restrict__ part,
                              cplx_t<R> alpha, cplx_t<R> beta, cplx_t<R>* C, long ldc) {
    chain_begin();
    using T = cplx_t<R>;
    const long total = (long)M * N;
    const bool use_beta = (beta.x != R(0) || beta.y != R(0));
    for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total;
         idx += (long)gridDim.x * blockDim.x) {
        const int m = static_cast<int>(idx % M);
        const int n = static_cast<int>(idx / M);
        T s = splits > 0 ? part[idx] : czero<T>();
        for (int z = 1; z < splits; ++z) s = s + part[(long)z * total + idx];
        T v = cmul(alpha, s);
        T* c = C + m + (long)n * ldc;
        if (use_beta) v = v + cmul(beta, *c);
        *c = v;
    }
}

// Clocks a product takes on the busiest SM, for choosing tiles and K ranges: a
// block of a bm x bn tile spends 4 bm bn / 64 clocks of the FP64 units on a step
// of K, at the share of their rate its kernel reaches (0.6 here, 0.72 with the
// large tiles, both measured), and about `start` steps before and after them.
constexpr double kPipeRate = 0.6, kBigRate = 0.72;
constexpr int kPipeStart = 48, kBigStart = 30;
inline double busiest(long blocks, int k, int start, int bm, int bn, double rate) {
    const long sms = device_sms(), waves = (blocks + sms - 1) / sms;
    return (double)waves * (k + start) * (bm * bn / 16.0) / rate;
}

// The tile and the K ranges of a product on the pipelined tiles.
//   tile: 64 x 64 or 32 x 32, whichever takes fewer clocks (64 x 64 where a grid has
//     no room for the tiles of 32 rows); 32 x 16 where 32 columns would leave a
//     quarter or more of them empty;
//   ranges (C,N only): the count with the least clocks, each costing two steps of K
//     for its share of the sum.  At most 64, of at least 32 steps, and as many tiles
//     as there are counters.
constexpr int kMaxGridRows = 65535;
struct PipePlan {
    int tm, tn, splits, kchunk;
    size_t part;   // complex values of the partial sums
    double clocks;
};
PipePlan pipe_plan(bool conj_a, int M, int N, int K) {
    PipePlan best{2, 2, 1, K, 0, -1.0};
    auto consider = [&](int tm, int tn) {
        const int bm = 16 * tm, bn = 16 * tn;
        const long tiles = (long)ceil_div(M, bm) * ceil_div(N, bn);
        for (int s = 1; s == 1 || (conj_a && tiles <= GemmWorkspace::kCounters && s <= 64 && K >= 32 * s); ++s) {
            const double c = busiest(tiles * s, ceil_div(K, s), kPipeStart, bm, bn, kPipeRate) +
                             (s > 1 ? 2.0 * s * (bm * bn / 16.0) : 0.0);
            if (best.clocks >= 0.0 && c >= best.clocks) continue;
            best = PipePlan{tm, tn, 1, K, 0, c};
            if (s > 1) {
                best.kchunk = ceil_div(ceil_div(K, s), kBK) * kBK;
                best.splits = ceil_div(K, best.kchunk);
                best.part = best.splits > 1 ? (size_t)best.splits * tiles * (256 * tm * tn) : 0;
            }
        }
    };
    if (ceil_div(M, 32) <= kMaxGridRows) consider(2, ceil_div(N, 16) * 16 * 4 <= ceil_div(N, 32) * 32 * 3 ? 1 : 2);
    consider(4, 4);
    return best;
}

template <typename R, bool CONJ_A, int TM, int TN>
void pipe_run(cudaStream_t st, dim3 grid, int M, int N, int K, cplx_t<R> alpha, const cplx_t<R>* A, long lda,
              const cplx_t<R>* B, long ldb, cplx_t<R> beta, cplx_t<R>* C, long ldc, int kchunk, cplx_t<R>* part,
              unsigned* counters) {
    constexpr size_t smem = PipeTile<R, TM, TN>::smem;
    static PerDeviceOnce once;
    once.run([] {
        Q3B_CUDA(cudaFuncSetAttribute(cgemm_pipe<R, CONJ_A, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)PipeTile<R, TM, TN>::smem));
    });
    launch_chained(cgemm_pipe<R, CONJ_A, TM, TN>, grid, kThreads, smem, st, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk,
                                                                part, counters);
    Q3B_LAUNCH_CHECK();
}

// K splits of a large-tile C,N product: at most 64, at most one per 256 of K,
// and a workspace of at most 64 MB
constexpr size_t kBigSplitBytes = 64ull << 20;
inline int big_max_splits(int M, int N, int K) {
    const long by_ws = static_cast<long>(kBigSplitBytes / ((size_t)M * N * sizeof(double2)));
    long s = std::min<long>(64, ceil_div(K, 256));
    s = std::min(s, by_ws);
    return s < 1 ? 1 : static_cast<int>(s);
}

// The tile height (128 or 96 rows) and K ranges of zgemm_big: the least rows of
// work per SM over whole waves; a C,N product splits K into as many chunks as fill
// whole waves (at least two, at most 64).
struct BigPlan {
    int tm, splits;
    double clocks;
};
BigPlan big_plan(bool conj_a, int M, int N, int K) {
    BigPlan best{8, 1, -1.0};
    const int most = conj_a ? big_max_splits(M, N, K) : 1;
    for (int tm : {8, 6}) {
        const long tiles = (long)ceil_div(M, 16 * tm) * ceil_div(N, big::BN);
        for (int s = 1; s <= most; ++s) {
            const double c = busiest(tiles * s, ceil_div(K, s), kBigStart, 16 * tm, big::BN, kBigRate);
            if (best.clocks < 0.0 || c < best.clocks) best = BigPlan{tm, s, c};
        }
    }
    // the split sums' own kernel, about 5 us
    if (best.splits > 1) best.clocks += 1e4;
    return best;
}

// FP64 products of at least one 128 x 64 tile take the large tiles where these
// are the faster: 23847 x 256 x 512 (N,N) and 256 x 128 x 12000 (C,N) do;
// 3000 x 96 x 96 (38 us there), 128 x 64 x 6000 (87) and 160 x 80 x 9000 (89) do not
inline bool big_tiles(bool conj_a, int M, int N, int K) {
    return M >= big::BM && N >= big::BN && big_plan(conj_a, M, N, K).clocks < pipe_plan(conj_a, M, N, K).clocks;
}

template <bool CONJ_A, int TM>
void zgemm_big_run(cudaStream_t st, dim3 grid, int M, int N, int K, double2 alpha, const double2* A, long lda,
                   const double2* B, long ldb, double2 beta, double2* C, long ldc, int kchunk, double2* part) {
    constexpr size_t smem = big::Shape<TM>::smem;
    static_assert(smem <= 227 * 1024, "zgemm_big stages exceed shared memory");
    // the attribute belongs to the function on one device
    static PerDeviceOnce once;
    once.run([] {
        Q3B_CUDA(cudaFuncSetAttribute(zgemm_big<CONJ_A, TM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)big::Shape<TM>::smem));
    });
    launch_chained(zgemm_big<CONJ_A, TM>, grid, big::THREADS, smem, st, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk,
                                                             part);
    Q3B_LAUNCH_CHECK();
}

void zgemm_big_launch(cudaStream_t st, bool conj_a, int M, int N, int K, double2 alpha, const double2* A,
                      long lda, const double2* B, long ldb, double2 beta, double2* C, long ldc,
                      const GemmWorkspace& ws) {
    const BigPlan plan = big_plan(conj_a, M, N, K);
    const int tm = plan.tm;
    int splits = plan.splits;
    const size_t need = (size_t)splits * M * N * sizeof(double2);
    if (splits > 1 && (ws.ptr == nullptr || ws.bytes < need)) splits = 1;
    int kchunk = K;
    if (splits > 1) {
        kchunk = ceil_div(K, splits);
        kchunk = ceil_div(kchunk, big::BK) * big::BK;
        splits = ceil_div(K, kchunk);
    }
    const int bm = 16 * tm;
    if (ceil_div(M, bm) > 65535) throw std::runtime_error("complex GEMM: M too large");
    dim3 grid(ceil_div(N, big::BN), ceil_div(M, bm), splits);
    double2* part = splits > 1 ? static_cast<double2*>(ws.ptr) : nullptr;
    if (conj_a) {
        if (tm == 6) zgemm_big_run<true, 6>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, part);
        else zgemm_big_run<true, 8>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, part);
    } else {
        if (tm == 6) zgemm_big_run<false, 6>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, part);
        else zgemm_big_run<false, 8>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, kchunk, part);
    }
    if (splits > 1) {
        const long total = (long)M * N;
        int blocks = ceil_div(total, 256);
        if (blocks > 4096) blocks = 4096;
        launch_chained(splitk_reduce<double>, blocks, 256, 0, st, M, N, splits, part, alpha, beta, C, ldc);
        Q3B_LAUNCH_CHECK();
    }
}


}  // namespace

bool use_tensor_cores(int M, int N, int K) { return (double)M * N * K >= kTensorCoreMinMacs; }

template <typename R> size_t cgemm_workspace_bytes(int M, int N, int K) {
    size_t simt = pipe_plan(true, M, N, K).part * sizeof(cplx_t<R>);
    if constexpr (std::is_same<R, float>::value) return std::max(simt, tc::workspace_bytes(M, N, K));
    const int s = big_max_splits(M, N, K);
    if (big_tiles(true, M, N, K) && s > 1) simt = std::max(simt, (size_t)s * M * N * sizeof(cplx_t<R>));
    return simt;
}

double fp64_units_seconds(bool conj_a, int M, int N, int K) {
    double clocks = pipe_plan(conj_a, M, N, K).clocks;
    if (M >= big::BM && N >= big::BN) clocks = std::min(clocks, big_plan(conj_a, M, N, K).clocks);
    return clocks / 1.93e9 + 4e-6;
}

template <typename R> size_t cgemm_wanted_bytes(bool conj_a, int M, int N, int K) {
    if constexpr (std::is_same<R, double>::value) {
        if (zmod::worth(conj_a, M, N, K, false)) return zmod::workspace_bytes(conj_a, M, N, K, false);
    }
    return 0;
}

template <typename R>
void cgemm(cudaStream_t st, bool conj_a, int M, int N, int K, cplx_t<R> alpha, const cplx_t<R>* A,
           long lda, const cplx_t<R>* B, long ldb, cplx_t<R> beta, cplx_t<R>* C, long ldc,
           const GemmWorkspace& ws) {
    using T = cplx_t<R>;
    if (M <= 0 || N <= 0) return;
    if constexpr (std::is_same<R, float>::value) {
        // small products stay on the CUDA cores: a tensor-core block takes a
        // whole SM's shared memory, which small problems, often several at
        // once on separate streams, cannot keep busy
        if (K > 0 && use_tensor_cores(M, N, K)) {
            tc::cgemm(st, conj_a, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, ws);
            return;
        }
    }
    if (K <= 0) {
        // C = beta * C
        dim3 g(ceil_div((long)M * N, 256));
        launch_chained(splitk_reduce<R>, g, 256, 0, st, M, N, 0, nullptr, alpha, beta, C, ldc);
        Q3B_LAUNCH_CHECK();
        return;
    }
    if constexpr (std::is_same<R, double>::value) {
        if (ws.wanted && zmod::worth(conj_a, M, N, K, false) &&
            ws.bytes >= zmod::workspace_bytes(conj_a, M, N, K, false) && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
            reinterpret_cast<uintptr_t>(B) % 16 == 0) {
            zmod::zgemm(st, conj_a, M, N, K, alpha, A, lda, nullptr, B, ldb, beta, C, ldc, ws);
            return;
        }
        if (big_tiles(conj_a, M, N, K) && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
            reinterpret_cast<uintptr_t>(B) % 16 == 0) {
            zgemm_big_launch(st, conj_a, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, ws);
            return;
        }
    }
    PipePlan p = pipe_plan(conj_a, M, N, K);
    if (p.splits > 1 && (!ws.ptr || !ws.counters || ws.bytes < p.part * sizeof(T))) {
        p.splits = 1;
        p.kchunk = K;
    }
    if (ceil_div(M, 16 * p.tm) > kMaxGridRows) throw std::runtime_error("complex GEMM: M too large");
    const dim3 grid(ceil_div(N, 16 * p.tn), ceil_div(M, 16 * p.tm), p.splits);
    T* part = p.splits > 1 ? static_cast<T*>(ws.ptr) : nullptr;
    auto run = [&](auto conj) {
        constexpr bool CA = decltype(conj)::value;
        if (p.tm == 4)
            pipe_run<R, CA, 4, 4>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, p.kchunk, part, ws.counters);
        else if (p.tn == 2)
            pipe_run<R, CA, 2, 2>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, p.kchunk, part, ws.counters);
        else
            pipe_run<R, CA, 2, 1>(st, grid, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc, p.kchunk, part, ws.counters);
    };
    if (conj_a) run(std::true_type{});
    else run(std::false_type{});
}

namespace {
// an A packed whole for two products takes at most this; a larger one is packed a panel
// at a time for each of them (zgemm_mod.cu)
constexpr size_t kPackedOnceBytes = 4ull << 30;
size_t packed_once_bytes(int M, int K) {
    return zmod::packed_a_bytes(M, K) + ((zmod::packed_a_exps(M) * sizeof(int) + 255) & ~size_t(255));
}
}  // namespace

template <typename R> size_t cgemm_two_wanted_bytes(int M, int N, int K) {
    if constexpr (std::is_same<R, double>::value) {
        if (zmod::worth(true, M, N, K, false) && packed_once_bytes(M, K) <= kPackedOnceBytes)
            return packed_once_bytes(M, K) + zmod::workspace_bytes(true, M, N, K, true);
    }
    return 0;
}

template <typename R>
void cgemm_two(cudaStream_t st, int M, int N, int K, const cplx_t<R>* A, long lda, const cplx_t<R>* B1,
               const cplx_t<R>* B2, long ldb, cplx_t<R>* C1, cplx_t<R>* C2, long ldc, const GemmWorkspace& ws) {
    const cplx_t<R> one = mk(R(1), R(0)), zero = mk(R(0), R(0));
    if constexpr (std::is_same<R, double>::value) {
        const size_t want = cgemm_two_wanted_bytes<R>(M, N, K);
        if (want && ws.wanted && ws.bytes >= want && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
            reinterpret_cast<uintptr_t>(B1) % 16 == 0 && reinterpret_cast<uintptr_t>(B2) % 16 == 0) {
            unsigned char* tiles = static_cast<unsigned char*>(ws.ptr);
            int* exps = reinterpret_cast<int*>(tiles + zmod::packed_a_bytes(M, K));
            zmod::pack_a(st, M, K, A, lda, true, nullptr, tiles, exps);
            const zmod::PackedA pk{tiles, exps, M, K};
            const size_t used = packed_once_bytes(M, K);
            const GemmWorkspace rest{tiles + used, ws.bytes - used, ws.counters, true};
            zmod::zgemm(st, true, M, N, K, one, nullptr, 0, &pk, B1, ldb, zero, C1, ldc, rest);
            zmod::zgemm(st, true, M, N, K, one, nullptr, 0, &pk, B2, ldb, zero, C2, ldc, rest);
            return;
        }
    }
    cgemm<R>(st, true, M, N, K, one, A, lda, B1, ldb, zero, C1, ldc, ws);
    cgemm<R>(st, true, M, N, K, one, A, lda, B2, ldb, zero, C2, ldc, ws);
}

double measure_dfma_tflops(cudaStream_t st) {
    int dev = 0, sms = 0;
    Q3B_CUDA(cudaGetDevice(&dev));
    Q3B_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int blocks = sms * 8, iters = 4096;
    double* out = nullptr;
    Q3B_CUDA(cudaMallocAsync(&out, blocks * sizeof(double), st));
    cudaEvent_t e0, e1;
    Q3B_CUDA(cudaEventCreate(&e0));
    Q3B_CUDA(cudaEventCreate(&e1));
    float best = 1e30f;
    for (int rep = 0; rep < 4; ++rep) {
        Q3B_CUDA(cudaEventRecord(e0, st));
        dfma_probe<<<blocks, 256, 0, st>>>(iters, 1.0, out);
        Q3B_LAUNCH_CHECK();
        Q3B_CUDA(cudaEventRecord(e1, st));
        Q3B_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        Q3B_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (rep > 0 && ms < best) best = ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    Q3B_CUDA(cudaFreeAsync(out, st));
    const double flops = 2.0 * 8.0 * iters * 256.0 * blocks;
    return flops / (best * 1e-3) / 1e12;
}

template void cgemm<double>(cudaStream_t, bool, int, int, int, double2, const double2*, long,
                            const double2*, long, double2, double2*, long, const GemmWorkspace&);
template void cgemm<float>(cudaStream_t, bool, int, int, int, float2, const float2*, long,
                           const float2*, long, float2, float2*, long, const GemmWorkspace&);
template size_t cgemm_workspace_bytes<double>(int, int, int);
template size_t cgemm_workspace_bytes<float>(int, int, int);
template size_t cgemm_two_wanted_bytes<double>(int, int, int);
template void cgemm_two<double>(cudaStream_t, int, int, int, const double2*, long, const double2*, const double2*,
                                long, double2*, double2*, long, const GemmWorkspace&);
template size_t cgemm_wanted_bytes<double>(bool, int, int, int);
template size_t cgemm_wanted_bytes<float>(bool, int, int, int);

}  // namespace q3b
