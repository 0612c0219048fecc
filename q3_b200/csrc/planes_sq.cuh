// Plane pass of the local H|psi> term for square planes of a compile-time size
// (pass B of hpsi_local.cu).
//
// The same seven in-place shared-memory passes as the general plane kernel
// (rows backward, the columns' round trip with V, rows forward; fft_core.cuh
// has the passes), with the line length, its factors, the pitch and the block
// size known to the compiler: element offsets become immediates of the
// shared-memory instructions, a line's DFT is the only one in the code, and the
// twiddles of a pass lie in the order its items read them, [item][k].  The
// general kernel issues 29.1 k warp instructions for an 80 x 80 FP64 plane, of
// which 13 k are FP64 arithmetic and 4 k shared-memory accesses; most of the
// rest, address arithmetic and control, goes away here, and the FP64 kernel fits
// 80 registers, so that an SM holds 24 warps of it instead of 16.  Bound: the
// latency of the passes (shared memory, FP64 or FP32 arithmetic) between barriers.
// Plane pass of 64 bands, general kernel against this, each at its best block:
//   40^3, 48 bands   FP64 45.3 -> 33.1 us    FP32 29.0 -> 21.0 us
//   54^3, 77 bands   FP64 133.5 -> 100.9     FP32 86.1 -> 61.7
//   64^3, 65 bands   FP64 162.2 -> 133.4     FP32 104.6 -> 80.4
//   80^3             FP64 334.6 -> 242.5     FP32 188.7 -> 139.5
//   108^3, 32 bands  FP64 525.5 -> 406.8     FP32 286.9 -> 205.4
#pragma once

#include "fft_core.cuh"
#include "hpsi_local.cuh"

namespace q3b {
namespace psq {

// n = na * nb, na >= nb, na the smallest such factor (Context's factor_line)
constexpr bool is_factor(int a) { return (a >= 1 && a <= 6) || a == 8 || a == 9 || a == 10 || a == 12 || a == 15 || a == 16; }
constexpr int factor_a(int n) {
    for (int a = 1; a <= 16; ++a)
        if (is_factor(a) && n % a == 0 && is_factor(n / a) && a >= n / a) return a;
    return 0;
}

template <typename R, int N> struct Geometry {
    static constexpr int NA = factor_a(N), NB = N / factor_a(N);
    static constexpr int PITCH = N | 1;
    static constexpr int MASK_WORDS = 16;
    static size_t smem(int nrows) {
        return (size_t)(2 * N + N * PITCH) * sizeof(cplx_t<R>) + (size_t)nrows * sizeof(int) +
               MASK_WORDS * sizeof(unsigned);
    }
    // blocks of NT threads an SM holds by shared memory (half the rows holding sticks)
    static constexpr int smem_blocks = 232448 / static_cast<int>((2 * N + N * PITCH) * sizeof(cplx_t<R>) + 4 * N + 1088);
};

// Items of a pass over `lines` lines with Q items each: lines run fastest
// across the threads.
template <int NT, typename F> __device__ __forceinline__ void items(int lines, int Q, const F& f) {
    const int total = lines * Q, bq = NT / lines, br = NT - bq * lines;
    int q = static_cast<int>(threadIdx.x) / lines, l = static_cast<int>(threadIdx.x) - q * lines;
#pragma unroll 1
    for (int it = threadIdx.x; it < total; it += NT) {
        f(l, q);
        l += br;
        q += bq;
        if (l >= lines) {
            l -= lines;
            ++q;
        }
    }
}

// The shared memory of a plane block and its set-up: twiddles in item order, the
// rows that hold sticks, and for each item of the columns' first pass the
// positions in such rows.  Ends with a barrier.
template <typename R, int N> struct PlaneSmem {
    using T = cplx_t<R>;
    T *twa, *twb, *plane;  // w^(q k) at [q < NB][k < NA], at [q < NA][k < NB]
    int* rowb;
    unsigned* colmask;
    template <int NT> __device__ __forceinline__ void init(const LocalPlan<R>& p, unsigned char* smem) {
        using G = Geometry<R, N>;
        twa = reinterpret_cast<T*>(smem);
        twb = twa + N;
        plane = twb + N;
        rowb = reinterpret_cast<int*>(plane + N * G::PITCH);
        colmask = reinterpret_cast<unsigned*>(rowb + p.nrows);
        const int tid = threadIdx.x;
        for (int i = tid; i < N; i += NT) {
            twa[i] = p.tw1[(i / G::NA) * (i % G::NA)];
            twb[i] = p.tw1[(i / G::NB) * (i % G::NB)];
        }
        for (int i = tid; i < p.nrows; i += NT) rowb[i] = p.row_base[i];
        if (tid < G::MASK_WORDS) colmask[tid] = 0u;
        __syncthreads();
        for (int i = tid; i < p.nrows; i += NT) {
            const int w1 = rowb[i] / G::PITCH;
            atomicOr(&colmask[w1 % G::NB], 1u << (w1 / G::NB));
        }
        __syncthreads();
    }
};

// The rows' outer passes take their values from the stick buffer and leave them
// there, element by element through the plan's map from (row, w2) to sticks
// (LocalPlan::row_map), so no row is cleared, filled or emptied by passes of its
// own: six barriers a plane instead of ten (80^3, 64 bands: FP64 267 -> 243 us,
// FP32 152 -> 140; the density of the 64-atom cell 875 -> 824).  Their items run
// along q first, so that neighbouring lanes meet neighbouring sticks.
template <int NT, int NB, typename F> __device__ __forceinline__ void items_along_row(int nrows, const F& f) {
#pragma unroll 1
    for (int it = threadIdx.x; it < nrows * NB; it += NT) f(it / NB, it % NB);
}

// Rows backward from the sticks of one plane, the columns' first pass backward.
// Only the rows that hold sticks are written and read.  Ends with a barrier.
template <typename R, int N, int NT>
__device__ __forceinline__ void plane_in(const LocalPlan<R>& p, const PlaneSmem<R, N>& s, const cplx_t<R>* xp) {
    using T = cplx_t<R>;
    using G = Geometry<R, N>;
    constexpr int NA = G::NA, NB = G::NB, P = G::PITCH;
    const int nrows = p.nrows;
    items_along_row<NT, NB>(nrows, [&](int l, int q) {
        T* b = s.plane + s.rowb[l] + q;
        const T* w = s.twa + q * NA;
        const short* at = p.row_map + l * N + q;
        int from[NA];
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) from[r] = at[NB * r];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = from[r] >= 0 ? xp[from[r]] : czero<T>();
        fft::dft<NA, +1>(x, w, 0);
#pragma unroll
        for (int k = 0; k < NA; ++k) b[NB * k] = k ? cmulc(w[k], x[k]) : x[k];
    });
    __syncthreads();
    items<NT>(nrows, NA, [&](int l, int q) {
        T* b = s.plane + s.rowb[l] + q * NB;
        T x[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = b[r];
        fft::dft<NB, +1>(x, s.twa, 0);
#pragma unroll
        for (int k = 0; k < NB; ++k) b[k] = x[k];
    });
    __syncthreads();
    items<NT>(N, NB, [&](int l, int q) {
        T* b = s.plane + l + q * P;
        const T* w = s.twa + q * NA;
        const unsigned m = s.colmask[q];
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = (m >> r) & 1u ? b[r * NB * P] : czero<T>();
        fft::dft<NA, +1>(x, w, 0);
#pragma unroll
        for (int k = 0; k < NA; ++k) b[k * NB * P] = k ? cmulc(w[k], x[k]) : x[k];
    });
    __syncthreads();
}

template <typename R, int N, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) planes_sq(LocalPlan<R> p, cplx_t<R>* X) {
    chain_begin();
    using T = cplx_t<R>;
    using G = Geometry<R, N>;
    constexpr int NA = G::NA, NB = G::NB, P = G::PITCH;
    extern __shared__ __align__(16) unsigned char smem[];
    PlaneSmem<R, N> s;
    s.template init<NT>(p, smem);
    const int i3 = blockIdx.x, band = blockIdx.y, nrows = p.nrows;
    T* xp = X + ((long)band * p.n3 + i3) * p.xpitch;
    plane_in<R, N, NT>(p, s, xp);
    // columns: the rest of backward, V, forward (only the stick rows are wanted of it)
    const R* vp = p.vplane + (long)i3 * N * N;
    items<NT>(N, NA, [&](int l, int q) {
        T* b = s.plane + l + q * NB * P;
        const T* w = s.twb + q * NB;
        const R* v = vp + q * N + l;
        R pot[NB];
        T x[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) pot[r] = v[r * NA * N];
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = b[r * P];
        fft::dft<NB, +1>(x, w, 0);
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = pot[r] * x[r];
        fft::dft<NB, -1>(x, w, 0);
#pragma unroll
        for (int k = 0; k < NB; ++k) b[k * P] = k ? cmul(x[k], w[k]) : x[k];
    });
    __syncthreads();
    items<NT>(N, NB, [&](int l, int q) {
        T* b = s.plane + l + q * P;
        const unsigned m = s.colmask[q];
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = b[r * NB * P];
        fft::dft<NA, -1>(x, s.twa, 0);
#pragma unroll
        for (int k = 0; k < NA; ++k)
            if ((m >> k) & 1u) b[k * NB * P] = x[k];
    });
    __syncthreads();
    items<NT>(nrows, NA, [&](int l, int q) {
        T* b = s.plane + s.rowb[l] + q * NB;
        const T* w = s.twb + q * NB;
        T x[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = b[r];
        fft::dft<NB, -1>(x, w, 0);
#pragma unroll
        for (int k = 0; k < NB; ++k) b[k] = k ? cmul(x[k], w[k]) : x[k];
    });
    __syncthreads();
    items_along_row<NT, NB>(nrows, [&](int l, int q) {
        const T* b = s.plane + s.rowb[l] + q;
        const short* at = p.row_map + l * N + q;
        int to[NA];
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) to[r] = at[NB * r];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = b[NB * r];
        fft::dft<NA, -1>(x, s.twa, 0);
#pragma unroll
        for (int k = 0; k < NA; ++k)
            if (to[k] >= 0) xp[to[k]] = x[k];
    });
}

// Charge density of one band group on one plane (density_reduce in
// hpsi_local.cu sums the groups): the backward half of the plane pass for each
// band of the group in order, with w |psi|^2 added into the group's slab by the
// items of the columns' last pass, straight from registers.  The slab is
// [w3 pos][w1][w2 pos], w1 in natural order (the last pass knows it); its old
// values are loaded before the item's DFT.  Bands of weight 0 are skipped.
template <int N, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB)
density_sq(LocalPlan<double> p, const double2* X, int nb, const double* __restrict__ wt, double* partial, int groups) {
    chain_begin();
    using G = Geometry<double, N>;
    constexpr int NA = G::NA, NB = G::NB, P = G::PITCH;
    extern __shared__ __align__(16) unsigned char smem[];
    PlaneSmem<double, N> s;
    s.template init<NT>(p, smem);
    const int i3 = blockIdx.x, g = blockIdx.y, per = (nb + groups - 1) / groups;
    const int b0 = g * per, b1 = min(nb, b0 + per);
    double* acc = partial + ((size_t)g * p.n3 + i3) * (N * N);
    for (int b = b0; b < b1; ++b) {
        const double wb = wt[b];
        if (wb == 0.0) continue;
        plane_in<double, N, NT>(p, s, X + ((long)b * p.n3 + i3) * p.xpitch);
        items<NT>(N, NA, [&](int l, int q) {
            const double2* c = s.plane + l + q * NB * P;
            double* a = acc + q * N + l;
            double old[NB];
            double2 x[NB];
#pragma unroll
            for (int r = 0; r < NB; ++r) old[r] = a[r * NA * N];
#pragma unroll
            for (int r = 0; r < NB; ++r) x[r] = c[r * P];
            fft::dft<NB, +1>(x, s.twb, 0);
#pragma unroll
            for (int r = 0; r < NB; ++r) a[r * NA * N] = old[r] + wb * (x[r].x * x[r].x + x[r].y * x[r].y);
        });
        __syncthreads();
    }
}

// ------------------------------------------------------------------ sticks
// Passes A and C (hpsi_local.cu) for a compile-time line length, 32 sticks a
// block, one a lane where the stick buffer is read or written, so that no index
// is divided there.  Bound: the latency of the gathers and of the buffer's L2
// accesses.  Backward, the pass next to the sphere takes its values from psi
// through the plan's map from (stick, w3) to plane waves (LocalPlan::stick_map),
// its items running along q first so that neighbouring lanes meet neighbouring
// entries, instead of clearing and filling the lines beforehand (the density of
// the 64-atom cell 824 -> 816 us, FP32 backward 95 -> 90).  Forward, the values go
// through the lines: handing them to H psi from that pass's registers took
// 164 us instead of 98 (FP32, 256 bands of 80^3).  The general kernels took 130
// and 176 us there.
constexpr int kGroup = 32;      // sticks a block
constexpr int kStickNT = 256;
constexpr int kGathers = 4;     // global gathers a thread keeps in flight

template <typename R, int N> struct StickSmem {
    static constexpr int P = N | 1;
    static constexpr size_t bytes = (size_t)(N + kGroup * P) * sizeof(cplx_t<R>);
};
template <typename R, int N> constexpr int stick_blocks() {
    constexpr int regs = Geometry<R, N>::NA <= 10 ? (sizeof(R) == 8 ? 80 : 48) : (sizeof(R) == 8 ? 112 : 64);
    constexpr int by_regs = 65536 / (kStickNT * regs);
    constexpr int by_smem = static_cast<int>(232448 / (StickSmem<R, N>::bytes + 1024));
    return by_regs < by_smem ? by_regs : by_smem;
}

template <typename R, int N>
__global__ void __launch_bounds__(kStickNT, (stick_blocks<R, N>()))
sticks_back(LocalPlan<R> p, const cplx_t<R>* __restrict__ psi, long ldpsi, cplx_t<R>* X) {
    chain_begin();
    using T = cplx_t<R>;
    constexpr int NA = Geometry<R, N>::NA, NB = Geometry<R, N>::NB, P = StickSmem<R, N>::P, W = kStickNT / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    T* twa = reinterpret_cast<T*>(smem);  // w^(q k) at [q < NB][k < NA]
    T* lines = twa + N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int band = blockIdx.y, s0 = blockIdx.x * kGroup, ns = min(kGroup, p.nsticks - s0);
    for (int i = tid; i < N; i += kStickNT) twa[i] = p.tw3[(i / NA) * (i % NA)];
    __syncthreads();
    const T* ps = psi + (long)band * ldpsi;
#pragma unroll 1
    for (int it = tid; it < ns * NB; it += kStickNT) {
        const int l = it / NB, q = it % NB;
        const int* at = p.stick_map + (long)(s0 + l) * N + q;
        const T* w = twa + q * NA;
        int from[NA];
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) from[r] = at[NB * r];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = from[r] >= 0 ? ps[from[r]] : czero<T>();
        fft::dft<NA, +1>(x, w, 0);
        T* b = lines + l * P + q;
#pragma unroll
        for (int k = 0; k < NA; ++k) b[NB * k] = k ? cmulc(w[k], x[k]) : x[k];
    }
    __syncthreads();
    if (lane >= ns) return;
    // the second pass leaves its values at positions NB q + k
    const T* line = lines + lane * P;
    T* xb = X + (long)band * p.n3 * p.xpitch + s0 + lane;
#pragma unroll 1
    for (int q = warp; q < NA; q += W) {
        T x[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = line[NB * q + r];
        fft::dft<NB, +1>(x, twa, 0);
#pragma unroll
        for (int k = 0; k < NB; ++k) xb[(long)(NB * q + k) * p.xpitch] = x[k];
    }
}

template <typename R, int N>
__global__ void __launch_bounds__(kStickNT, (stick_blocks<R, N>()))
sticks_fwd(LocalPlan<R> p, const cplx_t<R>* __restrict__ X, const cplx_t<R>* __restrict__ psi, long ldpsi,
           cplx_t<R>* hpsi, long ldh) {
    chain_begin();
    using T = cplx_t<R>;
    constexpr int NA = Geometry<R, N>::NA, NB = Geometry<R, N>::NB, P = StickSmem<R, N>::P, W = kStickNT / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    T* twb = reinterpret_cast<T*>(smem);  // w^(q k) at [q < NA][k < NB]
    T* lines = twb + N;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int band = blockIdx.y, s0 = blockIdx.x * kGroup, ns = min(kGroup, p.nsticks - s0);
    for (int i = tid; i < N; i += kStickNT) twb[i] = p.tw3[(i / NB) * (i % NB)];
    __syncthreads();
    T* line = lines + lane * P;
    // the first pass takes positions NB q + r: straight from X
    const T* xb = X + (long)band * p.n3 * p.xpitch + s0 + lane;
#pragma unroll 1
    for (int q = warp; q < NA; q += W) {
        const T* w = twb + q * NB;
        T x[NB];
#pragma unroll
        for (int r = 0; r < NB; ++r) x[r] = lane < ns ? xb[(long)(NB * q + r) * p.xpitch] : czero<T>();
        fft::dft<NB, -1>(x, w, 0);
#pragma unroll
        for (int k = 0; k < NB; ++k) line[NB * q + k] = k ? cmul(x[k], w[k]) : x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int q = warp; q < NB; q += W) {
        T x[NA];
#pragma unroll
        for (int r = 0; r < NA; ++r) x[r] = line[q + NB * r];
        fft::dft<NA, -1>(x, twb, 0);
#pragma unroll
        for (int k = 0; k < NA; ++k) line[q + NB * k] = x[k];
    }
    __syncthreads();
    const T* ps = psi + (long)band * ldpsi;
    T* hs = hpsi + (long)band * ldh;
    const int e1 = p.stick_start[s0 + ns];
    for (int eb = p.stick_start[s0] + tid; eb < e1; eb += kGathers * kStickNT) {
        int gi[kGathers];
        R ke[kGathers];
        T x[kGathers], v[kGathers];
#pragma unroll
        for (int u = 0; u < kGathers; ++u) {
            const int e = eb + u * kStickNT;
            gi[u] = -1;
            if (e < e1) {
                gi[u] = p.entry_g[e];
                v[u] = lines[p.entry_at[e]];
            }
        }
#pragma unroll
        for (int u = 0; u < kGathers; ++u) {
            if (gi[u] >= 0) {
                ke[u] = p.ke[gi[u]];
                x[u] = ps[gi[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kGathers; ++u)
            if (gi[u] >= 0) hs[gi[u]] = ke[u] * x[u] + v[u];
    }
}

// registers a thread may use: what keeps the line of a pass (R complex values)
// and its DFT without spilling to memory
template <typename R, int N> constexpr int register_need() {
    return Geometry<R, N>::NA <= 10 ? (sizeof(R) == 8 ? 80 : 56) : (sizeof(R) == 8 ? 112 : 64);
}
template <typename R, int N, int NT> constexpr int min_blocks() {
    constexpr int by_regs = 65536 / (NT * register_need<R, N>());
    constexpr int by_threads = 2048 / NT;
    constexpr int b = by_regs < by_threads ? by_regs : by_threads;
    constexpr int c = b < Geometry<R, N>::smem_blocks ? b : Geometry<R, N>::smem_blocks;
    return c < 1 ? 1 : c;
}

template <typename R, int N, int NT> void launch(const LocalPlan<R>& p, cplx_t<R>* X, int nb, cudaStream_t st) {
    constexpr int MINB = min_blocks<R, N, NT>();
    static PerDeviceOnce once;
    once.run([] {
        auto* k = planes_sq<R, N, NT, MINB>;
        Q3B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        Q3B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    });
    launch_chained(planes_sq<R, N, NT, MINB>, dim3(p.n3, nb), NT, Geometry<R, N>::smem(p.nrows), st, p, X);
}

template <typename R, int N>
void launch_back(const LocalPlan<R>& p, const cplx_t<R>* psi, long ldpsi, cplx_t<R>* X, int nb, cudaStream_t st) {
    constexpr size_t smem = StickSmem<R, N>::bytes;
    static PerDeviceOnce once;
    once.run([] {
        Q3B_CUDA(cudaFuncSetAttribute(sticks_back<R, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    });
    launch_chained(sticks_back<R, N>, dim3(ceil_div(p.nsticks, kGroup), nb), kStickNT, smem, st, p, psi, ldpsi, X);
}
template <typename R, int N>
void launch_fwd(const LocalPlan<R>& p, const cplx_t<R>* X, const cplx_t<R>* psi, long ldpsi, cplx_t<R>* hpsi,
                long ldh, int nb, cudaStream_t st) {
    constexpr size_t smem = StickSmem<R, N>::bytes;
    static PerDeviceOnce once;
    once.run([] {
        Q3B_CUDA(cudaFuncSetAttribute(sticks_fwd<R, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    });
    launch_chained(sticks_fwd<R, N>, dim3(ceil_div(p.nsticks, kGroup), nb), kStickNT, smem, st, p, X, psi, ldpsi, hpsi, ldh);
}

// ------------------------------------------------------------------ dispatch
// The lengths with kernels of their own: every product of two supported factors
// (context.cu's factor_line) from 16 to 108, the longest whose FP64 plane fits an
// SM's shared memory, that a plane-wave cell's grid takes (2/3/5-smooth).  Each
// source file that includes this instantiates one half of them in one precision.
#define Q3B_SQ_SMALL(X) X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48)
#define Q3B_SQ_LARGE(X) X(50) X(54) X(60) X(64) X(72) X(75) X(80) X(81) X(90) X(96) X(100) X(108)

// threads of the small, middle and large block (LocalPlan::plane_threads 128, 256,
// 512): the large FP64 one is the most of which two fit an SM without spilling
// (80^3, 64 bands: 256 threads 290 us, 320 280, 384 267, 448 and 512 above 359)
template <typename R, int N> bool planes_of(const LocalPlan<R>& p, cplx_t<R>* X, int nb, cudaStream_t st) {
    constexpr int large = sizeof(R) == 8 && N < 96 ? 384 : 512;
    if (p.plane_threads >= 512) launch<R, N, large>(p, X, nb, st);
    else if (p.plane_threads >= 256) launch<R, N, 256>(p, X, nb, st);
    else launch<R, N, 128>(p, X, nb, st);
    return true;
}

// the density's block: as the large plane block, the most threads that fit
template <int N> struct DensityBlock {
    static constexpr int NT = N < 32 ? 128 : N < 96 ? 384 : 512;
    static constexpr int MINB = min_blocks<double, N, NT>();
};
template <int N> void density_limits() {
    static PerDeviceOnce once;
    once.run([] {
        auto* k = density_sq<N, DensityBlock<N>::NT, DensityBlock<N>::MINB>;
        Q3B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        Q3B_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    });
}
// nb > 0: launch; nb == 0: the blocks an SM holds, in *per_sm
template <int N>
void density_of(const LocalPlan<double>& p, const double2* X, int nb, const double* w, double* partial, int groups,
                cudaStream_t st, int* per_sm) {
    using B = DensityBlock<N>;
    density_limits<N>();
    const size_t smem = Geometry<double, N>::smem(p.nrows);
    if (nb > 0)
        launch_chained(density_sq<N, B::NT, B::MINB>, dim3(p.n3, groups), B::NT, smem, st, p, X, nb, w, partial, groups);
    else
        Q3B_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, density_sq<N, B::NT, B::MINB>, B::NT, smem));
}

}  // namespace psq
}  // namespace q3b

// FP64 only: the density kernels
#define Q3B_SQ_DENSITY_INSTANTIATE(NAME, SIZES)                                                                \
    namespace q3b {                                                                                            \
    namespace psq {                                                                                            \
    bool NAME##_density(const LocalPlan<double>& p, const double2* X, int nb, const double* w, double* partial, \
                        int groups, cudaStream_t st, int* per_sm) {                                            \
        if (p.n1 != p.n2) return false;                                                                        \
        switch (p.n1) {                                                                                        \
            SIZES(Q3B_SQ_DENSITY)                                                                              \
            default: return false;                                                                             \
        }                                                                                                      \
        return true;                                                                                           \
    }                                                                                                          \
    }                                                                                                          \
    }
#define Q3B_SQ_DENSITY(N) case N: density_of<N>(p, X, nb, w, partial, groups, st, per_sm); break;

#define Q3B_SQ_INSTANTIATE(NAME, R, SIZES)                                                                     \
    namespace q3b {                                                                                            \
    namespace psq {                                                                                            \
    bool NAME##_planes(const LocalPlan<R>& p, cplx_t<R>* X, int nb, cudaStream_t st) {                         \
        if (p.n1 != p.n2) return false;                                                                        \
        switch (p.n1) {                                                                                        \
            SIZES(Q3B_SQ_PLANE_##R)                                                                            \
            default: return false;                                                                             \
        }                                                                                                      \
    }                                                                                                          \
    bool NAME##_back(const LocalPlan<R>& p, const cplx_t<R>* psi, long ldpsi, cplx_t<R>* X, int nb,            \
                     cudaStream_t st) {                                                                        \
        if (!p.stick_map) return false;                                                                        \
        switch (p.n3) {                                                                                        \
            SIZES(Q3B_SQ_BACK_##R)                                                                             \
            default: return false;                                                                             \
        }                                                                                                      \
        return true;                                                                                           \
    }                                                                                                          \
    bool NAME##_fwd(const LocalPlan<R>& p, const cplx_t<R>* X, const cplx_t<R>* psi, long ldpsi,               \
                    cplx_t<R>* hpsi, long ldh, int nb, cudaStream_t st) {                                      \
        switch (p.n3) {                                                                                        \
            SIZES(Q3B_SQ_FWD_##R)                                                                              \
            default: return false;                                                                             \
        }                                                                                                      \
        return true;                                                                                           \
    }                                                                                                          \
    }                                                                                                          \
    }
#define Q3B_SQ_PLANE_double(N) case N: return planes_of<double, N>(p, X, nb, st);
#define Q3B_SQ_PLANE_float(N) case N: return planes_of<float, N>(p, X, nb, st);
#define Q3B_SQ_BACK_double(N) case N: launch_back<double, N>(p, psi, ldpsi, X, nb, st); break;
#define Q3B_SQ_BACK_float(N) case N: launch_back<float, N>(p, psi, ldpsi, X, nb, st); break;
#define Q3B_SQ_FWD_double(N) case N: launch_fwd<double, N>(p, X, psi, ldpsi, hpsi, ldh, nb, st); break;
#define Q3B_SQ_FWD_float(N) case N: launch_fwd<float, N>(p, X, psi, ldpsi, hpsi, ldh, nb, st); break;
