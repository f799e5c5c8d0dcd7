// The exact batched 4 x 4 product (the reference's benchmarks/experiments/exact_gemm4: README.md "Contract and
// dispatch", prototype.hpp:5-24): fixed row-major 4 x 4 matrices, matrix t of A, B and C at t * stride elements
// (stride 0 broadcasts an input).  Each real output component is RN(C_old + sum_k a_ik b_kj) with one rounding of the
// exact sum (C_old left out without accumulation), negated when asked; a complex component sums its eight signed real
// products.  Statuses: zero with the OR of every operand the component reads and C_old; no nonzero product gives C_old
// (or zero).  One thread per output component; the exact sum is a register window when the terms' spread fits it, else
// cluster_round over the component's terms (a window per cluster, streamed when a cluster is wider), so every spread
// is summed on the GPU.
#pragma once
#include "lf_linalg.cuh"
#include "lf_carveout.h"

namespace lfd {

struct Eg4Params {
    const u32* A; const u32* B; u32* C; u64 count, sa, sb, sc; int accumulate, negative;
    int wide;                             // every matrix starts on a 16-byte boundary
};

// Factors and sign of a component's term k (real: k < 4; complex: k < 8).
template <int N, bool CX> __device__ __forceinline__ void eg4_term(const u32* a, const u32* b, int k, int part, const u32*& x,
                                                                 const u32*& y, int& sg) {
    constexpr u64 E = N + 3, S = CX ? 2 * E : E;
    if (!CX) { x = a + (u64)k * S; y = b + (u64)k * 4 * S; sg = 1; return; }
    const int kk = k >> 1, h = k & 1;
    const u32* ak = a + (u64)kk * S;
    const u32* bk = b + (u64)kk * 4 * S;
    if (part == 0) { x = ak + h * E; y = bk + h * E; sg = h ? -1 : 1; }             // re: a.re b.re - a.im b.im
    else { x = ak + h * E; y = bk + (1 - h) * E; sg = 1; }                        // im: a.re b.im + a.im b.re
}
// Terms of one component for cluster_round: the signed products, and the old value as the last term.  add's word counts are
// constants, so a product stays in registers (added with a run-time count it went to thread-local memory and was read back
// word by word: 5567 complex 1024-bit matrices took 3.7 ms, this way 1.1).
template <int N, bool CX> struct Eg4Terms {
    static constexpr int CNT = CX ? 8 : 4;
    const u32* a; const u32* b; int part; Num<N> c;
    __device__ u64 count() const { return CNT + 1; }
    __device__ bool term(u64 k, i64& scale, i64& top, int& sign) const {
        if ((int)k == CNT) {
            if (!c.s) return false;
            scale = (i64)c.e - (32 * N - 1); top = scale + 32 * N; sign = c.s;
            return true;
        }
        const u32 *x, *y; int sg;
        eg4_term<N, CX>(a, b, (int)k, part, x, y, sg);
        const int sa = (int)x[N + 1], sb = (int)y[N + 1];
        if (!sa || !sb) return false;
        scale = (i64)(int)x[N] + (int)y[N] - 2 * (32 * N - 1);
        top = scale + 64 * N;
        sign = sg * sa * sb;
        return true;
    }
    __device__ void add(u64 k, u32* acc, int len, i64 off) const {
        if ((int)k == CNT) { acc_add(acc, len, c.m, off); return; }
        const u32 *x, *y; int sg;
        eg4_term<N, CX>(a, b, (int)k, part, x, y, sg);
        const Num<N> xa = load_plain<N>(x);
        u32 prod[2 * N];
        mant_mul<N>(xa.m, y, prod);
        acc_add(acc, len, prod, off);
    }
};

// Register window for components whose terms span at most 32 W - 5 bits (the usual case): every product is added
// exactly into a two's-complement window of W = 2N + 8 words held in registers and rounded once; the term pointers
// follow from the term index, so nothing is indexed at run time.  Wider spreads (and widths above 512 bits, where
// the window would not fit in registers) take cluster_round.  Returns false to ask for the cluster path.
template <int N> constexpr int eg4_window() { return N <= 16 ? 2 * N + 8 : 0; }
template <int N, bool CX> __device__ bool eg4_window_sum(const u32* a, const u32* b, int part, const Num<N>& c, Num<N>& out) {
    constexpr int W = eg4_window<N>();
    if constexpr (W == 0) {
        return false;
    } else {
        constexpr int CNT = CX ? 8 : 4;
        i64 lo = INT64_MAX, hi = INT64_MIN;
#pragma unroll 1
        for (int k = 0; k < CNT; ++k) {
            const u32 *x, *y; int sg;
            eg4_term<N, CX>(a, b, k, part, x, y, sg);
            if (!x[N + 1] || !y[N + 1]) continue;
            const i64 sc = (i64)(int)x[N] + (int)y[N] - 2 * (32 * N - 1);
            lo = sc < lo ? sc : lo; hi = sc + 64 * N > hi ? sc + 64 * N : hi;
        }
        const i64 cs = (i64)c.e - (32 * N - 1);
        if (c.s) { lo = cs < lo ? cs : lo; hi = cs + 32 * N > hi ? cs + 32 * N : hi; }
        if (hi - lo + 5 > 32 * (i64)W) return false;
        u32 acc[W], t[W];
#pragma unroll
        for (int w = 0; w < W; ++w) acc[w] = 0;
#pragma unroll 1
        for (int k = 0; k < CNT; ++k) {
            const u32 *x, *y; int sg;
            eg4_term<N, CX>(a, b, k, part, x, y, sg);
            const int sa = (int)x[N + 1], sb = (int)y[N + 1];
            if (!sa || !sb) continue;
            const Num<N> xa = load_plain<N>(x);
            u32 pr[2 * N];
            mant_mul<N>(xa.m, y, pr);                              // y's words come from shared memory as their rows need them
            place_words<W, 2 * N>(t, pr, (i64)xa.e + (int)y[N] - 2 * (32 * N - 1) - lo);
            accumulate<W>(acc, t, sg * sa * sb < 0);
        }
        if (c.s) {
            place_words<W, N>(t, c.m, cs - lo);
            accumulate<W>(acc, t, c.s < 0);
        }
        const bool neg = acc[W - 1] >> 31;
        negate_words<W>(acc, neg);                                  // the magnitude
        out = round_general<N, W>(acc, lo, neg ? -1 : 1, 0);
        return true;
    }
}

// Where eg4_staged() says so, the A and B matrices of a block (four complex or eight real ones, a thread per output component) pass
// through shared memory: every entry is read by eight threads, and from global memory a warp's load of one word touched a cache line
// an entry.  The results replace A's matrices in the tile and leave as whole matrices (the padding between output matrices is kept).
// The tiles take L1 from the thread-local windows of cluster_round, so components that need it lose what the others gain:
//   - above 16 limbs every component sums by clusters: unstaged (20,000 complex matrices of 32 limbs: 5.25 ms staged, 2.66 not);
//   - real matrices up to 7 limbs have few lines an entry, and staging gains nothing (7 limbs: 39 us either way; exponents of +-1000,
//     by clusters: 1.96 ms staged, 1.52 not);
//   - the others stage and leave the rest of the array to L1 (eg4_carveout).
constexpr int kEg4Threads = 128;
template <bool CX> constexpr int eg4_matrices() { return kEg4Threads / (CX ? 32 : 16); }
template <int N, bool CX> constexpr int eg4_matrix_words() { return 16 * (CX ? 2 : 1) * (N + 3); }
template <int N, bool CX> constexpr size_t eg4_smem_bytes() { return (size_t)4 * 2 * eg4_matrices<CX>() * eg4_matrix_words<N, CX>(); }
// Matrices t0 .. t0 + nm - 1 of one operand, `stride` words apart.
template <int MW> __device__ __forceinline__ void eg4_fetch(u32* tile, const u32* src, u64 t0, int nm, u64 stride, bool wide) {
    if (wide) {
        for (int x = threadIdx.x; x < nm * (MW / 4); x += kEg4Threads) {
            const int m = x / (MW / 4), w = 4 * (x - m * (MW / 4));
            cp_async16(tile + m * MW + w, src + (t0 + m) * stride + w);
        }
    } else {
        for (int x = threadIdx.x; x < nm * MW; x += kEg4Threads) {
            const int m = x / MW, w = x - m * MW;
            cp_async4(tile + x, src + (t0 + m) * stride + w);
        }
    }
}
template <int N, bool CX> constexpr bool eg4_staged() { return N <= 16 && (CX || N > 7); }
// Shared memory to set aside, in percent of 228 KB: the hardware's step of 32, 64 or 100 KB that holds four blocks (N + 4 KB each, the system's
// included).  Left to the driver, shared memory got what it could and cluster sums slowed: 20,000 complex matrices of 14 limbs with
// exponents of +-200 took 6.6 ms, so 1.11; +-30: 0.23 either way.  Real matrices of 13 limbs do with three blocks (72 us,
// four 68; +-1000: 2.9 ms at 64 KB, 4.0 at 100).
template <int N, bool CX> constexpr int eg4_carveout() { return N <= 4 ? 14 : N <= (CX ? 12 : 13) ? 28 : 43; }
// One component: RN(c + sum) from its row of A and column of B (a, b: in memory or in the tiles) and its old value c.
template <int N, bool CX> __device__ __forceinline__ Num<N> eg4_component(const u32* a, const u32* b, int part, const Num<N>& c, bool negative) {
    constexpr int CNT = CX ? 8 : 4;
    u32 st = c.st;
    bool products = false;
#pragma unroll 1
    for (int k = 0; k < CNT; ++k) {
        const u32 *x, *y; int sg;
        eg4_term<N, CX>(a, b, k, part, x, y, sg);
        st |= x[N + 2] | y[N + 2];
        products = products || (x[N + 1] && y[N + 1]);
    }
    Num<N> r;
    if (st) r = zero<N>(st);
    else if (!products) r = c;
    else if (!eg4_window_sum<N, CX>(a, b, part, c, r)) {
        const Eg4Terms<N, CX> src{a, b, part, c};
        r = cluster_round<N, 8 * N + 8>(src, nullptr);
    }
    if (negative) r = negate<N>(r);
    return r;
}
template <int N, bool CX> __global__ void __launch_bounds__(kEg4Threads) exact_gemm4_kernel(Eg4Params p) {
    constexpr u64 E = N + 3, S = CX ? 2 * E : E, P = CX ? 2 : 1;
    constexpr int NM = eg4_matrices<CX>(), MW = eg4_matrix_words<N, CX>();
    const u64 t0 = (u64)blockIdx.x * NM;
    const int nm = p.count - t0 < (u64)NM ? (int)(p.count - t0) : NM;
    const int t = threadIdx.x / (int)(16 * P), rest = threadIdx.x % (int)(16 * P), oi = rest / (int)P, part = rest % (int)P;
    if constexpr (!eg4_staged<N, CX>()) {
        if (t >= nm) return;
        u32* out = p.C + ((t0 + t) * p.sc + oi) * S + part * E;
        const Num<N> c = p.accumulate ? load_plain<N>(out) : zero<N>();
        store<N>(out, eg4_component<N, CX>(p.A + ((t0 + t) * p.sa + oi / 4 * 4) * S, p.B + ((t0 + t) * p.sb + oi % 4) * S, part, c, p.negative));
    } else {
        extern __shared__ __align__(16) u32 eg4_tiles[];
        u32* const tA = eg4_tiles;
        u32* const tB = tA + NM * MW;
        eg4_fetch<MW>(tA, p.A, t0, nm, p.sa * S, p.wide);
        eg4_fetch<MW>(tB, p.B, t0, nm, p.sb * S, p.wide);
        cp_async_commit();
        Num<N> r = zero<N>();
        if (p.accumulate && t < nm) r = load_plain<N>(p.C + ((t0 + t) * p.sc + oi) * S + part * E);
        cp_async_wait<0>();
        __syncthreads();
        if (t < nm) r = eg4_component<N, CX>(tA + t * MW + (oi / 4) * 4 * S, tB + t * MW + (oi % 4) * S, part, r, p.negative);
        __syncthreads();                                            // every component has read A
        if (t < nm) store<N>(tA + t * MW + oi * S + part * E, r);
        __syncthreads();
        if (p.wide) {
            for (int x = threadIdx.x; x < nm * (MW / 4); x += kEg4Threads) {
                const int m = x / (MW / 4), w = 4 * (x - m * (MW / 4));
                *reinterpret_cast<uint4*>(p.C + (t0 + m) * p.sc * S + w) = *reinterpret_cast<const uint4*>(tA + m * MW + w);
            }
        } else {
            for (int x = threadIdx.x; x < nm * MW; x += kEg4Threads) {
                const int m = x / MW, w = x - m * MW;
                p.C[(t0 + m) * p.sc * S + w] = tA[x];
            }
        }
    }
}

struct Eg4Kernels { void (*run)(const Eg4Params&, bool complex_, cudaStream_t); };
const Eg4Kernels* eg4_kernels(int limbs);

template <int N, bool CX> void eg4_launch_v(const Eg4Params& pin, cudaStream_t s) {
    constexpr size_t smem = eg4_staged<N, CX>() ? eg4_smem_bytes<N, CX>() : 0;
    constexpr u64 S = (CX ? 2 : 1) * (N + 3);
    Eg4Params p = pin;
    // a lone matrix has no stride (its argument may be anything); the others start stride * S words apart
    const u64 strides = p.count > 1 ? (p.sa | p.sb | p.sc) * S : 0;
    p.wide = !(((uintptr_t)p.A | (uintptr_t)p.B | (uintptr_t)p.C | 4 * strides) & 15);
    static_assert(smem <= 48 * 1024, "tiles need no larger limit");
    if constexpr (smem > 0) {
        static std::atomic<uint64_t> asked{0};
        prefer_carveout(exact_gemm4_kernel<N, CX>, eg4_carveout<N, CX>(), asked);
    }
    const unsigned blocks = (unsigned)((p.count + eg4_matrices<CX>() - 1) / eg4_matrices<CX>());
    exact_gemm4_kernel<N, CX><<<blocks, kEg4Threads, smem, s>>>(p);
}
template <int N> void eg4_launch(const Eg4Params& p, bool cx, cudaStream_t s) {
    if (!p.count) return;
    if (cx) eg4_launch_v<N, true>(p, s); else eg4_launch_v<N, false>(p, s);
}

}  // namespace lfd

#define LF_EG4_INSTANTIATE(N)                                                         \
    namespace lfd {                                                                   \
    extern const Eg4Kernels eg4_kernels_##N;                                          \
    const Eg4Kernels eg4_kernels_##N = {eg4_launch<N>};                               \
    }
