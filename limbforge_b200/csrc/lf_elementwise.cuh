// Element-wise kernels: one value per thread (one component of a complex value), the reference's element layout (AoS) in HBM.
// Broadcast operands are read at (i / stride) % period (kernels.metal:7).  Op codes follow
// limbforge::Operation (engine.hpp:13).  The mul-chain kernel keeps the running value in
// registers across every step (the fused form of a resident CommandBatch chain).
#pragma once
#include "lf_arith.cuh"
#include "lf_carveout.h"
#include <cuda_runtime.h>
#include <cstdint>

namespace lfd {

struct EwParams {
    const u32* a; const u32* b; const u32* c; u32* out;
    u64 count, bs, bp, cs, cp;
    int aligned;                          // every operand and the output start on 16-byte boundaries
};
struct ChainStep { const u32* b; u32* out; u64 bs, bp; int op; int pad; };
constexpr int kMaxChain = 32;
struct ChainParams {
    const u32* a; u64 count; int steps; int lanes;      // lanes: 2 runs stageable multiplication chains on lane pairs
    ChainStep step[kMaxChain];
};

__device__ __forceinline__ u64 bidx(u64 i, u64 s, u64 p) { u64 j = s > 1 ? i / s : i; return p ? j % p : j; }

constexpr int kEwThreads = 128;

// A block's rows (elements, or components of complex values) pass through shared memory: a thread's own N + 3 words lie
// (N + 3) words from its neighbour's, so a load of one word by a warp touches some N + 3 cache lines, and the element-wise
// kernels were bound by those (300,000 512-bit sums: 35 us, 1.9 TB/s).  Tiles are copied with cp.async, in
// 16-byte pieces where the block is whole and the arrays are aligned, word by word otherwise (a last block, an even row
// length: those rows are padded to an odd stride, free of bank conflicts).  A thread copies its own row of a broadcast operand, whose few
// elements L1 holds, and forms its index once (formed for every word, the index's two divisions cost 500,000 96-bit products
// 6 us of 41).
template <int N> constexpr int ew_stride() { return (N + 3) | 1; }
template <int N> __device__ __forceinline__ void ew_fetch(u32* tile, const u32* src, u64 row0, int rows, u64 bs, u64 bp, int parts, bool wide) {
    constexpr int E = N + 3, S = ew_stride<N>();
    if (bs == 1 && !bp) {
        src += row0 * E;
        if (S == E && wide) {
            for (int c = threadIdx.x; c < kEwThreads * E / 4; c += kEwThreads) cp_async16(tile + 4 * c, src + 4 * c);
        } else {
            for (int w = threadIdx.x; w < rows * E; w += kEwThreads) cp_async4(tile + w + (w / E) * (S - E), src + w);
        }
    } else if ((int)threadIdx.x < rows) {
        const u64 row = row0 + threadIdx.x, j = parts == 2 ? 2 * bidx(row >> 1, bs, bp) + (row & 1) : bidx(row, bs, bp);
        u32* const mine = tile + threadIdx.x * S;
#pragma unroll
        for (int w = 0; w < E; ++w) mine[w] = __ldg(src + j * E + w);
    }
}
template <int N> __device__ __forceinline__ void ew_put(const u32* tile, u32* dst, u64 row0, int rows, bool wide) {
    constexpr int E = N + 3, S = ew_stride<N>();
    dst += row0 * E;
    if (S == E && wide) {
        for (int c = threadIdx.x; c < kEwThreads * E / 4; c += kEwThreads)
            reinterpret_cast<uint4*>(dst)[c] = reinterpret_cast<const uint4*>(tile)[c];
    } else {
        for (int w = threadIdx.x; w < rows * E; w += kEwThreads) dst[w] = tile[w + (w / E) * (S - E)];
    }
}
constexpr bool ew_complex(int op) { return op == 4 || op == 5 || op == 6 || op == 11 || op == 12; }
constexpr int ew_inputs(int op) { return op == 7 || op == 8 ? 1 : op >= 9 ? 3 : 2; }
// Fused complex operations whose exponents lie far apart sum by clusters in thread-local windows, which need L1: shared memory that the driver sets
// aside for more blocks costs them more than it brings.  Up to 12 limbs the kernels therefore read the addend straight from memory (two
// tiles) and run in the 64 KB step of shared memory (28% of 228 KB), four blocks of 12 limbs.  200,000 values, us, a thread a value / three tiles by
// default / this: 8 limbs, near exponents 91 / 52 / 51, +-300 238 / 254 / 223, +-3000 292 / 335 / 284; 12 limbs 173 / 79 / 75, 448 / 343 / 321,
// 661 / 618 / 568; 5 limbs 62 / 38 / 38, 163 / 198 / 175, 158 / 173 / 154; 3 limbs 34 / 32 / 30, 95 / 120 / 104, 84 / 94 / 82.  (32 KB would
// take 5 limbs to 131 and 125 there, and from 38 to 44 with near exponents.)  Wider kernels hold few blocks anyway (13 limbs, near: default
// 89, 64 KB 95).
template <int N> constexpr int ew_tiles(int op) { return op >= 11 && N <= 12 ? 2 : ew_inputs(op); }
template <int N> constexpr size_t ew_smem_bytes(int op) { return (size_t)ew_tiles<N>(op) * kEwThreads * ew_stride<N>() * 4; }
// The block's rows of every operand, in tiles of kEwThreads rows; returns how many rows the block has.
template <int N, int OP> __device__ __forceinline__ int ew_load_tiles(const EwParams& p, u32* tile, u64 row0, bool& wide) {
    constexpr int parts = ew_complex(OP) ? 2 : 1, T = kEwThreads * ew_stride<N>();
    const u64 left = parts * p.count - row0;
    const int rows = left < (u64)kEwThreads ? (int)left : kEwThreads;
    wide = p.aligned && rows == kEwThreads;
    ew_fetch<N>(tile, p.a, row0, rows, 1, 0, parts, wide);
    if constexpr (ew_inputs(OP) > 1) ew_fetch<N>(tile + T, p.b, row0, rows, p.bs, p.bp, parts, wide);
    if constexpr (ew_tiles<N>(OP) > 2) ew_fetch<N>(tile + 2 * T, p.c, row0, rows, p.cs, p.cp, parts, wide);
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    return rows;
}

template <int N, int OP> __global__ void __launch_bounds__(kEwThreads) ew_kernel(EwParams p) {
    constexpr int S = ew_stride<N>(), T = kEwThreads * S;
    extern __shared__ __align__(16) u32 ew_park[];
    const u64 row0 = (u64)blockIdx.x * kEwThreads;
    bool wide;
    const int rows = ew_load_tiles<N, OP>(p, ew_park, row0, wide);
    u32* const mine = ew_park + threadIdx.x * S;
    if ((int)threadIdx.x < rows) {
        const Num<N> x = load_plain<N>(mine);
        Num<N> z;
        if constexpr (OP == 7) z = mul_mem<N>(x, mine);
        else if constexpr (OP == 8) z = lfd::sqrt<N>(x);
        else if constexpr (OP == 2) z = mul_mem<N>(x, mine + T);
        else {
            const Num<N> y = load_plain<N>(mine + T);
            if constexpr (OP == 0) z = add<N>(x, y);
            else if constexpr (OP == 1) z = sub<N>(x, y);
            else if constexpr (OP == 3) z = div<N>(x, y);
            else {
                const Num<N> w = load_plain<N>(mine + 2 * T);
                z = OP == 9 ? fma<N>(x, y, w) : fms<N>(x, y, w);
            }
        }
        store<N>(mine, z);
    }
    __syncthreads();
    ew_put<N>(ew_park, p.out, row0, rows, wide);
}

// Complex operations: two lanes per value, one component each (lane 2q real, 2q + 1 imaginary).  The components are
// independent rounding sequences but for the quotient's denominator |b|^2, whose two squares the lanes form and
// exchange.  A thread then holds one running sum beside a product instead of two whole complex values, and the serial
// chain of a quotient is three products and one division instead of six and two: at 1024 bits, where 65,536 pairs are
// few warps, the operation is bound by that chain's latency.  The products run as one rolled loop whose second factors
// are read from memory, so the code of one product is fetched once.  Both lanes have read all their operands before
// either writes its result over the first operand's row.
template <int N, int OP> __global__ void __launch_bounds__(kEwThreads, (N > 16 && OP <= 6 ? 3 : 1)) ew_pair_kernel(EwParams p) {
    constexpr int S = ew_stride<N>(), T = kEwThreads * S;
    extern __shared__ __align__(16) u32 ew_park[];
    const u64 row0 = (u64)blockIdx.x * kEwThreads;
    constexpr bool kAddendTile = ew_tiles<N>(OP) > 2;
    Num<N> w = zero<N>();
    if constexpr (OP >= 11 && !kAddendTile) {                     // this lane's component of the addend
        const u64 row = row0 + threadIdx.x;
        if (row < 2 * p.count) w = load<N>(p.c + (p.cs == 1 && !p.cp ? row : 2 * bidx(row >> 1, p.cs, p.cp) + (row & 1)) * (N + 3));
    }
    bool wide;
    const int rows = ew_load_tiles<N, OP>(p, ew_park, row0, wide);
    const int im = (int)(threadIdx.x & 1);
    u32* const a = ew_park + (threadIdx.x & ~1u) * S;            // the value's real row; its imaginary row follows
    const u32* const b = a + T;
    if ((int)threadIdx.x < rows) {                                // rows is even: both lanes of a pair, or neither
        const u32 pair = 3u << (threadIdx.x & 30u);
        Num<N> z;
        if constexpr (OP == 4) {
            z = add<N>(load_plain<N>(a + im * S), load_plain<N>(b + im * S));
        } else if constexpr (OP == 5 || OP == 6) {
            // product:  re = a.re b.re - a.im b.im          im = a.re b.im + a.im b.re
            // quotient: re = (a.re b.re + a.im b.im) / d    im = (a.im b.re - a.re b.im) / d
            z = zero<N>();
            Num<N> first = z;
#pragma unroll 1
            for (int s = 0; s < (OP == 6 ? 3 : 2); ++s) {
                const u32* x; const u32* y;
                if constexpr (OP == 5) { x = a + s * S; y = b + (s ^ im) * S; }
                else { x = s == 2 ? b + im * S : a + (s ^ im) * S; y = s == 2 ? x : b + s * S; }
                Num<N> q = mul_mem<N>(load_plain<N>(x), y);
                if (s == 0) { first = q; continue; }
                if (s == 1) { if (OP == 5 ? !im : im) q.s = -q.s; }
                else {
                    z = first;                                        // the numerator waits for the denominator
#pragma unroll
                    for (int w = 0; w < N; ++w) first.m[w] = __shfl_xor_sync(pair, q.m[w], 1);
                    first.e = __shfl_xor_sync(pair, q.e, 1);
                    first.s = __shfl_xor_sync(pair, q.s, 1);
                    first.st = __shfl_xor_sync(pair, q.st, 1);
                }
                first = add<N>(first, q);
            }
            if constexpr (OP == 6) z = div<N>(z, first); else z = first;
        } else {
            if constexpr (kAddendTile) w = load_plain<N>(a + 2 * T + im * S);
            const Num<N> ai = load_plain<N>(a + S);
            z = dot2_add<N>(load_plain<N>(a), load_plain<N>(b + im * S), im ? ai : negate<N>(ai), load_plain<N>(b + (im ^ 1) * S), OP == 12 ? negate<N>(w) : w);
        }
        __syncwarp(pair);
        store<N>(a + im * S, z);
    }
    __syncthreads();
    ew_put<N>(ew_park, p.out, row0, rows, wide);
}

// v <- op_s(v, b_s[...]) for every step; out_s written where non-null.  Steps are uniform across
// the grid, so the switch never diverges.  Products read the factor's words from memory inside the
// product (mul_mem), which keeps the kernel at about 120 registers; 64-thread blocks spread a
// one-wave grid evenly over the SMs.
constexpr int kChainThreads = 64;
template <int N, bool MUL_ONLY> __global__ void __launch_bounds__(kChainThreads) chain_kernel(const __grid_constant__ ChainParams p) {
    const u64 i = (u64)blockIdx.x * kChainThreads + threadIdx.x;
    if (i >= p.count) return;
    constexpr u64 E = N + 3;
    Num<N> v = load_plain<N>(p.a + E * i);
#pragma unroll 1
    for (int s = 0; s < p.steps; ++s) {
        const ChainStep& st = p.step[s];
        const u32* y = st.b + E * bidx(i, st.bs, st.bp);
        if constexpr (MUL_ONLY) v = mul_mem<N>(v, y);
        else switch (st.op) {
        case 0: v = add<N>(v, load_plain<N>(y)); break;
        case 1: v = sub<N>(v, load_plain<N>(y)); break;
        case 2: v = mul_mem<N>(v, y); break;
        default: v = div<N>(v, load_plain<N>(y)); break;
        }
        if (st.out) store<N>(st.out + E * i, v);
    }
}

// Multiplication chains whose factors are contiguous (no broadcast) and read nowhere that a step writes:
// a block of 32 values copies the next step's 32 factors (one contiguous tile of 32 (N+3) words, a
// multiple of 16 bytes) into shared memory with cp.async while the current products run, so the product
// reads its factor words from shared memory.  A partial last block reads its factors directly.
// Above 24 limbs the registers are held to 128, 16 blocks an SM, where the compiler would take some 160 (12 blocks): a block is one warp, and the
// products leave the pipe idle with twelve.  Eight products of 1,000 to 500,000 values at 800, 896, 960 and 1024 bits, 12 blocks against 16:
// 65,536 values 45 / 63 / 70 / 71 us and 42 / 54 / 59 / 67, 500,000 values 224 / 292 / 324 / 358 and 218 / 278 / 306 / 347; of 32 counts and
// widths two were slower (1024 bits: 30,000 values by 2%, 131,072 by 5%).
constexpr int kStagedThreads = 32;
template <int N> __global__ void __launch_bounds__(kStagedThreads, (N > 24 ? 16 : 1)) chain_staged_kernel(const __grid_constant__ ChainParams p) {
    constexpr u64 E = N + 3;
    constexpr int T = kStagedThreads, TILE = T * (int)E, CH = TILE / 4;
    static_assert(TILE % 4 == 0, "tiles of whole 16-byte chunks");
    const u64 base = (u64)blockIdx.x * T, i = base + threadIdx.x;
    if (base + T > p.count) {
        if (i >= p.count) return;
        Num<N> v = load_plain<N>(p.a + E * i);
#pragma unroll 1
        for (int s = 0; s < p.steps; ++s) {
            v = mul_mem<N>(v, p.step[s].b + E * i);
            if (p.step[s].out) store<N>(p.step[s].out + E * i, v);
        }
        return;
    }
    extern __shared__ __align__(16) u32 chain_stage[];
    const auto fetch = [&](int s) {
        const u32* src = p.step[s].b + E * base;
        u32* dst = chain_stage + (s & 1) * TILE;
        for (int c = threadIdx.x; c < CH; c += T) cp_async16(dst + 4 * c, src + 4 * c);
        cp_async_commit();
    };
    fetch(0);
    Num<N> v = load_plain<N>(p.a + E * i);
#pragma unroll 1
    for (int s = 0; s < p.steps; ++s) {
        if (s + 1 < p.steps) { fetch(s + 1); cp_async_wait<1>(); } else cp_async_wait<0>();
        __syncthreads();                                     // every thread's chunks of this step's tile
        v = mul_mem<N>(v, chain_stage + (s & 1) * TILE + threadIdx.x * E);
        if (p.step[s].out) store<N>(p.step[s].out + E * i, v);
        __syncthreads();                                     // the tile is refilled for step s + 2
    }
}
// ---- Lane pairs: one value over two lanes (N even, N >= 12).  Both lanes hold the running value a.  Lane p forms
// the rows j = 2m + p of the upper part T of a * y (the products a_i y_j with i + j >= N - 2, as mant_mul_high),
// each row a carry chain, into its own window; lane p's window index w'' stands for word w'' - 1 + p of T, which
// keeps every index static.  Lane 1's row 2m + 1 starts one product earlier than lane 0's row 2m; lane 0 takes that
// product with a zero operand.  One exchange of the windows (a shuffle per word) gives both lanes T, and both round
// it exactly as mul does, so the pair ends the step holding RN(a * y) bit for bit as one thread would.
template <int N> __device__ __forceinline__ Num<N> mul_pair(const Num<N>& a, const u32* y, int pl) {
    static_assert(N % 2 == 0 && N >= kShortMulLimbs, "lane pairs need an even width of at least kShortMulLimbs");
    constexpr int B = N - 2, W = N + 2;
    const int ys = (int)y[N + 1];
    const u32 st = a.st | y[N + 2];
    if (st || !a.s || !ys) return zero<N>(st);
    u32 h[W + 1];
#pragma unroll
    for (int k = 0; k <= W; ++k) h[k] = 0;
#pragma unroll
    for (int m = 0; m < N / 2; ++m) {
        const u32 bj = y[2 * m + pl];
        const int i1 = B - 2 * m - 1 > 0 ? B - 2 * m - 1 : 0;           // lane 1's first product (static)
        const bool mask0 = B - 2 * m - 1 >= 0;                           // lane 0 starts one later: zero operand
        u32 c = 0;
#pragma unroll
        for (int i = i1; i < N; ++i) {
            const u32 ai = (i == i1 && mask0 && !pl) ? 0u : a.m[i];
            const u64 t = (u64)ai * bj + h[i + 2 * m - B + 1] + c;
            h[i + 2 * m - B + 1] = (u32)t;
            c = (u32)(t >> 32);
        }
        h[2 * m + 3] = c;                                                // N - 1 + 2m - B + 2
    }
    // T word w = h0[w + 1] + h1[w]: each lane sends its share of word w and adds the partner's.  The exchange names
    // only the two lanes of the pair: other pairs of the warp may have left (a zero or status operand above, or a
    // value past the end), and both lanes of a pair always take the same path (they hold the same a and y).
    const u32 pair = 3u << ((threadIdx.x & 31) & ~1u);
    u32 cy = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        const u32 mine = pl ? h[w] : h[w + 1];
        const u32 other = __shfl_xor_sync(pair, mine, 1);
        const u64 t = (u64)mine + other + cy;
        h[w] = (u32)t;
        cy = (u32)(t >> 32);
    }
    const u32 sh = (h[N + 1] >> 31) ? 0u : 1u;
    const u32 lw = h[1] << sh;
    const u32 low = lw & 0x7fffffffu;
    const bool rb = lw >> 31;
    if (low >= 0x80000000u - ((u32)N << sh) || (rb && low == 0)) return mul_exact_mem_call<N>(a, y);
    u32 m[N];
#pragma unroll
    for (int i = 0; i < N; ++i) m[i] = __funnelshift_l(h[i + 1], h[i + 2], sh);
    return finish<N>(m, (i64)a.e + (int)y[N] + 1 - (i64)sh, a.s * ys, rb, 0);
}
constexpr int kPairThreads = 64;                          // 32 values per block
template <int N> __global__ void __launch_bounds__(kPairThreads, 10) chain_pair_kernel(const __grid_constant__ ChainParams p) {
    constexpr u64 E = N + 3;
    constexpr int V = kPairThreads / 2, TILE = V * (int)E, CH = TILE / 4;
    static_assert(TILE % 4 == 0, "tiles of whole 16-byte chunks");
    const int pl = threadIdx.x & 1, vi = threadIdx.x >> 1;
    const u64 base = (u64)blockIdx.x * V, i = base + vi;
    if (base + V > p.count) {                                       // partial block: factors straight from memory
        if (i >= p.count) return;                                    // both lanes of a pair leave together
        Num<N> v = load_plain<N>(p.a + E * i);
#pragma unroll 1
        for (int s = 0; s < p.steps; ++s) {
            v = mul_pair<N>(v, p.step[s].b + E * i, pl);
            if (p.step[s].out && !pl) store<N>(p.step[s].out + E * i, v);
        }
        return;
    }
    extern __shared__ __align__(16) u32 pair_stage[];
    const auto fetch = [&](int s) {
        const u32* src = p.step[s].b + E * base;
        u32* dst = pair_stage + (s & 1) * TILE;
        for (int c = threadIdx.x; c < CH; c += kPairThreads) cp_async16(dst + 4 * c, src + 4 * c);
        cp_async_commit();
    };
    fetch(0);
    Num<N> v = load_plain<N>(p.a + E * i);
#pragma unroll 1
    for (int s = 0; s < p.steps; ++s) {
        if (s + 1 < p.steps) { fetch(s + 1); cp_async_wait<1>(); } else cp_async_wait<0>();
        __syncthreads();
        v = mul_pair<N>(v, pair_stage + (s & 1) * TILE + vi * E, pl);
        if (p.step[s].out && !pl) store<N>(p.step[s].out + E * i, v);
        __syncthreads();
    }
}

// The staged kernel applies when every factor is contiguous, 16-byte aligned and disjoint from every output.
inline bool chain_can_stage(const ChainParams& p, u64 E) {
    const u64 bytes = p.count * E * 4;
    for (int k = 0; k < p.steps; ++k) {
        const ChainStep& st = p.step[k];
        if (st.op != 2 || st.bs != 1 || st.bp != 0 || ((uintptr_t)st.b & 15)) return false;
        const uintptr_t b0 = (uintptr_t)st.b, b1 = b0 + bytes;
        for (int q = 0; q < p.steps; ++q) {
            if (!p.step[q].out) continue;
            const uintptr_t o0 = (uintptr_t)p.step[q].out, o1 = o0 + bytes;
            if (b0 < o1 && o0 < b1) return false;
        }
    }
    return true;
}

template <int N, int OP> void launch_ew_op(const EwParams& p, cudaStream_t s) {
    constexpr size_t smem = ew_smem_bytes<N>(OP);
    const unsigned blocks = (unsigned)(((ew_complex(OP) ? 2 * p.count : p.count) + kEwThreads - 1) / kEwThreads);
    if constexpr (ew_complex(OP)) {
        if constexpr (smem > 48 * 1024) cudaFuncSetAttribute(ew_pair_kernel<N, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if constexpr (ew_tiles<N>(OP) < ew_inputs(OP)) {
            static std::atomic<uint64_t> asked{0};
            prefer_carveout(ew_pair_kernel<N, OP>, 28, asked);
        }
        ew_pair_kernel<N, OP><<<blocks, kEwThreads, smem, s>>>(p);
    } else {
        if constexpr (smem > 48 * 1024) cudaFuncSetAttribute(ew_kernel<N, OP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        ew_kernel<N, OP><<<blocks, kEwThreads, smem, s>>>(p);
    }
}
template <int N> int launch_ew(int op, const EwParams& pin, cudaStream_t s) {
    if (!pin.count) return 0;
    EwParams p = pin;
    p.aligned = !(((uintptr_t)p.a | (uintptr_t)p.b | (uintptr_t)p.c | (uintptr_t)p.out) & 15);
    switch (op) {
    case 0: launch_ew_op<N, 0>(p, s); break;
    case 1: launch_ew_op<N, 1>(p, s); break;
    case 2: launch_ew_op<N, 2>(p, s); break;
    case 3: launch_ew_op<N, 3>(p, s); break;
    case 4: launch_ew_op<N, 4>(p, s); break;
    case 5: launch_ew_op<N, 5>(p, s); break;
    case 6: launch_ew_op<N, 6>(p, s); break;
    case 7: launch_ew_op<N, 7>(p, s); break;
    case 8: launch_ew_op<N, 8>(p, s); break;
    case 9: launch_ew_op<N, 9>(p, s); break;
    case 10: launch_ew_op<N, 10>(p, s); break;
    case 11: launch_ew_op<N, 11>(p, s); break;
    case 12: launch_ew_op<N, 12>(p, s); break;
    default: return 1;
    }
    return 0;
}
template <int N> int launch_chain(const ChainParams& p, cudaStream_t s) {
    if (!p.count) return 0;
    const unsigned blocks = (unsigned)((p.count + kChainThreads - 1) / kChainThreads);
    bool mul_only = true;
    for (int k = 0; k < p.steps; ++k) mul_only = mul_only && p.step[k].op == 2;
    if (mul_only && chain_can_stage(p, N + 3)) {
        if constexpr (N % 2 == 0 && N >= kShortMulLimbs) {
            if (p.lanes == 2) {
                const unsigned pb = (unsigned)((p.count + kPairThreads / 2 - 1) / (kPairThreads / 2));
                chain_pair_kernel<N><<<pb, kPairThreads, 2 * (kPairThreads / 2) * (N + 3) * 4, s>>>(p);
                return 0;
            }
        }
        const unsigned sb = (unsigned)((p.count + kStagedThreads - 1) / kStagedThreads);
        chain_staged_kernel<N><<<sb, kStagedThreads, 2 * kStagedThreads * (N + 3) * 4, s>>>(p);
    } else if (mul_only) chain_kernel<N, true><<<blocks, kChainThreads, 0, s>>>(p);     // registers of mul alone
    else chain_kernel<N, false><<<blocks, kChainThreads, 0, s>>>(p);
    return 0;
}

// Attributes of the element-wise kernel of one operation (the query also loads the kernel's module, which a
// first launch would otherwise do): Engine::prewarm and Engine::pipeline_info.
template <int N> int ew_attributes(int op, cudaFuncAttributes* a) {
    switch (op) {
    case 0: return cudaFuncGetAttributes(a, ew_kernel<N, 0>);
    case 1: return cudaFuncGetAttributes(a, ew_kernel<N, 1>);
    case 2: return cudaFuncGetAttributes(a, ew_kernel<N, 2>);
    case 3: return cudaFuncGetAttributes(a, ew_kernel<N, 3>);
    case 4: return cudaFuncGetAttributes(a, ew_pair_kernel<N, 4>);
    case 5: return cudaFuncGetAttributes(a, ew_pair_kernel<N, 5>);
    case 6: return cudaFuncGetAttributes(a, ew_pair_kernel<N, 6>);
    case 7: return cudaFuncGetAttributes(a, ew_kernel<N, 7>);
    case 8: return cudaFuncGetAttributes(a, ew_kernel<N, 8>);
    case 9: return cudaFuncGetAttributes(a, ew_kernel<N, 9>);
    case 10: return cudaFuncGetAttributes(a, ew_kernel<N, 10>);
    case 11: return cudaFuncGetAttributes(a, ew_pair_kernel<N, 11>);
    case 12: return cudaFuncGetAttributes(a, ew_pair_kernel<N, 12>);
    default: return (int)cudaErrorInvalidValue;
    }
}

// Dispatch tables filled by the per-width translation units (lf_ew_*.cu).
typedef int (*EwLauncher)(int, const EwParams&, cudaStream_t);
typedef int (*ChainLauncher)(const ChainParams&, cudaStream_t);
typedef int (*EwAttributes)(int, cudaFuncAttributes*);
EwLauncher ew_launcher(int limbs);
ChainLauncher chain_launcher(int limbs);
EwAttributes ew_attributes_of(int limbs);

}  // namespace lfd

#define LF_EW_INSTANTIATE(N)                                                             \
    namespace lfd {                                                                      \
    int ew_launch_##N(int op, const EwParams& p, cudaStream_t s) { return launch_ew<N>(op, p, s); } \
    int chain_launch_##N(const ChainParams& p, cudaStream_t s) { return launch_chain<N>(p, s); } \
    int ew_attr_##N(int op, cudaFuncAttributes* a) { return ew_attributes<N>(op, a); } \
    }
