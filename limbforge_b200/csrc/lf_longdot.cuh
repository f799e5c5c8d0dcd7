// Exact products with few outputs and long sums that the residue engine does not take (exponents too far apart): a block per
// output, its 256 or 512 threads sharing the terms (block_exact_sum of the QR panels), the old entry as one more term.
// The tiled limb kernel gives an output one thread, whose K products follow one another: the 64 x 4 sums of 1600 terms by
// which a complex QR factor's block meets the right-hand sides took it 7.8 ms.
// An output whose terms do not fit the block's window is left to a second launch (long_rest_kernel), a warp for each: the cluster method is
// one lane's work, and a block of 512 threads that waits for it is most of an SM (16 x 32 outputs of 1000 256-bit terms with
// exponents of +-3000: 1.89 s in the blocks, 0.81 in the tiled kernel, 0.66 by warps).  Where it is the old entry that does not
// fit, the block sums the products alone and rounds their sum with it.
#pragma once
#include "lf_qr.cuh"
#include "lf_residue.cuh"

namespace lfd {

// c - sum x_k y_k or sum x_k y_k as terms a_k b_k: the products, then c times one.
template <int N> struct AddedDot {
    const u32* c; bool subtract; const u32* x; i64 sx; const u32* y; i64 sy; u64 K;
    int* spilled;                          // shared: set where the terms do not fit the window
    __device__ void operands(u64 k, Num<N>& a, Num<N>& b) const {
        constexpr i64 E = N + 3;
        if (k < K) {
            a = ldn<N, true>(x + (i64)k * sx * E); b = ldn<N, true>(y + (i64)k * sy * E);
            if (subtract) a.s = -a.s;
        } else {
            a = load_plain<N>(c); b = qr_pow2<N>(0);
        }
    }
    __device__ Num<N> fallback(u32*) const { *spilled = 1; return zero<N>(); }       // one thread, before a barrier
};
// Where a block per output is the faster form.  At 256 bits and 1600 terms, some 296 outputs at a time take 0.1 ms, and the tiled
// kernel some 1.6 us a term for any number of outputs up to a hundred thousand: the lines cross at 6600 outputs, at 128 terms
// at 2400.  spread: the widest line's exponent spread where the analysis showed it, which must leave the products inside the
// block's window (wider, the tiled kernel's windows follow the spread); -1 where nobody looked, and then only
// products too small to fill the tiled kernel's blocks.  Shorter sums leave most of a block's threads without a term.
inline bool long_dot_fits(int limbs, u64 M, u64 Nc, u64 K, int spread) {
    if (K < 128) return false;
    if (spread < 0) return M * Nc <= 512;
    int logk = 0;
    while ((1ull << logk) < K) ++logk;
    const int spare = 32 * (limbs <= 16 ? 26 : 14);              // qr_window beyond a product's 2 N words
    return M * Nc <= 2048 && 2 * (i64)spread + logk + 3 < spare;
}
template <int N> struct LongOutput {
    const u32 *x, *y; u32* out; bool live;
    __device__ LongOutput(const DotParams& p, u64 o) {
        constexpr u64 E = N + 3;
        const u64 i = o / p.Nc, j = o % p.Nc;
        live = i < p.M && !(p.lower && j > i);
        out = p.C + (i * p.ldc + j) * E; x = p.left.base + i * p.left.ls * E; y = p.right.base + j * p.right.ls * E;
    }
};
// rest[o]: whether output o is left to long_rest_kernel.
template <int N> __global__ void __launch_bounds__(qr_threads<N>()) long_dot_kernel(DotParams p, u32* rest) {
    constexpr int W = qr_window<N>();
    __shared__ __align__(16) u32 sm[qr_dot_words<N>()];
    __shared__ u32 keep[qr_keep_words<N>()];
    __shared__ int spilled;
    const LongOutput<N> o(p, blockIdx.x);
    if (!o.live) return;
    if (threadIdx.x == 0) spilled = 0;                             // block_exact_sum has a barrier before it asks for the fallback
    const AddedDot<N> src{p.subtract ? o.out : nullptr, p.subtract != 0, o.x, (i64)p.left.ks, o.y, (i64)p.right.ks, p.K, &spilled};
    Num<N> v = block_exact_sum<N>(src, p.K + (p.subtract ? 1 : 0), sm, p.error);
    if (spilled && p.subtract) {                                   // the products alone, and their sum with the old entry in one rounding
        __syncthreads();
        if (threadIdx.x == 0) spilled = 0;
        block_exact_sum<N>(src, p.K, sm, p.error, keep);
        if (!spilled && threadIdx.x == 0) {
            v = load_plain<N>(o.out);
            if (keep[0]) {
                u32 X[W], scratch[round_sum2_words<N>(W)];
                const bool neg = keep[6 + W - 1] >> 31;
                for (int w = 0; w < W; ++w) X[w] = keep[6 + w];
                negate_words<W>(X, neg);
                v = round_sum2<N>(X, W, (i64)((u64)keep[1] | ((u64)keep[2] << 32)), neg ? -1 : 1, v, scratch);
            }
        }
    }
    if (threadIdx.x == 0) {                                        // every thread read its terms before the sum's last barrier
        rest[blockIdx.x] = spilled;
        if (!spilled) store<N>(o.out, v);
    }
}
template <int N> __global__ void __launch_bounds__(32) long_rest_kernel(DotParams p, const u32* rest) {
    const LongOutput<N> o(p, blockIdx.x);
    if (threadIdx.x || !o.live || !rest[blockIdx.x]) return;
    store<N>(o.out, exact_dot_add_dev<N, true>(p.subtract ? o.out : nullptr, p.subtract, o.x, (i64)p.left.ks, o.y, (i64)p.right.ks, p.K, p.error));
}
template <int N> void long_dot_launch(const DotParams& p, u32* rest, cudaStream_t s) {
    if (!p.M || !p.Nc) return;
    const unsigned outputs = (unsigned)(p.M * p.Nc);
    long_dot_kernel<N><<<outputs, qr_threads<N>(), 0, s>>>(p, rest);
    long_rest_kernel<N><<<outputs, 32, 0, s>>>(p, rest);
}
typedef void (*LongDotFn)(const DotParams&, u32* rest, cudaStream_t);       // rest: M Nc words of scratch
LongDotFn long_dot_launcher(int limbs);

}  // namespace lfd

#define LF_LONG_DOT_INSTANTIATE(N) namespace lfd { void long_dot_##N(const DotParams& p, u32* rest, cudaStream_t s) { long_dot_launch<N>(p, rest, s); } }
