// Exact products with few outputs and long sums that the residue engine does not take (exponents too far apart): a block per
// output, its 256 threads sharing the terms (block_exact_sum of the QR panels), the old entry as one more term.
// The tiled limb kernel gives an output one thread, whose K products follow one another: the 64 x 4 sums of 1600 terms by
// which a complex QR factor's block meets the right-hand sides took it 7.8 ms.
#pragma once
#include "lf_qr.cuh"

namespace lfd {

// c - sum x_k y_k or sum x_k y_k as terms a_k b_k: the products, then c times one.
template <int N> struct AddedDot {
    const u32* c; bool subtract; const u32* x; i64 sx; const u32* y; i64 sy; u64 K;
    __device__ void operands(u64 k, Num<N>& a, Num<N>& b) const {
        constexpr i64 E = N + 3;
        if (k < K) {
            a = ldn<N, true>(x + (i64)k * sx * E); b = ldn<N, true>(y + (i64)k * sy * E);
            if (subtract) a.s = -a.s;
        } else {
            a = load_plain<N>(c); b = qr_pow2<N>(0);
        }
    }
    __device__ Num<N> fallback(u32* error) const { return exact_dot_add_dev<N, true>(c, subtract, x, sx, y, sy, K, error); }
};
// Where a block per output is the faster form.  At 256 bits and 1600 terms, some 296 outputs at a time take 0.1 ms, and the tiled
// kernel some 1.6 us a term for any number of outputs up to a hundred thousand: the lines cross at 6600 outputs, at 128 terms
// at 2400.  spread: the widest line's exponent spread where the analysis showed it, which must leave the products inside the
// block's window (a sum that does not fit is one lane's work); -1 where nobody looked, and then only
// products too small to fill the tiled kernel's blocks.  Shorter sums leave most of a block's threads without a term.
inline bool long_dot_fits(int limbs, u64 M, u64 Nc, u64 K, int spread) {
    if (K < 128) return false;
    if (spread < 0) return M * Nc <= 512;
    int logk = 0;
    while ((1ull << logk) < K) ++logk;
    const int spare = 32 * (limbs <= 16 ? 26 : 14);              // qr_window beyond a product's 2 N words
    return M * Nc <= 2048 && 2 * (i64)spread + logk + 3 < spare;
}
template <int N> __global__ void __launch_bounds__(qr_threads<N>()) long_dot_kernel(DotParams p) {
    constexpr u64 E = N + 3;
    __shared__ __align__(16) u32 sm[qr_dot_words<N>()];
    const u64 i = blockIdx.x / p.Nc, j = blockIdx.x % p.Nc;
    if (p.lower && j > i) return;
    u32* out = p.C + (i * p.ldc + j) * E;
    const AddedDot<N> src{p.subtract ? out : nullptr, p.subtract != 0, p.left.base + i * p.left.ls * E, (i64)p.left.ks,
                          p.right.base + j * p.right.ls * E, (i64)p.right.ks, p.K};
    const Num<N> v = block_exact_sum<N>(src, p.K + (p.subtract ? 1 : 0), sm, p.error);
    if (threadIdx.x == 0) store<N>(out, v);                        // every thread read its terms before the sum's last barrier
}
template <int N> void long_dot_launch(const DotParams& p, cudaStream_t s) {
    if (p.M && p.Nc) long_dot_kernel<N><<<(unsigned)(p.M * p.Nc), qr_threads<N>(), 0, s>>>(p);
}
DotFn long_dot_launcher(int limbs);

}  // namespace lfd

#define LF_LONG_DOT_INSTANTIATE(N) namespace lfd { void long_dot_##N(const DotParams& p, cudaStream_t s) { long_dot_launch<N>(p, s); } }
