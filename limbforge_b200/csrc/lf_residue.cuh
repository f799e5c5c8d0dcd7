// Int8-residue / CRT exact products (the reference's plan D6, linalg.mm:305-404 and
// linalg.metal:23-152, redesigned for sm_100a):
//
//  1. digits: every entry of a line becomes the exact integer X = mantissa * 2^(e - bottom(line))
//     (< 2^(32N+G), G = widest line spread), reduced modulo L primes m_l < 2^16 to a balanced
//     residue r = 256 d1 + d0 with int8 digits; planes D1/D0 [L][rows][Kp] (K-major, zero padded).
//  2. mma: per modulus and 128x80 output tile, tcgen05.mma kind::i8 with int32 accumulators in
//     TMEM: S11 = D1a D1b^T, S00 = D0a D0b^T, Smid = D1a D0b^T + D0a D1b^T; operands fed by TMA
//     (128-byte swizzle, no multicast); epilogue r = (65536 S11 + 256 Smid + S00) mod m -> uint16, for the tensor-core
//     CRT already weighted: t = r (M/m_l)^-1 mod m_l.
//  3. reconstruct: per output, CRT of the L residues (X = sum_l t_l (M/m_l) - q M, q = round of the
//     fixed-point sum of t_l/m_l; the modulus product exceeds 4 max|X| so the rounding of q is never
//     close), then RN(c - X 2^scale) (or RN(X 2^scale)) with one rounding; the sums over l are a second int8 product.
// Every step is exact integer arithmetic, so the outputs equal the generic limb kernel's bit for bit.
#pragma once
#include "lf_linalg.cuh"
#include <cuda.h>

namespace lfd {

constexpr int kResMaxModuli = 160;
constexpr int kResMaxQWords = 80;          // words of M / m_l
struct ResTables {
    u32 m[kResMaxModuli];                  // moduli, descending primes < 2^16
    u64 barrett[kResMaxModuli];            // floor(2^64 / m)
    u32 w[kResMaxModuli];                  // (M / m_l)^{-1} mod m_l
    u64 frac[kResMaxModuli];               // floor(2^48 / m_l)
    u32 q[kResMaxModuli][kResMaxQWords];   // M / m_l, little-endian words
    u32 M[kResMaxQWords + 1];              // product of the moduli
    u32 pw[kResMaxModuli][40];             // 2^(32 w) mod m_l for the integer words (<= 40)
};

__device__ __forceinline__ u32 mod_barrett(u64 x, u32 m, u64 r) {
    u64 q = __umul64hi(x, r);
    u64 t = x - q * m;
    while (t >= m) t -= m;                 // at most twice
    return (u32)t;
}

// ---------------------------------------------------------------- 1. digit planes
struct DigitParams {
    LineView v; u64 lines, K, Kp, rows_pad; int L; int xwords;
    const LineInfo* info; const ResTables* tab;
    signed char* d1; signed char* d0;      // [L][rows_pad][Kp]
};
template <int N> __global__ void __launch_bounds__(128) digits_kernel(DigitParams p) {
    const u64 k = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const u64 line = blockIdx.y;                          // rows_pad lines: padding rows are zero
    if (k >= p.Kp || line >= p.rows_pad) return;
    u32 x[40];
    for (int w = 0; w < 40; ++w) x[w] = 0;
    bool nz = false, negative = false;
    if (k < p.K && line < p.lines) {
        const Num<N> a = load<N>(p.v.base + (line * p.v.ls + k * p.v.ks) * (u64)(N + 3));
        if (!a.st && a.s) {
            nz = true; negative = a.s < 0;
            const int sh = a.e - p.info[line].bottom;       // 0 <= sh <= G
            const int ws = sh >> 5, bs = sh & 31;
            for (int i = 0; i <= N; ++i) {
                u32 v = i < N ? a.m[i] << bs : 0u;
                if (bs && i > 0) v |= a.m[i - 1] >> (32 - bs);
                x[i + ws] = v;
            }
        }
    }
    const u64 plane = p.rows_pad * p.Kp;
    for (int l = 0; l < p.L; ++l) {
        int r = 0;
        if (nz) {
            const u32 m = p.tab->m[l];
            u64 acc = 0;
            for (int w = 0; w < p.xwords; ++w) acc += (u64)x[w] * p.tab->pw[l][w];     // < 2^54
            u32 u = mod_barrett(acc, m, p.tab->barrett[l]);
            if (negative && u) u = m - u;                     // residue of -X
            r = (int)u;
            if (r > (int)(m >> 1)) r -= (int)m;               // balanced: |r| <= (m-1)/2 <= 32639
        }
        const int lo = (int)(signed char)(r & 0xff);
        const int hi = (r - lo) >> 8;                         // in [-128, 127] because m <= 65279
        p.d1[l * plane + line * p.Kp + k] = (signed char)hi;
        p.d0[l * plane + line * p.Kp + k] = (signed char)lo;
    }
}

// ---------------------------------------------------------------- 2. tcgen05 residue products
// Output tiles of 128 x 80: the three accumulators take 240 of 256 allocated TMEM columns and two stages 104 KB, so two
// CTAs share an SM and one's epilogue runs under the other's loads and MMAs (a 128 x 128 tile fills TMEM and leaves
// the tensor pipe idle during its epilogue: 33% active).  The operands' way from L2 then bounds the kernel (128 x 64 tiles: 8.5 TB/s
// over 1024^3 products of 75 moduli, 0.435 ms), so the tile is the widest that leaves room for the second CTA (0.374 ms).
constexpr int kTileM = 128, kTileN = 80, kTileK = 128;       // K tile in int8 elements = one 128-byte row
constexpr int kKAlign = 32;                                   // planes hold K rounded up to one MMA step, not a whole tile
constexpr int kStages = 2;
constexpr int kTileABytes = kTileM * kTileK, kTileBBytes = kTileN * kTileK;
constexpr int kStageBytes = 2 * (kTileABytes + kTileBBytes);  // D1a, D0a, D1b, D0b
constexpr u32 kMmaTmem = 256;
constexpr u32 kSpinLimit = 1u << 28;                          // bounded mbarrier waits
constexpr int kMmaThreads = 256;                              // warps w and w + 4 share TMEM lanes 32 (w % 4) ..
constexpr int kDigitThreads = 256;                            // digit planes: the same lane sharing
constexpr int kCrtThreads = 256;                              // CRT column sums: the same lane sharing

struct MmaParams {
    u16* res;                               // L times [M][Nc] residues (0 <= r < m), times w_l mod m_l when weighted
    const ResTables* tab;
    u64 M, Nc, Kp;
    int lower;                              // skip tiles strictly above the diagonal (SYRK)
    u32* error;
    const ResPlan* plan;                    // planned on the GPU: moduli at or above plan->L have no work
    u32 poll_limit;                         // polls of a barrier wait before it gives up (0: kSpinLimit)
    int no_loads;                           // failure test only: the producer issues no loads, so the first wait runs out
    int weighted;                           // store t_l = r w_l mod m_l, the operand of the tensor-core CRT
    u64 pitch;                              // residues from one modulus to the next, 0: M * Nc
};

__device__ __forceinline__ u32 smem_u32(const void* p) { return (u32)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(u64* bar, u32 count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(u64* bar, u32 bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(u64* bar, u32 phase) {
    u32 ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(phase) : "memory");
    return ok != 0;
}
// Bounded wait: false (and the error flag set) when the barrier has not completed after `limit` polls.
__device__ __forceinline__ bool mbar_wait(u64* bar, u32 phase, u32* error, u32 limit = kSpinLimit) {
    for (u32 it = 0; it < limit; ++it)
        if (mbar_try_wait(bar, phase)) return true;
    atomicExch(error, 2u);
    return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, u64* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 :: "r"(smem_u32(dst)), "l"((u64)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// K-major operand in 128-byte-swizzled 8-row atoms (1024 B): LBO 16 B, SBO 1024 B, layout SWIZZLE_128B.
__device__ __forceinline__ u64 smem_desc(const void* p) {
    const u64 start = (smem_u32(p) >> 4) & 0x3FFFu;
    return start | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// kind::i8: D s32, A s8, B s8, both K-major, M = 128, N = kTileN.
constexpr u32 kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((u32)(kTileN >> 3) << 17) | ((u32)(kTileM >> 4) << 24);

__device__ __forceinline__ void mma_i8(u32 d_tmem, u64 a, u64 b, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 :: "r"(d_tmem), "l"(a), "l"(b), "r"(kIdesc), "r"((u32)accumulate), "r"(0u));
}
__device__ __forceinline__ void mma_commit(u64* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(u32 taddr, u32 (&r)[32]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld16(u32 taddr, u32 (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}

#ifdef LF_RESIDUE_MMA_KERNEL
// x mod m in [0, 2m) for any 32-bit x, rr = floor(2^32 / m).
__device__ __forceinline__ u32 mod_lazy(u32 x, u32 m, u32 rr) { return x - __umulhi(x, rr) * m; }
// One CTA = one 128 x 80 output tile of one modulus (grid z).  Warp 0 lane 0 issues TMA loads,
// warp 1 lane 0 issues the MMAs; then all eight warps reduce the accumulators: warp w reads TMEM lanes
// 32 (w % 4) .. + 31 (rows) for every second group of 16 columns and stores 16 residues of a row with two
// 16-byte stores when the row stride allows.  The planes end at K rounded up to one MMA step of 32; the last
// K tile's rows beyond it are zeros that the TMA load fills in, and no MMA reads them.
__global__ void __launch_bounds__(kMmaThreads, 2) residue_mma_kernel(const __grid_constant__ CUtensorMap ta1, const __grid_constant__ CUtensorMap ta0,
                                                              const __grid_constant__ CUtensorMap tb1, const __grid_constant__ CUtensorMap tb0,
                                                              MmaParams p) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) u64 full[kStages], empty[kStages], done;
    __shared__ u32 tmem_slot;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const ResTables* tab = p.tab;
    if (p.plan) {
        if (p.plan->mode != 1 || blockIdx.z >= (unsigned)p.plan->L) return;
        tab = static_cast<const ResTables*>(p.plan->tab);
    }
    const int tm = blockIdx.y, tn = blockIdx.x, l = blockIdx.z;
    if (p.lower && (u64)tn * kTileN > (u64)tm * kTileM + kTileM - 1) return;      // whole tile above the diagonal
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_slot)), "r"(kMmaTmem));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const u32 tmem = tmem_slot;
    const u32 acc11 = tmem, acc00 = tmem + kTileN, accm = tmem + 2 * kTileN;
    const int kblocks = (int)((p.Kp + kTileK - 1) / kTileK);
    const u32 polls = p.poll_limit ? p.poll_limit : kSpinLimit;
    __shared__ int abort_flag, issued, consumed;          // stages loaded by the producer / read by the MMA issuer
    if (threadIdx.x == 0) { abort_flag = 0; issued = 0; consumed = kblocks; }
    __syncthreads();
    if (warp == 0 && lane == 0) {
        // producer; stops issuing once the MMA issuer has given up
        for (int kb = 0; kb < kblocks && !p.no_loads; ++kb) {
            const int s = kb % kStages;
            const u32 ph = (u32)((kb / kStages) & 1);
            if (kb >= kStages && !mbar_wait(&empty[s], ph ^ 1u, p.error, polls)) { abort_flag = 1; break; }
            if (*(volatile int*)&abort_flag) break;
            unsigned char* st = smem + s * kStageBytes;
            mbar_expect_tx(&full[s], kStageBytes);
            tma_load_3d(st, &ta1, &full[s], kb * kTileK, tm * kTileM, l);
            tma_load_3d(st + kTileABytes, &ta0, &full[s], kb * kTileK, tm * kTileM, l);
            tma_load_3d(st + 2 * kTileABytes, &tb1, &full[s], kb * kTileK, tn * kTileN, l);
            tma_load_3d(st + 2 * kTileABytes + kTileBBytes, &tb0, &full[s], kb * kTileK, tn * kTileN, l);
            issued = kb + 1;
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        bool ok = true;
        for (int kb = 0; kb < kblocks && ok; ++kb) {
            const int s = kb % kStages;
            const u32 ph = (u32)((kb / kStages) & 1);
            if (!mbar_wait(&full[s], ph, p.error, polls)) { ok = false; consumed = kb; *(volatile int*)&abort_flag = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;");
            unsigned char* st = smem + s * kStageBytes;
            const u64 a1 = smem_desc(st), a0 = smem_desc(st + kTileABytes), b1 = smem_desc(st + 2 * kTileABytes),
                      b0 = smem_desc(st + 2 * kTileABytes + kTileBBytes);
            const int left = (int)(p.Kp - (u64)kb * kTileK) / 32, steps = left < kTileK / 32 ? left : kTileK / 32;
            for (int kk = 0; kk < steps; ++kk) {
                const u64 off = (u64)(kk * 32) >> 4;           // 32 bytes along K inside the swizzled row
                const bool acc = kb > 0 || kk > 0;
                mma_i8(acc11, a1 + off, b1 + off, acc);
                mma_i8(acc00, a0 + off, b0 + off, acc);
                mma_i8(accm, a1 + off, b0 + off, acc);
                mma_i8(accm, a0 + off, b1 + off, true);
            }
            mma_commit(&empty[s]);                            // stage free once these MMAs have read it
        }
        mma_commit(&done);                                    // arrives after every MMA issued above
    }
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) {
        // An abandoned wait leaves loads in flight into shared memory: let every stage that was loaded and
        // not read complete (bounded) before the CTA releases its resources.
        for (int kb = consumed; kb < issued; ++kb) mbar_wait(&full[kb % kStages], (u32)((kb / kStages) & 1), p.error, polls);
    }
    const bool fine = mbar_wait(&done, 0, p.error, polls) && !abort_flag;
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (fine) {
        const u32 m = tab->m[l];
        const u32 rr = (u32)(tab->barrett[l] >> 32);          // floor(2^64 / m) >> 32 = floor(2^32 / m)
        const u32 w = p.weighted ? tab->w[l] : 1u;
        // multiples of m that make the sums nonnegative: |S11|, |S00| < 2^30 and |Smid| < 2^31 for K <= kMaxK
        const u32 off30 = ((1u << 30) / m + 1) * m, off31 = ((1u << 31) / m) * m;
        const int q = warp & 3, half = warp >> 2;
        const u64 row = (u64)tm * kTileM + q * 32 + lane;
        const u32 lane_base = (u32)(q * 32) << 16;
        const bool vec = (p.Nc & 7) == 0;                      // rows start on 16-byte boundaries
        const u64 pitch = p.pitch ? p.pitch : p.M * p.Nc;
        for (int c0 = half * 16; c0 < kTileN; c0 += 32) {
            u32 s11[16], s00[16], sm[16];
            tmem_ld16(acc11 + lane_base + c0, s11);
            tmem_ld16(acc00 + lane_base + c0, s00);
            tmem_ld16(accm + lane_base + c0, sm);
            asm volatile("tcgen05.wait::ld.sync.aligned;");
            if (row < p.M) {
                const u64 col0 = (u64)tn * kTileN + c0;
                u16* out = p.res + (u64)l * pitch + row * p.Nc + col0;
                u32 r[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    // 65536 S11 + 256 Smid + S00 by Horner's rule in 32-bit words: every mod_lazy leaves [0, 2m), 2m < 2^17
                    const u32 hi = mod_lazy(s11[c] + off30, m, rr) * 256u + mod_lazy(sm[c] + off31, m, rr);
                    const u32 x = mod_lazy(hi, m, rr) * 256u + (s00[c] + off30);
                    u32 t = mod_lazy(x, m, rr);
                    t = min(t, t - m);                         // [0, m)
                    t = mod_lazy(t * w, m, rr);
                    r[c] = min(t, t - m);
                }
                if (vec && col0 + 16 <= p.Nc) {
                    uint4* o = reinterpret_cast<uint4*>(out);
#pragma unroll
                    for (int v = 0; v < 2; ++v)
                        o[v] = make_uint4(r[8 * v] | (r[8 * v + 1] << 16), r[8 * v + 2] | (r[8 * v + 3] << 16),
                                          r[8 * v + 4] | (r[8 * v + 5] << 16), r[8 * v + 6] | (r[8 * v + 7] << 16));
                } else {
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        if (col0 + c < p.Nc) out[c] = (u16)r[c];
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kMmaTmem));
}

// Plans a product on the GPU from its line analysis (the rule of the host driver): the residue engine
// when some line is nonzero and status free, every such line spans at most max_band bits (G = the
// widest) and 0 < K <= max_k; L is then the smallest count whose log2 product cum[L] exceeds
// 2(32 limbs + G) + ceil(log2 K) + 3.  Otherwise the limb kernel.  One block.
struct PlanParams {
    const LineInfo* linfo; const LineInfo* rinfo; u64 M, Nc, K; int limbs;
    const ResPlan* cands; const double* cum; int Lmin, count;     // candidate i is L = Lmin + i
    int max_band; u64 max_k;
    ResPlan* out;
};
__global__ void __launch_bounds__(256) plan_kernel(PlanParams p) {
    __shared__ int sg[256], sa[256];
    int G = 0, any = 0;
    for (u64 i = threadIdx.x; i < p.M + p.Nc; i += blockDim.x) {
        const LineInfo li = i < p.M ? p.linfo[i] : p.rinfo[i - p.M];
        if (!li.status && li.nonzero) { G = max(G, li.top - li.bottom); any = 1; }
    }
    sg[threadIdx.x] = G; sa[threadIdx.x] = any;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
        if ((int)threadIdx.x < o) { sg[threadIdx.x] = max(sg[threadIdx.x], sg[threadIdx.x + o]); sa[threadIdx.x] |= sa[threadIdx.x + o]; }
        __syncthreads();
    }
    if (threadIdx.x) return;
    ResPlan r{};
    r.mode = 0; r.G = sg[0];
    if (sa[0] && sg[0] <= p.max_band && p.K && p.K <= p.max_k) {
        int logk = 0;
        while ((1ull << logk) < p.K) ++logk;
        const double need = 2.0 * (32 * p.limbs + sg[0]) + logk + 3;
        for (int i = 0; i < p.count; ++i)
            if (p.cum[i] > need) { r = p.cands[i]; r.mode = 1; r.G = sg[0]; break; }
    }
    *p.out = r;
}

#endif  // LF_RESIDUE_MMA_KERNEL

// ---------------------------------------------------------------- 3. reconstruction and rounding
struct RecParams {
    const u16* res; const ResTables* tab; int L; int qwords;
    const LineInfo* linfo; const LineInfo* rinfo;
    u32* C; u64 ldc, M, Nc;
    int subtract, lower;
};
// RN(sign_x * X * 2^sx + c) with one rounding for an exact multiword X: both terms in one exact
// window when they are close, otherwise the far smaller term as a sticky unit (as in fma).
// acc (len words, two's complement) -= t << off (t has tw words), borrow carried to the top.
__device__ __forceinline__ void acc_sub(u32* acc, int len, const u32* t, int tw, i64 off) {
    const int ws = (int)(off >> 5), bs = (int)(off & 31);
    u32 bo = 0;
    int k = ws;
    for (int q = 0; q <= tw && k < len; ++q, ++k) {
        u32 v = q < tw ? t[q] << bs : 0u;
        if (bs && q > 0) v |= t[q - 1] >> (32 - bs);
        const u64 d = (u64)v + bo;
        const u32 old = acc[k];
        acc[k] = (u32)((u64)old - d);
        bo = (u64)old < d;
    }
    for (; bo && k < len; ++k) { const u32 old = acc[k]; acc[k] = old - 1u; bo = old == 0u; }
}
__device__ __forceinline__ void acc_unit(u32* acc, int len, bool negative) {   // acc +-= 1
    if (negative) { for (int k = 0; k < len; ++k) { const u32 old = acc[k]; acc[k] = old - 1u; if (old) break; } }
    else { for (int k = 0; k < len; ++k) { if (++acc[k]) break; } }
}
// Scratch words round_sum2 needs for an X of xw words (the window below); callers pass that much.
template <int N> __host__ __device__ constexpr int round_sum2_words(int xw) { return xw + 2 * N + 8; }
template <int N> __device__ Num<N> round_sum2(const u32* X, int xw, i64 sx, int signx, const Num<N>& c, u32* acc) {
    // One two's-complement window of xw + 2N + 8 words under the larger top, two bits of headroom
    // above it: a term below the window lies at least 2N + 6 words under that top, beyond every
    // rounding decision, and counts as +-1 in the lowest word.  The window lives in the caller's
    // scratch (shared memory in crt_round_kernel).
    const int CW = round_sum2_words<N>(xw);
    int tx = -1;
    for (int w = xw - 1; w >= 0; --w) if (X[w]) { tx = w; break; }
    if (tx < 0) return c;                                       // no product term left
    const i64 topx = sx + 32 * (i64)tx + 31 - __clz(X[tx]);
    if (!c.s) {
        Rounded<N> R; round_info<N>(X, xw, sx, R);
        return finish<N>(R.m, R.e, signx, R.rb && (R.sb || (R.m[0] & 1u)), 0);
    }
    const i64 sc = (i64)c.e - (32 * N - 1), topc = c.e;
    const i64 hi = topx > topc ? topx : topc;
    const i64 lo = hi + 3 - 32 * (i64)(CW - 1);               // exponent of window bit 32
    for (int w = 0; w < CW; ++w) acc[w] = 0;
    if (sx >= lo) { if (signx > 0) acc_add(acc, CW, X, xw, 32 + (sx - lo)); else acc_sub(acc, CW, X, xw, 32 + (sx - lo)); }
    else acc_unit(acc, CW, signx < 0);
    if (sc >= lo) { if (c.s > 0) acc_add(acc, CW, c.m, N, 32 + (sc - lo)); else acc_sub(acc, CW, c.m, N, 32 + (sc - lo)); }
    else acc_unit(acc, CW, c.s < 0);
    const bool negative = acc[CW - 1] >> 31;
    if (negative) { u32 cy = 1; for (int w = 0; w < CW; ++w) { const u32 v = ~acc[w] + cy; cy = cy && v == 0; acc[w] = v; } }
    Rounded<N> R;
    if (!round_info<N>(acc, CW, lo - 32, R)) return zero<N>();   // exact cancellation
    return finish<N>(R.m, R.e, negative ? -1 : 1, R.rb && (R.sb || (R.m[0] & 1u)), 0);
}

// From S = sum_l t_l (M / m_l) (qwords + 2 words, clobbered) and F = sum_l t_l floor(2^48 / m_l):
// X = S - round(F / 2^48) M, the signed exact product sum; returns RN(c -/+ X 2^scale) (subtract) or
// RN(X 2^scale), one rounding.  The modulus product exceeds 4 max|X|, so the quotient's rounding is
// never close.
template <int N> __device__ __forceinline__ Num<N> crt_tail(u32* S, int qwords, u64 F, const ResTables* tab, i64 scale,
                                                          bool subtract, const Num<N>& c, u32* scratch) {
    const u64 q = (F + (1ull << 47)) >> 48;                  // round(F): X = S - q M
    // D = S - q*M (two's complement over qwords+2 words)
    u64 borrow = 0;
    for (int w = 0; w <= qwords + 1; ++w) {
        const u64 qm = (w <= qwords ? (u64)tab->M[w] : 0ull) * q + borrow;
        const u32 lo = (u32)qm;
        const u32 old = S[w];
        S[w] = old - lo;
        borrow = (qm >> 32) + (old < lo ? 1u : 0u);
    }
    int sign = 1;
    const int xw = qwords + 2;
    if (S[xw - 1] >> 31) {
        sign = -1; u64 c1 = 1;
        for (int w = 0; w < xw; ++w) { u64 v = (u64)(u32)~S[w] + c1; S[w] = (u32)v; c1 = v >> 32; }
    }
    // a zero exact sum X with the addend falls back to c itself, as exact_dot_add
    return round_sum2<N>(S, xw, scale, subtract ? -sign : sign, c, scratch);
}

// ---------------------------------------------------------------- 4. tiled limb-kernel product
// The generic limb kernel's fast form: C[i][j] = RN(c -/+ sum_k L(i,k) R(j,k)) with every product summed exactly in
// one window per output and rounded once (round_sum2 with the old entry), the same bits as exact_dot_add.  The line
// analysis bounds every product of output (i, j): a nonzero, status-free entry of line i has its exponent in
// [bottom_i, top_i], so the products' scales lie in [base, base + spread_i + spread_j] with base = bottom_i +
// bottom_j - 2(32N - 1), each below 2^(scale + 64N), and K of them sum below 2^(base + spread_i + spread_j + 64N +
// ceil(log2 K)).  When that fits kWinWords(N) words, the output adds each signed product, shifted to its bit offset
// (scale - base), word by word into signed 64-bit column sums: no carry runs between the words of a product, so the
// adds of one product are independent, and K < 2^28 products of 32-bit words cannot overflow a column.  One carry pass
// at the end turns the columns into a two's-complement window that is rounded once with the old entry; wider
// outputs take exact_dot_add_dev's cluster method in the same kernel.  A block computes an 8 x 8 tile of outputs and
// stages the 8 + 8 lines' next kWinTK entries in shared memory, so each entry is read from memory once per tile
// instead of once per output; the column sums live in shared memory (one row per thread, an odd number of 64-bit
// words apart).
// The window has p.words words: win_words(N) for lines whose spread is not known or narrow, up to win_max_words(N) where
// the host saw it (each word more costs a block 512 bytes of shared memory, two passes over a word an output, and at
// 1024 bits the widest window still leaves two blocks an SM); the cluster method costs each output some six passes over
// its terms' exponents in memory and one lane's sums in local memory (178 x 226 x 47 at 192 bits and exponents of +-185:
// 0.64 ms by clusters, 0.14 ms in wide windows; 250 x 280 x 250 at 736 bits: 61.7 and 4.0).
constexpr int kWinTM = 8, kWinTN = 8, kWinThreads = kWinTM * kWinTN, kWinTK = 8;
template <int N> __host__ __device__ constexpr int win_words() { return 2 * N + 8; }
// Row of one thread: W + 1 64-bit column sums (the sum's sign in the last), later the window (round_sum2's scratch is
// thread-local, used once per output); the row is an odd number of 64-bit words long.
__host__ __device__ constexpr int win_row_words(int words) { return 2 * ((words + 1) | 1); }
template <int N> __host__ __device__ constexpr int win_max_words() { return 2 * N + 64; }
constexpr unsigned long long kWinMaxK = 1ull << 28;          // column sums of 32-bit words stay below 2^62
template <int N> __host__ __device__ constexpr size_t win_smem_bytes(int words) {
    return (size_t)4 * ((kWinTM + kWinTN) * kWinTK * (N + 3) + kWinThreads * win_row_words(words));
}
// col (len signed 64-bit column sums) +/-= t (TW words) << (32 ws + bs), one independent add per word
template <int TW> __device__ __forceinline__ void win_add_cols(long long* col, int len, const u32 (&t)[TW], int ws, int bs, bool negative) {
#pragma unroll
    for (int q = 0; q <= TW; ++q) {
        const int k = ws + q;
        if (k >= len) break;
        const u32 v = lf_fshl(q ? t[q - 1] : 0u, q < TW ? t[q] : 0u, (u32)bs);
        col[k] += negative ? -(long long)v : (long long)v;
    }
}
struct WinParams {
    DotParams d;                    // operands, output, modes, error word
    const LineInfo* linfo; const LineInfo* rinfo;   // analysis of the M left and Nc right lines
    int spread = -1;                // the widest line's exponent spread where the host knows it, or -1
    int words = 0;                  // of a window (set by the launch)
};
template <int N> __global__ void __launch_bounds__(kWinThreads) window_dot_kernel(const WinParams wp) {
    const DotParams& p = wp.d;
    constexpr int E = N + 3;
    const int W = wp.words;
    extern __shared__ __align__(16) u32 win_park[];
    u32* sA = win_park;                                  // [kWinTK][kWinTM] entries
    u32* sB = sA + kWinTK * kWinTM * E;                  // [kWinTK][kWinTN] entries
    const int t = threadIdx.x, r = t / kWinTN, q = t % kWinTN;
    u32* row = sB + kWinTK * kWinTN * E + t * win_row_words(W);
    long long* col = reinterpret_cast<long long*>(row);  // W column sums; then the window
    const u64 r0 = (u64)blockIdx.y * kWinTM, q0 = (u64)blockIdx.x * kWinTN;
    const u64 ro = r0 + r, qo = q0 + q;                  // this thread's output (local row, column)
    const u64 i = p.row0 + ro, j = p.col0 + qo;          // its lines
    bool live = ro < p.M && qo < p.Nc && !(p.lower && j > i);
    u32* out = p.C + (ro * p.ldc + qo) * E;
    const Num<N> c = (live && p.subtract) ? load_plain<N>(out) : zero<N>();
    LineInfo li{}, ri{};
    if (live) { li = wp.linfo[ro]; ri = wp.rinfo[qo]; }
    const u32 st = (p.subtract ? c.st : 0u) | li.status | ri.status;
    const bool products = li.nonzero && ri.nonzero;
    int logk = 0;
    while ((1ull << logk) < p.K) ++logk;
    const i64 span = products ? (i64)(li.top - li.bottom) + (ri.top - ri.bottom) + 64 * N + logk : 0;
    const bool window = live && !st && products && span <= 32 * W && p.K < kWinMaxK;
    const int W1 = W + 1;                                // one more column for the sign of the signed sum
    if (window) for (int w = 0; w < W1; ++w) col[w] = 0;
    const int ebase = li.bottom + ri.bottom;
    // all threads stage the tiles (the barriers include threads without a window)
    for (u64 k0 = 0; k0 < p.K; k0 += kWinTK) {
        __syncthreads();
        // word by word over the staged entries, consecutive words to consecutive threads: entries of one k that
        // are consecutive in memory (unit line stride) make coalesced runs
        for (int x = t; x < (kWinTM + kWinTN) * kWinTK * E; x += kWinThreads) {
            const int e = x / E, w = x - e * E;
            const bool left = e < kWinTM * kWinTK;
            const int y = left ? e : e - kWinTM * kWinTK;
            const int kk = y / (left ? kWinTM : kWinTN), line = y - kk * (left ? kWinTM : kWinTN);
            const u64 lo_line = (left ? r0 : q0) + line, k = k0 + kk;
            const bool in = k < p.K && lo_line < (left ? p.M : p.Nc);
            const LineView& v = left ? p.left : p.right;
            win_park[x] = in ? __ldg(v.base + (((left ? p.row0 : p.col0) + lo_line) * v.ls + k * v.ks) * (u64)E + w) : 0u;
        }
        __syncthreads();
        if (!window) continue;
        const int kmax = p.K - k0 < (u64)kWinTK ? (int)(p.K - k0) : kWinTK;
        for (int kk = 0; kk < kmax; ++kk) {
            const u32* a = sA + (kk * kWinTM + r) * E;
            const u32* b = sB + (kk * kWinTN + q) * E;
            const int sa = (int)a[N + 1], sb = (int)b[N + 1];
            if (!sa || !sb) continue;
            u32 am[N], bm[N], pr[2 * N];
#pragma unroll
            for (int w = 0; w < N; ++w) { am[w] = a[w]; bm[w] = b[w]; }
            mant_mul<N>(am, bm, pr);
            const int off = (int)a[N] + (int)b[N] - ebase;           // 0 <= off <= spread_i + spread_j
            win_add_cols<2 * N>(col, W1, pr, off >> 5, off & 31, (sa * sb > 0) == (p.subtract != 0));
        }
    }
    if (!live) return;
    if (st) { store<N>(out, zero<N>(st)); return; }
    if (!products) { store<N>(out, p.subtract ? c : zero<N>()); return; }
    if (!window) {                                       // wide output: the cluster method, from memory
        const Num<N> v = exact_dot_add_dev<N>(p.subtract ? out : nullptr, p.subtract, p.left.base + i * p.left.ls * E, (i64)p.left.ks,
                                              p.right.base + j * p.right.ls * E, (i64)p.right.ks, p.K, p.error);
        store<N>(out, v);
        return;
    }
    // one carry pass: the columns become the two's-complement window X (in place: word w is written after column w,
    // which starts at word 2w, has been read), its sign the final carry's
    u32* X = row;
    long long carry = 0;
    for (int w = 0; w < W1; ++w) {
        const long long v = col[w] + carry;
        X[w] = (u32)v;
        carry = v >> 32;
    }
    int cmp = carry < 0 ? -1 : 0;
    if (cmp < 0) {
        u32 cy = 1;
        for (int w = 0; w < W1; ++w) { const u32 v = ~X[w] + cy; cy = cy && v == 0; X[w] = v; }
    } else {
        for (int w = 0; w < W1 && !cmp; ++w) if (X[w]) cmp = 1;
    }
    // round_sum2 adds the old entry c with its own sign (it computes RN(sign * X * 2^scale + c))
    u32 scratch[round_sum2_words<N>(win_max_words<N>() + 1)];
    store<N>(out, round_sum2<N>(X, W1, (i64)ebase - 2 * (32 * N - 1), cmp, c, scratch));
}

template <int N> __global__ void __launch_bounds__(128) reconstruct_kernel(RecParams p) {
    const u64 j = (u64)blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if (j >= p.Nc || i >= p.M) return;
    if (p.lower && j > i) return;
    constexpr u64 E = N + 3;
    u32* out = p.C + (i * p.ldc + j) * E;
    const Num<N> c = p.subtract ? load_plain<N>(out) : zero<N>();
    const LineInfo li = p.linfo[i], ri = p.rinfo[j];
    const u32 st = (p.subtract ? c.st : 0u) | li.status | ri.status;
    if (st) { store<N>(out, zero<N>(st)); return; }
    if (!li.nonzero || !ri.nonzero) { store<N>(out, p.subtract ? c : zero<N>()); return; }
    // S = sum_l t_l (M/m_l) in 64-bit column sums, F = sum_l t_l floor(2^48/m_l)
    u64 col[kResMaxQWords + 1];
    for (int w = 0; w <= p.qwords; ++w) col[w] = 0;
    u64 F = 0;
    bool any = false;
    for (int l = 0; l < p.L; ++l) {
        const u32 r = p.res[((u64)l * p.M + i) * p.Nc + j];
        any |= r != 0;
        const u32 m = p.tab->m[l];
        const u32 t = mod_barrett((u64)r * p.tab->w[l], m, p.tab->barrett[l]);
        F += (u64)t * p.tab->frac[l];
        for (int w = 0; w < p.qwords; ++w) col[w] += (u64)t * p.tab->q[l][w];
    }
    if (!any) { store<N>(out, p.subtract ? c : zero<N>()); return; }       // X == 0
    u32 S[kResMaxQWords + 2];
    u64 cy = 0;
    for (int w = 0; w <= p.qwords; ++w) { u64 v = col[w] + cy; S[w] = (u32)v; cy = v >> 32; }
    S[p.qwords + 1] = (u32)cy;
    u32 scratch[round_sum2_words<N>(kResMaxQWords + 2)];
    store<N>(out, crt_tail<N>(S, p.qwords, F, p.tab, (i64)li.bottom + ri.bottom - 2 * (32 * N - 1), p.subtract != 0, c, scratch));
}

// ---------------------------------------------------------------- 3b. CRT on the tensor cores
// S and F as one unsigned int8 GEMM.  With t_l = 256 th_l + tl_l (bytes) and q_{l,b} the bytes of
// M/m_l, byte column b of S gets P[b] = sum_l (tl_l q_{l,b} + th_l q_{l,b-1}), so that
// S = sum_b P[b] 2^(8b); F likewise from the bytes of floor(2^48/m_l).  Row o of the A operand holds
// (tl_0, th_0, tl_1, th_1, ...) for output o.  B is the constant [NB][Kp] byte matrix of those
// (shifted) bytes, uploaded once per modulus count already in the 128-byte-swizzled K-major layout
// of shared memory.  Each P[b] is below 2L * 255^2 < 2^25, so the int32 accumulators are exact.  One
// CTA computes 128 outputs per tile and is persistent over the tiles:
//   - the t_l that the residue products stored (16 bytes of one modulus at a time, its residues on a 16-byte boundary) arrive
//     while the tile before is carried; eight warps then write the rows of A, eight moduli a shared store, warps q and q + 4
//     taking alternate groups of eight moduli of the same rows.  Loaded when their tile began, 16 at a time, the t_l
//     left the warps waiting on memory (1024^2 outputs of 75 moduli: 0.284 ms, staged 0.136);
//   - one thread issues tcgen05.mma kind::i8 (u8 x u8 -> s32, M = 128, N <= 256 per instruction)
//     into TMEM;
//   - warps q and q + 4 read the same TMEM lanes and carry the byte columns of the lower and of the upper words into
//     S and F, which go to memory for crt_round_kernel; the lower words' last carry goes to a word of its own.
struct CrtParams {
    const u16* res; const ResTables* tab; const unsigned char* bimg;
    int L, qwords, NB, Kp, NS;             // B rows (multiple of 16), K bytes (multiple of 32), S byte columns
    u32 tmem_cols;
    const LineInfo* linfo; const LineInfo* rinfo;
    u32* C; u64 ldc, M, Nc;
    int subtract, lower;
    u32* error;
    const ResPlan* plan;                   // planned on the GPU: L and its operand come from the plan
    u32* sf;                               // S (qwords + 2 words), F (2 words) and the carry into word crt_split_word of
                                           // S, word-major (word w of output o at sf[w * M * Nc + o])
    u64 pitch;                             // residues of a modulus in res: M * Nc rounded up to 8
};
__host__ __device__ constexpr u64 crt_pitch(u64 outputs) { return (outputs + 7) / 8 * 8; }
__host__ __device__ constexpr size_t crt_smem_bytes(int Kp, int NB, int L) {
    return 1024 + (size_t)((Kp + 127) / 128) * (16384 + (size_t)NB * 128) + (size_t)L * 256;
}
constexpr int kCrtExtraWords = 5;          // words of an output in sf beyond qwords
// S words below this one are carried by warps 0-3, the others by warps 4-7: whole 32-column chunks, the larger part below
// (the chunk with F and the last words costs more).
__host__ __device__ __forceinline__ int crt_split_word(int qwords) {
    const int chunks = qwords / 8;
    return 8 * (chunks < 2 ? chunks : (chunks + 2) / 2);
}
__device__ __forceinline__ void mma_i8_u(u32 d_tmem, u64 a, u64 b, u32 idesc, bool accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
                 :: "r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"((u32)accumulate), "r"(0u));
}
__device__ __forceinline__ u64 crt_desc(u32 saddr) {       // K-major, SW128, SBO 1024 B, as smem_desc
    return (u64)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// byte offset of (row, k) in a [rows][128-byte K block] tile, 128-byte swizzle (the TMA SW128 image)
__host__ __device__ __forceinline__ u32 sw128_offset(u32 row, u32 k) {
    return (row >> 3) * 1024u + (row & 7u) * 128u + ((((k >> 4) ^ row) & 7u) << 4) + (k & 15u);
}
template <int N> __global__ void __launch_bounds__(kCrtThreads, 2) crt_mma_kernel(const CrtParams pin) {
    CrtParams p = pin;
    if (pin.plan) {
        const ResPlan& r = *pin.plan;
        if (r.mode != 1) return;
        p.tab = static_cast<const ResTables*>(r.tab); p.bimg = r.crt_bimg; p.L = r.L; p.qwords = r.qwords;
        p.NB = r.NB; p.Kp = r.Kp; p.NS = r.NS; p.tmem_cols = r.tmem_cols;
    }
    extern __shared__ __align__(1024) unsigned char crt_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)crt_raw + 1023) & ~(uintptr_t)1023);
    const int kblocks = p.Kp / 128 + (p.Kp % 128 ? 1 : 0);
    unsigned char* sA = smem;                                  // kblocks x [128 rows][128 B]
    unsigned char* sB = smem + kblocks * 16384;                // kblocks x [NB rows][128 B]
    u16* sR = reinterpret_cast<u16*>(sB + kblocks * p.NB * 128);     // [L][128 outputs]
    __shared__ __align__(8) u64 done;
    __shared__ u32 tmem_slot;
    const int warp = threadIdx.x >> 5;
    const u64 bbytes = (u64)kblocks * p.NB * 128;
    for (u64 o = (u64)threadIdx.x * 16; o < bbytes; o += (u64)blockDim.x * 16)
        *reinterpret_cast<uint4*>(sB + o) = *reinterpret_cast<const uint4*>(p.bimg + o);
    for (u32 o = threadIdx.x * 16u; o < (u32)kblocks * 16384u; o += blockDim.x * 16u)      // bytes beyond 2 L stay zero
        *reinterpret_cast<uint4*>(sA + o) = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_slot)), "r"(p.tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const u32 tmem = tmem_slot;
    const int N1 = p.NB < 256 ? p.NB : 256, N2 = p.NB - N1;
    const u32 id1 = (2u << 4) | ((u32)(N1 >> 3) << 17) | ((u32)(128 >> 4) << 24);
    const u32 id2 = (2u << 4) | ((u32)(N2 >> 3) << 17) | ((u32)(128 >> 4) << 24);
    const u64 outputs = p.M * p.Nc, tiles = (outputs + 127) / 128;
    // Warps q and q + 4 share the rows of A and the TMEM lanes 32 q ..
    const int half = warp >> 2;
    const u32 row = (u32)((warp & 3) * 32 + (threadIdx.x & 31)), lane_base = (u32)((warp & 3) * 32) << 16;
    auto following = [&](u64 t) {                              // the next tile from t on that is not wholly above the diagonal
        while (p.lower && t < tiles) {
            const u64 o0 = t * 128, o1 = (o0 + 127 < outputs ? o0 + 127 : outputs - 1);
            if (o0 / p.Nc != o1 / p.Nc || o0 % p.Nc <= o0 / p.Nc) break;
            t += gridDim.x;
        }
        return t;
    };
    auto stage = [&](u64 t) {
        if (t < tiles)
            for (int x = threadIdx.x; x < p.L * 16; x += kCrtThreads) {
                const u64 at = t * 128 + 8 * (x & 15);
                if (at < outputs) cp_async16(sR + (x >> 4) * 128 + 8 * (x & 15), p.res + (u64)(x >> 4) * p.pitch + at);
            }
        cp_async_commit();
    };
    u32 phase = 0;
    u64 tile = following(blockIdx.x);
    stage(tile);
    cp_async_wait<0>();
    __syncthreads();
    while (tile < tiles) {
        const u64 o = tile * 128 + row;
        const bool valid = o < outputs;
        for (int l0 = half * 8; l0 < p.L; l0 += 16) {           // row of A: t_l as two bytes
            u32 t[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) t[q] = l0 + q < p.L ? sR[(l0 + q) * 128 + row] : 0u;
            *reinterpret_cast<uint4*>(sA + (l0 >> 6) * 16384u + sw128_offset(row, 2u * (l0 & 63))) =
                make_uint4(t[0] | (t[1] << 16), t[2] | (t[3] << 16), t[4] | (t[5] << 16), t[6] | (t[7] << 16));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic writes -> tensor core reads
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            for (int ks = 0; ks < p.Kp / 32; ++ks) {
                const int kb = ks >> 2;
                const u64 koff = (u64)((ks & 3) * 32) >> 4;
                const u64 ad = crt_desc(smem_u32(sA + kb * 16384)) + koff;
                const u32 bbase = smem_u32(sB + (u64)kb * p.NB * 128);
                mma_i8_u(tmem, ad, crt_desc(bbase) + koff, id1, ks > 0);
                if (N2) mma_i8_u(tmem + 256, ad, crt_desc(bbase + 256 * 128) + koff, id2, ks > 0);
            }
            mma_commit(&done);
        }
        const u64 next = following(tile + gridDim.x);
        stage(next);                                            // every thread has read sR
        const bool fine = __syncthreads_and(mbar_wait(&done, phase, p.error));
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (!fine) break;
        // word w of S is the sum of its four byte columns and the carry from below (every thread of the warp reads its lane:
        // .sync.aligned); each column is below 2^25, so a word's sum stays below 2^50
        const int split = crt_split_word(p.qwords), chunks = p.qwords / 8;     // 8-word chunks wholly inside S
        u32* dst = p.sf + o;
        u64 acc = 0;
        for (int ch = half ? split / 8 : 0; ch < (half ? chunks : split / 8); ++ch) {
            u32 P[32];
            tmem_ld32(tmem + lane_base + (u32)ch * 32u, P);
            asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                acc += ((u64)P[4 * w + 1] << 8) + P[4 * w] + (((u64)P[4 * w + 3] << 24) + ((u64)P[4 * w + 2] << 16));
                if (valid) dst[(u64)(8 * ch + w) * outputs] = (u32)acc;
                acc >>= 32;
            }
        }
        if (half == 0) {
            if (valid) dst[(u64)(p.qwords + 4) * outputs] = (u32)acc;
        } else {
            int sw = 8 * chunks;
            u64 F = 0;
            for (int c0 = 4 * sw; c0 < p.NB; c0 += 32) {
                u32 P[32];
                tmem_ld32(tmem + lane_base + (u32)c0, P);
                asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const int col = c0 + c;
                    if (col < p.NS) {
                        acc += (u64)P[c] << (8 * (col & 3));
                        if ((col & 3) == 3) { if (valid) dst[(u64)sw * outputs] = (u32)acc; ++sw; acc >>= 32; }
                    } else if (col < p.NS + 6) {
                        F += (u64)P[c] << (8 * (col - p.NS));
                    }
                }
            }
            if (valid) {
                while (sw < p.qwords + 2) { dst[(u64)sw * outputs] = (u32)acc; ++sw; acc >>= 32; }
                dst[(u64)(p.qwords + 2) * outputs] = (u32)F;
                dst[(u64)(p.qwords + 3) * outputs] = (u32)(F >> 32);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        cp_async_wait<0>();
        __syncthreads();                                        // TMEM and A are free for the next tile, whose residues are here
        tile = next;
    }
    cp_async_wait<0>();
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(p.tmem_cols));
}

// ---------------------------------------------------------------- 1b. digit planes on the tensor cores
// X mod m_l for all L moduli as two unsigned int8 GEMMs: with x_b the bytes of X (4 xwords of them) and
// 2^(8b) mod m_l = 256 th + tl, P0 = [tl] x [x bytes] and P1 = [th] x [x bytes] give
// X == P0 + 256 P1 (mod m_l), each P below 160 * 255^2 < 2^24.  The moduli are the rows (TMEM lanes) and 128 padded
// entries (line, k) in plane order the columns: a thread then has its modulus in registers and 32 consecutive entries
// of one plane, whose digits it packs and stores as 32 bytes.  With entries as rows every digit was a store of
// its own byte and every residue two shared loads of its modulus (0.21 ms for 1024^2 512-bit entries).  Up to 64 (32)
// moduli the table's rows repeat two (four) times down the lanes, and each copy takes its share of the columns.
// B is the constant byte table, uploaded per (L, xwords) as its swizzled shared-memory image.  The epilogue reduces,
// balances, negates for negative entries and splits each residue into the two int8 digits.
struct DigitMmaParams {
    LineView v; u64 lines, K, Kp, rows_pad; int L; int xwords;
    const LineInfo* info; const ResTables* tab;
    const unsigned char* bimg; int KB;
    signed char* d1; signed char* d0;
    u32* error;
    const ResPlan* plan;                   // planned on the GPU: L and its operand come from the plan
};
constexpr int kDigitCols = 128;                                // entries per tile
__host__ __device__ constexpr int digit_row_tiles(int L) { return L > 128 ? 2 : 1; }
__host__ __device__ constexpr int digit_copies(int L) { return L <= 32 ? 4 : L <= 64 ? 2 : 1; }
__host__ __device__ constexpr u32 digit_tmem_cols(int L) { return 2u * kDigitCols * digit_row_tiles(L); }
__host__ __device__ constexpr size_t digit_smem_bytes(int row_tiles, int KB) {
    return 1024 + (size_t)(2 * row_tiles + 1) * ((KB + 127) / 128) * 16384;
}
__device__ __forceinline__ void store_bytes32(signed char* p, const u32 (&w)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" :: "l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
                 "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
}
template <int N> __global__ void __launch_bounds__(kDigitThreads, 2) digits_mma_kernel(const DigitMmaParams pin) {
    DigitMmaParams p = pin;
    if (pin.plan) {
        const ResPlan& r = *pin.plan;
        if (r.mode != 1) return;
        p.tab = static_cast<const ResTables*>(r.tab); p.bimg = r.dig_bimg; p.L = r.L;
    }
    extern __shared__ __align__(1024) unsigned char dig_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)dig_raw + 1023) & ~(uintptr_t)1023);
    const int kblocks = p.KB / 128 + (p.KB % 128 ? 1 : 0), row_tiles = digit_row_tiles(p.L);
    unsigned char* sX = smem;                                  // kblocks x [128 entries][128 B]
    unsigned char* sT = smem + kblocks * 16384;                // row tiles x (tl, th) x kblocks x [128 moduli][128 B]
    __shared__ __align__(8) u64 done;
    __shared__ u32 tmem_slot;
    __shared__ u32 s_neg[kDigitCols / 32];                     // negative entries of the tile, one bit each
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const u32 tbytes = 2u * row_tiles * kblocks * 16384u;
    for (u32 o = threadIdx.x * 16u; o < tbytes; o += blockDim.x * 16u)
        *reinterpret_cast<uint4*>(sT + o) = *reinterpret_cast<const uint4*>(p.bimg + o);
    if (threadIdx.x == 0) {
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const u32 tmem_cols = digit_tmem_cols(p.L);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&tmem_slot)), "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const u32 tmem = tmem_slot;
    constexpr u32 idesc = (2u << 4) | ((u32)(kDigitCols >> 3) << 17) | ((u32)(128 >> 4) << 24);
    const u64 plane = p.rows_pad * p.Kp, tiles = plane / kDigitCols;      // rows_pad is a multiple of 128
    const int q = warp & 3, half = warp >> 2;                  // warps q and q + 4 share TMEM lanes 32 q ..
    const u32 lane_base = (u32)(q * 32) << 16;
    const int copies = digit_copies(p.L), rows = 128 / copies, span = kDigitCols / copies;
    const int group = (q * 32) / rows;                         // the copy of the table this warp's lanes belong to
    // The first four warps stage the entries of a tile (one each a thread); the entry of the next tile is
    // loaded before the current tile's epilogue so that its latency hides behind the digit work.
    const u32 entry = (u32)(q * 32 + lane);
    Num<N> a = zero<N>();
    u64 aline = 0;
    auto fetch = [&](u64 t) {
        a = zero<N>();
        const u64 e = t * kDigitCols + entry;
        aline = e / p.Kp;
        const u64 k = e % p.Kp;
        if (t < tiles && k < p.K && aline < p.lines) a = load<N>(p.v.base + (aline * p.v.ls + k * p.v.ks) * (u64)(N + 3));
    };
    if (half == 0) fetch(blockIdx.x);
    u32 phase = 0;
    for (u64 tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        if (half == 0) {
            // column of B: the bytes of X = |entry| 2^(e - bottom) (0 <= shift <= G), zero beyond its words
#pragma unroll
            for (int c = 0; c < 16; ++c) {                      // up to 2 K blocks of 8 chunks
                if (c >= kblocks * 8) break;
                *reinterpret_cast<uint4*>(sX + (c >> 3) * 16384u + sw128_offset(entry, (u32)(c & 7) * 16u)) = make_uint4(0, 0, 0, 0);
            }
            bool negative = false;
            if (!a.st && a.s) {
                negative = a.s < 0;
                const int sh = a.e - p.info[aline].bottom;
                const int ws = sh >> 5, bs = sh & 31;
#pragma unroll
                for (int i = 0; i <= N; ++i) {
                    u32 v = i < N ? a.m[i] << bs : 0u;
                    if (bs && i > 0) v |= a.m[i - 1] >> (32 - bs);
                    const u32 byte = (u32)(i + ws) * 4u;      // word i + ws < xwords <= KB / 4
                    *reinterpret_cast<u32*>(sX + (byte >> 7) * 16384u + sw128_offset(entry, byte & 127u)) = v;
                }
            }
            const u32 neg = __ballot_sync(0xffffffffu, negative);
            if (lane == 0) s_neg[q] = neg;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;");
            for (int g = 0; g < 2 * row_tiles; ++g)
                for (int ks = 0; ks < p.KB / 32; ++ks) {
                    const u64 koff = (u64)((ks & 3) * 32) >> 4;
                    mma_i8_u(tmem + (u32)(g * kDigitCols), crt_desc(smem_u32(sT + (g * kblocks + (ks >> 2)) * 16384)) + koff,
                             crt_desc(smem_u32(sX + (ks >> 2) * 16384)) + koff, idesc, ks > 0);
                }
            mma_commit(&done);
        }
        const bool fine = __syncthreads_and(mbar_wait(&done, phase, p.error));
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (!fine) break;
        if (half == 0) fetch(tile + gridDim.x);                // sX is rewritten only after the barrier below
        for (int t = 0; t < row_tiles; ++t) {
            const int l = t * 128 + (int)entry - group * rows;
            const bool live = l < p.L;
            const u32 m = live ? p.tab->m[l] : 3u, rr = live ? (u32)(p.tab->barrett[l] >> 32) : 0u, h = m >> 1;
            const u64 at = (u64)(live ? l : 0) * plane + tile * kDigitCols;
            for (int ch = half; ch < span / 32; ch += 2) {
                const u32 c0 = (u32)(group * span + ch * 32);
                u32 P0[32], P1[32];
                tmem_ld32(tmem + lane_base + (u32)(2 * t * kDigitCols) + c0, P0);
                tmem_ld32(tmem + lane_base + (u32)((2 * t + 1) * kDigitCols) + c0, P1);
                asm volatile("tcgen05.wait::ld.sync.aligned;");
                if (live) {
                    const u32 neg = s_neg[c0 >> 5];
                    u32 w0[8], w1[8];
#pragma unroll
                    for (int g = 0; g < 8; ++g) {
                        int r[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const int c = 4 * g + b;
                            const u32 x = P0[c] + (P1[c] << 8);     // below 2^32: one Barrett step leaves [0, 2m)
                            u32 u = x - __umulhi(x, rr) * m;
                            u = min(u, u - m);
                            const int v = (int)u - (u > h ? (int)m : 0);       // balanced (m is odd): |v| <= 32639
                            r[b] = (neg >> c) & 1u ? -v : v;
                        }
                        // low digit: the byte of r; high digit: (r - low) >> 8 = byte 1 of r + 128
                        w0[g] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
                        w1[g] = __byte_perm(__byte_perm(r[0] + 128, r[1] + 128, 0x0051), __byte_perm(r[2] + 128, r[3] + 128, 0x0051), 0x5410);
                    }
                    store_bytes32(p.d1 + at + c0, w1);
                    store_bytes32(p.d0 + at + c0, w0);
                }
                __syncwarp();
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncthreads();
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(tmem_cols));
}

// The rounding half of the CRT: one thread per output, RN(c - X 2^scale) or RN(X 2^scale) with X = S - round(F) M.
// One pass over the words subtracts q M and adds the old entry in place (T = X - c at X's scale, negated when it is rounded),
// leaving T's words in shared memory (an odd stride: the lanes of a warp touch 32 banks); the rounding reads the N + 2 words
// under T's top and learns the sticky bit from the lowest nonzero word, which the pass recorded.  That needs the old
// entry's bits to lie inside X's words; an entry that reaches outside takes the two-window form (crt_tail, in thread-
// local memory).  The two-window form for every output took 0.32 ms for 1024^2 outputs at 512 bits, four passes over
// 82-word windows.
constexpr int kCrtRoundThreads = 128;
__host__ __device__ constexpr int crt_round_words(int qwords) { return (qwords + 2) | 1; }
template <int N> __device__ __noinline__ Num<N> crt_tail_call(const u32* S, int qwords, u64 F, const ResTables* tab, i64 scale,
                                                              bool subtract, const Num<N> c) {
    u32 X[kResMaxQWords + 2], scratch[round_sum2_words<N>(kResMaxQWords + 2)];
    for (int w = 0; w < qwords + 2; ++w) X[w] = S[w];
    return crt_tail<N>(X, qwords, F, tab, scale, subtract, c, scratch);
}
// One output: leaves its entry in T and returns whether there is one to write.  The words of S are loaded eight ahead of the pass
// (one a step left it waiting on memory: 1024^2 outputs at 512 bits took 0.217 ms, with this and the coalesced writes 0.146).
template <int N> __device__ __forceinline__ bool crt_round_one(const CrtParams& p, const u32* s_M, u64 o, u64 i, u64 j, u32* T, const u32* out) {
    const int xw = p.qwords + 2;
    const u64 outputs = p.M * p.Nc;
    const LineInfo li = p.linfo[i], ri = p.rinfo[j];
    int ce = 0, cs = 0;
    u32 cst = 0;
    if (p.subtract) { ce = (int)out[N]; cs = (int)out[N + 1]; cst = out[N + 2]; }
    const u32 st = cst | li.status | ri.status;
    if (st) { store<N>(T, zero<N>(st)); return true; }
    if (!li.nonzero || !ri.nonzero) { store<N>(T, zero<N>()); return !p.subtract; }      // C stays
    const u32* sf = p.sf + o;
    const u64 F = (u64)sf[(u64)(p.qwords + 2) * outputs] | ((u64)sf[(u64)(p.qwords + 3) * outputs] << 32);
    const int split = crt_split_word(p.qwords);
    const u32 up = sf[(u64)(p.qwords + 4) * outputs];            // carry of the lower words' columns
    const i64 scale = (i64)li.bottom + ri.bottom - 2 * (32 * N - 1);
    const i64 off = (i64)ce - (32 * N - 1) - scale;              // bit of T that the old entry's lowest bit falls on
    if (cs && (off < 0 || off + 32 * N > 32 * (i64)xw - 2)) {
        u64 cy = 0;
        for (int w = 0; w < xw; ++w) {
            const u64 v = (u64)sf[(u64)w * outputs] + (w == split ? up : 0u) + cy;
            T[w] = (u32)v; cy = v >> 32;
        }
        store<N>(T, crt_tail_call<N>(T, p.qwords, F, p.tab, scale, true, load_plain<N>(out)));
        return true;
    }
    // T = S - q M - c (two's complement); without an old entry T = X
    const u32 q = (u32)((F + (1ull << 47)) >> 48);              // round(F) <= L: X = S - q M
    const int ws = cs ? (int)(off >> 5) : xw, bs = cs ? (int)(off & 31) : 0;
    const u32 mask = cs > 0 ? 0xffffffffu : 0u;                   // c > 0 is subtracted
    u64 cy = 0, qm = 0, ca = mask & 1u;
    u32 prev = 0, low = 0xffffffffu;                              // lowest nonzero word of T
    int borrow = 0;
    for (int w0 = 0; w0 < xw; w0 += 8) {
        u32 sw[8], cw[8];
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            sw[x] = w0 + x < xw ? __ldg(sf + (u64)(w0 + x) * outputs) : 0u;
            cw[x] = (u32)(w0 + x - ws) < (u32)N ? out[w0 + x - ws] : 0u;
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int w = w0 + x;
            if (w >= xw) break;
            const u64 sv = (u64)sw[x] + (w == split ? up : 0u) + cy;
            cy = sv >> 32;
            qm += (u64)s_M[w] * q;
            const i64 d = (i64)(sv & 0xffffffffull) - (i64)(qm & 0xffffffffull) - borrow;
            qm >>= 32;
            borrow = d < 0;
            const u32 add = __funnelshift_l(prev, cw[x], bs);     // zero outside words [ws, ws + N]
            prev = cw[x];
            const u64 v = (u64)(u32)d + (add ^ mask) + ca;
            ca = v >> 32;
            T[w] = (u32)v;
            if ((u32)v && low == 0xffffffffu) low = (u32)w;
        }
    }
    if (low == 0xffffffffu) { store<N>(T, zero<N>()); return true; }
    const bool neg = T[xw - 1] >> 31;
    auto mag = [&](int w) -> u32 {                                // word w of |T|
        if (w < (int)low) return 0u;
        return neg ? (w == (int)low ? 0u - T[w] : ~T[w]) : T[w];
    };
    int t = xw - 1;
    while (!mag(t)) --t;
    u32 hi = mag(t);
    const int lz = __clz(hi);
    u32 m[N];
#pragma unroll
    for (int x = N - 1; x >= 0; --x) {
        const u32 below = mag(t - N + x);
        m[x] = __funnelshift_l(below, hi, lz);
        hi = below;
    }
    const u32 next = mag(t - N - 1), g = __funnelshift_l(next, hi, lz);
    const bool sticky = (g & 0x7fffffffu) || (next << lz) || (int)low < t - N - 1;
    // subtract: the result is c - X = -T
    store<N>(T, finish<N>(m, scale + 32 * (i64)t + 31 - lz, neg != (p.subtract != 0) ? -1 : 1, (g >> 31) && (sticky || (m[0] & 1u)), 0));
    return true;
}
template <int N> __global__ void __launch_bounds__(kCrtRoundThreads) crt_round_kernel(const CrtParams pin) {
    CrtParams p = pin;
    if (pin.plan) {
        if (pin.plan->mode != 1) return;
        p.tab = static_cast<const ResTables*>(pin.plan->tab); p.qwords = pin.plan->qwords;
    }
    extern __shared__ u32 crt_round_park[];
    __shared__ u32 s_M[kResMaxQWords + 2];
    const int xw = p.qwords + 2;
    for (int w = threadIdx.x; w < xw; w += kCrtRoundThreads) s_M[w] = w <= p.qwords ? p.tab->M[w] : 0u;
    __syncthreads();
    const u64 outputs = p.M * p.Nc, o = (u64)blockIdx.x * kCrtRoundThreads + threadIdx.x;
    const u64 i = o / p.Nc, j = o % p.Nc;
    constexpr u64 E = N + 3;
    u32* out = p.C + (i * p.ldc + j) * E;
    u32* T = crt_round_park + threadIdx.x * crt_round_words(p.qwords);
    const bool put = o < outputs && !(p.lower && j > i) && crt_round_one<N>(p, s_M, o, i, j, T, out);
    // a warp writes its 32 entries word by word, neighbouring words to neighbouring lanes
    const u32 live = __ballot_sync(0xffffffffu, put);
    if (!live) return;                                           // the whole warp: above the diagonal, or beyond the outputs
    __syncwarp();                                                // every lane's entry is in T: a vote orders no memory
    const u32 lane = threadIdx.x & 31;
    const u32* rows = T - lane * crt_round_words(p.qwords);
    for (u32 w = lane; w < 32 * E; w += 32) {
        const u32 r = w / (u32)E, x = w - r * (u32)E;
        u32* to = reinterpret_cast<u32*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(out), r));
        if ((live >> r) & 1u) to[x] = rows[r * crt_round_words(p.qwords) + x];
    }
}

typedef void (*DigitFn)(const DigitParams&, cudaStream_t);
typedef void (*RecFn)(const RecParams&, cudaStream_t);
typedef void (*CrtFn)(const CrtParams&, unsigned grid, size_t smem, cudaStream_t);
typedef void (*DigitMmaFn)(const DigitMmaParams&, unsigned grid, size_t smem, cudaStream_t);
typedef void (*WindowDotFn)(WinParams, cudaStream_t);
struct ResidueKernels { DigitFn digits; RecFn rec; CrtFn crt; DigitMmaFn digits_mma; WindowDotFn window_dot; };
const ResidueKernels* residue_kernels(int limbs);

template <int N> void digits_launch(const DigitParams& p, cudaStream_t s) {
    if (!p.rows_pad || !p.Kp) return;
    dim3 grid((unsigned)((p.Kp + 127) / 128), (unsigned)p.rows_pad);
    digits_kernel<N><<<grid, 128, 0, s>>>(p);
}
template <int N> void crt_launch(const CrtParams& p, unsigned grid, size_t smem, cudaStream_t s) {
    if (!p.M || !p.Nc) return;
    cudaFuncSetAttribute(crt_mma_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    crt_mma_kernel<N><<<grid, kCrtThreads, smem, s>>>(p);
    // the planned form learns qwords on the GPU: size the words of T for the largest table
    const size_t rsmem = (size_t)kCrtRoundThreads * crt_round_words(p.plan ? kResMaxQWords : p.qwords) * 4;
    if (rsmem > 48 * 1024) cudaFuncSetAttribute(crt_round_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem);
    crt_round_kernel<N><<<(unsigned)((p.M * p.Nc + kCrtRoundThreads - 1) / kCrtRoundThreads), kCrtRoundThreads, rsmem, s>>>(p);
}
template <int N> void digits_mma_launch(const DigitMmaParams& p, unsigned grid, size_t smem, cudaStream_t s) {
    if (!p.rows_pad || !p.Kp) return;
    cudaFuncSetAttribute(digits_mma_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    digits_mma_kernel<N><<<grid, kDigitThreads, smem, s>>>(p);
}
template <int N> void window_dot_launch(WinParams p, cudaStream_t s) {
    if (!p.d.M || !p.d.Nc) return;
    // a window for every output where the widest pair of lines fits one
    int logk = 0;
    while ((1ull << logk) < p.d.K) ++logk;
    const i64 need = p.spread < 0 ? 0 : (2 * (i64)p.spread + 64 * N + logk + 31) / 32;
    p.words = need <= win_words<N>() || need > win_max_words<N>() ? win_words<N>() : (int)need;
    const size_t smem = win_smem_bytes<N>(p.words);
    if (smem > 48 * 1024) cudaFuncSetAttribute(window_dot_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dim3 grid((unsigned)((p.d.Nc + kWinTN - 1) / kWinTN), (unsigned)((p.d.M + kWinTM - 1) / kWinTM));
    window_dot_kernel<N><<<grid, kWinThreads, smem, s>>>(p);
}
template <int N> void rec_launch(const RecParams& p, cudaStream_t s) {
    if (!p.M || !p.Nc) return;
    dim3 grid((unsigned)((p.Nc + 127) / 128), (unsigned)p.M);
    reconstruct_kernel<N><<<grid, 128, 0, s>>>(p);
}

}  // namespace lfd

#define LF_RESIDUE_INSTANTIATE(N)                                                                  \
    namespace lfd {                                                                                \
    extern const ResidueKernels residue_kernels_##N; const ResidueKernels residue_kernels_##N = {digits_launch<N>, rec_launch<N>, crt_launch<N>, digits_mma_launch<N>, window_dot_launch<N>}; \
    }
