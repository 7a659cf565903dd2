// fp32 Linears of prompts on the tensor cores (tcgen05): y = x W^T with every fp32 operand as three bf16 parts.
//
// An fp32 number is hi + mid / 2^8 + lo / 2^16 exactly: hi the nearest bf16, mid the nearest to 2^8 times what is left, lo 2^8 times the rest of that (at
// most 8 significant bits; the powers of two keep the parts of small numbers above bf16's smallest, down to 2^-126; of fp32's subnormal numbers hi has fewer bits, and a
// product of one is right to 2^-20).  x w is the sum of nine part
// products, of which the six largest are formed; the other three are below 2^-26 of x w, of either sign.  Products of bf16 numbers are exact in
// the tensor core; what it loses is in its running sum, so (a) the small products of a k-block are summed first, at their own scale -- the
// accumulator is divided by 2^8 where the next larger ones start -- and the four hi hi instructions last, and (b) the accumulator starts anew for
// every 64 columns of k and is added to fp32 registers with ordinary rounded additions.
// Error against float64 in units of 2^-24 (2-norm; operands normal, then in 1 .. 2), here and by a chain of FMAs: K = 8 0.78 / 0.92, 0.96 / 0.79;
// 16 0.81 / 1.28, 1.00 / 1.04; 64 1.3 / 2.4, 1.0 / 2.0; 2048 1.7 / 13.5, 1.2 / 11.4 (the same with operands of 2^-118).  Below FT_MIN_K columns the chain is the
// more exact one for operands of one sign and keeps the job (linear_tiled_fma).  With truncated parts and without the scales, as this began: 1.6 at any K,
// 7.8 for x = w = 1 + 2^-7 - 2^-23 and 300 at 2^-118.
//
// What bounds it: the MMAs, about 24 x (64 + w / 4) clocks a k-block of 64 for w tokens, and the power cap: 804 x 16384 x 2048 runs at 1.34 to 1.44 PFLOP/s of part products (225 us
// stored, 236 with the gated unit, where tiles of 128 x 128 with both operands split in every CTA took 480); few tokens by the way of a k-block through two stages
// (20 x 16384 x 2048: 51 us, 68 before, and 20 of them memory).
// A pair of CTAs (cta_group::2) has 256 features x up to 224 tokens: the weights are the MMA's rows, because its columns can be any multiple of 16 and its
// rows cannot.  x is split ahead, once, by a kernel of its own (f32_parts_kernel: 10 bytes an element) and comes in by TMA; W is split where it is used, each CTA its
// own 128 rows, since its parts written out would cost 10 bytes an element of a matrix that is several times as large.
//
// Warps: 0-7 load fp32 weights from global memory (one k-block ahead, in registers), split them and write the three part tiles (128B-swizzled, K-major) of a stage; 8-15 add
// the sums of each k-block to their registers; 16 TMA (parts of x); 17 issues the MMAs for both CTAs.  Splitting and adding are warps of their own because each is a
// chain of latencies of 1500 to 2500 clocks a k-block (a round trip to tensor memory alone is 300), and one warp that did both took 4000 of them for MMAs of 2800.
// Two stages, two accumulators.  Clusters are persistent; a last round that is not full is cut along k, and f32_combine_kernel adds the parts in the order of k, so nobody waits for another
// cluster and the result is the same every time.
//
// An infinity or a NaN in the operands of a tile, or a number from 2^120 on (256 x is formed): its outputs are computed again with FMAs (ft_fma_rows; one NaN among 804 x 16384 x 2048: 2046 us).
//
// The parts of x and the slots are room that the caller brings; without it, and where x is the larger operand, hybrid_linear_f32_cta.cuh runs.
#pragma once
#include <cuda.h>

#include "hybrid_linear.cuh"

namespace mbh {

constexpr int FT_MIN_K = 16;  // shorter rows: linear_tiled_fma
constexpr int FT_BN = 128, FT_BK = 64;  // features of a CTA (a pair: 256), columns of a k-block
constexpr int FT_MAX_W = 224, FT_CHUNKS = FT_MAX_W / 32;  // tokens of a tile at most; blocks of 16 of them a warp adds up
constexpr int FT_SPLIT_WARPS = 8, FT_SUM_WARPS = 8, FT_THREADS = 32 * (FT_SPLIT_WARPS + FT_SUM_WARPS + 4);
// Registers a thread: 20 warps are launched with 96 each; the sums get 152 of them, the splitting warps 72 and the last four 32 (2 x 152 + 2 x 72 + 32 = 5 x 96).
constexpr int FT_REGS = 96, FT_SPLIT_REGS = 72, FT_SUM_REGS = 152, FT_REST_REGS = 32;
static_assert(2 * FT_SPLIT_REGS + 2 * FT_SUM_REGS + FT_REST_REGS <= 5 * FT_REGS, "a split of more than was launched with waits forever");
constexpr int FT_TILE = FT_BN * FT_BK * 2, FT_STAGE = 3 * FT_TILE + 3 * (FT_MAX_W / 2) * FT_BK * 2;  // a part of W: 128 rows of 128 bytes; a stage: three of W, three of half the tile's tokens
constexpr int FT_SMEM = 2 * FT_STAGE + 1024;
constexpr int FT_REDO_WORDS = 512;  // a bit per tile of a cluster

__device__ __forceinline__ uint32_t ft_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ft_bar_init(uint64_t* b, uint32_t count) { asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(ft_smem(b)), "r"(count) : "memory"); }
__device__ __forceinline__ void ft_bar_arrive(uint32_t b) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(b) : "memory"); }  // b: ft_first_cta
__device__ __forceinline__ void ft_bar_expect(uint64_t* b, uint32_t bytes) { asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(ft_smem(b)), "r"(bytes) : "memory"); }
// Waits a bounded time.  false: gave up: the caller marks its CTA (`lost`), whose sums from then on are NaN, goes on to the end without waiting again, and says nothing more that
// would let the other CTA of the pair take what is not there (no arrival, no copy, no commit): that one gives up too.
__device__ __forceinline__ bool ft_bar_wait(uint64_t* b, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(ft_smem(b)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// K-major, 128B-swizzled tile of 128-byte rows: 8-row groups 1024 B apart, version 1, layout SWIZZLE_128B.  The upper word of a descriptor is this, the lower the tile's address
// in units of 16 bytes (and 1 << 16).
constexpr uint32_t FT_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t ft_desc_lo(uint32_t addr) { return ((addr & 0x3ffff) >> 4) | (1u << 16); }
constexpr uint32_t FT_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * FT_BN >> 4) << 24);  // bf16 x bf16 -> fp32, 256 rows; + the width / 8 at bit 17
// D = A B (ACC false), A B + D / 2^DOWN, by the pair.  a, b: lower words of the descriptors (one addition each: the thread that issues is what bounds narrow tiles)
template <bool ACC, int DOWN>
__device__ __forceinline__ void ft_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t idesc) {
    if constexpr (DOWN > 0)
        asm volatile("{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %4};\nmov.b64 db, {%2, %4};\nsetp.ne.b32 p, 1, 0;\n"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p, %5;\n}\n" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "n"(FT_DESC_HI), "n"(DOWN)
                     : "memory");
    else
        asm volatile("{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %4};\nmov.b64 db, {%2, %4};\nsetp.ne.b32 p, %5, 0;\n"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(d), "r"(a), "r"(b), "r"(idesc), "n"(FT_DESC_HI), "n"(ACC ? 1 : 0)
                     : "memory");
}
__device__ __forceinline__ bool ft_elect() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0u;
}
// on the barrier at this offset in both CTAs, once the MMAs issued so far have completed
__device__ __forceinline__ void ft_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(ft_smem(b)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void ft_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_ld16(uint32_t addr, float (&v)[16]) {  // (ft_wait_ld before the numbers are used)
    uint32_t* u = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]),
                   "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(addr));
}
template <int R>
__device__ __forceinline__ void ft_more_regs() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R>
__device__ __forceinline__ void ft_fewer_regs() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }
__device__ __forceinline__ void ft_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// two numbers to the nearest bf16, and back
__device__ __forceinline__ uint32_t ft_pack(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
// pairs of fp32 numbers in a 64-bit register
__device__ __forceinline__ uint64_t ft_two(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float ft_first(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float ft_second(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t ft_unpack(uint32_t u) { return ft_two(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ uint64_t ft_mul2(uint64_t v, float f) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(v), "l"(ft_two(f, f)));
    return r;
}
__device__ __forceinline__ uint64_t ft_fma2(uint64_t v, float f, uint64_t add) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(v), "l"(ft_two(f, f)), "l"(add));
    return r;
}
// four numbers as three times four bf16 parts; every subtraction is exact; 256 x first, so that both steps of a part are one instruction for two numbers
__device__ __forceinline__ void ft_split4(const float4& v, uint2 (&part)[3]) {
    const float f[4] = {v.x, v.y, v.z, v.w};
    uint32_t p[3][2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const uint64_t v8 = ft_mul2(ft_two(f[2 * e], f[2 * e + 1]), 256.f);
        const uint32_t h = ft_pack(f[2 * e], f[2 * e + 1]);
        const uint64_t r1 = ft_fma2(ft_unpack(h), -256.f, v8);
        const uint32_t m = ft_pack(ft_first(r1), ft_second(r1));
        const uint64_t r2 = ft_fma2(ft_unpack(m), -256.f, ft_mul2(r1, 256.f));
        p[0][e] = h;
        p[1][e] = m;
        p[2][e] = __byte_perm(__float_as_uint(ft_first(r2)), __float_as_uint(ft_second(r2)), 0x7632);  // at most 8 significant bits are left: exact
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) part[q] = make_uint2(p[q][0], p[q][1]);
}
// shared::cluster address of `p`'s offset in the cluster's first CTA
__device__ __forceinline__ uint32_t ft_first_cta(const void* p) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(ft_smem(p)), "r"(0u));
    return r;
}
__device__ __forceinline__ void ft_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Up to 128 rows of x times a CTA's features with FMAs in the order of k, through shared memory (the stages: the parts are not needed any more).  A thread takes four
// columns of every 16th row.  About the time the whole tile takes with FMAs, once per tile that holds an infinity or a NaN.  lost: copies may still be on their way to
// the stages; NaN in place of the sums.
template <bool VEC, int THREADS>
__device__ __noinline__ void ft_fma_rows(const LinearArgs& a, const float* X, const float* W, float* sm, int m0, int n0, int rows, int cols, bool lost) {
    constexpr int KB = 64, XP = KB + 4, WP = FT_BN + 4, share = 128;
    float *xs = sm, *ws = sm + share * XP;  // [share][XP], [KB][WP]
    static_assert((share * XP + KB * WP) * 4 <= 2 * FT_STAGE, "both blocks fit in the stages");
    const int tid = threadIdx.x, c4 = (tid & 31) * 4, r0 = tid >> 5, nr = (rows + 15) / 16;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = lost ? __int_as_float(0x7fffffff) : 0.f;
    for (int k0 = 0; k0 < a.K && !lost; k0 += KB) {
        __syncthreads();
        for (int i = tid; i < (share + FT_BN) * (KB / 4); i += THREADS) {
            const int r = i / (KB / 4), kc = (i % (KB / 4)) * 4, k = k0 + kc, n = r - share;
            const bool is_x = r < share, ok = is_x ? r < rows : n < cols;
            const float* src = is_x ? X + (size_t)r * a.x_pitch() + k : W + (size_t)n * a.K + k;
            float v[4];
            if (VEC) {
                const float4 u = ok && k < a.K ? *reinterpret_cast<const float4*>(src) : make_float4(0.f, 0.f, 0.f, 0.f);
                v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[e] = ok && k + e < a.K ? src[e] : 0.f;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) (is_x ? xs[r * XP + kc + e] : ws[(kc + e) * WP + n]) = v[e];
        }
        __syncthreads();
        if (tid < 512)
#pragma unroll 4
            for (int k = 0; k < KB; ++k) {
                const float4 w = *reinterpret_cast<const float4*>(ws + k * WP + c4);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < nr) {
                        const float x = xs[(r0 + 16 * i) * XP + k];
                        acc[i][0] = fmaf(x, w.x, acc[i][0]); acc[i][1] = fmaf(x, w.y, acc[i][1]);
                        acc[i][2] = fmaf(x, w.z, acc[i][2]); acc[i][3] = fmaf(x, w.w, acc[i][3]);
                    }
            }
    }
    if (tid >= 512) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = r0 + 16 * i;
        if (i >= nr || r >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; j += 2)
            if (c4 + j < cols) epilogue_pair<float>(a, m0 + r, n0 + c4 + j, acc[i][j], acc[i][j + 1], n0 + c4 + j + 1 < a.N);
    }
}

// x [M, K] fp32 -> three bf16 part matrices [3][M][kp], kp = K rounded up to 8 (the columns past K are zero).  Bound by memory: 10 bytes an element.
constexpr int FP_THREADS = 256;
template <bool VEC>
__global__ void __launch_bounds__(FP_THREADS) f32_parts_kernel(const float* x, int ldx, int M, int K, int kp, bf16* parts, unsigned* counters, int n_counters) {
    pdl_trigger();
    pdl_wait();
    if (blockIdx.x == 0)
        for (int i = threadIdx.x; i < n_counters; i += FP_THREADS) counters[i] = 0u;
    const int64_t per_row = kp / 8, total = (int64_t)M * per_row;
    for (int64_t i = (int64_t)blockIdx.x * FP_THREADS + threadIdx.x; i < total; i += (int64_t)gridDim.x * FP_THREADS) {
        const int m = (int)(i / per_row), k = (int)(i % per_row) * 8;
        const float* src = x + (size_t)m * ldx + k;
        float v[8];
        if (VEC && k + 8 <= K) {
            load4(src, v);
            load4(src + 4, v + 4);
        } else {
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = k + e < K ? src[e] : 0.f;
        }
        uint2 lo[3], hi[3];
        ft_split4(make_float4(v[0], v[1], v[2], v[3]), lo);
        ft_split4(make_float4(v[4], v[5], v[6], v[7]), hi);
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(parts + ((size_t)q * M + m) * kp + k) = make_uint4(lo[q].x, lo[q].y, hi[q].x, hi[q].y);
    }
}

// How a Linear is dealt: tiles of 256 features x w tokens, token tiles fastest; items [0, whole) are tiles, the others parts of the tiles of the last round.
struct F32Plan {
    int w, tok_tiles, clusters, whole, cut, items;
};
inline F32Plan f32_plan(int M, int N, int K, int units) {
    const int nkb = (K + FT_BK - 1) / FT_BK, n_tiles = (N + 2 * FT_BN - 1) / (2 * FT_BN), least = (M + FT_MAX_W - 1) / FT_MAX_W;
    F32Plan best = {};
    double best_cost = 0;
    // A round costs 256 + w clocks a k-block and product.  More and narrower token tiles than needed pay where they fill a round better.
    for (int tt = least; tt <= least + 5; ++tt) {
        F32Plan p;
        p.tok_tiles = tt;
        p.w = ((M + tt - 1) / tt + 15) / 16 * 16;
        if (tt > least && (p.w < 128 || (long long)(tt - 1) * p.w >= M)) break;  // (narrow tiles cost little less; a tile without tokens)
        const long long tiles = (long long)tt * n_tiles;
        const int rest = (int)(tiles % units);
        int cut = rest ? units / rest : 1;
        if (cut > 8) cut = 8;
        while (cut > 1 && nkb < 4 * cut) --cut;  // (parts of fewer k-blocks cost more in slots than they save: 300 x 1024 x 1024 20.8 us with two, 17.2; 2000 x 1024 x 256 21.8, 15.9)
        p.cut = cut;
        p.whole = (int)(cut > 1 ? tiles - rest : tiles);
        p.items = (int)(p.whole + (tiles - p.whole) * cut);
        p.clusters = p.items < units ? p.items : units;
        const double rounds = (double)(tiles / units) + (rest ? 1.0 / cut : 0.0), cost = rounds * (256 + p.w) * (1 + (rest ? 0.03 * cut : 0.0));
        if (tt == least || cost < best_cost) best = p, best_cost = cost;
    }
    return best;
}

// A tile's sums go where the Linear's result goes, straight from the registers, if nothing but a bias follows; else, and for parts of cut tiles, to a slot of
// [w tokens][128 features], and f32_combine_kernel takes them from there.  (With the residual add from the registers, whose loads stand in the open, 804 x 16384 x 2048 took 314 us
// instead of 236.)
enum { FT_TO_SLOTS = 0, FT_TO_OUT = 1 };
inline int f32_step_of(const LinearArgs& a) {
    return (a.epi == EPI_STORE && a.n_act <= 0) || (a.epi == EPI_F32 && a.limit <= 0.f && a.alpha == 0.f) ? FT_TO_OUT : FT_TO_SLOTS;
}
struct F32Args {
    LinearArgs a;
    F32Plan p;
    int slot0;           // the first item that has slots (0, or p.whole)
    float* slots;        // [items - slot0][2 CTAs][w][128]
    unsigned* counters;  // [2 * tiles from slot0 on], zero: parts that are there, 2^16 for each that holds a number that is not finite
};

// The step after the Linear for the tiles whose sums (or parts of them, added in the order of k) lie in slots: four features of two tokens a thread.  Bound by memory.  A launch of its
// own spreads the parts of cut tiles over the chip (added by the cluster that arrives last, 804 x 2048 x 2048 took 70 us instead of 49), and keeps the steps' code away from the registers of
// the kernel before (with it inside, unrolled over a thread's tokens, 804 x 16384 x 2048 took 507 us).
constexpr int FC_THREADS = 256, FC_TOKENS = 16;
__global__ void __launch_bounds__(FC_THREADS) f32_combine_kernel(const __grid_constant__ F32Args args) {
    pdl_trigger();
    pdl_wait();
    const LinearArgs& a = args.a;
    const F32Plan& p = args.p;
    const int blocks = (p.w + FC_TOKENS - 1) / FC_TOKENS, half = blockIdx.x / blocks, rank = half & 1, nth = half >> 1, tile = args.slot0 + nth;
    if (args.counters[half] >> 16) return;  // computed again
    const int parts = tile < p.whole ? 1 : p.cut, item = tile < p.whole ? tile : p.whole + (tile - p.whole) * p.cut;
    const int t0 = tile % p.tok_tiles * p.w, n = (tile / p.tok_tiles * 2 + rank) * FT_BN + (threadIdx.x & 31) * 4, t = blockIdx.x % blocks * FC_TOKENS + (threadIdx.x >> 5);
    if (n >= a.N) return;
    const size_t slot = (size_t)p.w * FT_BN;
    const float* src = args.slots + ((size_t)(item - args.slot0) * 2 + rank) * slot + (threadIdx.x & 31) * 4;
    constexpr int U = FC_TOKENS * 32 / FC_THREADS;
    float4 v[U];
    const int end = min(p.w, a.M - t0);
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (t + u * (FC_THREADS / 32) < end) v[u] = __ldcg(reinterpret_cast<const float4*>(src + (size_t)(t + u * (FC_THREADS / 32)) * FT_BN));
#pragma unroll 2
    for (int s = 1; s < parts; ++s)
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (t + u * (FC_THREADS / 32) < end) {
                const float4 x = __ldcg(reinterpret_cast<const float4*>(src + 2 * s * slot + (size_t)(t + u * (FC_THREADS / 32)) * FT_BN));
                v[u].x += x.x, v[u].y += x.y, v[u].z += x.z, v[u].w += x.w;
            }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int m = t0 + t + u * (FC_THREADS / 32);
        if (t + u * (FC_THREADS / 32) >= end) continue;
        epilogue_pair<float>(a, m, n, v[u].x, v[u].y, n + 1 < a.N);
        if (n + 2 < a.N) epilogue_pair<float>(a, m, n + 2, v[u].z, v[u].w, n + 3 < a.N);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(FT_THREADS, 1) linear_f32_pair(const __grid_constant__ CUtensorMap parts, const __grid_constant__ F32Args args) {
    extern __shared__ __align__(1024) unsigned char ft_raw[];
    unsigned char* const sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[2], done[2], taken[2];  // a stage is there; its MMAs have completed; their sums have been added (full and taken: the first CTA's)
    __shared__ uint32_t tmem_slot;
    __shared__ unsigned redo[FT_REDO_WORDS];
    __shared__ volatile int lost;  // a wait of this CTA ran out
    const LinearArgs& a = args.a;
    const F32Plan& p = args.p;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = blockIdx.x & 1, cluster = blockIdx.x >> 1;
    const int nkb = (a.K + FT_BK - 1) / FT_BK;
    const float* const W = static_cast<const float*>(a.w);
    struct Item { int t0, n0, kb0, kb1, part; };  // first token, this CTA's first feature, k-blocks, part of a cut tile (-1: whole)
    auto item_of = [&](int i) {
        Item it;
        int tile = i;
        it.part = -1, it.kb0 = 0, it.kb1 = nkb;
        if (i >= p.whole) {
            tile = p.whole + (i - p.whole) / p.cut;
            it.part = (i - p.whole) % p.cut;
            it.kb0 = (int)((long long)nkb * it.part / p.cut);
            it.kb1 = (int)((long long)nkb * (it.part + 1) / p.cut);
        }
        it.t0 = tile % p.tok_tiles * p.w;
        it.n0 = (tile / p.tok_tiles * 2 + rank) * FT_BN;
        return it;
    };

    if (tid == 0) {
        lost = 0;
        for (int i = 0; i < 2; ++i) { ft_bar_init(&full[i], 2 * FT_SPLIT_WARPS + 1); ft_bar_init(&done[i], 1); ft_bar_init(&taken[i], 2 * FT_SUM_WARPS); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&parts) : "memory");
    }
    for (int i = tid; i < FT_REDO_WORDS; i += FT_THREADS) redo[i] = 0u;
    if (warp == FT_SPLIT_WARPS + FT_SUM_WARPS + 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ft_smem(&tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    ft_fence_before();
    ft_cluster_sync();  // the other CTA's barriers are there before any copy or commit reaches them
    ft_fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_trigger();
    if (warp < FT_SPLIT_WARPS) {
        ft_fewer_regs<FT_SPLIT_REGS>();
        constexpr int NF = FT_BN * FT_BK / 4 / (32 * FT_SPLIT_WARPS), RS = FT_BN / NF;  // float4s of a thread a k-block, and their row step
        static_assert(RS % 8 == 0, "a thread's rows lie at the same place of the swizzle");
        // float4 i of this thread: row (i * RS + tid / 16), columns 4 (tid % 16) .. of the k-block; the next block's are in flight while this one is split
        const int r0 = tid >> 4, c4 = (tid & 15) * 4;
        const size_t step = (size_t)RS * a.K;
        float4 v[NF];
        int item = cluster, kb = 0, cols = 0;
        Item c = {};
        const float* src = nullptr;
        auto start = [&]() {  // the rows of `item`
            if (item >= p.items) return;
            c = item_of(item);
            kb = c.kb0;
            cols = a.N - c.n0 - r0;
            src = W + (size_t)(c.n0 + r0) * a.K + c4;
#pragma unroll
            for (int i = 0; i < NF; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);  // rows past N stay zero
        };
        auto fetch = [&]() {
            const int k = kb * FT_BK;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                if (VEC) {
                    if (RS * i < cols) v[i] = __ldg(reinterpret_cast<const float4*>(src + i * step + k));
                } else {
                    float* w = reinterpret_cast<float*>(&v[i]);
#pragma unroll
                    for (int e = 0; e < 4; ++e) w[e] = RS * i < cols && k + c4 + e < a.K ? src[i * step + k + e] : 0.f;
                }
            }
        };
        auto fetch_vec_tail = [&]() {  // a block that runs past K, by whole float4s
            const bool in = kb * FT_BK + c4 < a.K;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in && RS * i < cols) v[i] = __ldg(reinterpret_cast<const float4*>(src + i * step + kb * FT_BK));
            }
        };
        auto next = [&]() {
            if (item >= p.items) return;
            if (VEC && (kb + 1) * FT_BK > a.K) fetch_vec_tail();
            else fetch();
            if (++kb == c.kb1) item += p.clusters, kb = -1;
        };
        start();
        next();
        const uint32_t full_at[2] = {ft_first_cta(&full[0]), ft_first_cta(&full[1])};
        unsigned char* const at = sm + r0 * 128 + (((c4 * 2) ^ ((r0 & 7) << 4)) & 0x7f);  // 16-byte units XORed with the row
        int total = 0;
        for (int i = cluster; i < p.items; i += p.clusters) {
            const Item t = item_of(i);
            total += t.kb1 - t.kb0;
        }
        bool alive = true;
        for (int it = 0; it < total; ++it) {
            if (it == 2) pdl_wait();  // nothing is multiplied before the predecessor's end: the wait's limit counts from there
            if (it >= 2 && alive && !ft_bar_wait(&done[it & 1], ((it >> 1) - 1) & 1)) { alive = false; lost = 1; }
            unsigned char* st = at + (it & 1) * FT_STAGE;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                uint2 part[3];
                ft_split4(v[i], part);
#pragma unroll
                for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(st + q * FT_TILE + i * RS * 128) = part[q];
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0 && alive) ft_bar_arrive(full_at[it & 1]);
            if (kb < 0) start();
            next();  // (behind the arrival, which would wait for the loads)
        }
        __syncwarp();
        ft_more_regs<FT_REGS>();
    } else if (warp < FT_SPLIT_WARPS + FT_SUM_WARPS) {
        ft_more_regs<FT_SUM_REGS>();
        pdl_wait();
        // this warp's sums: features 32 (warp % 4) .., tokens in blocks of 16, every second block
        constexpr int THREADS = 32 * FT_SUM_WARPS;
        const int etid = tid - 32 * FT_SPLIT_WARPS, g = (warp - FT_SPLIT_WARPS) >> 2, row = (warp & 3) * 32 + lane, n_ch = p.w / 16;
        const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + g * 16;
        const uint32_t taken_at[2] = {ft_first_cta(&taken[0]), ft_first_cta(&taken[1])};
        float acc[FT_CHUNKS][16];
        bool alive = true;
        int it = 0, ord = 0;
        for (int i = cluster; i < p.items; i += p.clusters, ++ord) {
            const Item c = item_of(i);
#pragma unroll
            for (int q = 0; q < FT_CHUNKS; ++q)
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[q][j] = 0.f;
            for (int kb = c.kb0; kb < c.kb1; ++kb, ++it) {
                if (alive && !ft_bar_wait(&done[it & 1], (it >> 1) & 1)) { alive = false; lost = 1; }
                __syncwarp();
                ft_fence_after();
                const uint32_t from = mine + (it & 1) * 256;
                // two blocks a round trip (300 clocks each)
#pragma unroll
                for (int q = 0; q < FT_CHUNKS; q += 2) {
                    if (g + 2 * q >= n_ch) break;
                    float u[16], v[16];
                    const bool two = q + 1 < FT_CHUNKS && g + 2 * q + 2 < n_ch;
                    ft_ld16(from + q * 32, u);
                    if (two) ft_ld16(from + q * 32 + 32, v);
                    ft_wait_ld();
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[q][j] += u[j];
                    if (q + 1 < FT_CHUNKS && two)
#pragma unroll
                        for (int j = 0; j < 16; ++j) acc[q + 1 < FT_CHUNKS ? q + 1 : q][j] += v[j];
                }
                ft_fence_before();
                __syncwarp();
                if (lane == 0 && alive) ft_bar_arrive(taken_at[it & 1]);
            }
            // The tile's sums.  An operand that is not finite makes a part that is NaN (inf - inf), so every sum it enters is NaN: found here, once.
            int strange = 0;
            if (lost) alive = false;
#pragma unroll
            for (int q = 0; q < FT_CHUNKS; ++q)
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    strange |= not_finite(acc[q][j]);
                    if (!alive) acc[q][j] = __int_as_float(0x7fffffff);
                }
            if (!alive) strange = 0;
            asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %0, 0;\nbarrier.cta.red.or.pred q, 1, %1, p;\nselp.b32 %0, 1, 0, q;\n}\n" : "+r"(strange) : "n"(THREADS) : "memory");
            const bool slotted = i >= args.slot0;
            if (strange && (!slotted || c.part < 0)) {  // computed again at the end
                if (etid == 0) {
                    redo[ord >> 5] |= 1u << (ord & 31);
                    if (slotted) args.counters[2 * (i - args.slot0) + rank] = 0x10001u;
                }
                continue;
            }
            if (slotted) {
                float* const slot = args.slots + ((size_t)(i - args.slot0) * 2 + rank) * p.w * FT_BN + row;
#pragma unroll
                for (int q = 0; q < FT_CHUNKS; ++q)
                    if (g + 2 * q < n_ch)
#pragma unroll
                        for (int j = 0; j < 16; ++j) slot[((g + 2 * q) * 16 + j) * FT_BN] = acc[q][j];
                if (c.part >= 0 && etid == 0) {  // of a cut tile with a number that is not finite the last part to arrive computes the tile again
                    const unsigned before = atomicAdd(args.counters + 2 * (p.whole - args.slot0 + (i - p.whole) / p.cut) + rank, strange ? 0x10001u : 1u);
                    if ((before & 0xffffu) + 1u == (unsigned)p.cut && (strange || before >> 16)) redo[ord >> 5] |= 1u << (ord & 31);
                }
                continue;
            }
            const int n = c.n0 + row;
            const float bias = a.bias && n < a.N ? static_cast<const float*>(a.bias)[n] : 0.f;
            float* const to = (a.epi == EPI_STORE ? static_cast<float*>(a.out) : a.out32) + n;
#pragma unroll
            for (int q = 0; q < FT_CHUNKS; ++q) {
                const int t = c.t0 + (g + 2 * q) * 16;
                if (g + 2 * q >= n_ch || n >= a.N) continue;
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if (t + j < a.M) to[(size_t)(t + j) * a.N] = acc[q][j] + bias;
            }
        }
        __syncwarp();
        ft_fewer_regs<FT_REGS>();
    } else {
        ft_fewer_regs<FT_REST_REGS>();
        if (warp == FT_SPLIT_WARPS + FT_SUM_WARPS && lane == 0) {
            pdl_wait();
            const int half = p.w / 2;
            bool alive = true;
            int it = 0;
            for (int i = cluster; i < p.items; i += p.clusters) {
                const Item c = item_of(i);
                for (int kb = c.kb0; kb < c.kb1; ++kb, ++it) {
                    if (it >= 2 && alive && !ft_bar_wait(&done[it & 1], ((it >> 1) - 1) & 1)) { alive = false; lost = 1; }
                    if (!alive) continue;
                    // the pair's copies count on the first CTA's barrier (the other CTA's may land before it is armed)
                    if (rank == 0) ft_bar_expect(&full[it & 1], 2u * 3u * (uint32_t)half * 128u);
                    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
                                     ft_smem(sm + (it & 1) * FT_STAGE + 3 * FT_TILE)),
                                 "l"(&parts), "r"(ft_first_cta(&full[it & 1])), "r"(kb * FT_BK), "r"(c.t0 + rank * half), "r"(0)
                                 : "memory");
                }
            }
        }
        if (warp == FT_SPLIT_WARPS + FT_SUM_WARPS + 1 && rank == 0) {
            // (the whole warp walks, one thread of it issues: so the operands are uniform.  In a thread's own registers the 24 instructions of a k-block took longer to
            // issue than to run)
            pdl_wait();  // (the copies begin behind it: the waits' limits count from there)
            bool alive = true;
            int it = 0;
            const uint32_t idesc = FT_IDESC | (uint32_t)(p.w >> 3) << 17, x_part = (uint32_t)(p.w / 2) * 128u >> 4, first = ft_desc_lo(ft_smem(sm));
            for (int i = cluster; i < p.items; i += p.clusters) {
                const Item c = item_of(i);
                for (int kb = c.kb0; kb < c.kb1; ++kb, ++it) {
                    if (it >= 2 && alive && !ft_bar_wait(&taken[it & 1], ((it >> 1) - 1) & 1)) alive = false;
                    if (alive && !ft_bar_wait(&full[it & 1], (it >> 1) & 1)) alive = false;
                    if (!__all_sync(0xffffffffu, alive)) { alive = false; lost = 1; continue; }
                    ft_fence_after();
                    const uint32_t w0 = first + (it & 1) * (FT_STAGE >> 4), w1 = w0 + (FT_TILE >> 4), w2 = w1 + (FT_TILE >> 4), d = tmem + (it & 1) * 256;
                    const uint32_t x0 = w2 + (FT_TILE >> 4), x1 = x0 + x_part, x2 = x1 + x_part;  // parts: 0 hi, 1 mid, 2 lo
                    if (ft_elect()) {
                        // the small products first; the scale of the parts changes twice: 2^16, 2^8, 1
                        ft_mma<false, 0>(d, w1, x1, idesc);
#pragma unroll
                        for (int k = 2; k < 8; k += 2) ft_mma<true, 0>(d, w1 + k, x1 + k, idesc);
#pragma unroll
                        for (int k = 0; k < 8; k += 2) ft_mma<true, 0>(d, w2 + k, x0 + k, idesc);
#pragma unroll
                        for (int k = 0; k < 8; k += 2) ft_mma<true, 0>(d, w0 + k, x2 + k, idesc);
                        ft_mma<true, 8>(d, w1, x0, idesc);
#pragma unroll
                        for (int k = 2; k < 8; k += 2) ft_mma<true, 0>(d, w1 + k, x0 + k, idesc);
#pragma unroll
                        for (int k = 0; k < 8; k += 2) ft_mma<true, 0>(d, w0 + k, x1 + k, idesc);
                        ft_mma<true, 8>(d, w0, x0, idesc);
#pragma unroll
                        for (int k = 2; k < 8; k += 2) ft_mma<true, 0>(d, w0 + k, x0 + k, idesc);
                        ft_commit(&done[it & 1]);
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
        ft_more_regs<FT_REGS>();
    }
    ft_fence_before();
    ft_cluster_sync();  // every MMA has completed, nothing reaches the other CTA any more: the stages are free
    ft_fence_after();
    if (warp == FT_SPLIT_WARPS + FT_SUM_WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
    for (int i = cluster, ord = 0; i < p.items; i += p.clusters, ++ord) {
        if (!(redo[ord >> 5] >> (ord & 31) & 1u)) continue;
        const Item c = item_of(i);
        const int end = min(a.M, c.t0 + p.w);
        for (int m = c.t0; m < end; m += 128)
            ft_fma_rows<VEC, FT_THREADS>(a, static_cast<const float*>(a.x) + (size_t)m * a.x_pitch(), W + (size_t)c.n0 * a.K, reinterpret_cast<float*>(sm), m, c.n0, min(128, end - m),
                             min(FT_BN, a.N - c.n0), lost);
    }
}

typedef CUresult (*FtEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline FtEncode ft_encode() {  // the driver's entry point through the runtime: no link against libcuda
    static const FtEncode fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult found;
        return cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<FtEncode>(ptr) : nullptr;
    }();
    return fn;
}
inline int ft_units() {  // pairs of SMs
    const int sms = device_info::sm_count();
    return sms >= 2 ? sms / 2 : 1;
}

// scratch: counters, slots, the parts of x
struct F32Scratch {
    int64_t counters, slots, parts, bytes;
    int kp;
};
inline F32Scratch f32_scratch(int M, int K, const F32Plan& p, int step) {
    F32Scratch s;
    const int64_t items = step == FT_TO_SLOTS ? p.items : p.items - p.whole;
    s.kp = (K + 7) / 8 * 8;
    s.counters = 2 * (step == FT_TO_SLOTS ? p.whole + (p.items - p.whole) / p.cut : (p.items - p.whole) / p.cut);
    s.slots = (s.counters * 4 + 1023) / 1024 * 1024;
    s.parts = s.slots + items * 2 * p.w * FT_BN * 4;
    s.bytes = s.parts + 3 * (int64_t)M * s.kp * 2;
    return s;
}
// Rows of a launch: 4096, because the slots of a longer prompt would take as much memory as its result, and more only where slots and parts stay below 128 MB; equal shares, since a launch
// of a few rows takes as long as one of a few hundred (5000 x 384 x 128 in 4096 + 904 rows 25 us, 15.1 so).
inline int f32_launch_rows(int M, int N, int K) {
    const int64_t room = ((int64_t)128 << 20) / (4 * (int64_t)N + 6 * (int64_t)K), most = room < 4096 ? 4096 : room > 16384 ? 16384 : room;
    const int launches = (int)((M + most - 1) / most);
    return ((M + launches - 1) / launches + 15) / 16 * 16;
}
// of a Linear of M rows
inline int64_t f32_scratch_bytes(int M, int N, int K, int step) {
    const int rows = f32_launch_rows(M, N, K), m = M < rows ? M : rows, rest = M > m ? M % m : 0;
    const int64_t bytes = f32_scratch(m, K, f32_plan(m, N, K, ft_units()), step).bytes, more = rest ? f32_scratch(rest, K, f32_plan(rest, N, K, ft_units()), step).bytes : 0;
    return bytes > more ? bytes : more;
}

inline cudaError_t launch_f32_tokens(const LinearArgs& a, const F32Plan& p, int step, void* scratch, bool& taken, cudaStream_t st) {
    const F32Scratch s = f32_scratch(a.M, a.K, p, step);
    const F32Args args{a, p, step == FT_TO_SLOTS ? 0 : p.whole, reinterpret_cast<float*>(static_cast<char*>(scratch) + s.slots), static_cast<unsigned*>(scratch)};
    bf16* const parts = reinterpret_cast<bf16*>(static_cast<char*>(scratch) + s.parts);
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)s.kp, (cuuint64_t)a.M, 3}, strides[2] = {(cuuint64_t)s.kp * 2, (cuuint64_t)a.M * s.kp * 2};
    const cuuint32_t box[3] = {FT_BK, (cuuint32_t)p.w / 2, 3}, unit[3] = {1, 1, 1};
    taken = ft_encode()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, parts, dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    if (!taken) return cudaSuccess;
    const auto aligned = [](const void* q) { return reinterpret_cast<uintptr_t>(q) % 16 == 0; };
    const bool x_vec = a.x_pitch() % 4 == 0 && aligned(a.x), vec = x_vec && a.K % 4 == 0 && aligned(a.w);
    const int64_t blocks = ((int64_t)a.M * (s.kp / 8) + FP_THREADS - 1) / FP_THREADS;
    cudaError_t e = launch_pdl(x_vec ? f32_parts_kernel<true> : f32_parts_kernel<false>, dim3((unsigned)(blocks < 4096 ? blocks : 4096)), dim3(FP_THREADS), 0, st, static_cast<const float*>(a.x),
                               a.x_pitch(), a.M, a.K, s.kp, parts, args.counters, (int)s.counters);
    if (e) return e;
    auto kernel = vec ? linear_f32_pair<true> : linear_f32_pair<false>;
    e = vec ? device_info::allow_shared<linear_f32_pair<true>>(FT_SMEM) : device_info::allow_shared<linear_f32_pair<false>>(FT_SMEM);
    if (e) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)p.clusters);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = FT_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = device_info::pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, map, args);
    if (!e && s.counters) e = launch_pdl(f32_combine_kernel, dim3((unsigned)s.counters * (unsigned)((p.w + FC_TOKENS - 1) / FC_TOKENS)), dim3(FC_THREADS), 0, st, args);
    return e ? e : cudaGetLastError();
}

// Few features over many tokens: hybrid_linear_f32_cta.cuh, which reads x once or a few times and writes nothing of it.  us there and here: 4096 x 8 x 2048 21, 39; 4096 x 128 x 4096 43, 73;
// 804 x 32 x 2048 16, 19; 300 x 32 x 4096 21.5, 22.7; 2000 x 128 x 1024 19, 23; but 300 x 128 x 2048 20, 17.5, 2000 x 32 x 2048 29, 25 (its clusters of eight CTAs fill a second round),
// 4096 x 256 x 2048 43, 43.  Up to 384 features where its tiles fill the SMs once and K is short: 3000 x 384 x 512 20, 24; 2000 x 256 x 1024 20, 22; 1200 x 384 x 1024 20, 22.5.
inline bool f32_few_features(int M, int N, int K) {
    if (N <= 128) return M > 4096 || (K >= 512 && (M > 2048 || (M > 1024 && K <= 1024) || (N <= 64 && M >= 256 && M <= 1024 && K >= 1024)));
    return N <= 384 && M > 1024 && K >= 512 && K <= 1024 && ((M + 127) / 128) * ((N + 127) / 128) <= ft_units();
}
// false: not for this kernel (no room, few features, more tiles a cluster than `redo` has bits)
inline bool launch_linear_f32_pair(const LinearArgs& a, void* scratch, int64_t scratch_bytes, cudaStream_t st, cudaError_t& e) {
    const int step = f32_step_of(a), rows = f32_launch_rows(a.M, a.N, a.K);
    if (f32_few_features(a.M, a.N, a.K) || !scratch || scratch_bytes < f32_scratch_bytes(a.M, a.N, a.K, step) || reinterpret_cast<uintptr_t>(scratch) % 16 || !ft_encode()) return false;
    {
        const F32Plan p = f32_plan(a.M < rows ? a.M : rows, a.N, a.K, ft_units());
        if (p.items / p.clusters >= 32 * FT_REDO_WORDS) return false;
    }
    for (int m = 0; m < a.M; m += rows) {  // (rows of everything that a row of x makes)
        LinearArgs b = a;
        b.M = a.M - m < rows ? a.M - m : rows;
        b.ldx = a.x_pitch();
        const bool half = a.epi == EPI_GLU || a.epi == EPI_SWIGLU || a.epi == EPI_GEGLU;
        b.x = static_cast<const float*>(a.x) + (size_t)m * a.x_pitch();
        if (a.out) b.out = static_cast<float*>(a.out) + (size_t)m * (half ? a.N / 2 : a.N);
        if (a.out32) b.out32 = a.out32 + (size_t)m * a.N;
        if (a.rowscale) b.rowscale = a.rowscale + (size_t)m * a.rs_pitch;
        bool taken = false;
        e = launch_f32_tokens(b, f32_plan(b.M, b.N, b.K, ft_units()), step, scratch, taken, st);
        if (!taken) return false;  // (of the first rows: the map's sizes are the same for the others)
        if (e) return true;
    }
    return true;
}

}  // namespace mbh
