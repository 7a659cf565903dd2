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
// What bounds it: the sixteen warps that load, split, store and add.  750 x 16384 x 2048 under ncu: tensor pipe 38 % of the cycles, shared memory 41 %, both with
// room.  The 64 x 64 FMA tiles it replaces (24 TFLOP/s of 74): 8870 us of Linears for 3 x ~250 tokens, width 2048, two layers; about 1820 here.
//
// CTA = 128 x 128 outputs, or one of `splits` parts of their k range (a cluster; the parts are added through distributed shared memory in
// rank order, so a small problem fills the chip and the result is the same every time).  17 warps: sixteen load fp32 from global memory
// (one k-block ahead, in registers), split, write the six part tiles (128B-swizzled, K-major) of a stage and add the block before to
// their registers; one thread of the last issues the MMAs (with eight workers the loads' latency was in the open: 3530 us of Linears against 1870).  Two stages: the MMAs of a block run under the splitting of the next.
// An infinity or a NaN in the operands of a tile, or a number from 2^120 on (256 x is formed): its outputs are computed again with FMAs (ft_fma_rows).
#pragma once
#include "hybrid_linear.cuh"

namespace mbh {

constexpr int FT_BM = 128, FT_BN = 128, FT_BK = 64, FT_WARPS = 16 /* workers */, FT_THREADS = 32 * (FT_WARPS + 1), FT_TILE = 128 * 64 * 2;  // a part tile: 128 rows of 128 bytes
constexpr int FT_MIN_K = 16;
constexpr int FT_STAGE = 6 * FT_TILE, FT_SMEM = 2 * FT_STAGE + 1024, FT_LD = FT_BN + 4;
static_assert(FT_BM * FT_LD * 4 <= 2 * FT_STAGE, "the sums of a tile fit in the stages");

__device__ __forceinline__ uint32_t ft_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ft_bar_init(uint64_t* b, uint32_t count) { asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(ft_smem(b)), "r"(count) : "memory"); }
__device__ __forceinline__ void ft_bar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(ft_smem(b)) : "memory"); }
// Waits a bounded time.  false: gave up (the caller marks the CTA dead and goes on to the end without waiting again).
__device__ __forceinline__ bool ft_bar_wait(uint64_t* b, uint32_t parity) {
    for (int i = 0; i < (1 << 22); ++i) {
        uint32_t ok;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok) : "r"(ft_smem(b)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
// K-major, 128B-swizzled tile of 128-byte rows: 8-row groups 1024 B apart, version 1, layout SWIZZLE_128B
__device__ __forceinline__ uint64_t ft_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
constexpr uint32_t FT_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FT_BN >> 3) << 17) | ((uint32_t)(FT_BM >> 4) << 24);  // bf16 x bf16 -> fp32
// D = A B (accumulate 0) or A B + D / 2^DOWN
template <int DOWN>
__device__ __forceinline__ void ft_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, %5;\n}\n" ::"r"(d), "l"(a), "l"(b), "r"(FT_IDESC), "r"(accumulate),
                 "n"(DOWN)
                 : "memory");
}
__device__ __forceinline__ void ft_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ft_smem(b)) : "memory");
}
__device__ __forceinline__ void ft_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_ld16(uint32_t addr, float (&v)[16]) {
    uint32_t* u = reinterpret_cast<uint32_t*>(v);
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]),
                   "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
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
__device__ __forceinline__ float ft_ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}
__device__ __forceinline__ void ft_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// `share` rows of a tile from row `first` on (a multiple of 16, at most 128) with FMAs in the order of k, through shared memory (the stages: the parts are not needed
// any more).  A thread takes four columns of every 16th row.  About the time the whole tile takes with FMAs, once per tile that holds an infinity or a NaN.
template <bool VEC>
__device__ __noinline__ void ft_fma_rows(const LinearArgs& a, const float* X, const float* W, float* sm, int m0, int n0, int first, int share, int rows, int cols) {
    constexpr int KB = 64, XP = KB + 4, WP = FT_BN + 4;
    float *xs = sm, *ws = sm + FT_BM * XP;  // [share][XP], [KB][WP]
    static_assert((FT_BM * XP + KB * WP) * 4 <= 2 * FT_STAGE, "both blocks fit in the stages");
    const int tid = threadIdx.x, c4 = (tid & 31) * 4, r0 = tid >> 5, nr = share / 16;
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    for (int k0 = 0; k0 < a.K; k0 += KB) {
        __syncthreads();
        for (int i = tid; i < (share + FT_BN) * (KB / 4); i += FT_THREADS) {
            const int r = i / (KB / 4), kc = (i % (KB / 4)) * 4, k = k0 + kc, n = r - share;
            const bool is_x = r < share, ok = is_x ? first + r < rows : n < cols;
            const float* src = is_x ? X + (size_t)(first + r) * a.x_pitch() + k : W + (size_t)n * a.K + k;
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
        const int r = first + r0 + 16 * i;
        if (i >= nr || r >= rows) continue;
#pragma unroll
        for (int j = 0; j < 4; j += 2)
            if (c4 + j < cols) epilogue_pair<float>(a, m0 + r, n0 + c4 + j, acc[i][j], acc[i][j + 1], n0 + c4 + j + 1 < a.N);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(FT_THREADS, 1) linear_f32_parts(LinearArgs a, int splits) {
    extern __shared__ __align__(1024) unsigned char ft_raw[];
    unsigned char* const sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[2], done[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int flags;  // 1: a sum that is not finite; 2: a wait that ended without its event
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // row tiles fastest: the CTAs that share a tile of W run together
    const int tiles_m = (a.M + FT_BM - 1) / FT_BM, tile = blockIdx.x / splits, rank = blockIdx.x % splits;
    const int n0 = tile / tiles_m * FT_BN, m0 = tile % tiles_m * FT_BM;
    const float* X = static_cast<const float*>(a.x) + (size_t)m0 * a.x_pitch();
    const float* W = static_cast<const float*>(a.w) + (size_t)n0 * a.K;
    const int rows = min(FT_BM, a.M - m0), cols = min(FT_BN, a.N - n0);
    const int nkb = (a.K + FT_BK - 1) / FT_BK, kb0 = (int)((long long)nkb * rank / splits), kb1 = (int)((long long)nkb * (rank + 1) / splits);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { ft_bar_init(&full[i], FT_WARPS); ft_bar_init(&done[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        flags = 0;
    }
    if (warp == FT_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ft_smem(&tmem_slot)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // rows of x and W past the end stay zero in both stages
    for (int i = tid; i < 2 * FT_STAGE / 16; i += FT_THREADS) {
        const int r = (i % (FT_TILE / 16)) / 8, part = (i / (FT_TILE / 16)) % 6;
        if (r >= (part < 3 ? rows : cols)) reinterpret_cast<uint4*>(sm)[i] = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    const uint32_t tmem = tmem_slot;
    constexpr int NF = FT_BM * FT_BK / 4 / (32 * FT_WARPS), RS = FT_BM / NF, NC = FT_BN / (FT_WARPS / 4);  // float4s and row step of a worker, its columns of the sums
    float acc[NC];
    int strange = 0;  // a sum that is not finite
    if (warp < FT_WARPS) {
        // float4 i of this thread: row (i * RS + tid / 16), columns 4 (tid % 16) .. of the k-block
        const int r0 = tid >> 4, c4 = (tid & 15) * 4;
        float4 px[NF], pw[NF];
        auto fetch = [&](int kb) {
            const int k = kb * FT_BK + c4;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                const int r = r0 + RS * i;
                px[i] = pw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                const float *xp = X + (size_t)r * a.x_pitch() + k, *wp = W + (size_t)r * a.K + k;
                if (VEC) {
                    if (k < a.K) {
                        if (r < rows) px[i] = *reinterpret_cast<const float4*>(xp);
                        if (r < cols) pw[i] = __ldg(reinterpret_cast<const float4*>(wp));
                    }
                } else {
                    float *x = reinterpret_cast<float*>(&px[i]), *w = reinterpret_cast<float*>(&pw[i]);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (k + e < a.K) {
                            if (r < rows) x[e] = xp[e];
                            if (r < cols) w[e] = wp[e];
                        }
                }
            }
        };
        auto put = [&](unsigned char* tile, int r, const float4& v) {
            const float* f = reinterpret_cast<const float*>(&v);
            uint32_t part[3][2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                // every subtraction is exact; 256 x first, so that both steps of a part are one instruction for two numbers
                const uint64_t v8 = ft_mul2(ft_two(f[2 * e], f[2 * e + 1]), 256.f);
                const uint32_t h = ft_pack(f[2 * e], f[2 * e + 1]);
                const uint64_t r1 = ft_fma2(ft_unpack(h), -256.f, v8);
                const uint32_t m = ft_pack(ft_first(r1), ft_second(r1));
                const uint64_t r2 = ft_fma2(ft_unpack(m), -256.f, ft_mul2(r1, 256.f));
                part[0][e] = h;
                part[1][e] = m;
                part[2][e] = __byte_perm(__float_as_uint(ft_first(r2)), __float_as_uint(ft_second(r2)), 0x7632);  // at most 8 significant bits are left: exact
            }
            unsigned char* at = tile + r * 128 + (((c4 * 2) ^ ((r & 7) << 4)) & 0x7f);  // 16-byte units XORed with the row
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(at + q * FT_TILE) = make_uint2(part[q][0], part[q][1]);
        };
#pragma unroll
        for (int j = 0; j < NC; ++j) acc[j] = 0.f;
        const uint32_t mine = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * NC;
        bool alive = true;
        auto promote = [&](int it) {
            if (alive && !ft_bar_wait(&done[it & 1], (it >> 1) & 1)) { alive = false; atomicOr(&flags, 2); }
            __syncwarp();
            ft_fence_after();
            float v[16];  // (32 at once spill beside the operands in flight)
#pragma unroll
            for (int c = 0; c < NC / 16; ++c) {
                ft_ld16(mine + (it & 1) * 128 + c * 16, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c * 16 + j] += v[j];
            }
            ft_fence_before();
        };
        if (kb0 < kb1) fetch(kb0);
        // Block it may overwrite stage it & 1 and accumulator it & 1 once block it - 2 has been added up: promote() of it - 2 waited for its
        // MMAs, and every warp arrives on full[] after that.
        for (int it = 0; it < kb1 - kb0; ++it) {
            unsigned char* st = sm + (it & 1) * FT_STAGE;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                const int r = r0 + RS * i;
                if (r < rows) put(st, r, px[i]);
                if (r < cols) put(st + 3 * FT_TILE, r, pw[i]);
            }
            if (kb0 + it + 1 < kb1) fetch(kb0 + it + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) ft_bar_arrive(&full[it & 1]);
            if (it > 0) promote(it - 1);
        }
        if (kb0 < kb1) promote(kb1 - kb0 - 1);
        // an operand that is not finite makes a part that is NaN (inf - inf), so every sum it enters is NaN: found here, once
#pragma unroll
        for (int j = 0; j < NC; ++j) strange |= not_finite(acc[j]);
        if (strange) atomicOr(&flags, 1);
    } else if (lane == 0) {
        bool alive = true;
        for (int it = 0; it < kb1 - kb0; ++it) {
            if (alive && !ft_bar_wait(&full[it & 1], (it >> 1) & 1)) { alive = false; atomicOr(&flags, 2); }
            ft_fence_after();
            const uint32_t base = ft_smem(sm + (it & 1) * FT_STAGE), d = tmem + (it & 1) * 128;
            // (x part, W part), the small products first: 0 hi, 1 mid, 2 lo
            constexpr int PX[6] = {1, 0, 2, 0, 1, 0}, PW[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint64_t xd = ft_desc(base + PX[p] * FT_TILE) + (uint64_t)(2 * k), wd = ft_desc(base + (3 + PW[p]) * FT_TILE) + (uint64_t)(2 * k);
                    if (k == 0 && (p == 3 || p == 5)) ft_mma<8>(d, xd, wd, 1u);  // the scale of the parts changes: 2^16, 2^8, 1
                    else ft_mma<0>(d, xd, wd, (p | k) ? 1u : 0u);
                }
            ft_commit(&done[it & 1]);
        }
    }
    ft_fence_before();
    __syncthreads();  // every MMA has completed (the last promote waited for it): the stages are free
    ft_fence_after();
    float(*sum)[FT_LD] = reinterpret_cast<float(*)[FT_LD]>(sm);
    if (warp < FT_WARPS) {
        const int r = (warp & 3) * 32 + lane, c = (warp >> 2) * NC;
#pragma unroll
        for (int j = 0; j < NC; j += 4) *reinterpret_cast<float4*>(&sum[r][c + j]) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
    }
    if (warp == FT_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u));
    int mark = 0;
    if (splits > 1) {
        ft_cluster_sync();
        for (int s = 0; s < splits; ++s) mark |= __float_as_int(ft_ld_cluster(ft_smem(&flags), s));
    } else {
        __syncthreads();
        mark = flags;
    }
    // this CTA's share of the tile's rows: sums over the ranks in order, then the step that follows the Linear, a pair of columns per thread
    const int share = FT_BM / splits, first = rank * share;
    if (mark == 1) {
        ft_fma_rows<VEC>(a, X, W, reinterpret_cast<float*>(sm), m0, n0, first, share, rows, cols);
    } else {
        for (int i = tid; i < share * (FT_BN / 2); i += FT_THREADS) {
            const int r = first + i / (FT_BN / 2), c = (i % (FT_BN / 2)) * 2;
            if (r >= rows || c >= cols) continue;
            float v0 = 0.f, v1 = 0.f;
            if (mark & 2) {
                v0 = v1 = __int_as_float(0x7fffffff);
            } else if (splits > 1) {
                for (int s = 0; s < splits; ++s) { v0 += ft_ld_cluster(ft_smem(&sum[r][c]), s); v1 += ft_ld_cluster(ft_smem(&sum[r][c + 1]), s); }
            } else {
                const float2 v = *reinterpret_cast<const float2*>(&sum[r][c]);
                v0 = v.x; v1 = v.y;
            }
            epilogue_pair<float>(a, m0 + r, n0 + c, v0, v1, n0 + c + 1 < a.N);
        }
    }
    if (splits > 1) ft_cluster_sync();  // nobody leaves while its sums are being read
}

inline cudaError_t launch_linear_f32_parts(const LinearArgs& a, cudaStream_t st) {
    const int tiles_n = (a.N + FT_BN - 1) / FT_BN, tiles_m = (a.M + FT_BM - 1) / FT_BM, nkb = (a.K + FT_BK - 1) / FT_BK;
    // split k until the CTAs fill the chip (148 SMs, one CTA each), at least four k-blocks a part
    int splits = 1;
    while (splits < 8 && (long long)tiles_n * tiles_m * splits * 2 <= 160 && nkb >= 8 * splits) splits *= 2;
    const bool vec = a.K % 4 == 0 && a.x_pitch() % 4 == 0 && (reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) % 16 == 0;
    auto kernel = vec ? linear_f32_parts<true> : linear_f32_parts<false>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FT_SMEM);
    if (e) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles_n * (unsigned)tiles_m * (unsigned)splits);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = FT_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kernel, a, splits);
    return e ? e : cudaGetLastError();
}

}  // namespace mbh
