// fp32 Linears of prompts by single CTAs, with no memory beside their operands: the arithmetic of hybrid_linear_f32.cuh, both operands split where they are used.
//
// For calls that bring no room for the parts of x (the entries of mistral_b200_hybrid.h allocate nothing) and for matrices of few features, where
// x is the larger operand and its parts, written out ahead and read back, cost more than splitting it once or twice here (f32_few_features).
//
// CTA = 128 tokens x 128 features, or one of `splits` parts of their k range (a cluster; the parts are added through distributed shared memory in
// rank order, so a small problem fills the chip and the result is the same every time).  17 warps: sixteen load fp32 from global memory
// (one k-block ahead, in registers), split, write the six part tiles (128B-swizzled, K-major) of a stage and add the block before to
// their registers; one thread of the last issues the MMAs.  Two stages: the MMAs of a block run under the splitting of the next.  What bounds it: the sixteen warps that load, split,
// store and add (750 x 16384 x 2048: tensor pipe 38 % of the cycles, shared memory 41 %).
#pragma once
#include "hybrid_linear_f32.cuh"

namespace mbh {

constexpr int F1_BM = 128, F1_WARPS = 16 /* workers */, F1_THREADS = 32 * (F1_WARPS + 1);
constexpr int F1_STAGE = 6 * FT_TILE, F1_SMEM = 2 * F1_STAGE + 1024, F1_LD = FT_BN + 4;
static_assert(F1_BM * F1_LD * 4 <= 2 * F1_STAGE, "the sums of a tile fit in the stages");
constexpr uint32_t F1_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FT_BN >> 3) << 17) | ((uint32_t)(F1_BM >> 4) << 24);  // bf16 x bf16 -> fp32
// D = A B (accumulate 0) or A B + D / 2^DOWN.  a, b: lower words of the descriptors
template <int DOWN>
__device__ __forceinline__ void f1_mma(uint32_t d, uint32_t a, uint32_t b, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\n.reg .b64 da, db;\nmov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p, %6;\n}\n" ::"r"(d), "r"(a), "r"(b), "r"(F1_IDESC), "r"(accumulate), "n"(FT_DESC_HI), "n"(DOWN)
                 : "memory");
}
__device__ __forceinline__ void f1_commit(uint64_t* b) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(ft_smem(b)) : "memory");
}
__device__ __forceinline__ float f1_ld_cluster(uint32_t addr, uint32_t rank) {
    uint32_t remote;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
    return v;
}

template <bool VEC>
__global__ void __launch_bounds__(F1_THREADS, 1) linear_f32_parts(LinearArgs a, int splits) {
    extern __shared__ __align__(1024) unsigned char ft_raw[];
    unsigned char* const sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ft_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t full[2], done[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int flags;  // 1: a sum that is not finite; 2: a wait that ended without its event
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // row tiles fastest: the CTAs that share a tile of W run together
    const int tiles_m = (a.M + F1_BM - 1) / F1_BM, tile = blockIdx.x / splits, rank = blockIdx.x % splits;
    const int n0 = tile / tiles_m * FT_BN, m0 = tile % tiles_m * F1_BM;
    const float* X = static_cast<const float*>(a.x) + (size_t)m0 * a.x_pitch();
    const float* W = static_cast<const float*>(a.w) + (size_t)n0 * a.K;
    const int rows = min(F1_BM, a.M - m0), cols = min(FT_BN, a.N - n0);
    const int nkb = (a.K + FT_BK - 1) / FT_BK, kb0 = (int)((long long)nkb * rank / splits), kb1 = (int)((long long)nkb * (rank + 1) / splits);

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { ft_bar_init(&full[i], F1_WARPS); ft_bar_init(&done[i], 1); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        flags = 0;
    }
    if (warp == F1_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ft_smem(&tmem_slot)), "r"(256u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // rows of x and W past the end stay zero in both stages
    for (int i = tid; i < 2 * F1_STAGE / 16; i += F1_THREADS) {
        const int r = (i % (FT_TILE / 16)) / 8, part = (i / (FT_TILE / 16)) % 6;
        if (r >= (part < 3 ? rows : cols)) reinterpret_cast<uint4*>(sm)[i] = make_uint4(0, 0, 0, 0);
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    const uint32_t tmem = tmem_slot;
    constexpr int NF = F1_BM * FT_BK / 4 / (32 * F1_WARPS), RS = F1_BM / NF, NC = FT_BN / (F1_WARPS / 4);  // float4s and row step of a worker, its columns of the sums
    float acc[NC];
    int strange = 0;  // a sum that is not finite
    if (warp < F1_WARPS) {
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
            uint2 part[3];
            ft_split4(v, part);
            unsigned char* at = tile + r * 128 + (((c4 * 2) ^ ((r & 7) << 4)) & 0x7f);  // 16-byte units XORed with the row
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(at + q * FT_TILE) = part[q];
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
                ft_wait_ld();
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c * 16 + j] += v[j];
            }
            ft_fence_before();
        };
        if (kb0 < kb1) fetch(kb0);
        // Block it may overwrite stage it & 1 and accumulator it & 1 once block it - 2 has been added up: promote() of it - 2 waited for its
        // MMAs, and every warp arrives on full[] after that.
        for (int it = 0; it < kb1 - kb0; ++it) {
            unsigned char* st = sm + (it & 1) * F1_STAGE;
#pragma unroll
            for (int i = 0; i < NF; ++i) {
                const int r = r0 + RS * i;
                if (r < rows) put(st, r, px[i]);
                if (r < cols) put(st + 3 * FT_TILE, r, pw[i]);
            }
            if (kb0 + it + 1 < kb1) fetch(kb0 + it + 1);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) ft_bar_arrive(ft_smem(&full[it & 1]));
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
            const uint32_t base = ft_smem(sm + (it & 1) * F1_STAGE), d = tmem + (it & 1) * 128;
            // (x part, W part), the small products first: 0 hi, 1 mid, 2 lo
            constexpr int PX[6] = {1, 0, 2, 0, 1, 0}, PW[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
            for (int p = 0; p < 6; ++p)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t xd = ft_desc_lo(base + PX[p] * FT_TILE) + 2 * k, wd = ft_desc_lo(base + (3 + PW[p]) * FT_TILE) + 2 * k;
                    if (k == 0 && (p == 3 || p == 5)) f1_mma<8>(d, xd, wd, 1u);  // the scale of the parts changes: 2^16, 2^8, 1
                    else f1_mma<0>(d, xd, wd, (p | k) ? 1u : 0u);
                }
            f1_commit(&done[it & 1]);
        }
    }
    ft_fence_before();
    __syncthreads();  // every MMA has completed (the last promote waited for it): the stages are free
    ft_fence_after();
    float(*sum)[F1_LD] = reinterpret_cast<float(*)[F1_LD]>(sm);
    if (warp < F1_WARPS) {
        const int r = (warp & 3) * 32 + lane, c = (warp >> 2) * NC;
#pragma unroll
        for (int j = 0; j < NC; j += 4) *reinterpret_cast<float4*>(&sum[r][c + j]) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
    }
    if (warp == F1_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u));
    int mark = 0;
    if (splits > 1) {
        ft_cluster_sync();
        for (int s = 0; s < splits; ++s) mark |= __float_as_int(f1_ld_cluster(ft_smem(&flags), s));
    } else {
        __syncthreads();
        mark = flags;
    }
    // this CTA's share of the tile's rows: sums over the ranks in order, then the step that follows the Linear, a pair of columns per thread
    const int share = F1_BM / splits, first = rank * share;
    if (mark == 1) {
        if (rows > first)
            ft_fma_rows<VEC, F1_THREADS>(a, X + (size_t)first * a.x_pitch(), W, reinterpret_cast<float*>(sm), m0 + first, n0, min(share, rows - first), cols, false);
    } else {
        for (int i = tid; i < share * (FT_BN / 2); i += F1_THREADS) {
            const int r = first + i / (FT_BN / 2), c = (i % (FT_BN / 2)) * 2;
            if (r >= rows || c >= cols) continue;
            float v0 = 0.f, v1 = 0.f;
            if (mark & 2) {
                v0 = v1 = __int_as_float(0x7fffffff);
            } else if (splits > 1) {
                for (int s = 0; s < splits; ++s) { v0 += f1_ld_cluster(ft_smem(&sum[r][c]), s); v1 += f1_ld_cluster(ft_smem(&sum[r][c + 1]), s); }
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
    const int tiles_n = (a.N + FT_BN - 1) / FT_BN, tiles_m = (a.M + F1_BM - 1) / F1_BM, nkb = (a.K + FT_BK - 1) / FT_BK;
    // split k until the CTAs fill the chip (148 SMs, one CTA each), at least four k-blocks a part
    int splits = 1;
    while (splits < 8 && (long long)tiles_n * tiles_m * splits * 2 <= 160 && nkb >= 8 * splits) splits *= 2;
    const bool vec = a.K % 4 == 0 && a.x_pitch() % 4 == 0 && (reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.w)) % 16 == 0;
    auto kernel = vec ? linear_f32_parts<true> : linear_f32_parts<false>;
    cudaError_t e = vec ? device_info::allow_shared<linear_f32_parts<true>>(F1_SMEM) : device_info::allow_shared<linear_f32_parts<false>>(F1_SMEM);
    if (e) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)tiles_n * (unsigned)tiles_m * (unsigned)splits);
    cfg.blockDim = dim3(F1_THREADS);
    cfg.dynamicSmemBytes = F1_SMEM;
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
