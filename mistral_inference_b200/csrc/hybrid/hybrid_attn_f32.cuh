// Prompt attention in true fp32 (fp32 storage): flash-style, one CTA per (32-query tile, head), FMAs out of shared memory.
//
// attn_bias_kernel gives every (token, head) a CTA of its own, which reads each of its keys a lane at a time: ~800 queries x 16 heads over ~270 keys of 128 took 496 us for
// 0.9 GFLOP.  Here 32 queries share the keys: tiles of 32 keys and values come by cp.async, two stages; 256 threads form the 32 x 32 scores (2 queries x 2 keys each:
// 4 16-byte loads for 16 FMAs, a dot product is one chain over d as before), the running (maximum, sum) of a query lives in the 16 lanes that hold its scores, and the weights
// go transposed through shared memory to the threads that own 4 queries x E / 32 columns of the output.  68 us.  What bounds it now: the loads out of shared
// memory (about 1.5 cycles to each of FMA) and, for prompts this short, the few tiles in flight.  Few rows over many keys, whose tiles would be a handful of CTAs that
// walk all keys in turn, stay with attn_bias_kernel (the caller's choice).
//
// Bias, soft cap, sinks, gates, windows, chunks and rings as in attn_bias_kernel.  A key that a query does not see enters nothing, whatever its numbers: on tiles that
// some query's range cuts, products are taken by index and not by a weight of zero (0 x infinity).
#pragma once
#include "hybrid_mixers.cuh"

namespace mbh {

constexpr int F3_BQ = 32, F3_BK = 32, F3_THREADS = 256, F3_PP = F3_BQ + 4;

template <int D, int E> struct F3Smem {
    static constexpr int KP = D + 4;  // rows 16 bytes apart in the banks
    float q[F3_BQ * KP], k[2][F3_BK * KP], v[2][F3_BK * E], pt[F3_BK * F3_PP], corr[F3_BQ], l[F3_BQ];
};

__device__ __forceinline__ void f3_copy16(float* dst, const float* src, bool ok) {
    const uint32_t addr = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(addr), "l"(src), "r"(ok ? 16 : 0));
}

template <int D, int E>
__global__ void __launch_bounds__(F3_THREADS, 2) attn_f32_kernel(AttnArgs a) {
    using S_ = F3Smem<D, E>;
    constexpr int KP = S_::KP, CPL = E / 32;  // output columns of a thread
    extern __shared__ __align__(16) float f3_raw[];
    S_& sm = *reinterpret_cast<S_*>(f3_raw);
    const int h = blockIdx.x, g = h / (a.H / a.G), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // tile blockIdx.y of all sequences' tiles, the last (longest) ones first
    int idx = (int)gridDim.y - 1 - (int)blockIdx.y, b = 0;
    for (; b < a.B; ++b) {
        const int tiles = (a.q_start[b + 1] - a.q_start[b] + F3_BQ - 1) / F3_BQ;
        if (idx < tiles) break;
        idx -= tiles;
    }
    if (b == a.B) return;
    const int t0 = a.q_start[b] + idx * F3_BQ, nq = min(F3_BQ, a.q_start[b + 1] - t0), pos0 = a.positions[t0];
    const size_t base = (size_t)a.slots[b] * a.W, kr = (size_t)a.G * D, vr = (size_t)a.G * E;
    const int own_from = a.own_k ? a.seqpos[b] : 0x7fffffff;
    const size_t own_row = a.own_k ? (size_t)a.q_start[b] : 0;
    const KeySource<float> K{static_cast<const float*>(a.cache_k) + base * kr + (size_t)g * D, static_cast<const float*>(a.own_k) + own_row * kr + (size_t)g * D, kr, kr, a.W, own_from};
    const KeySource<float> V{static_cast<const float*>(a.cache_v) + base * vr + (size_t)g * E, static_cast<const float*>(a.own_v) + own_row * vr + (size_t)g * E, vr, vr, a.W, own_from};
    const int lo = first_key(a, pos0), hi = pos0 + nq;  // keys lo .. hi - 1
    for (int i = tid; i < F3_BQ * (D / 4); i += F3_THREADS) {
        const int r = i / (D / 4), c = (i % (D / 4)) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < nq) v = *reinterpret_cast<const float4*>(static_cast<const float*>(a.q) + ((size_t)(t0 + r) * a.H + h) * D + c);
        *reinterpret_cast<float4*>(sm.q + r * KP + c) = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
    }
    auto load = [&](int j0, int stage) {  // eight threads to a row
        const int r = tid >> 3, j = j0 + r;
        const bool ok = j < hi;
        const float* ks = K.row(ok ? j : lo);
        const float* vs = V.row(ok ? j : lo);
#pragma unroll
        for (int c = (tid & 7) * 4; c < D; c += 32) f3_copy16(sm.k[stage] + r * KP + c, ks + c, ok);
#pragma unroll
        for (int c = (tid & 7) * 4; c < E; c += 32) f3_copy16(sm.v[stage] + r * E + c, vs + c, ok);
        asm volatile("cp.async.commit_group;\n");
    };
    load(lo, 0);
    const int tq = tid >> 4, tk = tid & 15;  // scores: queries 2 tq, 2 tq + 1; keys tk, tk + 16
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f}, acc[4][CPL];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < CPL; ++c) acc[i][c] = 0.f;
    int from[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) from[i] = first_key(a, pos0 + 2 * tq + i);
    int stage = 0;
    for (int j0 = lo; j0 < hi; j0 += F3_BK, stage ^= 1) {
        if (j0 + F3_BK < hi) {
            load(j0 + F3_BK, stage ^ 1);
            asm volatile("cp.async.wait_group 1;\n");
        } else {
            asm volatile("cp.async.wait_group 0;\n");
        }
        __syncthreads();
        const float *sk = sm.k[stage] + tk * KP, *sq = sm.q + 2 * tq * KP;
        float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll 8
        for (int c = 0; c < D; c += 4) {
            const float4 q0 = *reinterpret_cast<const float4*>(sq + c), q1 = *reinterpret_cast<const float4*>(sq + KP + c);
            const float4 k0 = *reinterpret_cast<const float4*>(sk + c), k1 = *reinterpret_cast<const float4*>(sk + 16 * KP + c);
            s[0][0] = fmaf(q0.w, k0.w, fmaf(q0.z, k0.z, fmaf(q0.y, k0.y, fmaf(q0.x, k0.x, s[0][0]))));
            s[0][1] = fmaf(q0.w, k1.w, fmaf(q0.z, k1.z, fmaf(q0.y, k1.y, fmaf(q0.x, k1.x, s[0][1]))));
            s[1][0] = fmaf(q1.w, k0.w, fmaf(q1.z, k0.z, fmaf(q1.y, k0.y, fmaf(q1.x, k0.x, s[1][0]))));
            s[1][1] = fmaf(q1.w, k1.w, fmaf(q1.z, k1.z, fmaf(q1.y, k1.y, fmaf(q1.x, k1.x, s[1][1]))));
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int pos = pos0 + 2 * tq + i;
            bool sees[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int j = j0 + tk + 16 * k;
                sees[k] = j <= pos && j >= from[i];
                if (a.softcap > 0.f) s[i][k] = a.softcap * tanhf(s[i][k] / a.softcap);
                if (a.bias_tab && sees[k]) s[i][k] += a.bias_tab[(size_t)min(pos - j, a.n_tab - 1) * a.H + h];
                if (!sees[k]) s[i][k] = -INFINITY;
            }
            float mx = fmaxf(s[i][0], s[i][1]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            mx = fmaxf(m[i], mx);
            const float z = mx == -INFINITY ? 0.f : mx;  // keys of nothing but -infinity so far weigh 0 (-infinity less itself is no number)
            const float f = m[i] == -INFINITY ? 0.f : expf(m[i] - z);
            float p[2], sum;
#pragma unroll
            for (int k = 0; k < 2; ++k) p[k] = sees[k] ? expf(s[i][k] - z) : 0.f;
            sum = p[0] + p[1];
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l[i] = l[i] * f + sum;
            m[i] = mx;
            sm.pt[tk * F3_PP + 2 * tq + i] = p[0];
            sm.pt[(tk + 16) * F3_PP + 2 * tq + i] = p[1];
            if (tk == 0) sm.corr[2 * tq + i] = f;
        }
        __syncthreads();
        const float* sv = sm.v[stage] + lane * CPL;
        const float* sp = sm.pt + 4 * warp;
        const float4 f4 = *reinterpret_cast<const float4*>(sm.corr + 4 * warp);
        const float f[4] = {f4.x, f4.y, f4.z, f4.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < CPL; ++c) acc[i][c] *= f[i];
        auto value = [&](int k, float (&v)[CPL]) {
            if constexpr (CPL == 4) {
                const float4 u = *reinterpret_cast<const float4*>(sv + k * E);
                v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w;
            } else {
                const float2 u = *reinterpret_cast<const float2*>(sv + k * E);
                v[0] = u.x; v[1] = u.y;
            }
        };
        const int qp = pos0 + 4 * warp;
        if (j0 + F3_BK - 1 <= qp && j0 >= first_key(a, qp + 3)) {  // every query of this warp sees the whole tile (first_key grows with the position)
#pragma unroll 8
            for (int k = 0; k < F3_BK; ++k) {
                const float4 p = *reinterpret_cast<const float4*>(sp + k * F3_PP);
                float v[CPL];
                value(k, v);
#pragma unroll
                for (int c = 0; c < CPL; ++c) {
                    acc[0][c] = fmaf(p.x, v[c], acc[0][c]);
                    acc[1][c] = fmaf(p.y, v[c], acc[1][c]);
                    acc[2][c] = fmaf(p.z, v[c], acc[2][c]);
                    acc[3][c] = fmaf(p.w, v[c], acc[3][c]);
                }
            }
        } else {
            int first[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) first[i] = first_key(a, qp + i);
#pragma unroll 4
            for (int k = 0; k < F3_BK; ++k) {
                const float4 p4 = *reinterpret_cast<const float4*>(sp + k * F3_PP);
                const float p[4] = {p4.x, p4.y, p4.z, p4.w};
                float v[CPL];
                value(k, v);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (j0 + k <= qp + i && j0 + k >= first[i]) {
#pragma unroll
                        for (int c = 0; c < CPL; ++c) acc[i][c] = fmaf(p[i], v[c], acc[i][c]);
                    }
            }
        }
        __syncthreads();  // the stage, the weights and the factors are free
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (tk == 0) sm.l[2 * tq + i] = a.sink ? sink_denominator(m[i], l[i], a.sink[h]) : l[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 4 * warp + i;
        if (r >= nq) continue;
        float* out = static_cast<float*>(a.out) + ((size_t)(t0 + r) * a.H + h) * E + lane * CPL;
        float y[CPL];
#pragma unroll
        for (int c = 0; c < CPL; ++c) y[c] = acc[i][c] / sm.l[r] * out_gate<float>(a.gate, a.gate_pitch, a.gate_entry, t0 + r, h, E, lane * CPL + c);
        if constexpr (CPL == 4) *reinterpret_cast<float4*>(out) = make_float4(y[0], y[1], y[2], y[3]);
        else *reinterpret_cast<float2*>(out) = make_float2(y[0], y[1]);
    }
}

template <int D, int E> inline cudaError_t launch_attn_f32_de(const AttnArgs& a, int tiles, cudaStream_t st) {
    cudaError_t e = cudaFuncSetAttribute(attn_f32_kernel<D, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(F3Smem<D, E>));
    if (e) return e;
    attn_f32_kernel<D, E><<<dim3((unsigned)a.H, (unsigned)tiles), F3_THREADS, sizeof(F3Smem<D, E>), st>>>(a);
    return cudaGetLastError();
}
// Prompts of fp32 layers, softmax over one map per head, head sizes 64 and 128, rows of whole 16-byte pieces.  tiles64: 64-query tiles of all sequences; twice as many
// of 32 are at least enough (the rest leave at once).  false: attn_bias_kernel.
inline bool launch_attn_f32(const AttnArgs& a, int64_t tiles64, cudaStream_t st, cudaError_t& err) {
    if (a.maps != 1 || a.sigmoid || a.k_pitch || a.v_pitch || a.own_k_pitch || a.own_v_pitch || 2 * tiles64 > 65535) return false;
    const uintptr_t p = reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.cache_k) | reinterpret_cast<uintptr_t>(a.cache_v) | reinterpret_cast<uintptr_t>(a.out) |
                        reinterpret_cast<uintptr_t>(a.own_k) | reinterpret_cast<uintptr_t>(a.own_v);
    if (p % 16) return false;
    if (a.d == 128 && a.e == 128) err = launch_attn_f32_de<128, 128>(a, (int)(2 * tiles64), st);
    else if (a.d == 64 && a.e == 64) err = launch_attn_f32_de<64, 64>(a, (int)(2 * tiles64), st);
    else return false;
    return true;
}

}  // namespace mbh
