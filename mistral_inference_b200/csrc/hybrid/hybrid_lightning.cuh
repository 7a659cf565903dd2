// Lightning attention of prompts in chunks, on tensor cores (bf16 storage, fp32 state).
//
//     S_i = a S_(i-1) + k_i v_i^T,   o_i = S_i^T q_i          per head, a the head's decay
//
// is, inside a chunk of C tokens that starts from state S,
//
//     o_i = a^(i+1) S^T q_i + sum_(j <= i) a^(i-j) (q_i . k_j) v_j,        S' = a^C S + sum_j a^(C-1-j) k_j v_j^T:
//
// three small matrix products instead of C dependent updates of d x e numbers (the scan of hybrid_mixers.cuh, one column per thread, is a chain of
// T steps on H CTAs: 4.6 ms for 4096 tokens whatever the width).  Here a CTA walks the chunks of one (sequence, head, 32 value columns)
// with the state in registers: 32 heads x 4 column blocks = 128 CTAs, about 10 MFLOP a chunk on mma.sync; 4.6 -> 0.32 ms.  What bounds it now
// is the chain from chunk to chunk (about 5 us each: the parts, two barriers, 100 products a warp), not the products.
//
// Nothing that was 32 bits wide loses any: q, k, v are bf16 as stored; the state, the decayed values a^(C-1-j) v_j and the decayed scores
// a^(i-j) (q_i . k_j) are fp32 and enter the products as three bf16 parts each (8 + 8 + 8 significant bits: the parts add up to the
// number exactly or to its last bit; of numbers below 2^-110 what lies under bf16's smallest, 2^-133, is gone), accumulated in fp32; powers of the
// decay come from a table made in double precision.
// A chunk with an infinity or a NaN anywhere (or in the state) is walked token by token instead, so that a token's numbers reach no earlier one.
#pragma once
#include "hybrid_attn_flash.cuh"

namespace mbh {

constexpr int LC_C = 64, LC_E = 32, LC_THREADS = 256, LC_VP = LC_E + 8;

template <int D> struct LcSmem {
    static constexpr int KP = D + 8;
    bf16 q[2][LC_C * KP], k[2][LC_C * KP], v[2][LC_C * LC_VP];
    bf16 vd[3][LC_C * LC_VP];      // a^(C-1-j) v_j in three parts
    bf16 s[3][LC_E * KP];          // the chunk's start state, transposed (row: value column), in three parts
    float o[LC_C][LC_E + 4];       // a^(i+1) S^T q_i
    float pw[LC_C + 1];
};

// x = hi + mid + lo, 8 significant bits each (truncated, so hi never overflows)
__device__ __forceinline__ void split3(float x, float& hi, float& mid, float& lo) {
    hi = __uint_as_float(__float_as_uint(x) & 0xffff0000u);
    const float r = x - hi;
    mid = __uint_as_float(__float_as_uint(r) & 0xffff0000u);
    lo = r - mid;
}
// two numbers -> three registers of bf16 pairs
__device__ __forceinline__ void split3_pack(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    float xh, xm, xl, yh, ym, yl;
    split3(x, xh, xm, xl);
    split3(y, yh, ym, yl);
    hi = pack_bf16(xh, yh); mid = pack_bf16(xm, ym); lo = pack_bf16(xl, yl);
}

template <int D>
__global__ void __launch_bounds__(LC_THREADS) lightning_chunk_kernel(LightningArgs a) {
    using S_ = LcSmem<D>;
    constexpr int KP = S_::KP;
    constexpr int NT = D > 64 ? 2 : 1;  // a warp's part of the transposed state: 32 rows x 8 NT columns (D = 32: four of the warps have one)
    extern __shared__ __align__(16) unsigned char lc_smem[];
    S_& sm = *reinterpret_cast<S_*>(lc_smem);
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, c0 = blockIdx.y * LC_E;
    const int t0 = a.q_start[b], t1 = a.q_start[b + 1];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
    const int stride = 2 * a.H * D + 2 * a.H * a.e;
    const bf16* X = static_cast<const bf16*>(a.qkvg);
    float* st = a.state + (((size_t)a.slots[b] * a.H + h) * D) * a.e + c0;
    const float dec = a.decay[h];
    if (tid <= LC_C) {
        double p = 1.0;
        for (int i = 0; i < tid; ++i) p *= (double)dec;
        sm.pw[tid] = (float)p;
    }
    // state: transposed, rows = value columns: tile (mt, nt) element (mt * 16 + gid (+8), warp * D / 8 + nt * 8 + tig * 2 (+1))
    const bool fresh = a.seqpos[b] == 0;
    float S[2][NT][4];
    const bool has_state = warp * 8 * NT < D;
    const int d0 = warp * 8 * NT;
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int col = mt * 16 + gid + (r >> 1) * 8, d = d0 + nt * 8 + tig * 2 + (r & 1);
                S[mt][nt][r] = has_state && !fresh ? st[(size_t)d * a.e + col] : 0.f;
            }
    auto load = [&](int tb, int stage) {
        const int n = t1 - tb;
#pragma unroll 4
        for (int c = tid; c < 2 * LC_C * (D / 8); c += LC_THREADS) {
            const int which = c / (LC_C * (D / 8)), rem = c % (LC_C * (D / 8)), r = rem / (D / 8), kc = (rem % (D / 8)) * 8;
            const bool ok = r < n;
            cp_async16((which ? sm.k[stage] : sm.q[stage]) + r * KP + kc, ok ? X + (size_t)(tb + r) * stride + (which ? a.H * D : 0) + h * D + kc : X, ok);
        }
        {
            const int r = tid >> 2, ec = (tid & 3) * 8;
            const bool ok = r < n;
            cp_async16(sm.v[stage] + r * LC_VP + ec, ok ? X + (size_t)(tb + r) * stride + 2 * a.H * D + h * a.e + c0 + ec : X, ok);
        }
        cp_async_commit();
    };
    if (t0 < t1) load(t0, 0);
    int stage = 0;
    for (int tb = t0; tb < t1; tb += LC_C, stage ^= 1) {
        const int n = min(LC_C, t1 - tb);
        if (tb + LC_C < t1) { load(tb + LC_C, stage ^ 1); cp_async_wait<1>(); }
        else cp_async_wait<0>();
        __syncthreads();  // the tiles have landed; everybody is done with vd, s and o of the chunk before
        const bf16 *sq = sm.q[stage], *sk = sm.k[stage], *sv = sm.v[stage];
        int bad = 0;
        {
            const int r = tid >> 2, ec = (tid & 3) * 8;
            float x[8];
            Vec<bf16>::load(sv + r * LC_VP + ec, x);
            const float f = r < n ? sm.pw[n - 1 - r] : 0.f;
            uint32_t p[3][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                bad |= not_finite(x[2 * i]) | not_finite(x[2 * i + 1]);
                split3_pack(x[2 * i] * f, x[2 * i + 1] * f, p[0][i], p[1][i], p[2][i]);
            }
#pragma unroll
            for (int q = 0; q < 3; ++q) *reinterpret_cast<uint4*>(sm.vd[q] + r * LC_VP + ec) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
        }
#pragma unroll 4
        for (int c = tid; c < 2 * LC_C * (D / 8); c += LC_THREADS) {
            const int which = c / (LC_C * (D / 8)), rem = c % (LC_C * (D / 8)), r = rem / (D / 8), kc = (rem % (D / 8)) * 8;
            const uint4 u = *reinterpret_cast<const uint4*>((which ? sk : sq) + r * KP + kc);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) bad |= ((w[i] & 0x7f80u) == 0x7f80u) | ((w[i] & 0x7f800000u) == 0x7f800000u);
        }
        if (has_state) {
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        const float x = S[mt][nt][2 * hf], y = S[mt][nt][2 * hf + 1];
                        bad |= not_finite(x) | not_finite(y);
                        uint32_t p[3];
                        split3_pack(x, y, p[0], p[1], p[2]);
                        const int at = (mt * 16 + gid + 8 * hf) * KP + d0 + nt * 8 + tig * 2;
#pragma unroll
                        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint32_t*>(sm.s[q] + at) = p[q];
                    }
        }
        if (__syncthreads_or(bad)) {
            // token by token: thread (column, eighth of the keys); the state passes through shared memory (over vd and s)
            float* sf = reinterpret_cast<float*>(sm.vd[0]);  // [LC_E][D + 1]
            static_assert(sizeof(float) * LC_E * (D + 1) <= sizeof(sm.vd) + sizeof(sm.s), "the state fits");
            float(*red)[LC_E + 4] = sm.o;
            const int col = tid & 31, g = tid >> 5;
            if (has_state)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int r = 0; r < 4; ++r) sf[(mt * 16 + gid + (r >> 1) * 8) * (D + 1) + d0 + nt * 8 + tig * 2 + (r & 1)] = S[mt][nt][r];
            __syncthreads();
            float* mine = sf + col * (D + 1) + g * (D / 8);
            for (int i = 0; i < n; ++i) {
                const float v = to_f(sv[i * LC_VP + col]);
                float o = 0.f;
                for (int d = 0; d < D / 8; ++d) {
                    const float s = fmaf(dec, mine[d], to_f(sk[i * KP + g * (D / 8) + d]) * v);
                    mine[d] = s;
                    o = fmaf(s, to_f(sq[i * KP + g * (D / 8) + d]), o);
                }
                red[g][col] = o;
                __syncthreads();
                if (g == 0) {
                    float sum = 0.f;
                    for (int q = 0; q < 8; ++q) sum += red[q][col];
                    a.o[(size_t)(tb + i) * a.H * a.e + h * a.e + c0 + col] = sum;
                }
                __syncthreads();
            }
            if (has_state)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                        for (int r = 0; r < 4; ++r) S[mt][nt][r] = sf[(mt * 16 + gid + (r >> 1) * 8) * (D + 1) + d0 + nt * 8 + tig * 2 + (r & 1)];
            __syncthreads();
            continue;
        }
        const int mi = warp & 3;  // 16 query rows
        const bool live = mi * 16 < n;
        float o[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) o[nt][0] = o[nt][1] = o[nt][2] = o[nt][3] = 0.f;
        const bf16* qa = sq + (mi * 16 + (lane & 15)) * KP + (lane >> 4) * 8;
        if (warp >= 4 && live) {
            // a^(i+1) q_i . S
            const bf16* sb = sm.s[0] + ((lane >> 4) * 8 + (lane & 7)) * KP + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int part = 2; part >= 0; --part)
#pragma unroll
                for (int kk = 0; kk < D / 16; ++kk) {
                    uint32_t qf[4];
                    ldmatrix4(qf, qa + kk * 16);
#pragma unroll
                    for (int np = 0; np < 2; ++np) {
                        uint32_t bf[4];
                        ldmatrix4(bf, sb + part * LC_E * KP + np * 16 * KP + kk * 16);
                        mma_bf16(o[2 * np], qf, bf[0], bf[1]);
                        mma_bf16(o[2 * np + 1], qf, bf[2], bf[3]);
                    }
                }
            const float w0 = sm.pw[mi * 16 + gid + 1], w1 = sm.pw[mi * 16 + gid + 9];
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                *reinterpret_cast<float2*>(&sm.o[mi * 16 + gid][nt * 8 + tig * 2]) = make_float2(w0 * o[nt][0], w0 * o[nt][1]);
                *reinterpret_cast<float2*>(&sm.o[mi * 16 + gid + 8][nt * 8 + tig * 2]) = make_float2(w1 * o[nt][2], w1 * o[nt][3]);
            }
        } else if (live) {
            float s[8][4];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.f;
            const bf16* kb = sk + ((lane >> 4) * 8 + (lane & 7)) * KP + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                uint32_t qf[4];
                ldmatrix4(qf, qa + kk * 16);
#pragma unroll
                for (int np = 0; np < 4; ++np)
                    if (np <= mi) {  // keys after the last row of this warp: nothing
                        uint32_t kf[4];
                        ldmatrix4(kf, kb + np * 16 * KP + kk * 16);
                        mma_bf16(s[2 * np], qf, kf[0], kf[1]);
                        mma_bf16(s[2 * np + 1], qf, kf[2], kf[3]);
                    }
            }
            const bf16* vb = sv + (((lane >> 3) & 1) * 8 + (lane & 7)) * LC_VP + (lane >> 4) * 8;
            const int i0 = mi * 16 + gid, i1 = i0 + 8;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                if (kk <= mi) {
                    uint32_t p[3][4];
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        const int j = kk * 16 + u * 8 + tig * 2;
                        const float* sc = s[2 * kk + u];
                        split3_pack(j <= i0 ? sc[0] * sm.pw[i0 - j] : 0.f, j + 1 <= i0 ? sc[1] * sm.pw[i0 - j - 1] : 0.f, p[0][2 * u], p[1][2 * u], p[2][2 * u]);
                        split3_pack(j <= i1 ? sc[2] * sm.pw[i1 - j] : 0.f, j + 1 <= i1 ? sc[3] * sm.pw[i1 - j - 1] : 0.f, p[0][2 * u + 1], p[1][2 * u + 1], p[2][2 * u + 1]);
                    }
#pragma unroll
                    for (int np = 0; np < 2; ++np) {
                        uint32_t vf[4];
                        ldmatrix4_trans(vf, vb + kk * 16 * LC_VP + np * 16);
#pragma unroll
                        for (int part = 2; part >= 0; --part) {
                            mma_bf16(o[2 * np], p[part], vf[0], vf[1]);
                            mma_bf16(o[2 * np + 1], p[part], vf[2], vf[3]);
                        }
                    }
                }
        }
        // S' = a^n S + sum_j (a^(n-1-j) v_j) k_j^T
        if (has_state) {
            float u[2][NT][4];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt) u[mt][nt][0] = u[mt][nt][1] = u[mt][nt][2] = u[mt][nt][3] = 0.f;
            const bf16* va = sm.vd[0] + ((lane >> 4) * 8 + (lane & 7)) * LC_VP + ((lane >> 3) & 1) * 8;
            const bf16* kb = sk + (((lane >> 3) & 1) * 8 + (lane & 7)) * KP + d0 + (NT == 2 ? (lane >> 4) * 8 : 0);
#pragma unroll
            for (int kk = 0; kk < LC_C / 16; ++kk) {
                uint32_t kf[4];
                ldmatrix4_trans(kf, kb + kk * 16 * KP);
#pragma unroll
                for (int part = 2; part >= 0; --part)
#pragma unroll
                    for (int mt = 0; mt < 2; ++mt) {
                        uint32_t vf[4];
                        ldmatrix4_trans(vf, va + part * LC_C * LC_VP + kk * 16 * LC_VP + mt * 16);
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) mma_bf16(u[mt][nt], vf, kf[2 * nt], kf[2 * nt + 1]);
                    }
            }
            const float f = sm.pw[n];
#pragma unroll
            for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int r = 0; r < 4; ++r) S[mt][nt][r] = fmaf(f, S[mt][nt][r], u[mt][nt][r]);
        }
        __syncthreads();
        if (warp < 4 && live) {
            const int i0 = mi * 16 + gid, i1 = i0 + 8;
            float* out = a.o + (size_t)tb * a.H * a.e + h * a.e + c0 + tig * 2;
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) {
                const float2 x = *reinterpret_cast<const float2*>(&sm.o[i0][nt * 8 + tig * 2]), y = *reinterpret_cast<const float2*>(&sm.o[i1][nt * 8 + tig * 2]);
                if (i0 < n) *reinterpret_cast<float2*>(out + (size_t)i0 * a.H * a.e + nt * 8) = make_float2(x.x + o[nt][0], x.y + o[nt][1]);
                if (i1 < n) *reinterpret_cast<float2*>(out + (size_t)i1 * a.H * a.e + nt * 8) = make_float2(y.x + o[nt][2], y.y + o[nt][3]);
            }
        }
    }
    if (has_state)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int r = 0; r < 4; ++r) st[(size_t)(d0 + nt * 8 + tig * 2 + (r & 1)) * a.e + mt * 16 + gid + (r >> 1) * 8] = S[mt][nt][r];
}

template <int D> inline cudaError_t run_lightning_chunk(const LightningArgs& a, cudaStream_t st) {
    const cudaError_t e = cudaFuncSetAttribute(lightning_chunk_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LcSmem<D>));
    if (e) return e;
    lightning_chunk_kernel<D><<<dim3((unsigned)(a.B * a.H), (unsigned)(a.e / LC_E)), LC_THREADS, sizeof(LcSmem<D>), st>>>(a);
    return cudaGetLastError();
}

}  // namespace mbh
