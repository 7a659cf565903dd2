// Decode attention on tensor cores (bf16 storage): one token per sequence, every key and value row read once for all query heads of its group.
//
// grid (sequence * key/value head, splits), four warps.  The (up to 16) query heads of the group are the M side of m16n8k16 tiles; every warp walks
// its own 16-key pieces of the ring (pieces are dealt out over warps and splits) with its own running (max, sum) and value accumulators, its
// pieces arriving by cp.async in a private ring of DA_STAGES buffers -- warps never wait for one another before the end, when they are merged
// through shared memory.  The splits' partial results have the layout of attn_bias_kernel's and go through the same merge kernels (sinks,
// differences of two maps, gates).  With MAPS 2 both maps of a head are computed here: their keys are one row, their values are shared.
// BIAS: AttnArgs::bias_tab is added to the scores by distance, and the weights stay 32 bits wide -- they multiply the values as three bf16 parts
// (hybrid_lightning.cuh); they come from ex2.approx in log2 units, a few 2^-23 each, where the fp32 kernel of hybrid_mixers.cuh that these layers ran on
// has expf.  A step's error against float64 is 0.00676 here and 0.00675 there (bf16 roundings).  That kernel reads a ring row once per query head:
// 116 us for 8 sequences of ~1800 tokens, 16 / 4 heads, against 16 us here and 4 us of merging.
#pragma once
#include "hybrid_lightning.cuh"

namespace mbh {

constexpr int DA_WARPS = 4, DA_KEYS = 16, DA_STAGES = 3, DA_MAX_GROUP = 16;

template <int D, int E, int MAPS> constexpr size_t attn_decode_smem() {
    constexpr size_t stages = sizeof(bf16) * (size_t)DA_WARPS * DA_STAGES * DA_KEYS * (MAPS * D + 8 + E + 8);
    constexpr size_t merge = sizeof(float) * (size_t)DA_WARPS * MAPS * 16 * (E + 2);
    return stages > merge ? stages : merge;
}

// The warps' results, [warp][map][row] of (max in log2 units, sum, E values), to one per (query head, map): this split's partial result
template <int E, int MAPS>
__device__ __forceinline__ void merge_warps(const AttnArgs& a, const float* mrg, int b, int g, int R, int split) {
    constexpr float LN2 = 0.6931471805599453f;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int rm = warp; rm < R * MAPS; rm += DA_WARPS) {  // a warp per (query head, map)
        const int row = rm / MAPS, m = rm % MAPS;
        const float* p = mrg + ((size_t)m * 16 + row) * (E + 2);
        constexpr size_t WS = (size_t)MAPS * 16 * (E + 2);
        float M = -INFINITY, L = 0.f, f[DA_WARPS];
#pragma unroll
        for (int w = 0; w < DA_WARPS; ++w) M = fmaxf(M, p[w * WS]);
#pragma unroll
        for (int w = 0; w < DA_WARPS; ++w) {
            f[w] = p[w * WS] == -INFINITY ? 0.f : exp2_fast(p[w * WS] - M);
            L += f[w] * p[w * WS + 1];
        }
        float* out = a.scratch + ((((size_t)b * a.H + g * R + row) * MAPS + m) * a.splits + split) * (2 + E);
        if (lane == 0) { out[0] = M * LN2; out[1] = L; }
        for (int c = lane; c < E; c += 32) {
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < DA_WARPS; ++w) v = fmaf(f[w], p[w * WS + 2 + c], v);
            out[2 + c] = v;
        }
    }
}

template <int D, int E, int MAPS, bool BIAS = false>
__global__ void __launch_bounds__(DA_WARPS * 32) attn_decode_mma_kernel(AttnArgs a) {
    static_assert(!BIAS || MAPS == 1, "a bias with two maps is not built");
    constexpr int PARTS = BIAS ? 3 : 1;
    constexpr int KP = MAPS * D + 8, VP = E + 8, STAGE = DA_KEYS * (KP + VP);
    constexpr float LOG2E = 1.4426950408889634f;
    extern __shared__ __align__(16) unsigned char da_smem[];
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.x / a.G, g = blockIdx.x % a.G, R = a.H / a.G, split = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    bf16* const mine = reinterpret_cast<bf16*>(da_smem) + warp * DA_STAGES * STAGE;
    const int pos = a.positions[b], lo = first_key(a, pos);
    const size_t base = (size_t)a.slots[b] * a.W, kstride = (size_t)a.G * MAPS * D, vstride = (size_t)a.G * E;
    const bf16* K = static_cast<const bf16*>(a.cache_k) + base * kstride + (size_t)g * MAPS * D;
    const bf16* V = static_cast<const bf16*>(a.cache_v) + base * vstride + (size_t)g * E;
    const bf16* Q = static_cast<const bf16*>(a.q) + ((size_t)b * a.H + g * R) * MAPS * D;

    const int step = a.splits * DA_WARPS * DA_KEYS;
    auto load = [&](int c0, int stage) {  // keys c0 .. c0 + 15 (those up to pos)
        bf16* ks = mine + stage * STAGE;
        bf16* vs = ks + DA_KEYS * KP;
        if (c0 <= pos) {
            const int s0 = c0 % a.W;
            constexpr int CK = MAPS * D / 8, CV = E / 8;
#pragma unroll
            for (int c = lane; c < DA_KEYS * CK; c += 32) {
                const int r = c / CK, kc = (c % CK) * 8, s = s0 + r;
                const bool ok = c0 + r <= pos;
                cp_async16(ks + r * KP + kc, ok ? K + (size_t)(s < a.W ? s : s % a.W) * kstride + kc : K, ok);
            }
#pragma unroll
            for (int c = lane; c < DA_KEYS * CV; c += 32) {
                const int r = c / CV, ec = (c % CV) * 8, s = s0 + r;
                const bool ok = c0 + r <= pos;
                cp_async16(vs + r * VP + ec, ok ? V + (size_t)(s < a.W ? s : s % a.W) * vstride + ec : V, ok);
            }
        }
        cp_async_commit();
    };
    const int first = lo + (split * DA_WARPS + warp) * DA_KEYS;
#pragma unroll
    for (int i = 0; i < DA_STAGES - 1; ++i) load(first + i * step, i);

    uint32_t qf[MAPS][D / 16][4];
#pragma unroll
    for (int m = 0; m < MAPS; ++m)
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int row = gid + (u & 1) * 8, col = kk * 16 + tig * 2 + (u >> 1) * 8;
                qf[m][kk][u] = row < R ? *reinterpret_cast<const uint32_t*>(Q + ((size_t)row * MAPS + m) * D + col) : 0u;
            }
    float o[MAPS][E / 8][4], mx[MAPS][2], l[MAPS][2];  // maxima in units of log2
#pragma unroll
    for (int m = 0; m < MAPS; ++m) {
        mx[m][0] = mx[m][1] = -INFINITY; l[m][0] = l[m][1] = 0.f;
#pragma unroll
        for (int ne = 0; ne < E / 8; ++ne) o[m][ne][0] = o[m][ne][1] = o[m][ne][2] = o[m][ne][3] = 0.f;
    }
    const bool capped = a.softcap > 0.f;
    const float unit = (capped ? 1.f : a.scale) * LOG2E, capf = capped ? 2.f * a.scale / a.softcap : 0.f;

    int stage = 0;
    for (int c0 = first; c0 <= pos; c0 += step) {
        load(c0 + (DA_STAGES - 1) * step, (stage + DA_STAGES - 1) % DA_STAGES);
        cp_async_wait<DA_STAGES - 1>();
        __syncwarp();
        const bf16* ks = mine + stage * STAGE;
        const bf16* vs = ks + DA_KEYS * KP;
        uint32_t pa[MAPS * PARTS][4];
        float bias[2][4];  // in log2 units, requested before the products
        if constexpr (BIAS) {
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int row = gid + (c >> 1) * 8, dist = min(max(pos - (c0 + nt * 8 + tig * 2 + (c & 1)), 0), a.n_tab - 1);
                    bias[nt][c] = row < R ? __ldg(a.bias_tab + (size_t)dist * a.H + g * R + row) * LOG2E : 0.f;
                }
        }
#pragma unroll
        for (int m = 0; m < MAPS; ++m) {
            float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            const bf16* kp = ks + ((lane >> 4) * 8 + (lane & 7)) * KP + m * D + ((lane >> 3) & 1) * 8;
#pragma unroll
            for (int kk = 0; kk < D / 16; ++kk) {
                uint32_t kf[4];
                ldmatrix4(kf, kp + kk * 16);
                mma_bf16(s[0], qf[m][kk], kf[0], kf[1]);
                mma_bf16(s[1], qf[m][kk], kf[2], kf[3]);
            }
            float t0 = -INFINITY, t1 = -INFINITY;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const bool ok = c0 + nt * 8 + tig * 2 + c <= pos;
                    float x0 = s[nt][c], x1 = s[nt][2 + c];
                    if (capped) { x0 = softcap_fast(x0, a.softcap, capf); x1 = softcap_fast(x1, a.softcap, capf); }
                    x0 = BIAS ? fmaf(x0, unit, bias[nt][c]) : x0 * unit;
                    x1 = BIAS ? fmaf(x1, unit, bias[nt][2 + c]) : x1 * unit;
                    s[nt][c] = ok ? x0 : -INFINITY; s[nt][2 + c] = ok ? x1 : -INFINITY;
                    t0 = fmaxf(t0, s[nt][c]); t1 = fmaxf(t1, s[nt][2 + c]);
                }
            // key c0 is visible, so the new maxima are finite
            t0 = fmaxf(mx[m][0], quad_max(t0)); t1 = fmaxf(mx[m][1], quad_max(t1));
            const float f0 = exp2_fast(mx[m][0] - t0), f1 = exp2_fast(mx[m][1] - t1);
            mx[m][0] = t0; mx[m][1] = t1;
            float q0 = 0.f, q1 = 0.f;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    s[nt][c] = exp2_fast(s[nt][c] - t0); s[nt][2 + c] = exp2_fast(s[nt][2 + c] - t1);
                    q0 += s[nt][c]; q1 += s[nt][2 + c];
                }
            l[m][0] = l[m][0] * f0 + q0; l[m][1] = l[m][1] * f1 + q1;
#pragma unroll
            for (int ne = 0; ne < E / 8; ++ne) { o[m][ne][0] *= f0; o[m][ne][1] *= f0; o[m][ne][2] *= f1; o[m][ne][3] *= f1; }
            if constexpr (BIAS) {
#pragma unroll
                for (int u = 0; u < 4; ++u) split3_pack(s[u >> 1][(u & 1) * 2], s[u >> 1][(u & 1) * 2 + 1], pa[0][u], pa[1][u], pa[2][u]);
            } else {
                pa[m][0] = pack_bf16(s[0][0], s[0][1]); pa[m][1] = pack_bf16(s[0][2], s[0][3]);
                pa[m][2] = pack_bf16(s[1][0], s[1][1]); pa[m][3] = pack_bf16(s[1][2], s[1][3]);
            }
        }
        const bf16* vp = vs + (((lane >> 3) & 1) * 8 + (lane & 7)) * VP + (lane >> 4) * 8;
#pragma unroll
        for (int np = 0; np < E / 16; ++np) {
            uint32_t vf[4];
            ldmatrix4_trans(vf, vp + np * 16);
#pragma unroll
            for (int m = 0; m < MAPS; ++m)
#pragma unroll
                for (int q = PARTS - 1; q >= 0; --q) {  // the smallest part first
                    mma_bf16(o[m][2 * np], pa[m * PARTS + q], vf[0], vf[1]);
                    mma_bf16(o[m][2 * np + 1], pa[m * PARTS + q], vf[2], vf[3]);
                }
        }
        __syncwarp();  // the buffer is used up
        stage = (stage + 1) % DA_STAGES;
    }
    cp_async_wait<0>();
    __syncthreads();
    // the warps' results: [warp][map][row] of (max, sum, E values)
    float* mrg = reinterpret_cast<float*>(da_smem);
#pragma unroll
    for (int m = 0; m < MAPS; ++m) {
        float* p0 = mrg + ((size_t)(warp * MAPS + m) * 16 + gid) * (E + 2);
        float* p1 = p0 + 8 * (E + 2);
        const float s0 = quad_sum(l[m][0]), s1 = quad_sum(l[m][1]);
        if (tig == 0) { p0[0] = mx[m][0]; p0[1] = s0; p1[0] = mx[m][1]; p1[1] = s1; }
#pragma unroll
        for (int ne = 0; ne < E / 8; ++ne) {
            const int col = 2 + ne * 8 + tig * 2;
            *reinterpret_cast<float2*>(p0 + col) = make_float2(o[m][ne][0], o[m][ne][1]);
            *reinterpret_cast<float2*>(p1 + col) = make_float2(o[m][ne][2], o[m][ne][3]);
        }
    }
    __syncthreads();
    merge_warps<E, MAPS>(a, mrg, b, g, R, split);
}

// The same for groups of up to 8 query heads and one map, with the KEYS as the MMAs' 16 rows and the heads as their 8 columns: S^T = K Q^T, O^T = V^T P^T (the
// weights change sides by movmatrix).  Half the MMAs of the kernel above, whose 16 rows a group of 4 heads fills to a quarter, half the accumulators to rescale (and only when a maximum
// grew), one score a lane and key pair, and the addresses of a piece that neither wraps nor ends inside reduced to one addition a copy: what bounds both is the instructions of a
// warp's piece (985 above, eight warps an SM, 5 clocks each), then latency.  us with the merge, 16 / 4 heads: 8 sequences of ~1800 tokens 20.0, 14.7; 32 / 8 heads, 16 sequences of
// ~2600 71.7, 42.0 (4.1 TB/s), of ~430 18.7, 14.9, of which 17.1, 50.3 and 16.2 with the number of splits as it was (a few CTAs more than run at once).  Three CTAs an SM with two stages: 14.5, 39.1
// and 14.6, but slower for few sequences (4 of ~2600 13.6, 14.1).
template <int D, int E, bool BIAS>
__global__ void __launch_bounds__(DA_WARPS * 32) attn_decode_keys_kernel(AttnArgs a) {
    constexpr int PARTS = BIAS ? 3 : 1, KP = D + 8, VP = E + 8, STAGE = DA_KEYS * (KP + VP), CK = D / 8, CV = E / 8;
    constexpr float LOG2E = 1.4426950408889634f;
    extern __shared__ __align__(16) unsigned char da_smem[];
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.x / a.G, g = blockIdx.x % a.G, R = a.H / a.G, split = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    bf16* const mine = reinterpret_cast<bf16*>(da_smem) + warp * DA_STAGES * STAGE;
    const int pos = a.positions[b], lo = first_key(a, pos);
    const unsigned kstride = (unsigned)a.G * D, vstride = (unsigned)a.G * E;
    const size_t base = (size_t)a.slots[b] * a.W;
    const bf16* K = static_cast<const bf16*>(a.cache_k) + base * kstride + (size_t)g * D;
    const bf16* V = static_cast<const bf16*>(a.cache_v) + base * vstride + (size_t)g * E;
    const bf16* Q = static_cast<const bf16*>(a.q) + ((size_t)b * a.H + g * R) * D;
    const int step = a.splits * DA_WARPS * DA_KEYS, step_w = step % a.W, first = lo + (split * DA_WARPS + warp) * DA_KEYS;
    int s0 = first % a.W;  // ring row of the next piece to load
    auto load = [&](int c0, int stage) {  // keys c0 .. c0 + 15 (those up to pos)
        bf16* ks = mine + stage * STAGE;
        bf16* vs = ks + DA_KEYS * KP;
        if (c0 + DA_KEYS - 1 <= pos && s0 + DA_KEYS <= a.W) {
            const bf16 *kb = K + (size_t)s0 * kstride, *vb = V + (size_t)s0 * vstride;
#pragma unroll
            for (int c = lane; c < DA_KEYS * CK; c += 32) cp_async16(ks + (c / CK) * KP + (c % CK) * 8, kb + (unsigned)(c / CK) * kstride + (c % CK) * 8, true);
#pragma unroll
            for (int c = lane; c < DA_KEYS * CV; c += 32) cp_async16(vs + (c / CV) * VP + (c % CV) * 8, vb + (unsigned)(c / CV) * vstride + (c % CV) * 8, true);
        } else if (c0 <= pos) {
            for (int c = lane; c < DA_KEYS * CK; c += 32) {
                const int r = c / CK, s = s0 + r;
                const bool ok = c0 + r <= pos;
                cp_async16(ks + r * KP + (c % CK) * 8, ok ? K + (size_t)(s < a.W ? s : s % a.W) * kstride + (c % CK) * 8 : K, ok);
            }
            for (int c = lane; c < DA_KEYS * CV; c += 32) {
                const int r = c / CV, s = s0 + r;
                const bool ok = c0 + r <= pos;
                cp_async16(vs + r * VP + (c % CV) * 8, ok ? V + (size_t)(s < a.W ? s : s % a.W) * vstride + (c % CV) * 8 : V, ok);
            }
        }
        s0 += step_w;
        if (s0 >= a.W) s0 -= a.W;
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < DA_STAGES - 1; ++i) load(first + i * step, i);

    uint32_t qf[D / 16][2];  // Q^T: head gid, dimensions 16 kk + 2 tig .. and 8 more
#pragma unroll
    for (int kk = 0; kk < D / 16; ++kk)
#pragma unroll
        for (int u = 0; u < 2; ++u) qf[kk][u] = gid < R ? *reinterpret_cast<const uint32_t*>(Q + (size_t)gid * D + kk * 16 + u * 8 + tig * 2) : 0u;
    // heads 2 tig, 2 tig + 1: accumulators (value columns 16 ne + gid and 8 more), running maximum (log2 units) and this lane's keys' sum
    float o[E / 16][4], mx[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int ne = 0; ne < E / 16; ++ne) o[ne][0] = o[ne][1] = o[ne][2] = o[ne][3] = 0.f;
    const bool capped = a.softcap > 0.f;
    const float unit = (capped ? 1.f : a.scale) * LOG2E, capf = capped ? 2.f * a.scale / a.softcap : 0.f;
    // the bias of a piece's keys, fetched a piece ahead
    float bias[4], ahead[4];
    const float* const tab = BIAS ? a.bias_tab + g * R + tig * 2 : nullptr;
    auto biases = [&](int c0) {
        if constexpr (BIAS) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float* row = tab + (size_t)min(max(pos - (c0 + gid + 8 * h), 0), a.n_tab - 1) * a.H;
                ahead[2 * h] = tig * 2 < R ? __ldg(row) * LOG2E : 0.f;
                ahead[2 * h + 1] = tig * 2 + 1 < R ? __ldg(row + 1) * LOG2E : 0.f;
            }
        }
    };
    biases(first);
    int stage = 0;
    for (int c0 = first; c0 <= pos; c0 += step) {
        load(c0 + (DA_STAGES - 1) * step, (stage + DA_STAGES - 1) % DA_STAGES);
#pragma unroll
        for (int i = 0; i < 4; ++i) bias[i] = ahead[i];
        biases(c0 + step);
        cp_async_wait<DA_STAGES - 1>();
        __syncwarp();
        const bf16* ks = mine + stage * STAGE;
        const bf16* vs = ks + DA_KEYS * KP;
        float s[4] = {0.f, 0.f, 0.f, 0.f}, z[4] = {0.f, 0.f, 0.f, 0.f};  // keys gid, gid + 8 x heads 2 tig, 2 tig + 1; two sums, so that the MMAs wait less for one another
        const bf16* kp = ks + (lane & 15) * KP + (lane >> 4) * 8;
#pragma unroll
        for (int kk = 0; kk < D / 16; ++kk) {
            uint32_t kf[4];
            ldmatrix4(kf, kp + kk * 16);
            mma_bf16(kk & 1 ? z : s, kf, qf[kk][0], qf[kk][1]);
        }
        float t[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float x = s[i] + z[i];
            if (capped) x = softcap_fast(x, a.softcap, capf);
            x = BIAS ? fmaf(x, unit, bias[i]) : x * unit;
            s[i] = c0 + gid + (i >> 1) * 8 <= pos ? x : -INFINITY;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            t[h] = fmaxf(s[h], s[2 + h]);
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) t[h] = fmaxf(t[h], __shfl_xor_sync(0xffffffffu, t[h], off));
            t[h] = fmaxf(mx[h], t[h]);
        }
        if (__any_sync(0xffffffffu, t[0] > mx[0] || t[1] > mx[1])) {
            const float f0 = mx[0] == -INFINITY ? 0.f : exp2_fast(mx[0] - t[0]), f1 = mx[1] == -INFINITY ? 0.f : exp2_fast(mx[1] - t[1]);
            mx[0] = t[0]; mx[1] = t[1];
            l[0] *= f0; l[1] *= f1;
#pragma unroll
            for (int ne = 0; ne < E / 16; ++ne) { o[ne][0] *= f0; o[ne][1] *= f1; o[ne][2] *= f0; o[ne][3] *= f1; }
        }
        const float m0 = mx[0] == -INFINITY ? 0.f : mx[0], m1 = mx[1] == -INFINITY ? 0.f : mx[1];  // (a piece of nothing but -infinity weighs nothing)
        s[0] = exp2_fast(s[0] - m0); s[1] = exp2_fast(s[1] - m1); s[2] = exp2_fast(s[2] - m0); s[3] = exp2_fast(s[3] - m1);
        l[0] += s[0] + s[2]; l[1] += s[1] + s[3];
        uint32_t pb[PARTS][2];  // P^T: keys 2 tig .. (and 8 more) x head gid
        if constexpr (BIAS) {
            split3_pack(s[0], s[1], pb[0][0], pb[1][0], pb[2][0]);
            split3_pack(s[2], s[3], pb[0][1], pb[1][1], pb[2][1]);
        } else {
            pb[0][0] = pack_bf16(s[0], s[1]); pb[0][1] = pack_bf16(s[2], s[3]);
        }
#pragma unroll
        for (int q = 0; q < PARTS; ++q)
#pragma unroll
            for (int u = 0; u < 2; ++u) asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(pb[q][u]) : "r"(pb[q][u]));
        const bf16* vp = vs + ((lane >> 4) * 8 + (lane & 7)) * VP + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int ne = 0; ne < E / 16; ++ne) {
            uint32_t vf[4];
            ldmatrix4_trans(vf, vp + ne * 16);
#pragma unroll
            for (int q = PARTS - 1; q >= 0; --q) mma_bf16(o[ne], vf, pb[q][0], pb[q][1]);  // the smallest part first
        }
        __syncwarp();  // the buffer is used up
        stage = stage + 1 == DA_STAGES ? 0 : stage + 1;
    }
    cp_async_wait<0>();
    __syncthreads();
    float* mrg = reinterpret_cast<float*>(da_smem);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float* p = mrg + ((size_t)warp * 16 + tig * 2 + h) * (E + 2);
#pragma unroll
        for (int off = 4; off < 32; off <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], off);
        if (gid == 0) { p[0] = mx[h]; p[1] = l[h]; }
#pragma unroll
        for (int ne = 0; ne < E / 16; ++ne) { p[2 + ne * 16 + gid] = o[ne][h]; p[2 + ne * 16 + gid + 8] = o[ne][2 + h]; }
    }
    __syncthreads();
    merge_warps<E, 1>(a, mrg, b, g, R, split);
}

template <int D, int E, int MAPS, bool BIAS = false> inline cudaError_t run_attn_decode(const AttnArgs& a, cudaStream_t st) {
    constexpr size_t smem = attn_decode_smem<D, E, MAPS>();
    auto go = [&](auto kernel) {
        if (smem > 48 * 1024) {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e) return e;
        }
        return launch_pdl(kernel, dim3((unsigned)(a.B * a.G), (unsigned)a.splits), dim3(DA_WARPS * 32), smem, st, a);
    };
    if constexpr (MAPS == 1)
        if (a.H / a.G <= 8) return go(attn_decode_keys_kernel<D, E, BIAS>);
    return go(attn_decode_mma_kernel<D, E, MAPS, BIAS>);
}

// true when a (D, E, maps) instantiation exists; launches it (partial results only)
inline bool launch_attn_decode(const AttnArgs& a, cudaStream_t st, cudaError_t& err) {
    if (a.H / a.G > DA_MAX_GROUP) return false;
    if (a.bias_tab) {
#define MBH_DAB(DD, EE) if (a.d == DD && a.e == EE && a.maps == 1) { err = run_attn_decode<DD, EE, 1, true>(a, st); return true; }
        MBH_DAB(32, 32) MBH_DAB(64, 64) MBH_DAB(64, 128) MBH_DAB(128, 64) MBH_DAB(128, 128)
#undef MBH_DAB
        return false;
    }
#define MBH_DA(DD, EE, MM) if (a.d == DD && a.e == EE && a.maps == MM) { err = run_attn_decode<DD, EE, MM>(a, st); return true; }
    MBH_DA(32, 32, 1) MBH_DA(64, 32, 1) MBH_DA(64, 64, 1) MBH_DA(64, 128, 1) MBH_DA(128, 64, 1) MBH_DA(128, 128, 1) MBH_DA(96, 64, 1) MBH_DA(96, 96, 1)
    MBH_DA(32, 32, 2) MBH_DA(32, 64, 2) MBH_DA(48, 96, 2) MBH_DA(64, 64, 2) MBH_DA(64, 128, 2) MBH_DA(96, 96, 2) MBH_DA(128, 128, 2)
#undef MBH_DA
    return false;
}

}  // namespace mbh
