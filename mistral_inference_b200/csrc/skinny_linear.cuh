// Weight-streaming linears for a decode step's few tokens:  y[t, n] = sum_k x[t, k] * W[n, k]
//
// skinny_mma_kernel (2 to 4 tokens, rows above 4096; 4 with the norm in front).  y^T = W x^T on mma.sync: 16 weight rows of a CTA are the M side of m16n8k16 tiles, the
// tokens the N side; the CTA's 8 warps split K, a lane takes 16 contiguous bytes of two weight rows and of a token per step (the k order inside a
// step is permuted alike on both sides).  The weights of the first eight steps are requested BEFORE the programmatic-dependent-launch wait -- no
// kernel writes weights -- so they stream in while the predecessor finishes.  HBM-bound like skinny_linear_kernel, whose FMAs and staging of
// T * K * 2 bytes per CTA bind first there; figures at skinny_mma_better.  At 8 tokens the stream-K kernel is ahead (637 us a step of 4 layers
// against 753: it reads the tokens once per 128 weight rows, not per 16).
//
// skinny_linear_kernel (1 token, other rows up to 4096; up to 4 tokens where there is no workspace for the normed rows), FMA:
// Roofline: HBM.  Algorithmic bytes = N*K*2 (every weight read exactly once); the activations
// (T*K*2 bytes) are re-read by every CTA from L2.  Each warp owns 2 adjacent weight rows (one RoPE pair /
// one gate-up pair) and streams them with 16-byte no-allocate loads, 4 in flight per row per lane; x lives in
// shared memory (optionally RMS-normalised in place by every CTA -- 8..28 KB, cheaper than a kernel boundary).
#pragma once
#include "epilogue.cuh"

namespace mb200 {

constexpr int kSkinnyThreads = 256;
constexpr int kSkinnyWarps = kSkinnyThreads / 32;
constexpr int kSkinnyRowsPerWarp = 2;
constexpr int kSkinnyRowsPerCta = kSkinnyWarps * kSkinnyRowsPerWarp;

struct SkinnyParams {
  const void* x;       // [T, K] bf16
  const void* norm_w;  // [K] bf16 (NORM only)
  const void* w;       // [N, K] bf16
  int N, K;
  float eps;
  EpiParams epi;
};

template <int T, int MODE, bool NORM>
__global__ void __launch_bounds__(kSkinnyThreads) skinny_linear_kernel(const SkinnyParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  uint4* xs = reinterpret_cast<uint4*>(smem_raw);  // [T][K/8] 16-byte chunks
  __shared__ float red[T][kSkinnyWarps];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kc = p.K >> 3;  // chunks per row

  // ---- stage x (and normalise) ----
  const uint4* xg = reinterpret_cast<const uint4*>(p.x);
  for (int i = tid; i < T * kc; i += kSkinnyThreads) xs[i] = xg[i];
  if constexpr (NORM) {
    __syncthreads();
    float ss[T];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      ss[t] = 0.f;
      for (int c = tid; c < kc; c += kSkinnyThreads) {
        const uint4 v = xs[t * kc + c];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float a = bf16lo(u[j]), b = bf16hi(u[j]);
          ss[t] = fmaf(a, a, ss[t]);
          ss[t] = fmaf(b, b, ss[t]);
        }
      }
      ss[t] = warp_sum(ss[t]);
      if (lane == 0) red[t][warp] = ss[t];
    }
    __syncthreads();
    const uint4* wn = reinterpret_cast<const uint4*>(p.norm_w);
#pragma unroll
    for (int t = 0; t < T; ++t) {
      float tot = 0.f;
#pragma unroll
      for (int w = 0; w < kSkinnyWarps; ++w) tot += red[t][w];
      const float r = ref_rsqrt(tot / (float)p.K + p.eps);
      for (int c = tid; c < kc; c += kSkinnyThreads) {
        const uint4 v = xs[t * kc + c];
        const uint4 g = wn[c];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
        const uint32_t gw[4] = {g.x, g.y, g.z, g.w};
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // bf16( bf16(x * r) * w )
          const float a = round_bf16(bf16lo(u[j]) * r) * bf16lo(gw[j]);
          const float b = round_bf16(bf16hi(u[j]) * r) * bf16hi(gw[j]);
          o[j] = pack_bf16x2(a, b);
        }
        xs[t * kc + c] = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
  __syncthreads();

  // ---- stream the two rows of this warp ----
  const int n0 = (blockIdx.x * kSkinnyWarps + warp) * kSkinnyRowsPerWarp;
  if (n0 >= p.N) return;
  const uint4* w0 = reinterpret_cast<const uint4*>(p.w) + (int64_t)n0 * kc;
  const uint4* w1 = w0 + kc;

  float acc[2][T];
#pragma unroll
  for (int t = 0; t < T; ++t) acc[0][t] = acc[1][t] = 0.f;

  constexpr int U = 4;  // 16-byte loads in flight per row per lane
  int c = lane;
  for (; c + (U - 1) * 32 < kc; c += U * 32) {
    uint4 a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ldg_stream16(w0 + c + u * 32);
      b[u] = ldg_stream16(w1 + c + u * 32);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
      const uint32_t bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const uint4 xv = xs[t * kc + c + u * 32];
        const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float xl = bf16lo(xw[j]), xh = bf16hi(xw[j]);
          acc[0][t] = fmaf(bf16lo(aw[j]), xl, acc[0][t]);
          acc[0][t] = fmaf(bf16hi(aw[j]), xh, acc[0][t]);
          acc[1][t] = fmaf(bf16lo(bw[j]), xl, acc[1][t]);
          acc[1][t] = fmaf(bf16hi(bw[j]), xh, acc[1][t]);
        }
      }
    }
  }
  for (; c < kc; c += 32) {  // tail (K/8 not a multiple of 128)
    const uint4 a = ldg_stream16(w0 + c), b = ldg_stream16(w1 + c);
    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
    const uint32_t bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int t = 0; t < T; ++t) {
      const uint4 xv = xs[t * kc + c];
      const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float xl = bf16lo(xw[j]), xh = bf16hi(xw[j]);
        acc[0][t] = fmaf(bf16lo(aw[j]), xl, acc[0][t]);
        acc[0][t] = fmaf(bf16hi(aw[j]), xh, acc[0][t]);
        acc[1][t] = fmaf(bf16lo(bw[j]), xl, acc[1][t]);
        acc[1][t] = fmaf(bf16hi(bw[j]), xh, acc[1][t]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < T; ++t) {
    acc[0][t] = warp_sum(acc[0][t]);
    acc[1][t] = warp_sum(acc[1][t]);
  }
#pragma unroll
  for (int t = 0; t < T; ++t)
    if (lane == t) epi_pair<MODE>(p.epi, t, n0, acc[0][t], acc[1][t]);
}

// ---- tensor cores ------------------------------------------------------------------------------------------------------------------
constexpr int SM_WARPS = 8, SM_AHEAD = 8;

// Which of the two takes 2 to 4 tokens: what an FMA CTA stages and multiplies grows with T * K.  Steps of 4 layers (K = 4096 and 14336 in the 7B
// shape; 4096, 5120 and 14336 in the Nemo shape), FMAs alone / this rule / tensor cores alone, us: 2 tokens 612 / 548 / 665 and 842 / 729 / -;
// 3 tokens 666 / 596 / 682 and 1051 / 745 / 927; 4 tokens 780 / 492 / 664 and 1283 / 765 / 969.  Four tokens with the norm in front take tensor
// cores at any K (7B: 704 without that); the Linear behind the attention (K = 4096, no norm) is the one that loses by them.
inline bool skinny_mma_better(int64_t T, int64_t K, bool norm) { return (T >= 2 && K > 4096) || (T == 4 && norm); }

__device__ __forceinline__ void skinny_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int MODE>
__global__ void __launch_bounds__(SM_WARPS * 32, 2) skinny_mma_kernel(const SkinnyParams p, int T) {
  __shared__ float part[SM_WARPS][16][9];
  const bf16* X = reinterpret_cast<const bf16*>(p.x);
  const bf16* W = reinterpret_cast<const bf16*>(p.w);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int n0 = blockIdx.x * 16, k0 = warp * 32 + tig * 8;
  constexpr int STEP = SM_WARPS * 32;
  const bf16* wa = W + (int64_t)min(n0 + gid, p.N - 1) * p.K + k0;
  const bf16* wb = W + (int64_t)min(n0 + gid + 8, p.N - 1) * p.K + k0;
  uint4 va[SM_AHEAD], vb[SM_AHEAD];
  const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
  for (int u = 0; u < SM_AHEAD; ++u) {
    const bool ok = k0 + u * STEP < p.K;
    va[u] = ok ? ldg_stream16(wa + u * STEP) : zero;
    vb[u] = ok ? ldg_stream16(wb + u * STEP) : zero;
  }
  pdl_trigger();
  pdl_wait();
  float c[4] = {0.f, 0.f, 0.f, 0.f};
  const bf16* xr = X + (int64_t)min(gid, T - 1) * p.K + k0;  // rows past the end repeat the last one: their sums go nowhere
  const int steps = (p.K + STEP - 1) / STEP;
  for (int i = 0; i < steps; i += SM_AHEAD) {
#pragma unroll
    for (int u = 0; u < SM_AHEAD; ++u) {
      const int k = (i + u) * STEP;
      const uint4 vx = k0 + k < p.K ? *reinterpret_cast<const uint4*>(xr + k) : zero;
      skinny_mma(c, va[u].x, vb[u].x, va[u].y, vb[u].y, vx.x, vx.y);
      skinny_mma(c, va[u].z, vb[u].z, va[u].w, vb[u].w, vx.z, vx.w);
      const bool more = k0 + k + SM_AHEAD * STEP < p.K;
      va[u] = more ? ldg_stream16(wa + k + SM_AHEAD * STEP) : zero;
      vb[u] = more ? ldg_stream16(wb + k + SM_AHEAD * STEP) : zero;
    }
  }
  part[warp][gid][tig * 2] = c[0];
  part[warp][gid][tig * 2 + 1] = c[1];
  part[warp][gid + 8][tig * 2] = c[2];
  part[warp][gid + 8][tig * 2 + 1] = c[3];
  __syncthreads();
  if (threadIdx.x < 64) {
    const int t = threadIdx.x & 7, r = (threadIdx.x >> 3) * 2, n = n0 + r;
    if (t < T && n < p.N) {
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int w = 0; w < SM_WARPS; ++w) {
        s0 += part[w][r][t];
        s1 += part[w][r + 1][t];
      }
      epi_pair<MODE>(p.epi, t, n, s0, s1);
    }
  }
}

template <int MODE>
int launch_skinny_mma(const SkinnyParams& p, int T, cudaStream_t stream) {
  MB_CHECK_ARG(p.K % 8 == 0 && p.N % 2 == 0, "skinny linear: K=%d must be a multiple of 8, N=%d even", p.K, p.N);
  MB_CHECK_ARG((size_t)T * p.K * 2 <= 200 * 1024, "skinny linear: T*K too large (%d x %d)", T, p.K);  // the limit of both kernels
  MB_CHECK_CUDA(launch_pdl(skinny_mma_kernel<MODE>, dim3((unsigned)ceil_div(p.N, 16)), dim3(SM_WARPS * 32), 0, stream, p, T));
  return MB200_OK;
}

template <int MODE, bool NORM>
int launch_skinny(const SkinnyParams& p, int T, cudaStream_t stream) {
  MB_CHECK_ARG(T >= 1 && T <= MB200_SKINNY_MAX_T, "skinny linear: T=%d out of range", T);
  MB_CHECK_ARG(p.K % 8 == 0 && p.N % kSkinnyRowsPerWarp == 0, "skinny linear: K=%d must be a multiple of 8, N=%d even", p.K, p.N);
  const size_t smem = (size_t)T * p.K * 2;
  MB_CHECK_ARG(smem <= 200 * 1024, "skinny linear: T*K too large for shared memory (%zu B)", smem);
  const dim3 grid(ceil_div(p.N, kSkinnyRowsPerCta));
  auto go = [&](auto kernel) -> int {
    if (smem > 48 * 1024) MB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<grid, kSkinnyThreads, smem, stream>>>(p);
    MB_CHECK_LAUNCH("skinny_linear_kernel");
    return MB200_OK;
  };
  switch (T) {
    case 1: return go(skinny_linear_kernel<1, MODE, NORM>);
    case 2: return go(skinny_linear_kernel<2, MODE, NORM>);
    case 3: return go(skinny_linear_kernel<3, MODE, NORM>);
    default: return go(skinny_linear_kernel<4, MODE, NORM>);
  }
}

}  // namespace mb200
