// C[T, N] = A[T, K] * W[N, K]^T for a few dozen to a few hundred tokens: every weight byte is read once, by all SMs at the same rate, and HBM or the way from L2 bounds it.
//
// The weights are the MMA's 128 rows and the tokens its columns (any multiple of 16 up to 256), so a k-block of 64 costs what its tokens cost.  N / 128 tiles do not divide over 148 SMs, so
// the (tile, k-block) units are one sequence of which CTA c takes the c-th contiguous part, and the fp32 sums of each piece of a tile go to a slot of their own; a second
// kernel, launched programmatically, adds a tile's pieces in the order of k and runs the step behind the Linear on the whole chip.  Nobody waits for another CTA, and the exchange is 3 us of a
// launch that overlaps the first one's end, where the owner of a tile that waits for its contributors (gemm_streamk.cuh, which remains for the mixtures and for matrices whose
// slots would not fit) took 6 to 10 with memory idle.  Lanes of an accumulator are features: a token's 32 features of a warp are one 128-byte line of the slot.
//
// us from a cold L2, stream-K and this one: 64 tokens 6144 x 4096 35, 26; 4096 x 14336 55, 42; 28672 x 4096 72, 60 (40 tokens); 96 tokens 4096 x 4096 49, 24; 5120 x 14336 66, 48.
// Steps and prompts: four layers of the 7B shape, 48 sequences 837, 616; one layer, 100 tokens 228, 153; two layered ones of width 4096, 100 tokens 556, 320.
#pragma once
#include "gemm_tcgen05.cuh"

namespace mb200 {

constexpr int ST_ROWS = 128, ST_MAX_T = 256, ST_THREADS = 192;
constexpr int ST_W_BYTES = ST_ROWS * TG_BK * 2, ST_RING = 190 * 1024, ST_MAX_STAGES = 12;
constexpr size_t ST_SLOT_BYTES = 28u << 20;  // of slots: what a workspace has room for

struct StParams {
  int T, N, K, cols /* T rounded up to 16 */, stages, grid;
  EpiParams epi;
  float* slots;  // [grid + tiles - 1] x [T][128] (st_piece): the piece of tile t that CTA c computes is slot c + t
};
// Floats of a slot: more than T x 128, so that the CTAs' slots, which fill at the same time, do not lie a power of two apart.
MB_HD size_t st_piece(int64_t T) { return (size_t)T * ST_ROWS + 416; }
// which units CTA c has, and which CTA has unit u
struct StSchedule {
  long long per, rem;
  MB_HD StSchedule(long long total, int grid) : per(total / grid), rem(total % grid) {}
  MB_HD long long first(int c) const { return (long long)c * per + (c < rem ? c : rem); }
  MB_HD int cta(long long u) const { return (int)(u < rem * (per + 1) ? u / (per + 1) : rem + (u - rem * (per + 1)) / per); }
};

__global__ void __launch_bounds__(ST_THREADS, 1) stream_tiles_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const __grid_constant__ StParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[ST_MAX_STAGES], empty[ST_MAX_STAGES], tmem_full[2], tmem_empty[2];
  __shared__ uint32_t tmem_base_slot;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, cta = (int)blockIdx.x;
  const int tiles = p.N / ST_ROWS, num_k = p.K / TG_BK;
  const StSchedule sched((long long)tiles * num_k, p.grid);
  const long long u_begin = sched.first(cta), u_end = sched.first(cta + 1);
  const uint32_t stage_bytes = ST_W_BYTES + (uint32_t)p.cols * TG_BK * 2;
  const uint32_t half_cols = p.cols <= 32 ? 32u : p.cols <= 64 ? 64u : p.cols <= 128 ? 128u : 256u;
  if (threadIdx.x == 0) {
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 4);  // one arrive per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(&tmem_base_slot, 2 * half_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  if (threadIdx.x == 0) pdl_trigger();

  if (warp == 0) {
    // ================= TMA producer: the weights of the first ring before the wait for the predecessor, its tokens after it =================
    if (lane == 0) {
      const int n_it = (int)(u_end - u_begin), head = min(n_it, p.stages);
      int tile = (int)(u_begin / num_k), kb = (int)(u_begin % num_k), x_kb = kb;
      auto weights = [&](int s) {
        tma_load_2d(smem + s * stage_bytes, &map_w, &full[s], kb * TG_BK, tile * ST_ROWS);
        if (++kb == num_k) kb = 0, ++tile;
      };
      auto tokens = [&](int s) {
        tma_load_2d(smem + s * stage_bytes + ST_W_BYTES, &map_a, &full[s], x_kb * TG_BK, 0);
        if (++x_kb == num_k) x_kb = 0;
      };
      for (int it = 0; it < head; ++it) {
        mbar_arrive_expect_tx(&full[it], stage_bytes);
        weights(it);
      }
      pdl_wait();
      for (int it = 0; it < head; ++it) tokens(it);
      int s = 0, par = 0;
      for (int it = head; it < n_it; ++it) {
        mbar_wait(&empty[s], par, 31, it);
        mbar_arrive_expect_tx(&full[s], stage_bytes);
        weights(s);
        tokens(s);
        if (++s == p.stages) s = 0, par ^= 1;
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (one thread, elected by the warp) =================
    pdl_wait();  // (the tokens come behind it: the waits' limits count from there)
    const uint32_t ring = umma_desc_lo(smem_u32(smem)), idesc = (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t)(p.cols >> 3) << 17 | (uint32_t)(ST_ROWS >> 4) << 24;
    int s = 0, par = 0;
    uint32_t seg = 0;
    for (long long u = u_begin; u < u_end; ++seg) {
      const int n_kb = (int)min((long long)num_k - u % num_k, u_end - u);
      const uint32_t acc = seg & 1, d_tmem = tmem_base + acc * half_cols;
      mbar_wait(&tmem_empty[acc], ((seg >> 1) & 1) ^ 1, 32, seg);
      tc_fence_after();
      for (int kb = 0; kb < n_kb; ++kb) {
        mbar_wait(&full[s], par, 33, kb);
        tc_fence_after();
        const uint32_t wdesc = ring + s * (stage_bytes >> 4), xdesc = wdesc + (ST_W_BYTES >> 4);
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < TG_BK / 16; ++k) umma_bf16(d_tmem, wdesc + 2 * k, xdesc + 2 * k, idesc, (kb > 0 || k) ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        __syncwarp();
        if (++s == p.stages) s = 0, par ^= 1;
      }
      if (elect_one()) umma_commit(&tmem_full[acc]);
      __syncwarp();
      u += n_kb;
    }
  } else {
    // ================= warps 2..5: sums to the slots, TMEM lanes (features) 32 * (warp % 4) .. + 31 =================
    pdl_wait();  // (the slots may still be read by the predecessor)
    const int lane_base = (warp & 3) * 32;
    uint32_t seg = 0;
    for (long long u = u_begin; u < u_end; ++seg) {
      const int tile = (int)(u / num_k), n_kb = (int)min((long long)num_k - u % num_k, u_end - u);
      const uint32_t acc = seg & 1, trow = tmem_base + ((uint32_t)lane_base << 16) + acc * half_cols;
      float* const slot = p.slots + (size_t)(cta + tile) * st_piece(p.T) + lane_base + lane;
      mbar_wait(&tmem_full[acc], (seg >> 1) & 1, 34, seg);
      tc_fence_after();
      uint32_t v[32];
#pragma unroll 1
      for (int c = 0; c < p.T; c += 32) {
        tmem_ld_32x32b_x32(trow + c, v);
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (c + j < p.T) slot[(size_t)(c + j) * ST_ROWS] = __uint_as_float(v[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty[acc]);
      u += n_kb;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, 2 * half_cols);
}

// The pieces of a tile, added in the order of k, and the step behind the Linear: 32 features of a token a thread.
constexpr int SC_THREADS = 128;
template <int MODE>
__global__ void __launch_bounds__(SC_THREADS) stream_tiles_combine_kernel(const __grid_constant__ StParams p) {
  pdl_trigger();
  const int i = blockIdx.x * SC_THREADS + threadIdx.x, chunk = i & 3, t = (i >> 2) % p.T, tile = (i >> 2) / p.T, num_k = p.K / TG_BK, tiles = p.N / ST_ROWS;
  pdl_wait();
  if (tile >= tiles) return;
  const StSchedule sched((long long)tiles * num_k, p.grid);
  const int c0 = sched.cta((long long)tile * num_k), c1 = sched.cta((long long)(tile + 1) * num_k - 1);
  const size_t piece = st_piece(p.T);
  const float4* src = reinterpret_cast<const float4*>(p.slots + (size_t)(c0 + tile) * piece + (size_t)t * ST_ROWS + chunk * 32);
  const int n = tile * ST_ROWS + chunk * 32;
  float4 v[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) v[q] = src[q];
#pragma unroll 2
  for (int c = c0 + 1; c <= c1; ++c) {
    src += piece / 4;
    float4 x[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) x[q] = src[q];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q].x += x[q].x, v[q].y += x[q].y, v[q].z += x[q].z, v[q].w += x[q].w;
  }
  uint32_t y[32];
#pragma unroll
  for (int q = 0; q < 8; ++q) y[4 * q] = __float_as_uint(v[q].x), y[4 * q + 1] = __float_as_uint(v[q].y), y[4 * q + 2] = __float_as_uint(v[q].z), y[4 * q + 3] = __float_as_uint(v[q].w);
  epi_chunk32<MODE>(p.epi, t, n, y);
}

// ---- host ----
// Below 128 tokens always; above, where single CTAs (gemm_tcgen05.cuh) would leave most of the chip idle along a long k.  us from a cold L2, there and here: 160 tokens 1024 x 14336 57, 34;
// 2048 x 8192 37, 28; 3072 x 14336 43, 38 (pairs); 4096 x 8192 37, 36; 4096 x 4096 25, 28; 5120 x 14336 51, 52 (pairs).
// (128 tokens, which run on no pairs: 5120 x 5120 31, 30, 5120 x 14336 66, 50, but 6144 x 4096 29, 30.)
inline bool stream_tiles_better(int64_t T, int64_t N, int64_t K) { return T < TG_BM || (T == TG_BM && K >= 5120) || (T <= ST_MAX_T && K >= 8192 && N <= 4096); }

// CTAs: every SM, but at most twelve a tile where tiles are few: a tile's pieces are added one after another.  us with all SMs and with twelve a tile: 128 tokens 256 x 8192 58, 16; 128 x 5120
// 54, 14; 1024 x 8192 21, 20; with more than 128 tokens from seven tiles on the pieces' own length counts for more: 160 tokens 768 x 8192 26, 18.5; 1024 x 14336 23.6, 24.9.
inline int stream_tiles_grid(int64_t T, int64_t N, int64_t K, int sms) {
  const int64_t tiles = N / ST_ROWS, units = tiles * (K / TG_BK), most = T <= TG_BM || tiles <= 6 ? 12 * tiles : sms;
  return (int)(units < sms ? (units < most ? units : most) : most < sms ? most : sms);
}

// bytes of slots, 0: not for this kernel
inline size_t stream_tiles_bytes(int64_t T, int64_t N, int64_t K, int sms) {
  const char* e = getenv("MB200_STREAMK");
  if (sms < 1 || (e != nullptr && e[0] == '0') || T < 1 || !stream_tiles_better(T, N, K) || N % ST_ROWS != 0 || K % TG_BK != 0) return 0;
  const int64_t tiles = N / ST_ROWS, grid = stream_tiles_grid(T, N, K, sms);
  const size_t bytes = (size_t)(grid + tiles - 1) * st_piece(T) * sizeof(float);
  return bytes <= ST_SLOT_BYTES ? bytes : 0;
}

template <int MODE>
int launch_stream_tiles(const GemmParams& g, int sms, void* slots, cudaStream_t stream) {
  StParams p;
  p.T = g.T;
  p.N = g.N;
  p.K = g.K;
  p.cols = (g.T + 15) / 16 * 16;
  if (p.cols == 128 || p.cols == 192) p.cols += 16;  // measured: 128 tokens 5120 x 14336 56 us at 128 columns, 50 at 144; 192 60, (224: 56).  The stages are then 16-KB multiples; why that costs is not known
  const int stage_bytes = ST_W_BYTES + p.cols * TG_BK * 2;
  p.stages = ST_RING / stage_bytes < ST_MAX_STAGES ? ST_RING / stage_bytes : ST_MAX_STAGES;
  p.grid = stream_tiles_grid(g.T, g.N, g.K, sms);
  p.epi = g.epi;
  p.slots = reinterpret_cast<float*>(slots);
  CUtensorMap map_a, map_w;
  int rc = make_tensor_map_2d(&map_a, g.a, g.T, g.K, p.cols);
  if (rc) return rc;
  rc = make_tensor_map_2d(&map_w, g.w, g.N, g.K, ST_ROWS);
  if (rc) return rc;
  const size_t smem = (size_t)p.stages * stage_bytes + 1024;
  MB_CHECK_CUDA(device_info::allow_shared<stream_tiles_kernel>(ST_RING + 1024));
  MB_CHECK_CUDA(launch_pdl(stream_tiles_kernel, dim3((unsigned)p.grid), dim3(ST_THREADS), smem, stream, map_a, map_w, p));
  const long long threads = (long long)(g.N / 32) * g.T;
  MB_CHECK_CUDA(launch_pdl(stream_tiles_combine_kernel<MODE>, dim3((unsigned)((threads + SC_THREADS - 1) / SC_THREADS)), dim3(SC_THREADS), 0, stream, p));
  return MB200_OK;
}

}  // namespace mb200
