// Mixture of experts for T > 1 tokens (prefill and batched decode): device-side router + grouped tensor-core expert GEMMs.
// Replaces MoeLayer.forward (moe.py:24-32) -- gate Linear, torch.topk, softmax, and the per-expert `torch.where` / index /
// FeedForward / weighted `+=` loop with its host synchronisations -- by five launches with NO host round trip:
//
//   moe_route_kernel    logits = bf16(hn . gate^T); top-k on the bf16 logits (ties: lower expert index first); fp32 softmax over
//                       the k selected -> bf16 weights (moe.py:25-27); the k (expert, weight) pairs of a token are stored in
//                       ASCENDING expert index: the order the reference's `results[idx] += w * expert(x)` loop visits them.
//   moe_plan_kernel     one CTA: per-expert row counts, segment starts (each expert's segment padded to a multiple of the GEMM's
//                       m-tile), a DETERMINISTIC slot for every (token, expert) pair (token order inside a segment: identical on
//                       every rank of an expert-parallel group, which is what lets ranks write each other's rows), and the list
//                       of m tiles of the experts this rank owns.
//   moe_gather_kernel   xs[slot] = hn[token], row_w[slot] = routing weight  (rows of local experts only)
//   grouped GEMM x2     g = silu(xs W1_e^T) * (xs W3_e^T);  yw = bf16(w * bf16(g W2_e^T)), the second one storing every row on ALL
//                       ranks of the group (peer stores over NVLink) -- the exchange step of expert parallelism is the epilogue of
//                       the down projection, an all-gather of rows with no reduction.  gemm_streamk.cuh for few tokens,
//                       gemm_tcgen05.cuh, and from ~128 rows an expert gemm_pair.cuh.
//   moe_combine_kernel  (expert parallel: signal the peers / wait for theirs) out[t] = bf16(h[t] + sum_j yw[slot(t, j)]) with the
//                       sum taken in ascending expert index, each step rounded to bf16 like `results +=`: the reference's
//                       order for any k and any number of ranks.  (The rows themselves are the same on any number of ranks but for
//                       stream-K's, whose sums are cut by the tiles that a rank has.)
// Roofline: tensor pipe for prefill (2 * rows * 3 * dim * hidden flop), HBM for decode (every touched expert's weights once).
#pragma once
#include "gemm_pair.cuh"
#include "gemm_streamk.cuh"
#include "gemm_tcgen05.cuh"

namespace mb200 {

constexpr int MOE_MAX_TOPK = 8;

// ---- router: one warp per token (WIDE = false: prefill) or one CTA per token with the 8 warps splitting the row (WIDE = true:
// decode-sized batches, where a single warp walking 4096 dims x 8 experts is pure load latency: 36 us measured for 8 tokens) ------
template <int E, bool WIDE>
__global__ void __launch_bounds__(256) moe_route_kernel(const bf16* hn, const bf16* __restrict__ gate_w, int T, int dim, int k,
                                                        int32_t* __restrict__ sel, bf16* __restrict__ wts) {
  pdl_trigger();
  pdl_wait();  // hn is the preceding RMSNorm's output
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = WIDE ? (int)blockIdx.x : (int)blockIdx.x * 8 + warp;
  if (t >= T) return;
  const int kc = dim >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(hn + (int64_t)t * dim);
  float acc[E];
#pragma unroll
  for (int e = 0; e < E; ++e) acc[e] = 0.f;
#pragma unroll 2
  for (int c = WIDE ? (int)threadIdx.x : lane; c < kc; c += WIDE ? 256 : 32) {
    const uint4 xv = xr[c];
    const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const uint4 gv = __ldg(reinterpret_cast<const uint4*>(gate_w + (int64_t)e * dim) + c);
      const uint32_t gw[4] = {gv.x, gv.y, gv.z, gv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[e] = fmaf(bf16lo(gw[j]), bf16lo(xw[j]), acc[e]);
        acc[e] = fmaf(bf16hi(gw[j]), bf16hi(xw[j]), acc[e]);
      }
    }
  }
  if constexpr (WIDE) {  // fold the 8 warps' partial sums in a fixed order
    __shared__ float part[8][E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float v = warp_sum(acc[e]);
      if (lane == 0) part[warp][e] = v;
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) v += part[w][e];
      acc[e] = round_bf16(v);  // the router Linear's bf16 output (moe.py:25)
    }
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) acc[e] = round_bf16(warp_sum(acc[e]));  // the router Linear's bf16 output (moe.py:25)
  }
  if (lane != 0) return;
  int se[MOE_MAX_TOPK];
  float sv[MOE_MAX_TOPK];
  unsigned taken = 0u;
  for (int j = 0; j < k; ++j) {  // top-k on the bf16 logits, ties -> lower index
    int best = -1;
    float bv = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (!((taken >> e) & 1u) && (best < 0 || acc[e] > bv)) {
        best = e;
        bv = acc[e];
      }
    taken |= 1u << best;
    se[j] = best;
    sv[j] = bv;
  }
  float den = 0.f, ex[MOE_MAX_TOPK];
  for (int j = 0; j < k; ++j) {
    ex[j] = expf(sv[j] - sv[0]);  // sv[0] is the maximum
    den += ex[j];
  }
  for (int j = 0; j < k; ++j) sv[j] = round_bf16(ex[j] / den);  // softmax in fp32, then .to(bf16) (moe.py:27)
  for (int a = 1; a < k; ++a)  // ascending expert index, weights travelling with their experts
    for (int b = a; b > 0 && se[b] < se[b - 1]; --b) {
      const int ts = se[b];
      se[b] = se[b - 1];
      se[b - 1] = ts;
      const float tv = sv[b];
      sv[b] = sv[b - 1];
      sv[b - 1] = tv;
    }
  for (int j = 0; j < k; ++j) {
    sel[(int64_t)t * k + j] = se[j];
    wts[(int64_t)t * k + j] = __float2bfloat16_rn(sv[j]);
  }
}

// ---- plan: one CTA ---------------------------------------------------------------------------------------------------------
// plan layout (int32): [0] m tiles owned by this rank, [1] padded rows in total, [2] tile capacity, [3] (token, expert) pairs, [4]/[5] statistics, [6] token tiles for
// pairs of CTAs, [7] tiles that these have drawn (zero between launches), [8 + e] start of expert e's segment (e = 0..E), then from word MOE_PLAN_HEADER four lists of `capacity` words: tile_expert, tile_row0 (m tiles),
// pair_expert, pair_info (token tiles: first row | width / 32).
constexpr int MP_THREADS = 1024, MP_ROW = MP_THREADS + MP_THREADS / 32;
// A plan of up to this many (token, expert) pairs lists no token tiles for pairs of CTAs: whoever launches on them asks here first.
constexpr int MOE_SHORT_PLAN = 512;
MB_HD bool moe_plan_lists_pairs(int64_t pairs) { return pairs > MOE_SHORT_PLAN; }
inline size_t moe_plan_smem(int64_t E) { return ((size_t)E * MP_ROW + 2 * E + 1) * sizeof(int32_t); }
__global__ void __launch_bounds__(MP_THREADS) moe_plan_kernel(const int32_t* sel, int pairs, int E, int tile_rows, int shard_rank,
                                                              int shard_world, int tile_cap, int32_t* __restrict__ slot, int32_t* __restrict__ plan) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ int32_t sm[];  // cnt[E][MP_ROW], then seg[E + 1], total[E]
  int32_t* cnt = sm;
  int32_t* seg = sm + E * MP_ROW;
  int32_t* total = seg + E + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (!moe_plan_lists_pairs(pairs)) {
    // decode-sized batch: thread e walks the whole (short) pair list for expert e -- same deterministic plan, a few hundred cycles
    if (tid < E) {
      int n = 0;
      for (int i = 0; i < pairs; ++i)
        if (sel[i] == tid) slot[i] = n++;  // position inside the expert's segment; the segment start is added below
      total[tid] = n;  // (a choice >= E names no expert with weights: it gets no row)
    }
    __syncthreads();
    if (tid == 0) {
      int rows = 0, n = 0, touched = 0;
      for (int e = 0; e < E; ++e) {
        seg[e] = rows;
        plan[8 + e] = rows;
        const int m_tiles = (total[e] + tile_rows - 1) / tile_rows;
        touched += total[e] > 0;
        if (e % shard_world == shard_rank)
          for (int m = 0; m < m_tiles && n < tile_cap; ++m, ++n) {
            plan[MOE_PLAN_HEADER + n] = e;
            plan[MOE_PLAN_HEADER + tile_cap + n] = rows + m * tile_rows;
          }
        rows += m_tiles * tile_rows;
      }
      plan[8 + E] = rows;
      plan[0] = n;
      plan[1] = rows;
      plan[2] = tile_cap;
      plan[3] = pairs;
      plan[4] += touched;
      plan[5] += 1;
      plan[6] = 0;
      plan[7] = 0;
    }
    __syncthreads();
    for (int i = tid; i < pairs; i += MP_THREADS) slot[i] = sel[i] < E ? slot[i] + seg[sel[i]] : -1;
    return;
  }
  // This thread counts `per` neighbouring pairs, eight loads in flight at a time.  Row e of cnt has thread t's count at t + t / 32: the scan below, whose lanes take 32
  // neighbouring counts each, would otherwise have all of them in one bank.
  const int per = (pairs + MP_THREADS - 1) / MP_THREADS, mine = tid + (tid >> 5);
  const int p0 = min(tid * per, pairs), p1 = min(p0 + per, pairs);
  for (int e = 0; e < E; ++e) cnt[e * MP_ROW + mine] = 0;
  for (int i0 = p0; i0 < p1; i0 += 8) {
    int v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i0 + i < p1 ? sel[i0 + i] : E;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (v[i] < E) cnt[v[i] * MP_ROW + mine] += 1;
  }
  __syncthreads();
  // exclusive scan of every expert's 1024 counts: warp w takes experts w, w + 32, ...; lane l scans entries [32 l, 32 l + 32)
  for (int e = warp; e < E; e += MP_THREADS / 32) {
    int32_t* c = cnt + e * MP_ROW + lane * 33;
    int run = 0;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) {
      const int v = c[i];
      c[i] = run;
      run += v;
    }
    int incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    const int base = incl - run;
#pragma unroll 8
    for (int i = 0; i < 32; ++i) c[i] += base;
    if (lane == 31) total[e] = incl;
  }
  __syncthreads();
  if (warp == 0) {  // segment starts and the tile lists, an expert per lane
    int rows = 0, n = 0, np = 0, touched = 0;
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane;
      const bool here = e < E, own = here && e % shard_world == shard_rank;
      const int have = here ? total[e] : 0, m_tiles = (have + tile_rows - 1) / tile_rows;
      const int units = (have + 31) / 32, items = (units + 7) / 8;  // token tiles of pairs of CTAs: at most 256 wide, widths differ by at most 32
      int r = m_tiles * tile_rows, k = own ? m_tiles : 0, q = own ? items : 0;
      const int r_own = r, k_own = k, q_own = q;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int ur = __shfl_up_sync(0xffffffffu, r, o), uk = __shfl_up_sync(0xffffffffu, k, o), uq = __shfl_up_sync(0xffffffffu, q, o);
        if (lane >= o) r += ur, k += uk, q += uq;
      }
      const int row0 = rows + r - r_own, n0 = n + k - k_own, np0 = np + q - q_own;
      if (here) {
        seg[e] = row0;
        plan[8 + e] = row0;
      }
      for (int m = 0; m < k_own && n0 + m < tile_cap; ++m) {
        plan[MOE_PLAN_HEADER + n0 + m] = e;
        plan[MOE_PLAN_HEADER + tile_cap + n0 + m] = row0 + m * tile_rows;
      }
      for (int m = 0; m < q_own && np0 + m < tile_cap; ++m) {
        const int u0 = units * m / items, u1 = units * (m + 1) / items;
        plan[MOE_PLAN_HEADER + 2 * tile_cap + np0 + m] = e;
        plan[MOE_PLAN_HEADER + 3 * tile_cap + np0 + m] = (row0 + 32 * u0) | (u1 - u0);
      }
      rows += __shfl_sync(0xffffffffu, r, 31);
      n += __shfl_sync(0xffffffffu, k, 31);
      np += __shfl_sync(0xffffffffu, q, 31);
      touched += __popc(__ballot_sync(0xffffffffu, have > 0));
    }
    if (lane == 0) {
      plan[0] = min(n, tile_cap);
      plan[1] = rows;
      plan[2] = tile_cap;
      plan[3] = pairs;
      plan[4] += touched;  // statistics (never reset by the kernel): experts with at least one row, summed over calls ...
      plan[5] += 1;        // ... and the number of calls: the measured "distinct experts per layer" of bench.py
      plan[6] = min(np, tile_cap);
      plan[7] = 0;
      seg[E] = rows;
      plan[8 + E] = rows;
    }
  }
  __syncthreads();
  for (int i0 = p0; i0 < p1; i0 += 8) {  // this thread's column of cnt is its own: the next free place of each expert
    int v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = i0 + i < p1 ? sel[i0 + i] : E;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i0 + i < p1) slot[i0 + i] = v[i] < E ? seg[v[i]] + cnt[v[i] * MP_ROW + mine]++ : -1;
  }
}

// ---- gather: one warp per (token, expert) pair ------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint4* hn, const int32_t* sel, const bf16* wts, const int32_t* slot, int pairs, int k, int row_chunks, int shard_rank,
                                                         int shard_world, uint4* __restrict__ xs, bf16* __restrict__ row_w) {
  pdl_trigger();
  pdl_wait();
  const int pair = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (pair >= pairs) return;
  if (sel[pair] % shard_world != shard_rank) return;  // another rank's expert
  const int t = pair / k, s = slot[pair];
  if (lane == 0) row_w[s] = wts[pair];
  const uint4* src = hn + (int64_t)t * row_chunks;
  uint4* dst = xs + (int64_t)s * row_chunks;
  for (int c = lane; c < row_chunks; c += 32) dst[c] = src[c];
}

// ---- combine (+ the expert-parallel handshake) --------------------------------------------------------------------------------
struct MoeCombineParams {
  const uint4* yw;        // [rows, dim] weighted expert outputs (all ranks' rows once the handshake is through)
  const int32_t* slot;    // [T, k]
  const uint4* residual;  // h [T, dim] or null
  uint4* out;             // [T, dim]
  int T, k, row_chunks;
  // expert parallel (n_ranks > 1): flags[r] of THIS rank is written by rank r when all its rows of this call have landed here
  int n_ranks, my_rank;
  unsigned* my_flags;               // [n_ranks] in this rank's comm buffer
  unsigned* peer_flags[kMaxPeers];  // the same array on the other ranks (mapped)
  unsigned* epoch;                  // local device word: completed calls on this buffer
  int* done_counter;                // local, self-resetting
};
__device__ __forceinline__ unsigned ld_acquire_sys_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sys_u32(unsigned* p, unsigned v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__global__ void __launch_bounds__(128) moe_combine_kernel(const MoeCombineParams p) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  if (p.n_ranks > 1) {
    // This kernel starts after this rank's down projection has finished (stream order), i.e. after its peer stores were issued
    // and completed.  Block 0 tells every peer; every block then waits until every peer has told this rank.
    __shared__ unsigned target;
    if (threadIdx.x == 0) {
      const unsigned e = *reinterpret_cast<volatile unsigned*>(p.epoch) + 1u;
      target = e;
      if (blockIdx.x == 0) {
        __threadfence_system();
        for (int r = 0; r < p.n_ranks - 1; ++r) st_release_sys_u32(p.peer_flags[r] + p.my_rank, e);
        st_release_sys_u32(p.my_flags + p.my_rank, e);
      }
      for (int r = 0; r < p.n_ranks; ++r) {
        unsigned long long spins = 0;
        while ((int)(ld_acquire_sys_u32(p.my_flags + r) - e) < 0) {
          if (++spins == (1ull << 26)) {
            printf("[mb200 watchdog] rank %d block %d: no signal from rank %d for MoE exchange %u (have %u)\n", p.my_rank, (int)blockIdx.x, r, e,
                   ld_acquire_sys_u32(p.my_flags + r));
            __trap();
          }
        }
      }
    }
    __syncthreads();
    (void)target;
  }
  const int32_t* sl = p.slot + (int64_t)t * p.k;
  for (int c = threadIdx.x; c < p.row_chunks; c += 128) {
    float r[8];
    {
      const uint4 v = p.yw[(int64_t)sl[0] * p.row_chunks + c];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        r[2 * j] = bf16lo(u[j]);  // results starts at zero: bf16(0 + t) == t
        r[2 * j + 1] = bf16hi(u[j]);
      }
    }
    for (int q = 1; q < p.k; ++q) {
      const uint4 v = p.yw[(int64_t)sl[q] * p.row_chunks + c];
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        r[2 * j] = round_bf16(r[2 * j] + bf16lo(u[j]));  // results[idx] += ... in bf16 (moe.py:31)
        r[2 * j + 1] = round_bf16(r[2 * j + 1] + bf16hi(u[j]));
      }
    }
    uint32_t o[4];
    if (p.residual != nullptr) {
      const uint4 h = p.residual[(int64_t)t * p.row_chunks + c];
      const uint32_t hu[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(bf16lo(hu[j]) + r[2 * j], bf16hi(hu[j]) + r[2 * j + 1]);  // h + r (transformer_layers.py:168)
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) o[j] = pack_bf16x2(r[2 * j], r[2 * j + 1]);
    }
    p.out[(int64_t)t * p.row_chunks + c] = make_uint4(o[0], o[1], o[2], o[3]);
  }
  if (p.n_ranks > 1) {  // the last block to finish publishes the epoch for the next call on this buffer
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      const int prev = atomicAdd(p.done_counter, 1);
      if (prev == (int)gridDim.x - 1) {
        *p.done_counter = 0;
        __threadfence();
        *reinterpret_cast<volatile unsigned*>(p.epoch) = *reinterpret_cast<volatile unsigned*>(p.epoch) + 1u;
      }
    }
  }
}

// ---- host side -------------------------------------------------------------------------------------------------------------
inline int moe_tile_rows(int64_t T) { return T <= 32 ? 32 : (T <= 64 ? 64 : 128); }  // an expert gets at most one row per token: decode batches fit ONE short m tile
inline int64_t moe_tile_cap(int64_t pairs, int64_t E, int tile_rows) { return (pairs + tile_rows - 1) / tile_rows + E; }
inline int64_t moe_plan_words(int64_t pairs, int64_t E, int tile_rows) { return MOE_PLAN_HEADER + 4 * moe_tile_cap(pairs, E, tile_rows); }
inline int64_t moe_row_cap(int64_t pairs, int64_t E, int tile_rows) { return moe_tile_cap(pairs, E, tile_rows) * tile_rows; }

// tensor maps of the experts' weights, boxes of `rows` rows; another rank's experts (never referenced by this rank's tiles) get `map_a`
inline int make_expert_maps(MoeWeightMaps* maps, const CUtensorMap& map_a, const void* const* w_host, int E, int64_t N, int64_t K, int rows) {
  for (int e = 0; e < MOE_MAX_EXPERTS; ++e) {
    if (e >= E || w_host[e] == nullptr) {
      maps->m[e] = map_a;
      continue;
    }
    const int rc = make_tensor_map_2d(&maps->m[e], w_host[e], N, K, rows);
    if (rc) return rc;
  }
  return MB200_OK;
}

template <int MODE, int BN, int TA>
int launch_grouped_bn(const void* a, int64_t rows_cap, int64_t K, int64_t N, const void* const* w_host, int E, const int32_t* plan, const EpiParams& epi,
                      int sms, cudaStream_t stream) {
  using Cfg = TgCfg<BN, TA, kEpiSmem<MODE>>;
  CUtensorMap map_a;
  MoeWeightMaps maps;
  int rc = make_tensor_map_2d(&map_a, a, rows_cap, K, TA);
  if (rc) return rc;
  rc = make_expert_maps(&maps, map_a, w_host, E, N, K, BN);
  if (rc) return rc;
  TcGemmParams p;
  p.T = (int)rows_cap;
  p.N = (int)N;
  p.K = (int)K;
  p.epi = epi;
  MB_CHECK_CUDA((device_info::allow_shared<gemm_tcgen05_grouped_kernel<MODE, BN, TA>>(Cfg::kSmem)));
  gemm_tcgen05_grouped_kernel<MODE, BN, TA><<<sms, TG_THREADS, Cfg::kSmem, stream>>>(map_a, maps, p, plan);
  MB_CHECK_LAUNCH("gemm_tcgen05_grouped_kernel");
  return MB200_OK;
}

// Pairs of CTAs over the plan's token tiles (packed experts: w_n | w_k != 0, one map).  No tile is cut along k: how many tiles a rank has depends on the
// experts it owns, and a row's sum must not, so that every number of ranks gives the same bits.  (With cuts the layer, eight experts of ~512 rows at 4096 x 14336, took
// 1535 us instead of 1550.)
template <int MODE>
int launch_grouped_pair(const CUtensorMap& map_a, const MoeWeightMaps& maps, int64_t rows_cap, int64_t K, int64_t N, int64_t w_n, int64_t w_k, const int32_t* plan,
                        const EpiParams& epi, int sms, cudaStream_t stream) {
  PairParams p;
  p.T = (int)rows_cap;
  p.N = (int)N;
  p.K = (int)K;
  p.epi = epi;
  p.w_n = (int)w_n;
  p.w_k = (int)w_k;
  p.units = sms / 2;
  if (K >= GP_DRAW_MIN_K) p.draw = reinterpret_cast<unsigned*>(const_cast<int32_t*>(plan) + 7);
  MB_CHECK_CUDA(device_info::allow_shared<gemm_pair_grouped_kernel<MODE>>(GP_SMEM));
  return launch_pairs(gemm_pair_grouped_kernel<MODE>, p.units, stream, map_a, maps, p, plan);
}

// tile width: prefill (128-row tiles) takes the widest tile that divides N; decode-sized calls (32-row tiles, HBM-bound) pick the
// width that fills the rounds of the persistent schedule best for the EXPECTED number of touched experts
// decode-sized calls: the stream-K weight-streaming kernel over (expert segment, n tile, k block) units
template <int MODE, int TA>
int launch_grouped_streamk(const void* a, int64_t rows_cap, int64_t K, int64_t N, const void* const* w_host, int E, const int32_t* plan,
                           const EpiParams& epi, void* workspace, size_t workspace_bytes, size_t header, int sms, cudaStream_t stream) {
  using Cfg = TgCfg<SK_BN, TA>;
  if (sms > SK_MAX_CTAS) sms = SK_MAX_CTAS;
  if (workspace == nullptr || workspace_bytes < header + SK_PARTIAL_BYTES) return fail(MB200_E_WORKSPACE, "grouped stream-K gemm: workspace %zu < %zu", workspace_bytes, header + SK_PARTIAL_BYTES);
  CUtensorMap map_a;
  MoeWeightMaps maps;
  int rc = make_tensor_map_2d(&map_a, a, rows_cap, K, TA);
  if (rc) return rc;
  rc = make_expert_maps(&maps, map_a, w_host, E, N, K, SK_BN);
  if (rc) return rc;
  SkParams p;
  p.T = (int)rows_cap;
  p.N = (int)N;
  p.K = (int)K;
  p.epi = epi;
  p.partials = reinterpret_cast<float*>((uint8_t*)workspace + header);
  p.flags = reinterpret_cast<unsigned*>((uint8_t*)workspace + SK_FLAGS_OFFSET);
  MB_CHECK_CUDA((device_info::allow_shared<gemm_streamk_grouped_kernel<MODE, TA>>(Cfg::kSmem)));
  MB_CHECK_CUDA(launch_pdl(gemm_streamk_grouped_kernel<MODE, TA>, dim3((unsigned)sms), dim3(TG_THREADS), (size_t)Cfg::kSmem, stream, map_a, maps, p, plan));
  return MB200_OK;
}

template <int MODE>
int launch_grouped(const void* a, int64_t rows_cap, int64_t K, int64_t N, const void* const* w_host, int E, int64_t pairs, int est_mtiles, int tile_rows,
                   const int32_t* plan, const EpiParams& epi, void* workspace, size_t workspace_bytes, size_t header, cudaStream_t stream) {
  const int sms = device_info::sm_count();
  if (sms == 0) return fail(MB200_E_CUDA, "no device");
  MB_CHECK_ARG(K % TG_BK == 0 && N % 32 == 0, "grouped gemm: K=%lld must be a multiple of 64, N=%lld of 32", (long long)K, (long long)N);
  if (tile_rows < 128 && streamk_eligible(tile_rows, N, K)) {
    if (tile_rows == 32) return launch_grouped_streamk<MODE, 32>(a, rows_cap, K, N, w_host, E, plan, epi, workspace, workspace_bytes, header, sms, stream);
    return launch_grouped_streamk<MODE, 64>(a, rows_cap, K, N, w_host, E, plan, epi, workspace, workspace_bytes, header, sms, stream);
  }
  if (tile_rows == 128) {
    // From about 128 rows an expert, where the GEMMs below begin to need two tiles of tokens for one.  The layer of eight experts of 4096 x 14336 with the GEMMs below and with pairs, us:
    // 300 tokens (75 rows an expert) 527, 550, 450 530, 562, 600 681, 594, 800 695, 631, 1000 829, 781, 1300 948, 938; of 6144 x 16384: 400 872, 876, 800 1192, 1018, 1200 1678, 1584.
    if (N % 128 == 0 && tcgen05_cluster_enabled() && moe_plan_lists_pairs(pairs) && rows_cap >= (int64_t)E * 256) {
      CUtensorMap map_a;
      MoeWeightMaps maps;
      int rc = make_tensor_map_2d(&map_a, a, rows_cap, K, TG_BM);
      if (rc) return rc;
      rc = make_expert_maps(&maps, map_a, w_host, E, N, K, TG_BM);
      if (rc) return rc;
      return launch_grouped_pair<MODE>(map_a, maps, rows_cap, K, N, 0, 0, plan, epi, sms, stream);
    }
    if (N % 256 == 0) return launch_grouped_bn<MODE, 256, 128>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    if (N % 128 == 0) return launch_grouped_bn<MODE, 128, 128>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    if (N % 64 == 0) return launch_grouped_bn<MODE, 64, 128>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    return launch_grouped_bn<MODE, 32, 128>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
  }
  int best = 32;
  double best_score = -1.0;
  const int forced = tcgen05_forced_bn();
  const int cand[4] = {256, 128, 64, 32};
  for (int i = 0; i < 4; ++i) {
    const int bn = cand[i];
    if (N % bn != 0) continue;
    if (forced == bn) {
      best = bn;
      break;
    }
    const int64_t tiles = (int64_t)est_mtiles * (N / bn), rounds = (tiles + sms - 1) / sms;
    const double score = (double)tiles / (double)(rounds * sms);
    if (score > best_score + 0.02) {  // wider tiles (bigger TMA boxes) unless a narrower one fills the rounds clearly better
      best_score = score;
      best = bn;
    }
  }
  if (tile_rows == 64) {
    switch (best) {
      case 256: return launch_grouped_bn<MODE, 256, 64>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
      case 128: return launch_grouped_bn<MODE, 128, 64>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
      case 64: return launch_grouped_bn<MODE, 64, 64>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
      default: return launch_grouped_bn<MODE, 32, 64>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    }
  }
  switch (best) {
    case 256: return launch_grouped_bn<MODE, 256, 32>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    case 128: return launch_grouped_bn<MODE, 128, 32>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    case 64: return launch_grouped_bn<MODE, 64, 32>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
    default: return launch_grouped_bn<MODE, 32, 32>(a, rows_cap, K, N, w_host, E, plan, epi, sms, stream);
  }
}

// ---- the mixtures of layered decoders ---------------------------------------------------------------------------------------
// Prompts of a layered decoder ran EVERY expert on every token (two plain Linears, unchosen experts scaled by 0): E / top times the
// useful flops.  With the plan and the grouped GEMMs of this file only the chosen (token, expert) rows are computed:
//   layer_moe_gather   xs[slot] = hn[token], row_w[slot] = routing weight (fp32)
//   grouped GEMM       act = step(xs W13_e^T) * row_w            (EPI_LAYER; the roundings of the dense form)
//   grouped GEMM       rows32 = act W2_e^T                       (fp32 rows: the sum over a token's experts is never below fp32)
//   layer_moe_combine  y32[t] (+)= sum_j rows32[slot(t, j)]      in the order of the token's choices: no atomics, the same bits each time
// The experts lie packed in one matrix each (w13 [E * units, width], w2 [width, E * ff]): one tensor map, offsets by expert.
// Choices >= E (identity experts) get no row; the combine adds them as the token itself.  A mixture's prompt of 2500 tokens, 16 experts of 1408, top 4 of 20 outputs,
// width 2048: 800 us before (all experts on all tokens), 248 us now, of which ~150 us are the grouped GEMMs, 24 the router and 12 the plan.
__global__ void __launch_bounds__(256) layer_moe_gather_kernel(const uint4* hn, const float* wsel, const int32_t* slot,
                                                               int pairs, int k, int row_chunks, uint4* __restrict__ xs, float* __restrict__ row_w) {
  pdl_trigger();
  pdl_wait();
  const int pair = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (pair >= pairs) return;
  const int s = slot[pair];
  if (s < 0) return;
  if (lane == 0) row_w[s] = wsel[pair];
  const uint4* src = hn + (int64_t)(pair / k) * row_chunks;
  uint4* dst = xs + (int64_t)s * row_chunks;
#pragma unroll 4
  for (int c = lane; c < row_chunks; c += 32) dst[c] = src[c];
}

// identity: a choice without a row is an identity expert, the token itself (hn) times the choice's weight
__global__ void __launch_bounds__(256) layer_moe_combine_kernel(const float4* rows, const int32_t* slot, const float* wsel, const uint2* hn, float4* __restrict__ y, int k, int row_quads, int add, int identity) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * 256 + threadIdx.x, t = blockIdx.y;
  if (c >= row_quads) return;
  const int32_t* sl = slot + (int64_t)t * k;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  float4* dst = y + (int64_t)t * row_quads + c;
  float4 o = acc;
  if (add) o = *dst;
  float own = 0.f;  // the identity experts' weights
  for (int j0 = 0; j0 < k; j0 += 8) {
    float4 v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int s = j0 + j < k ? sl[j0 + j] : -1;
      v[j] = s >= 0 ? __ldcs(rows + (int64_t)s * row_quads + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (identity && s < 0 && j0 + j < k) own += wsel[(int64_t)t * k + j0 + j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) acc.x += v[j].x, acc.y += v[j].y, acc.z += v[j].z, acc.w += v[j].w;
  }
  if (own != 0.f) {
    const uint2 h = hn[(int64_t)t * row_quads + c];
    acc.x = fmaf(own, bf16lo(h.x), acc.x), acc.y = fmaf(own, bf16hi(h.x), acc.y);
    acc.z = fmaf(own, bf16lo(h.y), acc.z), acc.w = fmaf(own, bf16hi(h.y), acc.w);
  }
  if (add) {
    acc.x += o.x, acc.y += o.y, acc.z += o.z, acc.w += o.w;
  }
  *dst = acc;
}

// w: rows x cols, expert e at row e * w_n, column e * w_k.  N % 128 == 0, K % 64 == 0.
inline int launch_grouped_packed(const void* a, int64_t rows_cap, int64_t K, int64_t N, const void* w, int64_t w_rows, int64_t w_cols, int64_t w_n, int64_t w_k,
                                 int64_t pairs, int64_t E, const int32_t* plan, const EpiParams& epi, cudaStream_t stream) {
  const int sms = device_info::sm_count();
  if (sms == 0) return fail(MB200_E_CUDA, "no device");
  CUtensorMap map_a;
  MoeWeightMaps maps;
  int rc = make_tensor_map_2d(&map_a, a, rows_cap, K, TG_BM);
  if (rc) return rc;
  rc = make_tensor_map_2d(&maps.m[0], w, w_rows, w_cols, TG_BM);
  if (rc) return rc;
  for (int e = 1; e < MOE_MAX_EXPERTS; ++e) maps.m[e] = maps.m[0];
  // Wherever the plan lists token tiles of pairs (more than 512 rows in all).  16 experts of 1408, width 2048, with the GEMM below and with pairs, us: 130 tokens 117, 114, 250 102, 97,
  // 450 104, 103, 800 135, 123, 1300 162, 143; eight of 14336, width 4096: 300 tokens 539, 523, 600 772, 580, 1000 923, 776, 1300 1126, 998.
  if (tcgen05_cluster_enabled() && moe_plan_lists_pairs(pairs))
    return launch_grouped_pair<EPI_LAYER>(map_a, maps, rows_cap, K, N, w_n, w_k, plan, epi, sms, stream);
  using Cfg = TgCfg<128, 128, kEpiSmem<EPI_LAYER>>;
  TcGemmParams p;
  p.T = (int)rows_cap;
  p.N = (int)N;
  p.K = (int)K;
  p.epi = epi;
  p.w_n = (int)w_n;
  p.w_k = (int)w_k;
  MB_CHECK_CUDA((device_info::allow_shared<gemm_tcgen05_grouped_kernel<EPI_LAYER, 128, 128>>(Cfg::kSmem)));
  gemm_tcgen05_grouped_kernel<EPI_LAYER, 128, 128><<<sms, TG_THREADS, Cfg::kSmem, stream>>>(map_a, maps, p, plan);
  MB_CHECK_LAUNCH("gemm_tcgen05_grouped_kernel<layer>");
  return MB200_OK;
}

}  // namespace mb200
