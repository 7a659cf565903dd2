// Prompt attention (varlen, causal, sliding window, optional bias by distance; head size 128) on tcgen05 / TMEM / TMA.
//
// Keys and values come from up to three runs of consecutive positions: the old ring (one run, or two when it wraps) and the call's own
// rows.  One kernel serves first prompts, portions of prompts over a partly filled ring, and the layered decoders' attention, whose keys
// all lie in the ring.
//
// Roofline: tensor pipe and MUFU alike (a 128 x 128 tile is 1024 cycles of MMA for S and P V and 1024 of exp2; 4096 tokens under
// ncu: tensor pipe 44 % of the cycles).  CTA = (two query heads
// of one key/value head, 128 queries, sequence): the two S tiles share every K and V tile, and while the softmax warps of one head work the
// tensor cores work for the other.  10 warps:
//   warp 0    TMA producer: both Q tiles once, then K, V, K, V, ... tiles of 128 keys (two 128B-swizzled [128 x 64] boxes) into a ring of 32 KB slots
//   warp 1    MMA issuer: S_u = Q_u K^T (both K-major from shared memory); O_u += P_u V with P from TENSOR MEMORY and V MN-major.  Order per tile:
//             PV_0(t) S_0(t+1) PV_1(t) S_1(t+1): S_u(t+1) overwrites P_u(t), which lies in S_u's own columns, after PV_u(t) (in-order pipe)
//   warps 2-5, 6-9  softmax of head 0, head 1: one thread per query row: its 128 scores are read once, masked on the tiles that an edge cuts,
//             maximum and sum stay in the thread.  O is rescaled only when a maximum grew by more than 2^8 (P stays far inside bf16's range)
// TMEM columns: S_0 / P_0 at 0, S_1 / P_1 at 128, O_0 at 256, O_1 at 384.
//
// Key tiles are laid from the END of a run backwards: rows before the run are older tokens, another sequence's rows (own rows) or, below row 0,
// zeros of the copy engine.  A tile laid forwards would read ring rows that nothing has written yet.  The mask makes the weights of rows before the
// run 0, but 0 x NaN is not 0: on a run's first tile (three at most per CTA) the softmax warps of head 0 overwrite those rows of V with zeros, so
// that a sequence's infinities stay its own and tokens before a tile's window do not count at all.
//
// One head per CTA, two S buffers, two threads per row (before): 191 us a layer at T = 4096, 32 / 8 heads; portions of prompts and the
// layered decoders went through mma.sync kernels: 520 us for 3 x ~650 queries over ~2900 keys, 1997 us for 4096 queries with a bias.
#pragma once
#include "gemm_tcgen05.cuh"

namespace mb200 {

constexpr int FA_BM = 128, FA_BN = 128, FA_THREADS = 320;
constexpr int FA_TILE_BYTES = 128 * kHeadDim * 2;  // one [128 x 128] bf16 tile = two swizzled [128 x 64] boxes = 32 KB
constexpr int FA_SLOTS = 4;
constexpr int FA_TMEM_COLS = 512, FA_COL_O = 256;
constexpr int FA_SMEM_BASE = FA_TILE_BYTES * (2 + FA_SLOTS) + 256;       // Q_0, Q_1, the ring, barriers
constexpr int FA_BIAS_PAD = 128;                                          // distances below 0 (masked) before a table, above its end behind it
constexpr int FA_MAX_TAB = (232448 - FA_SMEM_BASE) / 8 - 3 * FA_BIAS_PAD;  // entries of a distance table that fit beside the tiles, two heads
constexpr float FA_LAZY = 8.f;                                            // log2 units a maximum may grow before O is rescaled

struct FaParams {
  const int32_t* q_start;  // [B+1]
  const int32_t* seqpos;   // [B] tokens before this call, or null: none
  const int32_t* slots;    // [B] ring row block of each sequence, or null: sequence b in block b
  const float* bias;       // [n_tab, H] added to the scaled scores by distance (larger distances: the last row), or null
  bf16* out;               // [T, H*hd]
  int B, W, window, H, KV; // W: rows of a ring block; window: positions a query sees, itself included
  int own;                 // 1: keys from seqpos on are the call's own rows; 0: every key is in the ring
  int n_tab;
  float scale_log2;
};

constexpr uint32_t kIdescQK = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(FA_BN >> 3) << 17) | ((uint32_t)(FA_BM >> 4) << 24);
constexpr uint32_t kIdescPV = kIdescQK | (1u << 16);  // b_major = MN: V tile rows are keys (K), contiguous along head_dim (N)

// MN-major, 128B-swizzled operand made of [keys x 64 dims] boxes: 8-key groups 1024 B apart (SBO), 64-dim blocks one box apart (LBO)
__device__ __forceinline__ uint64_t umma_desc_sw128_mn(uint32_t smem_addr, uint32_t box_bytes) {
  return (uint64_t)((smem_addr & 0x3ffff) >> 4) | ((uint64_t)(box_bytes >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
         ((uint64_t)2 << 61);
}
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n"
      "}\n" ::"r"(tmem_d),
      "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
               "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}

// The key tiles of one query tile.  A run [lo, hi) of positions is cut into tiles of 128 that end at hi; position pos of the run is row
// pos - shift of its source.
struct FaRuns {
  int lo[3], hi[3], shift[3], first[4];  // first[i]: tile index at which run i starts; runs 0 and 1: ring, run 2: own rows
  __device__ __forceinline__ void run_of(int t, int& pos0, int& run_lo, int& row, bool& ring) const {
    const int i = t >= first[2] ? 2 : (t >= first[1] ? 1 : 0);
    run_lo = i == 2 ? lo[2] : (i == 1 ? lo[1] : lo[0]);
    const int h = i == 2 ? hi[2] : (i == 1 ? hi[1] : hi[0]), end = i == 2 ? first[3] : (i == 1 ? first[2] : first[1]);
    pos0 = h - (end - t) * FA_BN;
    row = pos0 - (i == 2 ? shift[2] : (i == 1 ? shift[1] : shift[0]));
    ring = i != 2;
  }
};
__device__ __forceinline__ FaRuns fa_runs(const FaParams& p, int seqpos, int tok0, int q_first, int q_last) {
  FaRuns r;
  const int lo = max(0, q_first - p.window + 1);  // the first position any query of the tile sees
  const int ring_hi = p.own ? seqpos : q_last + 1;
  r.lo[0] = r.hi[0] = r.shift[0] = 0;
  r.lo[1] = r.hi[1] = r.shift[1] = 0;
  if (lo < ring_hi) {
    const int turn = ring_hi - 1 - (ring_hi - 1) % p.W;  // position in row 0 of the ring's present turn
    if (lo < turn) {  // the run wraps: all rows have been written
      r.lo[0] = lo;
      r.hi[0] = turn;
      r.shift[0] = turn - p.W;
    }
    r.lo[1] = max(lo, turn);
    r.hi[1] = ring_hi;
    r.shift[1] = turn;
  }
  r.lo[2] = p.own ? max(lo, seqpos) : 0;
  r.hi[2] = p.own ? q_last + 1 : 0;
  r.shift[2] = seqpos - tok0;
  r.first[0] = 0;
  r.first[1] = (r.hi[0] - r.lo[0] + FA_BN - 1) / FA_BN;
  r.first[2] = r.first[1] + (r.hi[1] - r.lo[1] + FA_BN - 1) / FA_BN;
  r.first[3] = r.first[2] + (r.hi[2] - r.lo[2] + FA_BN - 1) / FA_BN;
  return r;
}

// NU: query heads per CTA (2; 1 when a key/value head has an odd number of query heads)
template <int NU, bool BIAS>
__global__ void __launch_bounds__(FA_THREADS, 1)
    attn_prompt_tcgen05_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                               const __grid_constant__ CUtensorMap ring_k, const __grid_constant__ CUtensorMap ring_v, const FaParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];  // SW128 tiles want 1024-byte alignment; there is no room left to pad by hand
  uint8_t* smem = smem_raw;
  if ((smem_u32(smem) & 1023u) != 0) __trap();
  uint8_t* sQ = smem;
  uint8_t* sKV = smem + FA_TILE_BYTES * 2;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + FA_TILE_BYTES * (2 + FA_SLOTS));
  uint64_t* q_full = bars;                    // TMA -> MMA
  uint64_t* kv_full = bars + 1;               // [FA_SLOTS] TMA -> MMA
  uint64_t* kv_empty = kv_full + FA_SLOTS;    // [FA_SLOTS] MMA (commit) -> TMA
  uint64_t* s_full = kv_empty + FA_SLOTS;     // [2] MMA (commit) -> softmax
  uint64_t* p_full = s_full + 2;              // [2] softmax (4 warps) -> MMA
  uint64_t* pv_done = p_full + 2;             // [2] MMA (commit) -> softmax: the product of a tile has read P and written O
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  float* tab = reinterpret_cast<float*>(smem + FA_SMEM_BASE);  // [2][FA_BIAS_PAD + n_tab + 2 * FA_BIAS_PAD], in log2 units

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h0 = blockIdx.x * NU, b = blockIdx.z, g = h0 / (p.H / p.KV);
  const int tok0 = p.q_start[b], s_len = p.q_start[b + 1] - tok0;
  // Heads vary fastest and the heavier (later) query tiles start first: longest-processing-time order for the causal triangle, and the
  // heads of one KV group read the same K/V tiles at the same time (L2 locality).
  const int qt = (int)gridDim.y - 1 - (int)blockIdx.y;
  const int i0 = qt * FA_BM;
  if (i0 >= s_len) return;
  const int seqpos = p.seqpos != nullptr ? p.seqpos[b] : 0;
  const int q_first = seqpos + i0, q_last = seqpos + min(i0 + FA_BM, s_len) - 1;  // positions
  const FaRuns runs = fa_runs(p, seqpos, tok0, q_first, q_last);
  const int n_tiles = runs.first[3];

  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int i = 0; i < FA_SLOTS; ++i) {
      mbar_init(&kv_full[i], 1);
      mbar_init(&kv_empty[i], 1);
    }
    for (int u = 0; u < 2; ++u) {
      mbar_init(&s_full[u], 1);
      mbar_init(&p_full[u], 4);  // one arrive per softmax warp
      mbar_init(&pv_done[u], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, FA_TMEM_COLS);
  if constexpr (BIAS) {
    const int len = p.n_tab + 3 * FA_BIAS_PAD;
    for (int i = threadIdx.x; i < NU * len; i += FA_THREADS) {
      const int u = i / len, d = min(max(i % len - FA_BIAS_PAD, 0), p.n_tab - 1);
      tab[i] = p.bias[(int64_t)d * p.H + h0 + u] * 1.4426950408889634f;
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ================= TMA producer =================
    if (lane == 0) {
      mbar_arrive_expect_tx(q_full, NU * FA_TILE_BYTES);
#pragma unroll
      for (int u = 0; u < NU; ++u) {
        tma_load_2d(sQ + u * FA_TILE_BYTES, &map_q, q_full, (h0 + u) * kHeadDim, tok0 + i0);
        tma_load_2d(sQ + u * FA_TILE_BYTES + FA_TILE_BYTES / 2, &map_q, q_full, (h0 + u) * kHeadDim + 64, tok0 + i0);
      }
      const int block = p.slots != nullptr ? p.slots[b] : b;
      for (int it = 0; it < 2 * n_tiles; ++it) {  // K, V, K, V, ...
        const int s = it % FA_SLOTS, par = (it / FA_SLOTS) & 1;
        int pos0, run_lo, row;
        bool ring;
        runs.run_of(it >> 1, pos0, run_lo, row, ring);
        mbar_wait(&kv_empty[s], par ^ 1, 21, it);
        mbar_arrive_expect_tx(&kv_full[s], FA_TILE_BYTES);
        uint8_t* dst = sKV + s * FA_TILE_BYTES;
        if (ring) {
          const CUtensorMap* m = (it & 1) ? &ring_v : &ring_k;
          tma_load_3d(dst, m, &kv_full[s], g * kHeadDim, row, block);
          tma_load_3d(dst + FA_TILE_BYTES / 2, m, &kv_full[s], g * kHeadDim + 64, row, block);
        } else {
          const CUtensorMap* m = (it & 1) ? &map_v : &map_k;
          tma_load_2d(dst, m, &kv_full[s], g * kHeadDim, row);
          tma_load_2d(dst + FA_TILE_BYTES / 2, m, &kv_full[s], g * kHeadDim + 64, row);
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (one thread, elected by the warp) =================
    {
      mbar_wait(q_full, 0, 22, 0);
      auto issue_s = [&](int u, int t) {  // S_u = Q_u K_t^T: 8 k-steps of 16 dims; dims 0..63 / 64..127 in two boxes 16 KB apart
        const int it = 2 * t, s = it % FA_SLOTS;
        if (u == 0) {
          mbar_wait(&kv_full[s], (it / FA_SLOTS) & 1, 23, t);
          tc_fence_after();
        }
        const uint32_t q_desc = umma_desc_lo(smem_u32(sQ + u * FA_TILE_BYTES)), k_desc = umma_desc_lo(smem_u32(sKV + s * FA_TILE_BYTES));
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            const uint32_t off = ((ks >> 2) * (FA_TILE_BYTES / 2) + (ks & 3) * 32) >> 4;
            umma_bf16(tmem + u * 128, q_desc + off, k_desc + off, kIdescQK, ks ? 1u : 0u);
          }
          umma_commit(&s_full[u]);
          if (u == NU - 1) umma_commit(&kv_empty[s]);
        }
        __syncwarp();
      };
#pragma unroll
      for (int u = 0; u < NU; ++u) issue_s(u, 0);
      for (int t = 0; t < n_tiles; ++t) {
        const int it = 2 * t + 1, s = it % FA_SLOTS;
        const uint32_t v_addr = smem_u32(sKV + s * FA_TILE_BYTES);
#pragma unroll
        for (int u = 0; u < NU; ++u) {
          mbar_wait(&p_full[u], t & 1, 24, t);  // the softmax warps have written P (and rescaled O)
          if (u == 0) mbar_wait(&kv_full[s], (it / FA_SLOTS) & 1, 25, t);
          tc_fence_after();
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks)  // 16 keys per step: P columns 8*ks (bf16 pairs), V rows 16*ks (128 B each)
              umma_bf16_ts(tmem + FA_COL_O + u * 128, tmem + u * 128 + ks * 8, umma_desc_sw128_mn(v_addr + ks * 2048, FA_TILE_BYTES / 2), kIdescPV,
                           (t | ks) ? 1u : 0u);
            umma_commit(&pv_done[u]);
            if (u == NU - 1) umma_commit(&kv_empty[s]);
          }
          __syncwarp();
          if (t + 1 < n_tiles) issue_s(u, t + 1);
        }
      }
    }
  } else if (warp < 2 + 4 * NU) {
    // ================= softmax warps: one thread per query row =================
    const int u = (warp - 2) >> 2;
    const int lane_base = (warp & 3) * 32;  // a warp may touch TMEM lanes 32 * (warp % 4) .. + 31
    const int r = lane_base + lane;         // row in the tile = TMEM lane
    const int q_pos = q_first + r;
    const bool row_valid = i0 + r < s_len;
    const int q_min = row_valid ? q_pos - p.window : 0x3fffffff;  // a key is seen iff q_min < pos <= q_pos (and pos >= its run's first)
    const uint32_t srow = tmem + ((uint32_t)lane_base << 16) + u * 128, orow = srow + FA_COL_O;
    const float* my_tab = tab + u * (p.n_tab + 3 * FA_BIAS_PAD) + FA_BIAS_PAD;
    const float scale = p.scale_log2;
    float m_run = -1.0e30f, l_run = 0.f;
    for (int t = 0; t < n_tiles; ++t) {
      int pos0, run_lo, row;
      bool ring;
      runs.run_of(t, pos0, run_lo, row, ring);
      // Only tiles that an edge cuts need masks (tile-uniform test): the diagonal, the window's lower end, a run's start, rows past the end
      const bool edge = (pos0 + FA_BN - 1 > q_first) || (pos0 <= q_first + FA_BM - 1 - p.window) || (pos0 < run_lo) || (i0 + FA_BM > s_len);
      mbar_wait(&s_full[u], t & 1, 26, t);
      tc_fence_after();
      uint32_t sv[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32_nowait(srow + c * 32, sv[c]);
      tmem_wait_ld();
      if constexpr (BIAS) {
        if (q_first - (pos0 + FA_BN - 1) >= p.n_tab - 1) {  // every distance of the tile is in the table's last row
          const float far = my_tab[p.n_tab - 1];
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[c][e] = __float_as_uint(fmaf(__uint_as_float(sv[c][e]), scale, far));
        } else {
          // distance of column 0; at most n_tab - 2 + 127 + 127 for the rows that count (the table is padded), at least -127
          const float* at = my_tab + min(q_pos - pos0, p.n_tab - 1 + 2 * FA_BIAS_PAD - 1);
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int e = 0; e < 32; ++e) sv[c][e] = __float_as_uint(fmaf(__uint_as_float(sv[c][e]), scale, at[-(c * 32 + e)]));
        }
      }
      if (edge) {
        const int lo = max(q_min + 1, run_lo) - pos0, hi = q_pos - pos0;  // columns lo .. hi are seen
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (c * 32 + e < lo || c * 32 + e > hi) sv[c][e] = 0xff800000u;  // -inf: its exponential is exactly 0
      }
      float mx4[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx4[c] = __uint_as_float(sv[c][0]);
#pragma unroll
        for (int e = 1; e < 32; ++e) mx4[c] = fmaxf(mx4[c], __uint_as_float(sv[c][e]));
      }
      float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      if constexpr (!BIAS) mx *= scale;  // (scale > 0)
      mx = fmaxf(mx, -1.0e30f);          // a row that sees nothing in this tile
      const bool grew = t == 0 ? mx > m_run : mx > m_run + FA_LAZY;
      if (t == 0) {
        m_run = mx;
      } else if (__any_sync(0xffffffffu, grew)) {
        mbar_wait(&pv_done[u], (t - 1) & 1, 27, t);
        tc_fence_after();
        const float m_new = grew ? mx : m_run, corr = ex2_approx(m_run - m_new);
        l_run *= corr;
        m_run = m_new;
        uint32_t v[32];
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          tmem_ld_32x32b_x32(orow + c * 32, v);
#pragma unroll
          for (int e = 0; e < 32; ++e) v[e] = __float_as_uint(__uint_as_float(v[e]) * corr);
          tmem_st_32x32b_x32(orow + c * 32, v);
        }
      }
      // P = exp2(s * scale - m) as bf16 pairs -> TMEM, over the scores' own columns (A operand of the product with V)
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint32_t pk[16];
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float s0 = __uint_as_float(sv[c][e]), s1 = __uint_as_float(sv[c][e + 1]);
          const float e0 = ex2_approx(BIAS ? s0 - m_run : fmaf(s0, scale, -m_run)), e1 = ex2_approx(BIAS ? s1 - m_run : fmaf(s1, scale, -m_run));
          l4[c] += e0 + e1;
          pk[e >> 1] = pack2_rn(e0, e1);
        }
        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(srow + c * 16),
                     "r"(pk[0]), "r"(pk[1]), "r"(pk[2]), "r"(pk[3]), "r"(pk[4]), "r"(pk[5]), "r"(pk[6]), "r"(pk[7]), "r"(pk[8]), "r"(pk[9]),
                     "r"(pk[10]), "r"(pk[11]), "r"(pk[12]), "r"(pk[13]), "r"(pk[14]), "r"(pk[15])
                     : "memory");
      }
      l_run += (l4[0] + l4[1]) + (l4[2] + l4[3]);
      if (pos0 < run_lo && u == 0) {  // (a row's 128 bytes of each box keep their place under the swizzle)
        const int it = 2 * t + 1, s = it % FA_SLOTS, bytes = (run_lo - pos0) * 128;
        mbar_wait(&kv_full[s], (it / FA_SLOTS) & 1, 29, t);
        uint8_t* const v = sKV + s * FA_TILE_BYTES;
        for (int i = r * 16; i < bytes; i += FA_BM * 16) {
          *reinterpret_cast<uint4*>(v + i) = make_uint4(0, 0, 0, 0);
          *reinterpret_cast<uint4*>(v + FA_TILE_BYTES / 2 + i) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[u]);
    }
    // O / l -> bf16 -> global: 256 contiguous bytes per thread
    mbar_wait(&pv_done[u], (n_tiles - 1) & 1, 28, 0);
    tc_fence_after();
    const float inv = row_valid ? 1.f / l_run : 0.f;
    bf16* dst = p.out + (int64_t)(tok0 + i0 + r) * p.H * kHeadDim + (int64_t)(h0 + u) * kHeadDim;
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      uint32_t v[32];
      tmem_ld_32x32b_x32(orow + c * 32, v);
      if (row_valid) {
#pragma unroll
        for (int e = 0; e < 32; e += 8) {
          uint4 o;
          o.x = pack2_rn(__uint_as_float(v[e]) * inv, __uint_as_float(v[e + 1]) * inv);
          o.y = pack2_rn(__uint_as_float(v[e + 2]) * inv, __uint_as_float(v[e + 3]) * inv);
          o.z = pack2_rn(__uint_as_float(v[e + 4]) * inv, __uint_as_float(v[e + 5]) * inv);
          o.w = pack2_rn(__uint_as_float(v[e + 6]) * inv, __uint_as_float(v[e + 7]) * inv);
          *reinterpret_cast<uint4*>(dst + c * 32 + e) = o;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem, FA_TMEM_COLS);
}

// [blocks, rows, cols] bf16 row-major (blocks == 0: a 2-D map [rows, cols]), box = [128 rows x 64 cols], 128-byte swizzle; rows outside 0 .. rows - 1
// read as zero
inline int make_tensor_map_rows(CUtensorMap* map, const void* base, int64_t rows, int64_t cols, int64_t blocks = 0) {
  PFN_encodeTiled enc = get_encode_tiled();
  if (enc == nullptr) return fail(MB200_E_CUDA, "cuTensorMapEncodeTiled entry point not available");
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)(blocks ? blocks : 1)};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)(rows * cols) * 2};
  const cuuint32_t box[3] = {64, 128, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, blocks ? 3 : 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MB200_E_CUDA, "cuTensorMapEncodeTiled (attention) failed (%d)", (int)r);
  return MB200_OK;
}

// MB200_ATTN=mma forces the mma.sync kernel
inline bool tcgen05_attn_enabled() {
  static int forced = -1;
  if (forced < 0) {
    const char* e = getenv("MB200_ATTN");
    forced = (e != nullptr && e[0] == 'm') ? 1 : 0;
  }
  return !forced;
}

// k_new / v_new null: every key is in the ring; cache null: no key is (p.seqpos must be null or all zero)
inline int launch_attn_prompt_tcgen05(FaParams p, const void* q, const void* k_new, const void* v_new, const void* cache_k, const void* cache_v, int64_t blocks,
                                      int64_t T, int64_t max_seqlen, cudaStream_t stream) {
  CUtensorMap mq, mk, mv, rk, rv;
  int rc = make_tensor_map_rows(&mq, q, T, (int64_t)p.H * kHeadDim);
  if (rc) return rc;
  const int64_t cols = (int64_t)p.KV * kHeadDim;
  if (cache_k != nullptr) {
    if ((rc = make_tensor_map_rows(&rk, cache_k, p.W, cols, blocks)) != 0) return rc;
    if ((rc = make_tensor_map_rows(&rv, cache_v, p.W, cols, blocks)) != 0) return rc;
  }
  if (k_new != nullptr) {
    if ((rc = make_tensor_map_rows(&mk, k_new, T, cols)) != 0) return rc;
    if ((rc = make_tensor_map_rows(&mv, v_new, T, cols)) != 0) return rc;
  } else {
    mk = rk;
    mv = rv;
  }
  if (cache_k == nullptr) {
    rk = mk;
    rv = mv;
  }
  p.own = k_new != nullptr;
  const bool two = (p.H / p.KV) % 2 == 0;
  const size_t smem = FA_SMEM_BASE + (p.bias != nullptr ? (size_t)2 * (p.n_tab + 3 * FA_BIAS_PAD) * sizeof(float) : 0);
  auto kernel = p.bias != nullptr ? (two ? attn_prompt_tcgen05_kernel<2, true> : attn_prompt_tcgen05_kernel<1, true>)
                                  : (two ? attn_prompt_tcgen05_kernel<2, false> : attn_prompt_tcgen05_kernel<1, false>);
  MB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const dim3 grid((unsigned)(p.H / (two ? 2 : 1)), (unsigned)ceil_div(max_seqlen, FA_BM), (unsigned)p.B);
  kernel<<<grid, FA_THREADS, smem, stream>>>(mq, mk, mv, rk, rv, p);
  MB_CHECK_LAUNCH("attn_prompt_tcgen05_kernel");
  return MB200_OK;
}

}  // namespace mb200
