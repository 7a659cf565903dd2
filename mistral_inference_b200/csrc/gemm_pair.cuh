// C[T, N] = A[T, K] * W[N, K]^T for prompts, on pairs of CTAs that share MMAs (cta_group::2): 256 features x up to 256 tokens a tile.
//
// Roofline: tensor pipe (2*T*N*K flops), under the power cap for launches of milliseconds.  A cluster of two CTAs is one worker; each CTA copies 128 rows
// of the weight tile and HALF of the token tile, the MMA reads both shared memories: 32 KB per CTA and k-block of 64 out of L2 where a CTA by itself takes
// 48 KB for the same flops.  No copy is multicast: each tile is read by the CTA that holds it.
//
// The WEIGHTS are the MMA's 256 rows and the TOKENS its columns, because the number of columns of an MMA is free (any multiple of 32 up to 256) and that of its rows is not:
// T tokens are dealt to ceil(T / 256) tiles whose widths differ by at most 32, and at most 31 columns of all are padding.  With the tokens as rows the last tile ran
// as 256 rows whatever it held (an MMA of 128 rows over a pair takes as long): 1102 tokens cost 1280 rows, now 1120 columns; eight experts of ~512 rows
// each cost 640 or 768, now what they have, to the next 32.  A k-block of a tile w wide takes 2 w clocks
// and little more.  (256 + w, while one diverged lane issued the MMAs and the copies: see umma_bf16.)
//
// Accumulators therefore lie transposed in TMEM: lane = feature, column = token.  Epilogues work on pairs of features (exchange_pairs, epilogue.cuh); fp32 results
// need not even that, a warp's 32 features of a token are one 128-byte line.  Shared memory stays out of it: the MMAs' operands and the copies take all of its
// bandwidth (64 + 64 bytes a clock), and a turn of 32 x 32 fp32 blocks through it cost 3 to 5 % of a prompt.
//
// Warps: 0 TMA producer, 1 MMA issuer (one thread of the first CTA, for both) and TMEM, 2-9 epilogue (two to a quarter of the lanes, taking turns at its columns).  Both CTAs' copies count on the first CTA's full[]
// barrier; its commits free the stage, and publish the accumulator, in both; both CTAs' epilogues release an accumulator on the first CTA's tmem_empty[].
//
// A last round of tiles that is at most half full is cut along k (split_schedule.cuh); the parts' fp32 sums meet in the first part's epilogue, in the order of k.
//
// GROUPED: the mixtures' form, token tiles from the plan of moe.cuh (pair_expert, pair_info), weights by expert; nothing is cut.  Token tiles there are 32 to 256 wide, and a tile's time
// follows its width: clusters that take every n_cta-th tile drift apart by rounds, and the two or three that share an expert's weight tile no longer meet in L2 (2048 tokens, eight
// experts of 4096 x 14336: 5.4 GB read from memory, 3.9 with the draw).  So a cluster takes the next tile that nobody has: the first CTA's producer draws it from a counter shortly before
// it needs it and hands it to the warps of both CTAs (tile_full, tile_empty): 1545 us without, 1470 with.  Short tiles are dealt, their hand-over costs more (both GEMMs of a layer,
// dealt and drawn, us: 16 experts of 2048 x 1408, 2500 tokens 195, 207; 3072 x 1408 278, 287; eight of 2560 x 5120 349, 361; 3072 x 8192 640, 643; 3584 x 10240 901, 901; 4096 x 14336 1459, 1428): the line
// is GP_DRAW_MIN_K.
#pragma once
#include <type_traits>

#include "gemm_tcgen05.cuh"

namespace mb200 {

constexpr int GP_ROWS = 256;                         // features a tile
constexpr int GP_EPI_WARPS = 8, GP_THREADS = 64 + 32 * GP_EPI_WARPS;
constexpr int GP_W_BYTES = TG_BM * TG_BK * 2;        // a CTA's half of the weight tile, per stage
constexpr int GP_MAX_STAGES = 7, GP_SHAPES = 16, GP_INFO = 32, GP_DRAWN = 4;
constexpr int GP_DRAW_MIN_K = 4096;
constexpr int GP_DRAW_AHEAD = 24, GP_HAND_AHEAD = 14;  // k-blocks before a tile's last: the draw's way to memory and back, and the hand-over's to the other CTA, lie under copies
static_assert(GP_SHAPES > GP_MAX_STAGES + 1, "see shape_s");
template <int MODE>
constexpr int kPairTurn = MODE == EPI_LOGPROB ? GP_EPI_WARPS * 2048 : 0;
template <int MODE>
constexpr int kPairRing = 227 * 1024 - 1024 /*align*/ - 512 /*barriers*/ - kPairTurn<MODE>;
constexpr uint32_t GP_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(GP_ROWS >> 4) << 24);  // + the width in units of 8 at bit 17
constexpr unsigned CUT_GIVEN_UP = 2u;  // a flag: 0, 1 (the part is there), or this
constexpr int TG_MAX_CUTS = 56;        // (cut - 1) * cut_pairs at most: 256 KB each
constexpr size_t TG_CUT_BYTES = (size_t)TG_MAX_CUTS * 2 * TG_BM * 256 * sizeof(float);

// Tiles in the order of tile_mn (gemm_tcgen05.cuh) with blocks of 8 x 9, by steps
struct TileWalk {
  int q, mb, nb, gm, gn;  // place in the block, the block's first token and weight tile, its extents (m fastest)
  __device__ __forceinline__ void block(int num_m, int num_n) {
    const bool one = num_m <= 16;
    gm = one ? num_m : min(8, num_m - mb);
    gn = one ? num_n : min(9, num_n - nb);
  }
  __device__ __forceinline__ void start(int num_m, int num_n) {
    q = mb = nb = 0;
    block(num_m, num_n);
  }
  __device__ __forceinline__ void advance(int by, int num_m, int num_n) {
    q += by;
    while (q >= gm * gn && nb < num_n) {
      q -= gm * gn;
      mb += gm;
      if (mb >= num_m) mb = 0, nb += gn;
      block(num_m, num_n);
    }
  }
  __device__ __forceinline__ int m() const { return mb + (int)((unsigned)q % (unsigned)gm); }
  __device__ __forceinline__ int n() const { return nb + (int)((unsigned)q / (unsigned)gm); }
};

struct PairParams {
  int T, N, K;
  EpiParams epi;
  int w_n = 0, w_k = 0;       // grouped, experts packed in one matrix: see TcGemmParams
  int tok_tiles = 0;          // dense: the tokens are dealt to that many tiles
  int box = 128;              // rows of a CTA's token box: at least half of the widest tile
  int units = 0;              // clusters on the chip
  float* partials = nullptr;  // [TG_MAX_CUTS][2 CTAs][256 / 4][128] float4: what the parts but the first leave for it; null: nothing is cut
  unsigned* flags = nullptr;  // [TG_MAX_CUTS * 2], zero between launches
  unsigned* draw = nullptr;   // grouped: tiles drawn, zero between launches; null: tiles are dealt
};

// (a ring of a fixed number of fixed slots: with both in registers the loop that issues the MMAs took 4 % longer)
constexpr int GP_STAGE_BYTES = 2 * GP_W_BYTES;
template <int MODE>
constexpr int kPairStages = kPairRing<MODE> / GP_STAGE_BYTES;
constexpr int GP_SMEM = 227 * 1024;

// Waits for what the other CTA of the pair has written.
__device__ __forceinline__ void mbar_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok = 0, spins = 0;
  do {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (!ok && ++spins == MB200_WATCHDOG_SPINS) {
      printf("[mb200 watchdog] block %d thread %d: no tile was handed out\n", (int)blockIdx.x, (int)threadIdx.x);
      __trap();
    }
  } while (!ok);
}
// a tile's number into both CTAs' shared memories, and word of it on their barriers
__device__ __forceinline__ void hand_tile(uint32_t* at, uint64_t* bar, uint32_t tile) {
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r)
    asm volatile(
        "{\n"
        ".reg .b32 a, b;\n"
        "mapa.shared::cluster.u32 a, %0, %3;\n"
        "mapa.shared::cluster.u32 b, %1, %3;\n"
        "st.shared::cluster.u32 [a], %2;\n"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [b];\n"
        "}\n" ::"r"(smem_u32(at)),
        "r"(smem_u32(bar)), "r"(tile), "r"(r)
        : "memory");
}

template <int MODE, bool GROUPED>
__device__ __forceinline__ void pair_gemm_body(const CUtensorMap& map_a, const CUtensorMap* map_w_base, const PairParams& p, const int32_t* plan) {
  extern __shared__ uint8_t smem_raw[];
  if (GROUPED) pdl_wait();  // the plan
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);  // SW128 wants 1024-B tiles
  uint8_t* turn = smem + kPairRing<MODE>;
  uint64_t* full = reinterpret_cast<uint64_t*>(turn + kPairTurn<MODE>);
  uint64_t* empty = full + GP_MAX_STAGES;
  uint64_t* tmem_full = empty + GP_MAX_STAGES;  // [2]
  uint64_t* tmem_empty = tmem_full + 2;         // [2]
  uint64_t* cut_full = tmem_empty + 2;          // copies of another part's sums
  uint32_t* tmem_base_slot = reinterpret_cast<uint32_t*>(cut_full + 1);
  volatile uint32_t* cut_lost = tmem_base_slot + 1;
  uint64_t* tile_full = cut_full + 2;              // [GP_DRAWN] grouped: a drawn tile is there (each CTA's own)
  uint64_t* tile_empty = tile_full + GP_DRAWN;     // [GP_DRAWN] everybody has read it (the first CTA's)
  uint32_t* drawn_s = reinterpret_cast<uint32_t*>(tile_empty + GP_DRAWN);  // [GP_DRAWN]
  volatile uint32_t* shape_s = drawn_s + GP_DRAWN;  // [GP_SHAPES] (width / 32) << 24 | k-blocks
  int32_t* info_s = reinterpret_cast<int32_t*>(drawn_s + GP_DRAWN + GP_SHAPES);  // [GP_INFO] grouped: the plan's first token tiles

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = (int)cluster_ctarank();
  const int cta = (int)blockIdx.x >> 1, n_cta = (int)gridDim.x >> 1;  // cluster index / clusters in the grid
  constexpr int stages = kPairStages<MODE>, stage_bytes = GP_STAGE_BYTES;
  const uint32_t arriving = 2u * (uint32_t)(GP_W_BYTES + p.box * TG_BK * 2);  // bytes of a k-block, in both CTAs
  const int num_n = (p.N + GP_ROWS - 1) / GP_ROWS, num_k = p.K / TG_BK;
  const int num_m = GROUPED ? plan[6] : p.tok_tiles;
  const CutPlan cuts = !GROUPED && p.partials != nullptr ? cut_plan((long long)num_m * num_n, num_k, p.units, TG_MAX_CUTS) : CutPlan{0, 1};
  const int whole = num_m * num_n - cuts.cut_pairs, num_tiles = whole + cuts.cut * cuts.cut_pairs;
  const int32_t* item_expert = GROUPED ? plan + MOE_PLAN_HEADER + 2 * plan[2] : nullptr;
  const int32_t* item_info = GROUPED ? item_expert + plan[2] : nullptr;
  const int tok_base = GROUPED ? 0 : (p.T + 31) / 32 / num_m, tok_more = GROUPED ? 0 : (p.T + 31) / 32 % num_m;
  struct Item {
    int mu, t0, width, n0, kb0, kb1;
    int part, slot;  // part of a cut tile (0: the owner, which adds the others' sums), -1: not cut
  };
  // This cluster's items one after the other, without a division by anything but a block's few rows: the walk stands between two tiles' copies, and with the general
  // arithmetic (~1500 cycles) it cost 3 % of a tile with K = 4096.
  struct Walk {
    TileWalk at;
    int prev = 0;
  };
  Walk walk;
  auto next_item = [&](int tile) {
    Item it;
    it.kb0 = 0, it.kb1 = num_k, it.part = -1, it.slot = 0;
    int t = tile;
    if (t >= whole) {
      const CutItem c = cut_item(t - whole, cuts.cut, cuts.cut_pairs);
      it.part = c.part;
      it.slot = c.slot;
      it.kb0 = num_k * it.part / cuts.cut;
      it.kb1 = num_k * (it.part + 1) / cuts.cut;
      t = whole + it.slot;
    }
    walk.at.advance(t - walk.prev, num_m, num_n);
    walk.prev = t;
    it.mu = walk.at.m();
    it.n0 = walk.at.n() * GP_ROWS;
    if (GROUPED) {
      const int info = it.mu < GP_INFO ? info_s[it.mu] : item_info[it.mu];
      it.t0 = info & ~31;
      it.width = 32 * (info & 31);
    } else {  // the first tok32 % num_m tiles are 32 wider
      const int u0 = tok_base * it.mu + min(it.mu, tok_more);
      it.t0 = 32 * u0;
      it.width = 32 * (tok_base + (it.mu < tok_more ? 1 : 0));
    }
    return it;
  };
  walk.at.start(num_m, num_n);
  const bool draws = GROUPED && p.draw != nullptr;
  // The tile behind this cluster's nth.  Every reader of a drawn one (a whole warp, or the other CTA's producer) says so; >= num_tiles: there is none.
  auto tile_after = [&](int tile, uint32_t nth) {
    if (!draws) return tile + n_cta;
    const uint32_t slot = nth % GP_DRAWN;
    mbar_wait_cluster(&tile_full[slot], (nth / GP_DRAWN) & 1);
    const int next = (int)*(volatile uint32_t*)&drawn_s[slot];
    return next;
  };
  auto tile_read = [&](uint32_t nth) { mbar_arrive_cluster(cluster_first(&tile_empty[nth % GP_DRAWN])); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], 2 * GP_EPI_WARPS);  // one arrive per epilogue warp of both CTAs
    }
    mbar_init(cut_full, 1);
    if (GROUPED)
      for (int i = 0; i < GP_DRAWN; ++i) {
        mbar_init(&tile_full[i], 1);
        mbar_init(&tile_empty[i], 2 + 2 * GP_EPI_WARPS);  // the issuing warp, the other CTA's producer, the epilogue warps
      }
    *cut_lost = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    if (!GROUPED) asm volatile("prefetch.tensormap [%0];" ::"l"(map_w_base) : "memory");
  }
  if (GROUPED && warp == 2 && lane < min(num_m, GP_INFO)) info_s[lane] = item_info[lane];
  if (warp == 1) tmem_alloc<2>(tmem_base_slot, 512);
  tc_fence_before();
  cluster_sync_all();  // the peer's barriers must be initialised before any copy or commit reaches them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_slot;
  pdl_trigger();
  if (!GROUPED) pdl_wait();  // barriers, tensor memory and the cluster's meeting are behind the predecessor's end

  if (warp == 0) {
    // ================= TMA producer (one thread, elected by the warp, which walks as a whole) =================
    const uint32_t full_first = cluster_first(full);
    uint32_t s = 0, par = 0, it = 0, nth = 0;
    for (int tile = cta; tile < num_tiles; ++nth) {
      const Item w = next_item(tile);
      const uint32_t shape = (uint32_t)(w.width / 32) << 24 | (uint32_t)(w.kb1 - w.kb0);
      const int expert = GROUPED ? item_expert[w.mu] : 0;
      const bool packed = GROUPED && (p.w_n | p.w_k) != 0;
      const CUtensorMap* wmap = map_w_base + (packed ? 0 : expert);
      const int wr = w.n0 + rank * TG_BM + (packed ? expert * p.w_n : 0), wc = packed ? expert * p.w_k : 0;
      const int t0 = w.t0 + rank * (w.width / 2);
      if (elect_one()) shape_s[nth & (GP_SHAPES - 1)] = shape;  // for the MMA warp; more slots than stages: the one it still reads is not overwritten
      auto copy = [&](int kb0, int kb1) {
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          mbar_wait(&empty[s], par ^ 1, 11, it);
          if (elect_one()) {
            // the pair's four tiles count on the first CTA's barrier (the other CTA's may land before it is armed: the count goes negative)
            if (rank == 0) mbar_arrive_expect_tx(&full[s], arriving);
            uint8_t* const st = smem + s * stage_bytes;
            const uint32_t bar = full_first + s * 8u;
            tma_load_2d_pair(st, wmap, bar, wc + kb * TG_BK, wr);
            tma_load_2d_pair(st + GP_W_BYTES, &map_a, bar, kb * TG_BK, t0);
          }
          __syncwarp();
          if (++s == (uint32_t)stages) {
            s = 0;
            par ^= 1;
          }
        }
      };
      if (!draws) {
        copy(w.kb0, w.kb1);
        tile += n_cta;
      } else if (rank == 0) {  // every cluster that had a tile draws once in vain, so there are num_tiles draws: the last puts the counter back
        const uint32_t slot = nth % GP_DRAWN;
        const int draw_at = max(w.kb1 - GP_DRAW_AHEAD, w.kb0), hand_at = max(w.kb1 - GP_HAND_AHEAD, w.kb0);
        unsigned drawn = 0;
        copy(w.kb0, draw_at);
        if (lane == 0) drawn = atomicAdd(p.draw, 1u);
        copy(draw_at, hand_at);
        tile = n_cta + (int)__shfl_sync(0xffffffffu, drawn, 0);
        mbar_wait(&tile_empty[slot], ((nth / GP_DRAWN) & 1) ^ 1, 16, nth);
        if (lane == 0) {
          hand_tile(&drawn_s[slot], &tile_full[slot], (uint32_t)tile);
          if (drawn == (unsigned)num_tiles - 1u) *(volatile unsigned*)p.draw = 0u;
        }
        __syncwarp();
        copy(hand_at, w.kb1);
      } else {
        copy(w.kb0, w.kb1);
        tile = tile_after(tile, nth);
        __syncwarp();
        if (lane == 0) tile_read(nth);
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (one thread, for both CTAs) =================
    // The warp walks as a whole and elects a lane to issue, so that descriptors and counters are uniform.
    if (rank == 0) {
      const uint32_t ring = umma_desc_lo(smem_u32(smem));
      uint32_t s = 0, par = 0, it = 0, acc_it = 0;
      for (int tile = cta; tile < num_tiles; ++acc_it) {
        const uint32_t acc = acc_it & 1, acc_par = (acc_it >> 1) & 1;
        mbar_wait(&tmem_empty[acc], acc_par ^ 1, 12, acc_it);  // the epilogue has drained this accumulator buffer
        mbar_wait(&full[s], par, 13, it);
        tc_fence_after();
        const uint32_t shape = shape_s[acc_it & (GP_SHAPES - 1)];  // written before the producer armed this stage
        const int n_kb = (int)(shape & 0xffffff);
        const uint32_t d_tmem = tmem_base + acc * 256;
        auto k_blocks = [&](auto width32) {  // (the width a constant of the instructions: as a register it took 3 % of the tile)
          constexpr uint32_t idesc = GP_IDESC | (decltype(width32)::value * 4u) << 17;
          for (int kb = 0; kb < n_kb; ++kb, ++it) {
            if (kb > 0) mbar_wait(&full[s], par, 13, it);
            tc_fence_after();
            const uint32_t wdesc = ring + s * (stage_bytes >> 4), tdesc = wdesc + (GP_W_BYTES >> 4);
            if (elect_one()) {
              umma_bf16_pair(d_tmem, wdesc, tdesc, idesc, kb > 0 ? 1u : 0u);
#pragma unroll
              for (int k = 1; k < TG_BK / 16; ++k)  // +32 bytes (= 2 in 16-byte units) per K = 16 step inside the 128-byte swizzled row
                umma_bf16_pair(d_tmem, wdesc + 2 * k, tdesc + 2 * k, idesc, 1u);
              umma_commit_pair(&empty[s]);  // frees the stage in both CTAs when these MMAs have read it
            }
            __syncwarp();
            if (++s == (uint32_t)stages) {
              s = 0;
              par ^= 1;
            }
          }
        };
        switch (shape >> 24) {
          case 1: k_blocks(std::integral_constant<uint32_t, 1>()); break;
          case 2: k_blocks(std::integral_constant<uint32_t, 2>()); break;
          case 3: k_blocks(std::integral_constant<uint32_t, 3>()); break;
          case 4: k_blocks(std::integral_constant<uint32_t, 4>()); break;
          case 5: k_blocks(std::integral_constant<uint32_t, 5>()); break;
          case 6: k_blocks(std::integral_constant<uint32_t, 6>()); break;
          case 7: k_blocks(std::integral_constant<uint32_t, 7>()); break;
          default: k_blocks(std::integral_constant<uint32_t, 8>()); break;
        }
        if (elect_one()) umma_commit_pair(&tmem_full[acc]);  // accumulator complete, in both CTAs
        tile = tile_after(tile, acc_it);
        __syncwarp();
        if (draws && lane == 0) tile_read(acc_it);
      }
    }
  } else {
    // ========== epilogue warps 2..9: TMEM lanes (features) 32 * (warp % 4) .. + 31, every second block of 32 columns (tokens) ==========
    const int lane_base = (warp & 3) * 32, row = lane_base + lane, first = (warp - 2) >> 2;
    uint32_t acc_it = 0;
    auto after = [&](int tile) {
      const int next = tile_after(tile, acc_it);
      __syncwarp();
      if (draws && lane == 0) tile_read(acc_it);
      return next;
    };
    for (int tile = cta; tile < num_tiles; tile = after(tile), ++acc_it) {
      const Item w = next_item(tile);
      const int n = w.n0 + rank * TG_BM + lane_base;  // this warp's 32 features
      const int chunks = w.width / 32;
      const uint32_t acc = acc_it & 1, acc_par = (acc_it >> 1) & 1;
      // what the first block's step reads is requested while the MMAs run, what the next one's reads while this one is stored
      const bool mine = n < p.N && w.part <= 0, f32_step = MODE == EPI_LAYER && layer_step_is_f32(p.epi.layer);  // (the last weight tile may run past N)
      const int half = (lane & 1) * 16, n2 = n + (lane & ~1);  // a lane's share of a block of 32 x 32: tokens half .. + 15, features n2, n2 + 1 (of fp32 results: all tokens, feature n + lane)
      auto rows_of = [&](int c) { return mine && c < chunks ? min(f32_step ? 32 : 16, p.T - w.t0 - c * 32 - (f32_step ? 0 : half)) : 0; };
      uint32_t next[MODE == EPI_LAYER ? 32 : 16];
      auto fetch = [&](int c) {
        if constexpr (MODE == EPI_LAYER) {
          if (f32_step)
            epi_layer32_f32_lanes_fetch(p.epi, w.t0 + c * 32, rows_of(c), n + lane, next);
          else if (p.epi.rowscale != nullptr && p.epi.rs_pitch == 1)
            epi_pairs16_fetch<MODE>(p.epi, w.t0 + c * 32 + half, rows_of(c), n2, reinterpret_cast<uint32_t(&)[16]>(next));
        } else {
          epi_pairs16_fetch<MODE>(p.epi, w.t0 + c * 32 + half, rows_of(c), n2, next);
        }
      };
      fetch(first);
      mbar_wait(&tmem_full[acc], acc_par, 14, acc_it);
      tc_fence_after();
      const uint32_t trow = tmem_base + ((uint32_t)lane_base << 16) + acc * 256;
      uint32_t va[32];
      bool lost = false;  // a part of this tile never came
      auto add_part = [&](int c) {  // columns 32 c .. + 31 of the part that lies in the ring: quads of 128 rows side by side
        const float4* src = reinterpret_cast<const float4*>(smem) + row;
        const float none = __uint_as_float(0x7fffffffu);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float4 x = lost ? make_float4(none, none, none, none) : src[(c * 8 + q) * TG_BM];
          va[4 * q] = __float_as_uint(__uint_as_float(va[4 * q]) + x.x);
          va[4 * q + 1] = __float_as_uint(__uint_as_float(va[4 * q + 1]) + x.y);
          va[4 * q + 2] = __float_as_uint(__uint_as_float(va[4 * q + 2]) + x.z);
          va[4 * q + 3] = __float_as_uint(__uint_as_float(va[4 * q + 3]) + x.w);
        }
      };
      auto release = [&]() {  // the MMA thread may overwrite this accumulator buffer
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(cluster_first(&tmem_empty[acc]));
      };
      if (w.part > 0) {
        // a later part of a cut tile: its fp32 sums go to the owner, column quads of 128 rows side by side
        const int at = ((w.part - 1) * cuts.cut_pairs + w.slot) * 2 + rank;
        float4* dst = reinterpret_cast<float4*>(p.partials) + (size_t)at * 64 * TG_BM + row;
#pragma unroll 1
        for (int c = first; c < chunks; c += 2) {
          tmem_ld_32x32b_x32(trow + c * 32, va);
#pragma unroll
          for (int q = 0; q < 8; ++q)
            dst[(c * 8 + q) * TG_BM] = make_float4(__uint_as_float(va[4 * q]), __uint_as_float(va[4 * q + 1]), __uint_as_float(va[4 * q + 2]), __uint_as_float(va[4 * q + 3]));
        }
        asm volatile("fence.proxy.async;" ::: "memory");
        __threadfence();
        asm volatile("bar.sync 2, 256;" ::: "memory");
        if (threadIdx.x == 64) {
          __threadfence();
          if (atomicExch(p.flags + at, 1u) == CUT_GIVEN_UP) atomicExch(p.flags + at, 0u);
        }
        release();
        continue;
      }
      if (w.part == 0) {
        // The owner: the other parts lie on lower clusters (cut_item).  This CTA's ring is free (its last MMA has completed): each part's sums (128 KB at
        // full width) come in by bulk copies and are added in the order of k -- all but the last into the accumulator, the last in the epilogue below.
        // (Loaded 128 bytes per thread and column chunk instead, a launch paid ~12 us of L2 latency here.)
        for (int o = 0; o < cuts.cut - 1; ++o) {
          if (threadIdx.x == 64) {
            const int at = (o * cuts.cut_pairs + w.slot) * 2 + rank;
            unsigned spins = 0, there = 0u;
            while ((there = ld_acquire_u32(p.flags + at)) == 0u && ++spins < MB200_WATCHDOG_SPINS) {
            }
            if (there == 0u) {  // gives up: the flag says so to a part that comes after all and puts it back; the tile's results are NaN
              there = atomicCAS(p.flags + at, 0u, CUT_GIVEN_UP);
              __threadfence();
            }
            if (there == 0u) {
              printf("[mb200 watchdog] cluster %d: part %d of tile %d never came\n", cta, o + 1, w.slot);
              *cut_lost = 1u;
            } else {
              p.flags[at] = 0u;  // ready for the next launch
              if (!lost) {
                asm volatile("fence.proxy.async;" ::: "memory");  // written with ordinary stores, read by the copy engine
                const uint32_t copy = TG_BM * 32 * 4;  // 32 columns
                mbar_arrive_expect_tx(cut_full, copy * (uint32_t)chunks);
                const uint8_t* src = reinterpret_cast<const uint8_t*>(p.partials) + (size_t)at * (TG_BM * 256 * 4);
                for (int i = 0; i < chunks; ++i) bulk_load(smem + i * copy, src + i * copy, copy, cut_full);
              }
            }
          }
          asm volatile("bar.sync 2, 256;" ::: "memory");
          lost = *cut_lost != 0u;
          if (lost) continue;  // the other parts' flags still go back to zero
          mbar_wait(cut_full, o & 1, 15, o);
          if (o + 1 < cuts.cut - 1) {
#pragma unroll 1
            for (int c = first; c < chunks; c += 2) {
              tmem_ld_32x32b_x32(trow + c * 32, va);
              add_part(c);
              tmem_st_32x32b_x32(trow + c * 32, va);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("bar.sync 2, 256;" ::: "memory");  // everybody has read: the next part may come
          }
        }
      }
      // One block: this warp's 32 features of tokens w.t0 + 32 c ..
      if (first < chunks) tmem_ld_32x32b_x32_nowait(trow + first * 32, va);
      if constexpr (MODE == EPI_LAYER) {
        if (f32_step) {
#pragma unroll 1
          for (int c = first; c < chunks; c += 2) {
            tmem_wait_ld();
            if (w.part == 0) add_part(c);
            epi_layer32_f32_lanes(p.epi, n + lane, va, next, mine);
            fetch(c + 2);
            epi_layer32_f32_lanes_store(p.epi, w.t0 + c * 32, rows_of(c), n + lane, va);
            if (c + 2 < chunks) tmem_ld_32x32b_x32_nowait(trow + (c + 2) * 32, va);
          }
          release();
          continue;
        }
      }
      const float bias = MODE == EPI_LAYER && p.epi.bias != nullptr && mine ? bf16_to_float(reinterpret_cast<const uint16_t*>(p.epi.bias)[n + lane]) : 0.f;
#pragma unroll 1
      for (int c = first; c < chunks; c += 2) {
        tmem_wait_ld();
        if (w.part == 0) add_part(c);
        uint32_t own[16], y0[8], y1[8], r[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          float lo = __uint_as_float(va[2 * q]), hi = __uint_as_float(va[2 * q + 1]);
          if constexpr (MODE == EPI_LAYER) {
            if (p.epi.bias != nullptr) lo += bias, hi += bias;
          }
          own[q] = pack2_rn(lo, hi);
          r[q] = next[q];
        }
        const int t0 = w.t0 + c * 32, rows = rows_of(c);
        if (c + 2 < chunks) tmem_ld_32x32b_x32_nowait(trow + (c + 2) * 32, va);
        fetch(c + 2);
        exchange_pairs(own, y0, y1);
        if constexpr (MODE == EPI_LOGPROB) {
          // (maximum, sum) per 64 features of a token: a thread takes a token's 32 features of this warp out of shared memory (rows of 64 bytes, 16-byte units
          // XORed with the row), and the odd warp of two hands its pair over there.
          uint32_t* const blk = reinterpret_cast<uint32_t*>(turn + (first * 4 + (warp & 3)) * 2048);
#pragma unroll
          for (int j = 0; j < 16; ++j)
            blk[(half + j) * 16 + ((((lane >> 3) ^ (j >> 1)) & 3) << 2) + ((lane >> 1) & 3)] = __byte_perm(y0[j >> 1], y1[j >> 1], j & 1 ? 0x7632 : 0x5410);
          __syncwarp();
          uint32_t v[32];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 x = *reinterpret_cast<const uint4*>(blk + lane * 16 + (((q ^ (lane >> 1)) & 3) << 2));
            const uint32_t u[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) v[8 * q + 2 * i] = u[i] << 16, v[8 * q + 2 * i + 1] = u[i] & 0xffff0000u;
          }
          const int t = t0 + lane;
          const bool live = mine && t < p.T;
          const long long tgt = live ? p.epi.target[t] : -1;
          const int keep = live ? p.epi.keep_row[t] : -1;
          float m = -INFINITY, sum = 0.f;
          if (live) epi_logprob32(p.epi, t, n, v, tgt, keep, m, sum);
          __syncwarp();
          float2* const meet = reinterpret_cast<float2*>(turn + (first * 4 + ((warp & 3) | 1)) * 2048) + lane;
          const uint32_t id = 4 + first * 2 + (lane_base >> 6);
          if (lane_base & 32) *meet = make_float2(m, sum);
          asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
          if (!(lane_base & 32)) {
            const float2 o = *meet;
            const float mx = fmaxf(m, o.x);
            if (mx != -INFINITY) {  // (a part of nothing but -infinity holds 0, or NaN)
              sum = (m != -INFINITY ? sum * expf(m - mx) : sum) + (o.x != -INFINITY ? o.y * expf(o.x - mx) : o.y);
              m = mx;
            } else {
              sum += o.y;
            }
            if (tgt >= 0) p.epi.partial[(int64_t)t * (p.N / 64) + n / 64] = make_float2(m, sum);
          }
          asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
        } else if (mine) {
          if constexpr (MODE == EPI_LAYER) {
            if (p.epi.rowscale != nullptr)
              epi_layer_pairs16<true>(p.epi, t0 + half, rows, n2, y0, y1, r);
            else
              epi_layer_pairs16<false>(p.epi, t0 + half, rows, n2, y0, y1, r);
          } else
            epi_pairs16<MODE>(p.epi, t0 + half, rows, n2, y0, y1, r);
        }
      }
      release();
    }
  }
  tc_fence_before();
  cluster_sync_all();  // the peer's last commits and arrivals still reach this CTA's barriers, its MMAs this CTA's memory
  if (warp == 1) tmem_dealloc<2>(tmem_base, 512);
}

template <int MODE>
__global__ void __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const PairParams p) {
  pair_gemm_body<MODE, false>(map_a, &map_w, p, nullptr);
}
template <int MODE>
__global__ void __launch_bounds__(GP_THREADS, 1)
    gemm_pair_grouped_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ MoeWeightMaps maps_w, const PairParams p, const int32_t* plan) {
  pair_gemm_body<MODE, true>(map_a, maps_w.m, p, plan);
}

// ---- host -------------------------------------------------------------------------------------------------------------
template <class Kernel, class... Args>
int launch_pairs(Kernel kernel, int clusters, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2u * (unsigned)clusters);
  cfg.blockDim = dim3(GP_THREADS);
  cfg.dynamicSmemBytes = GP_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  MB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
  MB_CHECK_LAUNCH("gemm_pair_kernel");
  return MB200_OK;
}

inline int pair_token_tiles(int64_t T) { return (int)((T + 255) / 256); }

// Whether pairs (and, for k of at least 8192, the parts their tiles would be cut into) fill half of the chip's `units` pairs
inline bool pairs_fill(int64_t T, int64_t N, int64_t K, int units, bool cuts) {
  const int64_t tiles = pair_token_tiles(T) * ((N + GP_ROWS - 1) / GP_ROWS);
  const CutPlan c = cuts && K >= 8192 ? cut_plan(tiles, (int)(K / TG_BK), units, TG_MAX_CUTS) : CutPlan{0, 1};
  return 2 * (tiles + (c.cut - 1) * c.cut_pairs) >= units;
}

// scratch: TG_CUT_BYTES for the sums of cut tiles, flags: 2 * TG_MAX_CUTS words, zero (or neither)
template <int MODE>
int launch_gemm_pair(const GemmParams& g, int sms, cudaStream_t stream, void* scratch, unsigned* flags) {
  PairParams p;
  p.T = g.T;
  p.N = g.N;
  p.K = g.K;
  p.epi = g.epi;
  p.tok_tiles = pair_token_tiles(g.T);
  p.box = 16 * ceil_div(ceil_div(g.T, 32), p.tok_tiles);
  p.units = sms / 2;
  p.partials = reinterpret_cast<float*>(scratch);
  p.flags = flags;
  CUtensorMap map_a, map_w;
  int rc = make_tensor_map_2d(&map_a, g.a, g.T, g.K, p.box);
  if (rc) return rc;
  rc = make_tensor_map_2d(&map_w, g.w, g.N, g.K, TG_BM);
  if (rc) return rc;
  const long long tiles = (long long)p.tok_tiles * ceil_div(g.N, GP_ROWS);
  MB_CHECK_CUDA(device_info::allow_shared<gemm_pair_kernel<MODE>>(GP_SMEM));
  const bool cut = scratch != nullptr && cut_plan(tiles, g.K / TG_BK, p.units, TG_MAX_CUTS).cut_pairs > 0;
  return launch_pairs(gemm_pair_kernel<MODE>, cut || tiles > p.units ? p.units : (int)tiles, stream, map_a, map_w, p);  // (cut: item s of the last round runs on cluster s, so all of them are there)
}

// T >= TG_BM
template <int MODE>
int launch_gemm_tcgen05_prompt(const GemmParams& g, cudaStream_t stream, void* scratch = nullptr, unsigned* flags = nullptr) {
  const int sms = device_info::sm_count();
  if (sms == 0) return fail(MB200_E_CUDA, "no device");
  const int forced = tcgen05_forced_bn();
  const bool pairs = tcgen05_cluster_enabled() && g.N % 128 == 0;
  if ((forced == 128 || forced == 192 || forced == 256) && g.N % forced == 0) {
    if (forced == 256 && pairs && g.T >= 4 * TG_BM) return launch_gemm_pair<MODE>(g, sms, stream, nullptr, nullptr);  // (a pinned width is a plain schedule: nothing is cut)
    if (forced == 256) return launch_gemm_tcgen05_bn<MODE, 256>(g, sms, stream);
    return forced == 192 ? launch_gemm_tcgen05_bn<MODE, 192>(g, sms, stream) : launch_gemm_tcgen05_bn<MODE, 128>(g, sms, stream);
  }
  if (pairs && g.T > TG_BM && pairs_fill(g.T, g.N, g.K, sms / 2, scratch != nullptr)) return launch_gemm_pair<MODE>(g, sms, stream, scratch, flags);
  if (g.N % 256 == 0 && (int64_t)ceil_div(g.T, TG_BM) * (g.N / 256) >= sms) return launch_gemm_tcgen05_bn<MODE, 256>(g, sms, stream);
  if (g.N % 128 == 0) return launch_gemm_tcgen05_bn<MODE, 128>(g, sms, stream);
  return launch_gemm_tcgen05_bn<MODE, 192>(g, sms, stream);
}

template <int MODE>
int launch_gemm_tcgen05(const GemmParams& g, cudaStream_t stream, void* scratch, unsigned* flags) {
  if (g.T >= TG_BM) return launch_gemm_tcgen05_prompt<MODE>(g, stream, scratch, flags);
  const int sms = device_info::sm_count();
  if (sms == 0) return fail(MB200_E_CUDA, "no device");
  return launch_gemm_tcgen05_small<MODE>(g, sms, stream);
}

}  // namespace mb200
