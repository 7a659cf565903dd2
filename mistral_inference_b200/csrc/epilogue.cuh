// Pair epilogues shared by the weight-streaming GEMV (skinny_linear.cuh) and the tensor-core GEMMs.
// Every linear on the hot path hands the epilogue two adjacent fp32 accumulators (columns n, n+1 of
// token t).  That is the natural unit: RoPE rotates the interleaved pair (x[2i], x[2i+1]) (rope.py:18-23)
// and the packed gate/up weight puts w1[i], w3[i] on rows 2i, 2i+1.
#pragma once
#include "common.cuh"
#include "sigmoid.cuh"

namespace mb200 {

enum EpiMode : int {
  EPI_STORE = 0,     // out[t, n] = bf16(acc)
  EPI_RESIDUAL = 1,  // out[t, n] = bf16( bf16(acc) + residual[t, n] )           (transformer_layers.py:166,168)
  EPI_F32 = 2,       // logits[t, n] = float(bf16(acc))                           (transformer.py:235,240)
  EPI_SWIGLU = 3,    // g[t, n/2] = bf16( bf16(silu(bf16(acc0))) * bf16(acc1) )   (transformer_layers.py:106)
  EPI_QKV_ROPE = 4,  // split into q/k/v, rotate q,k pairs, optional ring scatter  (transformer_layers.py:66-70, cache.py:91-92)
  EPI_MOE_SCALE = 5, // yw[row, n] = bf16( w[row] * bf16(acc) ), stored on every rank of an expert-parallel group  (moe.py:31)
  EPI_LAYER = 6,     // the Linears of layered decoders: bias, then the step named by EpiParams::layer (LayerEpi)
  EPI_LOGPROB = 7,   // scoring: the logits bf16(acc) of 64 columns -> (maximum, sum of exp(. - maximum)), the target's logit, whole rows of
                     // logits only where asked for                              (generate.py:97-118)
};

// What follows a layered decoder's Linear (numbers shared with csrc/hybrid/hybrid_linear.cuh, which states the formulas).
enum LayerEpi : int { LAYER_STORE = 0, LAYER_RESIDUAL = 1, LAYER_GLU = 2, LAYER_F32 = 3, LAYER_SWIGLU = 4, LAYER_RESIDUAL_SCALED = 5, LAYER_RELU2 = 6, LAYER_GEGLU = 7 };

constexpr int kMaxPeers = 8;

struct EpiParams {
  void* out = nullptr;             // bf16 [T, ld_out]
  const void* residual = nullptr;  // bf16 [T, ld_out]
  float* out_f32 = nullptr;        // fp32 [T, ld_out]
  int64_t ld_out = 0;
  // EPI_QKV_ROPE
  void* q_out = nullptr;  // [T, q_dim]
  void* k_out = nullptr;  // [T, kv_dim]
  void* v_out = nullptr;  // [T, kv_dim]
  void* cache_k = nullptr;  // [rows, kv_dim]
  void* cache_v = nullptr;
  const int32_t* positions = nullptr;   // [T]
  const int32_t* cache_rows = nullptr;  // [T] or null
  const float* rope = nullptr;          // [n_pos, 64, 2]
  int q_dim = 0, kv_dim = 0;
  // EPI_MOE_SCALE: routing weight of each (token, expert) row; the weighted expert output goes to `out` and to the same offset
  // of the mapped buffers of the other ranks (NVLink peer stores; n_peers == 0 when unsharded)
  const void* row_w = nullptr;  // bf16 [rows]
  void* peer_out[kMaxPeers] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
  int n_peers = 0;
  // EPI_LOGPROB
  const long long* target = nullptr;     // [T]: rows with a negative target need no partial sums
  const int32_t* keep_row = nullptr;     // [T]: row of out_f32 that takes this row's logits, or -1
  float2* partial = nullptr;             // [T, N / 64]
  float* target_logit = nullptr;         // [T]
  // EPI_LAYER
  int layer = 0, n_act = 0;              // LayerEpi; columns below n_act go through SiLU (LAYER_STORE)
  float limit = 0.f, alpha = 0.f;
  const void* bias = nullptr;            // bf16 [N] or null
  const float* rowscale = nullptr;       // fp32 [T, rs_pitch] or null: hidden unit c of row t is scaled by rowscale[t, c / rs_group]
  int rs_pitch = 0, rs_group = 1;
};

template <int MODE>
__device__ __forceinline__ void epi_pair(const EpiParams& p, int t, int n, float acc0, float acc1) {
  // the Linear's own output rounding (bf16 result of nn.Linear)
  const float y0 = round_bf16(acc0), y1 = round_bf16(acc1);
  if constexpr (MODE == EPI_STORE) {
    *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + n) = pack_bf16x2(y0, y1);
  } else if constexpr (MODE == EPI_RESIDUAL) {
    const uint32_t r = *reinterpret_cast<const uint32_t*>(reinterpret_cast<const uint16_t*>(p.residual) + (int64_t)t * p.ld_out + n);
    *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + n) =
        pack_bf16x2(y0 + bf16lo(r), y1 + bf16hi(r));
  } else if constexpr (MODE == EPI_F32) {
    *reinterpret_cast<float2*>(p.out_f32 + (int64_t)t * p.ld_out + n) = make_float2(y0, y1);
  } else if constexpr (MODE == EPI_SWIGLU) {
    const float s = round_bf16(ref_silu(y0));
    reinterpret_cast<bf16*>(p.out)[(int64_t)t * p.ld_out + (n >> 1)] = __float2bfloat16_rn(s * y1);
  } else if constexpr (MODE == EPI_MOE_SCALE) {
    const float w = bf16_to_float(reinterpret_cast<const uint16_t*>(p.row_w)[t]);
    const uint32_t packed = pack_bf16x2(w * y0, w * y1);
    const int64_t off = (int64_t)t * p.ld_out + n;
    *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.out) + off) = packed;
    for (int r = 0; r < p.n_peers; ++r) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.peer_out[r]) + off) = packed;
  } else if constexpr (MODE == EPI_QKV_ROPE) {
    if (n < p.q_dim + p.kv_dim) {  // q or k: rotate
      const int pos = p.positions[t];
      const int i = (n & (kHeadDim - 1)) >> 1;
      const float2 cs = *reinterpret_cast<const float2*>(p.rope + ((int64_t)pos * (kHeadDim / 2) + i) * 2);
      float re, im;
      ref_cmul(y0, y1, cs.x, cs.y, re, im);
      const uint32_t packed = pack_bf16x2(re, im);
      if (n < p.q_dim) {
        *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.q_out) + (int64_t)t * p.q_dim + n) = packed;
      } else {
        const int c = n - p.q_dim;
        *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.k_out) + (int64_t)t * p.kv_dim + c) = packed;
        if (p.cache_rows != nullptr) {
          const int row = p.cache_rows[t];
          if (row >= 0) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.cache_k) + (int64_t)row * p.kv_dim + c) = packed;
        }
      }
    } else {  // v: stored as projected
      const int c = n - p.q_dim - p.kv_dim;
      const uint32_t packed = pack_bf16x2(y0, y1);
      *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.v_out) + (int64_t)t * p.kv_dim + c) = packed;
      if (p.cache_rows != nullptr) {
        const int row = p.cache_rows[t];
        if (row >= 0) *reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(p.cache_v) + (int64_t)row * p.kv_dim + c) = packed;
      }
    }
  }
}

// ---- row-chunk epilogues for the tcgen05 GEMM -------------------------------------------------------------------------------
// There one thread owns one output row and reads its accumulator out of TMEM 32 columns at a time, so the natural unit is
// (row t, columns n .. n+31) with n a multiple of 32: the chunk never straddles a head or the q|k|v boundaries, every store is
// a 16-byte vector, and the per-row metadata (position, ring row) is read once per chunk instead of once per pair.  The
// arithmetic is the same as epi_pair's, except that SiLU uses the hardware exp2/reciprocal (relative error ~1e-6, i.e. a
// one-ulp bf16 flip in ~0.03 % of the gate values -- far below what the accumulation order already does).
__device__ __forceinline__ uint32_t pack2_rn(float lo, float hi) {
  const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);  // one F2FP: .x (low half) = lo
  return *reinterpret_cast<const uint32_t*>(&b);
}
__device__ __forceinline__ float fast_silu(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// What epi_chunk32 will READ for row t, columns n0 .. n0 + 127, requested ahead of time (the thread is about to wait for its
// accumulator): the residual row segment, or the row's position and its RoPE table lines.  Prefetches only -- no registers held.
__device__ __forceinline__ void prefetch_l1(const void* ptr) { asm volatile("prefetch.global.L1 [%0];" ::"l"(ptr)); }
template <int MODE>
__device__ __forceinline__ void epi_prefetch128(const EpiParams& p, int t, int n0) {
  if constexpr (MODE == EPI_RESIDUAL) {
    const uint8_t* src = reinterpret_cast<const uint8_t*>(reinterpret_cast<const uint16_t*>(p.residual) + (int64_t)t * p.ld_out + n0);
    prefetch_l1(src);
    prefetch_l1(src + 128);
  } else if constexpr (MODE == EPI_QKV_ROPE) {
    if (n0 < p.q_dim + p.kv_dim) {
      const int pos = p.positions[t];
      const uint8_t* cs = reinterpret_cast<const uint8_t*>(p.rope + (int64_t)pos * kHeadDim);  // [n_pos, 64, 2] floats: 512 B per position
#pragma unroll
      for (int i = 0; i < 4; ++i) prefetch_l1(cs + 128 * i);
    }
    if (n0 >= p.q_dim && p.cache_rows != nullptr) prefetch_l1(p.cache_rows + t);
  }
}

// EPI_LOGPROB, columns n .. n + 31 of row t.  m, s: running maximum and sum of this row's current 64 columns.
__device__ __forceinline__ void epi_logprob32(const EpiParams& p, int t, int n, const uint32_t (&v)[32], long long tgt, int keep, float& m, float& s) {
  float y[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) y[j] = round_bf16(__uint_as_float(v[j]));
  if (keep >= 0) {
    float4* dst = reinterpret_cast<float4*>(p.out_f32 + (int64_t)keep * p.ld_out + n);
#pragma unroll
    for (int q = 0; q < 8; ++q) dst[q] = make_float4(y[4 * q], y[4 * q + 1], y[4 * q + 2], y[4 * q + 3]);
  }
  if (tgt < 0) return;
  float mx = y[0];
#pragma unroll
  for (int j = 1; j < 32; ++j) mx = fmaxf(mx, y[j]);
  mx = fmaxf(m, mx);
  if (mx != -INFINITY) {
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      a0 += expf(y[j] - mx);
      a1 += expf(y[j + 1] - mx);
    }
    s = s * expf(m - mx) + (a0 + a1);
    m = mx;
  } else {  // nothing but -infinity adds nothing; a NaN, which fmaxf passes over, counts
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (y[j] != y[j]) s = y[j];
  }
  if (tgt >= n && tgt < n + 32) {
    float x = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) x = n + j == (int)tgt ? y[j] : x;
    p.target_logit[t] = x;
  }
}

// EPI_LAYER.  The step is chosen at run time (uniform over the launch): one kernel per tile shape serves every layered decoder.  The
// choice is made once per 32 columns, never inside a loop over them: with the branches inside, the chains of exponential and
// reciprocal ran one after the other and a tile's epilogue took longer than its MMAs (gate/up of 4096 x 28672 x 4096: 1015 us against
// 642 us for the plain store).  The Linear's sum (+ bias) is rounded to bf16 once before the step, except for fp32 results.
__device__ __forceinline__ float layer_sigmoid(float x) {
  return sigmoid_by(
      x,
      [](float v) {
        float r;
        asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
        return r;
      },
      [](float v) {
        float r;
        asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
        return r;
      });
}
__device__ __forceinline__ float layer_gelu(float z) { return 0.5f * z * (1.f + tanhf(0.7978845608028654f * fmaf(0.044715f * z * z, z, z))); }

__device__ __forceinline__ bool layer_step_is_f32(int step) { return step == LAYER_F32 || step == LAYER_RESIDUAL || step == LAYER_RESIDUAL_SCALED; }

__device__ __forceinline__ void layer_sums(const EpiParams& p, int n, const uint32_t (&v)[32], float (&x)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j) x[j] = __uint_as_float(v[j]);
  if (p.bias != nullptr) {
    const uint4* b4 = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.bias) + n);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint4 b = __ldg(b4 + q);
      const uint32_t u[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        x[8 * q + 2 * j] += bf16lo(u[j]);
        x[8 * q + 2 * j + 1] += bf16hi(u[j]);
      }
    }
  }
}

// fp32 results and the fp32 residual stream, for the 32 rows t0 .. of one warp (all lanes call; rows from `rows` on are not stored).  A
// thread owns a row of the accumulator, but 16-byte accesses of 32 different rows are half a sector each: the 32 x 32 block goes
// through 4 KB of shared memory (the warp's own; 16-byte units XORed with the row: no bank conflicts) and out as whole 128-byte lines.
__device__ __forceinline__ void epi_layer32_f32(const EpiParams& p, int t0, int rows, int n, const uint32_t (&v)[32], float4* stg) {
  const int lane = (int)(threadIdx.x & 31), step = p.layer;
  float4* const base = reinterpret_cast<float4*>(p.out_f32 + (int64_t)t0 * p.ld_out + n) + (lane & 7);
  const int64_t pitch = p.ld_out / 4;
  float4 r[8];
  if (step != LAYER_F32) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 4 * i + (lane >> 3);
      if (row < rows) r[i] = base[row * pitch];
    }
  }
  float x[32];
  layer_sums(p, n, v, x);
  if (step == LAYER_F32) {
    if (p.limit > 0.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = p.limit * tanhf(x[j] / p.limit);
    }
    const float f = p.alpha != 0.f ? p.alpha : 1.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] *= f;
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j) x[j] = round_bf16(x[j]);
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 8; ++q) stg[lane * 8 + (q ^ (lane & 7))] = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
  __syncwarp();
  const float f = step == LAYER_RESIDUAL_SCALED ? p.alpha : 1.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = 4 * i + (lane >> 3);
    float4 o = stg[row * 8 + ((lane & 7) ^ (row & 7))];
    if (row < rows) {
      if (step != LAYER_F32) o = make_float4(r[i].x + f * o.x, r[i].y + f * o.y, r[i].z + f * o.z, r[i].w + f * o.w);
      base[row * pitch] = o;
    }
  }
}

// the same for a warp whose lanes hold the columns: v[j] is row t0 + j of column n, an access is one 128-byte line.  First what is there already (_fetch, into
// r), then the step, then _store.  (Row offsets are 32-bit products of the pitch: as 64-bit ones they cost the registers that the rows need.)
__device__ __forceinline__ void epi_layer32_f32_lanes_fetch(const EpiParams& p, int t0, int rows, int n, uint32_t (&r)[32]) {
  if (p.layer == LAYER_F32) return;
  const float* base = p.out_f32 + (int64_t)t0 * p.ld_out + n;
  const int ld = (int)p.ld_out;
  if (rows >= 32) {
#pragma unroll
    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(base[j * ld]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < rows) r[j] = __float_as_uint(base[j * ld]);
  }
}
__device__ __forceinline__ void epi_layer32_f32_lanes(const EpiParams& p, int n, uint32_t (&v)[32], const uint32_t (&r)[32], bool valid) {
  if (p.bias != nullptr) {
    const float b = valid ? bf16_to_float(reinterpret_cast<const uint16_t*>(p.bias)[n]) : 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + b);
  }
  if (p.layer == LAYER_F32) {
    if (p.limit > 0.f) {
#pragma unroll 1
      for (int j = 0; j < 32; ++j) {  // (a soft cap: heads only; one copy of tanhf, the registers by a select)
        float x = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) x = i == j ? __uint_as_float(v[i]) : x;
        x = p.limit * tanhf(x / p.limit);
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = i == j ? __float_as_uint(x) : v[i];
      }
    }
    const float f = p.alpha != 0.f ? p.alpha : 1.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * f);
  } else {
    const float f = p.layer == LAYER_RESIDUAL_SCALED ? p.alpha : 1.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(r[j]) + f * round_bf16(__uint_as_float(v[j])));
  }
}
__device__ __forceinline__ void epi_layer32_f32_lanes_store(const EpiParams& p, int t0, int rows, int n, const uint32_t (&v)[32]) {
  float* const base = p.out_f32 + (int64_t)t0 * p.ld_out + n;
  const int ld = (int)p.ld_out;
  if (rows >= 32) {
#pragma unroll
    for (int j = 0; j < 32; ++j) base[j * ld] = __uint_as_float(v[j]);
  } else {
#pragma unroll
    for (int j = 0; j < 32; ++j)
      if (j < rows) base[j * ld] = __uint_as_float(v[j]);
  }
}

// the same for one row by one thread (the few rows of the stream-K kernel)
__device__ __forceinline__ void epi_layer32_f32_row(const EpiParams& p, int t, int n, const uint32_t (&v)[32]) {
  float x[32];
  layer_sums(p, n, v, x);
  float4* dst = reinterpret_cast<float4*>(p.out_f32 + (int64_t)t * p.ld_out + n);
  if (p.layer == LAYER_F32) {
    if (p.limit > 0.f) {
#pragma unroll
      for (int j = 0; j < 32; ++j) x[j] = p.limit * tanhf(x[j] / p.limit);
    }
    const float f = p.alpha != 0.f ? p.alpha : 1.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) dst[q] = make_float4(x[4 * q] * f, x[4 * q + 1] * f, x[4 * q + 2] * f, x[4 * q + 3] * f);
    return;
  }
  const float f = p.layer == LAYER_RESIDUAL_SCALED ? p.alpha : 1.f;
  float4 r[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) r[q] = dst[q];
#pragma unroll
  for (int q = 0; q < 8; ++q)
    dst[q] = make_float4(r[q].x + f * round_bf16(x[4 * q]), r[q].y + f * round_bf16(x[4 * q + 1]), r[q].z + f * round_bf16(x[4 * q + 2]), r[q].w + f * round_bf16(x[4 * q + 3]));
}

// the bf16 results: row t, columns n .. n + 31 of the accumulator
__device__ __forceinline__ void epi_layer32_bf16(const EpiParams& p, int t, int n, const uint32_t (&v)[32]) {
  const int step = p.layer;
  float x[32];
  layer_sums(p, n, v, x);
#pragma unroll
  for (int j = 0; j < 32; ++j) x[j] = round_bf16(x[j]);
  if (step == LAYER_STORE || step == LAYER_RELU2) {
    if (step == LAYER_STORE) {
      if (n + 32 <= p.n_act) {
#pragma unroll
        for (int j = 0; j < 32; ++j) x[j] *= layer_sigmoid(x[j]);
      } else if (n < p.n_act) {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (n + j < p.n_act) x[j] *= layer_sigmoid(x[j]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float y = fmaxf(x[j], 0.f);
        x[j] = y * y;
      }
      if (p.rowscale != nullptr) {
        const float* rs = p.rowscale + (int64_t)t * p.rs_pitch;
        const int g = n / p.rs_group;
        if ((n + 31) / p.rs_group == g) {
          const float f = rs[g];
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] = f == 0.f ? 0.f : x[j] * f;
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) x[j] *= rs[(n + j) / p.rs_group];
        }
      }
    }
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + n);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      dst[q] = make_uint4(pack2_rn(x[8 * q], x[8 * q + 1]), pack2_rn(x[8 * q + 2], x[8 * q + 3]), pack2_rn(x[8 * q + 4], x[8 * q + 5]),
                          pack2_rn(x[8 * q + 6], x[8 * q + 7]));
    return;
  }
  // gated units: 16 (gate, up) pairs -> 16 outputs
  const int c = n >> 1;
  uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + c);
  float s0 = 1.f;
  float s[16];
  bool one = true;  // one scale for the 16 outputs
  if (p.rowscale != nullptr) {
    const float* row = p.rowscale + (int64_t)t * p.rs_pitch;
    const int g = c / p.rs_group;
    one = (c + 15) / p.rs_group == g;
    if (one) {
      s0 = row[g];
      if (s0 == 0.f) {  // an expert that the token did not choose: nothing of it counts, not even an infinity
        dst[0] = dst[1] = make_uint4(0, 0, 0, 0);
        return;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) s[j] = row[(c + j) / p.rs_group];
    }
  }
  if (one) {
#pragma unroll
    for (int j = 0; j < 16; ++j) s[j] = s0;
  }
  if (step == LAYER_GLU) {  // the scale multiplies the expert's INPUT: gate and up, before the clamps
    const float limit = p.limit, alpha = p.alpha;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float g = fminf(x[2 * j] * s[j], limit), u = fminf(fmaxf(x[2 * j + 1] * s[j], -limit), limit);
      x[j] = g * layer_sigmoid(alpha * g) * (u + 1.f);
    }
  } else if (step == LAYER_SWIGLU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = x[2 * j] * layer_sigmoid(x[2 * j]) * x[2 * j + 1] * s[j];
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = layer_gelu(x[2 * j]) * x[2 * j + 1] * s[j];
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    dst[q] = make_uint4(pack2_rn(x[8 * q], x[8 * q + 1]), pack2_rn(x[8 * q + 2], x[8 * q + 3]), pack2_rn(x[8 * q + 4], x[8 * q + 5]),
                        pack2_rn(x[8 * q + 6], x[8 * q + 7]));
}

template <int MODE>
__device__ __forceinline__ void epi_chunk32(const EpiParams& p, int t, int n, const uint32_t (&v)[32]) {
  if constexpr (MODE == EPI_LAYER) {
    if (layer_step_is_f32(p.layer))
      epi_layer32_f32_row(p, t, n, v);  // few rows; many: epi_layer32_f32, by whole warps
    else
      epi_layer32_bf16(p, t, n, v);
  } else if constexpr (MODE == EPI_STORE || MODE == EPI_RESIDUAL) {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + n);
    uint32_t o[16];
    if constexpr (MODE == EPI_RESIDUAL) {
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.residual) + (int64_t)t * p.ld_out + n);
      uint4 r4[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) r4[q] = src[q];
      const uint32_t* r = reinterpret_cast<const uint32_t*>(r4);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        o[j] = pack2_rn(round_bf16(__uint_as_float(v[2 * j])) + bf16lo(r[j]), round_bf16(__uint_as_float(v[2 * j + 1])) + bf16hi(r[j]));
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] = pack2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
  } else if constexpr (MODE == EPI_MOE_SCALE) {
    const float w = bf16_to_float(reinterpret_cast<const uint16_t*>(p.row_w)[t]);
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) o[j] = pack2_rn(w * round_bf16(__uint_as_float(v[2 * j])), w * round_bf16(__uint_as_float(v[2 * j + 1])));
    const int64_t off = (int64_t)t * p.ld_out + n;
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + off);
#pragma unroll
    for (int q = 0; q < 4; ++q) dst[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    for (int r = 0; r < p.n_peers; ++r) {  // the same row on the other ranks (NVLink peer stores, 64 B per thread and chunk)
      uint4* pd = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.peer_out[r]) + off);
#pragma unroll
      for (int q = 0; q < 4; ++q) pd[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    }
  } else if constexpr (MODE == EPI_F32) {
    float4* dst = reinterpret_cast<float4*>(p.out_f32 + (int64_t)t * p.ld_out + n);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      dst[q] = make_float4(round_bf16(__uint_as_float(v[4 * q])), round_bf16(__uint_as_float(v[4 * q + 1])),
                           round_bf16(__uint_as_float(v[4 * q + 2])), round_bf16(__uint_as_float(v[4 * q + 3])));
  } else if constexpr (MODE == EPI_SWIGLU) {
    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t * p.ld_out + (n >> 1));
    uint32_t o[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a0 = round_bf16(__uint_as_float(v[4 * j])), b0 = round_bf16(__uint_as_float(v[4 * j + 1]));
      const float a1 = round_bf16(__uint_as_float(v[4 * j + 2])), b1 = round_bf16(__uint_as_float(v[4 * j + 3]));
      o[j] = pack2_rn(round_bf16(fast_silu(a0)) * b0, round_bf16(fast_silu(a1)) * b1);
    }
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
  } else if constexpr (MODE == EPI_QKV_ROPE) {
    uint32_t o[16];
    uint16_t* dst;
    uint16_t* ring = nullptr;
    if (n < p.q_dim + p.kv_dim) {  // q or k: rotate the 16 interleaved pairs of this chunk
      const int pos = p.positions[t];
      const float4* cs4 = reinterpret_cast<const float4*>(p.rope + ((int64_t)pos * (kHeadDim / 2) + ((n & (kHeadDim - 1)) >> 1)) * 2);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 cs = __ldg(cs4 + j);  // (cos, sin) of pairs 2j, 2j+1
        float re, im;
        ref_cmul(round_bf16(__uint_as_float(v[4 * j])), round_bf16(__uint_as_float(v[4 * j + 1])), cs.x, cs.y, re, im);
        o[2 * j] = pack2_rn(re, im);
        ref_cmul(round_bf16(__uint_as_float(v[4 * j + 2])), round_bf16(__uint_as_float(v[4 * j + 3])), cs.z, cs.w, re, im);
        o[2 * j + 1] = pack2_rn(re, im);
      }
      if (n < p.q_dim) {
        dst = reinterpret_cast<uint16_t*>(p.q_out) + (int64_t)t * p.q_dim + n;
      } else {
        dst = reinterpret_cast<uint16_t*>(p.k_out) + (int64_t)t * p.kv_dim + (n - p.q_dim);
        if (p.cache_rows != nullptr) {
          const int row = p.cache_rows[t];
          if (row >= 0) ring = reinterpret_cast<uint16_t*>(p.cache_k) + (int64_t)row * p.kv_dim + (n - p.q_dim);
        }
      }
    } else {  // v: stored as projected
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] = pack2_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
      const int c = n - p.q_dim - p.kv_dim;
      dst = reinterpret_cast<uint16_t*>(p.v_out) + (int64_t)t * p.kv_dim + c;
      if (p.cache_rows != nullptr) {
        const int row = p.cache_rows[t];
        if (row >= 0) ring = reinterpret_cast<uint16_t*>(p.cache_v) + (int64_t)row * p.kv_dim + c;
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(dst)[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    if (ring != nullptr) {
#pragma unroll
      for (int q = 0; q < 4; ++q) reinterpret_cast<uint4*>(ring)[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    }
  }
}

// ---- feature-lane epilogues (gemm_pair.cuh) ------------------------------------------------------------------------------------
// There a warp's accumulator block has the 32 features in its lanes and 32 tokens in each lane's registers.  Lanes 2i and 2i + 1 exchange halves, as bf16 pairs, and
// then hold both features of pair i for 16 tokens each: what epi_pair takes.  For a store four features of a token come together (exchange_rows8).
// y0, y1: features n, n + 1 of tokens t0 + j, as packed pairs of tokens (2q, 2q + 1); tokens from `rows` on are not stored.
__device__ __forceinline__ float bf16_of(const uint32_t (&y)[8], int j) { return j & 1 ? bf16hi(y[j >> 1]) : bf16lo(y[j >> 1]); }

// words q of own[16] hold tokens 2q, 2q + 1 of this lane's feature
__device__ __forceinline__ void exchange_pairs(const uint32_t (&own)[16], uint32_t (&y0)[8], uint32_t (&y1)[8]) {
  const bool odd = threadIdx.x & 1;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? own[q] : own[8 + q], 1);
    y0[q] = odd ? other : own[q];
    y1[q] = odd ? own[8 + q] : other;
  }
}

// What the step reads for these tokens, requested a block ahead: the residual's pairs, the positions, the rows' weights.
template <int MODE>
__device__ __forceinline__ void epi_pairs16_fetch(const EpiParams& p, int t0, int rows, int n, uint32_t (&r)[16]) {
  if constexpr (MODE == EPI_RESIDUAL) {
    const uint16_t* src = reinterpret_cast<const uint16_t*>(p.residual) + (int64_t)t0 * p.ld_out + n;
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = j < rows ? *reinterpret_cast<const uint32_t*>(src + j * (int)p.ld_out) : 0u;
  } else if constexpr (MODE == EPI_MOE_SCALE) {
    const uint16_t* src = reinterpret_cast<const uint16_t*>(p.row_w) + t0;
#pragma unroll
    for (int j = 0; j < 16; ++j) r[j] = j < rows ? (uint32_t)src[j] << 16 : 0u;
  } else if constexpr (MODE == EPI_QKV_ROPE) {
    if (n < p.q_dim + p.kv_dim) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = j < rows ? (uint32_t)p.positions[t0 + j] : 0u;
    }
  } else if constexpr (MODE == EPI_LAYER) {  // one scale per row (the mixtures)
    if (p.rowscale != nullptr && p.rs_pitch == 1) {
#pragma unroll
      for (int j = 0; j < 16; ++j) r[j] = j < rows ? __float_as_uint(p.rowscale[t0 + j]) : 0u;
    }
  }
}

// A lane has features n, n + 1 (o[j]) of 16 tokens; lanes whose numbers differ by 2 exchange halves, and v[q] are features n & ~3 .. | 3 of token rows8() + q: eight
// stores of 8 bytes where sixteen of 4 held up the MMAs, whose operands come out of L2 while a tile's results go there.  4096 x 18944 x 2048 219.6 -> 217.1 us,
// 4096 x 4096 x 2048 60.3 -> 59.2, 4096 x 9472 x 4096 205.3 -> 203.8.  (Four stores of 16 bytes, one more exchange: 216.6, 59.9, 203.8.  Gated units by 8
// bytes instead of 4: 1024 x 16384 x 2048 58 -> 61 in a loop, so they keep 4.)
__device__ __forceinline__ int rows8() { return threadIdx.x & 2 ? 8 : 0; }
__device__ __forceinline__ void exchange_rows8(const uint32_t (&o)[16], uint2 (&v)[8]) {
  const bool hi = threadIdx.x & 2;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t own = hi ? o[8 + q] : o[q], other = __shfl_xor_sync(0xffffffffu, hi ? o[q] : o[8 + q], 2);
    v[q] = hi ? make_uint2(other, own) : make_uint2(own, other);
  }
}
// base: features n & ~3 of the first of the 16 tokens, `rows` of which are there
__device__ __forceinline__ void store_rows8(uint16_t* base, int ld, int rows, const uint2 (&v)[8]) {
  const int t = rows8();
  uint16_t* dst = base + (int64_t)t * ld;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    if (t + q < rows) *reinterpret_cast<uint2*>(dst + q * ld) = v[q];
}

// Gated units: 16 tokens of unit c (in lane pair by lane pair).  Two lane pairs exchange halves, so that a store is 4 bytes, units c & ~1 and c | 1 of a token.
__device__ __forceinline__ void store_units16(void* out, int ld, int t0, int rows, int c, const float (&x)[16]) {
  const bool hi = threadIdx.x & 2;
  uint16_t* dst = reinterpret_cast<uint16_t*>(out) + (int64_t)(t0 + (hi ? 8 : 0)) * ld + (c & ~1);
  const int left = rows - (hi ? 8 : 0);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t a = pack2_rn(x[2 * q], x[2 * q + 1]), b = pack2_rn(x[8 + 2 * q], x[9 + 2 * q]);
    const uint32_t other = __shfl_xor_sync(0xffffffffu, hi ? a : b, 2);
    const uint32_t u0 = hi ? other : a, u1 = hi ? b : other;  // tokens 2q, 2q + 1 (+ 8) of the two units
    if (2 * q < left) *reinterpret_cast<uint32_t*>(dst + 2 * q * ld) = __byte_perm(u0, u1, 0x5410);
    if (2 * q + 1 < left) *reinterpret_cast<uint32_t*>(dst + (2 * q + 1) * ld) = __byte_perm(u0, u1, 0x7632);
  }
}

template <int MODE>
__device__ __forceinline__ void epi_pairs16(const EpiParams& p, int t0, int rows, int n, const uint32_t (&y0)[8], const uint32_t (&y1)[8], const uint32_t (&r)[16]) {
  if constexpr (MODE == EPI_STORE || MODE == EPI_RESIDUAL || MODE == EPI_MOE_SCALE) {
    const int64_t off = (int64_t)t0 * p.ld_out + (n & ~3);
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float a = bf16_of(y0, j), b = bf16_of(y1, j);
      if constexpr (MODE == EPI_RESIDUAL)
        o[j] = pack2_rn(a + bf16lo(r[j]), b + bf16hi(r[j]));
      else if constexpr (MODE == EPI_MOE_SCALE)
        o[j] = pack2_rn(__uint_as_float(r[j]) * a, __uint_as_float(r[j]) * b);
      else
        o[j] = __byte_perm(y0[j >> 1], y1[j >> 1], j & 1 ? 0x7632 : 0x5410);
    }
    uint2 v[8];
    exchange_rows8(o, v);
    store_rows8(reinterpret_cast<uint16_t*>(p.out) + off, (int)p.ld_out, rows, v);
    if constexpr (MODE == EPI_MOE_SCALE) {
      for (int k = 0; k < p.n_peers; ++k) store_rows8(reinterpret_cast<uint16_t*>(p.peer_out[k]) + off, (int)p.ld_out, rows, v);  // the same rows on the other ranks (NVLink peer stores)
    }
  } else if constexpr (MODE == EPI_F32) {
    float* dst = p.out_f32 + (int64_t)t0 * p.ld_out + n;
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < rows) *reinterpret_cast<float2*>(dst + j * (int)p.ld_out) = make_float2(bf16_of(y0, j), bf16_of(y1, j));
  } else if constexpr (MODE == EPI_SWIGLU) {
    float x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = round_bf16(fast_silu(bf16_of(y0, j))) * bf16_of(y1, j);
    store_units16(p.out, (int)p.ld_out, t0, rows, n >> 1, x);
  } else if constexpr (MODE == EPI_QKV_ROPE) {
    const bool rotate = n < p.q_dim + p.kv_dim, ring = n >= p.q_dim && p.cache_rows != nullptr;  // (the warp's 32 features lie in one head)
    uint32_t o[16];
    if (rotate) {
      const float* tab = p.rope + (n & (kHeadDim - 1));
      float2 cs[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) cs[j] = j < rows ? __ldg(reinterpret_cast<const float2*>(tab + (int64_t)(int)r[j] * kHeadDim)) : make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float re, im;
        ref_cmul(bf16_of(y0, j), bf16_of(y1, j), cs[j].x, cs[j].y, re, im);
        o[j] = pack2_rn(re, im);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] = __byte_perm(y0[j >> 1], y1[j >> 1], j & 1 ? 0x7632 : 0x5410);
    }
    uint2 v[8];
    exchange_rows8(o, v);
    const bool is_q = n < p.q_dim;
    const int width = is_q ? p.q_dim : p.kv_dim, c = (is_q ? n : (rotate ? n - p.q_dim : n - p.q_dim - p.kv_dim)) & ~3;
    store_rows8(reinterpret_cast<uint16_t*>(is_q ? p.q_out : (rotate ? p.k_out : p.v_out)) + (int64_t)t0 * width + c, width, rows, v);
    if (ring) {
      uint16_t* cache = reinterpret_cast<uint16_t*>(rotate ? p.cache_k : p.cache_v) + c;
      const int t = rows8();
      int row[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) row[q] = t + q < rows ? p.cache_rows[t0 + t + q] : -1;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (row[q] >= 0) *reinterpret_cast<uint2*>(cache + (int64_t)row[q] * p.kv_dim) = v[q];
    }
  }
}

// EPI_LAYER's bf16 results (bias added and sums rounded before the exchange).  SCALED: the rows have scales; r: those of rs_pitch 1 (the mixtures), fetched ahead.
template <bool SCALED>
__device__ __forceinline__ void epi_layer_pairs16(const EpiParams& p, int t0, int rows, int n, const uint32_t (&y0)[8], const uint32_t (&y1)[8], const uint32_t (&r)[16]) {
  const int step = p.layer;
  if (step == LAYER_STORE || step == LAYER_RELU2) {
    uint32_t o[16];
    if (step == LAYER_STORE) {
      const bool act0 = n < p.n_act, act1 = n + 1 < p.n_act;
      if (__any_sync(0xffffffffu, act0)) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float a = bf16_of(y0, j), b = bf16_of(y1, j);
          o[j] = pack2_rn(act0 ? a * layer_sigmoid(a) : a, act1 ? b * layer_sigmoid(b) : b);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) o[j] = __byte_perm(y0[j >> 1], y1[j >> 1], j & 1 ? 0x7632 : 0x5410);
      }
    } else {
      const float* rs0 = nullptr;
      const float* rs1 = nullptr;
      if constexpr (SCALED) {
        rs0 = p.rowscale + (int64_t)t0 * p.rs_pitch + n / p.rs_group;
        rs1 = p.rowscale + (int64_t)t0 * p.rs_pitch + (n + 1) / p.rs_group;
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const float a = fmaxf(bf16_of(y0, j), 0.f), b = fmaxf(bf16_of(y1, j), 0.f);
        float u = a * a, v = b * b;
        if constexpr (SCALED) {
          const float f0 = j < rows ? rs0[j * p.rs_pitch] : 0.f, f1 = rs1 == rs0 ? f0 : (j < rows ? rs1[j * p.rs_pitch] : 0.f);
          u = f0 == 0.f ? 0.f : u * f0;
          v = f1 == 0.f ? 0.f : v * f1;
        }
        o[j] = pack2_rn(u, v);
      }
    }
    uint2 v[8];
    exchange_rows8(o, v);
    store_rows8(reinterpret_cast<uint16_t*>(p.out) + (int64_t)t0 * p.ld_out + (n & ~3), (int)p.ld_out, rows, v);
    return;
  }
  float s[16], x[16];
  if constexpr (SCALED) {
    if (p.rs_pitch == 1) {
#pragma unroll
      for (int j = 0; j < 16; ++j) s[j] = __uint_as_float(r[j]);
    } else {
      const float* rs = p.rowscale + (int64_t)t0 * p.rs_pitch + (n >> 1) / p.rs_group;
#pragma unroll
      for (int j = 0; j < 16; ++j) s[j] = j < rows ? rs[j * p.rs_pitch] : 0.f;
    }
  }
  if (step == LAYER_GLU) {  // the scale multiplies the expert's INPUT: gate and up, before the clamps
    const float limit = p.limit, alpha = p.alpha;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float g = bf16_of(y0, j), u = bf16_of(y1, j);
      if constexpr (SCALED) g *= s[j], u *= s[j];
      g = fminf(g, limit);
      x[j] = g * layer_sigmoid(alpha * g) * (fminf(fmaxf(u, -limit), limit) + 1.f);
    }
  } else if (step == LAYER_SWIGLU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = bf16_of(y0, j) * layer_sigmoid(bf16_of(y0, j)) * bf16_of(y1, j);
  } else {
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = layer_gelu(bf16_of(y0, j)) * bf16_of(y1, j);
  }
  if constexpr (SCALED) {
    const bool glu = step == LAYER_GLU;
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = s[j] == 0.f ? 0.f : (glu ? x[j] : x[j] * s[j]);  // (an expert that the token did not choose: nothing of it counts, not even an infinity)
  }
  store_units16(p.out, (int)p.ld_out, t0, rows, n >> 1, x);
}

}  // namespace mb200
