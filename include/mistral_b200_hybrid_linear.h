/* libmb200_hybrid.so: the Linears of mistral_b200_hybrid.h with memory that the caller keeps for them.
 *
 * fp32 prompts (M > 8, K >= 16) run on tensor cores as products of bf16 parts.  mbh_linear and its kin form the parts where they are used, over and over for matrices of many
 * features; with room for the parts of x, which a caller with an allocator passes here, they are formed once. */
#ifndef MISTRAL_B200_HYBRID_LINEAR_H
#define MISTRAL_B200_HYBRID_LINEAR_H
#include <stdint.h>
#ifdef __cplusplus
extern "C" {
#endif

/* Bytes of device memory that mbh_linear_any uses for these sizes and this step (0: none); mbh_linear_scratch: enough for every step. */
int64_t mbh_linear_any_scratch(int64_t M, int64_t N, int64_t K, int epi, int64_t n_act, float limit, float alpha, int dt);
int64_t mbh_linear_scratch(int64_t M, int64_t N, int64_t K, int dt);

/* mbh_linear with every epilogue: 0 to 3 and 5 as there; 4 and 7 mbh_linear_swiglu (SiLU, gelu), 6 mbh_linear_relu2, 8 mbh_linear_decay (a_log, groups in rs_group); with
 * rowscale epilogue 2 is mbh_linear_glu.  scratch: mbh_linear_any_scratch bytes, 16-byte aligned, of any content and this call's alone until it has run; null
 * or smaller: as mbh_linear. */
int mbh_linear_any(const void* x, int64_t ldx, const void* w, const void* bias, void* out, void* out32, int64_t M, int64_t N, int64_t K, int epi, int64_t n_act, float limit,
                   float alpha, const void* rowscale, int64_t rs_pitch, int64_t rs_group, const void* a_log, void* scratch, int64_t scratch_bytes, int dt, void* stream);

#ifdef __cplusplus
}
#endif
#endif
