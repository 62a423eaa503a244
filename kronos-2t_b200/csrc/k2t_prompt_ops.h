// Small operators of a prompt batch (k2t_prompt_ops.cu).
#pragma once
#include "k2t_gemm_f16.h"
#include "k2t_model_kernels.h"

namespace k2t {

// Signs of the rotation, a byte per eight values, for chunks 0 .. chunks - 1: made once, read by every launch below.
size_t sign_table_bytes(uint32_t chunks);
cudaError_t launch_sign_table(cudaStream_t s, uint8_t *table, uint32_t chunks);

struct PromptAct {
    int8_t *q;                 // [n_tok][cols], with scale and sum per chunk
    float *scales;
    int32_t *sums;
    ActHalf image{};           // img == null: none wanted
    uint32_t tok_pad = 0;      // act_half_tokens(n_tok)
};
// Results of launch_rmsnorm_quant_x, launch_swiglu_quant / launch_expert_swiglu_quant (exact_exp) and launch_qkv_post, and the image.
cudaError_t launch_norm_batch(cudaStream_t s, float *hidden, const float *delta, const float *w, uint32_t n, float eps, float *x_norm, uint32_t n_tok, const uint8_t *signs,
                              const PromptAct &a, bool pdl);
cudaError_t launch_swiglu_batch(cudaStream_t s, bool exact_exp, const float *gate_up, uint32_t inter, uint32_t n_tok, uint32_t chunk0, const uint8_t *signs, const PromptAct &a, bool pdl);
bool heads_batch_takes(const QkvPostArgs &a);
cudaError_t launch_heads_batch(cudaStream_t s, const QkvPostArgs &a, uint32_t n_tok, const uint8_t *signs, bool pdl);

}  // namespace k2t
