// Prompt GEMM over half-precision operand images (k2t_gemm_f16.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "k2t_kernels.h"

namespace k2t {

// Operand and scale image of a batch's activations: device scratch of the caller, rewritten by every launch.
struct ActHalf {
    uint8_t *img = nullptr;          // act_half_bytes, 1024-byte aligned
    uint8_t *scales = nullptr;       // act_half_scale_bytes, 16-byte aligned
    uint32_t *zero = nullptr;        // images of k2t_prompt_ops.cu: set when a chunk without a scale was written since the caller cleared it
};
inline size_t act_half_tokens(size_t n_tok) { return (n_tok + 127) & ~(size_t)127; }
bool gemm_f16_takes(size_t n_tok);          // batches whose padded tokens, 32 to a CTA of either launch, fit a grid
// Whether a batch of int8 activations is better off converted and multiplied here than by the integer GEMM, which needs no conversion
// launch.  Product of both, conversion included, cold weights, integer -> this one: as long as the integer GEMM fills less than half the SMs with
// its tiles of 16 tokens it is up to 40% faster for rows of up to 64 chunks (576 columns x 960 rows, 100 tokens 5.7 -> 7.9 us; 2048 x 2048, 128 tokens 16.6 ->
// 17.6; 3584 x 4608, 32 tokens 29.0 -> 29.9), beyond that slower (2048 x 6144, 33 tokens 20.4 -> 17.9; 18944 x 3584, 65 tokens 265 -> 135; 2048 x 49152,
// 512 tokens 605 -> 253) - but for few chunks, whose launches weigh more (576 x 960, 512 tokens 9.2 -> 9.4 in tiles of 32; 576 x 1536 9.7 -> 8.4
// in tiles of 64).  The line is older than k2t_gemm_prompt.cu: on the integer side of it rows of 96 chunks and more would gain 2 to 15% by that kernel (8192 x 2048 b4,
// 64 tokens 56.9 -> 56.0; 18944 x 3584 151 -> 135; b6 x 8192 65 -> 56), and 2048 x 49152, 16 tokens 51 -> 40; nf5 (65 -> 73) and rows below a tile would lose.
bool gemm_f16_pays(uint32_t rows, uint32_t nc, size_t n_tok, int sm_count);
size_t act_half_bytes(size_t n_tok, uint32_t cols);
size_t act_half_scale_bytes(size_t n_tok, uint32_t cols);

// y[t] = W x[t] for activations in the form the library's own quantizers leave them (the sums of a chunk are those of its values):
// two launches, the image and the product; image_ready: the kernel that quantized them has left the image (k2t_prompt_ops.cu).
cudaError_t launch_gemm_f16(cudaStream_t stream, const DeviceMatrix &m, const int8_t *xq, const float *xs, uint32_t n_tok, const ActHalf &h,
                            float *out, size_t out_stride, int sm_count, uint32_t *err_flag, uint32_t *launches, bool pdl, bool image_ready = false);

// The (token, route) pairs of a batch in tiles of 32 of one expert: device scratch of the caller.
struct ExpertTiles {
    uint32_t *n_tiles = nullptr;     // one word
    uint32_t *expert = nullptr;      // [expert_tiles_max]
    uint32_t *pairs = nullptr;       // [expert_tiles_max][32]: pair = token * k + route, 0xffffffff behind the expert's last one
};
constexpr uint32_t EXPERT_TILES_MAX_EXPERTS = 256;
uint32_t expert_tiles_max(size_t n_pair, uint32_t n_experts);
cudaError_t launch_expert_tiles(cudaStream_t stream, const uint32_t *route_ids, uint32_t n_tok, uint32_t k, uint32_t route_stride, uint32_t n_experts,
                                const uint8_t *const *bases, const ExpertTiles &t, uint32_t *err_flag, bool pdl);

// Whether the expert projections of a batch run in tiles (below) or as a GEMV per pair.  Tiles are a tensor-core form: only for batches that
// gemm_tc_min_tokens() hands over.  Their time goes with the weights of the experts that the pairs meet, a GEMV's per pair, with the weights
// of one expert and the cost of its decode.  Measured with 2048 columns, prompts of 2 layers: tokens at which tiles (first) and GEMVs take the same, by
// experts / routes / width / bits: 128 / 8 / 768 / 3 38 (32: 619 and 565 us, 48: 654 and 720), 4 24; 64 / 6 / 768 / 3 29, 4 20; 64 / 6 / 1408 / 3 36 (32: 610
// and 560, 40: 624 and 667); fewer than 16: 5 and 2 bits of both, 16 / 4 / 2816 / 3 (16: 440 and 446) and 4, 8 / 2 / 4096 / 4, 4 / 2 / 2048 / 3.
bool experts_grouped(uint32_t n_tok, uint32_t n_pair, uint32_t n_experts, uint32_t hidden, uint32_t d_ff, uint32_t bits);

// (k2t_gemm_prompt.cu) The expert projections of all pairs of `t`, an expert's weights expanded once per 32 pairs; out = [n_pair][rows].  Same bits as
// launch_gemv_experts, for activations in the form the library's own quantizers leave them.
cudaError_t launch_gemm_experts(cudaStream_t stream, const DeviceMatrix &m0, int fmt, const ExpertCodebook *books, const uint8_t *const *bases, uint32_t n_experts,
                                const ExpertTiles &t, uint32_t n_pair, uint32_t act_group, const int8_t *xq, const float *xs, float *out, int sm_count, uint32_t *err_flag, bool pdl);

}  // namespace k2t
