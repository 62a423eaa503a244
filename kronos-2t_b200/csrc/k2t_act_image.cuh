// The operand image of a batch's activations (k2t_gemm_f16.cu): per chunk 128 bytes per token - 64 halves in the 128-byte-swizzled K-major
// layout, tokens padded to 128 - and per (chunk, 32 tokens) a record of their scales.
#pragma once
#include <cuda_fp16.h>

#include "k2t_device.cuh"
#include "k2t_gemm_f16.h"

namespace k2t {

constexpr uint32_t HF_REC = 144;             // bytes per (chunk, 32 tokens) of the scale image: 32 scales, a flag (all of them set; not where the image was left by the quantizing kernel), padding

// four bytes (each 0..255, standing for byte - 1024 - add) -> four halves: 0x6400 | b is the half 1024 + b
__device__ __forceinline__ void hf_widen(uint32_t bytes, __half2 add, uint32_t &h0, uint32_t &h1) {
    const uint32_t a = prmt(bytes, 0x64646464u, 0x4140u), b = prmt(bytes, 0x64646464u, 0x4342u);
    const __half2 x = __hadd2(*reinterpret_cast<const __half2 *>(&a), add), y = __hadd2(*reinterpret_cast<const __half2 *>(&b), add);
    h0 = *reinterpret_cast<const uint32_t *>(&x);
    h1 = *reinterpret_cast<const uint32_t *>(&y);
}
// piece `piece` (columns 8 piece .. 8 piece + 7, as int8 in b) of token t in chunk c
__device__ __forceinline__ void image_piece(uint8_t *img, uint32_t tok_pad, uint32_t c, uint32_t t, uint32_t piece, uint2 b) {
    const __half2 add = __half2half2(__int2half_rn(-1152));
    uint4 h;
    hf_widen(b.x ^ 0x80808080u, add, h.x, h.y);
    hf_widen(b.y ^ 0x80808080u, add, h.z, h.w);
    *reinterpret_cast<uint4 *>(img + ((size_t)c * tok_pad + t) * 128 + ((piece ^ (t & 7u)) << 4)) = h;
}
__device__ __forceinline__ void image_scale(uint8_t *scales, uint32_t tok_pad, uint32_t c, uint32_t t, float s) {
    reinterpret_cast<float *>(scales + ((size_t)c * (tok_pad / 32) + t / 32) * HF_REC)[t % 32] = s;
}

}  // namespace k2t
