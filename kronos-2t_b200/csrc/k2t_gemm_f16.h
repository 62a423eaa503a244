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
};
size_t act_half_bytes(size_t n_tok, uint32_t cols);
size_t act_half_scale_bytes(size_t n_tok, uint32_t cols);

// y[t] = W x[t] for activations in the form the library's own quantizers leave them (the sums of a chunk are those of its values):
// two launches, the image and the product.
cudaError_t launch_gemm_f16(cudaStream_t stream, const DeviceMatrix &m, const int8_t *xq, const float *xs, uint32_t n_tok, const ActHalf &h,
                            float *out, size_t out_stride, int sm_count, uint32_t *err_flag, uint32_t *launches, bool pdl);

}  // namespace k2t
