// The small operators between the projections of a prompt batch: residual + norm, SwiGLU and the head preparation, each ending in the
// signed FWHT-64 and int8 quantization, bit for bit what the one-token kernels of k2t_model_kernels.cu compute.
//
// Those give a warp one 64-value block (two values per lane: five exchange steps for the rotation, five each for maximum and sum), which
// is the shortest way for one token; a batch is bound by the instructions (issue slots 73-79% busy, 260 to 420 per block).  Here eight
// lanes share a block, eight consecutive values per lane: three of the six rotation stages stay in the lane, the other three and both
// reductions serve four blocks per warp with three exchanges, and the signs (a SplitMix64 round per value) come from a table.
// The kernels also leave the operand image of the projection that follows, which saves its conversion launch.
// 512 tokens of the 1.7B shape, before -> now: norm 11.3 -> 10.0 us (2048 columns), SwiGLU 24.0 -> 15.7 us
// (8192 columns), head preparation 30.1 -> 12.9 us (96 heads), and the conversion launches 3.9 to 6.1 us each -> none.  Batches below
// sixteen tokens, which the weight passes of four take, keep the one-token kernels: nothing reads an image there.
#include <algorithm>

#include "k2t_act_image.cuh"
#include "k2t_model_device.cuh"
#include "k2t_prompt_ops.h"

namespace k2t {
namespace {

constexpr uint32_t PO_THREADS = 256, PO_BLOCKS = PO_THREADS / 8;          // 64-value blocks a CTA has in hand at a time

__global__ void __launch_bounds__(256) sign_table_kernel(uint8_t *table, uint32_t n) {          // byte i: the signs of values 8 i .. 8 i + 7
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    uint32_t b = 0;
    for (uint32_t k = 0; k < 8; ++k) b |= (rademacher_sign(i / 8, (i % 8) * 8 + k) >> 31) << k;
    table[i] = (uint8_t)b;
}

// Eight lanes = one block, lane o = values 8 o .. 8 o + 7.  The butterflies of warp_fwht64, in its order.
__device__ __forceinline__ void oct_fwht64(float (&v)[8], uint32_t signs, uint32_t lane) {
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) v[k] = __fmul_rn(__uint_as_float(__float_as_uint(v[k]) ^ ((signs << (31 - k)) & 0x80000000u)), 0.125f);
#pragma unroll
    for (uint32_t s = 1; s < 8; s <<= 1)
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k)
            if ((k & s) == 0) {
                const float a = __fadd_rn(v[k], v[k + s]), b = __fsub_rn(v[k], v[k + s]);
                v[k] = a; v[k + s] = b;
            }
#pragma unroll
    for (uint32_t m = 1; m < 8; m <<= 1) {
        const bool hi = (lane & m) != 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            const float o = __shfl_xor_sync(0xffffffffu, v[k], m);
            v[k] = hi ? __fsub_rn(o, v[k]) : __fadd_rn(v[k], o);
        }
    }
}
// largest magnitude over the LANES lanes that share it
template <uint32_t LANES> __device__ __forceinline__ float oct_max(const float (&v)[8]) {
    float mx = fabsf(v[0]);
#pragma unroll
    for (int k = 1; k < 8; ++k) mx = fmaxf(mx, fabsf(v[k]));
#pragma unroll
    for (uint32_t m = 1; m < LANES; m <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
    return mx;
}
__device__ __forceinline__ uint2 oct_int8(const float (&v)[8], float mx) {          // warp_quant64's rounding; zeros below its limit
    if (mx <= 1.1920929e-07f) return make_uint2(0, 0);
    const float inv = __fdiv_rn(127.0f, mx);
    uint32_t q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = (uint32_t)__float2int_rn(__fmul_rn(v[k], inv));
    return make_uint2(prmt(prmt(q[0], q[1], 0x0040u), prmt(q[2], q[3], 0x0040u), 0x5410u), prmt(prmt(q[4], q[5], 0x0040u), prmt(q[6], q[7], 0x0040u), 0x5410u));
}
__device__ __forceinline__ float int8_scale(float mx) { return mx <= 1.1920929e-07f ? 0.0f : __fdiv_rn(mx, 127.0f); }

// a rotated block of token t -> int8 activation, scale, sum, and the image
__device__ __forceinline__ void oct_store(const float (&v)[8], const PromptAct &a, uint32_t nc, uint32_t c, uint32_t t, uint32_t lane, bool on) {
    const uint32_t o = lane & 7u;
    const float mx = oct_max<8>(v);
    const uint2 b = oct_int8(v, mx);
    int sum = __dp4a((int)b.x, 0x01010101, __dp4a((int)b.y, 0x01010101, 0));
#pragma unroll
    for (uint32_t m = 1; m < 8; m <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, m);
    if (!on) return;
    const size_t at = (size_t)t * nc + c;
    reinterpret_cast<uint2 *>(a.q + at * 64)[o] = b;
    if (a.image.img != nullptr) image_piece(a.image.img, a.tok_pad, c, t, o, b);
    if (o == 0) {
        const float s = int8_scale(mx);
        a.scales[at] = s;
        a.sums[at] = sum;
        if (a.image.img != nullptr) {
            image_scale(a.image.scales, a.tok_pad, c, t, s);
            if (s == 0.0f) *a.image.zero = 1u;
        }
    }
}
__device__ __forceinline__ void load8(const float *p, float (&v)[8]) {
    const float4 a = __ldcg(reinterpret_cast<const float4 *>(p)), b = __ldcg(reinterpret_cast<const float4 *>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

// One or two tokens per CTA, eight lanes per block up to 1024 threads: the sums of squares of two tokens are two half-warps' sixteen
// chains each (the order of rmsnorm_quant_kernel).
template <uint32_t NORM_TOKENS>
__global__ void __launch_bounds__(1024) norm_batch_kernel(float *__restrict__ hidden, const float *__restrict__ delta, const float *__restrict__ w, uint32_t n, float eps,
                                                                float *__restrict__ x_norm, uint32_t n_tok, const uint8_t *__restrict__ signs, const PromptAct a) {
    extern __shared__ __align__(16) float s_x[];
    __shared__ float s_inv[NORM_TOKENS];
    const uint32_t tid = threadIdx.x, lane = tid & 31, tok0 = blockIdx.x * NORM_TOKENS, nc = n / 64, pitch = n + 16, nthr = blockDim.x;          // the half-warps' rows in different banks
    const uint32_t toks = min(NORM_TOKENS, n_tok - tok0);
    float *s_w = s_x + NORM_TOKENS * pitch;          // the layer's norm weights, from HBM: requested before the wait
    for (uint32_t i = tid; i < n / 4; i += nthr) reinterpret_cast<float4 *>(s_w)[i] = __ldg(reinterpret_cast<const float4 *>(w) + i);
    pdl_wait();
    pdl_trigger();
    for (uint32_t t = 0; t < toks; ++t) {
        float4 *hp = reinterpret_cast<float4 *>(hidden + (size_t)(tok0 + t) * n);
        const float4 *dp = reinterpret_cast<const float4 *>(delta + (size_t)(tok0 + t) * n);
#pragma unroll 4
        for (uint32_t i = tid; i < n / 4; i += nthr) {
            float4 v = __ldcg(hp + i);
            if (delta != nullptr) {
                const float4 d = __ldcg(dp + i);
                v.x = __fadd_rn(v.x, d.x); v.y = __fadd_rn(v.y, d.y); v.z = __fadd_rn(v.z, d.z); v.w = __fadd_rn(v.w, d.w);
                hp[i] = v;
            }
            reinterpret_cast<float4 *>(s_x + t * pitch)[i] = v;
        }
    }
    __syncthreads();
    if (tid < 32) {
        const uint32_t t = min(lane >> 4, NORM_TOKENS - 1), i0 = lane & 15u;
        const float *x = s_x + min(t, toks - 1) * pitch;
        float acc = 0.0f;
#pragma unroll 16
        for (uint32_t i = i0; i < n; i += 16) { const float v = x[i]; acc = __fmaf_rn(v, v, acc); }
        float r = __fadd_rn(acc, __shfl_down_sync(0xffffffffu, acc, 4, 16));      // lanes 0..3: a0+a1, lanes 8..11: a2+a3
        r = __fadd_rn(r, __shfl_down_sync(0xffffffffu, r, 8, 16));
        r = __fadd_rn(r, __shfl_down_sync(0xffffffffu, r, 1, 16));
        r = __fadd_rn(r, __shfl_down_sync(0xffffffffu, r, 2, 16));
        if (i0 == 0) s_inv[t] = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(r, (float)n), eps)));
    }
    __syncthreads();
    const uint32_t items = toks * nc, o = lane & 7u;
    for (uint32_t i0 = 0; i0 < items; i0 += nthr / 8) {
        const uint32_t i = i0 + (tid >> 3);
        const bool on = i < items;
        const uint32_t t = on ? i / nc : 0, c = on ? i % nc : 0;
        float v[8], ww[8];
        const float4 *xp = reinterpret_cast<const float4 *>(s_x + t * pitch + c * 64 + o * 8), *wp = reinterpret_cast<const float4 *>(s_w + c * 64 + o * 8);
        const float4 x0 = xp[0], x1 = xp[1], w0 = wp[0], w1 = wp[1];
        v[0] = x0.x; v[1] = x0.y; v[2] = x0.z; v[3] = x0.w; v[4] = x1.x; v[5] = x1.y; v[6] = x1.z; v[7] = x1.w;
        ww[0] = w0.x; ww[1] = w0.y; ww[2] = w0.z; ww[3] = w0.w; ww[4] = w1.x; ww[5] = w1.y; ww[6] = w1.z; ww[7] = w1.w;
        const float inv = s_inv[t];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(__fmul_rn(v[k], inv), ww[k]);
        if (x_norm != nullptr && on) {
            float4 *p = reinterpret_cast<float4 *>(x_norm + (size_t)(tok0 + t) * n + c * 64 + o * 8);
            p[0] = make_float4(v[0], v[1], v[2], v[3]);
            p[1] = make_float4(v[4], v[5], v[6], v[7]);
        }
        oct_fwht64(v, __ldg(signs + c * 8 + o), lane);
        oct_store(v, a, nc, c, tok0 + t, lane, on);
    }
}

// gate = values [0, inter) of a token's row, up = the rest; EXACT_EXP: the scalar-path exp of the experts (chunk0 = 0 there)
template <bool EXACT_EXP>
__global__ void __launch_bounds__(PO_THREADS) swiglu_batch_kernel(const float *__restrict__ gate_up, uint32_t inter, uint32_t n_tok, uint32_t chunk0,
                                                                  const uint8_t *__restrict__ signs, const PromptAct a) {
    const uint32_t lane = threadIdx.x & 31, o = lane & 7u, nc = inter / 64, i = blockIdx.x * PO_BLOCKS + (threadIdx.x >> 3);
    const bool on = i < n_tok * nc;
    const uint32_t t = on ? i / nc : 0, c = on ? i % nc : 0, sg = __ldg(signs + (chunk0 + c) * 8 + o);
    pdl_wait();
    if (!EXACT_EXP) pdl_trigger();          // an expert projection cannot start before it has read its activations: it would only sit on the SMs
    float g[8], u[8];
    const float *p = gate_up + (size_t)t * 2 * inter + c * 64 + o * 8;
    load8(p, g);
    load8(p + inter, u);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const float e = EXACT_EXP ? (float)exp((double)-g[k]) : exp_poly(-g[k]);
        g[k] = __fmul_rn(__fdiv_rn(g[k], __fadd_rn(1.0f, e)), u[k]);
    }
    oct_fwht64(g, sg, lane);
    oct_store(g, a, nc, c, t, lane, on);
}

// qkv_post_kernel for the int8 cache: HD / 8 lanes per head.  The first `turned_ctas` CTAs take queries and keys, the others the values of
// one block of sixteen positions: their second copy (ExactAttnArgs.v_t, [position / 16][dimension][16], sign flipped) leaves through
// shared memory in 8-byte words (byte by byte, a store per value, it was 24 us of stores).
template <uint32_t HD>
__global__ void __launch_bounds__(PO_THREADS) heads_batch_kernel(const QkvPostArgs a, uint32_t n_tok, uint32_t turned_ctas, const uint8_t *__restrict__ signs) {
    constexpr uint32_t LPH = HD / 8, HALF = HD / 2;
    constexpr uint32_t PER = PO_THREADS / LPH, VH = PER / 16;          // heads in hand; value heads of a CTA
    __shared__ __align__(8) uint8_t s_t[VH * HD * 16];
    const uint32_t lane = threadIdx.x & 31, o = lane % LPH, heads = a.n_q + 2 * a.n_kv, sg = __ldg(signs + o);          // block within the head
    const bool values = blockIdx.x >= turned_ctas;
    pdl_wait();
    pdl_trigger();
    const uint32_t p0 = __ldcg(a.pos) + a.pos_offset;
    uint32_t tok, head;
    bool on;
    if (!values) {
        const uint32_t n = a.n_q + a.n_kv, i = blockIdx.x * PER + threadIdx.x / LPH;
        on = i < n_tok * n;
        tok = on ? i / n : 0; head = on ? i % n : 0;
    } else {
        const uint32_t groups = (a.n_kv + VH - 1) / VH, b = blockIdx.x - turned_ctas, at = (p0 / 16 + b / groups) * 16 + (threadIdx.x / LPH) % 16;
        const uint32_t kvh = (b % groups) * VH + threadIdx.x / LPH / 16;
        on = at >= p0 && at - p0 < n_tok && kvh < a.n_kv;
        tok = on ? at - p0 : 0; head = a.n_q + a.n_kv + (on ? kvh : 0);
    }
    const bool is_q = head < a.n_q, is_k = !is_q && head < a.n_q + a.n_kv, turned = is_q || is_k;
    const uint32_t pos = p0 + tok;
    float v[8], c[8], s[8];
    load8(a.qkv + ((size_t)tok * heads + head) * HD + o * 8, v);
    {
        const float *r = a.rope + (size_t)pos * HD + (o % (LPH / 2)) * 8;
        load8(r, c);
        load8(r + HALF, s);
    }
    if (a.bias != nullptr) {
        float b[8];
        load8(a.bias + (size_t)head * HD + o * 8, b);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __fadd_rn(v[k], b[k]);
    }
    auto do_rope = [&]() {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float other = __shfl_xor_sync(0xffffffffu, v[k], LPH / 2);
            const float x = o < LPH / 2 ? __fsub_rn(__fmul_rn(v[k], c[k]), __fmul_rn(other, s[k])) : __fadd_rn(__fmul_rn(v[k], c[k]), __fmul_rn(other, s[k]));
            v[k] = turned ? x : v[k];
        }
    };
    auto do_norm = [&]() {
        // sixteen fma accumulators over strides of 16 values: the lanes of either parity walk through eight of them together
        float acc[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < HD / 16; ++j)
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const float x = __shfl_sync(0xffffffffu, v[k], (lane & ~(LPH - 1)) + 2 * j + (lane & 1u));
                acc[k] = __fmaf_rn(x, x, acc[k]);
            }
        float u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            u[k] = __fadd_rn(acc[k], acc[k + 4]);
            u[k] = __fadd_rn(u[k], __shfl_xor_sync(0xffffffffu, u[k], 1));
        }
        const float ss = __fadd_rn(__fadd_rn(u[0], u[1]), __fadd_rn(u[2], u[3]));
        const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fmul_rn(ss, __fdiv_rn(1.0f, (float)HD)), a.eps)));
        const float *norm_w = is_q ? a.q_norm : is_k ? a.k_norm : nullptr;
        if (norm_w != nullptr) {
            float w[8];
            load8(norm_w + o * 8, w);
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(__fmul_rn(v[k], inv), w[k]);
        }
    };
    const bool norm = a.q_norm != nullptr || a.k_norm != nullptr;
    if (a.qk_norm_after_rope) do_rope();
    if (norm) do_norm();
    if (!a.qk_norm_after_rope) do_rope();
    oct_fwht64(v, sg, lane);
    const float mx = oct_max<LPH>(v);          // one scale for the whole head
    const uint2 b = oct_int8(v, mx);
    if (values && a.v_t != nullptr) {          // no window then: row = position
        const uint32_t vh = threadIdx.x / LPH / 16, j = (threadIdx.x / LPH) % 16;
        uint8_t *p = s_t + vh * (HD * 16) + o * 128 + j;
#pragma unroll
        for (int k = 0; k < 8; ++k) p[k * 16] = (uint8_t)(((k < 4 ? b.x >> (8 * k) : b.y >> (8 * (k - 4))) & 255u) ^ 0x80u);
        __syncthreads();
        const uint32_t groups = (a.n_kv + VH - 1) / VH, blk = blockIdx.x - turned_ctas, base = (p0 / 16 + blk / groups) * 16;
        const uint32_t at = threadIdx.x * 8, kvh = (blk % groups) * VH + at / (HD * 16), first = base + at % 16;          // eight positions of one dimension
        if (kvh < a.n_kv) {
            int8_t *dst = a.v_t + (((size_t)a.layer * a.n_kv + kvh) * a.max_seq + base) * HD + at % (HD * 16);
            if (first >= p0 && first + 8 <= p0 + n_tok) {
                *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(s_t + at);
            } else {
                for (uint32_t k = 0; k < 8; ++k)
                    if (first + k >= p0 && first + k < p0 + n_tok) dst[k] = (int8_t)s_t[at + k];
            }
        }
    }
    if (!on) return;
    int8_t *dst;
    float *dst_s;
    if (is_q) {
        dst = a.q_i8 + ((size_t)tok * a.n_q + head) * HD;
        dst_s = a.q_scale + (size_t)tok * a.n_q + head;
    } else {
        const size_t kvh = is_k ? head - a.n_q : head - a.n_q - a.n_kv, row = a.ring.slot_of_pos(pos), base = ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
        dst = (is_k ? a.k_q8 : a.v_q8) + (base + row) * HD;
        dst_s = (is_k ? a.k_scale : a.v_scale) + base + row;
    }
    reinterpret_cast<uint2 *>(dst)[o] = b;
    if (o == 0) *dst_s = int8_scale(mx);
}

}  // namespace

size_t sign_table_bytes(uint32_t chunks) { return (size_t)chunks * 8; }
cudaError_t launch_sign_table(cudaStream_t s, uint8_t *table, uint32_t chunks) {
    return launch_kernel(sign_table_kernel, dim3((chunks * 8 + 255) / 256), dim3(256), 0, s, false, table, chunks * 8);
}

cudaError_t launch_norm_batch(cudaStream_t s, float *hidden, const float *delta, const float *w, uint32_t n, float eps, float *x_norm, uint32_t n_tok, const uint8_t *signs,
                              const PromptAct &a, bool pdl) {
    // two tokens per CTA once that still leaves a CTA per SM
    const bool two = n_tok >= 2u * 148u && (3 * n + 32) * 4 <= 96 * 1024;
    const size_t smem = (size_t)(two ? 3 * n + 32 : 2 * n + 16) * 4;
    if (smem > 220 * 1024) return cudaErrorInvalidValue;
    const void *k = two ? reinterpret_cast<const void *>(norm_batch_kernel<2>) : reinterpret_cast<const void *>(norm_batch_kernel<1>);
    cudaError_t e = allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    const dim3 block(std::min(1024u, std::max(256u, (n / 4 + 31) & ~31u)));
    return two ? launch_kernel(norm_batch_kernel<2>, dim3((n_tok + 1) / 2), block, smem, s, pdl, hidden, delta, w, n, eps, x_norm, n_tok, signs, a)
               : launch_kernel(norm_batch_kernel<1>, dim3(n_tok), block, smem, s, pdl, hidden, delta, w, n, eps, x_norm, n_tok, signs, a);
}
cudaError_t launch_swiglu_batch(cudaStream_t s, bool exact_exp, const float *gate_up, uint32_t inter, uint32_t n_tok, uint32_t chunk0, const uint8_t *signs, const PromptAct &a, bool pdl) {
    const dim3 grid((uint32_t)(((size_t)n_tok * (inter / 64) + PO_BLOCKS - 1) / PO_BLOCKS));
    return exact_exp ? launch_kernel(swiglu_batch_kernel<true>, grid, dim3(PO_THREADS), 0, s, pdl, gate_up, inter, n_tok, chunk0, signs, a)
                     : launch_kernel(swiglu_batch_kernel<false>, grid, dim3(PO_THREADS), 0, s, pdl, gate_up, inter, n_tok, chunk0, signs, a);
}
bool heads_batch_takes(const QkvPostArgs &a) { return a.kv_bits == 8 && (a.head_dim == 64 || a.head_dim == 128); }
cudaError_t launch_heads_batch(cudaStream_t s, const QkvPostArgs &a, uint32_t n_tok, const uint8_t *signs, bool pdl) {
    if (!heads_batch_takes(a)) return cudaErrorInvalidValue;
    const uint32_t per = PO_THREADS / (a.head_dim / 8), vh = per / 16, turned = (n_tok * (a.n_q + a.n_kv) + per - 1) / per;
    const dim3 grid(turned + ((n_tok + 15) / 16 + 1) * ((a.n_kv + vh - 1) / vh));          // the batch may start inside a block of sixteen positions
    return a.head_dim == 64 ? launch_kernel(heads_batch_kernel<64>, grid, dim3(PO_THREADS), 0, s, pdl, a, n_tok, turned, signs)
                            : launch_kernel(heads_batch_kernel<128>, grid, dim3(PO_THREADS), 0, s, pdl, a, n_tok, turned, signs);
}

}  // namespace k2t
