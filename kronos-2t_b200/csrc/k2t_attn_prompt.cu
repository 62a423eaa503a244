// Attention of a prompt batch over the int8 Hadamard cache (full causal context) in the reference's summation order
// (causal_gqa_group_q8, src/model/real_llm.rs:8471-8594), bit for bit what attn_scores_kernel / attn_values_kernel compute for one
// token at a time.
//
// The order that has to be kept is per (token, query head): four interleaved denominators over the positions and one
// position-ascending fma chain per dimension.  Different rows (token, head) are independent, and the rows of a kv head read the same
// keys and values.  So a CTA takes R = 16 (8 for long contexts) consecutive rows of a kv head and keeps their scores in shared memory,
// position-major, through all phases - nothing goes through global scratch:
//   scores      thread = position: its key row in registers against the rows' int8 queries (dp4a), row maxima
//   exp         thread = position: polynomial exp (correctly rounded exp for the last ctx % 4 positions of a row)
//   denominator lane = (row, accumulator): 64 serial sums side by side
//   weights     thread = position: (p * inv) * v_scale; zero beyond a row's own context
//   chains      thread = (dimension, R / 2 rows): a value byte is converted once for all of its rows, the rows' weights come as
//               128-bit broadcasts, two chain steps per packed fma
// One token per CTA, as in decoding, converts every value byte for a single chain step and has four lanes busy with the
// denominator while the others wait.
// Sixteen rows: enough to share a value byte and to fill two warps with denominators, few enough that three CTAs fit an SM at a
// thousand positions (64 bytes of scores per position).
// Measured (B200): 256 tokens of 32 heads of 64 at 0 .. 1000 positions 58 us on average against 193 us (scores + values, a token and head
// per CTA); a 1000-token prompt through 12 layers of the 1.7B shape 18.4 -> 11.9 ms.  Bound by shared memory (0.25 broadcast
// wavefronts per chain step) and fp32 issue together.
#include <algorithm>

#include "k2t_model_device.cuh"

namespace k2t {
namespace {

template <int HD, int R> struct PromptAttn {
    static constexpr uint32_t NT = 2 * HD;                 // two row groups x one thread per dimension
    static constexpr uint32_t NR = R / 2;                  // chains per thread
    static constexpr uint32_t HEAD = R * HD + R * 16 + 2 * R * 4 + (NT / 32) * R * 4 + R * HD * 4;      // queries, row constants, maxima and inverses, reduction, outputs
    static __host__ __device__ size_t bytes(uint32_t ctx) { return ((HEAD + 127u) & ~127u) + (size_t)((ctx + 15u) & ~15u) * R * 4; }
};

// float4 q of position t lies at index q ^ swz(t): eight consecutive positions then write eight different bank groups
template <int R> __device__ __forceinline__ constexpr uint32_t pos_swz(uint32_t t) { return R == 16 ? (t >> 1) & 3u : (t >> 2) & 1u; }

__device__ __forceinline__ unsigned long long dup_f32(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1,%1};" : "=l"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

template <int HD, int R>
__global__ void __launch_bounds__(2 * HD) attn_prompt_kernel(const ExactAttnArgs a) {
    using P = PromptAttn<HD, R>;
    constexpr uint32_t NT = P::NT, NR = P::NR, NW = NT / 32, NB = HD / 64, KW = HD / 16, RQ = R / 4;
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t *s_q = smem;                                                       // [R][HD] int8 queries
    float4 *s_row = reinterpret_cast<float4 *>(smem + R * HD);                 // {scale, context, positions in whole groups of eight, -} per row
    float *s_max = reinterpret_cast<float *>(smem + R * HD + R * 16);          // [R] maxima, then [R] 1 / denominator
    float *s_inv = s_max + R;
    float *s_red = s_inv + R;                                                  // [NW][R]
    float *s_o = s_red + NW * R;                                               // [R][HD]
    float *s_p = reinterpret_cast<float *>(smem + ((P::HEAD + 127u) & ~127u));  // [ctx][R]
    const uint32_t p_sa = (uint32_t)__cvta_generic_to_shared(s_p);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t G = a.group, n_q = a.n_kv * G, kvh = blockIdx.x;
    const uint32_t n_rows = a.n_tok * G, r0 = (gridDim.y - 1 - blockIdx.y) * R;          // the longest contexts first
    pdl_wait();
    const uint32_t pos0 = __ldcg(a.pos) + a.pos_offset;
    const uint32_t tok_lo = r0 / G, tok_hi = min(r0 + R - 1, n_rows - 1) / G;
    const uint32_t ctx_lo = pos0 + tok_lo + 1, ctx = pos0 + tok_hi + 1, ctx16 = (ctx + 15u) & ~15u;          // of the first / last row
    if (ctx > a.ctx_cap) {                 // the launcher sizes shared memory by the batch's last position: cannot happen
        if (tid == 0 && a.err_flag != nullptr) atomicExch(a.err_flag, 5u);
        return;
    }
    const size_t slot0 = ((size_t)a.layer * a.n_kv + kvh) * a.max_seq;
    for (uint32_t i = tid; i < R * HD / 4; i += NT) {
        const uint32_t r = r0 + i / (HD / 4);
        int v = 0;
        if (r < n_rows) v = __ldcg(reinterpret_cast<const int *>(a.q_i8 + ((size_t)(r / G) * n_q + kvh * G + r % G) * HD) + i % (HD / 4));
        reinterpret_cast<int *>(s_q)[i] = v;
    }
    if (tid < R) {
        const uint32_t r = r0 + tid, c = r < n_rows ? pos0 + r / G + 1 : 0u;
        const float qas = r < n_rows ? __fmul_rn(__ldcg(a.q_scale + (size_t)(r / G) * n_q + kvh * G + r % G), a.attn_scale) : 0.0f;
        s_row[tid] = make_float4(qas, __uint_as_float(c), __uint_as_float((c & ~255u) + (c & 255u & ~7u)), 0.0f);
    }
    __syncthreads();
    const bool full_rows = r0 + R <= n_rows;
    // ---- scores: dot * (ks * qas) in whole groups of eight positions of a 256-position tile, (dot * ks) * qas behind them
    {
        float m[R];
#pragma unroll
        for (int r = 0; r < R; ++r) m[r] = -INFINITY;
        const uint32_t plain_end = full_rows ? (ctx_lo & ~255u) + (ctx_lo & 255u & ~7u) : 0u;          // below: no row is masked or outside its groups
        const uint4 *K = reinterpret_cast<const uint4 *>(a.k_q8 + slot0 * HD);
        const float *ks_p = a.k_scale + slot0;
#pragma unroll 1
        for (uint32_t t = tid; t < ctx16; t += NT) {
            uint4 k[KW];
            const bool in = t < ctx;
#pragma unroll
            for (uint32_t i = 0; i < KW; ++i) k[i] = in ? __ldcg(K + (size_t)t * KW + i) : make_uint4(0, 0, 0, 0);
            const float ks = in ? __ldcg(ks_p + t) : 0.0f;
            const bool plain = t < plain_end;
#pragma unroll
            for (uint32_t rq = 0; rq < RQ; ++rq) {
                float s[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t r = rq * 4 + j;
                    int d = 0;
#pragma unroll
                    for (uint32_t i = 0; i < KW; ++i) {
                        const int4 q = *reinterpret_cast<const int4 *>(s_q + r * HD + i * 16);
                        d = __dp4a((int)k[i].x, q.x, d); d = __dp4a((int)k[i].y, q.y, d); d = __dp4a((int)k[i].z, q.z, d); d = __dp4a((int)k[i].w, q.w, d);
                    }
                    const float4 c = s_row[r];
                    const float df = (float)d;
                    s[j] = __fmul_rn(df, __fmul_rn(ks, c.x));
                    if (!plain) {
                        if (t >= __float_as_uint(c.z)) s[j] = __fmul_rn(__fmul_rn(df, ks), c.x);
                        if (t >= __float_as_uint(c.y)) s[j] = -INFINITY;
                    }
                    m[r] = fmaxf(m[r], s[j]);
                }
                *reinterpret_cast<float4 *>(s_p + (size_t)t * R + ((rq ^ pos_swz<R>(t)) << 2)) = make_float4(s[0], s[1], s[2], s[3]);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float v = warp_max(m[r]);
            if (lane == 0) s_red[warp * R + r] = v;
        }
    }
    __syncthreads();
    if (tid < R) {
        float v = s_red[tid];
        for (uint32_t w = 1; w < NW; ++w) v = fmaxf(v, s_red[w * R + tid]);
        s_max[tid] = v;
    }
    __syncthreads();
    // ---- exp
    {
        const uint32_t plain_end = full_rows ? ctx_lo & ~3u : 0u;
#pragma unroll 1
        for (uint32_t t = tid; t < ctx16; t += NT) {
            const bool plain = t < plain_end;
#pragma unroll
            for (uint32_t rq = 0; rq < RQ; ++rq) {
                float4 *p = reinterpret_cast<float4 *>(s_p + (size_t)t * R + ((rq ^ pos_swz<R>(t)) << 2));
                const float4 v = *p, mx = *reinterpret_cast<const float4 *>(s_max + rq * 4);
                float x[4] = {__fsub_rn(v.x, mx.x), __fsub_rn(v.y, mx.y), __fsub_rn(v.z, mx.z), __fsub_rn(v.w, mx.w)};
                if (plain) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) x[j] = exp_poly(x[j]);
                } else {
#pragma unroll 1
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t c = __float_as_uint(s_row[rq * 4 + j].y);
                        x[j] = t < (c & ~3u) ? exp_poly(x[j]) : t < c ? (float)exp((double)x[j]) : 0.0f;
                    }
                }
                *p = make_float4(x[0], x[1], x[2], x[3]);
            }
        }
    }
    __syncthreads();
    // ---- denominators: lane = (row, accumulator); accumulator i adds the terms 4 k + i, k ascending, then (a0 + a1) + (a2 + a3) and
    // the terms behind the last whole group of four
    if (tid < 4 * R) {
        const uint32_t r = tid % R, i = tid / R, c = __float_as_uint(s_row[r].y), n = c / 4;
        const uint32_t r4 = r >> 2, rl = r & 3u;
        auto term = [&](uint32_t t) { return s_p[(size_t)t * R + (((r4 ^ pos_swz<R>(t)) << 2) | rl)]; };
        float acc = 0.0f;
        const uint32_t n_all = full_rows ? (ctx_lo / 4) & ~7u : 0u;          // terms every row has, in rounds of eight
        uint32_t k = 0;
        if (n_all > 0) {
            float A[8], B[8];
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) A[u] = term(4 * u + i);
            for (; k + 8 < n_all; k += 8) {
#pragma unroll
                for (uint32_t u = 0; u < 8; ++u) B[u] = term(4 * (k + 8 + u) + i);
#pragma unroll
                for (uint32_t u = 0; u < 8; ++u) { acc = __fadd_rn(acc, A[u]); A[u] = B[u]; }
            }
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) acc = __fadd_rn(acc, A[u]);
            k += 8;
        }
        for (; k < n; ++k) acc = __fadd_rn(acc, term(4 * k + i));
        s_o[i * R + r] = acc;
    }
    __syncthreads();
    if (tid < R) {
        const uint32_t r = tid, c = __float_as_uint(s_row[r].y);
        float acc = __fadd_rn(__fadd_rn(s_o[r], s_o[R + r]), __fadd_rn(s_o[2 * R + r], s_o[3 * R + r]));
        for (uint32_t t = c & ~3u; t < c; ++t) acc = __fadd_rn(acc, s_p[(size_t)t * R + ((((r >> 2) ^ pos_swz<R>(t)) << 2) | (r & 3u))]);
        s_inv[r] = __fdiv_rn(1.0f, acc);
    }
    __syncthreads();
    // ---- value weights
    {
        const float *vs_p = a.v_scale + slot0;
#pragma unroll 1
        for (uint32_t t = tid; t < ctx16; t += NT) {
            const float vs = t < ctx ? __ldcg(vs_p + t) : 0.0f;
            const bool plain = full_rows && t < ctx_lo;
#pragma unroll
            for (uint32_t rq = 0; rq < RQ; ++rq) {
                float4 *p = reinterpret_cast<float4 *>(s_p + (size_t)t * R + ((rq ^ pos_swz<R>(t)) << 2));
                const float4 v = *p, inv = *reinterpret_cast<const float4 *>(s_inv + rq * 4);
                float w[4] = {__fmul_rn(__fmul_rn(v.x, inv.x), vs), __fmul_rn(__fmul_rn(v.y, inv.y), vs), __fmul_rn(__fmul_rn(v.z, inv.z), vs), __fmul_rn(__fmul_rn(v.w, inv.w), vs)};
                if (!plain) {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (t >= __float_as_uint(s_row[rq * 4 + j].y)) w[j] = 0.0f;
                }
                *p = make_float4(w[0], w[1], w[2], w[3]);
            }
        }
    }
    __syncthreads();
    // ---- chains: thread = dimension d, rows g * NR .. g * NR + NR - 1; sixteen positions per 16-byte load of the block-transposed values
    {
        const uint32_t g = tid / HD, d = tid % HD;
        const uint4 *V = reinterpret_cast<const uint4 *>(a.v_t + slot0 * HD) + d;
        unsigned long long o[NR / 2];
#pragma unroll
        for (uint32_t r = 0; r < NR / 2; ++r) o[r] = 0;
        const uint32_t nblk = ctx16 / 16;
        uint4 x = __ldcg(V), xn = nblk > 1 ? __ldcg(V + HD) : x;
        // float4 j of the group at position k: index (g * NR / 4 + j) ^ swz(k)
        const uint32_t base0 = p_sa + g * (NR * 4), base1 = p_sa + (g ^ 1u) * (NR * 4);
#pragma unroll 1
        for (uint32_t b = 0; b < nblk; ++b) {
            const uint4 x2 = b + 2 < nblk ? __ldcg(V + (size_t)(b + 2) * HD) : x;
            const uint32_t off = b * (16 * R * 4), w0 = base0 + off, w1 = base1 + off;
            const uint32_t xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (uint32_t k = 0; k < 16; ++k) {
                // 0x4B000000 | (b ^ 0x80) is the float 2^23 + 128 + (int8)b
                const unsigned long long v = dup_f32(__fsub_rn(__uint_as_float(prmt(xs[k / 4], 0x4B000000u, 0x7440u + (k % 4))), 8388736.0f));
                const uint32_t f = pos_swz<R>(k);
#pragma unroll
                for (uint32_t j = 0; j < NR / 4; ++j) {
                    unsigned long long wa, wb;
                    const uint32_t at = R == 16 ? ((f >> 1) ? w1 : w0) + ((j ^ (f & 1u)) << 4) : (f ? w1 : w0);
                    asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(wa), "=l"(wb) : "r"(at + k * (R * 4)));
                    o[2 * j] = fma_f32x2(v, wa, o[2 * j]);
                    o[2 * j + 1] = fma_f32x2(v, wb, o[2 * j + 1]);
                }
            }
            x = xn; xn = x2;
        }
        pdl_trigger();
#pragma unroll
        for (uint32_t r = 0; r < NR; ++r) s_o[(g * NR + r) * HD + d] = __uint_as_float((r & 1u) ? (uint32_t)(o[r / 2] >> 32) : (uint32_t)o[r / 2]);
    }
    __syncthreads();
    // ---- inverse rotation (block index within the head), forward rotation with the global chunk index, int8 for o_proj
    for (uint32_t u = warp; u < R * NB; u += NW) {
        const uint32_t r = r0 + u / NB, b = u % NB;
        if (r >= n_rows) continue;
        const uint32_t tok = r / G, qh = kvh * G + r % G, c = qh * NB + b;
        float x0 = s_o[(u / NB) * HD + b * 64 + 2 * lane], x1 = s_o[(u / NB) * HD + b * 64 + 2 * lane + 1];
        warp_ifwht64(x0, x1, b, lane);
        if (a.attn_out != nullptr && tok + 1 == a.n_tok) reinterpret_cast<float2 *>(a.attn_out + (size_t)qh * HD + b * 64)[lane] = make_float2(x0, x1);
        warp_fwht64(x0, x1, a.out_chunk0 + c, lane);
        int q0, q1, sum;
        float scl;
        warp_quant64(x0, x1, q0, q1, scl, sum);
        const size_t row = (size_t)tok * n_q * NB;           // o_proj activation row of this token, in chunks
        reinterpret_cast<char2 *>(a.out_q + (row + c) * 64)[lane] = make_char2((signed char)q0, (signed char)q1);
        if (lane == 0) { a.out_scales[row + c] = scl; a.out_sums[row + c] = sum; }
    }
}

template <int HD, int R> cudaError_t launch_prompt(cudaStream_t s, const ExactAttnArgs &a, bool pdl) {
    const size_t smem = PromptAttn<HD, R>::bytes(a.ctx_cap);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(attn_prompt_kernel<HD, R>), smem);
    if (e != cudaSuccess) return e;
    return launch_kernel(attn_prompt_kernel<HD, R>, dim3(a.n_kv, (a.n_tok * a.group + R - 1) / R), dim3(2 * HD), smem, s, pdl, a);
}
constexpr size_t PROMPT_SMEM_MAX = 220 * 1024;

}  // namespace

bool attention_prompt_fits(uint32_t head_dim, uint32_t ctx) {
    return head_dim == 64 ? PromptAttn<64, 8>::bytes(ctx) <= PROMPT_SMEM_MAX : head_dim == 128 && PromptAttn<128, 8>::bytes(ctx) <= PROMPT_SMEM_MAX;
}
uint32_t attention_prompt_rows(uint32_t head_dim, uint32_t ctx) {
    if (!attention_prompt_fits(head_dim, ctx)) return 0;
    return (head_dim == 64 ? PromptAttn<64, 16>::bytes(ctx) : PromptAttn<128, 16>::bytes(ctx)) <= PROMPT_SMEM_MAX ? 16 : 8;
}
bool attention_prompt_pays(uint32_t n_tok, uint32_t n_q, uint32_t n_kv, uint32_t head_dim, uint32_t ctx) {
    const uint32_t rows = n_tok * n_q;
    if (n_tok < PROMPT_ATTN_MIN_TOKENS) return false;
    if (n_q == n_kv) return rows >= 1536 || ctx <= (rows >= 1024 ? 512u : 256u);
    if (head_dim == 128) return rows >= 896 || ctx <= 768;
    return rows >= 1152 || ctx <= (rows >= 576 ? 896u : 384u);
}
bool attention_prompt_takes(const ExactAttnArgs &a, uint32_t n_tok) {
    return a.kv_bits == 8 && a.v_t != nullptr && a.ring.window == 0 && attention_prompt_fits(a.head_dim, a.ctx_cap) &&
           attention_prompt_pays(n_tok, a.n_kv * a.group, a.n_kv, a.head_dim, a.ctx_cap);
}

cudaError_t launch_attention_prompt(cudaStream_t s, const ExactAttnArgs &args, bool pdl, uint32_t n_tok) {
    if (args.kv_bits != 8 || args.v_t == nullptr || args.ring.window != 0 || args.group == 0 || n_tok == 0) return cudaErrorInvalidValue;
    const uint32_t rows = attention_prompt_rows(args.head_dim, args.ctx_cap);
    if (rows == 0) return cudaErrorInvalidValue;
    ExactAttnArgs a = args;
    a.n_tok = n_tok;
    if (a.head_dim == 64) return rows == 16 ? launch_prompt<64, 16>(s, a, pdl) : launch_prompt<64, 8>(s, a, pdl);
    return rows == 16 ? launch_prompt<128, 16>(s, a, pdl) : launch_prompt<128, 8>(s, a, pdl);
}

}  // namespace k2t
