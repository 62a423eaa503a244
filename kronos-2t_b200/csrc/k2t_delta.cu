// Generalized delta rule of the block engine (k2t_block_kernels.h), fp32 throughout: per head a state S [key][value] with
//   S_t = diag(w) S_(t-1) - (a u)(u^T S_(t-1)) + k v^T,   o_t = S_t^T r,
// w the decay and a the removal rate per key channel, u the unit key.  Columns of S do not meet, so a column group of a head is
// an independent chain.
//   * delta_step_kernel (one token): a cluster per head.  The state is requested before the dependency wait (only the same
//     layer's previous step wrote it), then coefficients, recurrence, per-head norm, output gate and the activation of the output
//     projection in one launch.
//   * prompts: delta_chunk_kernel turns sixteen tokens of a head into one record of coefficients, delta_scan_kernel walks the records -
//     a CTA holds sixteen columns of a head's state - and delta_post_kernel norms and gates.
#include <algorithm>
#include <cmath>

#include "k2t_block_kernels.h"
#include "k2t_dense.cuh"

namespace k2t {
namespace {

__device__ __forceinline__ float sigmoidf(float x) { return 1.0f / (1.0f + expf(-x)); }
// Decays are kept as w - 1: a channel that decays by a hair per token would lose that hair in the rounding of w, the same way
// at every token, and a state carried over thousands of tokens would show it.
__device__ __forceinline__ float decay_minus_one(float scale, float logit) { return expm1f(-scale * sigmoidf(logit)); }

// ------------------------------------------------------------------------------------------------ one token
// A cluster of drow / 32 CTAs per head, CTA = 32 columns: thread = (four columns, KPS = drow / 32 keys).  Every CTA makes the
// head's coefficients; only the sum of squares of o crosses the cluster.
constexpr uint32_t ST_THREADS = 256, ST_COLS = 32, ST_SLICES = ST_THREADS / (ST_COLS / 4);
constexpr uint32_t ST_WAIT_LIMIT = 1u << 22;
inline size_t step_vec_smem(uint32_t drow, uint32_t rank_pad) { return (((size_t)5 * drow + ST_COLS + ST_SLICES * ST_COLS + rank_pad) * 4 + 127) & ~(size_t)127; }

template <bool F32, int KPS, bool STAGED>
__global__ void __launch_bounds__(ST_THREADS) delta_step_kernel(const DeltaArgs a, uint32_t weights_at) {
    extern __shared__ __align__(128) float sm[];
    __shared__ float scratch[32], slots[8];
    __shared__ __align__(8) uint64_t bar_w;
    constexpr uint32_t D = 32 * KPS, SLICES = ST_SLICES;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cs = cluster_size(), me = cluster_rank(), h = blockIdx.x / cs, dim = a.dim;
    const uint32_t q = tid & 7u, sl = tid >> 3, col0 = me * ST_COLS, rank_pad = (a.rank + 63) / 64 * 64;
    float *s_w = sm, *s_au = s_w + D, *s_u = s_au + D, *s_k = s_u + D, *s_r = s_k + D, *s_v = s_r + D, *s_red = s_v + ST_COLS, *s_t = s_red + SLICES * ST_COLS;
    float4 st[KPS];
    float *state = a.state + (size_t)h * D * D + (size_t)(sl * KPS) * D + col0 + q * 4;
#pragma unroll
    for (uint32_t i = 0; i < KPS; ++i) st[i] = __ldcg(reinterpret_cast<const float4 *>(state + (size_t)i * D));
    for (uint32_t i = tid; i < 5 * D + ST_COLS; i += ST_THREADS) sm[i] = 0.0f;
    for (uint32_t i = tid; i < rank_pad; i += ST_THREADS) s_t[i] = 0.0f;
    DenseView decay = a.decay;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&bar_w), row0 = h * dim & ~7u;          // the head's rows, from a whole swizzle octet on
    if (STAGED) {       // the head's rows of the decay product: weights, copied while the predecessor runs
        uint8_t *s_d = reinterpret_cast<uint8_t *>(sm) + weights_at;
        const uint32_t rows = h * dim + dim - row0;
        if (tid == 0) {
            mbar_init(bar, 1);
            fence_mbar_init();
            mbar_expect_tx(bar, rows * 128 * decay.panels);
            for (uint32_t p = 0; p < decay.panels; ++p)
                bulk_g2s((uint32_t)__cvta_generic_to_shared(s_d) + p * rows * 128, static_cast<const uint8_t *>(a.decay.base) + ((size_t)p * a.decay.rows_pad + row0) * 128, rows * 128, bar);
        }
        decay.base = s_d; decay.rows_pad = rows;
    }
    const float norm_w = tid < ST_COLS && col0 + tid < dim ? __ldg(a.norm + h * dim + col0 + tid) : 0.0f;
    if (cs > 1) cluster_sync_all();             // every CTA of the cluster runs before its shared memory is written from outside
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    const uint32_t HD = a.heads * dim;
    const float *in = a.in + h * dim;
    float kk[1] = {0.0f}, rate = 0.0f, gate = 0.0f, bias = 0.0f;
    if (tid < dim) {                            // dim <= 256 = threads
        const float k = __ldcg(in + HD + tid);
        s_r[tid] = __ldcg(in + tid);
        s_k[tid] = k;
        rate = __ldcg(in + 4 * HD + tid) + __ldg(a.rate_bias + h * dim + tid);
        bias = __ldg(a.decay_bias + h * dim + tid);
        kk[0] = k * k;
    }
    if (tid < ST_COLS && col0 + tid < dim) { s_v[tid] = __ldcg(in + 2 * HD + col0 + tid); gate = __ldcg(in + 3 * HD + col0 + tid); }
    for (uint32_t i = tid; i < a.rank; i += ST_THREADS) s_t[i] = tanhf(__ldcg(a.in + 5 * HD + i));
    block_sum<1>(kk, scratch);                          // its barriers also publish s_t, s_k
    const float inv_k = 1.0f / sqrtf(kk[0] + a.unit_eps);
    if (tid < dim) { const float u = s_k[tid] * inv_k; s_u[tid] = u; s_au[tid] = sigmoidf(rate) * u; }
    if (STAGED) {
        bool ok = false;
        for (uint32_t spin = 0; spin < ST_WAIT_LIMIT && !ok; ++spin) ok = mbar_try_wait(bar, 0u);
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    }
    const uint32_t sub = lane & 7u;
#pragma unroll 1
    for (uint32_t r0 = warp * 4; r0 < dim; r0 += ST_THREADS / 8) {
        const uint32_t i = r0 + (lane >> 3), c = h * dim + min(i, dim - 1);
        const float z = row_dot8<F32, STAGED>(decay, STAGED ? c - row0 : c, 0, decay.panels, s_t, sub);
        if (i < dim && sub == 0) s_w[i] = z;
    }
    __syncthreads();
    if (tid < dim) s_w[tid] = decay_minus_one(a.decay_scale, s_w[tid] + bias);
    __syncthreads();
    float4 c = make_float4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t i = 0; i < KPS; ++i) {
        const float u = s_u[sl * KPS + i];
        c.x = __fmaf_rn(u, st[i].x, c.x); c.y = __fmaf_rn(u, st[i].y, c.y); c.z = __fmaf_rn(u, st[i].z, c.z); c.w = __fmaf_rn(u, st[i].w, c.w);
    }
    *reinterpret_cast<float4 *>(s_red + sl * ST_COLS + q * 4) = c;
    __syncthreads();
    c = make_float4(0, 0, 0, 0);
#pragma unroll 8
    for (uint32_t s = 0; s < SLICES; ++s) {
        const float4 p = *reinterpret_cast<const float4 *>(s_red + s * ST_COLS + q * 4);
        c.x += p.x; c.y += p.y; c.z += p.z; c.w += p.w;
    }
    const float4 v = *reinterpret_cast<const float4 *>(s_v + q * 4);
    float4 o = make_float4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t i = 0; i < KPS; ++i) {
        const uint32_t key = sl * KPS + i;
        const float w = s_w[key], au = -s_au[key], k = s_k[key], r = s_r[key];
        st[i].x = __fmaf_rn(au, c.x, __fmaf_rn(w, st[i].x, __fmaf_rn(k, v.x, st[i].x))); st[i].y = __fmaf_rn(au, c.y, __fmaf_rn(w, st[i].y, __fmaf_rn(k, v.y, st[i].y)));
        st[i].z = __fmaf_rn(au, c.z, __fmaf_rn(w, st[i].z, __fmaf_rn(k, v.z, st[i].z))); st[i].w = __fmaf_rn(au, c.w, __fmaf_rn(w, st[i].w, __fmaf_rn(k, v.w, st[i].w)));
        o.x = __fmaf_rn(r, st[i].x, o.x); o.y = __fmaf_rn(r, st[i].y, o.y); o.z = __fmaf_rn(r, st[i].z, o.z); o.w = __fmaf_rn(r, st[i].w, o.w);
        *reinterpret_cast<float4 *>(state + (size_t)i * D) = st[i];
    }
    __syncthreads();                                    // every thread has read the partial sums
    *reinterpret_cast<float4 *>(s_red + sl * ST_COLS + q * 4) = o;
    __syncthreads();
    float so[1] = {0.0f}, mine = 0.0f;
    if (tid < ST_COLS) {
#pragma unroll 8
        for (uint32_t s = 0; s < SLICES; ++s) mine += s_red[s * ST_COLS + tid];          // columns beyond dim hold zeros
        so[0] = warp_sum(mine * mine);
        if (tid == 0) scratch[0] = so[0];
    }
    __syncthreads();
    so[0] = scratch[0];
    cluster_sum<1>(so, slots);
    const float inv = 1.0f / sqrtf(so[0] / (float)dim + a.eps);
    if (tid < ST_COLS && col0 + tid < dim) act_store<F32>(a.out, 0, h * dim + col0 + tid, mine * inv * norm_w * sigmoidf(gate));
    if (cs > 1) cluster_sync_all();                     // no CTA leaves while a peer may still write to it
}

// ------------------------------------------------------------------------------------------------ prompts
template <bool F32>
__global__ void __launch_bounds__(256) delta_tanh_kernel(const float *__restrict__ in, size_t in_stride, uint32_t rank, uint32_t n_tok, const Act out) {
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    pdl_wait();
    pdl_trigger();
    if (i >= n_tok * rank) return;
    act_store<F32>(out, i / rank, i % rank, tanhf(__ldcg(in + (i / rank) * in_stride + i % rank)));
}

// Prompts run in chunks of sixteen tokens, each a step of matrix products.  With S the state ahead of a chunk, W_t = w_1 .. w_t by key channel,
//   c_t = u_t^T S_(t-1) = U_t^T S + sum over s < t of (G_ts v_s - H_ts c_s),     U_t = u_t W_(t-1),
//   o_t = S_t^T r_t     = R_t^T S + sum over s <= t of (P_ts v_s - Q_ts c_s),    R_t = r_t W_t,
// G, H, P, Q the products by key channel of U or R with k_s / W_s and (a u)_s / W_s.  The triangular system for the c is solved ahead
// of the scan, on the coefficients: c = A1 S + B1 v, o = A2 S + B2 v, and S <- W S + K^T v - A^T c, K_s = k_s w_(s+1) .. w_last, A alike.
// What is left in sequence is one step of three products per sixteen tokens, where groups of four took a round of shuffles and 26 dependent
// multiply-adds each.  The error against 64 bits stays that of groups of four (2048 random tokens, outputs: 1.1e-7 both; slow decays and
// alike keys 2.5e-7 and 2.6e-7; fast decays 1.0e-7 both): W is a product and W - 1 a sum of its own, neither is had from the other.
// A chunk's record: [drow + 16][32] (A1 | A2 by key, then B1 | B2 by source token), [32][drow] (K, then -A), W - 1 [drow],
// v [drow / 16][16][16].  A decay is at least exp(-decay_scale), so W stays above exp(-40) over the tokens chunk_len allows a chunk.
constexpr uint32_t CHUNK = 16, CCOLS = 16;
__host__ __device__ constexpr uint32_t chunk_shared_floats(uint32_t drow) { return (drow + CHUNK) * 2 * CHUNK + 2 * CHUNK * drow + drow; }      // what every column group reads
__host__ __device__ constexpr uint32_t chunk_floats(uint32_t drow) { return chunk_shared_floats(drow) + CHUNK * drow; }

// One CTA per (chunk, head), thread = key channel.  2048 tokens of 16 heads of 128: 103 us (with the 1 / W, 90 MB of records and loads whose
// latency four CTAs an SM do not hide); the records of groups of four took 71.
template <int D>
__global__ void __launch_bounds__(D, 512 / D) delta_chunk_kernel(const DeltaArgs a, uint32_t n_tok, uint32_t len) {
    extern __shared__ __align__(16) float cm[];
    constexpr uint32_t PITCH = D + 4, SP = 36;          // rows 16 bytes apart in the banks
    float *sa = cm, *sb = sa + 32 * PITCH, *sp = sb + 32 * PITCH, *s_inv = sp + 32 * SP, *sd = s_inv + CHUNK, *su = sd + CHUNK * D;          // sd, su: a thread's own decays and removals
    const uint32_t c = threadIdx.x, lane = c & 31, warp = c >> 5, h = blockIdx.y, tok0 = blockIdx.x * len, dim = a.dim, HD = a.heads * dim;
    pdl_wait();
    pdl_trigger();
    float *rec = a.rec + ((size_t)h * gridDim.x + blockIdx.x) * chunk_floats(D);
    const float *in = a.in + (size_t)tok0 * a.in_stride + h * dim + c;
    const uint32_t n = min(len, n_tok - tok0);
    float k[CHUNK];
#pragma unroll
    for (uint32_t t = 0; t < CHUNK; ++t) {
        const bool on = t < n && c < dim;
        k[t] = on ? __ldcg(in + t * a.in_stride + HD) : 0.0f;
        sd[t * D + c] = on ? __ldcg(a.decay_logit + (size_t)(tok0 + t) * a.logit_stride + h * dim + c) : 0.0f;
        su[t * D + c] = on ? __ldcg(in + t * a.in_stride + 4 * HD) : 0.0f;
        sb[t * PITCH + c] = k[t];
    }
    __syncthreads();
#pragma unroll
    for (uint32_t t = warp; t < CHUNK; t += D / 32) {
        float kk = 0.0f;
#pragma unroll
        for (uint32_t i = 0; i < D / 32; ++i) { const float x = sb[t * PITCH + lane + 32 * i]; kk = __fmaf_rn(x, x, kk); }
        kk = warp_sum(kk);
        if (lane == 0) s_inv[t] = 1.0f / sqrtf(kk + a.unit_eps);
    }
    __syncthreads();
    const float bias = c < dim ? __ldg(a.decay_bias + h * dim + c) : 0.0f, rate = c < dim ? __ldg(a.rate_bias + h * dim + c) : 0.0f;
    float w = 1.0f, e = 0.0f;                // W_t, W_t - 1
#pragma unroll 4
    for (uint32_t t = 0; t < CHUNK; ++t) {
        const bool on = t < n && c < dim;
        const float kt = sb[t * PITCH + c], u = kt * s_inv[t], r = on ? __ldcg(in + t * a.in_stride) : 0.0f, v = on ? __ldcg(in + t * a.in_stride + 2 * HD) : 0.0f;
        const float d = on ? decay_minus_one(a.decay_scale, sd[t * D + c] + bias) : 0.0f, au = on ? sigmoidf(su[t * D + c] + rate) * u : 0.0f;
        sd[t * D + c] = d; su[t * D + c] = au;
        sa[t * PITCH + c] = u * w;
        e = __fmaf_rn(e, d, e + d);
        w = fmaxf(w * (1.0f + d), 1e-30f);          // what decays further in one token leaves nothing of what was there
        const float iw = 1.0f / w;
        sa[(CHUNK + t) * PITCH + c] = r * w;
        sb[t * PITCH + c] = kt * iw; sb[(CHUNK + t) * PITCH + c] = au * iw;
        rec[chunk_shared_floats(D) + (c / CCOLS) * CHUNK * CCOLS + t * CCOLS + c % CCOLS] = v;
    }
    {
        float *m2 = rec + (D + CHUNK) * 2 * CHUNK + c, suffix = 1.0f;
        m2[2 * CHUNK * D] = e;
#pragma unroll
        for (int t = CHUNK - 1; t >= 0; --t) {
            m2[t * D] = k[t] * suffix; m2[(CHUNK + t) * D] = -su[t * D + c] * suffix;
            suffix *= 1.0f + sd[t * D + c];
        }
    }
    __syncthreads();
    {          // the 32 x 32 products: a thread's rows lie 8 apart, its columns next to one another
        constexpr uint32_t NJ = D >= 256 ? 1 : D >= 128 ? 2 : 4, LJ = 32 / NJ;          // 4 x NJ products a thread, 8 LJ threads
        static_assert(8 * LJ <= D, "every product has a thread");
        const uint32_t i0 = c / LJ, j0 = (c % LJ) * NJ;
        if (c < 8 * LJ) {
            float acc[4][NJ];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < (int)NJ; ++j) acc[i][j] = 0.0f;
#pragma unroll 2
            for (uint32_t x = 0; x < D; x += 4) {
                float4 q[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4 *>(sa + (i0 + 8 * i) * PITCH + x);
#pragma unroll
                for (int j = 0; j < (int)NJ; ++j) {
                    const float4 y = *reinterpret_cast<const float4 *>(sb + (j0 + j) * PITCH + x);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][j] = __fmaf_rn(q[i].w, y.w, __fmaf_rn(q[i].z, y.z, __fmaf_rn(q[i].y, y.y, __fmaf_rn(q[i].x, y.x, acc[i][j]))));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < (int)NJ; ++j) sp[(i0 + 8 * i) * SP + j0 + j] = acc[i][j];
        }
    }
    __syncthreads();
    // rows of sp: U_t, then R_t; columns: k_s / W_s, then (a u)_s / W_s.  x1 solves the system (a row of H at a time), x2 follows from it;
    // both go to `to`, 32 floats in 16-byte pieces: A1 | A2
    auto solve = [&](auto first, auto second, auto to) {
        float x1[CHUNK];
        auto less = [&](float x, const float *row, uint32_t count) {
#pragma unroll
            for (uint32_t q = 0; q < CHUNK; q += 4)
                if (q < count) {
                    const float4 m = *reinterpret_cast<const float4 *>(row + q);
                    x = __fmaf_rn(-m.x, x1[q], x);
                    if (q + 1 < count) x = __fmaf_rn(-m.y, x1[q + 1], x);
                    if (q + 2 < count) x = __fmaf_rn(-m.z, x1[q + 2], x);
                    if (q + 3 < count) x = __fmaf_rn(-m.w, x1[q + 3], x);
                }
            return x;
        };
#pragma unroll
        for (uint32_t t = 0; t < CHUNK; ++t) {
            x1[t] = less(first(t), sp + t * SP + CHUNK, t);
            if (t % 4 == 3) { to(t / 4, make_float4(x1[t - 3], x1[t - 2], x1[t - 1], x1[t])); asm volatile("" ::: "memory"); }
        }
#pragma unroll
        for (uint32_t t = 0; t < CHUNK; t += 4) {
            float x2[4];
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) x2[i] = less(second(t + i), sp + (CHUNK + t + i) * SP + CHUNK, t + i + 1);
            to(4 + t / 4, make_float4(x2[0], x2[1], x2[2], x2[3]));
            asm volatile("" ::: "memory");
        }
    };
    // nobody reads sb any more: the key's 32 coefficients, pieces swizzled by key
    solve([&](uint32_t t) { return sa[t * PITCH + c]; }, [&](uint32_t t) { return sa[(CHUNK + t) * PITCH + c]; },
          [&](uint32_t q, float4 v) { *reinterpret_cast<float4 *>(sb + c * 2 * CHUNK + ((q ^ (c & 7u)) * 4)) = v; });
    if (c < CHUNK)          // the same for the values: source token c
        solve([&](uint32_t t) { return c < t ? sp[t * SP + c] : 0.0f; }, [&](uint32_t t) { return c <= t ? sp[(CHUNK + t) * SP + c] : 0.0f; },
              [&](uint32_t q, float4 v) { *reinterpret_cast<float4 *>(rec + (D + c) * 2 * CHUNK + q * 4) = v; });
    __syncthreads();
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t at = i * D + c, key = at >> 3, q = at & 7u;
        reinterpret_cast<float4 *>(rec)[at] = *reinterpret_cast<const float4 *>(sb + key * 2 * CHUNK + ((q ^ (key & 7u)) * 4));
    }
}

constexpr uint32_t SC_WAIT_LIMIT = 1u << 22, SC_THREADS = 256, SC_PITCH = 20;          // pitch: rows of 16 floats, four of them 16 banks on
template <int D> struct ScanLayout {
    static constexpr uint32_t STAGES = D > 192 ? 2 : 3, SHARED = chunk_shared_floats(D), STAGE = SHARED + CHUNK * CCOLS;
    static constexpr uint32_t X = STAGES * STAGE;                                      // [D + 48][20]: the state, v of two chunks, c
    static constexpr uint32_t PART = X + (D + 48) * SC_PITCH;                          // [8][32][20]: partial sums of c and o
    static constexpr uint32_t TOTAL = (PART + 8 * 32 * SC_PITCH) * 4;
};

// CTA = 16 columns of a head's state.  Per chunk: 8 warps share the rows of (A1 | A2)^T S + (B1 | B2)^T v, 4 x 4 products a lane; the warps' sums
// are added; then S takes its 32 updates, four keys x two columns at a time, those of v while the sums meet.  Bound by shared-memory reads
// (0.76 of wavefronts): 4 x 4 products per two 16-byte reads.  2048 tokens of 16 heads of 128: 216 us, in groups of four 337.
template <int D>
__global__ void __launch_bounds__(SC_THREADS, 1) delta_scan_kernel(const float *__restrict__ rec, uint32_t n_tok, uint32_t len, float *__restrict__ state, float *__restrict__ o, uint32_t heads,
                                                                   uint32_t *__restrict__ err_flag) {
    extern __shared__ __align__(128) float ring[];
    __shared__ __align__(8) uint64_t bars[3];
    using L = ScanLayout<D>;
    constexpr uint32_t NU = (2 * D + SC_THREADS - 1) / SC_THREADS, ROWS = (D + CHUNK) / 8, KG = D / 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, col0 = blockIdx.x * CCOLS;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(bars), rb = (uint32_t)__cvta_generic_to_shared(ring);
    const uint32_t chunks = (n_tok + len - 1) / len;
    const float *src = rec + (size_t)h * chunks * chunk_floats(D);
    float *X = ring + L::X, *part = ring + L::PART;
    if (tid == 0) {
        for (uint32_t i = 0; i < L::STAGES; ++i) mbar_init(bar + 8 * i, 1);
        fence_mbar_init();
    }
    // this thread's part of the state: keys 4 kg .., columns 2 cp, 2 cp + 1 of unit u (a warp: four key groups x eight column pairs)
    const uint32_t cp = lane & 7u, kg0 = warp * 4 + (lane >> 3);
    float *sp = state + (size_t)h * D * D + col0 + 2 * cp;
    float2 st[NU][4];
#pragma unroll
    for (uint32_t u = 0; u < NU; ++u) {
        const uint32_t kg = kg0 + 32 * u;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            st[u][i] = kg < KG ? __ldcg(reinterpret_cast<const float2 *>(sp + (size_t)(4 * kg + i) * D)) : make_float2(0.0f, 0.0f);
            if (kg < KG) *reinterpret_cast<float2 *>(X + (4 * kg + i) * SC_PITCH + 2 * cp) = st[u][i];
        }
    }
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    auto request = [&](uint32_t c) {
        const uint32_t b = bar + 8 * (c % L::STAGES), dst = rb + (c % L::STAGES) * L::STAGE * 4;
        const float *q = src + (size_t)c * chunk_floats(D);
        mbar_expect_tx(b, L::STAGE * 4);
        bulk_g2s(dst, q, L::SHARED * 4, b);
        bulk_g2s(dst + L::SHARED * 4, q + L::SHARED + blockIdx.x * CHUNK * CCOLS, CHUNK * CCOLS * 4, b);
    };
    auto landed = [&](uint32_t c) {          // and v of chunk c beside the state; false: gave up
        bool ok = mbar_try_wait(bar + 8 * (c % L::STAGES), (c / L::STAGES) & 1u);
        for (uint32_t spin = 0; spin < SC_WAIT_LIMIT && !ok; ++spin) ok = mbar_try_wait(bar + 8 * (c % L::STAGES), (c / L::STAGES) & 1u);
        X[(D + CHUNK * (c & 1u) + (tid >> 4)) * SC_PITCH + (tid & 15u)] = ring[(c % L::STAGES) * L::STAGE + L::SHARED + tid];
        return ok;
    };
    if (tid == 0)
        for (uint32_t c = 0; c < min(L::STAGES, chunks); ++c) request(c);
    bool ok = landed(0);
    const uint32_t oi = lane >> 2, cj = lane & 3u;
    for (uint32_t c = 0; c < chunks; ++c) {
        if (__syncthreads_or(!ok)) {            // a copy did not land: report, let the others in flight land, leave
            if (tid == 0 && err_flag != nullptr) atomicExch(err_flag, 1u);
            for (uint32_t d = c; d < min(c + L::STAGES, chunks); ++d)
                for (uint32_t spin = 0; spin < SC_WAIT_LIMIT && !mbar_try_wait(bar + 8 * (d % L::STAGES), (d / L::STAGES) & 1u); ++spin) {}
            return;
        }
        const float *stage = ring + (c % L::STAGES) * L::STAGE, *vrow = X + (D + CHUNK * (c & 1u)) * SC_PITCH;
        {          // partial sums of outputs 4 oi .. (c, then o) and columns 4 cj ..
            float acc[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
            const float *m1 = stage + warp * ROWS * 2 * CHUNK + 4 * oi;
#pragma unroll
            for (uint32_t r = 0; r < ROWS; ++r) {
                const uint32_t row = warp * ROWS + r;
                const float4 m = *reinterpret_cast<const float4 *>(m1 + r * 2 * CHUNK);
                const float4 x = *reinterpret_cast<const float4 *>((row < D ? X + row * SC_PITCH : vrow + (row - D) * SC_PITCH) + 4 * cj);
                const float mv[4] = {m.x, m.y, m.z, m.w}, xv[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = __fmaf_rn(mv[i], xv[j], acc[i][j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) *reinterpret_cast<float4 *>(part + (warp * 32 + 4 * oi + i) * SC_PITCH + 4 * cj) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        const float *m2 = stage + (D + CHUNK) * 2 * CHUNK, *crow = X + (D + 2 * CHUNK) * SC_PITCH;
        // updates s0 .. s0 + 15 of the state: v, then c
        auto update = [&](float2 (&add)[4], uint32_t kg, const float *y0, uint32_t s0) {
#pragma unroll
            for (uint32_t s = 0; s < CHUNK; ++s) {
                const float4 m = *reinterpret_cast<const float4 *>(m2 + (s0 + s) * D + 4 * kg);
                const float2 y = *reinterpret_cast<const float2 *>(y0 + s * SC_PITCH + 2 * cp);
                const float mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { add[i].x = __fmaf_rn(mv[i], y.x, add[i].x); add[i].y = __fmaf_rn(mv[i], y.y, add[i].y); }
            }
        };
        float2 add[NU][4];
#pragma unroll
        for (uint32_t u = 0; u < NU; ++u) {          // what needs no c goes on while the sums meet
            const uint32_t kg = kg0 + 32 * u;
            if (kg < KG) {
                const float4 e = *reinterpret_cast<const float4 *>(m2 + 2 * CHUNK * D + 4 * kg);
                const float ev[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) add[u][i] = make_float2(ev[i] * st[u][i].x, ev[i] * st[u][i].y);
                update(add[u], kg, vrow, 0);
            }
        }
        __syncthreads();
        {
            const uint32_t out = tid >> 3;
            float2 sum = make_float2(0.0f, 0.0f);
#pragma unroll
            for (uint32_t w = 0; w < 8; ++w) {
                const float2 p = *reinterpret_cast<const float2 *>(part + (w * 32 + out) * SC_PITCH + 2 * (tid & 7u));
                sum.x += p.x; sum.y += p.y;
            }
            if (out < CHUNK) *reinterpret_cast<float2 *>(X + (D + 2 * CHUNK + out) * SC_PITCH + 2 * (tid & 7u)) = sum;
            else if (out - CHUNK < len && c * len + out - CHUNK < n_tok) *reinterpret_cast<float2 *>(o + ((size_t)(c * len + out - CHUNK) * heads + h) * D + col0 + 2 * (tid & 7u)) = sum;
        }
        __syncthreads();
#pragma unroll
        for (uint32_t u = 0; u < NU; ++u) {
            const uint32_t kg = kg0 + 32 * u;
            if (kg < KG) {
                update(add[u], kg, crow, CHUNK);
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    st[u][i].x += add[u][i].x; st[u][i].y += add[u][i].y;
                    *reinterpret_cast<float2 *>(X + (4 * kg + i) * SC_PITCH + 2 * cp) = st[u][i];
                }
            }
        }
        if (c + 1 < chunks) ok = landed(c + 1);
        __syncthreads();                        // the stage is free
        if (tid == 0 && c + L::STAGES < chunks) request(c + L::STAGES);
    }
#pragma unroll
    for (uint32_t u = 0; u < NU; ++u) {
        const uint32_t kg = kg0 + 32 * u;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            if (kg < KG) *reinterpret_cast<float2 *>(sp + (size_t)(4 * kg + i) * D) = st[u][i];
    }
}

template <bool F32>
__global__ void __launch_bounds__(256) delta_post_kernel(const DeltaArgs a, uint32_t n_tok) {
    const uint32_t lane = threadIdx.x & 31, h = blockIdx.y, t = blockIdx.x * 8 + (threadIdx.x >> 5), dim = a.dim;
    pdl_wait();
    pdl_trigger();
    if (t >= n_tok) return;
    const float *o = a.o + ((size_t)t * a.heads + h) * a.drow, *g = a.in + t * a.in_stride + (size_t)3 * a.heads * dim + h * dim;
    float ss = 0.0f;
    for (uint32_t j = lane; j < dim; j += 32) { const float v = __ldcg(o + j); ss = __fmaf_rn(v, v, ss); }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dim + a.eps);
    for (uint32_t j = lane; j < dim; j += 32) act_store<F32>(a.out, t, h * dim + j, __ldcg(o + j) * inv * __ldg(a.norm + h * dim + j) * sigmoidf(__ldcg(g + j)));
}

// tokens of a chunk: all sixteen for decay scales up to 2.5
uint32_t chunk_len(float decay_scale) {
    const float x = 40.0f / std::fabs(decay_scale);
    return x >= 1.0f && x < (float)CHUNK ? (uint32_t)x : x < 1.0f ? 1u : CHUNK;
}

template <int D> cudaError_t scan(cudaStream_t s, const DeltaArgs &a, uint32_t n_tok, bool pdl) {
    constexpr size_t prep_smem = ((size_t)64 * (D + 4) + 32 * 36 + CHUNK + 2 * CHUNK * D) * 4;
    static_assert(ScanLayout<D>::TOTAL <= 227 * 1024, "shared memory");
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(delta_chunk_kernel<D>), prep_smem);
    if (e == cudaSuccess) e = allow_dynamic_smem(reinterpret_cast<const void *>(delta_scan_kernel<D>), ScanLayout<D>::TOTAL);
    const uint32_t len = chunk_len(a.decay_scale);
    if (e == cudaSuccess) e = launch_kernel(delta_chunk_kernel<D>, dim3((n_tok + len - 1) / len, a.heads), dim3(D), prep_smem, s, pdl, a, n_tok, len);
    if (e != cudaSuccess) return e;
    return launch_kernel(delta_scan_kernel<D>, dim3(D / CCOLS, a.heads), dim3(SC_THREADS), ScanLayout<D>::TOTAL, s, pdl, a.rec, n_tok, len, a.state, a.o, a.heads, a.err_flag);
}

}  // namespace

uint32_t delta_row(uint32_t dim) { return dim <= 256 ? (dim + 63u) & ~63u : 0u; }
size_t delta_record_floats(uint32_t n_tok, uint32_t heads, uint32_t drow, float decay_scale) {
    const uint32_t len = chunk_len(decay_scale);
    return ((size_t)n_tok + len - 1) / len * heads * chunk_floats(drow);
}
bool delta_step_fits(const DeltaArgs &a) { return step_vec_smem(a.drow, (a.rank + 63) / 64 * 64) <= 200 * 1024; }

template <bool F32, bool STAGED> static cudaError_t step_launch(cudaStream_t s, const DeltaArgs &a, size_t vec, size_t smem, bool pdl) {
    const uint32_t cs = a.drow / ST_COLS;
    auto k = a.drow == 64 ? delta_step_kernel<F32, 2, STAGED> : a.drow == 128 ? delta_step_kernel<F32, 4, STAGED> : a.drow == 192 ? delta_step_kernel<F32, 6, STAGED> : delta_step_kernel<F32, 8, STAGED>;
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(k), smem);
    return e != cudaSuccess ? e : launch_cluster(k, dim3(cs * a.heads), dim3(ST_THREADS), smem, s, pdl, cs, a, (uint32_t)vec);
}
cudaError_t launch_delta_step(cudaStream_t s, bool f32, const DeltaArgs &a, bool pdl) {
    const size_t vec = step_vec_smem(a.drow, (a.rank + 63) / 64 * 64), all = vec + (size_t)(a.dim + 8) * 128 * a.decay.panels;
    return f32 ? step_launch<true, false>(s, a, vec, vec, pdl) : all <= 200 * 1024 ? step_launch<false, true>(s, a, vec, all, pdl) : step_launch<false, false>(s, a, vec, vec, pdl);
}
cudaError_t launch_delta_tanh(cudaStream_t s, bool f32, const DeltaArgs &a, const Act &out, uint32_t n_tok, bool pdl) {
    return launch_kernel(f32 ? delta_tanh_kernel<true> : delta_tanh_kernel<false>, dim3((n_tok * a.rank + 255) / 256), dim3(256), 0, s, pdl,
                         a.in + (size_t)5 * a.heads * a.dim, a.in_stride, a.rank, n_tok, out);
}
cudaError_t launch_delta_prompt(cudaStream_t s, bool f32, const DeltaArgs &a, uint32_t n_tok, int sm_count, bool pdl) {
    const dim3 grid((n_tok + 7) / 8, a.heads);
    cudaError_t e = cudaErrorInvalidValue;
    switch (a.drow / 64) {
        case 1: e = scan<64>(s, a, n_tok, pdl); break;
        case 2: e = scan<128>(s, a, n_tok, pdl); break;
        case 3: e = scan<192>(s, a, n_tok, pdl); break;
        case 4: e = scan<256>(s, a, n_tok, pdl); break;
        default: break;
    }
    if (e != cudaSuccess) return e;
    return launch_kernel(f32 ? delta_post_kernel<true> : delta_post_kernel<false>, grid, dim3(256), 0, s, pdl, a, n_tok);
}

}  // namespace k2t
