// Sliding-window attention of the block engine (k2t_block_kernels.h): grouped queries, per-head score scale, a linear distance
// bias per head, unquantized (bf16 or fp32) key and value rows in a ring per layer.
//   * window_prep_kernel: per-head RMS norm of queries and keys of a prompt batch, cache rows, query rows (one warp per head).
//   * window_flash_kernel (bf16 prompts): CTA = 128 query rows of one kv head - row = (token, head of the group), so all heads
//     of a group share the key and value tiles.  S = Q K^T and O += P V by tcgen05.mma with S, P and O in tensor memory; scores,
//     bias and softmax in fp32, one row per thread; the next S is computed while the softmax of this one runs, and a row
//     of O is rescaled only when its own maximum has grown by more than 2^8.  Without a window the tiles of keys begin at position 0
//     and a row's bits depend on its keys alone; with one they begin at the first key that the CTA's first row sees, so that where a
//     prompt is cut moves them, and with them the last bits of a row (sums in another order).
//   * window_row_kernel: one token and kv head per thread-block cluster.  The positions are split over the CTAs of the cluster,
//     partial maxima, sums and outputs are merged through distributed shared memory, so a decode step is ONE launch: norms of
//     the new query and key, the new cache row, attention and the activation of the output projection.  With fp32 rows the same
//     kernel serves prompts (grid.z = token).
#include <algorithm>

#include "k2t_block_kernels.h"
#include "k2t_dense.cuh"
#include "k2t_flash_tc.cuh"

namespace k2t {
namespace {

constexpr uint32_t ROW_MAX = 256;

template <typename T> __device__ __forceinline__ void put(T *p, float v);
template <> __device__ __forceinline__ void put<float>(float *p, float v) { *p = v; }
template <> __device__ __forceinline__ void put<__nv_bfloat16>(__nv_bfloat16 *p, float v) { *p = __float2bfloat16_rn(v); }

// eight consecutive elements of a cached row (plain loads: the row may have been written by this CTA)
__device__ __forceinline__ void get8(const float *p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void get8(const __nv_bfloat16 *p, float (&v)[8]) {
    const uint4 a = *reinterpret_cast<const uint4 *>(p);
    v[0] = bf_lo(a.x); v[1] = bf_hi(a.x); v[2] = bf_lo(a.y); v[3] = bf_hi(a.y); v[4] = bf_lo(a.z); v[5] = bf_hi(a.z); v[6] = bf_lo(a.w); v[7] = bf_hi(a.w);
}

// one warp: dst[0 .. row) = x / rms(x) * w for dim values, zeros behind
template <typename T> __device__ __forceinline__ void norm_row(const float *x, const float *w, uint32_t dim, uint32_t row, float eps, T *dst, uint32_t lane) {
    float v[ROW_MAX / 32], ss = 0.0f;
#pragma unroll
    for (uint32_t i = 0; i < ROW_MAX / 32; ++i) {
        const uint32_t k = lane + 32 * i;
        v[i] = k < dim ? __ldcg(x + k) : 0.0f;
        ss = __fmaf_rn(v[i], v[i], ss);
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dim + eps);
#pragma unroll
    for (uint32_t i = 0; i < ROW_MAX / 32; ++i) {
        const uint32_t k = lane + 32 * i;
        if (k < row) put<T>(dst + k, k < dim ? v[i] * inv * __ldg(w + k) : 0.0f);
    }
}
template <typename T> __device__ __forceinline__ void copy_row(const float *x, uint32_t dim, uint32_t row, T *dst, uint32_t lane) {
    for (uint32_t k = lane; k < row; k += 32) put<T>(dst + k, k < dim ? __ldcg(x + k) : 0.0f);
}

struct AttnParams {
    WindowAttnArgs a;
    uint32_t n_tok, ring_rows, fused;       // ring_rows = cache rows per kv head
};

template <typename T>
__global__ void __launch_bounds__(256) window_prep_kernel(const AttnParams p) {
    const WindowAttnArgs &a = p.a;
    const uint32_t lane = threadIdx.x & 31, heads = a.n_q + 2 * a.n_kv, t = blockIdx.y, h = blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (h >= heads) return;
    const float *x = a.qkv + t * a.qkv_stride;
    const uint32_t slot = a.ring.slot_of_pos(__ldcg(a.pos) + t);
    if (h < a.n_q) {
        norm_row<T>(x + h * a.dim, a.q_norm, a.dim, a.row, a.eps, static_cast<T *>(a.q) + ((size_t)t * a.n_q + h) * a.row, lane);
    } else if (h < a.n_q + a.n_kv) {
        const uint32_t g = h - a.n_q;
        norm_row<T>(x + (a.n_q + g) * a.dim, a.k_norm, a.dim, a.row, a.eps, static_cast<T *>(a.k_cache) + ((size_t)g * p.ring_rows + slot) * a.row, lane);
    } else {
        const uint32_t g = h - a.n_q - a.n_kv;
        copy_row<T>(x + (a.n_q + a.n_kv) * a.dim + g * a.vdim, a.vdim, a.row, static_cast<T *>(a.v_cache) + ((size_t)g * p.ring_rows + slot) * a.row, lane);
    }
}

// ------------------------------------------------------------------------------------------------ one token per cluster
// The heads of a group run in passes of HB (the group is padded to full passes with zero queries), so the inner loops carry no
// branches.  Cached rows come in tiles by bulk copy (a CTA's positions are consecutive, so a tile is one run of the ring, two
// where it wraps); a decode step asks for its first tiles before its dependency wait - earlier steps wrote those rows - and lays
// the new position's row over the stale one once the tile has landed.
constexpr uint32_t RW_THREADS = 256, RW_MAX_CS = 8;
constexpr uint32_t RW_WAIT_LIMIT = 1u << 22;
// positions per tile: 64 KiB of keys (32 for long passes and fp32 rows), at most 256, a multiple of 16
template <typename T> __host__ __device__ constexpr uint32_t rw_tile(uint32_t row, uint32_t hb) {
    const uint32_t n = (hb > 4 || sizeof(T) == 4 ? 32768u : 65536u) / (row * (uint32_t)sizeof(T));
    return (n > 256u ? 256u : n) & ~15u;
}
__host__ __device__ inline uint32_t rw_pad(uint32_t group, uint32_t hb) { return (group + hb - 1) / hb * hb; }
template <typename T> inline size_t rw_smem(uint32_t group, uint32_t row, uint32_t hb) {
    const uint32_t tile = rw_tile<T>(row, hb);
    return (size_t)2 * tile * row * sizeof(T) + ((size_t)rw_pad(group, hb) * (2 * row + tile + 4 + 2 * RW_MAX_CS) + (size_t)8 * RW_THREADS * hb + 2 * row) * 4;
}

template <typename T, int D, int HB>
__global__ void __launch_bounds__(RW_THREADS) window_row_kernel(const AttnParams p) {
    extern __shared__ __align__(128) uint8_t smb[];
    __shared__ __align__(8) uint64_t bars[2];
    constexpr uint32_t TILE = rw_tile<T>(D, HB);
    const WindowAttnArgs &a = p.a;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, cs = cluster_size(), me = cluster_rank();
    const uint32_t g = blockIdx.y, t = blockIdx.z, group = a.n_q / a.n_kv, gp = rw_pad(group, HB);
    T *s_k = reinterpret_cast<T *>(smb), *s_v = s_k + TILE * D;
    float *s_q = reinterpret_cast<float *>(s_v + TILE * D), *s_o = s_q + gp * D, *s_red = s_o + gp * D, *s_new = s_red + 8 * RW_THREADS * HB, *s_p = s_new + 2 * D, *s_m = s_p + gp * TILE,
          *s_l = s_m + gp, *s_al = s_l + gp, *s_fm = s_al + 2 * gp, *s_fl = s_fm + gp * RW_MAX_CS;
    T *kc = static_cast<T *>(a.k_cache) + (size_t)g * p.ring_rows * D, *vc = static_cast<T *>(a.v_cache) + (size_t)g * p.ring_rows * D;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(bars), sk = (uint32_t)__cvta_generic_to_shared(s_k), sv = (uint32_t)__cvta_generic_to_shared(s_v);
    if (tid == 0) { mbar_init(bar, 1); mbar_init(bar + 8, 1); fence_mbar_init(); }
    if (!p.fused) { pdl_wait(); pdl_trigger(); }
    const uint32_t pos = __ldcg(a.pos) + t;                                              // a decode step's position was set before the step began
    const uint32_t n_seen = a.ring.active_len(pos + 1), lo = pos + 1 - n_seen;          // sinks are 0: the seen positions are consecutive
    const uint32_t per = (n_seen + cs - 1) / cs, j_lo = lo + min(n_seen, me * per), j_hi = lo + min(n_seen, (me + 1) * per);
    // rows of positions j0 .. of one tile; a stale row of the new position may come along
    auto request = [&](uint32_t dst, const T *cache, uint32_t j0, uint32_t b) {
        const uint32_t n = min(TILE, j_hi - j0), slot = a.ring.slot_of_pos(j0), first = min(n, p.ring_rows - slot);
        mbar_expect_tx(b, n * D * (uint32_t)sizeof(T));
        bulk_g2s(dst, cache + (size_t)slot * D, first * D * (uint32_t)sizeof(T), b);
        if (first < n) bulk_g2s(dst + first * D * (uint32_t)sizeof(T), cache, (n - first) * D * (uint32_t)sizeof(T), b);
    };
    auto landed = [&](uint32_t b, uint32_t parity) {
        bool ok = false;
        for (uint32_t spin = 0; spin < RW_WAIT_LIMIT && !ok; ++spin) ok = mbar_try_wait(b, parity);
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    };
    if (tid == 0 && j_lo < j_hi) { request(sk, kc, j_lo, bar); request(sv, vc, j_lo, bar + 8); }
    for (uint32_t i = tid; i < gp * D; i += RW_THREADS) s_o[i] = 0.0f;
    for (uint32_t i = group * D + tid; i < gp * D; i += RW_THREADS) s_q[i] = 0.0f;
    for (uint32_t i = tid; i < gp; i += RW_THREADS) { s_m[i] = -INFINITY; s_l[i] = 0.0f; s_al[i] = 0.0f; }
    const bool owner = p.fused && pos >= j_lo && pos < j_hi;          // this CTA attends to the new position and stores its rows
    if (p.fused) {
        pdl_wait();
        pdl_trigger();
        const float *x = a.qkv + t * a.qkv_stride;
        for (uint32_t h = warp; h < group + (owner ? 2u : 0u); h += RW_THREADS / 32) {
            if (h < group) norm_row<float>(x + (g * group + h) * a.dim, a.q_norm, a.dim, D, a.eps, s_q + h * D, lane);
            else if (h == group) norm_row<float>(x + (a.n_q + g) * a.dim, a.k_norm, a.dim, D, a.eps, s_new, lane);
            else copy_row<float>(x + (a.n_q + a.n_kv) * a.dim + g * a.vdim, a.vdim, D, s_new + D, lane);
        }
    } else {
        const T *qr = static_cast<const T *>(a.q) + ((size_t)t * a.n_q + g * group) * D;
        for (uint32_t i = tid * 8; i < group * D; i += RW_THREADS * 8) {
            float v[8];
            get8(qr + i, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) s_q[i + k] = v[k];
        }
    }
    __syncthreads();
    if (owner) {
        const size_t slot = (size_t)a.ring.slot_of_pos(pos) * D;
        for (uint32_t i = tid; i < D; i += RW_THREADS) { put<T>(kc + slot + i, s_new[i]); put<T>(vc + slot + i, s_new[D + i]); }
    }
    uint32_t phase = 0;
    for (uint32_t j0 = j_lo; j0 < j_hi; j0 += TILE, phase ^= 1) {
        const uint32_t n = min(TILE, j_hi - j0), j_next = j0 + TILE;
        const bool patch = owner && pos >= j0 && pos < j0 + n;
        landed(bar, phase);
        if (patch) {
            for (uint32_t i = tid; i < D; i += RW_THREADS) put<T>(s_k + (pos - j0) * D + i, s_new[i]);
            __syncthreads();
        }
        // scores: four lanes per key, sixteen keys per warp and step; neighbouring keys take their 64-byte pieces in another
        // order, so that the eight lanes of a shared-memory phase hit different banks
        const uint32_t sub = lane & 3u, ki = lane >> 2;
#pragma unroll 1
        for (uint32_t b = warp * 16; b < n; b += RW_THREADS / 2) {
            const uint32_t ja = b + ki, jb = b + 8 + ki;
            const T *ka = s_k + min(ja, n - 1) * D, *kb = s_k + min(jb, n - 1) * D;
#pragma unroll 1
            for (uint32_t h0 = 0; h0 < group; h0 += HB) {
                float da[HB], db[HB];
#pragma unroll
                for (uint32_t h = 0; h < HB; ++h) da[h] = db[h] = 0.0f;
#pragma unroll 1
                for (uint32_t c = 0; c < D / 32; ++c) {          // rolled: instruction fetch costs more than the loop
                    float va[8], vb[8];
                    const uint32_t k = (((c + (ki & 1u)) % (D / 32)) * 4 + sub) * 8;
                    get8(ka + k, va);
                    get8(kb + k, vb);
#pragma unroll
                    for (uint32_t h = 0; h < HB; ++h) {
                        const float4 q0 = *reinterpret_cast<const float4 *>(s_q + (h0 + h) * D + k), q1 = *reinterpret_cast<const float4 *>(s_q + (h0 + h) * D + k + 4);
                        const float q[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
                        for (int i = 0; i < 8; ++i) { da[h] = __fmaf_rn(q[i], va[i], da[h]); db[h] = __fmaf_rn(q[i], vb[i], db[h]); }
                    }
                }
#pragma unroll
                for (int m = 1; m < 4; m <<= 1)
#pragma unroll
                    for (uint32_t h = 0; h < HB; ++h) {
                        da[h] = __fadd_rn(da[h], __shfl_xor_sync(0xffffffffu, da[h], m));
                        db[h] = __fadd_rn(db[h], __shfl_xor_sync(0xffffffffu, db[h], m));
                    }
#pragma unroll
                for (uint32_t h = 0; h < HB; ++h)
                    if (sub == (h & 3u)) {
                        const uint32_t hh = g * group + min(h0 + h, group - 1);
                        const float sc = __ldg(a.head_scale + hh), sl = __ldg(a.head_slope + hh);
                        if (ja < n) s_p[(h0 + h) * TILE + ja] = da[h] * sc - sl * (float)(pos - (j0 + ja));
                        if (jb < n) s_p[(h0 + h) * TILE + jb] = db[h] * sc - sl * (float)(pos - (j0 + jb));
                    }
            }
        }
        __syncthreads();
        if (tid == 0 && j_next < j_hi) request(sk, kc, j_next, bar);         // everyone is done with the keys
#pragma unroll 1
        for (uint32_t h = warp; h < group; h += RW_THREADS / 32) {          // softmax terms of the tile, one warp per head
            float mx = -INFINITY;
            for (uint32_t j = lane; j < n; j += 32) mx = fmaxf(mx, s_p[h * TILE + j]);
#pragma unroll
            for (int m = 16; m > 0; m >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, m));
            const float m_old = s_m[h], m_new = fmaxf(m_old, mx);
            float sum = 0.0f;
            for (uint32_t j = lane; j < n; j += 32) { const float e = expf(s_p[h * TILE + j] - m_new); s_p[h * TILE + j] = e; sum += e; }
            sum = warp_sum(sum);
            if (lane == 0) { const float al = expf(m_old - m_new); s_al[h] = al; s_m[h] = m_new; s_l[h] = s_l[h] * al + sum; }
        }
        landed(bar + 8, phase);
        if (patch)
            for (uint32_t i = tid; i < D; i += RW_THREADS) put<T>(s_v + (pos - j0) * D + i, s_new[D + i]);
        __syncthreads();
        // values: thread = (key slice, eight columns); padding heads multiply finite leftovers that nobody reads
        constexpr uint32_t CPK = D / 8, KS = RW_THREADS / CPK;
        const uint32_t ks = tid / CPK, c = tid % CPK;
#pragma unroll 1
        for (uint32_t h0 = 0; h0 < group; h0 += HB) {
            float acc[HB][8];
#pragma unroll
            for (uint32_t h = 0; h < HB; ++h)
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[h][i] = 0.0f;
            if (ks < KS) {
#pragma unroll 2
                for (uint32_t j = ks; j < n; j += KS) {
                    float v[8];
                    get8(s_v + j * D + c * 8, v);
#pragma unroll
                    for (uint32_t h = 0; h < HB; ++h) {
                        const float e = s_p[(h0 + h) * TILE + j];
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[h][i] = __fmaf_rn(e, v[i], acc[h][i]);
                    }
                }
#pragma unroll
                for (uint32_t h = 0; h < HB; ++h) {
                    float4 *dst = reinterpret_cast<float4 *>(s_red + (ks * HB + h) * D + c * 8);
                    dst[0] = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
                    dst[1] = make_float4(acc[h][4], acc[h][5], acc[h][6], acc[h][7]);
                }
            }
            __syncthreads();
            for (uint32_t e = tid; e < HB * D; e += RW_THREADS) {
                float o = 0.0f;
#pragma unroll 8
                for (uint32_t k = 0; k < KS; ++k) o = __fadd_rn(o, s_red[k * HB * D + e]);
                s_o[h0 * D + e] = s_o[h0 * D + e] * s_al[h0 + e / D] + o;
            }
            __syncthreads();
        }
        if (tid == 0 && j_next < j_hi) request(sv, vc, j_next, bar + 8);     // everyone is done with the values
    }
    // merge over the cluster: factors of every (head, CTA), then the outputs shared out over all CTAs
    __syncthreads();
    if (cs > 1) cluster_sync_all();
    for (uint32_t i = tid; i < group * cs; i += RW_THREADS) {
        const uint32_t h = i / cs, r = i % cs;
        s_fm[h * RW_MAX_CS + r] = cs > 1 ? ld_cluster_f32(s_m + h, r) : s_m[h];
        s_fl[h * RW_MAX_CS + r] = cs > 1 ? ld_cluster_f32(s_l + h, r) : s_l[h];
    }
    __syncthreads();
    for (uint32_t h = tid; h < group; h += RW_THREADS) {
        float m = -INFINITY, l = 0.0f;
        for (uint32_t r = 0; r < cs; ++r) m = fmaxf(m, s_fm[h * RW_MAX_CS + r]);
        for (uint32_t r = 0; r < cs; ++r) { const float f = expf(s_fm[h * RW_MAX_CS + r] - m); s_fm[h * RW_MAX_CS + r] = f; l += f * s_fl[h * RW_MAX_CS + r]; }
        s_fl[h * RW_MAX_CS] = 1.0f / l;
    }
    __syncthreads();
    for (uint32_t e = me * RW_THREADS + tid; e < group * a.vdim; e += cs * RW_THREADS) {
        const uint32_t h = e / a.vdim, d = e % a.vdim;
        float o = 0.0f;
#pragma unroll
        for (uint32_t r = 0; r < RW_MAX_CS; ++r)
            if (r < cs) o = __fmaf_rn(s_fm[h * RW_MAX_CS + r], cs > 1 ? ld_cluster_f32(s_o + h * D + d, r) : s_o[h * D + d], o);
        act_store<sizeof(T) == 4>(a.out, t, (g * group + h) * a.vdim + d, o * s_fl[h * RW_MAX_CS]);
    }
    if (cs > 1) cluster_sync_all();
}

// ------------------------------------------------------------------------------------------------ prompts, bf16
constexpr uint32_t FL_M = 128, FL_LOADERS = 96, FL_THREADS = 128 + FL_LOADERS + 32, FL_HEADER = 1024, FL_TMEM = 512, FL_MARKS = 4096, FL_FEW = 32, FL_WAIT = 1u << 22;
__host__ __device__ constexpr uint32_t fl_tile(uint32_t d) { return d <= 128 ? 128 : 64; }          // keys per tile
__host__ __device__ constexpr uint32_t fl_panels(uint32_t d) { return (d + 63) / 64; }
__host__ __device__ constexpr uint32_t fl_smem(uint32_t d, uint32_t kt) { return 1024 + FL_HEADER + fl_panels(d) * 128 * (FL_M + 4 * kt); }

__device__ __forceinline__ void fl_cp16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
template <int N> __device__ __forceinline__ void fl_cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fl_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// A tile of 128 keys takes a CTA about 5000 cycles: 1050 are the tensor cores' for both products, about 1300 the issue slots of a
// softmax warp (nine instructions per key of a row).  Two softmax warps per row, half of the keys each, changed nothing (a prompt
// of 12 blocks within 3 us), so what is left is the fetch of 64 KB of keys and values per tile and the hand-offs between the roles;
// 256 rows per CTA over the same tiles would halve that fetch.  A value that is not finite would reach, as 0 x inf, all 128 rows: where
// an output is not finite the CTA goes over its tiles once more, with zeros for such values, and adds them to the rows that see them.
// The rows of the ring are row-major, so the tiles come in by
// 16-byte asynchronous copies of three warps, which put chunk c of row r at c ^ (r & 7) of its panel (the 128-byte swizzle) and
// fence them for the tensor cores; eight warps leave a softmax thread the registers for its 128 scores (nine: 168 and spills).  Keys per tile: 128, or 64 where the rows above
// 128 elements would not leave room for two tiles of keys and values.  The grid deals the rows of all kv heads in descending
// order of their contexts: a wave of 256 CTAs in ascending order left the longest to the end.
// 2048 tokens, 16 heads of 128 over 4 kv heads: 139 us with mma.sync and 64-key tiles, 45.5 now (378 TFLOP/s of causal
// work); a prompt of 12 blocks 6632 -> 6015 us, 300 tokens of 4 blocks 737 -> 648, 2 tokens behind 1000 positions 235 -> 207.
// Warps 0 .. 3: queries, softmax and output, one row per thread; warps 4 .. 6: key and value tiles; warp 7: tensor-core issue.
// Tensor memory: S of even and odd tiles (KT columns each, the softmax weights overwrite them as bf16 pairs), then O.
// A pass of the CTA over its tiles: whether an output of the thread is not finite.  AGAIN: the second one; the phases of the barriers go on, tile j is tile
// base + j of the CTA.
template <int D, uint32_t KT, bool AGAIN>
__device__ __forceinline__ bool flash_pass(const AttnParams &p, uint8_t *smem, uint32_t sbase, uint32_t tmem) {
    constexpr uint32_t PD = fl_panels(D), CH = D / 8, Q_BYTES = PD * FL_M * 128, T_BYTES = PD * KT * 128, PASS = AGAIN ? 1 : 0;
    const WindowAttnArgs &a = p.a;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = blockIdx.x, group = a.n_q / a.n_kv;
    const uint32_t rows = p.n_tok * group, r0 = (gridDim.y - 1 - blockIdx.y) * FL_M;          // the longest rows first, of all heads
    const uint32_t s_q = sbase + FL_HEADER, s_k = s_q + Q_BYTES, s_v = s_k + 2 * T_BYTES, t_o = tmem + 2 * KT;
    // barriers: queries, keys landed / free, values landed / free, S ready, weights ready, O updated, end of a pass
    const uint32_t b_q = sbase, b_kf = sbase + 8, b_ke = sbase + 24, b_vf = sbase + 40, b_ve = sbase + 56, b_s = sbase + 72, b_p = sbase + 88, b_o = sbase + 104, b_end = sbase + 112;
    volatile uint32_t *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 260);
    uint32_t *s_marked = reinterpret_cast<uint32_t *>(smem + 512);
    const uint32_t pos0 = __ldcg(a.pos), r_last = min(rows, r0 + FL_M) - 1;
    const uint32_t p_first = pos0 + r0 / group, p_last = pos0 + r_last / group;
    const uint32_t lo = p_first + 1 - a.ring.active_len(p_first + 1), n_tiles = (p_last - lo) / KT + 1, base = AGAIN ? n_tiles : 0;
    bool again = false;

    if (warp >= 4 && warp < 7) {
        const uint32_t lt = tid - 128;
        const __nv_bfloat16 *kc = static_cast<const __nv_bfloat16 *>(a.k_cache) + (size_t)g * p.ring_rows * D, *vc = static_cast<const __nv_bfloat16 *>(a.v_cache) + (size_t)g * p.ring_rows * D;
        // one tile of rows into the panels; positions beyond the last are clamped to it (masked below, rows finite)
        auto fetch = [&](const __nv_bfloat16 *src, uint32_t dst, uint32_t j) {
            const uint32_t j0 = lo + j * KT, slot0 = a.ring.slot_of_pos(j0), last = p_last - j0;
#pragma unroll 4
            for (uint32_t i = lt; i < KT * CH; i += FL_LOADERS) {
                const uint32_t r = i / CH, c = i % CH;
                uint32_t slot = slot0 + min(r, last);
                if (slot >= p.ring_rows) slot -= p.ring_rows;
                fl_cp16(dst + (c >> 3) * (KT * 128) + r * 128 + (((c & 7u) ^ (r & 7u)) << 4), src + (size_t)slot * D + c * 8);
            }
            fl_cp_commit();
        };
        // the thread's pieces of a tile of values without what is not finite; the tile is marked
        auto clean = [&](uint32_t dst, uint32_t j) {
            for (uint32_t i = lt; i < KT * CH; i += FL_LOADERS) {
                const uint32_t x = i / CH, c = i % CH, at = dst + (c >> 3) * (KT * 128) + x * 128 + (((c & 7u) ^ (x & 7u)) << 4);
                uint32_t w[4], mark = 0;
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(at));
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if ((w[k] & 0x7F80u) == 0x7F80u) { w[k] &= 0xFFFF0000u; mark = 1; }
                    if ((w[k] & 0x7F800000u) == 0x7F800000u) { w[k] &= 0x0000FFFFu; mark = 1; }
                }
                if (mark == 0) continue;
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(at), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
                atomicOr(s_marked + j % FL_MARKS / 32, 1u << (j % 32));
            }
        };
        // Every thread waits for its own copies, makes them visible to the tensor cores and announces them.  The keys of a tile are
        // announced as soon as they have landed, its values once the keys of the next tile have been requested.
        bool ok = true;
        for (uint32_t j = 0; j < n_tiles; ++j) {
            const uint32_t i = base + j, b = i & 1u;
            if (i >= 2) ok = mbar_wait_warp(b_ke + 8 * b, ((i >> 1) - 1u) & 1u, FL_WAIT, s_abort);
            if (!ok) break;
            fetch(kc, s_k + b * T_BYTES, j);
            if (j >= 1) {
                fl_cp_wait<1>();
                if (AGAIN) clean(s_v + (b ^ 1u) * T_BYTES, j - 1);
                fence_proxy_async();
                mbar_arrive(b_vf + 8 * (b ^ 1u));
            }
            fl_cp_wait<0>();
            fence_proxy_async();
            mbar_arrive(b_kf + 8 * b);
            if (i >= 2) ok = mbar_wait_warp(b_ve + 8 * b, ((i >> 1) - 1u) & 1u, FL_WAIT, s_abort);
            if (!ok) break;
            fetch(vc, s_v + b * T_BYTES, j);
        }
        fl_cp_wait<0>();                       // also after a wait that gave up: the copies land before the CTA leaves
        if (ok && AGAIN) clean(s_v + ((base + n_tiles - 1) & 1u) * T_BYTES, n_tiles - 1);
        fence_proxy_async();
        if (ok) mbar_arrive(b_vf + 8 * ((base + n_tiles - 1) & 1u));
        else if (lane == 0 && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    } else if (warp == 7) {
        if (lane == 0) {
            // fp32 accumulators, bf16 operands; A and B K-major for S, B with its columns consecutive for O
            constexpr uint32_t id_s = (1u << 4) | (1u << 7) | (1u << 10) | ((KT >> 3) << 17) | ((FL_M >> 4) << 24);
            constexpr uint32_t id_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((D >> 3) << 17) | ((FL_M >> 4) << 24);
            auto scores = [&](uint32_t i_tile) {
                const uint32_t b = i_tile & 1u, kb = s_k + b * T_BYTES;
                if (!mbar_wait_thread(b_kf + 8 * b, (i_tile >> 1) & 1u, FL_WAIT, s_abort)) return false;
                tc_fence_after();
#pragma unroll
                for (uint32_t i = 0; i < D / 16; ++i)
                    mma_ss(tmem + b * KT, desc_k(s_q + (i / 4) * FL_M * 128 + (i % 4) * 32), desc_k(kb + (i / 4) * KT * 128 + (i % 4) * 32), id_s, i != 0 ? 1u : 0u);
                tc_commit(b_s + 8 * b);
                tc_commit(b_ke + 8 * b);
                return true;
            };
            bool ok = mbar_wait_thread(b_q, 0, FL_WAIT, s_abort) && scores(base);
            for (uint32_t j = 0; j < n_tiles && ok; ++j) {
                const uint32_t i = base + j, b = i & 1u;
                if (j + 1 < n_tiles) {
                    if (i >= 1) ok = mbar_wait_thread(b_o, (i - 1) & 1u, FL_WAIT, s_abort);      // the weights of tile i - 1 lie where S of tile i + 1 goes
                    ok = ok && scores(i + 1);
                    if (!ok) break;
                }
                ok = mbar_wait_thread(b_p + 8 * b, (i >> 1) & 1u, FL_WAIT, s_abort) && mbar_wait_thread(b_vf + 8 * b, (i >> 1) & 1u, FL_WAIT, s_abort);
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (uint32_t k = 0; k < KT / 16; ++k)
                    mma_ts(t_o, tmem + b * KT + k * 8, desc_mn(s_v + b * T_BYTES + k * 16 * 128, KT * 128), id_o, (j | k) != 0 ? 1u : 0u);
                tc_commit(b_ve + 8 * b);
                tc_commit(b_o);
            }
            tc_commit(b_end);                 // also after a wait that gave up: completes when the issued products have
            mbar_arrive(b_end);               // with this thread's view of the marks
            if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
            for (uint32_t spin = 0; spin < FL_WAIT && !mbar_try_wait(b_end, PASS); ++spin) {}
        }
    } else {
        for (uint32_t i = tid; i < FL_M * CH && !AGAIN; i += 128) {          // rows beyond the last repeat it
            const uint32_t r = i / CH, c = i % CH, rr = min(r0 + r, rows - 1);
            fl_cp16(s_q + (c >> 3) * (FL_M * 128) + r * 128 + (((c & 7u) ^ (r & 7u)) << 4), static_cast<const __nv_bfloat16 *>(a.q) + ((size_t)(rr / group) * a.n_q + g * group + rr % group) * D + c * 8);
        }
        fl_cp_commit();
        const uint32_t r = r0 + tid, rr = min(r, rows - 1), t = rr / group, head = g * group + rr % group, qpos = pos0 + t, lanes = (warp * 32u) << 16;
        const uint32_t w_first = pos0 + min(r0 + warp * 32, rows - 1) / group, w_last = pos0 + min(r0 + warp * 32 + 31, rows - 1) / group;
        const uint32_t window = a.ring.window ? min(a.ring.window, 0x3fffffffu) : 0x3fffffffu;
        const float sc = __ldg(a.head_scale + head) * LOG2E, sl = __ldg(a.head_slope + head) * LOG2E;
        fl_cp_wait<0>();
        fence_proxy_async();
        if (!AGAIN) mbar_arrive(b_q);
        float m = -INFINITY, l = 0.0f;         // maximum the weights are taken against, and their sum
        bool ok = true;
        for (uint32_t j = 0; j < n_tiles; ++j) {
            const uint32_t i_tile = base + j, b = i_tile & 1u, t_s = tmem + b * KT + lanes, j0 = lo + j * KT;
            ok = mbar_wait_warp(b_s + 8 * b, (i_tile >> 1) & 1u, FL_WAIT, s_abort);
            if (!ok) break;
            tc_fence_after();
            uint32_t v[KT];
#pragma unroll
            for (int c = 0; c < (int)KT; c += 32) tm_ld32(t_s + c, v + c);
            tm_ld_wait();
            // bias of the tile's first key, the others follow in exact steps (small integers times the slope)
            const int rel = (int)(qpos - j0);
            const float f0 = (float)-rel;
#pragma unroll
            for (int c = 0; c < (int)KT; ++c) v[c] = __float_as_uint(__fmaf_rn(__uint_as_float(v[c]), sc, sl * (f0 + (float)c)));
            if (j0 + KT - 1 > w_first || w_last >= j0 + window) {            // some key of the tile is out of some row's sight
                const int from = rel - (int)window;
#pragma unroll
                for (int c = 0; c < (int)KT; ++c)
                    if (c > rel || c <= from) v[c] = 0xff800000u;
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < (int)KT; ++c) mx[c & 3] = fmaxf(mx[c & 3], __uint_as_float(v[c]));
            const float m_new = fmaxf(m, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
            if (j == 0) {
                m = m_new;
            } else if (__any_sync(0xffffffffu, m_new > m + 8.0f)) {
                ok = mbar_wait_warp(b_o, (i_tile - 1) & 1u, FL_WAIT, s_abort);
                if (!ok) break;
                tc_fence_after();
                const bool grown = m_new > m + 8.0f;          // row by row, whatever the rows beside it do
                const float al = grown ? exp2_approx(m - m_new) : 1.0f;
#pragma unroll 1
                for (uint32_t c = 0; c < D; c += 16) {
                    uint32_t o[16];
                    tm_ld16(t_o + lanes + c, o);
                    tm_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * al);
                    tm_st16(t_o + lanes + c, o);
                }
                l *= al;
                m = grown ? m_new : m;
            }
            const float mm = m == -INFINITY ? 0.0f : m;          // a row that has seen nothing yet: exp2(-inf) = 0
            float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < (int)KT; c += 2) {
                const float x = exp2_approx(__uint_as_float(v[c]) - mm), y = exp2_approx(__uint_as_float(v[c + 1]) - mm);
                sum[(c >> 1) & 3] += x + y;
                v[c >> 1] = pack_bf16(x, y);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
#pragma unroll
            for (int c = 0; c < (int)KT / 2; c += 32) {
                if constexpr (KT == 32) tm_st16(t_s, v);
                else tm_st32(t_s + c, v + c);
            }
            tm_st_wait();
            tc_fence_before();
            mbar_arrive(b_p + 8 * b);
        }
        // the last update by a barrier of its own: the phases of b_o may still be two behind here, and a parity tells only neighbours apart
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait_thread(b_end, PASS, FL_WAIT, s_abort) && *s_abort == 0);
        tc_fence_after();
        if (ok) {
            const float inv = 1.0f / l;
            float finite[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};          // NaN once an output is not finite
#pragma unroll 1
            for (uint32_t c = 0; c < D; c += 16) {
                uint32_t o[16];
                tm_ld16(t_o + lanes + c, o);
                tm_ld_wait();
                if (r < rows) {
                    float f[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) { f[i] = __uint_as_float(o[i]) * inv; finite[i & 7] = __fmaf_rn(f[i], 0.0f, finite[i & 7]); }
                    if (AGAIN) {
                        const __nv_bfloat16 *vc = static_cast<const __nv_bfloat16 *>(a.v_cache) + (size_t)g * p.ring_rows * D + c;
#pragma unroll 1
                        for (uint32_t x = lo; x <= qpos; ++x) {
                            const uint32_t j = (x - lo) / KT;
                            if ((s_marked[j % FL_MARKS / 32] >> (j % 32) & 1u) == 0) { x = lo + j * KT + KT - 1; continue; }
                            if (qpos - x >= window) continue;
                            float v[16];
                            get8(vc + (size_t)a.ring.slot_of_pos(x) * D, *reinterpret_cast<float(*)[8]>(v));
                            get8(vc + (size_t)a.ring.slot_of_pos(x) * D + 8, *reinterpret_cast<float(*)[8]>(v + 8));
#pragma unroll
                            for (int i = 0; i < 16; ++i)
                                if ((__float_as_uint(v[i]) & 0x7F800000u) == 0x7F800000u) f[i] += v[i];
                        }
                    }
                    const uint32_t k = head * a.vdim + c;
                    if (c + 16 <= a.vdim && (k & 7u) == 0) {
#pragma unroll
                        for (int i = 0; i < 16; i += 8)
                            *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(a.out.p) + panel_index(a.out.ld, t, k + i)) =
                                make_uint4(pack_bf16(f[i], f[i + 1]), pack_bf16(f[i + 2], f[i + 3]), pack_bf16(f[i + 4], f[i + 5]), pack_bf16(f[i + 6], f[i + 7]));
                    } else {
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (c + i < a.vdim) act_store<false>(a.out, t, k + i, f[i]);
                    }
                }
            }
            again = ((finite[0] + finite[1]) + (finite[2] + finite[3])) + ((finite[4] + finite[5]) + (finite[6] + finite[7])) != 0.0f;
        } else if (lane == 0 && a.err_flag != nullptr) {
            atomicExch(a.err_flag, 1u);
        }
    }
    return again;
}
template <int D, uint32_t KT> __device__ __noinline__ void flash_again(const AttnParams &p, uint8_t *smem, uint32_t sbase, uint32_t tmem) { flash_pass<D, KT, true>(p, smem, sbase, tmem); }

template <int D, uint32_t KT>
__global__ void __launch_bounds__(FL_THREADS, 1) window_flash_kernel(const __grid_constant__ AttnParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw), sbase = (raw + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (sbase - raw);
    const uint32_t b_q = sbase, b_kf = sbase + 8, b_ke = sbase + 24, b_vf = sbase + 40, b_ve = sbase + 56, b_s = sbase + 72, b_p = sbase + 88, b_o = sbase + 104, b_end = sbase + 112;
    volatile uint32_t *s_tmem = reinterpret_cast<volatile uint32_t *>(smem + 256), *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 260);
    if (tid < FL_MARKS / 32) reinterpret_cast<uint32_t *>(smem + 512)[tid] = 0;
    if (tid == 0) {
        mbar_init(b_q, 128);
        for (uint32_t i = 0; i < 2; ++i) {
            mbar_init(b_kf + 8 * i, FL_LOADERS); mbar_init(b_ke + 8 * i, 1); mbar_init(b_vf + 8 * i, FL_LOADERS); mbar_init(b_ve + 8 * i, 1);
            mbar_init(b_s + 8 * i, 1); mbar_init(b_p + 8 * i, 128);
        }
        mbar_init(b_o, 1);
        mbar_init(b_end, 2);
        *s_abort = 0;
        fence_mbar_init();
    }
    if (warp == 7) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + 256), "r"(FL_TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *s_tmem;
    pdl_wait();
    pdl_trigger();
    const bool again = flash_pass<D, KT, false>(p, smem, sbase, tmem);
    tc_fence_before();
    if (__syncthreads_or(again)) {
        tc_fence_after();
        flash_again<D, KT>(p, smem, sbase, tmem);
        tc_fence_before();
        __syncthreads();
    }
    if (warp == 7) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(FL_TMEM) : "memory");
    }
}

template <typename T, int D, int HB>
cudaError_t row_launch_hb(cudaStream_t s, const AttnParams &p, int sm_count, bool pdl) {
    const WindowAttnArgs &a = p.a;
    uint32_t cs = 1;                            // CTAs per (token, kv head): at least 64 positions each, about one wave of CTAs
    const uint32_t longest = a.ring.window ? a.ring.window : p.ring_rows;
    while (cs < RW_MAX_CS && cs * 2 * 64 <= longest && cs * 2 * a.n_kv * p.n_tok <= (uint32_t)sm_count) cs *= 2;
    const size_t smem = rw_smem<T>(a.n_q / a.n_kv, D, HB);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(window_row_kernel<T, D, HB>), smem);
    if (e != cudaSuccess) return e;
    return launch_cluster(window_row_kernel<T, D, HB>, dim3(cs, a.n_kv, p.n_tok), dim3(RW_THREADS), smem, s, pdl, cs, p);
}
inline uint32_t head_pass(bool f32, uint32_t group) { return f32 ? 4u : group == 1 ? 1u : group <= 4 ? 4u : 8u; }
template <int D>
cudaError_t row_launch(cudaStream_t s, bool f32, const AttnParams &p, int sm_count, bool pdl) {
    if (f32) return row_launch_hb<float, D, 4>(s, p, sm_count, pdl);
    switch (head_pass(false, p.a.n_q / p.a.n_kv)) {
        case 1: return row_launch_hb<__nv_bfloat16, D, 1>(s, p, sm_count, pdl);
        case 4: return row_launch_hb<__nv_bfloat16, D, 4>(s, p, sm_count, pdl);
        default: return row_launch_hb<__nv_bfloat16, D, 8>(s, p, sm_count, pdl);
    }
}
template <int D, uint32_t KT>
cudaError_t flash_launch_kt(cudaStream_t s, const AttnParams &p, bool pdl) {
    const uint32_t rows = p.n_tok * (p.a.n_q / p.a.n_kv);
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(window_flash_kernel<D, KT>), fl_smem(D, KT));
    if (e != cudaSuccess) return e;
    return launch_kernel(window_flash_kernel<D, KT>, dim3(p.a.n_kv, (rows + FL_M - 1) / FL_M), dim3(FL_THREADS), fl_smem(D, KT), s, pdl, p);
}
// Tiles of 32 keys where the batch ends by position 32: one tile either way, and a row's bits are the same (masked keys add zeros).  Both
// launches of 2 / 32 tokens from position 0: 16 heads of 64 6.0 / 6.4 us in tiles of 32, 7.6 / 8.2 in tiles of 128; 16 heads of 128 7.6 / 8.2 and 9.1 / 9.8.
template <int D>
cudaError_t flash_launch(cudaStream_t s, const AttnParams &p, bool pdl) {
    return p.a.ctx_bound != 0 && p.a.ctx_bound <= FL_FEW ? flash_launch_kt<D, FL_FEW>(s, p, pdl) : flash_launch_kt<D, fl_tile(D)>(s, p, pdl);
}

}  // namespace

uint32_t window_attn_row(uint32_t dim, uint32_t vdim) {
    const uint32_t d = std::max(dim, vdim);
    for (uint32_t c : {32u, 64u, 96u, 128u, 192u, 256u})
        if (d <= c) return c;
    return 0;
}

bool window_attn_fits(bool f32, uint32_t group, uint32_t row) { return (f32 ? rw_smem<float>(group, row, head_pass(f32, group)) : rw_smem<__nv_bfloat16>(group, row, head_pass(f32, group))) <= 224 * 1024; }

cudaError_t launch_window_attention(cudaStream_t s, bool f32, const WindowAttnArgs &a, uint32_t n_tok, int sm_count, uint32_t *launches, bool pdl) {
    AttnParams p{a, n_tok, 0, n_tok == 1 ? 1u : 0u};
    p.ring_rows = a.ring.ring_len;
    if (n_tok > 65535u || !window_attn_fits(f32, a.n_q / a.n_kv, a.row)) return cudaErrorInvalidValue;
    *launches = n_tok == 1 ? 1 : 2;
    if (n_tok > 1) {
        const dim3 grid((a.n_q + 2 * a.n_kv + 7) / 8, n_tok);
        cudaError_t e = f32 ? launch_kernel(window_prep_kernel<float>, grid, dim3(256), 0, s, pdl, p) : launch_kernel(window_prep_kernel<__nv_bfloat16>, grid, dim3(256), 0, s, pdl, p);
        if (e != cudaSuccess) return e;
    }
#define K2T_ROW(D) case D: return f32 || n_tok == 1 ? row_launch<D>(s, f32, p, sm_count, pdl) : flash_launch<D>(s, p, pdl)
    switch (a.row) {
        K2T_ROW(32);
        K2T_ROW(64);
        K2T_ROW(96);
        K2T_ROW(128);
        K2T_ROW(192);
        K2T_ROW(256);
        default: return cudaErrorInvalidValue;
    }
#undef K2T_ROW
}

}  // namespace k2t
