// Wide-batch quantized GEMM for prompts, integer dots as half-precision products on the tensor cores: the same arithmetic contract
// as k2t_gemm_tc.cu (reference batch forms src/kernels/simd_lut.rs:4228-4331, 6689-7029), bit for bit, for activations the library
// quantized itself.
//
// Weight codes and int8 activations are small integers: both are exact in fp16, a product needs at most 14 bits, and the 64
// products of a chunk sum to less than 2^21, so fp32 accumulation is exact in any order and the tensor cores hand out
// (float)dot itself.  Two things follow.  The bit-plane correction 2a - (2^B - 1) * xsum = sum (2 code - (2^B - 1)) q moves into
// the operand.  And a chain step f = fmaf(dot * xs, w_scale, f) is one multiply and one fma, which the packed forms do for two
// tokens per instruction: 1.3 instructions per (row, token, chunk) where the int32 accumulators of k2t_gemm_tc.cu take 4.75
// (integer correction, conversion, multiply, fma).
//
// Rows of 32 chunks and more go to k2t_gemm_prompt.cu where that is the faster one (gemm_prompt_takes); here are the others, the conversion of the
// activations, and the sorting of the experts' pairs.
//
// The activations come as an operand image (act_half_kernel below): per chunk 128 bytes per token in the 128-byte-swizzled
// K-major layout, so a tile of tokens is one contiguous run, plus the tokens' scales.  One CTA = 128 rows x N tokens:
//   * DECODE groups of 128 threads (thread = row) expand the row's cell of every chunk to 64 halves (A operand), from a ring
//     that `cp.async` keeps eight chunks ahead, and publish the row's weight scale;
//   * the PRODUCER thread brings the chunk's activations and scales (two bulk copies);
//   * the ISSUER thread multiplies (four tcgen05.mma kind::f16, K 16 each) into the stage's own accumulator buffer;
//   * EPILOGUE warps (lane = row, N / 4 or N / 2 tokens each) read the dots and advance their chains.
// The roles hand over two chunks at a time (a stage): half the barrier traffic of single chunks.
//
// Every wait is bounded; a wait that gives up raises the context's error word, and all roles come to their end.
// Measured (B200, 256 tokens, image included): 16384 x 2048 nf4g128 55 us against 98 us with int32 accumulators, 2048 x 8192 57 against
// 75; a 1000-token prompt through 12 layers of the 1.7B shape 21.5 -> 18.4 ms, 77 tokens through 4 layers of the 7B shape 2.09 -> 1.59 ms.
// What bounds it: issue and latency together (0.53 to 0.59 instructions per scheduler and cycle, 3000 per chunk of 128 rows x 128
// tokens and warp instruction: half of them chain steps and expansion, the rest waits and hand-overs; tensor pipe 8 to 15%).
#include <algorithm>
#include <cmath>

#include "k2t_gemm_half.cuh"

namespace k2t {

int fill_gemv_args(const DeviceMatrix &m, bool has_xsum, GemvArgs &a);      // k2t_gemv.cu

namespace {

constexpr uint32_t HF_M = 128;               // rows per CTA = UMMA M
constexpr uint32_t HF_SLOTS = 8;             // chunks whose scales (weights and activations) stay published: more than the stages in flight
constexpr uint32_t HF_WAIT_LIMIT = 1u << 21;
constexpr uint32_t HF_HEADER = 1024;
constexpr uint32_t HF_A_STAGE = HF_M * 128;

template <int N> struct HfRoles {
    static constexpr uint32_t EPI_WARPS = N >= 64 ? 16 : 8;
    static constexpr uint32_t GROUPS = N >= 64 ? 2 : 4;
    static constexpr uint32_t STAGES = N == 128 ? 2 : 3;       // a stage holds two chunks, each with an accumulator buffer of N tensor-memory columns
    static constexpr uint32_t NQ = N / (EPI_WARPS / 4);        // tokens per epilogue warp
    static constexpr uint32_t DEC_WARPS = 4 * GROUPS;
    static constexpr uint32_t THREADS = (EPI_WARPS + DEC_WARPS + 2) * 32;
    static constexpr uint32_t DEC_ARRIVALS = 8;                // decode warps that fill a stage: two groups, one per chunk
    static constexpr uint32_t TMEM = N == 32 ? 256 : 512;      // columns (a power of two)
};

template <int FMT, int N> struct HfLayout {
    static constexpr uint32_t PF = 8;          // ring slots of raw weights: chunks requested ahead
    static constexpr uint32_t PFG = PF / HfRoles<N>::GROUPS;                    // of them by one decode group
    static constexpr uint32_t A = HF_HEADER;
    static constexpr uint32_t B = A + HfRoles<N>::STAGES * 2 * HF_A_STAGE;
    static constexpr uint32_t XS = B + HfRoles<N>::STAGES * 2 * N * 128;
    static constexpr uint32_t WS = XS + HF_SLOTS * (N / 32) * HF_REC;
    static constexpr uint32_t RING = WS + HF_SLOTS * HF_M * 4;
    static constexpr uint32_t TOTAL = RING + PF * HF_M * (hf_cell<FMT>() + 4) + 1024;      // the base is rounded up to 1024 bytes
};

struct HfArgs {
    GemvArgs g;
    const uint8_t *img, *xs_img;
    const uint32_t *zero;              // image left by the kernel that quantized: not zero where any of its scales is; else null
    uint32_t n_tok, tok_pad;
};

template <int FMT, int N>
__global__ void __launch_bounds__(HfRoles<N>::THREADS, 1) gemm_f16_kernel(const HfArgs args) {
    extern __shared__ uint8_t smem_raw[];
    using R = HfRoles<N>;
    using L = HfLayout<FMT, N>;
    constexpr uint32_t EPI = R::EPI_WARPS, DEC = R::DEC_WARPS, S = R::STAGES, NQ = R::NQ, CELL = hf_cell<FMT>(), PF = L::PF;
    const GemvArgs &a = args.g;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nc = a.nc;
    const uint32_t row0 = blockIdx.x * HF_M, tok0 = blockIdx.y * N;
    const uint32_t raw = (uint32_t)__cvta_generic_to_shared(smem_raw), sbase = (raw + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (sbase - raw);
    // per stage: full (A written by a decode group, activations and scales landed), done (products in tensor memory), drained (the
    // epilogue has read them and has left the scales of earlier chunks)
    const uint32_t bar_full = sbase, bar_done = sbase + 64, bar_drained = sbase + 128, bar_last = sbase + 192;
    volatile uint32_t *s_tmem = reinterpret_cast<volatile uint32_t *>(smem + 256);
    volatile uint32_t *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 260);
    if (tid == 0) {
        for (uint32_t i = 0; i < S; ++i) { mbar_init(bar_full + 8 * i, R::DEC_ARRIVALS + 1); mbar_init(bar_done + 8 * i, 1); mbar_init(bar_drained + 8 * i, EPI); }
        mbar_init(bar_last, 1);
        *s_abort = 0;
        fence_mbar_init();
    }
    if (warp == EPI + DEC) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + 256), "r"(R::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    hf_fence_before();
    __syncthreads();
    hf_fence_after();
    const uint32_t tmem = *s_tmem;

    if (warp < EPI) {
        // ------------------------------------------------------------------ epilogue: lane = row, NQ chains
        const uint32_t quarter = warp & 3u, part = warp >> 2, row = row0 + quarter * 32 + lane;
        unsigned long long f[NQ / 2];
#pragma unroll
        for (uint32_t t = 0; t < NQ / 2; ++t) f[t] = 0;
        const uint32_t rec = (part * NQ) / 32, xs_sa = sbase + L::XS + rec * HF_REC + ((part * NQ) % 32) * 4, flag_sa = sbase + L::XS + rec * HF_REC + 128;
        // zero scales: a flag per record, or (image_ready) one word for the whole image and, where that is set, a look at the scales
        // themselves; a token behind the batch then has no scale of its own (its column is never stored)
        bool own_behind = false, all_plain = false, ready = false;
        const uint32_t xs_own = xs_sa + (lane % NQ) * 4;
        const uint32_t ws_sa = sbase + L::WS + (quarter * 32 + lane) * 4;
        const uint32_t taddr0 = tmem + ((quarter * 32u) << 16) + part * NQ;
        pdl_wait();
        own_behind = tok0 + part * NQ + lane % NQ >= args.n_tok;
        ready = args.zero != nullptr;
        all_plain = ready && __ldcg(args.zero) == 0;
        bool ok = true;
        uint32_t s = 0, ph = 0;
#pragma unroll 1
        for (uint32_t c0 = 0; c0 < nc; c0 += 2) {
            // `full` has completed by the time of `done`: waiting for it orders this thread after the scales' stores and copies
            ok = ok && mbar_wait_thread(bar_done + 8 * s, ph, HF_WAIT_LIMIT, s_abort) && mbar_wait_thread(bar_full + 8 * s, ph, HF_WAIT_LIMIT, s_abort);
            hf_fence_after();
            uint32_t ws_bits[2], any[2];          // of both chunks, requested together (a second chunk that does not exist: old ones, not used)
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k) {
                const uint32_t slot = (c0 + k) % HF_SLOTS;
                ws_bits[k] = hf_lds32(ws_sa + slot * (HF_M * 4));
                any[k] = all_plain ? 0u : hf_lds32((ready ? xs_own : flag_sa) + slot * ((N / 32) * HF_REC));
            }
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k) {
                if (c0 + k < nc) {
                    const uint32_t xo = ((c0 + k) % HF_SLOTS) * ((N / 32) * HF_REC);
                    const unsigned long long ws2 = hf_pack(ws_bits[k], ws_bits[k]);
                    bool plain = all_plain;
                    if (!plain) plain = ready ? __all_sync(0xffffffffu, own_behind || __uint_as_float(any[k]) != 0.0f) : any[k] != 0;
#pragma unroll
                    for (uint32_t h = 0; h < NQ / 16; ++h) {
                        uint32_t v[16];
                        hf_ld16(taddr0 + (2 * s + k) * N + h * 16, v);
                        if (plain) {
#pragma unroll
                            for (uint32_t t = 0; t < 16; t += 4) {
                                unsigned long long x0, x1;
                                hf_lds_pairs(xs_sa + xo + (h * 16 + t) * 4, x0, x1);
                                f[h * 8 + t / 2] = hf_step2(hf_pack(v[t], v[t + 1]), x0, ws2, f[h * 8 + t / 2]);
                                f[h * 8 + t / 2 + 1] = hf_step2(hf_pack(v[t + 2], v[t + 3]), x1, ws2, f[h * 8 + t / 2 + 1]);
                            }
                        } else {          // a token's zero scale skips its chain step (the reference skips the chunk)
#pragma unroll
                            for (uint32_t t = 0; t < 16; t += 2) {
                                const uint32_t x0 = hf_lds32(xs_sa + xo + (h * 16 + t) * 4), x1 = hf_lds32(xs_sa + xo + (h * 16 + t + 1) * 4);
                                const unsigned long long old = f[h * 8 + t / 2], r = hf_step2(hf_pack(v[t], v[t + 1]), hf_pack(x0, x1), ws2, old);
                                const uint32_t lo = __uint_as_float(x0) != 0.0f ? (uint32_t)r : (uint32_t)old, hi = __uint_as_float(x1) != 0.0f ? (uint32_t)(r >> 32) : (uint32_t)(old >> 32);
                                f[h * 8 + t / 2] = hf_pack(lo, hi);
                            }
                        }
                    }
                }
            }
            hf_fence_before();
            __syncwarp();
            if (lane == 0 && ok) hf_arrive(bar_drained + 8 * s);
            if (++s == S) { s = 0; ph ^= 1u; }
        }
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
        if (ok && row < a.rows) {
            const uint32_t t_first = tok0 + part * NQ;
            float *p = a.out + (size_t)t_first * a.out_stride + row;
#pragma unroll
            for (uint32_t t = 0; t < NQ; ++t) {
                if (t_first + t < args.n_tok) *p = __uint_as_float((t & 1u) ? (uint32_t)(f[t / 2] >> 32) : (uint32_t)f[t / 2]);
                p += a.out_stride;
            }
        }
    } else if (warp < EPI + DEC) {
        // ------------------------------------------------------------------ decode: group grp takes chunks grp, grp + GROUPS, ..; thread = row
        const uint32_t di = tid - EPI * 32, grp = di >> 7, i = di & 127u;
        const uint32_t row_c = min(row0 + i, a.rows_pad - 1);          // rows beyond the matrix repeat the last one (never stored)
        if (FMT == FMT_E8Q2) {
            uint32_t *tab = e8q2_templates_smem();
            if (di < 32) tab[di] = di < 28 ? E8Q2_TEMPLATE_WORDS[di] : 0u;
            asm volatile("bar.sync 2, %0;" ::"r"(DEC * 32) : "memory");
        }
        constexpr uint32_t B0 = Cell<FMT>::B0, B1 = Cell<FMT>::B1, B2 = Cell<FMT>::B2, SLOT = HF_M * (CELL + 4);
        const uint32_t ring = sbase + L::RING;
        const HfTables tables = hf_tables<FMT>(a);
        uint32_t p_cur = 0xffffffffu, ws_g0 = 0;
        const uint8_t *wb0 = nullptr, *wb1 = nullptr, *wb2 = nullptr, *wsb = nullptr;
        auto request = [&](uint32_t c) {          // the row's cell of chunk c and the word with its scale -> ring slot c % PF
            const uint32_t p = c >> 5;
            if (p != p_cur) {
                p_cur = p;
                const size_t r_n = (size_t)row_c * tile_chunks(nc, p);
                wb0 = a.plane[0] + tile_code_off(a.rows_pad, B0, p) + r_n * B0;
                if (B1) wb1 = a.plane[1] + tile_code_off(a.rows_pad, B1, p) + r_n * B1;
                if (B2) wb2 = a.plane[2] + tile_code_off(a.rows_pad, B2, p) + r_n * B2;
                wsb = reinterpret_cast<const uint8_t *>(a.scales) + tile_scale_off(a.rows_pad, p) + (size_t)row_c * tile_scale_pitch(nc, a.sgc, p);
                ws_g0 = scale_group_of(a, p * 32);
            }
            const uint32_t cc = c & 31u, slot = ring + (c % PF) * SLOT;
            hf_cp_async4(slot + HF_M * CELL + i * 4, wsb + (((scale_group_of(a, c) - ws_g0) * 2u) & ~3u));
            hf_cp_async16(slot + i * B0, wb0 + cc * B0);
            if (B1 == 16) hf_cp_async16(slot + HF_M * B0 + i * 16, wb1 + cc * 16);
            if (B1 == 8) hf_cp_async8(slot + HF_M * B0 + i * 8, wb1 + cc * 8);
            if (B2 == 16) hf_cp_async16(slot + HF_M * (B0 + B1) + i * 16, wb2 + cc * 16);
            if (B2 == 8) hf_cp_async8(slot + HF_M * (B0 + B1) + i * 8, wb2 + cc * 8);
        };
        // chunk `half` of the pairs pair0, pair0 + PSTEP, ..
        constexpr uint32_t PSTEP = R::GROUPS / 2;
        const uint32_t half = grp & 1u, pair0 = grp >> 1;
        for (uint32_t k = 0; k < L::PFG; ++k) {
            const uint32_t c = 2 * (pair0 + k * PSTEP) + half;
            if (c < nc) request(c);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        bool ok = true;
        uint32_t p = pair0;
#pragma unroll 1
        for (; 2 * p < nc; p += PSTEP) {
            const uint32_t s = p % S, c = 2 * p + half;
            asm volatile("cp.async.wait_group %0;" ::"n"(L::PFG - 1) : "memory");
            Raw<FMT> w;
            uint32_t ws_word;
            {
                const uint32_t slot = ring + (c % PF) * SLOT;          // nothing was requested for a chunk beyond the end: its bytes are not used
                ws_word = hf_lds32(slot + HF_M * CELL + i * 4);
                hf_lds128(slot + i * B0, w.w);
                if constexpr (B1 == 16) hf_lds128(slot + HF_M * B0 + i * 16, w.w + 4);
                if constexpr (B1 == 8) hf_lds64(slot + HF_M * B0 + i * 8, w.w[4], w.w[5]);
                if constexpr (B2 == 16) hf_lds128(slot + HF_M * (B0 + B1) + i * 16, w.w + 8);
                if constexpr (B2 == 8) hf_lds64(slot + HF_M * (B0 + B1) + i * 8, w.w[8], w.w[9]);
            }
            if (c + PF < nc) request(c + PF);          // the thread's own slot is free again
            asm volatile("cp.async.commit_group;" ::: "memory");
            uint32_t h[32];
            hf_expand<FMT>(w, tables, h);
            if (p >= S) {
                ok = mbar_wait_thread(bar_drained + 8 * s, ((p / S) - 1u) & 1u, HF_WAIT_LIMIT, s_abort);          // the products of the stage are done by then
                if (!ok) break;
            }
            if (c < nc) {
                const uint32_t dst = sbase + L::A + (2 * s + half) * HF_A_STAGE + i * 128;
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) hf_sts128(dst + ((k ^ (i & 7u)) << 4), h[4 * k], h[4 * k + 1], h[4 * k + 2], h[4 * k + 3]);
                const uint32_t g = scale_group_of(a, c) - scale_group_of(a, c & ~31u);
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(sbase + L::WS + ((c % HF_SLOTS) * HF_M + i) * 4), "r"((g & 1u) ? ws_word & 0xFFFF0000u : ws_word << 16) : "memory");
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) hf_arrive(bar_full + 8 * s);
        }
        for (; 2 * p < nc; p += PSTEP) __syncwarp();          // of a lane that has given up
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    } else if (warp == EPI + DEC) {
        if (lane == 0) {
            // ------------------------------------------------------------------ issue
            // instruction descriptor: fp32 accumulators, fp16 A and B, both K-major, N / 8, M / 16
            const uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((HF_M >> 4) << 24);
            bool ok = true;
            for (uint32_t p = 0; 2 * p < nc; ++p) {
                const uint32_t s = p % S;
                ok = mbar_wait_thread(bar_full + 8 * s, (p / S) & 1u, HF_WAIT_LIMIT, s_abort);
                if (!ok) break;
                hf_fence_after();
#pragma unroll
                for (uint32_t h = 0; h < 2; ++h) {
                    if (2 * p + h >= nc) break;
                    const uint64_t da = hf_desc(sbase + L::A + (2 * s + h) * HF_A_STAGE), db = hf_desc(sbase + L::B + (2 * s + h) * (N * 128));
#pragma unroll
                    for (uint32_t k = 0; k < 4; ++k) hf_mma(tmem + (2 * s + h) * N, da + 2 * k, db + 2 * k, idesc, k != 0 ? 1u : 0u);
                }
                hf_commit(bar_done + 8 * s);
            }
            if (!ok) {          // what was issued ends before the tensor memory is given back
                if (a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
                hf_commit(bar_last);
                for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar_last, 0u); ++spin) {}
            }
        }
    } else if (lane == 0) {
        // ------------------------------------------------------------------ activations and their scales
        constexpr uint32_t XB = (N / 32) * HF_REC;
        const uint8_t *src = args.img + (size_t)tok0 * 128, *xsrc = args.xs_img + (size_t)(tok0 / 32) * HF_REC;
        const size_t pitch = (size_t)args.tok_pad * 128, xpitch = (size_t)(args.tok_pad / 32) * HF_REC;
        pdl_wait();
        pdl_trigger();
        bool ok = true;
        uint32_t p = 0;
        for (; 2 * p < nc; ++p) {
            const uint32_t s = p % S, n = min(2u, nc - 2 * p);
            if (p >= S) {
                ok = mbar_wait_thread(bar_drained + 8 * s, ((p / S) - 1u) & 1u, HF_WAIT_LIMIT, s_abort);
                if (!ok) break;
            }
            mbar_expect_tx(bar_full + 8 * s, n * (N * 128 + XB));
            for (uint32_t h = 0; h < n; ++h) {
                const uint32_t c = 2 * p + h;
                bulk_g2s(sbase + L::B + (2 * s + h) * (N * 128), src + c * pitch, N * 128, bar_full + 8 * s);
                bulk_g2s(sbase + L::XS + (c % HF_SLOTS) * XB, xsrc + c * xpitch, XB, bar_full + 8 * s);
            }
        }
        if (!ok) {          // copies in flight land before the CTA leaves (their stages may lack decode arrivals: bounded by time)
            if (a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
            for (uint32_t k = p > S ? p - S : 0; k < p; ++k)
                for (uint32_t spin = 0; spin < 4096 && !mbar_try_wait(bar_full + 8 * (k % S), (k / S) & 1u); ++spin) {}
        }
    }
    hf_fence_before();
    __syncthreads();
    if (warp == EPI + DEC) {
        hf_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(R::TMEM) : "memory");
    }
}

// int8 activations [n_tok][cols] and their scales -> operand image and scale image.  CTA = 32 tokens x 4 chunks; thread = (token, chunk,
// half a chunk): 32 bytes in, 64 out.  Tokens beyond the batch are zeros with scale one.
__global__ void __launch_bounds__(256) act_half_kernel(const int8_t *q, const float *xs, uint32_t n_tok, uint32_t nc, uint32_t tok_pad, uint8_t *img, uint8_t *xs_img) {
    const uint32_t tid = threadIdx.x, tok0 = blockIdx.y * 32, c0 = blockIdx.x * 4;
    pdl_wait();
    pdl_trigger();
    {
        const uint32_t part = tid & 1u, ch = (tid >> 1) & 3u, c = c0 + ch, t = tok0 + (tid >> 3);
        if (c < nc) {
            uint4 v[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
            if (t < n_tok) {
                const uint4 *p = reinterpret_cast<const uint4 *>(q + ((size_t)t * nc + c) * 64 + part * 32);
                v[0] = __ldcg(p);
                v[1] = __ldcg(p + 1);
            }
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k)
                image_piece(img, tok_pad, c, t, part * 4 + k, (k & 1u) ? make_uint2(v[k >> 1].z, v[k >> 1].w) : make_uint2(v[k >> 1].x, v[k >> 1].y));
        }
    }
    if (tid < 128) {
        const uint32_t c = c0 + (tid >> 5), lane = tid & 31u, t = tok0 + lane;
        const float s = (t < n_tok && c < nc) ? __ldcg(xs + (size_t)t * nc + c) : 1.0f;
        const bool plain = __all_sync(0xffffffffu, s != 0.0f);
        if (c < nc) {
            image_scale(xs_img, tok_pad, c, t, s);
            if (lane == 0) *reinterpret_cast<uint32_t *>(xs_img + ((size_t)c * (tok_pad / 32) + blockIdx.y) * HF_REC + 128) = plain ? 1u : 0u;
        }
    }
}

// Sorts the (token, route) pairs of a batch by expert, in tiles of 32 of one expert: one CTA, two passes over the pairs.  A pair
// whose id is outside the layer's experts raises error word 4 and takes no part, nor does one whose expert another rank holds.  The
// order of an expert's pairs is free: every pair's product stands by itself.
__global__ void __launch_bounds__(1024) expert_tiles_kernel(const uint32_t *route_ids, uint32_t n_pair, uint32_t k, uint32_t route_stride, uint32_t n_experts,
                                                            const uint8_t *const *bases, uint32_t *n_tiles, uint32_t *tile_expert, uint32_t *tile_pairs, uint32_t *err_flag) {
    __shared__ uint32_t count[EXPERT_TILES_MAX_EXPERTS], first[EXPERT_TILES_MAX_EXPERTS], total;
    const uint32_t tid = threadIdx.x;
    for (uint32_t e = tid; e < n_experts; e += 1024) count[e] = 0;
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    auto expert_of = [&](uint32_t i) { return __ldcg(route_ids + (size_t)(i / k) * route_stride + i % k); };
    auto held = [&](uint32_t e) { return e < n_experts && bases[e] != nullptr; };
    for (uint32_t i = tid; i < n_pair; i += 1024) {
        const uint32_t e = expert_of(i);
        if (held(e)) atomicAdd(&count[e], 1u);
        else if (e >= n_experts && err_flag != nullptr) atomicExch(err_flag, 4u);
    }
    __syncthreads();
    if (tid < 32) {          // tiles in front of every expert's
        uint32_t run = 0;
        for (uint32_t e0 = 0; e0 < n_experts; e0 += 32) {
            const uint32_t e = e0 + tid, n = e < n_experts ? (count[e] + 31) / 32 : 0;
            uint32_t x = n;
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
                if (tid >= d) x += y;
            }
            if (e < n_experts) first[e] = run + x - n;
            run += __shfl_sync(0xffffffffu, x, 31);
        }
        if (tid == 0) { total = run; *n_tiles = run; }
    }
    __syncthreads();
    for (uint32_t i = tid; i < total * 32; i += 1024) tile_pairs[i] = HF_NO_PAIR;
    for (uint32_t e = tid; e < n_experts; e += 1024) {
        for (uint32_t j = 0; j < (count[e] + 31) / 32; ++j) tile_expert[first[e] + j] = e;
        count[e] = 0;
    }
    __syncthreads();
    for (uint32_t i = tid; i < n_pair; i += 1024) {
        const uint32_t e = expert_of(i);
        if (held(e)) tile_pairs[first[e] * 32 + atomicAdd(&count[e], 1u)] = i;
    }
}

template <int FMT, int N> cudaError_t launch_hf_n(cudaStream_t s, const HfArgs &args, bool pdl) {
    constexpr uint32_t smem = HfLayout<FMT, N>::TOTAL;
    static_assert(smem <= 227u * 1024u, "shared memory");
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(gemm_f16_kernel<FMT, N>), smem);
    if (e != cudaSuccess) return e;
    return launch_kernel(gemm_f16_kernel<FMT, N>, dim3((args.g.rows + HF_M - 1) / HF_M, (args.n_tok + N - 1) / N), dim3(HfRoles<N>::THREADS), smem, s, pdl, args);
}

template <int FMT> cudaError_t launch_hf_fmt(cudaStream_t s, const HfArgs &args, int sm_count, bool pdl) {
    const uint32_t row_tiles = (args.g.rows + HF_M - 1) / HF_M;
    // waves of the grid times a CTA's time per chunk
    auto cost = [&](uint32_t n, float t) { return (float)((row_tiles * ((args.n_tok + n - 1) / n) + sm_count - 1) / sm_count) * t; };
    const float c128 = cost(128, 1.0f), c64 = cost(64, 0.68f), c32 = cost(32, 0.5f);
    if (c128 <= c64 && c128 <= c32) return launch_hf_n<FMT, 128>(s, args, pdl);
    return c64 <= c32 ? launch_hf_n<FMT, 64>(s, args, pdl) : launch_hf_n<FMT, 32>(s, args, pdl);
}

}  // namespace

bool experts_grouped(uint32_t n_tok, uint32_t n_pair, uint32_t n_experts, uint32_t hidden, uint32_t d_ff, uint32_t bits) {
    const uint32_t min_tok = gemm_tc_min_tokens();
    if (min_tok == 0 || n_tok < min_tok || n_experts == 0 || bits < 2 || bits > 5) return false;
    // in units of a tile form's time per million weights (0.35 us)
    constexpr float START = 75.0f, PAIR[4] = {8.0f, 2.05f, 2.8f, 5.6f}, PAIR_PER_WEIGHT[4] = {0.8f, 0.326f, 0.5f, 0.73f};          // 2 .. 5 bits
    const float w = 3e-6f * (float)hidden * (float)d_ff, met = (float)n_experts * (1.0f - std::exp(-(float)n_pair / (float)n_experts));
    return (float)n_pair * std::max(PAIR[bits - 2], PAIR_PER_WEIGHT[bits - 2] * w) >= START + met * w;
}
uint32_t expert_tiles_max(size_t n_pair, uint32_t n_experts) { return (uint32_t)(n_pair / 32 + std::min<size_t>(n_pair, n_experts)); }

cudaError_t launch_expert_tiles(cudaStream_t stream, const uint32_t *route_ids, uint32_t n_tok, uint32_t k, uint32_t route_stride, uint32_t n_experts,
                                const uint8_t *const *bases, const ExpertTiles &t, uint32_t *err_flag, bool pdl) {
    if (n_experts > EXPERT_TILES_MAX_EXPERTS || expert_tiles_max((size_t)n_tok * k, n_experts) > 0xFFFFu) return cudaErrorInvalidValue;
    return launch_kernel(expert_tiles_kernel, dim3(1), dim3(1024), 0, stream, pdl, route_ids, n_tok * k, k, route_stride, n_experts, bases, t.n_tiles, t.expert, t.pairs, err_flag);
}

bool gemm_f16_takes(size_t n_tok) { return n_tok != 0 && act_half_tokens(n_tok) / 32 <= 0xFFFFu; }
bool gemm_f16_pays(uint32_t rows, uint32_t nc, size_t n_tok, int sm_count) {
    const uint32_t tile = gemm_tc_tile(rows, n_tok, sm_count);
    return tile == 64 || (tile == 32 && nc >= 16);
}
size_t act_half_bytes(size_t n_tok, uint32_t cols) { return act_half_tokens(n_tok) * cols * 2; }
size_t act_half_scale_bytes(size_t n_tok, uint32_t cols) { return act_half_tokens(n_tok) / 32 * (cols / 64) * HF_REC; }

cudaError_t launch_gemm_f16(cudaStream_t stream, const DeviceMatrix &m, const int8_t *xq, const float *xs, uint32_t n_tok, const ActHalf &h,
                            float *out, size_t out_stride, int sm_count, uint32_t *err_flag, uint32_t *launches, bool pdl, bool image_ready) {
    if (launches) *launches = 0;
    const uint32_t tok_pad = (uint32_t)act_half_tokens(n_tok);
    if (!gemm_f16_takes(n_tok) || (image_ready && h.zero == nullptr)) return cudaErrorInvalidValue;
    HfArgs args;
    const int fmt = fill_gemv_args(m, true, args.g);
    args.g.out = out; args.g.err_flag = err_flag; args.g.out_stride = out_stride;
    args.img = h.img; args.xs_img = h.scales; args.zero = image_ready ? h.zero : nullptr; args.n_tok = n_tok; args.tok_pad = tok_pad;
    cudaError_t e = image_ready ? cudaSuccess : launch_kernel(act_half_kernel, dim3((m.geom.nc + 3) / 4, tok_pad / 32), dim3(256), 0, stream, pdl, xq, xs, n_tok, m.geom.nc, tok_pad, h.img, h.scales);
    if (e != cudaSuccess) return e;
    if (gemm_prompt_takes(fmt, m.geom.rows, m.geom.nc, n_tok, sm_count)) {
        e = launch_gemm_prompt(stream, args.g, fmt, h, image_ready, n_tok, sm_count, pdl);
        if (e == cudaSuccess && launches) *launches = image_ready ? 1 : 2;
        return e;
    }
    switch (fmt) {
        case FMT_BP4: e = launch_hf_fmt<FMT_BP4>(stream, args, sm_count, pdl); break;
        case FMT_BP5: e = launch_hf_fmt<FMT_BP5>(stream, args, sm_count, pdl); break;
        case FMT_BP6: e = launch_hf_fmt<FMT_BP6>(stream, args, sm_count, pdl); break;
        case FMT_NF4: e = launch_hf_fmt<FMT_NF4>(stream, args, sm_count, pdl); break;
        case FMT_NF4G: e = launch_hf_fmt<FMT_NF4G>(stream, args, sm_count, pdl); break;
        case FMT_NF3: e = launch_hf_fmt<FMT_NF3>(stream, args, sm_count, pdl); break;
        case FMT_NF5: e = launch_hf_fmt<FMT_NF5>(stream, args, sm_count, pdl); break;
        case FMT_E8Q2: e = launch_hf_fmt<FMT_E8Q2>(stream, args, sm_count, pdl); break;
        default: return cudaErrorNotSupported;
    }
    if (e == cudaSuccess && launches) *launches = image_ready ? 1 : 2;
    return e;
}

}  // namespace k2t
