// Prompt GEMM of matrices with long rows: the arithmetic of k2t_gemm_f16.cu (exact integer dots as half-precision products, one fma chain per
// row and token in chunk order, bit for bit), organised by what bounds that kernel - the issue slots of the CUDA cores and the
// latency of every hand-over - and not by the tensor cores.
//
//   * Expanded weights go to tensor memory (tcgen05.st, thread = row) and are the A operand there: no stores of 128 bytes per row to shared
//     memory, and the products read only the activations from it (half the operand traffic).
//   * A chain warp reads its dots in the fragment shape (tcgen05.ld.16x256b): a lane has four rows and pairs of tokens, so a chunk takes 4 + NQ / 4
//     scales per lane where a lane per row takes NQ + 1 (broadcast reads of 16 bytes cost the shared-memory pipe two cycles each and were as
//     dear as the chains).
//   * One warp fetches the raw weights, four chunks of 128 rows at a time (64 consecutive bytes of a row per four lanes); a thread per
//     row fetching its own 16 bytes touches 32 lines per instruction.
//   * The issuer waits for ONE barrier per chunk; arrivals of activations are passed on to it by a warp of their own (three waits in a
//     row held it for 900 cycles a chunk: an instruction of a warp waits its turn behind busy ones).
//   * CTAs stay for several tiles: the next tile's weights are on their way while the last one is stored.
// Tiles of up to 192 tokens share one expansion (2.4 thousand warp instructions per chunk of 128 rows x 128 tokens instead of 3.0, half of
// the rest of them expansion and waits).  Measured on B200, nf4g128, image ready, k2t_gemm_f16.cu -> here: 2048 x 6144, 512 tokens
// 48.5 -> 32.5 us; 2048 x 16384 97.9 -> 82.6; 8192 x 2048 65.1 -> 59.3; b4, 77 tokens: 3584 x 37888 78.2 -> 57.7, 18944 x 3584 112.7 -> 104.1.
// Bound: 0.6 instructions per scheduler and cycle; what a chunk needs at least, packed chain steps, is a quarter of its time.  The instances of 192
// tokens spill 5 to 13 words of registers (80 a thread at launch), those of nf3, nf5 and b5 at 32 to 128 tokens 1 to 8.
// The experts of a prompt (EXP) run in the same kernel: a tile is 128 rows of one expert and up to 32 of its (token, route) pairs, which
// expert_tiles_kernel has gathered; two warps fetch the pairs' int8 rows where they lie and widen them on the way (one warp that did so
// held two CTAs an SM to a tile's chunk per 0.59 us).  2400 pairs of 128 experts, 3 bits: 1536 x 2048 202 -> 158 us, 2048 x 768 131 -> 94.
// Waits are bounded as in k2t_gemm_f16.cu.
#include <algorithm>
#include <type_traits>

#include "k2t_gemm_half.cuh"

namespace k2t {

int fill_gemv_args(const DeviceMatrix &m, bool has_xsum, GemvArgs &a);      // k2t_gemv.cu

namespace {

constexpr uint32_t GP_M = 128;               // rows per tile = UMMA M
constexpr uint32_t GP_WAIT_LIMIT = 1u << 21;
constexpr uint32_t GP_HEADER = 1024;
constexpr uint32_t GP_WS_SLOTS = 8;

// EXP: the pairs of an expert; two warps fetch and widen their activations instead of one thread that copies an image.
template <int FMT, int N, bool EXP = false> struct GpLayout {
    static constexpr uint32_t ND = N > 128 ? 2 : N > 64 ? 3 : 4;                     // accumulator buffers in tensor memory
    static constexpr uint32_t NA = 4;                                                // chunks of expanded weights there
    static constexpr uint32_t NB = N > 128 ? 4 : 6;                                  // chunks of activations in shared memory
    static constexpr uint32_t EPI = N > 128 ? 12 : 8, NG = N > 64 ? 2 : 4, DEC = 4 * NG, THREADS = (EPI + DEC + 4) * 32;          // warps: chains, expansion (groups of four)
    static constexpr uint32_t NQ = N > 128 ? 64 : N / 2;                             // tokens of a chain warp
    // registers a thread, at launch and by role
    static constexpr int R_ALL = N > 128 ? 80 : N > 64 ? 96 : 72, R_EPI = EXP ? 64 : N > 128 ? 112 : N > 64 ? 136 : 88, R_DEC = N > 128 ? 56 : N > 64 ? 80 : 72,
                         R_MISC = EXP ? 88 : N > 128 ? 32 : 40;
    static_assert(EPI * R_EPI + DEC * R_DEC + 4 * R_MISC <= (EPI + DEC + 4) * R_ALL && THREADS * R_ALL <= 65536, "registers");
    static constexpr uint32_t CELL = hf_cell<FMT>();
    static constexpr uint32_t GC = 4, NR = 4;                                        // chunks per slot of raw weights, slots
    static constexpr uint32_t TMEM = ND * N + 32 * NA <= 256 ? 256 : 512;
    static constexpr uint32_t SC_PITCH = 12;                                         // bytes of scales per row and slot
    static constexpr uint32_t XS_CHUNK = (N / 32) * HF_REC;
    static constexpr uint32_t B = GP_HEADER;
    static constexpr uint32_t XS = B + NB * N * 128;
    static constexpr uint32_t WS = XS + 2 * NB * XS_CHUNK;
    static constexpr uint32_t RAW = WS + GP_WS_SLOTS * GP_M * 8;
    static constexpr uint32_t RAW_SLOT = GP_M * (GC * CELL + SC_PITCH);
    static constexpr uint32_t TOTAL = RAW + NR * RAW_SLOT + 1024;                     // the base is rounded up to 1024 bytes
};

struct GpArgs {
    GemvArgs g;
    const uint8_t *img, *xs_img;
    const uint32_t *zero;              // image left by the kernel that quantized: not zero where any of its scales is; else null
    uint32_t n_tok, tok_pad, tok_tiles, tiles, width;          // width: tokens of a tile, a multiple of 32
};

// The pairs of a batch sorted into tiles of one expert each (k2t_gemm_f16.cu), and the experts' images.
struct GpExperts {
    GemvArgs g;                        // geometry and the first expert's planes; xq / xs = activation rows, out = one row per pair
    const uint32_t *n_tiles, *tile_expert, *tile_pairs;
    const ExpertCodebook *books;
    const uint8_t *const *bases;
    const uint8_t *base0;
    uint32_t act_group, row_tiles;     // activation row of a pair = pair / act_group
};
template <bool EXP> struct GpParam { using T = GpArgs; };
template <> struct GpParam<true> { using T = GpExperts; };

template <int R_ALL, int R> __device__ __forceinline__ void gp_registers() {
    if constexpr (R > R_ALL) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}
__device__ __forceinline__ void gp_arrive_n(uint32_t bar, uint32_t n) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(n) : "memory"); }
__device__ __forceinline__ bool gp_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
// products of 16 columns of the weights in tensor memory
__device__ __forceinline__ void gp_mma(uint32_t d, uint32_t a, uint64_t desc_b, uint32_t idesc, bool accumulate) {
    if (accumulate) asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc) : "memory");
    else asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(desc_b), "r"(idesc) : "memory");
}
__device__ __forceinline__ unsigned long long gp_lds_pair(uint32_t saddr) {
    unsigned long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(saddr));
    return v;
}
// sixteen lanes x 8 B columns: register 4 b + e of lane l is row l / 4 + 8 (e / 2), column 8 b + 2 (l % 4) + e % 2
template <int B> __device__ __forceinline__ void gp_ld(uint32_t taddr, uint32_t (&v)[4 * B]);
template <> __device__ __forceinline__ void gp_ld<1>(uint32_t taddr, uint32_t (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr + 0u) : "memory");
}
template <> __device__ __forceinline__ void gp_ld<2>(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr + 0u) : "memory");
}
template <> __device__ __forceinline__ void gp_ld<3>(uint32_t taddr, uint32_t (&v)[12]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr + 0u) : "memory");
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]) : "r"(taddr + 16u) : "memory");
}
template <> __device__ __forceinline__ void gp_ld<4>(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr + 0u) : "memory");
}
// the loaded registers are defined from here on (the loads name them as outputs, but fill them until the wait)
template <int N> __device__ __forceinline__ void gp_wait_ld(uint32_t (&v)[N]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < N; ++i) asm volatile("" : "+r"(v[i]));
}
__device__ __forceinline__ void gp_st32(uint32_t taddr, const uint32_t (&h)[32]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]), "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7]), "r"(h[8]), "r"(h[9]), "r"(h[10]), "r"(h[11]), "r"(h[12]), "r"(h[13]), "r"(h[14]), "r"(h[15]), "r"(h[16]), "r"(h[17]), "r"(h[18]), "r"(h[19]), "r"(h[20]), "r"(h[21]), "r"(h[22]), "r"(h[23]), "r"(h[24]), "r"(h[25]), "r"(h[26]), "r"(h[27]), "r"(h[28]), "r"(h[29]), "r"(h[30]), "r"(h[31]) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

template <int FMT, int N, bool EXP>
__global__ void __launch_bounds__(GpLayout<FMT, N, EXP>::THREADS, 1) gemm_prompt_kernel(const typename GpParam<EXP>::T args) {
    extern __shared__ uint8_t smem_raw[];
    using L = GpLayout<FMT, N, EXP>;
    constexpr uint32_t GP_EPI = L::EPI, GP_DEC = L::DEC, NG = L::NG, ND = L::ND, NA = L::NA, NB = L::NB, NQ = L::NQ, GC = L::GC, NR = L::NR, CELL = L::CELL, B0 = Cell<FMT>::B0, B1 = Cell<FMT>::B1, B2 = Cell<FMT>::B2;
    const GemvArgs &a = args.g;
    const uint32_t tid = threadIdx.x, hw_warp = tid >> 5, warp = hw_warp < 4 ? hw_warp + GP_EPI + GP_DEC : hw_warp - 4, lane = tid & 31, nc = a.nc;
    const uint32_t raw0 = (uint32_t)__cvta_generic_to_shared(smem_raw), sbase = (raw0 + 1023u) & ~1023u;
    uint8_t *smem = smem_raw + (sbase - raw0);
    // full: a chunk's weights are in tensor memory, its activations in shared memory and its accumulators read; done: its products are there, afree: its
    // weights have been used; bfull / bfree: activations; rfull / rfree: slots of raw weights
    const uint32_t bar_full = sbase, bar_afree = sbase + 32, bar_done = sbase + 64, bar_bfull = sbase + 96, bar_bfree = sbase + 144, bar_rfull = sbase + 192, bar_rfree = sbase + 224,
                   bar_last = sbase + 264;
    volatile uint32_t *s_tmem = reinterpret_cast<volatile uint32_t *>(smem + 256);
    volatile uint32_t *s_abort = reinterpret_cast<volatile uint32_t *>(smem + 260);
    if (tid == 0) {
        for (uint32_t i = 0; i < NA; ++i) { mbar_init(bar_full + 8 * i, 4 + GP_EPI + 1); mbar_init(bar_afree + 8 * i, 1); }
        for (uint32_t i = 0; i < ND; ++i) mbar_init(bar_done + 8 * i, 2);
        for (uint32_t i = 0; i < NB; ++i) { mbar_init(bar_bfull + 8 * i, 1); mbar_init(bar_bfree + 8 * i, 1); }
        for (uint32_t i = 0; i < NR; ++i) { mbar_init(bar_rfull + 8 * i, 32); mbar_init(bar_rfree + 8 * i, GC * 4); }
        mbar_init(bar_last, 1);
        *s_abort = 0;
        fence_mbar_init();
    }
    if (warp == GP_EPI + GP_DEC) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + 256), "r"(L::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (FMT == FMT_E8Q2 && tid < 32) e8q2_templates_smem()[tid] = tid < 28 ? E8Q2_TEMPLATE_WORDS[tid] : 0u;
    hf_fence_before();
    __syncthreads();
    hf_fence_after();
    const uint32_t tmem = *s_tmem, tmem_a = tmem + ND * N;
    uint32_t tiles;
    if constexpr (EXP) {          // the routes are the predecessor's: nothing can be requested before
        pdl_wait();
        tiles = __ldcg(args.n_tiles) * args.row_tiles;
    } else {
        tiles = args.tiles;
    }
    const uint32_t my_tiles = tiles > blockIdx.x ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0u, total = my_tiles * nc;
    auto first_row = [&](uint32_t tile) {
        if constexpr (EXP) return tile % args.row_tiles * GP_M;
        else return tile / args.tok_tiles * GP_M;
    };

    if (warp < GP_EPI) {
        gp_registers<L::R_ALL, L::R_EPI>();
        // ------------------------------------------------------------------ chains: lane = four rows (8 apart), NQ / 8 blocks of two tokens
        constexpr uint32_t NBLK = NQ / 8;
        const uint32_t quarter = warp & 3u, part = warp >> 2;
        if constexpr (!EXP) pdl_wait();
        uint32_t xs_at[NBLK];
#pragma unroll
        for (uint32_t b = 0; b < NBLK; ++b) {
            const uint32_t t = part * NQ + 8 * b + 2 * (lane & 3u);
            xs_at[b] = sbase + L::XS + (t / 32) * HF_REC + (t % 32) * 4;
        }
        const uint32_t ws_at = sbase + L::WS + (quarter * 32 + (lane >> 2) * 4) * 8;
        bool ok = true;
        uint32_t s8 = 0, ph = 0, f8 = (ND % NA) * 8, xo = 0, wo = 0, ta = tmem + ((quarter * 32u) << 16) + part * NQ;
        if (lane == 0)
            for (uint32_t i = 0; i < ND; ++i) hf_arrive(bar_full + 8 * (i % NA));          // nothing to read there yet
        auto run = [&](auto plain_image) {
            constexpr bool PLAIN = decltype(plain_image)::value;
#pragma unroll 1
            for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
                const uint32_t row0 = first_row(tile);
                uint32_t tok0 = 0, end = 0;
                bool live;          // any token of the warp
                const uint32_t *pairs = nullptr;
                if constexpr (EXP) {
                    pairs = args.tile_pairs + tile / args.row_tiles * N + part * NQ;
                    live = __ldcg(pairs) != HF_NO_PAIR;          // they fill their tile from the front
                } else {
                    tok0 = (tile % args.tok_tiles) * args.width; end = min(args.n_tok, tok0 + args.width);
                    live = tok0 + part * NQ < end;
                }
                unsigned long long f[4][NBLK];
#pragma unroll
                for (uint32_t r = 0; r < 4; ++r)
#pragma unroll
                    for (uint32_t b = 0; b < NBLK; ++b) f[r][b] = 0;
#pragma unroll 1
                for (uint32_t c = 0; c < nc; ++c) {
                    ok = ok && mbar_wait_thread(bar_done + s8, ph, GP_WAIT_LIMIT, s_abort);
                    hf_fence_after();
                    if (live) {
                        // pieces of PB blocks of sixteen lanes; with two buffers the next one is on its way while one is worked on
                        constexpr uint32_t PB = NBLK > 4 ? NBLK / 2 : NBLK, PIECES = 2 * NBLK / PB, BUF = L::R_EPI > 112 ? 2 : 1;
                        unsigned long long ws[4], xs[PB];
                        hf_lds_pairs(ws_at + wo, ws[0], ws[1]);
                        hf_lds_pairs(ws_at + wo + 16, ws[2], ws[3]);
                        uint32_t v[BUF][4 * PB];
                        auto at = [&](uint32_t p) { return ta + ((p & 1u) * 16u << 16) + (p >> 1) * PB * 8; };
                        gp_ld<PB>(at(0), v[0]);
                        bool plain = true;
#pragma unroll
                        for (uint32_t p = 0; p < PIECES; ++p) {
                            const uint32_t hr = p & 1u, b0 = (p >> 1) * PB;
                            if ((p & 1u) == 0) {
#pragma unroll
                                for (uint32_t b = 0; b < PB; ++b) xs[b] = gp_lds_pair(xs_at[b0 + b] + xo);
                                if constexpr (!PLAIN) {
                                    plain = true;
#pragma unroll
                                    for (uint32_t b = 0; b < PB; ++b) plain = plain && __uint_as_float((uint32_t)xs[b]) != 0.0f && __uint_as_float((uint32_t)(xs[b] >> 32)) != 0.0f;
                                    plain = __all_sync(0xffffffffu, plain);
                                }
                            }
                            gp_wait_ld(v[p % BUF]);
                            if (BUF == 2 && p + 1 < PIECES) gp_ld<PB>(at(p + 1), v[(p + 1) % BUF]);
                            if (PLAIN || plain) {
#pragma unroll
                                for (uint32_t b = 0; b < PB; ++b) {
                                    const uint32_t *d = v[p % BUF] + 4 * b;
                                    f[2 * hr][b0 + b] = hf_step2(hf_pack(d[0], d[1]), xs[b], ws[2 * hr], f[2 * hr][b0 + b]);
                                    f[2 * hr + 1][b0 + b] = hf_step2(hf_pack(d[2], d[3]), xs[b], ws[2 * hr + 1], f[2 * hr + 1][b0 + b]);
                                }
                            } else {          // a token's zero scale skips its chain step (the reference skips the chunk)
#pragma unroll
                                for (uint32_t b = 0; b < PB; ++b) {
                                    const uint32_t *d = v[p % BUF] + 4 * b;
                                    unsigned long long &f0 = f[2 * hr][b0 + b], &f1 = f[2 * hr + 1][b0 + b];
                                    const bool zx = __uint_as_float((uint32_t)xs[b]) == 0.0f, zy = __uint_as_float((uint32_t)(xs[b] >> 32)) == 0.0f;
                                    const unsigned long long r0 = hf_step2(hf_pack(d[0], d[1]), xs[b], ws[2 * hr], f0), r1 = hf_step2(hf_pack(d[2], d[3]), xs[b], ws[2 * hr + 1], f1);
                                    f0 = hf_pack(zx ? (uint32_t)f0 : (uint32_t)r0, zy ? (uint32_t)(f0 >> 32) : (uint32_t)(r0 >> 32));
                                    f1 = hf_pack(zx ? (uint32_t)f1 : (uint32_t)r1, zy ? (uint32_t)(f1 >> 32) : (uint32_t)(r1 >> 32));
                                }
                            }
                            if (BUF == 1 && p + 1 < PIECES) gp_ld<PB>(at(p + 1), v[0]);
                        }
                    }
                    hf_fence_before();
                    __syncwarp();
                    if (lane == 0 && ok) hf_arrive(bar_full + f8);          // the buffer is free for the chunk ND further on
                    s8 += 8; ta += N;
                    if (s8 == 8 * ND) { s8 = 0; ta -= ND * N; ph ^= 1u; }
                    f8 = (f8 + 8) & (8 * NA - 1);
                    xo += L::XS_CHUNK;
                    if (xo == 2 * NB * L::XS_CHUNK) xo = 0;
                    wo = (wo + GP_M * 8) & (GP_WS_SLOTS * GP_M * 8 - 1);
                }
                if constexpr (EXP) {
                    if (ok && live) {
#pragma unroll
                        for (uint32_t b = 0; b < NBLK; ++b) {
                            const uint2 pair = __ldcg(reinterpret_cast<const uint2 *>(pairs + 8 * b + 2 * (lane & 3u)));
#pragma unroll
                            for (uint32_t r = 0; r < 4; ++r) {
                                const uint32_t row = row0 + quarter * 32 + (lane >> 2) + 8 * r;
                                if (row < a.rows && pair.x != HF_NO_PAIR) a.out[(size_t)pair.x * a.out_stride + row] = __uint_as_float((uint32_t)f[r][b]);
                                if (row < a.rows && pair.y != HF_NO_PAIR) a.out[(size_t)pair.y * a.out_stride + row] = __uint_as_float((uint32_t)(f[r][b] >> 32));
                            }
                        }
                    }
                } else if (ok) {
#pragma unroll
                    for (uint32_t r = 0; r < 4; ++r) {
                        const uint32_t row = row0 + quarter * 32 + (lane >> 2) + 8 * r;
                        if (row < a.rows) {
#pragma unroll
                            for (uint32_t b = 0; b < NBLK; ++b) {
                                const uint32_t tok = tok0 + part * NQ + 8 * b + 2 * (lane & 3u);
                                float *o = a.out + (size_t)tok * a.out_stride + row;
                                if (tok < end) o[0] = __uint_as_float((uint32_t)f[r][b]);
                                if (tok + 1 < end) o[a.out_stride] = __uint_as_float((uint32_t)(f[r][b] >> 32));
                            }
                        }
                    }
                }
            }
        };
        if constexpr (EXP) run(std::false_type{});
        else if (args.zero != nullptr && __ldcg(args.zero) == 0) run(std::true_type{});
        else run(std::false_type{});
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    } else if (warp < GP_EPI + GP_DEC) {
        gp_registers<L::R_ALL, L::R_DEC>();
        // ------------------------------------------------------------------ expansion: groups of four warps, chunk by chunk in turn; thread = row
        const uint32_t di = (warp - GP_EPI) * 32 + lane, grp = di >> 7, row = di & 127u, quarter = row >> 5;
        HfTables tables;
        auto table_of = [&](uint32_t tile) {
            if constexpr (EXP) { if (tile < tiles) tables = hf_tables<FMT>(args.books[__ldcg(args.tile_expert + tile / args.row_tiles)]); }
        };
        if constexpr (EXP) table_of(blockIdx.x);
        else tables = hf_tables<FMT>(a);
        const uint32_t ta = tmem_a + ((quarter * 32u) << 16), sw = (row >> 1) & (GC - 1), sw8 = ((row >> 2) & 1u) * 16, spt = (nc + GC - 1) / GC;
        // the four rows of an epilogue lane side by side, each scale twice
        const uint32_t ws_at = sbase + L::WS + (quarter * 32 + (lane & 7u) * 4 + (lane >> 3)) * 8;
        bool ok = true;
        uint32_t tile = blockIdx.x, c = grp, base = 0, s = grp, ph = 1;          // chunk in its tile, raw slots of the tiles before, weight buffer and its phase
#pragma unroll 1
        for (uint32_t i = grp; i < total; i += NG, c += NG) {
            if (c >= nc) {
                while (c >= nc) { c -= nc; base += spt; tile += gridDim.x; }
                table_of(tile);
            }
            const uint32_t cc = c % GC, slot_n = base + c / GC, slot = slot_n % NR, rs = sbase + L::RAW + slot * L::RAW_SLOT;
            ok = ok && mbar_wait_thread(bar_rfull + 8 * slot, (slot_n / NR) & 1u, GP_WAIT_LIMIT, s_abort);
            Raw<FMT> w;
            hf_lds128(rs + row * (GC * B0) + ((cc ^ sw) * 16), w.w);
            if constexpr (B1 == 16) hf_lds128(rs + GP_M * GC * B0 + row * (GC * 16) + ((cc ^ sw) * 16), w.w + 4);
            if constexpr (B1 == 8) hf_lds64(rs + GP_M * GC * B0 + row * (GC * 8) + (cc * 8 ^ sw8), w.w[4], w.w[5]);
            if constexpr (B2 == 16) hf_lds128(rs + GP_M * GC * (B0 + B1) + row * (GC * 16) + ((cc ^ sw) * 16), w.w + 8);
            if constexpr (B2 == 8) hf_lds64(rs + GP_M * GC * (B0 + B1) + row * (GC * 8) + (cc * 8 ^ sw8), w.w[8], w.w[9]);
            // scale groups counted from the pass on; the slot's words begin with an even one
            const uint32_t g0 = scale_group_of(a, c & ~31u), g = scale_group_of(a, c) - g0, gs = (scale_group_of(a, c - cc) - g0) & ~1u;
            const uint32_t ws_word = hf_lds32(rs + GP_M * GC * CELL + row * L::SC_PITCH + (((g - gs) * 2) & ~3u));
            uint32_t h[32];
            if (L::R_DEC >= 72) hf_expand<FMT>(w, tables, h);          // where registers hold a whole cell it is ready before the buffer is
            if (i >= NA) ok = ok && mbar_wait_thread(bar_afree + 8 * s, ph, GP_WAIT_LIMIT, s_abort);
            hf_fence_after();
            if (L::R_DEC < 72) hf_expand<FMT>(w, tables, h);
            gp_st32(ta + s * 32, h);
            const uint32_t ws = (g & 1u) ? ws_word & 0xFFFF0000u : ws_word << 16;
            asm volatile("st.shared.v2.u32 [%0], {%1, %1};" ::"r"(ws_at + (i % GP_WS_SLOTS) * (GP_M * 8)), "r"(ws) : "memory");
            hf_fence_before();
            __syncwarp();
            if (lane == 0 && ok) {
                hf_arrive(bar_full + 8 * s);
                gp_arrive_n(bar_rfree + 8 * slot, c + 1 == nc ? GC - cc : 1);          // the last chunk of a tile also stands for those its slot does not hold
            }
            s += NG;
            if (s >= NA) { s -= NA; ph ^= 1u; }
        }
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    } else {
    gp_registers<L::R_ALL, L::R_MISC>();
    if (warp == GP_EPI + GP_DEC) {
        // ------------------------------------------------------------------ products
        uint32_t width = N;
        if constexpr (!EXP) width = args.width;
        const uint32_t idesc = (1u << 4) | ((width >> 3) << 17) | ((GP_M >> 4) << 24);
        const uint64_t db0 = hf_desc(sbase + L::B);
        bool ok = true;
        uint32_t s = 0, ph = 0, b = 0, d = 0;
#pragma unroll 1
        for (uint32_t i = 0; i < total; ++i) {
            ok = mbar_wait_warp(bar_full + 8 * s, ph, GP_WAIT_LIMIT, s_abort);
            if (!ok) break;
            hf_fence_after();
            if (gp_elect()) {
                const uint64_t db = db0 + (uint64_t)(b * (N * 128 / 16));
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) gp_mma(tmem + d * N, tmem_a + s * 32 + 8 * k, db + 2 * k, idesc, k != 0);
                hf_commit(bar_bfree + 8 * b);
                hf_commit(bar_afree + 8 * s);
                hf_commit(bar_done + 8 * d);
                hf_arrive(bar_done + 8 * d);          // with this thread's view of the scales: whoever sees the products sees them
            }
            __syncwarp();
            if (++s == NA) { s = 0; ph ^= 1u; }
            if (++d == ND) d = 0;
            if (++b == NB) b = 0;
        }
        if (!ok && lane == 0 && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
        if (gp_elect()) {          // what this thread issued ends before the tensor memory is given back, whichever role gave up
            hf_commit(bar_last);
            for (uint32_t spin = 0; spin < WAIT_LIMIT && !mbar_try_wait(bar_last, 0u); ++spin) {}
        }
        __syncwarp();
    } else if (warp == GP_EPI + GP_DEC + 1 || (EXP && warp == GP_EPI + GP_DEC + 3)) {
        if constexpr (EXP) {
            // ------------------------------------------------------------------ activations of the tile's pairs, widened on the way, the two warps chunk by chunk in
            // turn: eight tokens x four 16-byte pieces per load, the next chunk's values on their way
            const uint32_t piece = lane & 3u, r8 = lane >> 2, turn = warp == GP_EPI + GP_DEC + 1 ? 0u : 1u;
            if (turn == 0 && lane == 0) pdl_trigger();
            const __half2 add = __half2half2(__int2half_rn(-1152));
            const float *xs = nullptr;
            const uint8_t *xq[4];
            auto rows_of = [&](uint32_t tile) {
                const uint32_t own = tile < tiles ? __ldcg(args.tile_pairs + tile / args.row_tiles * N + lane) : HF_NO_PAIR;
                xs = own == HF_NO_PAIR ? nullptr : a.xs + (size_t)(own / args.act_group) * nc;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t pair = __shfl_sync(0xffffffffu, own, j * 8 + r8);
                    xq[j] = pair == HF_NO_PAIR ? nullptr : reinterpret_cast<const uint8_t *>(a.xq) + (size_t)(pair / args.act_group) * a.cols + piece * 16;
                }
            };
            uint4 v[4];
            float sc = 1.0f;
            auto load = [&](uint32_t c) {
                sc = xs != nullptr ? __ldcg(xs + c) : 1.0f;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) v[j] = xq[j] != nullptr ? __ldcg(reinterpret_cast<const uint4 *>(xq[j] + (size_t)c * 64)) : make_uint4(0, 0, 0, 0);
            };
            uint32_t tile = blockIdx.x, c = turn;
            auto settle = [&]() {          // the chunk's tile
                if (c < nc) return;
                while (c >= nc) { c -= nc; tile += gridDim.x; }
                rows_of(tile);
            };
            rows_of(tile);
            settle();
            if (turn < total) load(c);
            bool ok = true;
            for (uint32_t i = turn; i < total; i += 2) {
                const uint32_t b = i % NB, s = i % NA;
                // the products that read the slot are done; a buffer's arrivals belong to one chunk
                if (i >= NB) ok = ok && mbar_wait_thread(bar_bfree + 8 * b, (i / NB - 1u) & 1u, GP_WAIT_LIMIT, s_abort);
                if (i >= NA) ok = ok && mbar_wait_thread(bar_full + 8 * s, (i / NA - 1u) & 1u, GP_WAIT_LIMIT, s_abort);
                const uint32_t dst = sbase + L::B + b * (N * 128);
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const uint32_t t = j * 8 + r8;
                    uint32_t o[8];
                    hf_widen(v[j].x ^ 0x80808080u, add, o[0], o[1]);
                    hf_widen(v[j].y ^ 0x80808080u, add, o[2], o[3]);
                    hf_widen(v[j].z ^ 0x80808080u, add, o[4], o[5]);
                    hf_widen(v[j].w ^ 0x80808080u, add, o[6], o[7]);
                    hf_sts128(dst + t * 128 + (((2 * piece) ^ (t & 7u)) << 4), o[0], o[1], o[2], o[3]);
                    hf_sts128(dst + t * 128 + (((2 * piece + 1) ^ (t & 7u)) << 4), o[4], o[5], o[6], o[7]);
                }
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(sbase + L::XS + (i % (2 * NB)) * L::XS_CHUNK + lane * 4), "f"(sc) : "memory");
                c += 2;
                settle();
                if (i + 2 < total) load(c);
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && ok) hf_arrive(bar_full + 8 * s);
            }
            if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
        } else if (lane == 0) {
            // ------------------------------------------------------------------ activations and their scales
            const size_t pitch = (size_t)args.tok_pad * 128, xpitch = (size_t)(args.tok_pad / 32) * HF_REC;
            pdl_wait();
            pdl_trigger();
            bool ok = true;
            uint32_t i = 0, b = 0, ph = 1, xsl = 0;
            for (uint32_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
                const uint32_t tok0 = (tile % args.tok_tiles) * args.width, x0 = tok0 % 32, bytes = min(args.width, (args.n_tok - tok0 + 7u) & ~7u) * 128;          // whole groups of eight tokens; what lies behind is not stored
                const uint32_t xbytes = (x0 + bytes / 128 + 31) / 32 * HF_REC;
                const uint8_t *src = args.img + (size_t)tok0 * 128, *xsrc = args.xs_img + (size_t)(tok0 / 32) * HF_REC;
                for (uint32_t c = 0; c < nc; ++c, ++i) {
                    if (i >= NB) {          // the products that read the slot are done
                        ok = mbar_wait_thread(bar_bfree + 8 * b, ph, GP_WAIT_LIMIT, s_abort);
                        if (!ok) break;
                    }
                    mbar_expect_tx(bar_bfull + 8 * b, bytes + xbytes);
                    bulk_g2s(sbase + L::B + b * (N * 128), src, bytes, bar_bfull + 8 * b);
                    bulk_g2s(sbase + L::XS + xsl * L::XS_CHUNK, xsrc, xbytes, bar_bfull + 8 * b);
                    src += pitch; xsrc += xpitch;
                    if (++b == NB) { b = 0; ph ^= 1u; }
                    if (++xsl == 2 * NB) xsl = 0;
                }
            }
            if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
            for (uint32_t k = i > NB ? i - NB : 0; k < i; ++k)          // copies in flight land before the CTA leaves, whichever role gave up
                for (uint32_t spin = 0; spin < GP_WAIT_LIMIT && !mbar_try_wait(bar_bfull + 8 * (k % NB), (k / NB) & 1u); ++spin) {}
        }
    } else if (warp == GP_EPI + GP_DEC + 2) {
        // ------------------------------------------------------------------ raw weights, GC chunks of 128 rows at a time: GC lanes a row
        const uint32_t j = lane % GC, r8 = lane / GC;
        constexpr uint32_t STEP = 32 / GC;          // rows of a copy: eight, so that a lane's swizzle is the same in all of them
        const uint32_t d16 = r8 * GC * 16 + (j ^ ((r8 >> 1) & (GC - 1))) * 16;          // the lane's place among 16-byte pieces
        const uint32_t e8 = r8 * GC * 8 + (j * 8 ^ ((r8 >> 2) & 1u) * 16);              // among 8-byte pieces
        const uint32_t j2 = lane & 1u, r16 = lane >> 1, d8 = r16 * GC * 8 + (j2 ^ ((r16 >> 2) & 1u)) * 16;          // among pairs of them
        bool ok = true;
        uint32_t n_slot = 0;
        for (uint32_t tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
            const uint32_t row0 = first_row(tile);
            ptrdiff_t image = 0;          // this expert's image behind the first one's
            if constexpr (EXP) image = args.bases[__ldcg(args.tile_expert + tile / args.row_tiles)] - args.base0;
            for (uint32_t c0 = 0; c0 < nc; c0 += GC, ++n_slot) {
                const uint32_t slot = n_slot % NR, rs = sbase + L::RAW + slot * L::RAW_SLOT;
                if (n_slot >= NR) {
                    ok = mbar_wait_warp(bar_rfree + 8 * slot, (n_slot / NR - 1u) & 1u, GP_WAIT_LIMIT, s_abort);
                    if (!ok) break;
                }
                const uint32_t p = c0 >> 5, n = tile_chunks(nc, p), cc = (c0 & 31u) + j;
                if (n == 32 && row0 + GP_M <= a.rows_pad) {          // a full pass: the strides are constants, and pairs of 8-byte pieces lie on 16 bytes
                    const uint8_t *p0 = a.plane[0] + image + tile_code_off(a.rows_pad, B0, p) + (size_t)(row0 + r8) * (32 * B0) + cc * B0;
                    const uint8_t *p1 = a.plane[1] + image + tile_code_off(a.rows_pad, B1, p) + (size_t)(row0 + (B1 == 8 ? r16 : r8)) * (32 * B1) + (B1 == 8 ? (c0 & 31u) * 8 + j2 * 16 : cc * B1);
                    const uint8_t *p2 = a.plane[2] + image + tile_code_off(a.rows_pad, B2, p) + (size_t)(row0 + (B2 == 8 ? r16 : r8)) * (32 * B2) + (B2 == 8 ? (c0 & 31u) * 8 + j2 * 16 : cc * B2);
#pragma unroll
                    for (uint32_t r = 0; r < GP_M; r += STEP) {
                        hf_cp_async16(rs + d16 + r * GC * B0, p0 + r * 32 * B0);
                        if (B1 == 16) hf_cp_async16(rs + GP_M * GC * B0 + d16 + r * GC * 16, p1 + r * 32 * 16);
                        if (B2 == 16) hf_cp_async16(rs + GP_M * GC * (B0 + B1) + d16 + r * GC * 16, p2 + r * 32 * 16);
                    }
                    if (B1 == 8 || B2 == 8) {
#pragma unroll
                        for (uint32_t r = 0; r < GP_M; r += 16) {
                            if (B1 == 8) hf_cp_async16(rs + GP_M * GC * B0 + d8 + r * GC * 8, p1 + r * 32 * 8);
                            if (B2 == 8) hf_cp_async16(rs + GP_M * GC * (B0 + B1) + d8 + r * GC * 8, p2 + r * 32 * 8);
                        }
                    }
                } else if (cc < n) {
                    const uint8_t *p0 = a.plane[0] + image + tile_code_off(a.rows_pad, B0, p) + cc * B0, *p1 = a.plane[1] + image + tile_code_off(a.rows_pad, B1, p) + cc * B1,
                                  *p2 = a.plane[2] + image + tile_code_off(a.rows_pad, B2, p) + cc * B2;
                    auto row = [&](uint32_t r, const uint8_t *q0, const uint8_t *q1, const uint8_t *q2) {
                        hf_cp_async16(rs + d16 + r * GC * B0, q0);
                        if (B1 == 16) hf_cp_async16(rs + GP_M * GC * B0 + d16 + r * GC * 16, q1);
                        if (B1 == 8) hf_cp_async8(rs + GP_M * GC * B0 + e8 + r * GC * 8, q1);
                        if (B2 == 16) hf_cp_async16(rs + GP_M * GC * (B0 + B1) + d16 + r * GC * 16, q2);
                        if (B2 == 8) hf_cp_async8(rs + GP_M * GC * (B0 + B1) + e8 + r * GC * 8, q2);
                    };
                    if (EXP && row0 + GP_M <= a.rows_pad) {
                        const size_t at = (size_t)(row0 + r8) * n;
                        const uint32_t step = STEP * n;
                        p0 += at * B0; p1 += at * B1; p2 += at * B2;
#pragma unroll
                        for (uint32_t r = 0; r < GP_M; r += STEP) {
                            row(r, p0, p1, p2);
                            p0 += step * B0; p1 += step * B1; p2 += step * B2;
                        }
                    } else
#pragma unroll 2
                    for (uint32_t r = 0; r < GP_M; r += STEP) {          // rows beyond the matrix repeat the last one (never stored)
                        const size_t at = (size_t)min(row0 + r8 + r, a.rows_pad - 1) * n;
                        row(r, p0 + at * B0, p1 + at * B1, p2 + at * B2);
                    }
                }
                {          // the words that hold the scales of these chunks
                    const uint32_t g0 = scale_group_of(a, p * 32), off0 = ((scale_group_of(a, c0) - g0) * 2u) & ~3u;
                    const uint32_t last = min(c0 + GC, nc) - 1, words = ((scale_group_of(a, last) - g0) * 2u - off0) / 4u + 1u, pitch = tile_scale_pitch(nc, a.sgc, p);
                    const uint8_t *src = reinterpret_cast<const uint8_t *>(a.scales) + image + tile_scale_off(a.rows_pad, p) + off0;
#pragma unroll
                    for (uint32_t r = lane; r < GP_M; r += 32) {
                        const uint8_t *q = src + (size_t)min(row0 + r, a.rows_pad - 1) * pitch;
                        const uint32_t d = rs + GP_M * GC * CELL + r * L::SC_PITCH;
                        for (uint32_t w = 0; w < words; ++w) hf_cp_async4(d + 4 * w, q + 4 * w);
                    }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_rfull + 8 * slot) : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok && lane == 0 && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    } else if (lane == 0) {
        // ------------------------------------------------------------------ activations have landed: said where the issuer waits
        bool ok = true;
        uint32_t s = 0, sph = 1, b = 0, ph = 0;
        for (uint32_t i = 0; i < total; ++i) {
            ok = mbar_wait_thread(bar_bfull + 8 * b, ph, GP_WAIT_LIMIT, s_abort) && (i < NA || mbar_wait_thread(bar_full + 8 * s, sph, GP_WAIT_LIMIT, s_abort));          // a buffer's arrivals belong to one chunk
            if (!ok) break;
            hf_arrive(bar_full + 8 * s);
            if (++s == NA) { s = 0; sph ^= 1u; }
            if (++b == NB) { b = 0; ph ^= 1u; }
        }
        if (!ok && a.err_flag != nullptr) atomicExch(a.err_flag, 1u);
    }
    }
    hf_fence_before();
    __syncthreads();
    if (warp == GP_EPI + GP_DEC) {
        hf_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::TMEM) : "memory");
    }
}

template <int FMT> cudaError_t launch_gp_experts(cudaStream_t s, const GpExperts &args, uint32_t max_tiles, int sm_count, bool pdl) {
    constexpr uint32_t smem = GpLayout<FMT, 32, true>::TOTAL;
    static_assert(smem <= 227u * 1024u, "shared memory");
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(gemm_prompt_kernel<FMT, 32, true>), smem);
    if (e != cudaSuccess) return e;
    return launch_kernel(gemm_prompt_kernel<FMT, 32, true>, dim3((unsigned)std::min<uint64_t>((uint64_t)max_tiles * args.row_tiles, (uint64_t)sm_count)), dim3(GpLayout<FMT, 32, true>::THREADS), smem, s,
                         pdl, args);
}

template <int FMT, int N> cudaError_t launch_gp(cudaStream_t s, GpArgs args, int sm_count, bool pdl) {
    constexpr uint32_t smem = GpLayout<FMT, N>::TOTAL;
    static_assert(smem <= 227u * 1024u, "shared memory");
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(gemm_prompt_kernel<FMT, N, false>), smem);
    if (e != cudaSuccess) return e;
    args.tok_tiles = (args.n_tok + N - 1) / N;
    args.width = std::min<uint32_t>(N, ((args.n_tok + args.tok_tiles - 1) / args.tok_tiles + 31) / 32 * 32);
    args.tiles = ((args.g.rows + GP_M - 1) / GP_M) * args.tok_tiles;
    return launch_kernel(gemm_prompt_kernel<FMT, N, false>, dim3(std::min<uint32_t>(args.tiles, sm_count)), dim3(GpLayout<FMT, N>::THREADS), smem, s, pdl, args);
}
}  // namespace

template <int FMT> static cudaError_t launch_gp_fmt(cudaStream_t s, const GpArgs &args, int sm_count, bool pdl) {
    // the width with the fewest waves, times a chunk's time (us, 148 CTAs, 8192 columns): what is wide shares expansions, what is narrow spreads
    constexpr uint32_t WIDTH[5] = {32, 64, 96, 128, 192};
    constexpr float CHUNK[5] = {0.355f, 0.455f, 0.505f, 0.61f, 0.81f};
    const uint32_t row_tiles = (args.g.rows + GP_M - 1) / GP_M;
    uint32_t best = 0;
    float cost = 0.0f;
    for (uint32_t k = 0; k < 5; ++k) {
        const uint32_t tiles = row_tiles * ((args.n_tok + WIDTH[k] - 1) / WIDTH[k]);
        const float c = (float)((tiles + sm_count - 1) / sm_count) * CHUNK[k];
        if (k == 0 || c < cost) { cost = c; best = k; }
    }
    switch (best) {
        case 0: return launch_gp<FMT, 32>(s, args, sm_count, pdl);
        case 1: return launch_gp<FMT, 64>(s, args, sm_count, pdl);
        case 2: return launch_gp<FMT, 96>(s, args, sm_count, pdl);
        case 3: return launch_gp<FMT, 128>(s, args, sm_count, pdl);
        default: return launch_gp<FMT, 192>(s, args, sm_count, pdl);
    }
}

bool gemm_prompt_takes(int fmt, uint32_t rows, uint32_t nc, uint32_t n_tok, int sm_count) {
    if (nc < 32 || (nc % 32 != 0 && nc % 32 < 8)) return false;
    if (nc % 32 == 0 || (nc >= 64 && fmt != FMT_NF5)) return true;
    const uint32_t shared = fmt == FMT_BP5 ? 64 : fmt == FMT_NF3 || fmt == FMT_NF4 || fmt == FMT_NF4G || fmt == FMT_NF5 ? 32 : 0;          // tokens of the other kernel's tile
    return shared == 0 || (uint64_t)((rows + GP_M - 1) / GP_M) * ((n_tok + shared - 1) / shared) > (uint64_t)sm_count;
}

cudaError_t launch_gemm_prompt(cudaStream_t stream, const GemvArgs &g, int fmt, const ActHalf &h, bool image_ready, uint32_t n_tok, int sm_count, bool pdl) {
    GpArgs args;
    args.g = g; args.img = h.img; args.xs_img = h.scales; args.zero = image_ready ? h.zero : nullptr; args.n_tok = n_tok; args.tok_pad = (uint32_t)act_half_tokens(n_tok);
    switch (fmt) {
        case FMT_BP4: return launch_gp_fmt<FMT_BP4>(stream, args, sm_count, pdl);
        case FMT_BP5: return launch_gp_fmt<FMT_BP5>(stream, args, sm_count, pdl);
        case FMT_BP6: return launch_gp_fmt<FMT_BP6>(stream, args, sm_count, pdl);
        case FMT_NF4: return launch_gp_fmt<FMT_NF4>(stream, args, sm_count, pdl);
        case FMT_NF4G: return launch_gp_fmt<FMT_NF4G>(stream, args, sm_count, pdl);
        case FMT_NF3: return launch_gp_fmt<FMT_NF3>(stream, args, sm_count, pdl);
        case FMT_NF5: return launch_gp_fmt<FMT_NF5>(stream, args, sm_count, pdl);
        case FMT_E8Q2: return launch_gp_fmt<FMT_E8Q2>(stream, args, sm_count, pdl);
        default: return cudaErrorNotSupported;
    }
}

cudaError_t launch_gemm_experts(cudaStream_t stream, const DeviceMatrix &m0, int fmt, const ExpertCodebook *books, const uint8_t *const *bases, uint32_t n_experts,
                                const ExpertTiles &t, uint32_t n_pair, uint32_t act_group, const int8_t *xq, const float *xs, float *out, int sm_count, uint32_t *err_flag, bool pdl) {
    GpExperts args;
    if (fill_gemv_args(m0, true, args.g) < 0) return cudaErrorNotSupported;
    args.g.xq = xq; args.g.xs = xs; args.g.out = out; args.g.out_stride = m0.geom.rows; args.g.err_flag = err_flag;
    args.n_tiles = t.n_tiles; args.tile_expert = t.expert; args.tile_pairs = t.pairs;
    args.books = books; args.bases = bases; args.base0 = m0.d_base; args.act_group = act_group; args.row_tiles = (m0.geom.rows + GP_M - 1) / GP_M;
    const uint32_t tiles = expert_tiles_max(n_pair, n_experts);
    switch (fmt) {
        case FMT_NF4: return launch_gp_experts<FMT_NF4>(stream, args, tiles, sm_count, pdl);
        case FMT_NF4G: return launch_gp_experts<FMT_NF4G>(stream, args, tiles, sm_count, pdl);
        case FMT_NF3: return launch_gp_experts<FMT_NF3>(stream, args, tiles, sm_count, pdl);
        case FMT_NF5: return launch_gp_experts<FMT_NF5>(stream, args, tiles, sm_count, pdl);
        case FMT_E8Q2: return launch_gp_experts<FMT_E8Q2>(stream, args, tiles, sm_count, pdl);
        default: return cudaErrorNotSupported;       // experts are NF matrices (2..5 bits)
    }
}

}  // namespace k2t
