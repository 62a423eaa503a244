// Parts that the prompt GEMMs over half-precision operands share (k2t_gemm_f16.cu, k2t_gemm_prompt.cu): copies, tensor-core operations,
// the packed chain step, and the expansion of a cell to halves.
#pragma once
#include "k2t_act_image.cuh"
#include "k2t_gemv_core.cuh"

namespace k2t {

template <int FMT> __host__ __device__ constexpr uint32_t hf_cell() { return Cell<FMT>::B0 + Cell<FMT>::B1 + Cell<FMT>::B2; }

constexpr uint32_t HF_NO_PAIR = 0xffffffffu;          // behind the last pair of an expert's tile

__device__ __forceinline__ void hf_cp_async16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void hf_cp_async8(uint32_t dst, const void *src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void hf_cp_async4(uint32_t dst, const void *src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ uint32_t hf_lds32(uint32_t saddr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}
__device__ __forceinline__ void hf_lds64(uint32_t saddr, uint32_t &x, uint32_t &y) { asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(x), "=r"(y) : "r"(saddr)); }
__device__ __forceinline__ void hf_lds128(uint32_t saddr, uint32_t *v) {
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(saddr));
}
__device__ __forceinline__ void hf_lds_pairs(uint32_t saddr, unsigned long long &x, unsigned long long &y) {
    asm volatile("ld.shared.v2.b64 {%0,%1}, [%2];" : "=l"(x), "=l"(y) : "r"(saddr));
}
__device__ __forceinline__ void hf_sts128(uint32_t saddr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(saddr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void hf_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void hf_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void hf_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void hf_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void hf_mma(uint32_t d_tmem, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n" ::"r"(d_tmem), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ uint64_t hf_desc(uint32_t saddr) {      // K-major, 128-byte swizzle, groups of eight rows 1024 bytes apart
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// sixteen accumulators of the lane's row, waited for
__device__ __forceinline__ void hf_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
          "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ unsigned long long hf_pack(uint32_t lo, uint32_t hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1,%2};" : "=l"(d) : "r"(lo), "r"(hi));
    return d;
}
// two chain steps: f <- fma(dot * xs, ws, f) in both halves
__device__ __forceinline__ unsigned long long hf_step2(unsigned long long dot, unsigned long long xs, unsigned long long ws, unsigned long long f) {
    unsigned long long p, r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(dot), "l"(xs));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(p), "l"(ws), "l"(f));
    return r;
}
// A row's cell -> 64 halves in column order.  Bit-planes: 2 code - (2^B - 1), codebooks: the centroid.
struct HfTables { uint32_t cb[8], tab[4]; __half2 add; };
template <int FMT, typename T> __device__ __forceinline__ HfTables hf_tables(const T &a) {          // T: GemvArgs or ExpertCodebook

    HfTables t;
    // codebook bytes are stored + 128 (sign bit flipped) so that they are unsigned
#pragma unroll
    for (int i = 0; i < 8; ++i) t.cb[i] = a.cb[i] ^ 0x80808080u;
#pragma unroll
    for (int i = 0; i < 4; ++i) t.tab[i] = a.tab[i];
    int c = FMT == FMT_NF4 ? -1152 + a.nf4_offset : -1152;
    if constexpr (is_bitplane<FMT>()) c = -1024 - a.max_odd;
    t.add = __half2half2(__int2half_rn(c));
    return t;
}
template <int FMT> __device__ __forceinline__ void hf_expand(const Raw<FMT> &w, const HfTables &t, uint32_t (&h)[32]) {
    if (FMT == FMT_BP4) {            // twice the code, straight from the nibbles
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            hf_widen((w.w[i] << 1) & 0x1E1E1E1Eu, t.add, h[4 * i], h[4 * i + 1]);
            hf_widen((w.w[i] >> 3) & 0x1E1E1E1Eu, t.add, h[4 * i + 2], h[4 * i + 3]);
        }
        return;
    }
    if (FMT == FMT_NF4) {            // upper and lower half of the sorted codebook in two tables of non-negative bytes (see cell_dot)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t x = w.w[i], y = x ^ 0x88888888u;
            hf_widen(0x80808080u + prmt(t.tab[0], t.tab[1], y) - prmt(t.tab[2], t.tab[3], x), t.add, h[4 * i], h[4 * i + 1]);
            hf_widen(0x80808080u + prmt(t.tab[0], t.tab[1], __umulhi(y, 65536u)) - prmt(t.tab[2], t.tab[3], __umulhi(x, 65536u)), t.add, h[4 * i + 2], h[4 * i + 3]);
        }
        return;
    }
    uint32_t u[16];
    decode<FMT>(w, t.cb, u);
#pragma unroll
    for (int j = 0; j < 16; ++j) hf_widen(is_bitplane<FMT>() ? u[j] << 1 : FMT == FMT_E8Q2 ? u[j] ^ 0x80808080u : u[j], t.add, h[2 * j], h[2 * j + 1]);
}

// k2t_gemm_prompt.cu: the product for rows of 32 chunks and more whose last pass is not a stub of a few chunks (its fetch weighs as much as a
// whole one's); shorter rows end before the longer start of that kernel pays (576 x 960, 200 tokens 5.8 against 5.9 us, 576 x 3072 7.2 against
// 7.7; 4160 x 160 b5 29.5 against 32.5).  Of the others, rows of one whole pass and a part (nf5: of any passes and a part) stay with k2t_gemm_f16.cu while
// its tiles of 32 tokens (b5: 64) fit one wave: the part comes by copies of single chunks, 8 bytes each for b5, nf3 and nf5, of one warp, and nothing is
// shared yet.  There / here, us, image ready, cold weights: 3584 x 4608 b5, 77 tokens 29.1 / 31.7, 256 31.9 / 34.2, 300 43.6 / 38.1; 3584 x 4096 (rows) nf5,
// 128 32.6 / 36.4, 300 41.4 / 39.5; nf3 25.9 / 27.9, 200 30.4 / 29.6; nf4 26.1 / 27.5, 300 31.5 / 30.6; nf4g128 26.0 / 26.7.  b4, b6 and e8q2 are within 2% or
// faster here, and so are the other formats from nc = 64 on (4096 rows x 7168, 16 to 512 tokens: b5 55 to 83 / 53 to 72, nf3 49 to 78 / 46 to 70;
// nf5, 128 tokens 60.6 / 63.2, x 18944 147 / 153) and whole passes (2048, 4096, 8192 columns: 0.99 to 1.5 times as fast).
bool gemm_prompt_takes(int fmt, uint32_t rows, uint32_t nc, uint32_t n_tok, int sm_count);
cudaError_t launch_gemm_prompt(cudaStream_t stream, const GemvArgs &g, int fmt, const ActHalf &h, bool image_ready, uint32_t n_tok, int sm_count, bool pdl);

}  // namespace k2t
