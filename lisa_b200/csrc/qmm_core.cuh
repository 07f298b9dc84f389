// Pieces of the prefill GEMM kernels (qmm_affine.cu, qmm_pair.cu): tcgen05 / TMA wrappers, tile constants, and the decoder of the packed weights.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "common.cuh"

namespace lisa {

constexpr int kBN = 128;        // weight rows per CTA (MMA M)
constexpr int kWideBt = 384;    // the tall token tile (template WIDE)
constexpr int kBK = 64;         // k per MMA stage: 64 bf16 = one 128-byte swizzle row
constexpr int kStages = 5;      // operand ring of the one-CTA form: stage s = activation tile in shared memory + A tile in tensor memory
constexpr int kWpStages = 4;    // packed-weight ring: loads run a whole ring (12+ k-blocks) ahead of their use
constexpr int kQ4kBlock = 144;  // GGUF Q4_K: bytes of a 256-element block = one packed stage row (4 k-blocks)
constexpr int kQ2kBlock = 84;   // GGUF Q2_K: bytes of a block; a packed stage row is four of them (16 k-blocks)
constexpr int kACols = kBK / 2; // one k-block of A: 64 bf16 per lane = 32 columns
constexpr int kDequantWarps = 16;  // pairs: four sets of 4 warps, a thread per weight row; one CTA: two sets of 8 (even / odd k-blocks), two threads per row
constexpr int kWarpsPerKb = kDequantWarps / 2;  // (the one-CTA form)
constexpr int kThreads = (2 + kDequantWarps) * 32;
constexpr int kWpBytes = kBN * 128;       // 16 KiB

constexpr int kMaxSeg = 3;  // linears of one launch in the sibling form (q|k|v, gate|up)
struct QmmMaps {
    CUtensorMap m[kMaxSeg];
};

__device__ __forceinline__ uint32_t qmm_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void qmm_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void qmm_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// ---- tcgen05 / TMA wrappers ----
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    tma_load_2d(smem_u32(dst), map, x, y, smem_u32(bar));
}
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(cols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem descriptor {desc_lo, desc_hi}]; bf16 operands, f32 accumulate.
// A: lane = row, two consecutive k per 32-bit column (low half = even k), 8 columns per K=16 step.
__device__ __forceinline__ void umma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_lo, uint32_t desc_hi,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b64 d;\n\t"
        "mov.b64 d, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "r"(desc_lo), "r"(desc_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::
            "r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Shared-memory matrix descriptor, K-major, 128-byte swizzle, 8-row groups 1024 bytes apart, in two
// halves: low = start address >> 4 (bits 0-13) | leading byte offset 1 (bit 16, unused for swizzled
// K-major); high = stride byte offset 1024 >> 4 (bits 32-45) | version 1 (bit 46) | SWIZZLE_128B (2 << 61).
// Advancing k by 16 bf16 inside the 128-byte row adds 32 bytes = 2 to the low half.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr) { return (smem_addr >> 4) | (1u << 16); }
constexpr uint32_t kUmmaDescHiSw128 = (1024u >> 4) | (1u << 14) | (2u << 29);
// Instruction descriptor: D f32, A and B bf16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(128 >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// (a & b) | c in one LOP3 with all three operands in registers.
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// Packed bf16 arithmetic, one rounding per result.
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// Two codes of `src` -> two f32 weights, as a bf16 pair `hi` and the bf16 pair `lo` of what the rounding to bf16 left over: hi + lo
// carries 16 significant bits of each.  Code j sits at bit offset BITS*j of `src` and is masked in place (m0, m1), turned into the float
// 2^23 + q * 2^(BITS*j) by OR-ing the exponent of 2^23 (one LOP3 each), then both lanes at once: f - 2^23 (exact),
// (f - 2^23) * (s / 2^(BITS*j)) + b with one rounding -- the same real number as q * s + b.
__device__ __forceinline__ void dequant_pair_split(uint32_t src, uint32_t m0, uint32_t m1, uint32_t mbits,
                                                   unsigned long long neg_magic2, unsigned long long s2,
                                                   unsigned long long b2, uint32_t &hi, uint32_t &lo) {
    asm("{\n\t"
        ".reg .b32 q0, q1, h0, h1;\n\t"
        ".reg .f32 f0, f1;\n\t"
        ".reg .b64 t;\n\t"
        "lop3.b32 q0, %2, %3, %5, 0xEA;\n\t"
        "lop3.b32 q1, %2, %4, %5, 0xEA;\n\t"
        "mov.b64 t, {q0, q1};\n\t"
        "add.rn.f32x2 t, t, %6;\n\t"
        "fma.rn.f32x2 t, t, %7, %8;\n\t"
        "mov.b64 {f0, f1}, t;\n\t"
        "cvt.rn.bf16x2.f32 %0, f1, f0;\n\t"
        "shl.b32 h0, %0, 16;\n\t"
        "and.b32 h1, %0, 0xffff0000;\n\t"
        "sub.rn.f32 f0, f0, h0;\n\t"
        "sub.rn.f32 f1, f1, h1;\n\t"
        "cvt.rn.bf16x2.f32 %1, f1, f0;\n\t"
        "}\n"
        : "=r"(hi), "=r"(lo)
        : "r"(src), "r"(m0), "r"(m1), "r"(mbits), "l"(neg_magic2), "l"(s2), "l"(b2));
}

// Decoder of 32 codes of a row: `srow` is the row in its packed stage, (sub, half) the k-block of the stage and its half; scale sc and bias bi
// (GGUF: taken from the block header).  o: 16 pairs of bf16 weights, olo (GGUF only): what their rounding left over.
//
// GGUF = 4 (with BITS = 4): the packed rows are GGUF Q4_K blocks (crates/lisa-gguf/src/quant.rs:82-101):
// a stage row is one 144-byte block {f16 d, f16 dmin, 12 bytes of 6-bit scales and mins, 128 nibble bytes},
// a (k-block, half) is one 32-element sub-block g = 2*sub + half -- nibble `half` of bytes 32*sub .. +31 --
// i.e. an affine group with scale = d*sc_g and bias = -dmin*m_g, taken from the block header in shared
// memory.  GGUF = 2 (with BITS = 2): Q2_K blocks (quant.rs:64-80), four 84-byte blocks {16 scale/min
// bytes, 64 code bytes, f16 d, f16 dmin} per stage row; the 32 elements of (k-block, half) are the 2-bit
// fields at bit offset 2*shift of bytes 32*(kb4/2) .. +31, shift = 2*(kb4&1) + half, the first 16 under scale
// byte [half_of_block*8 + shift*2], the last 16 under the next one.  The output is f32.
template <int BITS, int GGUF>
struct QmmDecode {
    // masks and magic numbers, pinned in registers so that every extraction is one LOP3
    static constexpr int kMasks = GGUF == 0 ? (BITS == 4 ? 1 : 3) : (GGUF == 4 ? 4 : 8);
    uint32_t mk[kMasks], mbits, neg_magic;
    unsigned long long neg_magic2;
    __device__ __forceinline__ QmmDecode() {
#pragma unroll
        for (int j = 0; j < kMasks; ++j)
            asm volatile("mov.u32 %0, %1;" : "=r"(mk[j]) : "r"(GGUF == 0 ? (BITS == 4 ? 0x000f000fu : 0x00030003u << (2 * j)) : GGUF == 4 ? (0xfu << (4 * j)) : (0x3u << (2 * j))));
        asm volatile("mov.u32 %0, %1;" : "=r"(mbits) : "r"(GGUF == 0 ? 0x43004300u : 0x4b000000u));
        asm volatile("mov.u32 %0, %1;" : "=r"(neg_magic) : "r"(0xc300c300u));
        neg_magic2 = pack_f32x2(-8388608.0f, -8388608.0f);
    }
    __device__ __forceinline__ void operator()(uint32_t srow, int sub, int half, int swz, float sc, float bi, uint32_t (&o)[16], uint32_t (&olo)[16]) const {
        float sc1 = 0.f, bi1 = 0.f;  // Q2_K: scale and bias of the second 16 elements
        int qshift = 0;              // Q2_K: which 2-bit field of every byte
        // packed codes of (row, k-block, half): 32 codes
        uint32_t w[4];
        uint32_t wq[8];  // GGUF: the 32 bytes whose nibble `half` are this thread's codes
        if constexpr (GGUF == 2) {
            const int bq = sub >> 2, kb4 = sub & 3;  // block of the stage row, k-block of the block
            const uint32_t blk = srow + bq * kQ2kBlock;  // 4-byte aligned only
            const int hb = kb4 >> 1, shift = 2 * (kb4 & 1) + half;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                asm volatile("ld.shared.u32 %0, [%1];" : "=r"(wq[i]) : "r"(blk + 16 + hb * 32 + 4 * i));
            uint32_t sw, dd;
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(sw) : "r"(blk + hb * 8 + (shift >> 1) * 4));
            asm volatile("ld.shared.u32 %0, [%1];" : "=r"(dd) : "r"(blk + 80));
            // scale bytes [hb*8 + shift*2 + group], group 0 / 1 = first / last 16 elements
            const uint32_t sb0 = (sw >> (16 * (shift & 1))) & 255u, sb1 = (sw >> (16 * (shift & 1) + 8)) & 255u;
            float d, dmin;
            asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; cvt.f32.f16 %0, lo; cvt.f32.f16 %1, hi; }" : "=f"(d), "=f"(dmin) : "r"(dd));
            sc = d * static_cast<float>(sb0 & 15u);
            bi = -(dmin * static_cast<float>(sb0 >> 4));
            sc1 = d * static_cast<float>(sb1 & 15u);
            bi1 = -(dmin * static_cast<float>(sb1 >> 4));
            qshift = shift;
            w[0] = w[1] = w[2] = w[3] = 0;
        } else if constexpr (GGUF == 4) {
            const uint32_t blk = srow;
            uint32_t h0, h1, h2, h3;
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(h0), "=r"(h1), "=r"(h2), "=r"(h3) : "r"(blk));
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(wq[0]), "=r"(wq[1]), "=r"(wq[2]), "=r"(wq[3])
                         : "r"(blk + 16 + sub * 32));
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(wq[4]), "=r"(wq[5]), "=r"(wq[6]), "=r"(wq[7])
                         : "r"(blk + 32 + sub * 32));
            // 6-bit scale and min of sub-block g (quant.rs:88-96)
            const int g = 2 * sub + half, sh = 8 * (g & 3);
            const uint32_t b0 = (h1 >> sh) & 255u, b1 = (h2 >> sh) & 255u, b2 = (h3 >> sh) & 255u;
            const uint32_t sq = (g < 4) ? (b0 & 63u) : ((b2 & 15u) | ((b0 >> 6) << 4));
            const uint32_t mq = (g < 4) ? (b1 & 63u) : ((b2 >> 4) | ((b1 >> 6) << 4));
            float d, dmin;
            asm("{ .reg .b16 lo, hi; mov.b32 {lo, hi}, %2; cvt.f32.f16 %0, lo; cvt.f32.f16 %1, hi; }" : "=f"(d), "=f"(dmin) : "r"(h0));
            sc = d * static_cast<float>(sq);            // exact: 11 x 6 significant bits
            bi = -(dmin * static_cast<float>(mq));
            w[0] = w[1] = w[2] = w[3] = 0;
        } else if (BITS == 4) {
            const int c = sub * 2 + half;  // 16-byte chunk of the 128-byte packed row
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                         : "r"(srow + ((c ^ swz) << 4)));
        } else {
            uint32_t v0, v1;
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v0), "=r"(v1)
                         : "r"(srow + ((sub ^ swz) << 4) + half * 8));
            w[0] = v0;
            w[1] = v1;
        }
        [[maybe_unused]] const unsigned long long b2 = pack_f32x2(bi, bi);
        if constexpr (GGUF == 2) {
            // element 4i + b is the field at bit offset 2*shift of byte b of word i: offsets 2*shift and
            // 2*shift + 8 of each 16-bit half; mk[j] = 3 << 2j
            const float down = __uint_as_float((127u - 2u * qshift) << 23);  // 2^(-2*shift)
            const unsigned long long sg0 = pack_f32x2(sc * down, sc * down * 0.00390625f);
            const unsigned long long sg1 = pack_f32x2(sc1 * down, sc1 * down * 0.00390625f);
            const unsigned long long b21 = pack_f32x2(bi1, bi1);
            uint32_t m0 = mk[0], m1 = mk[4];
            if (qshift == 1) { m0 = mk[1]; m1 = mk[5]; }
            if (qshift == 2) { m0 = mk[2]; m1 = mk[6]; }
            if (qshift == 3) { m0 = mk[3]; m1 = mk[7]; }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                dequant_pair_split(wq[i], m0, m1, mbits, neg_magic2, i < 4 ? sg0 : sg1, i < 4 ? b2 : b21, o[2 * i + 0], olo[2 * i + 0]);
                dequant_pair_split(wq[i] >> 16, m0, m1, mbits, neg_magic2, i < 4 ? sg0 : sg1, i < 4 ? b2 : b21, o[2 * i + 1], olo[2 * i + 1]);
            }
        } else if constexpr (GGUF == 4) {
            // element 4i + b of the sub-block is nibble `half` of byte b of word i: bit offsets 4*half and
            // 4*half + 8 of each 16-bit half of the word
            const unsigned long long sg = half ? pack_f32x2(sc * 0.0625f, sc * 0.000244140625f)
                                               : pack_f32x2(sc, sc * 0.00390625f);
            const uint32_t m0 = half ? mk[1] : mk[0], m1 = half ? mk[3] : mk[2];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                dequant_pair_split(wq[i], m0, m1, mbits, neg_magic2, sg, b2, o[2 * i + 0], olo[2 * i + 0]);
                dequant_pair_split(wq[i] >> 16, m0, m1, mbits, neg_magic2, sg, b2, o[2 * i + 1], olo[2 * i + 1]);
            }
        } else {
            // bf16(q * s + b) for two codes at a time: a code goes to the low mantissa bits of 128.0 (one LOP3 for the codes 16 bits apart),
            // minus 128 (exact), times s plus b with one rounding; bytes are then paired up in the order of k.  That is the f32
            // multiply-add and its rounding to bf16 but where the first of the two roundings makes a tie of what is none, which takes a bias
            // below 2^-19 of the scale (all mantissas of both enumerated, for biases of 2^-40 to 2^23 of the scale).  2-bit codes 1, 2 of three
            // sit at 4 and 16 times their value: their scale is divided (a power of two).  Against packed f32 arithmetic (masks, add, fma, cvt, register moves) 76 instructions for 32 codes
            // instead of 112, which set the pace of a k-block.
            const uint32_t s2 = __float_as_uint(sc) | (__float_as_uint(sc) >> 16), bb = __float_as_uint(bi) | (__float_as_uint(bi) >> 16);
            if constexpr (BITS == 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t v[4];  // codes (j, j + 4)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[j] = fma_bf16x2(add_bf16x2(and_or(w[i] >> (4 * j), mk[0], mbits), neg_magic), s2, bb);
                    o[4 * i + 0] = __byte_perm(v[0], v[1], 0x5410);
                    o[4 * i + 1] = __byte_perm(v[2], v[3], 0x5410);
                    o[4 * i + 2] = __byte_perm(v[0], v[1], 0x7632);
                    o[4 * i + 3] = __byte_perm(v[2], v[3], 0x7632);
                }
            } else {
                const uint32_t sj[3] = {s2, mul_bf16x2(s2, 0x3e803e80u), mul_bf16x2(s2, 0x3d803d80u)};  // s, s / 4, s / 16
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    uint32_t v[8];  // codes (j, j + 8)
#pragma unroll
                    for (int j = 0; j < 8; ++j) v[j] = fma_bf16x2(add_bf16x2(and_or(w[i] >> (6 * (j / 3)), mk[j % 3], mbits), neg_magic), sj[j % 3], bb);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        o[8 * i + j] = __byte_perm(v[2 * j], v[2 * j + 1], 0x5410);
                        o[8 * i + 4 + j] = __byte_perm(v[2 * j], v[2 * j + 1], 0x7632);
                    }
                }
            }
        }
    }
};

}  // namespace lisa
