// Pieces of the mma.sync GEMV kernels (qmv_mm.cu, moe_mm.cu): asynchronous copies, the B fragments of the activations, and the products of a
// ring slot of packed rows with them.
#pragma once

#include "common.cuh"

namespace lisa {

__device__ __forceinline__ void mm_cp16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void mm_cp16z(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void mm_cp4z(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void mm_lds128(uint32_t addr, uint32_t *r) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mm_lds64(uint32_t addr, uint32_t *r) {
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
}
__device__ __forceinline__ uint32_t mm_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
// d = a . b + c, f16 16x16 by 16x8, f32
__device__ __forceinline__ void mm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, float c0,
                                       float c1, float c2, float c3) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
__device__ __forceinline__ uint32_t mm_pack_f16x2(float lo, float hi) {
    uint32_t out;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(out) : "f"(hi), "f"(lo));
    return out;
}

// How a 64-k group of a packed row is split over the four lanes of a fragment row: sixteen codes each.
template <int BITS>
struct MmShape {
    static constexpr int kGroups = 1024 / BITS / 64;       // 64-k groups of a step: 8 / 4 / 2
    static constexpr int kWords = BITS / 2;                // packed words of a lane and group: 1 / 2 / 4
    static constexpr int kPitch = BITS == 2 ? 144 : BITS == 4 ? 160 : 192;  // row pitch of a slot: reads free of bank conflicts
};

// Codes as f16 operands without arithmetic: a field masked in place is a subnormal f16, q * place * 2^-24 exactly (bits 0 to 9 of a half
// word), so that lifting a pair of codes is one AND, and a shift where the field lies higher: one per word of 4-bit codes (places 1 and
// 16) or 2-bit codes (places 1 .. 256), one for two 8-bit pairs.  As bf16 128 + q it took three shifts and the sums their
// start values.  x, normalised by a power of two per (group, token) to below 2^15, is divided by the place: exact where an element is
// above 2^-24 of the group's largest, and within 2^-32 of that one everywhere.
// An MMA cuts its sum some 24 bits below the largest product as the exponent fields of its operands have it, which for a subnormal code is up to
// ten bits above the product.  Error of the sums against 64 bits (2048 terms minus the same in another order, relative to one half, eight rows):
// 8-bit 0.9e-7 (the generic kernel 1.9e-7), 4-bit with group size 128 1.6e-7 and 2-bit 6e-7 (the bf16 mma.sync kernel 7e-7 and 36e-7); group size
// 64 the same, where the tensor-memory kernel's sums are exact on a grid of the activations of 2^-13.  All below the 2^-9 of a bf16 result; gguf_mm.cu,
// whose results are f32, uses normal numbers.

// A lane's sixteen elements of a (group, token), e[8] packed pairs -> its part of the B fragments and, with the other three lanes of the
// (group, token), the factor and the sum (whole warps call it: the four lanes are neighbours).  Pair q of the lane's
// packed words holds elements (4-bit) 8 (q / 4) + q % 4 and + 4; (2-bit) q and q + 8; (8-bit) 4 (q / 2) + q % 2 and + 2.  Pairs
// 0..3 are half 0, pairs 4..7 half 1.
template <int BITS, int MT>
__device__ __forceinline__ void mm_fragment(const uint32_t (&e)[8], uint32_t frag, uint32_t sums, int gl, int t, int cc, bool in) {
    constexpr int FRAG = MT * 128;  // bytes of a group's fragments: two halves of MT x 4 lanes x 16
    constexpr int SUMS = MT * 8;    // of a pair of tokens: factors {a, b}, sums of x {a, b}
    float sum = 0.f;
    uint32_t amax = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        sum += __uint_as_float(e[q] << 16) + __uint_as_float(e[q] & 0xffff0000u);
        amax = __vmaxu2(amax, e[q] & 0x7fff7fffu);
    }
#pragma unroll
    for (int off = 1; off < 4; off <<= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, off);
        amax = __vmaxu2(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    }
    // E: biased exponent of the group's largest magnitude, at least the one whose inverse is a float (smaller groups keep that grid).  An
    // infinity or NaN makes the factor NaN.
    const uint32_t ex0 = max(amax & 0xffffu, amax >> 16) >> 7, ex = max(ex0, 14u);
    const bool live = ex0 < 255u;
    const float up = live ? __uint_as_float((268u - ex) << 23) : 0.f;  // 2^(14 - (E - 127))
    auto lo = [&](int i) { return __uint_as_float(e[i] << 16); };
    auto hi = [&](int i) { return __uint_as_float(e[i] & 0xffff0000u); };
    uint32_t b[8];
    if constexpr (BITS == 2) {
        // pair q = elements (q, q + 8): even q: low halves of words q / 2 and q / 2 + 4, odd q: high halves; place 4^q, from q = 5 4^(q - 5)
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float s = up * (1.0f / static_cast<float>(1 << (2 * (q < 5 ? q : q - 5))));
            b[q] = (q & 1) ? mm_pack_f16x2(hi(q >> 1) * s, hi((q >> 1) + 4) * s) : mm_pack_f16x2(lo(q >> 1) * s, lo((q >> 1) + 4) * s);
        }
    } else if constexpr (BITS == 4) {
        // pairs 0 and 2 of a word have place 1, 1 and 3 place 16
        const float up16 = up * 0.0625f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            b[4 * h + 0] = mm_pack_f16x2(lo(4 * h) * up, lo(4 * h + 2) * up);
            b[4 * h + 1] = mm_pack_f16x2(hi(4 * h) * up16, hi(4 * h + 2) * up16);
            b[4 * h + 2] = mm_pack_f16x2(lo(4 * h + 1) * up, lo(4 * h + 3) * up);
            b[4 * h + 3] = mm_pack_f16x2(hi(4 * h + 1) * up16, hi(4 * h + 3) * up16);
        }
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            b[q] = (q & 1) ? mm_pack_f16x2(hi(q & ~1) * up, hi(q | 1) * up) : mm_pack_f16x2(lo(q & ~1) * up, lo(q | 1) * up);
    }
    if (in) {
        const uint32_t to = frag + gl * FRAG + (t * 4 + cc) * 16;
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + FRAG / 2), "r"(b[4]), "r"(b[5]), "r"(b[6]), "r"(b[7]) : "memory");
        if (cc == 0) {
            const uint32_t so = sums + gl * SUMS + (t >> 1) * 16 + (t & 1) * 4;
            // 2^((E - 127) - 14 + 24), less the 2^16 that the scale takes (each stays in range)
            const float factor = __uint_as_float(live ? (ex - 6u) << 23 : 0x7fc00000u);
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(so), "f"(factor) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(so + 8), "f"(sum) : "memory");
        }
    }
}

// Masks of the fields, pinned in registers.
template <int BITS>
struct MmLift {
    static constexpr int kMasks = BITS == 2 ? 5 : BITS == 4 ? 2 : 1;
    uint32_t mk[kMasks];
    __device__ __forceinline__ MmLift() {
#pragma unroll
        for (int i = 0; i < kMasks; ++i)
            asm volatile("mov.u32 %0, %1;" : "=r"(mk[i]) : "r"((BITS == 2 ? 0x00030003u : BITS == 4 ? 0x000f000fu : 0x00ff00ffu) << (BITS * i)));
    }
};

// Adds a ring slot (16 rows of 128 packed bytes, their scales and biases behind them, at `at`) against the fragments fa and sums sa of its
// groups to acc: rows g, g + 8; tokens 2c, 2c + 1.
template <int BITS, int MT, bool G128>
__device__ __forceinline__ void mm_step(uint32_t at, uint32_t fa, uint32_t sa, int g, int c, const MmLift<BITS> &lift, float (&acc)[2][2]) {
    using S = MmShape<BITS>;
    constexpr int G = S::kGroups, PITCH = S::kPitch, WSLOT = 16 * PITCH, FRAG = MT * 128, SUMS = MT * 8;
    constexpr int WPR = (G128 ? G / 2 : G) / 2;  // 32-bit words of scales (and of biases) per row and step: 4, 2 or 1
    uint32_t sw[4];
    const uint32_t wa = at + g * PITCH + c * (S::kWords * 4), sc = at + WSLOT + g * WPR * 4;
#pragma unroll
    for (int gi = 0; gi < G; ++gi) {
        uint32_t b[8], w0[S::kWords], w1[S::kWords];
        float fs[4];  // factors and sums of the two tokens
        mm_lds128(fa + gi * FRAG, b);
        mm_lds128(fa + gi * FRAG + FRAG / 2, b + 4);
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(fs[0]), "=f"(fs[1]), "=f"(fs[2]), "=f"(fs[3]) : "r"(sa + gi * SUMS));
        if constexpr (BITS == 2) {
            w0[0] = mm_lds32(wa + gi * 16);
            w1[0] = mm_lds32(wa + gi * 16 + 8 * PITCH);
        } else if constexpr (BITS == 4) {
            mm_lds64(wa + gi * 32, w0);
            mm_lds64(wa + gi * 32 + 8 * PITCH, w1);
        } else {
            mm_lds128(wa + gi * 64, w0);
            mm_lds128(wa + gi * 64 + 8 * PITCH, w1);
        }
        // scales and biases of rows g, g + 8: two groups a word
        constexpr int kGps = G128 ? 4 : 2;  // 64-k groups per word
        if (gi % kGps == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sw[i] = mm_lds32(sc + (gi / kGps) * 4 + i * (32 * WPR));
        }
        const bool hi = (gi / (kGps / 2)) & 1;
        auto pick = [&](uint32_t v) { return __uint_as_float(hi ? v & 0xffff0000u : v << 16); };
        const float s_0 = pick(sw[0]) * 65536.f, s_1 = pick(sw[1]) * 65536.f, b_0 = pick(sw[2]), b_1 = pick(sw[3]);
        float d[4] = {0.f, 0.f, 0.f, 0.f};
        if constexpr (BITS == 2) {
            const uint32_t h0 = w0[0] >> 10, h1 = w1[0] >> 10;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                auto field = [&](uint32_t w, uint32_t h, int q) { return q < 5 ? w & lift.mk[q] : h & lift.mk[q - 5]; };
                mm_mma(d, field(w0[0], h0, 2 * j), field(w1[0], h1, 2 * j), field(w0[0], h0, 2 * j + 1), field(w1[0], h1, 2 * j + 1), b[2 * j], b[2 * j + 1],
                       d[0], d[1], d[2], d[3]);
            }
        } else if constexpr (BITS == 4) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t u0 = w0[j >> 1] >> (8 * (j & 1)), u1 = w1[j >> 1] >> (8 * (j & 1));
                mm_mma(d, u0 & lift.mk[0], u1 & lift.mk[0], u0 & lift.mk[1], u1 & lift.mk[1], b[2 * j], b[2 * j + 1], d[0], d[1], d[2], d[3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mm_mma(d, w0[j] & lift.mk[0], w1[j] & lift.mk[0], (w0[j] >> 8) & lift.mk[0], (w1[j] >> 8) & lift.mk[0], b[2 * j], b[2 * j + 1], d[0], d[1],
                       d[2], d[3]);
        }
        acc[0][0] = fmaf(s_0 * fs[0], d[0], fmaf(b_0, fs[2], acc[0][0]));
        acc[0][1] = fmaf(s_0 * fs[1], d[1], fmaf(b_0, fs[3], acc[0][1]));
        acc[1][0] = fmaf(s_1 * fs[0], d[2], fmaf(b_1, fs[2], acc[1][0]));
        acc[1][1] = fmaf(s_1 * fs[1], d[3], fmaf(b_1, fs[3], acc[1][1]));
    }
}

}  // namespace lisa
