// Pieces of the dot-product GEMV kernels (qmv_dp.cu, moe_dp.cu): asynchronous copies, the integer form of the activations, and
// the products of a chunk of packed codes with it.
#pragma once

#include "common.cuh"

namespace lisa {

// d = c + sum of four products of unsigned bytes of a and signed bytes of b
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Asynchronous copies of 16 / 4 bytes to shared memory; the second form writes zeros where `in` is false (the address
// stays valid).
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16z(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4z(uint32_t dst, const void *src, bool in) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void lds128(uint32_t addr, uint32_t *r) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}

// The activations of one chunk in shared memory, as the words that meet the packed words: FIELDS fields of a packed
// word (its low and high nibbles; its four 2-bit fields; its bytes), PLANES planes of bytes (the highest first) each.
//
// Two planes: x on a grid of 2^-13 of the chunk's largest power of two, the documented form of group size 64 (2- and 4-bit).
// Four planes: 2^-29, which a bf16 value lies on when it is above 2^-22 of the chunk's largest and misses by at most 2^-30 of that one
// otherwise, less than the rounding of an f32 product with the largest: the form of every operator that promises the activations as they are
// (8-bit codes, group sizes 32 and 128, the routed block).
template <int BITS, int PLANES = 2>
struct DpShape {
    static constexpr int kWords = (BITS == 2) ? 4 : 8;               // packed words of a chunk
    static constexpr int kFields = 8 / BITS;                         // fields of a byte
    static constexpr int kCodes = kWords * 32 / BITS;                // 64 / 64 / 32
    static constexpr int kXWords = kWords * kFields * PLANES;        // activation words of a chunk: 16 / 16 / 8 a plane
    // the fields' place values make the chunk's integer 16 (4-bit) or 64 (2-bit) times the sum
    static constexpr int kPlace = (BITS == 4) ? 4 : (BITS == 2) ? 6 : 0;
    static constexpr int kGrid = PLANES == 2 ? 13 : 29;
};

// Vector i of a row of x (eight elements) -> its part of the chunk's activation words in xs ([steps][vectors of a chunk][8]) and
// {factor, sum(s)} in xf ([steps * 8][1 + SUB]); whole warps call it: the vectors of a chunk are adjacent lanes and share the exponent and the sums through shuffles
template <int BITS, bool G32, int PLANES = 2>
__device__ __forceinline__ void dp_convert(uint4 *xs, float *xf, int i, const uint4 &v) {
    using S = DpShape<BITS, PLANES>;
    constexpr int XV = S::kXWords / 4, SUB = G32 ? 2 : 1, PAIRS = PLANES / 2;
    constexpr int VPC = S::kCodes / 8;  // vectors per chunk: 8 / 8 / 4
    const uint32_t rw[4] = {v.x, v.y, v.z, v.w};
    float f[8];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f[2 * q] = __uint_as_float(rw[q] << 16);
        f[2 * q + 1] = __uint_as_float(rw[q] & 0xffff0000u);
    }
    float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
    uint32_t amax = __vmaxu2(__vmaxu2(rw[0] & 0x7fff7fffu, rw[1] & 0x7fff7fffu), __vmaxu2(rw[2] & 0x7fff7fffu, rw[3] & 0x7fff7fffu));
#pragma unroll
    for (int off = 1; off < VPC; off <<= 1) {
        amax = __vmaxu2(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        if (!(G32 && off == VPC / 2)) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    }
    // E: biased exponent of the chunk's largest magnitude, at least the one below which the factor would leave the range of a float
    // (smaller chunks keep that grid).  An infinity or NaN makes the chunk's factor NaN.
    const uint32_t e0 = max(amax & 0xffffu, amax >> 16) >> 7, e = max(e0, static_cast<uint32_t>(S::kGrid + S::kPlace + 1));
    const bool live = e0 < 255u;
    const float up = live ? __uint_as_float((254u + S::kGrid - e) << 23) : 0.f;  // 2^(kGrid - (E - 127))
    // digit p of x_int = rn(x * 2^(kGrid-E)), |x_int| < 2^(kGrid+1), is byte PLANES - 1 - p of word[p]
    uint32_t word[PLANES][8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if constexpr (PLANES == 2) {
            // through the mantissa of 1.5 * 2^23: the low bytes of the sum are those of x_int
            word[1][j] = __float_as_uint(fmaf(f[j], up, 12582912.f));
            word[0][j] = word[1][j] + 128u;
        } else {
            // signed digits: what a digit's sign takes away is carried into the next byte
            const uint32_t xi = static_cast<uint32_t>(live ? __float2int_rn(f[j] * up) : 0);
            word[3][j] = xi;
            word[2][j] = xi + 128u;
            word[1][j] = xi + 32896u;
            word[0][j] = xi + 8421504u;
        }
    }
    auto pack = [&](int p, int a, int b, int c, int d) {  // digit p of four elements
        constexpr uint32_t kSel[4] = {0x0040, 0x0051, 0x0062, 0x0073};
        const uint32_t sel = kSel[PLANES - 1 - p];
        return __byte_perm(__byte_perm(word[p][a], word[p][b], sel), __byte_perm(word[p][c], word[p][d], sel), 0x5410);
    };
    const int chunk = i / VPC, j = i - chunk * VPC;
    const int jf = j ^ ((BITS != 2 && (chunk & 4)) ? VPC / 2 : 0);  // (see the reads of the packed words)
    uint4 *dst = xs + static_cast<size_t>(chunk >> 3) * XV * 8 + (chunk & 7);
    if constexpr (BITS == 4) {
        // packed word j: low nibbles = codes 0, 2, 4, 6, high nibbles = 1, 3, 5, 7; a vector holds two planes
#pragma unroll
        for (int p = 0; p < PAIRS; ++p)
            dst[(jf * PAIRS + p) * 8] = make_uint4(pack(2 * p, 0, 2, 4, 6), pack(2 * p, 1, 3, 5, 7), pack(2 * p + 1, 0, 2, 4, 6), pack(2 * p + 1, 1, 3, 5, 7));
    } else if constexpr (BITS == 2) {
        // packed word j / 2 (16 codes): field f of byte c is code 4 c + f; this vector is bytes 2 (j & 1) and
        // 2 (j & 1) + 1, i.e. half-words of the four words of each plane, vector PLANES (j / 2) + plane
#pragma unroll
        for (int p = 0; p < PLANES; ++p) {
            constexpr uint32_t kSel[4] = {0x0040, 0x0051, 0x0062, 0x0073};
            uint16_t *to = reinterpret_cast<uint16_t *>(dst + ((j >> 1) * PLANES + p) * 8) + (j & 1);
#pragma unroll
            for (int q = 0; q < 4; ++q) to[2 * q] = static_cast<uint16_t>(__byte_perm(word[p][q], word[p][4 + q], kSel[PLANES - 1 - p]));
        }
    } else {
        // packed words 2j and 2j + 1 hold the eight codes as bytes
#pragma unroll
        for (int p = 0; p < PAIRS; ++p)
            dst[(jf * PAIRS + p) * 8] = make_uint4(pack(2 * p, 0, 1, 2, 3), pack(2 * p, 4, 5, 6, 7), pack(2 * p + 1, 0, 1, 2, 3), pack(2 * p + 1, 4, 5, 6, 7));
    }
    float *fo = xf + static_cast<size_t>(chunk) * (1 + SUB);
    if (j == 0) {
        fo[0] = live ? __uint_as_float((e - S::kGrid - S::kPlace) << 23) : __uint_as_float(0x7fc00000u);
        fo[1] = sum;
    }
    if (G32 && j == VPC / 2) fo[SUB] = sum;
}

// Takes a ring slot (eight rows x eight chunks at `at`, their scales and biases behind them) to registers.  Lanes 4 to 7 of a row
// read the halves of their 32-byte chunk in the other order (no bank conflicts); the activation words of those chunks are
// stored that way.
template <int BITS, bool G32>
struct DpTake {
    using S = DpShape<BITS>;
    static constexpr int kSub = G32 ? 2 : 1, kChunkBytes = S::kWords * 4, kWSlot = 64 * kChunkBytes, kSlot = kWSlot + 256 * kSub;
    int flip;
    uint32_t w_at, half0, half1, sc_at;
    __device__ __forceinline__ DpTake(int sl, int sub, int gshift) {
        flip = sl >> 2;
        w_at = (sub * 8 + sl) * kChunkBytes;
        half0 = flip * 16;
        half1 = 16 - half0;
        sc_at = kWSlot + sub * 16 + (kSub == 2 ? (sl >> 2) * 128 + (sl & 3) * 4 : ((sl * S::kCodes) >> gshift) * 2);
    }
    __device__ __forceinline__ void operator()(uint32_t at, uint32_t (&w)[2][S::kWords], uint32_t (&sc)[2][kSub], uint32_t (&bi)[2][kSub]) const {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int h = 0; h < kChunkBytes / 16; ++h) lds128(at + w_at + r * (4 * 8 * kChunkBytes) + (kChunkBytes == 32 ? (h ? half1 : half0) : 0u), w[r] + 4 * h);
#pragma unroll
            for (int g = 0; g < kSub; ++g) {
                const int gg = (kChunkBytes == 32 && kSub == 2) ? g ^ flip : g;
                sc[r][g] = lds_u16(at + sc_at + r * 64 + gg * 2);
                bi[r][g] = lds_u16(at + sc_at + r * 64 + gg * 2 + 128 * kSub);
            }
        }
    }
};

// Adds one chunk (64 or 32 codes of two rows, their scales and biases) against its activations to the rows' sums.  xt: the
// chunk's first activation vector, ft: its factor and sums; flip: see dp_take.
template <int BITS, bool G32, int PLANES = 2>
__device__ __forceinline__ void dp_chunk(const uint32_t (&w)[2][DpShape<BITS>::kWords], const uint32_t (&sc)[2][G32 ? 2 : 1],
                                         const uint32_t (&bi)[2][G32 ? 2 : 1], uint32_t xt, uint32_t ft, const uint32_t (&mask)[8 / BITS], int flip,
                                         float &acc0, float &acc1) {
    using S = DpShape<BITS, PLANES>;
    constexpr int SUB = G32 ? 2 : 1, CB = S::kWords * 4, PAIRS = PLANES / 2;
    constexpr int WORDS = BITS == 8 ? S::kWords / 2 : S::kWords;  // packed words, 8-bit: pairs of them
    float ff[1 + SUB];  // factor and sums of the chunk's activations
#pragma unroll
    for (int g = 0; g < 1 + SUB; ++g)
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(ff[g]) : "r"(ft + 4 * (CB == 32 && SUB == 2 && g ? 1 + ((g - 1) ^ flip) : g)));
#pragma unroll
    for (int g = 0; g < SUB; ++g) {
        float q[2] = {0.f, 0.f};
#pragma unroll
        for (int pp = 0; pp < PAIRS; ++pp) {  // two planes at a time
            int a[2][2][S::kFields];  // [row][plane][field]
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int f = 0; f < S::kFields; ++f) a[r][0][f] = a[r][1][f] = 0;
#pragma unroll
            for (int v = g * (WORDS / SUB); v < (g + 1) * (WORDS / SUB); ++v) {
                if constexpr (BITS == 2) {
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        uint32_t xw[4];
                        lds128(xt + (v * PLANES + 2 * pp + p) * 128, xw);
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int f = 0; f < 4; ++f) a[r][p][f] = dp4a_us(w[r][v] & mask[f], xw[f], a[r][p][f]);
                    }
                } else {
                    uint32_t xw[4];
                    lds128(xt + (v * PAIRS + pp) * 128, xw);  // (lanes of different rows read the same address: one wavefront)
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        if constexpr (BITS == 4) {
                            const uint32_t lo = w[r][v] & mask[0], hi = w[r][v] & mask[1];
                            a[r][0][0] = dp4a_us(lo, xw[0], a[r][0][0]);
                            a[r][0][1] = dp4a_us(hi, xw[1], a[r][0][1]);
                            a[r][1][0] = dp4a_us(lo, xw[2], a[r][1][0]);
                            a[r][1][1] = dp4a_us(hi, xw[3], a[r][1][1]);
                        } else {
                            a[r][0][0] = dp4a_us(w[r][2 * v], xw[0], a[r][0][0]);
                            a[r][0][0] = dp4a_us(w[r][2 * v + 1], xw[1], a[r][0][0]);
                            a[r][1][0] = dp4a_us(w[r][2 * v], xw[2], a[r][1][0]);
                            a[r][1][0] = dp4a_us(w[r][2 * v + 1], xw[3], a[r][1][0]);
                        }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                // field f carries 2^(f * BITS): bring all of them to the place value of the last one; below 2^30
                int v0 = a[r][0][0], v1 = a[r][1][0];
#pragma unroll
                for (int f = 1; f < S::kFields; ++f) {
                    v0 = v0 * (1 << BITS) + a[r][0][f];
                    v1 = v1 * (1 << BITS) + a[r][1][f];
                }
                const float part = static_cast<float>(v0 * 256 + v1);
                q[r] = pp == 0 ? part : fmaf(q[r], 65536.f, part);
            }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float &acc = r ? acc1 : acc0;
            acc = fmaf(bf16_bits_to_f32(sc[r][g]) * ff[0], q[r], fmaf(bf16_bits_to_f32(bi[r][g]), ff[1 + g], acc));
        }
    }
}

}  // namespace lisa
