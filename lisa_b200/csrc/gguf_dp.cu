// GGUF K-quant matvec and expert matvec for a few tokens on byte dot products: f32 activations and output.
//   y[z, r] = sum_k x[z, k] * W[e(z), r, k],  Q4_K and Q2_K blocks (crates/lisa-gguf/src/quant.rs:64-101)
// (deepseek41::packed_matvec / expert_matvec, crates/lisa-mlx/src/models/deepseek41.rs:93-283; their Metal kernels
// crates/lisa-mlx/src/shaders/deepseek41/iq.metal:1130-1363).
//
// The structure is that of qmv_dp.cu: a warp walks tasks (eight rows, a run of steps) through a ring of asynchronous copies
// of contiguous pieces of the rows -- block headers and codes as they lie in memory -- and multiplies bytes with dp4a.
// An activation is three or four signed bytes on an integer grid of its sub-block (32 elements, Q2_K: 16): with E the exponent of
// the sub-block's largest magnitude x_int = rn(x * 2^(21-E)) or rn(x * 2^(29-E)), exact on dyadic inputs; sums are
// exact in s32 and meet scale and min of the sub-block in f32.  Three bytes are the grid of the tensor-memory kernel, for the calls which that
// one takes (gguf_grid_call in api.cu); all others are promised f32 activations, of which four bytes lose less than
// f32 sums do: 2048 x 2304 of Q2_K, Gaussian activations, relative error 0.7e-7, the warp-per-row kernel 1.0e-7, three bytes 2.8e-7.
//
// Why not the tensor-memory kernel: its Q2_K stages took 42 KB, one CTA per SM and two stages, and both formats paid its
// hand-overs per pair of k-blocks.  This form is bound by its instruction stream, about 0.06 warp instructions per code
// (three planes: 0.75 dp4a), some 5 TB/s of Q4_K and 3.5 TB/s of Q2_K blocks.
//
// One CTA takes a share of the rows of one z (a token of the dense form, a (token, expert) slot of the expert form): the
// grid is z times the CTAs that fill the SMs.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace lisa {

namespace {

constexpr int kGdThreads = 512, kGdWarps = kGdThreads / 32, kGdDepth = 2;

struct GdParams {
    const uint8_t *w;
    const float *x;
    float *y;
    long long row_bytes;
    int rows, k, steps, parts, spt;
    int octets, ctas, base, extra;  // octets of rows of one z, its CTAs, octets of a CTA (the first `extra` one more)
    int tail_pieces;                // pieces of a row in its last step where that is ragged, else 0
    int ring_at, part_at;
    // expert form: z is a slot of the flat [tokens, top_k] id table; its activations are row (z / top_k) * slots + (z % top_k)
    // % slots of x; an id outside [0, experts) stores zeros and touches no weights
    const int32_t *ids;
    int experts, slots, top_k;
};

__device__ __forceinline__ int gd_dp4a(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
template <int B>
__device__ __forceinline__ void gd_copy(uint32_t dst, const void *src, bool in) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
}
template <int B>
__device__ __forceinline__ void gd_copy(uint32_t dst, const void *src) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void gd_lds128(uint32_t addr, uint32_t *r) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t gd_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void gd_half2(uint32_t v, float &lo, float &hi) {
    asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; cvt.f32.f16 %0, l; cvt.f32.f16 %1, h; }" : "=f"(lo), "=f"(hi) : "r"(v));
}

// The sum that the planes' sums (the highest first, below 2^22 each) stand for.
template <int PLANES>
__device__ __forceinline__ float gd_value(const int (&c)[PLANES]) {
    if constexpr (PLANES == 3) return fmaf(static_cast<float>(c[0]), 65536.f, static_cast<float>(c[1] * 256 + c[2]));
    else return fmaf(static_cast<float>(c[0] * 256 + c[1]), 65536.f, static_cast<float>(c[2] * 256 + c[3]));
}

// FMT 4: Q4_K, a step is two blocks of a row, a lane's chunk 64 elements (32 code bytes, two sub-blocks); FMT 2: Q2_K, a step is
// four blocks, a chunk 128 elements (32 code bytes, eight sub-blocks).  PIECE: bytes of a copy (16; 4 for Q2_K rows that are
// not whole 16-byte pieces).
template <int FMT, int PLANES = 3>
struct GdShape {
    static constexpr int kBlock = FMT == 4 ? 144 : 84;
    static constexpr int kBlocks = FMT == 4 ? 2 : 4;       // of a step
    static constexpr int kRow = kBlock * kBlocks;          // bytes of a row and step: 288 / 336
    static constexpr int kPitch = FMT == 4 ? 320 : 352;    // of the rows in a slot: room for 16 bytes of offset, whole sectors
    static constexpr int kElems = FMT == 4 ? 64 : 128;     // of a chunk
    static constexpr int kXV = PLANES * (FMT == 4 ? 4 : 8);  // 16-byte vectors of activation words of a chunk
    static constexpr int kSubs = FMT == 4 ? 2 : 8;         // sub-blocks of a chunk
    static constexpr int kGrid = PLANES == 3 ? 21 : 29;
};

template <int FMT, int PIECE, int PLANES>
__global__ void __launch_bounds__(kGdThreads, 1) gguf_dp_kernel(const GdParams p) {
    using S = GdShape<FMT, PLANES>;
    constexpr int SLOT = 8 * S::kPitch, PPR = S::kRow / PIECE;  // pieces per row
    constexpr int COPIES = (8 * PPR + 31) / 32;
    extern __shared__ __align__(128) uint8_t gd_smem[];
    const uint32_t xs = smem_u32(gd_smem);                                   // [steps][kXV][8 lanes] 16-byte vectors
    const uint32_t xf = xs + p.steps * (S::kXV * 128);                       // [steps * 8][kSubs] {factor, sum}
    float *part = reinterpret_cast<float *>(gd_smem + p.part_at);            // [rows of the CTA][parts]
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int sl = lane & 7, sub = lane >> 3;
    const int z = static_cast<int>(blockIdx.x) / p.ctas, cta = static_cast<int>(blockIdx.x) - z * p.ctas;
    const int qb = cta * p.base + min(cta, p.extra), sets = p.base + (cta < p.extra ? 1 : 0);
    const uint8_t *w = p.w;
    const float *x = p.x + static_cast<size_t>(z) * p.k;
    if (p.ids) {
        const int e = __ldg(p.ids + z);
        if (e < 0 || e >= p.experts) {
            for (int r = qb * 8 + tid; r < min((qb + sets) * 8, p.rows); r += kGdThreads) p.y[static_cast<size_t>(z) * p.rows + r] = 0.f;
            return;
        }
        w += static_cast<size_t>(e) * p.rows * p.row_bytes;
        const int token = z / p.top_k, slot = z - token * p.top_k;
        x = p.x + (static_cast<size_t>(token) * p.slots + slot % p.slots) * p.k;
    }

    // ---- the stream (see qmv_dp.cu): copy h moves piece h * 32 + lane of the eight rows
    const uint32_t ring = xs + p.ring_at + warp * (kGdDepth * SLOT);
    struct {
        int set, part, left, ragged;
        uint32_t slot;
        int shift;               // 16 in the steps whose rows start in the middle of a sector (Q2_K), else 0
        const uint8_t *w;        // the octet's first row in the next step (warp-uniform)
        uint32_t ow[COPIES];     // this lane's pieces of it (rows beyond the matrix repeat its last one)
    } ahead;
    // A row lies in its slot at the offset inside a 32-byte sector that it has in memory (0 or 16: of an odd row if rows are an odd
    // number of 16-byte pieces, of every second step of Q2_K): halves of one sector that do not stay one fetch it twice.
    const int odd = static_cast<int>(p.row_bytes >> 4) & 1;
    int cc[COPIES], cr[COPIES];  // piece of the row and row of the octet, copy by copy
#pragma unroll
    for (int h = 0; h < COPIES; ++h) {
        const int pc = min(h * 32 + lane, 8 * PPR - 1);
        cr[h] = pc / PPR;
        cc[h] = pc - cr[h] * PPR;
    }
    auto open_ahead = [&]() {
        while (ahead.set >= sets) {
            ahead.set -= sets;
            ++ahead.part;
        }
        if (ahead.part >= p.parts) {
            ahead.left = 0;
            return;
        }
        const int step = ahead.part * p.spt, row0 = (qb + ahead.set) * 8;
        ahead.left = min(p.spt, p.steps - step);
        ahead.shift = FMT == 2 ? (step & 1) * 16 : 0;
        ahead.ragged = p.tail_pieces && step + ahead.left == p.steps ? 1 : 0;
        const int last = p.rows - 1 - row0;
#pragma unroll
        for (int h = 0; h < COPIES; ++h) ahead.ow[h] = static_cast<uint32_t>(min(cr[h], last) * static_cast<int>(p.row_bytes) + cc[h] * PIECE);
        ahead.w = w + static_cast<size_t>(row0) * p.row_bytes + static_cast<size_t>(step) * S::kRow;
    };
    auto fetch = [&]() {
        if (ahead.left > 0) {
            const bool ragged = ahead.left == ahead.ragged;  // pieces beyond the row's end: zeros
#pragma unroll
            for (int h = 0; h < COPIES; ++h) {
                if (8 * PPR % 32 != 0 && h == COPIES - 1 && lane >= 8 * PPR % 32) break;
                const uint32_t to = ahead.slot + cr[h] * S::kPitch + cc[h] * PIECE + ((cr[h] & odd) ? 16 - ahead.shift : ahead.shift);
                if (!ragged) {
                    gd_copy<PIECE>(to, ahead.w + ahead.ow[h]);
                } else {
                    const bool in = cc[h] < p.tail_pieces;
                    gd_copy<PIECE>(to, ahead.w + (ahead.ow[h] - (in ? 0 : cc[h] * PIECE)), in);
                }
            }
            ahead.w += S::kRow;
            if (FMT == 2) ahead.shift ^= 16;
            ahead.slot = ahead.slot == ring ? ring + SLOT : ring;
            if (--ahead.left == 0) {
                ahead.set += kGdWarps;
                open_ahead();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    ahead.set = warp;
    ahead.part = 0;
    ahead.slot = ring;
    open_ahead();
#pragma unroll
    for (int i = 0; i < kGdDepth; ++i) fetch();

    // ---- activations: an item is eight consecutive elements; the items of a sub-block are neighbouring lanes
    constexpr int IPS = FMT == 4 ? 4 : 2;  // items per sub-block
    const int ni = p.steps * 8 * S::kElems / 8;  // (a multiple of 32: whole warps)
    for (int i0 = tid; i0 < ni; i0 += 2 * kGdThreads) {
        float4 v[2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + u * kGdThreads;
            const bool in = i < p.k / 8;
            const float4 *src = reinterpret_cast<const float4 *>(x) + 2 * static_cast<size_t>(i);
            v[u][0] = in ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[u][1] = in ? __ldg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = i0 + u * kGdThreads;
            if (i >= ni) break;
            const float f[8] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w, v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
            float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
            uint32_t amax = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = max(amax, __float_as_uint(f[j]) & 0x7fffffffu);
#pragma unroll
            for (int off = 1; off < IPS; off <<= 1) {
                amax = max(amax, __shfl_xor_sync(0xffffffffu, amax, off));
                sum += __shfl_xor_sync(0xffffffffu, sum, off);
            }
            // E: biased exponent of the sub-block's largest magnitude, at least the one whose factor is a float (smaller sub-blocks keep
            // that grid); an infinity or NaN makes its factor NaN
            const uint32_t e0 = amax >> 23, e = max(e0, S::kGrid + 7u);
            const bool live = e0 < 255u;
            const float up = live ? __uint_as_float((254u + S::kGrid - e) << 23) : 0.f;  // 2^(kGrid - (E - 127))
            uint32_t digit[PLANES][8];  // the signed bytes of x_int, the highest first, each with its carry: digit q in byte PLANES - 1 - q of its word
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t xi = static_cast<uint32_t>(live ? __float2int_rn(f[j] * up) : 0);  // below 2^(kGrid + 1)
                digit[PLANES - 1][j] = xi;
                digit[PLANES - 2][j] = xi + 128u;
                digit[PLANES - 3][j] = xi + 32896u;
                if constexpr (PLANES == 4) digit[0][j] = xi + 8421504u;
            }
            auto pack = [&](int q, int at) {
                constexpr uint32_t kSel[4] = {0x0040, 0x0051, 0x0062, 0x0073};
                const uint32_t sel = kSel[PLANES - 1 - q];
                return __byte_perm(__byte_perm(digit[q][at], digit[q][at + 1], sel), __byte_perm(digit[q][at + 2], digit[q][at + 3], sel), 0x5410);
            };
            const int chunk = i / (S::kElems / 8), j = i - chunk * (S::kElems / 8);
            const uint32_t to = xs + (chunk >> 3) * (S::kXV * 128) + (chunk & 7) * 16;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int v_ = (j & 3) * 2 + h;  // packed word of these four elements; j / 4: the half or field of it
                if constexpr (PLANES == 4) {
                    // a vector per packed word and half (Q4_K) or field (Q2_K)
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to + ((FMT == 4 ? 2 : 4) * v_ + (j >> 2)) * 128), "r"(pack(0, 4 * h)),
                                 "r"(pack(1, 4 * h)), "r"(pack(2, 4 * h)), "r"(pack(3, 4 * h)) : "memory");
                } else {
#pragma unroll
                    for (int q = 0; q < 3; ++q) {
                        // Q4_K: word v of half s (low / high nibbles) at 6 (v & 1) + 3 s + q of its pair; Q2_K: word v of field f at 3 f + q
                        const int idx = FMT == 4 ? 6 * (v_ & 1) + 3 * (j >> 2) + q : 3 * (j >> 2) + q;
                        const int vec = FMT == 4 ? 3 * (v_ >> 1) + (idx >> 2) : 3 * v_ + (idx >> 2);
                        asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + vec * 128 + (idx & 3) * 4), "r"(pack(q, 4 * h)) : "memory");
                    }
                }
            }
            if (j % IPS == 0) {
                // Q4_K: sub-block j / 4 (its high nibbles carry 16); Q2_K: field f = j / 4 (it carries 4^f), half (j & 3) / 2
                const int sb = FMT == 4 ? j >> 2 : (j >> 2) * 2 + ((j & 3) >> 1);
                const uint32_t place = FMT == 4 ? 4u * (j >> 2) : 2u * (j >> 2);
                const float factor = __uint_as_float(live ? (e - S::kGrid - place) << 23 : 0x7fc00000u);
                asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(xf + (chunk * S::kSubs + sb) * 8), "f"(factor), "f"(sum) : "memory");
            }
        }
    }
    __syncthreads();

    // ---- the tasks of this warp; a lane's rows of an octet are sub and sub + 4
    uint32_t mask[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) mask[f] = FMT == 4 ? (0x0f0f0f0fu << (4 * (f & 1))) : (0x03030303u << (2 * f));
    int set = warp, prt = 0;
    uint32_t at = ring;
    while (true) {
        while (set >= sets) {
            set -= sets;
            ++prt;
        }
        if (prt >= p.parts) break;
        float acc[2] = {0.f, 0.f};
        const int end = min((prt + 1) * p.spt, p.steps);
        for (int step = prt * p.spt; step < end; ++step) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kGdDepth - 1) : "memory");
            __syncwarp();
            const uint32_t xp = xs + step * (S::kXV * 128) + sl * 16, fp = xf + (step * 8 + sl) * (S::kSubs * 8);
            const uint32_t row0 = at + sub * S::kPitch + (((sub & odd) ^ (FMT == 2 ? step & 1 : 0)) << 4);  // (sub + 4: the same offset)
            if constexpr (FMT == 4) {
                uint32_t cw[2][8], hd[2][4];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t blk = row0 + r * (4 * S::kPitch) + (sl >> 2) * 144;
                    gd_lds128(blk, hd[r]);
                    gd_lds128(blk + 16 + (sl & 3) * 32, cw[r]);
                    gd_lds128(blk + 32 + (sl & 3) * 32, cw[r] + 4);
                }
                int c[2][2][PLANES];  // [row][low, high nibbles][plane]
#pragma unroll
                for (int r = 0; r < 2; ++r)
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int q = 0; q < PLANES; ++q) c[r][s][q] = 0;
                if constexpr (PLANES == 4) {
#pragma unroll
                    for (int v = 0; v < 8; ++v)
#pragma unroll
                        for (int s = 0; s < 2; ++s) {
                            uint32_t xw[4];
                            gd_lds128(xp + (2 * v + s) * 128, xw);
#pragma unroll
                            for (int r = 0; r < 2; ++r)
#pragma unroll
                                for (int q = 0; q < 4; ++q) c[r][s][q] = gd_dp4a(cw[r][v] & mask[s], xw[q], c[r][s][q]);
                        }
                } else
#pragma unroll
                for (int vp = 0; vp < 4; ++vp) {
                    uint32_t xw[12];
#pragma unroll
                    for (int u = 0; u < 3; ++u) gd_lds128(xp + (3 * vp + u) * 128, xw + 4 * u);
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int o = 0; o < 2; ++o) {
                            const uint32_t wv = cw[r][2 * vp + o], lo = wv & mask[0], hi = wv & mask[1];
#pragma unroll
                            for (int q = 0; q < 3; ++q) {
                                c[r][0][q] = gd_dp4a(lo, xw[6 * o + q], c[r][0][q]);
                                c[r][1][q] = gd_dp4a(hi, xw[6 * o + 3 + q], c[r][1][q]);
                            }
                        }
                }
                float fs[4];  // factor and sum of the two sub-blocks
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(fs[0]), "=f"(fs[1]), "=f"(fs[2]), "=f"(fs[3]) : "r"(fp));
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float d, dmin;
                    gd_half2(hd[r][0], d, dmin);
                    // 6-bit scales and mins of sub-blocks 2j, 2j + 1 (quant.rs:88-96), two at a time
                    const int sh = 16 * (sl & 1);
                    const uint32_t a = hd[r][1] >> sh, b = hd[r][2] >> sh, t = hd[r][3] >> sh;
                    const bool low = (sl & 3) < 2;
                    const uint32_t sc2 = low ? a & 0x3f3fu : (t & 0x0f0fu) | ((a >> 2) & 0x3030u);
                    const uint32_t mn2 = low ? b & 0x3f3fu : ((t >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u);
                    float as = 0.f, am = 0.f;  // sums under the block's d and dmin
#pragma unroll
                    for (int s = 0; s < 2; ++s) {
                        const float val = gd_value<PLANES>(c[r][s]);
                        as = fmaf(static_cast<float>((sc2 >> (8 * s)) & 255u), val * fs[2 * s], as);
                        am = fmaf(static_cast<float>((mn2 >> (8 * s)) & 255u), fs[2 * s + 1], am);
                    }
                    acc[r] = fmaf(d, as, fmaf(-dmin, am, acc[r]));
                }
            } else {
                uint32_t cw[2][8], sc[2][2];
                float d[2], dmin[2], as[2] = {0.f, 0.f}, am[2] = {0.f, 0.f};  // sums under the block's d and dmin
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t blk = row0 + r * (4 * S::kPitch) + (sl >> 1) * 84;
#pragma unroll
                    for (int i = 0; i < 8; ++i) cw[r][i] = gd_lds32(blk + 16 + (sl & 1) * 32 + 4 * i);
                    sc[r][0] = gd_lds32(blk + (sl & 1) * 8);
                    sc[r][1] = gd_lds32(blk + (sl & 1) * 8 + 4);
                    gd_half2(gd_lds32(blk + 80), d[r], dmin[r]);
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    int c[2][4][PLANES];  // [row][field][plane] of a 16-element sub-block
#pragma unroll
                    for (int r = 0; r < 2; ++r)
#pragma unroll
                        for (int f = 0; f < 4; ++f)
#pragma unroll
                            for (int q = 0; q < PLANES; ++q) c[r][f][q] = 0;
#pragma unroll
                    for (int v = 4 * half; v < 4 * half + 4; ++v) {
                        if constexpr (PLANES == 4) {
#pragma unroll
                            for (int f = 0; f < 4; ++f) {
                                uint32_t xw[4];
                                gd_lds128(xp + (4 * v + f) * 128, xw);
#pragma unroll
                                for (int r = 0; r < 2; ++r)
#pragma unroll
                                    for (int q = 0; q < 4; ++q) c[r][f][q] = gd_dp4a(cw[r][v] & mask[f], xw[q], c[r][f][q]);
                            }
                            continue;
                        } else {
                        uint32_t xw[12];
#pragma unroll
                        for (int u = 0; u < 3; ++u) gd_lds128(xp + (3 * v + u) * 128, xw + 4 * u);
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int f = 0; f < 4; ++f) {
                                const uint32_t wf = cw[r][v] & mask[f];
#pragma unroll
                                for (int q = 0; q < 3; ++q) c[r][f][q] = gd_dp4a(wf, xw[3 * f + q], c[r][f][q]);
                            }
                        }
                    }
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        float factor, sum;
                        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(factor), "=f"(sum) : "r"(fp + (2 * f + half) * 8));
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const uint32_t byte = (sc[r][f >> 1] >> (16 * (f & 1) + 8 * half)) & 255u;  // scale byte 2 f + half
                            const float val = gd_value<PLANES>(c[r][f]);
                            as[r] = fmaf(static_cast<float>(byte & 15u), val * factor, as[r]);
                            am[r] = fmaf(static_cast<float>(byte >> 4), sum, am[r]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) acc[r] = fmaf(d[r], as[r], fmaf(-dmin[r], am[r], acc[r]));
            }
            __syncwarp();
            fetch();
            at = at == ring ? ring + SLOT : ring;
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float v = acc[r];
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (sl == 0) part[(set * 8 + r * 4 + sub) * p.parts + prt] = v;
        }
        set += kGdWarps;
    }
    __syncthreads();
    for (int i = tid; i < sets * 8; i += kGdThreads) {
        const int row = qb * 8 + i;
        if (row >= p.rows) break;
        float tot = 0.f;
        for (int k = 0; k < p.parts; ++k) tot += part[i * p.parts + k];
        p.y[static_cast<size_t>(z) * p.rows + row] = tot;
    }
}

struct GdPlan {
    bool ok;
    GdParams p;
    int smem, piece;
};

GdPlan gd_make_plan(int fmt, int64_t zs, int64_t rows, int64_t row_bytes, bool exact) {
    GdPlan pl{};
    const int block = fmt == 4 ? 144 : 84, blocks = fmt == 4 ? 2 : 4;
    const int64_t nb = row_bytes / block;
    if (row_bytes % block != 0 || nb < 1 || rows < 1 || rows > (1 << 26) || nb > (1 << 16)) return pl;
    GdParams &p = pl.p;
    p.row_bytes = row_bytes;
    p.rows = static_cast<int>(rows);
    p.k = static_cast<int>(nb * 256);
    p.steps = static_cast<int>((nb + blocks - 1) / blocks);
    pl.piece = row_bytes % 16 == 0 ? 16 : 4;
    p.tail_pieces = nb % blocks ? static_cast<int>(nb % blocks) * block / pl.piece : 0;
    p.octets = static_cast<int>((rows + 7) / 8);
    const int xv = (exact ? 4 : 3) * (fmt == 4 ? 4 : 8), subs = fmt == 4 ? 2 : 8;
    const int64_t fixed = static_cast<int64_t>(p.steps) * (xv * 128 + 8 * subs * 8);
    if (fixed > (1 << 20)) return pl;
    p.ring_at = static_cast<int>((fixed + 127) & ~127);
    p.part_at = p.ring_at + kGdWarps * kGdDepth * 8 * (fmt == 4 ? 320 : 352);
    // CTAs of one z: those that fill the SMs once over all z, never more than octets
    p.ctas = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(p.octets, sm_count() / zs)));
    int64_t bytes = 0;
    for (;; p.ctas = std::min(p.octets, 2 * p.ctas)) {
        p.base = p.octets / p.ctas;
        p.extra = p.octets % p.ctas;
        const int per = p.base + (p.extra ? 1 : 0);
        double best = 1e30;
        for (int parts = 1; parts <= std::min(p.steps, 64); ++parts) {
            const int spt = (p.steps + parts - 1) / parts;
            if ((p.steps + spt - 1) / spt != parts) continue;
            const double cost = ((per * parts + kGdWarps - 1) / kGdWarps) * (spt + 0.1) + 0.01 * parts;
            if (cost < best) {
                best = cost;
                p.parts = parts;
                p.spt = spt;
            }
        }
        if (exact) {
            // Cut by the length of a row alone: a row has the same bits whatever the matrix and the slots.  Rows whose sums of so many parts do not
            // fit are dealt to more CTAs, so that what fits depends on the length too.
            p.spt = (p.steps + 15) / 16;
            p.parts = (p.steps + p.spt - 1) / p.spt;
        }
        bytes = p.part_at + static_cast<int64_t>(per) * 8 * p.parts * 4;
        if (bytes <= max_smem_optin() - 2048) break;
        if (!exact || p.ctas == p.octets) return pl;
    }
    pl.smem = static_cast<int>(bytes);
    pl.ok = true;
    return pl;
}

bool gd_plan(int fmt, int64_t zs, int64_t rows, int64_t row_bytes, bool exact, GdPlan &out) {
    static thread_local PlanTable<GdPlan> table;
    bool known;
    GdPlan *e = table.find(zs, rows, (row_bytes << 12) | (static_cast<int64_t>(current_device()) << 4) | (exact ? 8 : 0) | fmt, known);
    if (!known) *e = gd_make_plan(fmt, zs, rows, row_bytes, exact);
    out = *e;
    return out.ok;
}

template <int FMT, int PIECE, int PLANES>
int gd_launch(cudaStream_t stream, const GdPlan &pl, int64_t zs) {
    LISA_TRY((allow_smem_of<gguf_dp_kernel<FMT, PIECE, PLANES>>()));
    LISA_TRY(launch_kernel(stream, static_cast<unsigned>(zs * pl.p.ctas), kGdThreads, pl.smem, 0, gguf_dp_kernel<FMT, PIECE, PLANES>, pl.p));
    count_launch();
    return LISA_OK;
}

}  // namespace

// The formats and shapes the kernel takes: Q4_K and Q2_K, one token, or up to 1024 (token, expert) slots; 16-byte
// aligned packed rows (Q2_K: 4-byte aligned ones too).  `exact`: four bytes an activation instead of three.
bool gguf_dp_supported(int format, const void *w, int64_t zs, int64_t rows, int64_t row_bytes, bool experts, bool exact) {
    if (format != LISA_GGUF_Q4_K && format != LISA_GGUF_Q2_K) return false;
    if (zs < 1 || zs > (experts ? 1024 : 1)) return false;
    GdPlan pl;
    if (!gd_plan(format == LISA_GGUF_Q4_K ? 4 : 2, zs, rows, row_bytes, exact, pl)) return false;
    return (reinterpret_cast<uintptr_t>(w) & static_cast<uintptr_t>(pl.piece - 1)) == 0;
}

int gguf_dp(cudaStream_t stream, int format, const uint8_t *w, int64_t experts, int64_t rows, int64_t row_bytes, const float *x, int64_t zs,
            int64_t slots, const int32_t *ids, int64_t top_k, float *y, bool exact) {
    GdPlan pl;
    const bool q4 = format == LISA_GGUF_Q4_K;
    if (!gd_plan(q4 ? 4 : 2, zs, rows, row_bytes, exact, pl)) return fail(LISA_ERR_UNSUPPORTED, "gguf_dp: shape not supported");
    pl.p.w = w;
    pl.p.x = x;
    pl.p.y = y;
    pl.p.ids = ids;
    pl.p.experts = static_cast<int>(experts);
    pl.p.slots = static_cast<int>(slots);
    pl.p.top_k = static_cast<int>(top_k);
    if (exact) {
        if (q4) return gd_launch<4, 16, 4>(stream, pl, zs);
        return pl.piece == 16 ? gd_launch<2, 16, 4>(stream, pl, zs) : gd_launch<2, 4, 4>(stream, pl, zs);
    }
    if (q4) return gd_launch<4, 16, 3>(stream, pl, zs);
    return pl.piece == 16 ? gd_launch<2, 16, 3>(stream, pl, zs) : gd_launch<2, 4, 3>(stream, pl, zs);
}

}  // namespace lisa
