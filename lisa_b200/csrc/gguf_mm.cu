// GGUF K-quant matvec on mma.sync, for two tokens and more (and for one where gguf_dp.cu's grid is not asked for), with f16 operands: f32 activations and output.
//   y[z, r] = sum_k x[z, k] * W[e(z), r, k],  Q4_K and Q2_K blocks (crates/lisa-gguf/src/quant.rs:64-101)
// (deepseek41::packed_matvec, crates/lisa-mlx/src/models/deepseek41.rs:93-283; its Metal kernels crates/lisa-mlx/src/shaders/deepseek41/iq.metal:1130-1363).
//
// Operands without loss: a code in the mantissa of 1024 (one LOP3) goes through one f16 multiply-add with its sub-block's integer scale, divided by
// the code's place in the byte: q * scale exactly (at most ten bits); so all codes of a 256-element block meet one scale, and d, dmin
// follow per block in f32.  An f32 activation, normalised by a power of two per block, is the sum of three f16 (33 bits): three of
// the MMA's columns per token.  The minima are one more MMA per block against the sums of sixteen activations.
//
// Sums: an MMA aligns its products and its accumulator to the largest of them by its exponent field and cuts what is below some 24 bits.  So
// operands are normal numbers (with codes as subnormals, which the products' exponents do not tell from numbers near 2^-14, the sums of Q2_K
// lost five bits), and an accumulator takes two MMAs, 32 products; everything else is added in f32.  Relative error (2-norm) on Gaussian
// activations, Q4_K / Q2_K, 1208 x 1280, four tokens: 1.1e-7 / 0.8e-7 (one accumulator a block 2.9e-7 / 1.1e-7, the warp-per-row kernel
// 1.0e-7 / 1.0e-7), for 10 to 20 % of the time of a launch.
//
// What bounds it: per code 5/8 (4/8 at 2 bits) of an operation of the half-rate pipe and half a packed multiply-add, 0.055 warp
// instructions in all, against three dot products of four bytes (0.75 operations and 0.09 instructions) of the byte form in
// gguf_dp.cu, which takes a pass over the weights per token (and is the faster one for one token: it has less to stage).  Structure, streams and clusters are those of qmv_mm.cu: a warp
// takes tasks of sixteen rows and a run of steps (two Q4_K or four Q2_K blocks) through its own ring of asynchronous copies.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.h"

namespace lisa {

namespace {

constexpr int kGmThreads = 512, kGmWarps = kGmThreads / 32, kGmDepth = 2;
// The steps of a row are cut into up to eight leaves, by its length alone, and a row's sum is the balanced tree of theirs: clusters and tasks take
// whole subtrees, so that a result has the same bits whatever the rows of the matrix, the tokens of the call and the launch.
constexpr int gm_leaves(int steps) { return steps >= 8 ? 8 : steps >= 4 ? 4 : steps >= 2 ? 2 : 1; }

struct GmParams {
    const uint8_t *w;
    const float *x;
    float *y;
    long long row_bytes;
    int rows, k, blocks;     // rows of the matrix; k; 256-element blocks of a row
    int steps, leaves, splits, parts, warps;
    int shares, base, extra;  // shares of the 16-row tiles per z; tiles of a share (the first `extra` one more)
    int tail_pieces;          // pieces of a row in its last step where that is ragged, else 0
    int tokens;               // tokens of the call (dense form)
    int cols;                 // 3 * tokens of a launch column set
    int sums_at, fac_at, ring_at, part_at;
};

template <int B>
__device__ __forceinline__ void gm_copy(uint32_t dst, const void *src, bool in) {
    if constexpr (B == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %3, %2;" ::"r"(dst), "l"(src), "r"(in ? B : 0), "n"(B) : "memory");
}
__device__ __forceinline__ void gm_lds128(uint32_t addr, uint32_t *r) {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ uint32_t gm_lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void gm_half2(uint32_t v, float &lo, float &hi) {
    asm("{ .reg .b16 l, h; mov.b32 {l, h}, %2; cvt.f32.f16 %0, l; cvt.f32.f16 %1, h; }" : "=f"(lo), "=f"(hi) : "r"(v));
}
__device__ __forceinline__ uint32_t gm_mul(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t gm_fma(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t gm_and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t gm_f16(float v) {
    uint16_t h;
    asm("cvt.rn.f16.f32 %0, %1;" : "=h"(h) : "f"(v));
    return h;
}
__device__ __forceinline__ float gm_f32(uint32_t h) {
    float v;
    asm("cvt.f32.f16 %0, %1;" : "=f"(v) : "h"(static_cast<uint16_t>(h)));
    return v;
}
__device__ __forceinline__ void gm_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t gm_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void gm_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void gm_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void gm_st_cluster(float *local, uint32_t rank, float v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// FMT 4: Q4_K, a step is two blocks of a row; FMT 2: Q2_K, four.  A slot's row pitch keeps whole sectors and room for 16 bytes of offset, and
// spreads the reads of a quarter warp (two fragment rows, four 16-byte pieces each) over all banks where the second of the two rows is the
// next one (Q4_K) or the next but one (Q2_K): `row` is the matrix row of fragment row g.
template <int FMT>
struct GmShape {
    static constexpr int kBlock = FMT == 4 ? 144 : 84;
    static constexpr int kBlocks = FMT == 4 ? 2 : 4;
    static constexpr int kRow = kBlock * kBlocks;        // 288 / 336
    static constexpr int kPitch = FMT == 4 ? 320 : 352;
    static constexpr int kSlot = 16 * kPitch;
    __device__ static __forceinline__ int row(int g) { return FMT == 4 ? g : (g & 4) | ((g & 1) << 1) | ((g >> 1) & 1); }
};

// NT: column tiles (three columns a token); PIECE: bytes of a copy; CL: a cluster of CTAs divides the row's steps
template <int FMT, int PIECE, int NT, bool CL>
__global__ void __launch_bounds__(kGmThreads, 1) gguf_mm_kernel(const GmParams p) {
    using S = GmShape<FMT>;
    constexpr int PPR = S::kRow / PIECE, COPIES = 16 * PPR / 32 + (16 * PPR % 32 ? 1 : 0);
    extern __shared__ __align__(128) uint8_t gm_smem[];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int g = lane >> 2, t = lane & 3;
    const int splits = CL ? p.splits : 1, rank = CL ? static_cast<int>(gm_cluster_rank()) : 0;
    const int job = static_cast<int>(blockIdx.x) / splits, z = job / p.shares, share = job - z * p.shares;
    const int qb = share * p.base + min(share, p.extra), tiles = p.base + (share < p.extra ? 1 : 0);
    const int s0 = CL ? rank * p.steps / splits : 0, steps = CL ? (rank + 1) * p.steps / splits - s0 : p.steps;
    const int parts = p.parts, pieces = splits * parts;  // of all CTAs of the row: 1, 2, 4 or 8
    const int cols = p.cols, set_tokens = cols / 3, ntok = min(set_tokens, p.tokens - z * set_tokens);
    const float *x = p.x + static_cast<size_t>(z) * set_tokens * p.k;
    float *y = p.y + static_cast<size_t>(z) * set_tokens * p.rows;
    if (CL) gm_cluster_arrive();
    const uint32_t frag = smem_u32(gm_smem), sums = frag + p.sums_at, fac = frag + p.fac_at;
    float *part = reinterpret_cast<float *>(gm_smem + p.part_at);  // [rows of the share][pieces][tokens], in the first CTA
    const uint32_t ring = frag + p.ring_at + warp * kGmDepth * S::kSlot;

    // ---- the stream (see qmv_mm.cu): copy h moves piece h * 32 + lane of the sixteen rows.  With 16-byte pieces a row keeps the offset
    // inside its 32-byte sector that it has in memory (halves of a sector that part ways are fetched twice).
    const int odd = PIECE == 16 ? static_cast<int>(p.row_bytes >> 4) & 1 : 0;
    struct {
        int set, part, left, ragged, shift;
        uint32_t slot;
        const uint8_t *w;
        uint32_t ow[COPIES <= 12 ? COPIES : 1];
        int last;
    } ahead{};
    auto piece = [&](int h, int &r, int &c) {
        const int i = min(h * 32 + lane, 16 * PPR - 1);
        r = i / PPR;
        c = i - r * PPR;
    };
    auto open_ahead = [&]() {
        while (ahead.set >= tiles) {
            ahead.set -= tiles;
            ++ahead.part;
        }
        if (ahead.part >= parts) {
            ahead.left = 0;
            return;
        }
        const int at = rank * parts + ahead.part, step = at * p.steps / pieces, row0 = (qb + ahead.set) * 16;
        ahead.left = (at + 1) * p.steps / pieces - step;  // (at least one: pieces <= steps)
        ahead.ragged = p.tail_pieces && step + ahead.left == p.steps ? 1 : 0;
        ahead.shift = PIECE == 16 && FMT == 2 ? (step & 1) * 16 : 0;
        ahead.last = p.rows - 1 - row0;
        ahead.w = p.w + static_cast<size_t>(row0) * p.row_bytes + static_cast<size_t>(step) * S::kRow;
        if constexpr (COPIES <= 12) {
#pragma unroll
            for (int h = 0; h < COPIES; ++h) {
                int r, c;
                piece(h, r, c);
                ahead.ow[h] = static_cast<uint32_t>(min(r, ahead.last) * static_cast<int>(p.row_bytes) + c * PIECE);
            }
        }
    };
    auto fetch = [&]() {
        if (ahead.left > 0) {
            const bool ragged = ahead.left == ahead.ragged;  // pieces beyond the row's end: zeros
#pragma unroll
            for (int h = 0; h < COPIES; ++h) {
                if (16 * PPR % 32 != 0 && h == COPIES - 1 && lane >= 16 * PPR % 32) break;
                int r, c;
                piece(h, r, c);
                const uint32_t from = COPIES <= 12 ? ahead.ow[COPIES <= 12 ? h : 0] : static_cast<uint32_t>(min(r, ahead.last) * static_cast<int>(p.row_bytes) + c * PIECE);
                const bool in = !ragged || c < p.tail_pieces;
                gm_copy<PIECE>(ahead.slot + r * S::kPitch + c * PIECE + ((r & odd) ? 16 - ahead.shift : ahead.shift), ahead.w + (from - (in ? 0 : c * PIECE)), in);
            }
            ahead.w += S::kRow;
            if (PIECE == 16 && FMT == 2) ahead.shift ^= 16;
            ahead.slot = ahead.slot == ring ? ring + S::kSlot : ring;
            if (--ahead.left == 0) {
                ahead.set += p.warps;
                open_ahead();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    ahead.set = warp;
    ahead.slot = ring;
    if (warp < p.warps) open_ahead();
#pragma unroll
    for (int i = 0; i < kGmDepth; ++i) fetch();

    // ---- activations: a warp takes a (block, token), a lane eight consecutive elements of it
    const int b0 = s0 * S::kBlocks, nb = steps * S::kBlocks;  // blocks of this CTA (the last step's may lie beyond the row: zeros)
    const uint32_t blk_bytes = 512u * cols, sum_bytes = 32u * cols;
    for (int it = warp; it < nb * ntok; it += 2 * kGmWarps) {
        float4 v[2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = it + u * kGmWarps, tok = i / nb, b = i - tok * nb;
            const bool in = i < nb * ntok && b0 + b < p.blocks;
            const float4 *src = reinterpret_cast<const float4 *>(x + static_cast<size_t>(tok) * p.k + static_cast<size_t>(b0 + b) * 256) + 2 * lane;
            v[u][0] = in ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[u][1] = in ? __ldg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int i = it + u * kGmWarps;
            if (i >= nb * ntok) break;
            const int tok = i / nb, b = i - tok * nb;
            const float f[8] = {v[u][0].x, v[u][0].y, v[u][0].z, v[u][0].w, v[u][1].x, v[u][1].y, v[u][1].z, v[u][1].w};
            float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            uint32_t amax = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) amax = max(amax, __float_as_uint(f[j]) & 0x7fffffffu);
            // E: biased exponent of the block's largest magnitude, at least the one whose factor is a float (smaller blocks keep that
            // scale); an infinity or NaN makes its factor NaN
            const uint32_t e0 = __reduce_max_sync(0xffffffffu, amax) >> 23, e = max(e0, 14u);
            const bool live = e0 < 255u;
            const float up = live ? __uint_as_float((267u - e) << 23) : 0.f;  // 2^(13 - (E - 127))
            uint32_t h[3][8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float xn = f[j] * up;
                h[0][j] = gm_f16(xn);
                const float r1 = xn - gm_f32(h[0][j]);
                h[1][j] = gm_f16(r1);
                h[2][j] = gm_f16(r1 - gm_f32(h[1][j]));
            }
            const int byte = 8 * (lane & 3), sub = FMT == 4 ? (lane >> 2) & 1 : (lane >> 2) & 3;  // sub: nibble, or 2-bit field
            const int c = FMT == 4 ? lane >> 3 : lane >> 4;                                       // 32-byte run of the codes
            const int tt = FMT == 4 ? (c & 1) * 2 + (byte >> 4) : c * 2 + (byte >> 4);            // the fragment lane of these codes
            const int word = (FMT == 4 ? (c >> 1) * 4 : 0) + (byte & 15) / 4;                     // its words `word` and `word` + 1
#pragma unroll
            for (int pl = 0; pl < 3; ++pl) {
                const int col = tok * 3 + pl;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int vec = FMT == 4 ? word + q : 2 * (word + q) + (sub >> 1);
                    const uint32_t to = frag + b * blk_bytes + ((vec * cols + col) * 4 + tt) * 16 + (sub & 1) * 8;
                    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(to), "r"(h[pl][4 * q] | (h[pl][4 * q + 2] << 16)),
                                 "r"(h[pl][4 * q + 1] | (h[pl][4 * q + 3] << 16)) : "memory");
                }
            }
            if ((lane & 1) == 0) {
                // sums of sixteen, less 2^4; half word: (first, second) sub-block of the lane's low and high pair
                const float sn = sum * up * 0.0625f;
                uint32_t hs[3];
                hs[0] = gm_f16(sn);
                const float r1 = sn - gm_f32(hs[0]);
                hs[1] = gm_f16(r1);
                hs[2] = gm_f16(r1 - gm_f32(hs[1]));
                const int at = FMT == 4 ? (c >> 1) * 4 + sub * 2 : sub * 2;
#pragma unroll
                for (int pl = 0; pl < 3; ++pl)
                    asm volatile("st.shared.u16 [%0], %1;" ::"r"(sums + b * sum_bytes + ((tok * 3 + pl) * 4 + tt) * 8 + at), "h"(static_cast<uint16_t>(hs[pl])) : "memory");
                if (lane == 0) {
                    const float factor = __uint_as_float(live ? (e - 13u) << 23 : 0x7fc00000u);
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(fac + (b * (cols / 3) + tok) * 4), "f"(factor) : "memory");
                }
            }
        }
    }
    __syncthreads();
    if (CL) gm_cluster_wait();  // the first CTA of the cluster runs: its shared memory takes the others' partial sums

    // ---- the tasks of this warp
    uint32_t mk[4], magic;
#pragma unroll
    for (int i = 0; i < 4; ++i) asm volatile("mov.u32 %0, %1;" : "=r"(mk[i]) : "r"(FMT == 4 ? (0x000f000fu << (4 * (i & 1))) : (0x00030003u << (2 * i))));
    asm volatile("mov.u32 %0, 0x64006400;" : "=r"(magic));  // (1024, 1024)
    // fragment column g of tile n is column min(8 n + g, cols - 1): the rest repeats the last one and is not stored
    uint32_t bcol[NT], scol[NT];
    uint32_t fcol[NT][2];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int col = min(8 * n + g, cols - 1);
        bcol[n] = frag + (col * 4 + t) * 16;
        scol[n] = sums + (col * 4 + t) * 8;
#pragma unroll
        for (int j = 0; j < 2; ++j) fcol[n][j] = fac + min(8 * n + 2 * t + j, cols - 1) / 3 * 4;
    }
    const int rg = S::row(g);
    int set = warp, prt = 0;
    uint32_t at = ring;
    while (warp < p.warps) {
        while (set >= tiles) {
            set -= tiles;
            ++prt;
        }
        if (prt >= parts) break;
        // A lane's sums of the piece: rows g, g + 8 of tokens t, t + 4.  tree[l]: the subtree of 2^l leaves that waits for its right half, at the end the
        // piece (in local memory, by runtime indices: registers are short in the loop over the steps).
        constexpr int LT = (8 * NT / 3 + 3) / 4;
        float tree[4][LT * 2];
        const int leaves = p.leaves / pieces, leaf0 = (rank * parts + prt) * leaves;
        int step = leaf0 * p.steps / p.leaves - s0;
#pragma unroll 1
        for (int leaf = 0; leaf < leaves; ++leaf) {
            float acc[NT][4];  // rows g, g + 8 x columns 2t, 2t + 1
#pragma unroll
            for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
            const int end = (leaf0 + leaf + 1) * p.steps / p.leaves - s0;
#pragma unroll 1
            for (; step < end; ++step) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kGmDepth - 1) : "memory");
                __syncwarp();
                const uint32_t at_odd = ((rg & odd) ^ (PIECE == 16 && FMT == 2 ? (s0 + step) & 1 : 0)) << 4;  // (rows 8 apart: the same offset)
                const uint32_t r0 = at + rg * S::kPitch + at_odd;
#pragma unroll(FMT == 4 ? 1 : 4)
                for (int b = 0; b < S::kBlocks; ++b) {
                    const uint32_t bi = static_cast<uint32_t>(step * S::kBlocks + b);
                    constexpr int WORDS = FMT == 4 ? 8 : 4;
                    uint32_t cw[2][WORDS], mn[2][2], dm[2];
                    uint32_t sc[2][4], off[2][4];  // f16x2 scales of the lane's four sub-blocks, divided by their places; -1024 times that
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const uint32_t blk = r0 + r * (8 * S::kPitch) + b * S::kBlock;
                        uint32_t pair[2];
                        if constexpr (FMT == 4) {
                            uint32_t hd[4];
                            gm_lds128(blk, hd);
                            gm_lds128(blk + 16 + 16 * t, cw[r]);
                            gm_lds128(blk + 80 + 16 * t, cw[r] + 4);
                            dm[r] = hd[0];
                            // 6-bit scales and mins (quant.rs:88-96) of sub-blocks 2 (t / 2) + {0, 1} and 4 + 2 (t / 2) + {0, 1}
                            const int sh = 16 * (t >> 1);
                            const uint32_t a = hd[1] >> sh, m = hd[2] >> sh, hi = hd[3] >> sh;
                            pair[0] = __byte_perm(a & 0x3f3fu, magic, 0x5150);
                            pair[1] = __byte_perm((hi & 0x0f0fu) | ((a >> 2) & 0x3030u), magic, 0x5150);
                            mn[r][0] = gm_fma(__byte_perm(m & 0x3f3fu, magic, 0x5150), 0x3c003c00u, 0xe400e400u);
                            mn[r][1] = gm_fma(__byte_perm(((hi >> 4) & 0x0f0fu) | ((m >> 2) & 0x3030u), magic, 0x5150), 0x3c003c00u, 0xe400e400u);
                            // (1024 + s) - 1024, the second of a pair (high nibbles) divided by 16
#pragma unroll
                            for (int i = 0; i < 2; ++i) pair[i] = gm_fma(pair[i], 0x2c003c00u, 0xd400e400u);
                        } else {
                            // the block's codes start at word 4 + 21 b of the row: aligned vectors, the lane's four words in two of them
                            constexpr int kAligned[4] = {16, 96, 176, 256}, kWord[4] = {0, 1, 2, 3};
                            uint32_t v[8];
                            const uint32_t vec = r0 + r * (8 * S::kPitch) + kAligned[b] + 16 * t;
                            gm_lds128(vec, v);
                            if (kWord[b]) gm_lds128(vec + 16, v + 4);
#pragma unroll
                            for (int i = 0; i < 4; ++i) cw[r][i] = v[kWord[b] + i];
                            dm[r] = gm_lds32(blk + 80);
                            const int sh = 8 * (t & 1);
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                const uint32_t s = gm_lds32(blk + 8 * (t >> 1) + 4 * i) >> sh;  // scale bytes of fields 2 i, 2 i + 1
                                pair[i] = (s & 0x000f000fu) | 0x64006400u;
                                mn[r][i] = gm_fma(((s >> 4) & 0x000f000fu) | 0x64006400u, 0x3c003c00u, 0xe400e400u);
                            }
                            pair[0] = gm_fma(pair[0], 0x34003c00u, 0xdc00e400u);  // (s, s / 4)
                            pair[1] = gm_fma(pair[1], 0x24002c00u, 0xcc00d400u);  // (s / 16, s / 64)
                        }
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            sc[r][2 * i] = __byte_perm(pair[i], pair[i], 0x1010);
                            sc[r][2 * i + 1] = __byte_perm(pair[i], pair[i], 0x3232);
                            off[r][2 * i] = gm_mul(sc[r][2 * i], 0xe400e400u);
                            off[r][2 * i + 1] = gm_mul(sc[r][2 * i + 1], 0xe400e400u);
                        }
                    }
                    float cm[NT][4], total[NT][4];
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) cm[n][i] = total[n][i] = 0.f;
                        uint32_t bs[2];
                        asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(bs[0]), "=r"(bs[1]) : "r"(scol[n] + bi * sum_bytes));
                        gm_mma(cm[n], mn[0][0], mn[1][0], mn[0][1], mn[1][1], bs[0], bs[1]);
                    }
#pragma unroll
                    for (int v = 0; v < 8; ++v) {
                        // Q4_K: word v, low and high nibbles; Q2_K: word v / 2, fields 2 (v % 2) and + 1
                        const int wi = FMT == 4 ? v : v >> 1, f0 = FMT == 4 ? 0 : 2 * (v & 1), s_ = FMT == 4 ? 2 * (v >> 2) : f0;
                        uint32_t a[2][2][2];  // [row][field][bytes 0|2, 1|3]
#pragma unroll
                        for (int r = 0; r < 2; ++r)
#pragma unroll
                            for (int f = 0; f < 2; ++f) {
                                a[r][f][0] = gm_fma(gm_and_or(cw[r][wi], mk[f0 + f], magic), sc[r][s_ + f], off[r][s_ + f]);
                                a[r][f][1] = gm_fma(gm_and_or(cw[r][wi] >> 8, mk[f0 + f], magic), sc[r][s_ + f], off[r][s_ + f]);
                            }
#pragma unroll
                        for (int n = 0; n < NT; ++n) {
                            float c[4] = {0.f, 0.f, 0.f, 0.f};
                            uint32_t bf[4];
                            gm_lds128(bcol[n] + bi * blk_bytes + v * (cols * 64), bf);
                            gm_mma(c, a[0][0][0], a[1][0][0], a[0][0][1], a[1][0][1], bf[0], bf[1]);
                            gm_mma(c, a[0][1][0], a[1][1][0], a[0][1][1], a[1][1][1], bf[2], bf[3]);
#pragma unroll
                            for (int i = 0; i < 4; ++i) total[n][i] += c[i];
                        }
                    }
                    float d[2], dmin[2];
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        gm_half2(dm[r], d[r], dmin[r]);
                        dmin[r] *= -16.f;  // the sums' 2^4
                    }
#pragma unroll
                    for (int n = 0; n < NT; ++n) {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            float f;
                            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(f) : "r"(fcol[n][j] + bi * (cols / 3 * 4)));
#pragma unroll
                            for (int r = 0; r < 2; ++r) acc[n][2 * r + j] = fmaf(fmaf(d[r], total[n][2 * r + j], dmin[r] * cm[n][2 * r + j]), f, acc[n][2 * r + j]);
                        }
                    }
                }
                __syncwarp();
                fetch();
                at = at == ring ? ring + S::kSlot : ring;
            }
            // the three planes of a token lie in up to three lanes of the fragment row: their sum to lane (token % 4)
            float sum[LT * 2];
#pragma unroll
            for (int k = 0; k < 8 * NT / 3; ++k) {
                if (k >= ntok) break;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    float v[3];
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) {
                        const int col = 3 * k + pl;  // tile col / 8, lane (col % 8) / 2, its value col % 2
                        v[pl] = __shfl_sync(0xffffffffu, acc[col / 8][2 * r + (col & 1)], (lane & ~3) | ((col & 7) >> 1));
                    }
                    if (t == (k & 3)) sum[k / 4 * 2 + r] = v[0] + (v[1] + v[2]);
                }
            }
            int level = 0;
#pragma unroll 1
            for (; (leaf >> level) & 1; ++level)
#pragma unroll
                for (int i = 0; i < LT * 2; ++i) sum[i] = tree[level][i] + sum[i];
#pragma unroll
            for (int i = 0; i < LT * 2; ++i) tree[level][i] = sum[i];
        }
        const int top = 31 - __clz(leaves);
#pragma unroll
        for (int i = 0; i < LT; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r)
                if (4 * i + t < ntok) {
                    float *to = part + ((set * 16 + r * 8 + rg) * pieces + rank * parts + prt) * set_tokens + 4 * i + t;
                    if (CL) gm_st_cluster(to, 0, tree[top][i * 2 + r]);
                    else *to = tree[top][i * 2 + r];
                }
        set += p.warps;
    }
    if (CL) {
        gm_cluster_arrive();
        if (rank != 0) return;
        gm_cluster_wait();
    } else {
        __syncthreads();
    }

    // ---- the top of the tree; store
    for (int i = tid; i < tiles * 16 * ntok; i += kGmThreads) {
        const int tok = i / (tiles * 16), rr = i - tok * (tiles * 16), row = qb * 16 + rr;
        if (row >= p.rows) continue;
        const float *v = part + rr * pieces * set_tokens + tok;
        auto two = [&](int i) { return v[i * set_tokens] + v[(i + 1) * set_tokens]; };
        float tot;
        if (pieces == 1) tot = v[0];
        else if (pieces == 2) tot = two(0);
        else if (pieces == 4) tot = two(0) + two(2);
        else tot = (two(0) + two(2)) + (two(4) + two(6));
        y[static_cast<size_t>(tok) * p.rows + row] = tot;
    }
}

struct GmPlan {
    bool ok;
    GmParams p;
    int smem, piece, grid, nt;
};

// Clusters of `splits` CTAs of a whole SM each that the device runs at a time.
int gm_cluster_limit(int splits) {
    static std::atomic<int> known[64][4];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int> &slot = known[dev & 63][splits == 2 ? 0 : splits == 4 ? 1 : 2];
    int v = slot.load(std::memory_order_relaxed);
    if (v > 0) return v;
    v = std::max(1, sm_count() / splits - 4);  // (where the query fails)
    if (allow_smem_of<gguf_mm_kernel<4, 16, 1, true>>() == LISA_OK) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(sm_count() / splits * splits);
        cfg.blockDim = dim3(kGmThreads);
        cfg.dynamicSmemBytes = max_smem_optin() - 2048;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, gguf_mm_kernel<4, 16, 1, true>, &cfg) == cudaSuccess && n > 0) v = n;
        else cudaGetLastError();
    }
    slot.store(v, std::memory_order_relaxed);
    return v;
}

GmPlan gm_make_plan(int fmt, int64_t tokens, int64_t rows, int64_t row_bytes) {
    GmPlan pl{};
    const int block = fmt == 4 ? 144 : 84, blocks = fmt == 4 ? 2 : 4, slot = 16 * (fmt == 4 ? 320 : 352);
    const int64_t nb = row_bytes / block;
    if (row_bytes % block != 0 || nb < 1 || rows < 1 || rows > (1 << 26) || nb > (1 << 16)) return pl;
    GmParams &p = pl.p;
    p.row_bytes = row_bytes;
    p.rows = static_cast<int>(rows);
    p.blocks = static_cast<int>(nb);
    p.k = static_cast<int>(nb * 256);
    p.steps = static_cast<int>((nb + blocks - 1) / blocks);
    p.leaves = gm_leaves(p.steps);
    pl.piece = row_bytes % 16 == 0 ? 16 : row_bytes % 8 == 0 ? 8 : 4;
    p.tail_pieces = nb % blocks ? static_cast<int>(nb % blocks) * block / pl.piece : 0;
    const int64_t tiles = (rows + 15) / 16;
    p.tokens = static_cast<int>(tokens);
    double best = 1e30;
    // Tokens of a column set: eight, five or two fill three, two or one column tiles; more tokens run as several sets of nearly the same
    // size side by side (their weights meet in L2).  Single tokens, and any number of CTAs, where nothing else fits: what fits depends on the
    // length of a row alone.
    for (int most_tokens : {8, 5, 2, 1}) {
        const int64_t zs = (tokens + most_tokens - 1) / most_tokens, set = (tokens + zs - 1) / zs;
        const int64_t cols = 3 * set;
        const int nt = static_cast<int>((cols + 7) / 8);
        const bool last = most_tokens == 1;
        if (last && best < 1e30) break;
        for (int splits : {1, 2, 4, 8}) {
            if (splits > p.leaves) continue;
            const int64_t at_once = splits == 1 ? sm_count() : gm_cluster_limit(splits);
            const int most = (p.steps + splits - 1) / splits;
            const int64_t frag = static_cast<int64_t>(most) * blocks;
            const int64_t sums_at = frag * 512 * cols, fac_at = sums_at + frag * 32 * cols, ring_at = (fac_at + frag * set * 4 + 127) & ~static_cast<int64_t>(127);
            if (ring_at > max_smem_optin()) continue;
            // CTAs that run at a time, and two or four times as many, whose partial sums take less room
            int64_t shares = std::min<int64_t>(tiles, std::max<int64_t>(1, at_once / zs));
            for (int turn = 0;; ++turn, shares = std::min(tiles, 2 * shares)) {
                const int64_t per = (tiles + shares - 1) / shares, rounds = (shares * zs + at_once - 1) / at_once;
                bool fits = false;
                for (int warps : {16, 12, 8}) {
                    // time of a step: against sixteen warps and one column tile (three of them spill)
                    const double pace = (warps == 16 ? 1.0 : warps == 12 ? 0.85 : 0.7) * (nt == 1 ? 1.0 : nt == 2 ? 1.25 : 2.2);
                    for (int parts = 1; parts * splits <= p.leaves; parts *= 2) {
                        const int64_t part_at = ring_at + static_cast<int64_t>(warps) * kGmDepth * slot;
                        const int64_t bytes = part_at + per * 16 * splits * parts * set * 4;
                        if (bytes > max_smem_optin() - 2048) continue;
                        fits = true;
                        // ... the staging of the activations (about a fifth of a step per block and token and warp), and five steps for a CTA's start
                        const double cost = rounds * (((per * parts + warps - 1) / warps) * (static_cast<double>(most) / parts + 0.1) * pace + 0.2 * frag * static_cast<double>(set) / kGmWarps + 5.0) +
                                            0.01 * parts + (splits > 1 ? 0.5 * splits : 0);
                        if (cost < best) {
                            best = cost;
                            p.cols = static_cast<int>(cols);
                            pl.nt = nt;
                            p.splits = splits;
                            p.warps = warps;
                            p.parts = parts;
                            p.shares = static_cast<int>(shares);
                            p.base = static_cast<int>(tiles / shares);
                            p.extra = static_cast<int>(tiles % shares);
                            p.sums_at = static_cast<int>(sums_at);
                            p.fac_at = static_cast<int>(fac_at);
                            p.ring_at = static_cast<int>(ring_at);
                            p.part_at = static_cast<int>(part_at);
                            pl.smem = static_cast<int>(bytes);
                            pl.grid = static_cast<int>(zs * shares * splits);
                        }
                    }
                }
                if (shares == tiles || (turn >= 2 && (fits || !last))) break;
            }
        }
    }
    pl.ok = best < 1e30;
    return pl;
}

bool gm_plan(int fmt, int64_t tokens, int64_t rows, int64_t row_bytes, GmPlan &out) {
    static thread_local PlanTable<GmPlan> table;
    bool known;
    GmPlan *e = table.find(tokens, rows, (row_bytes << 12) | (static_cast<int64_t>(current_device()) << 4) | fmt, known);
    if (!known) *e = gm_make_plan(fmt, tokens, rows, row_bytes);
    out = *e;
    return out.ok;
}

template <int FMT, int PIECE, int NT, bool CL>
int gm_launch_one(cudaStream_t stream, const GmPlan &pl) {
    LISA_TRY((allow_smem_of<gguf_mm_kernel<FMT, PIECE, NT, CL>>()));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kGmThreads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = pl.p.splits;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CL ? 1 : 0;
    LISA_CUDA_TRY(cudaLaunchKernelEx(&cfg, gguf_mm_kernel<FMT, PIECE, NT, CL>, pl.p));
    count_launch();
    return LISA_OK;
}

template <int FMT, int PIECE>
int gm_launch(cudaStream_t stream, const GmPlan &pl) {
    const bool cl = pl.p.splits > 1;
    if (pl.nt == 1) return cl ? gm_launch_one<FMT, PIECE, 1, true>(stream, pl) : gm_launch_one<FMT, PIECE, 1, false>(stream, pl);
    if (pl.nt == 2) return cl ? gm_launch_one<FMT, PIECE, 2, true>(stream, pl) : gm_launch_one<FMT, PIECE, 2, false>(stream, pl);
    return cl ? gm_launch_one<FMT, PIECE, 3, true>(stream, pl) : gm_launch_one<FMT, PIECE, 3, false>(stream, pl);
}

}  // namespace

// Q4_K and Q2_K, any number of tokens (matrices that the tensor-core product does not take come here with all of theirs).
bool gguf_mm_supported(int format, const void *w, int64_t tokens, int64_t rows, int64_t row_bytes) {
    if ((format != LISA_GGUF_Q4_K && format != LISA_GGUF_Q2_K) || tokens < 1 || tokens > 65535) return false;
    GmPlan pl;
    if (!gm_plan(format == LISA_GGUF_Q4_K ? 4 : 2, tokens, rows, row_bytes, pl)) return false;
    return (reinterpret_cast<uintptr_t>(w) & static_cast<uintptr_t>(pl.piece - 1)) == 0;
}

int gguf_mm(cudaStream_t stream, int format, const uint8_t *w, int64_t rows, int64_t row_bytes, const float *x, int64_t tokens, float *y) {
    GmPlan pl;
    const bool q4 = format == LISA_GGUF_Q4_K;
    if (!gm_plan(q4 ? 4 : 2, tokens, rows, row_bytes, pl)) return fail(LISA_ERR_UNSUPPORTED, "gguf_mm: shape not supported");
    pl.p.w = w;
    pl.p.x = x;
    pl.p.y = y;
    if (q4) return gm_launch<4, 16>(stream, pl);
    return pl.piece == 16 ? gm_launch<2, 16>(stream, pl) : pl.piece == 8 ? gm_launch<2, 8>(stream, pl) : gm_launch<2, 4>(stream, pl);
}

}  // namespace lisa
