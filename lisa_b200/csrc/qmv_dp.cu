// Decode GEMV for MLX affine 2-/4-/8-bit weights, one or two rows of x: packed words straight from global memory to
// registers, four-way byte dot products (dp4a), no staging of the weights and no tensor memory.
//   y[m, n] = sum_k x[m, k] * (scale * q + bias)
//
// Same operator as qmv_tc.cu (affine_qmv_fast / affine_qmv_wide, crates/lisa-mlx/src/shaders/common/matmul/
// quantized.metal:762-1088) with the factorisation of the reference's qdot (quantized.metal:196-295) and the same
// integer grid for the activations: with E the exponent of the largest magnitude of a chunk of x, x * 2^(13-E) is
// rounded to an integer below 2^14 and split into two signed bytes; products and sums are exact in s32, scale and bias
// are applied per chunk in f32.  That grid is what the operator promises for 2- and 4-bit codes with group size 64; 8-bit codes and group sizes
// 32 and 128, whose other kernels take the activations as they are, use four bytes, 2^(29-E) (see dp_core.cuh).
//
// What bounds a decode launch is not the stream of weights (a 14 MB matrix is 95 KB per SM) but the chain in front of
// and behind it: launch, activations, conversion, reduction.  So the kernel keeps that chain short:
//  - a lane takes a chunk of one row -- 32 bytes (64 4-bit or 32 8-bit codes) or 16 (64 2-bit codes); eight lanes are
//    256 (128) contiguous bytes of a row, a warp four rows.  The bytes of a word are separated by AND alone
//    (w & 0x0f0f0f0f, w & 0xf0f0f0f0): the fields keep their place value, each field has its own accumulator, and
//    the place values meet in one integer per chunk.  About 0.033 warp instructions per code.
//  - rows are dealt in octets (two rows per lane share its activation words); an octet's k range is cut
//    into `parts` tasks of the CTA's warps, which makes short launches with long rows use every warp.  The partial sums
//    of a row meet in shared memory in the order of k.  The cut depends on n and k only: a row's result depends neither
//    on the number of rows of x nor on its place in the matrix.
//  - the weights of the first tasks are in flight before griddepcontrol.wait, and a CTA takes at most half an SM, so
//    that the loads of launch i+1 run while launch i drains (LISA_FLAG_PDL).
//  - every CTA converts the whole row of x (2.5 - 17 K elements by 512 threads); the residual add + RMSNorm or the
//    SwiGLU in front of the linear happens in registers on the way (FUSE), one read of the inputs.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "dp_core.cuh"
#include "kernels.h"

namespace lisa {

namespace {

constexpr int kDpThreads = 512, kDpWarps = kDpThreads / 32;
constexpr int kDpMaxSeg = 3;
constexpr int kDpKeepVec = 2;  // 16-byte vectors of x + r per thread that the NORM form keeps in registers (k <= 8192), the rest is read twice

struct DpParams {
    const uint8_t *w[kDpMaxSeg];
    const uint16_t *s[kDpMaxSeg], *b[kDpMaxSeg];
    uint16_t *y[kDpMaxSeg];
    int n[kDpMaxSeg];        // rows of every linear
    int q0[kDpMaxSeg];       // its first octet of rows
    int nseg, octets, k, m;
    int chunks;              // chunks of a row
    int gshift;              // chunk -> scale group: (chunk * codes) >> gshift
    int groups, row_bytes;
    int base, extra;         // octets of a CTA: base, the first `extra` CTAs one more
    int scale_words;         // words of scales (and of biases) per row and step
    int tail_bytes, tail_words;  // bytes of a row and scale words in its last step, where that is ragged (else 0)
    int ring_at;             // place of the warps' rings in shared memory
    int steps, parts, spt;   // eight-chunk steps of a row, tasks per octet, steps per task
    const uint16_t *x;
    const uint16_t *nr, *nw;  // FUSE 1: residual, norm weight; FUSE 2: nr = up projection
    float eps;
    uint16_t *nsum, *nnorm;
};

// MT rows of x; DEPTH slots in a warp's ring; PLANES bytes of an activation
template <int BITS, int FUSE, int MT, bool G32, int DEPTH, int PLANES>
__global__ void __launch_bounds__(kDpThreads, 2) qmv_dp_kernel(const DpParams p) {
    using S = DpShape<BITS, PLANES>;
    constexpr int XV = S::kXWords / 4;  // 16-byte vectors of activation words per chunk: 8 / 8 / 4 of two planes
    constexpr int SUB = G32 ? 2 : 1;    // scale groups of a chunk (group size 32 under 64 codes: two)
    constexpr int CB = S::kWords * 4;   // bytes of a chunk: 16 (2-bit) / 32
    constexpr int WSLOT = 64 * CB;      // packed bytes of a ring slot: eight rows x eight chunks
    constexpr int SLOT = WSLOT + 256 * SUB;
    extern __shared__ __align__(128) uint8_t dp_smem[];
    uint4 *xs = reinterpret_cast<uint4 *>(dp_smem);                                      // [MT][steps][XV][8 lanes]
    float *xf = reinterpret_cast<float *>(xs + static_cast<size_t>(MT) * p.steps * XV * 8);  // [MT][steps * 8][1 + SUB]: factor, sums
    float *part = xf + static_cast<size_t>(MT) * p.steps * 8 * (1 + SUB);                    // [rows of the CTA][parts][MT]
    __shared__ float red[kDpWarps];

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform for the compiler too
    const int sl = lane & 7, sub = lane >> 3;  // chunk of the step; the lane's rows of an octet are sub and sub + 4
    // octets of this CTA; its tasks are (octet, part), octet major inside a part
    const int qb = static_cast<int>(blockIdx.x) * p.base + min(static_cast<int>(blockIdx.x), p.extra);
    const int sets = p.base + (static_cast<int>(blockIdx.x) < p.extra ? 1 : 0);

    pdl_launch_dependents();

    // ---- the stream: every warp has a ring of DEPTH slots, one slot = one step of one task (eight rows x eight chunks and
    // their scales and biases), filled by asynchronous copies of contiguous pieces of the rows (rows beyond the linear
    // repeat its last one: their sums are not stored).  Everything an iteration needs is kept as pointers that move by
    // a constant; a division or a 64-bit product per step cost more than the arithmetic on it.
    const uint32_t ring = smem_u32(dp_smem) + p.ring_at + warp * (DEPTH * SLOT);
    const uint32_t ring_end = ring + DEPTH * SLOT;
    const int wpr = p.scale_words;  // 32-bit words of scales (and of biases) per row and step
    constexpr int H = CB / 8;       // 16-byte copies of a slot per lane: 4 / 2
    // 4-/8-bit: copy h takes the sixteen pieces of rows 2h and 2h + 1, 2-bit: the eight pieces of each of four rows.  The
    // slot keeps the order of memory (pieces of one 32-byte sector that go to different places fetch it twice).
    const int pc = CB == 32 ? lane & 15 : sl;  // this lane's piece of a row
    const int prow = CB == 32 ? lane >> 4 : sub;
    const uint32_t to_w = lane * 16;
    // this lane's row and word of the scales (where a step has fewer words than four, lanes repeat them)
    const int srow = lane >> 2, sword = lane & 3 & (wpr - 1);
    auto linear_of = [&](int q) { return (p.nseg > 2 && q >= p.q0[2]) ? 2 : (p.nseg > 1 && q >= p.q0[1]) ? 1 : 0; };
    struct {
        int set, part, left;     // octet, part, steps left of the task
        int ragged;              // the task holds the row's last step and that one is ragged: 1, else 0
        uint32_t slot;
        const uint8_t *w, *s, *b;  // the octet's first row in the next step (warp-uniform)
        uint32_t ow[H], os;      // this lane's pieces of it, its word of the scales and of the biases
    } ahead;
    auto open_ahead = [&]() {
        while (ahead.set >= sets) {
            ahead.set -= sets;
            ++ahead.part;
        }
        if (ahead.part >= p.parts) {
            ahead.left = 0;
            return;
        }
        const int q = qb + ahead.set, seg = linear_of(q), step = ahead.part * p.spt;
        ahead.left = min(p.spt, p.steps - step);
        ahead.ragged = p.tail_bytes && step + ahead.left == p.steps ? 1 : 0;
        const int row0 = (q - ((seg == 0) ? 0 : (seg == 1) ? p.q0[1] : p.q0[2])) * 8;
        const int end = ((seg == 0) ? p.n[0] : (seg == 1) ? p.n[1] : p.n[2]) - 1 - row0;
        ahead.w = ((seg == 0) ? p.w[0] : (seg == 1) ? p.w[1] : p.w[2]) + static_cast<size_t>(row0) * p.row_bytes + step * (8 * CB);
        const size_t g = (static_cast<size_t>(row0) * p.groups + step * 2 * wpr) * 2;
        ahead.s = reinterpret_cast<const uint8_t *>((seg == 0) ? p.s[0] : (seg == 1) ? p.s[1] : p.s[2]) + g;
        ahead.b = reinterpret_cast<const uint8_t *>((seg == 0) ? p.b[0] : (seg == 1) ? p.b[1] : p.b[2]) + g;
#pragma unroll
        for (int h = 0; h < H; ++h) ahead.ow[h] = static_cast<uint32_t>(min(prow + h * (8 / H), end) * p.row_bytes + pc * 16);
        ahead.os = static_cast<uint32_t>(min(srow, end) * p.groups * 2 + sword * 4);
    };
    auto fetch = [&]() {
        if (ahead.left > 0) {
            if (ahead.left == ahead.ragged) {
                // a ragged last step: pieces and scales beyond the row's end are zeros
                const bool in = pc * 16 < p.tail_bytes;
#pragma unroll
                for (int h = 0; h < H; ++h)
                    cp_async16z(ahead.slot + to_w + h * 512, ahead.w + (ahead.ow[h] - (in ? 0 : pc * 16)), in);
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    const bool in_s = sword + 4 * i < p.tail_words;
                    const uint32_t o = ahead.os + (in_s ? 16 * i : -sword * 4);
                    cp_async4z(ahead.slot + WSLOT + i * 128 + lane * 4, ahead.s + o, in_s);
                    cp_async4z(ahead.slot + WSLOT + (SUB + i) * 128 + lane * 4, ahead.b + o, in_s);
                }
            } else {
#pragma unroll
                for (int h = 0; h < H; ++h) cp_async16(ahead.slot + to_w + h * 512, ahead.w + ahead.ow[h]);
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    cp_async4(ahead.slot + WSLOT + i * 128 + lane * 4, ahead.s + (ahead.os + 16 * i));
                    cp_async4(ahead.slot + WSLOT + (SUB + i) * 128 + lane * 4, ahead.b + (ahead.os + 16 * i));
                }
            }
            ahead.w += 8 * CB;
            ahead.s += 4 * wpr;
            ahead.b += 4 * wpr;
            ahead.slot += SLOT;
            if (ahead.slot == ring_end) ahead.slot = ring;
            if (--ahead.left == 0) {
                ahead.set += kDpWarps;
                open_ahead();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    ahead.set = warp;
    ahead.part = 0;
    ahead.slot = ring;
    open_ahead();
    for (int i = 0; i < DEPTH; ++i) fetch();

    // ---- activations.  The norm's weights are constants of the model: fetched before the wait
    uint4 nw_keep[FUSE == 1 ? kDpKeepVec : 1];
    if constexpr (FUSE == 1) {
#pragma unroll
        for (int u = 0; u < kDpKeepVec; ++u) {
            const int i = tid + u * kDpThreads;
            nw_keep[u] = i < p.k / 8 ? __ldg(reinterpret_cast<const uint4 *>(p.nw) + i) : make_uint4(0, 0, 0, 0);
        }
    }
    pdl_wait();
    for (int t = 0; t < MT; ++t) {
        const uint16_t *xr = p.x + static_cast<size_t>(t) * p.k;
        uint4 *xs_t = xs + static_cast<size_t>(t) * p.steps * XV * 8;
        float *xf_t = xf + static_cast<size_t>(t) * p.steps * 8 * (1 + SUB);
        const int nv = p.k / 8;  // 16-byte vectors of a row
        const int nv_pad = p.steps * 8 * S::kCodes / 8;
        auto vec = [&](int i, uint4 v) {  // FUSE 2: activation = swiglu(x, up)
            if constexpr (FUSE == 2) {
                const uint4 u = __ldg(reinterpret_cast<const uint4 *>(p.nr + static_cast<size_t>(t) * p.k) + i);
                const uint32_t gw[4] = {v.x, v.y, v.z, v.w}, uw[4] = {u.x, u.y, u.z, u.w};
                uint32_t a[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) a[q] = swiglu_bf16x2(gw[q], uw[q]);
                v = make_uint4(a[0], a[1], a[2], a[3]);
                if (p.nnorm && blockIdx.x == 0) reinterpret_cast<uint4 *>(p.nnorm + static_cast<size_t>(t) * p.k)[i] = v;
            }
            return v;
        };
        if constexpr (FUSE == 1) {
            // residual add and RMSNorm: the row stays in registers between the sum of squares and the conversion
            uint4 keep[kDpKeepVec];
            float acc = 0.f;
            const uint4 *x4 = reinterpret_cast<const uint4 *>(xr), *r4 = reinterpret_cast<const uint4 *>(p.nr + static_cast<size_t>(t) * p.k);
            auto total = [&](int i, float &sq) {  // bf16(x + r) of vector i, its squares into sq
                const uint4 a = i < nv ? __ldg(x4 + i) : make_uint4(0, 0, 0, 0), b = i < nv ? __ldg(r4 + i) : make_uint4(0, 0, 0, 0);
                const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
                uint32_t sw[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    sw[q] = f32x2_to_bf16x2(__uint_as_float(aw[q] << 16) + __uint_as_float(bw[q] << 16),
                                            __uint_as_float(aw[q] & 0xffff0000u) + __uint_as_float(bw[q] & 0xffff0000u));
                    const float s0 = __uint_as_float(sw[q] << 16), s1 = __uint_as_float(sw[q] & 0xffff0000u);
                    sq = fmaf(s0, s0, sq);
                    sq = fmaf(s1, s1, sq);
                }
                return make_uint4(sw[0], sw[1], sw[2], sw[3]);
            };
#pragma unroll
            for (int u = 0; u < kDpKeepVec; ++u) keep[u] = u * kDpThreads < nv ? total(tid + u * kDpThreads, acc) : make_uint4(0, 0, 0, 0);
            for (int i = tid + kDpKeepVec * kDpThreads; i < nv; i += kDpThreads) total(i, acc);
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
            if (t > 0) __syncthreads();
            if (lane == 0) red[warp] = acc;
            __syncthreads();
            float tot = 0.f;
#pragma unroll
            for (int w = 0; w < kDpWarps; ++w) tot += red[w];
            const float inv = 1.0f / sqrtf(tot / static_cast<float>(p.k) + p.eps);
            auto emit = [&](int i, const uint4 &sv, const uint4 &wv) {
                uint4 v = make_uint4(0, 0, 0, 0);
                if (i < nv) {
                    const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w}, ww[4] = {wv.x, wv.y, wv.z, wv.w};
                    uint32_t nd[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t h = f32x2_to_bf16x2(__uint_as_float(sw[q] << 16) * inv, __uint_as_float(sw[q] & 0xffff0000u) * inv);
                        nd[q] = f32x2_to_bf16x2(__uint_as_float(ww[q] << 16) * __uint_as_float(h << 16),
                                                __uint_as_float(ww[q] & 0xffff0000u) * __uint_as_float(h & 0xffff0000u));
                    }
                    v = make_uint4(nd[0], nd[1], nd[2], nd[3]);
                    if (blockIdx.x == 0) {
                        reinterpret_cast<uint4 *>(p.nsum + static_cast<size_t>(t) * p.k)[i] = sv;
                        if (p.nnorm) reinterpret_cast<uint4 *>(p.nnorm + static_cast<size_t>(t) * p.k)[i] = v;
                    }
                }
                dp_convert<BITS, G32, PLANES>(xs_t, xf_t, i, v);
            };
            // (whole warps: nv_pad is a multiple of 32)
#pragma unroll
            for (int u = 0; u < kDpKeepVec; ++u)
                if (tid + u * kDpThreads < nv_pad) emit(tid + u * kDpThreads, keep[u], nw_keep[u]);
            for (int i = tid + kDpKeepVec * kDpThreads; i < nv_pad; i += kDpThreads) {
                float unused = 0.f;
                emit(i, total(i, unused), i < nv ? __ldg(reinterpret_cast<const uint4 *>(p.nw) + i) : make_uint4(0, 0, 0, 0));
            }
        } else {
            // whole warps (nv_pad is a multiple of 32; the conversion shuffles); vectors beyond the row are zeros
            for (int i0 = tid; i0 < nv_pad; i0 += 2 * kDpThreads) {
                const int i1 = i0 + kDpThreads;
                uint4 v0 = i0 < nv ? __ldg(reinterpret_cast<const uint4 *>(xr) + i0) : make_uint4(0, 0, 0, 0);
                uint4 v1 = i1 < nv ? __ldg(reinterpret_cast<const uint4 *>(xr) + i1) : make_uint4(0, 0, 0, 0);
                if (i0 < nv) v0 = vec(i0, v0);
                dp_convert<BITS, G32, PLANES>(xs_t, xf_t, i0, v0);
                if (i1 < nv_pad) {
                    if (i1 < nv) v1 = vec(i1, v1);
                    dp_convert<BITS, G32, PLANES>(xs_t, xf_t, i1, v1);
                }
            }
        }
    }
    __syncthreads();

    // ---- the tasks of this warp
    uint32_t mask[S::kFields];
#pragma unroll
    for (int f = 0; f < S::kFields; ++f) mask[f] = (BITS == 8) ? 0xffffffffu : ((BITS == 4) ? 0x0f0f0f0fu : 0x03030303u) << (f * BITS);
    float acc[2][MT];  // rows sub, sub + 4 of the octet
#pragma unroll
    for (int t = 0; t < MT; ++t) acc[0][t] = acc[1][t] = 0.f;
    int set = warp, prt = 0;
    uint32_t at = ring;
    const uint32_t xs32 = smem_u32(xs) + sl * 16, xf32 = smem_u32(xf) + sl * (4 + 4 * SUB);
    const DpTake<BITS, G32> take(sl, sub, p.gshift);
    while (true) {
        while (set >= sets) {
            set -= sets;
            ++prt;
        }
        if (prt >= p.parts) break;
        int step = prt * p.spt;
        const int end = min(step + p.spt, p.steps);
        uint32_t xp = xs32 + step * (XV * 128), fp = xf32 + step * (32 + 32 * SUB);
        for (; step < end; ++step, xp += XV * 128, fp += 32 + 32 * SUB) {
            // the oldest slot has landed (every lane's own copies, then everyone's), goes to registers and is filled again
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            __syncwarp();
            uint32_t w[2][S::kWords], sc[2][SUB], bi[2][SUB];
            take(at, w, sc, bi);
            __syncwarp();
            fetch();
            at += SLOT;
            if (at == ring_end) at = ring;
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                const uint32_t xt = xp + t * p.steps * (XV * 128), ft = fp + t * p.steps * (32 + 32 * SUB);
                dp_chunk<BITS, G32, PLANES>(w, sc, bi, xt, ft, mask, take.flip, acc[0][t], acc[1][t]);
            }
        }
        // the task's sums over its eight lanes, to their place in the order of k
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                float v = acc[r][t];
#pragma unroll
                for (int off = 4; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (sl == 0) part[((set * 8 + r * 4 + sub) * p.parts + prt) * MT + t] = v;
                acc[r][t] = 0.f;
            }
        set += kDpWarps;
    }
    __syncthreads();

    // ---- sum of the parts, store
    for (int i = tid; i < sets * 8 * MT; i += kDpThreads) {
        const int t = (MT == 1) ? 0 : i / (sets * 8), rr = i - t * sets * 8;
        const int q = qb + (rr >> 3), seg = linear_of(q);
        const int row = (q - ((seg == 0) ? 0 : (seg == 1) ? p.q0[1] : p.q0[2])) * 8 + (rr & 7);
        const int rows = (seg == 0) ? p.n[0] : (seg == 1) ? p.n[1] : p.n[2];
        if (row >= rows) continue;
        float tot = 0.f;
        for (int k = 0; k < p.parts; ++k) tot += part[(rr * p.parts + k) * MT + t];
        uint16_t *y = (seg == 0) ? p.y[0] : (seg == 1) ? p.y[1] : p.y[2];
        y[static_cast<size_t>(t) * rows + row] = static_cast<uint16_t>(f32_to_bf16_bits(tot));
    }
}

struct DpPlan {
    int smem, grid, depth;
};

// Bytes of an activation (see the head of the file).
constexpr int dp_planes(int group_size, int bits) { return bits == 8 || group_size != 64 ? 4 : 2; }

// Cut of k into tasks and shared memory, from n (all the linears of the launch) and k only.
bool dp_make_plan(int64_t octets, int64_t k, int group_size, int bits, int mt, DpParams &p, DpPlan &pl) {
    const int codes = bits == 8 ? 32 : 64;
    if ((bits != 2 && bits != 4 && bits != 8) || k % codes != 0 || octets > (1 << 24)) return false;
    p.k = static_cast<int>(k);
    if ((k / group_size) % 2 != 0) return false;  // scales are copied in pairs
    p.chunks = static_cast<int>(k / codes);
    p.gshift = group_size == 32 ? 5 : group_size == 64 ? 6 : 7;
    p.groups = static_cast<int>(k / group_size);
    p.row_bytes = static_cast<int>(k * bits / 8);
    p.steps = (p.chunks + 7) / 8;
    p.octets = static_cast<int>(octets);
    pl.grid = static_cast<int>(std::min<int64_t>(octets, sm_count()));
    p.base = static_cast<int>(octets / pl.grid);
    p.extra = static_cast<int>(octets % pl.grid);
    const int per = p.base + (p.extra ? 1 : 0);  // octets of the fullest CTA
    // cut of k: the busiest warp's steps plus about an eighth of a step per task (its reduction)
    double best = 1e30;
    p.parts = 1;
    p.spt = p.steps;
    for (int parts = 1; parts <= std::min(p.steps, 64); ++parts) {
        const int spt = (p.steps + parts - 1) / parts;
        if ((p.steps + spt - 1) / spt != parts) continue;
        const int rounds = (per * parts + kDpWarps - 1) / kDpWarps;
        const double cost = rounds * (spt + 0.125) + 0.01 * parts;
        if (cost < best) {
            best = cost;
            p.parts = parts;
            p.spt = spt;
        }
    }
    const int sub = (group_size == 32 && bits != 8) ? 2 : 1;
    p.scale_words = 4 * codes / group_size;
    if (p.chunks % 8) {
        p.tail_bytes = p.row_bytes - (p.steps - 1) * 8 * (bits == 2 ? 16 : 32);
        p.tail_words = p.groups / 2 - (p.steps - 1) * p.scale_words;
    }
    const size_t fixed = static_cast<size_t>(mt) * p.steps * 8 * (codes * dp_planes(group_size, bits) + 4 * (1 + sub)) + static_cast<size_t>(per) * 8 * p.parts * mt * 4;
    p.ring_at = static_cast<int>((fixed + 127) & ~static_cast<size_t>(127));
    const int slot = 64 * (bits == 2 ? 16 : 32) + 256 * sub;
    const int full = bits == 2 ? 4 : 2;
    // half an SM, so that the next launch's weights come in beside this one; four planes of a long row: a whole one
    for (int limit : {max_smem_optin() / 2 - 2048, dp_planes(group_size, bits) == 4 ? max_smem_optin() - 2048 : 0})
        for (int depth : {full, full / 2}) {
            const size_t bytes = p.ring_at + static_cast<size_t>(kDpWarps) * depth * slot;
            if (fixed < (1u << 20) && bytes <= static_cast<size_t>(limit)) {
                pl.depth = depth;
                pl.smem = static_cast<int>(bytes);
                return true;
            }
        }
    return false;
}

bool dp_plan(int64_t octets, int64_t k, int group_size, int bits, int mt, DpParams &p, DpPlan &pl) {
    struct Known {
        bool ok;
        DpParams p;
        DpPlan pl;
    };
    static thread_local PlanTable<Known> table;
    bool known;
    Known *e = table.find(octets, k, (static_cast<int64_t>(current_device()) << 32) | (group_size << 16) | (bits << 8) | mt, known);
    if (!known) {
        e->p = {};
        e->ok = dp_make_plan(octets, k, group_size, bits, mt, e->p, e->pl);
    }
    p = e->p;
    pl = e->pl;
    return e->ok;
}

template <int BITS, int FUSE, int MT, bool G32, int DEPTH, int PLANES>
int dp_launch_depth(cudaStream_t stream, const DpParams &p, const DpPlan &pl, unsigned flags) {
    LISA_TRY((allow_smem_of<qmv_dp_kernel<BITS, FUSE, MT, G32, DEPTH, PLANES>>()));
    LISA_TRY(launch_kernel(stream, pl.grid, kDpThreads, pl.smem, flags, qmv_dp_kernel<BITS, FUSE, MT, G32, DEPTH, PLANES>, p));
    count_launch();
    return LISA_OK;
}

template <int BITS, int FUSE, int MT, bool G32, int PLANES>
int dp_launch_one(cudaStream_t stream, const DpParams &p, const DpPlan &pl, unsigned flags) {
    constexpr int kFull = BITS == 2 ? 4 : 2;
    return pl.depth == kFull ? dp_launch_depth<BITS, FUSE, MT, G32, kFull, PLANES>(stream, p, pl, flags)
                             : dp_launch_depth<BITS, FUSE, MT, G32, kFull / 2, PLANES>(stream, p, pl, flags);
}

template <int BITS, int FUSE, bool G32, int PLANES>
int dp_launch_rows(cudaStream_t stream, const DpParams &p, const DpPlan &pl, int mt, unsigned flags) {
    return mt == 2 ? dp_launch_one<BITS, FUSE, 2, G32, PLANES>(stream, p, pl, flags) : dp_launch_one<BITS, FUSE, 1, G32, PLANES>(stream, p, pl, flags);
}

template <int BITS>
int dp_launch(cudaStream_t stream, const DpParams &p, const DpPlan &pl, int mt, int fuse, int group_size, unsigned flags) {
    if constexpr (BITS == 8) {
        return dp_launch_rows<8, 0, false, 4>(stream, p, pl, mt, flags);
    } else {
        if (fuse == 1) return dp_launch_rows<BITS, 1, false, 2>(stream, p, pl, mt, flags);
        if (fuse == 2) return dp_launch_rows<BITS, 2, false, 2>(stream, p, pl, mt, flags);
        if (group_size == 64) return dp_launch_rows<BITS, 0, false, 2>(stream, p, pl, mt, flags);
        return group_size == 32 ? dp_launch_rows<BITS, 0, true, 4>(stream, p, pl, mt, flags) : dp_launch_rows<BITS, 0, false, 4>(stream, p, pl, mt, flags);
    }
}

int64_t dp_octets(int count, const int64_t *n) {
    int64_t q = 0;
    for (int i = 0; i < count; ++i) q += (n[i] + 7) / 8;
    return q;
}

}  // namespace

// Rows of whole chunks (64 2- or 4-bit, 32 8-bit codes) and an even number of groups; the fused forms for group size 64.
bool qmv_dp_supported(int64_t m, int64_t k, int count, const int64_t *n, int group_size, int bits, bool fused) {
    if (m < 1 || count < 1 || count > kDpMaxSeg) return false;
    if (fused && (bits == 8 || group_size != 64)) return false;
    for (int i = 0; i < count; ++i)
        if (n[i] < 1 || n[i] > (1 << 26)) return false;
    DpParams p{};
    DpPlan pl;
    return dp_plan(dp_octets(count, n), k, group_size, bits, 1, p, pl);
}

int qmv_dp(cudaStream_t stream, const void *x, int64_t m, int64_t k, int count, const uint32_t *const *w, const void *const *scales,
           const void *const *biases, const int64_t *n, int group_size, int bits, void *const *y, unsigned flags, const TcNormArgs *norm) {
    const int64_t octets = dp_octets(count, n);
    for (int64_t done = 0; done < m;) {
        DpParams p{};
        DpPlan pl;
        int mt = m - done >= 2 ? 2 : 1;
        if (mt == 2 && !dp_plan(octets, k, group_size, bits, 2, p, pl)) mt = 1;
        if (mt == 1 && !dp_plan(octets, k, group_size, bits, 1, p, pl)) return fail(LISA_ERR_UNSUPPORTED, "qmv_dp: shape not supported");
        p.m = mt;
        p.nseg = count;
        int q = 0;
        for (int i = 0; i < count; ++i) {
            p.w[i] = reinterpret_cast<const uint8_t *>(w[i]);
            p.s[i] = reinterpret_cast<const uint16_t *>(scales[i]);
            p.b[i] = reinterpret_cast<const uint16_t *>(biases[i]);
            p.y[i] = reinterpret_cast<uint16_t *>(y[i]) + done * n[i];
            p.n[i] = static_cast<int>(n[i]);
            p.q0[i] = q;
            q += static_cast<int>((n[i] + 7) / 8);
        }
        p.x = reinterpret_cast<const uint16_t *>(x) + done * k;
        int fuse = 0;
        if (norm) {
            fuse = norm->weight ? 1 : 2;
            p.nr = reinterpret_cast<const uint16_t *>(norm->residual) + done * k;
            p.nw = reinterpret_cast<const uint16_t *>(norm->weight);
            p.eps = norm->eps;
            p.nsum = norm->sum ? reinterpret_cast<uint16_t *>(norm->sum) + done * k : nullptr;
            p.nnorm = norm->normed ? reinterpret_cast<uint16_t *>(norm->normed) + done * k : nullptr;
        }
        const int rc = bits == 4   ? dp_launch<4>(stream, p, pl, mt, fuse, group_size, flags)
                       : bits == 2 ? dp_launch<2>(stream, p, pl, mt, fuse, group_size, flags)
                                   : dp_launch<8>(stream, p, pl, mt, fuse, group_size, flags);
        if (rc != LISA_OK) return rc;
        done += mt;
    }
    return LISA_OK;
}

}  // namespace lisa
