// GEMV for MLX affine 2-/4-/8-bit weights and three to eight rows of x, on mma.sync with f16 operands:
//   y[m, n] = sum_k x[m, k] * (scale * q + bias)
// Same operator as qmv_dp.cu (which makes a pass over the weights per two rows) and qmv_tc.cu; the reference's
// affine_qmv_wide (crates/lisa-mlx/src/shaders/common/matmul/quantized.metal:890-1088).
//
// Codes and activations enter as f16 (mm_core.cuh: a masked field is a subnormal f16, x is normalised per 64-k group), products are
// exact, the sums those of the tensor core; scale and bias follow per 64-k group, in f32: no integer grid for the activations.
//
// What bounds it: the packed stream needs 46 4-bit (75 2-bit) codes per clock and SM at the measured copy rate; lifting
// codes costs 5/8 (9/16) of an operation of the half-rate pipe per code, the m16n8k16 MMAs run at 0.43 per clock (110
// codes), so the kernel is near the balance of the three.  Sixteen warps per SM, one CTA: each warp walks tasks
// (16 rows, a run of steps) through its own ring of asynchronous copies, like qmv_dp.cu; the B fragments of x lie
// in shared memory in fragment order.  Rows of more k than fit there are
// divided over a cluster of two or four CTAs, whose partial sums meet in the first one's shared memory.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "kernels.h"
#include "mm_core.cuh"

namespace lisa {

namespace {

constexpr int kMmThreads = 512, kMmWarps = kMmThreads / 32;
constexpr int kMmMaxSeg = 3;

struct MmParams {
    const uint8_t *w[kMmMaxSeg];
    const uint16_t *s[kMmMaxSeg], *b[kMmMaxSeg];
    uint16_t *y[kMmMaxSeg];
    int n[kMmMaxSeg];        // rows of every linear
    int q0[kMmMaxSeg];       // its first row block (16 rows)
    int nseg, k, m;
    int groups;              // scales of a row
    int g128;                // group size 128
    int row_bytes;
    int steps;               // 128-byte steps of a row
    int splits, max_steps;   // CTAs of a cluster; most steps of one
    int base, extra;         // row blocks of a share: base, the first `extra` shares one more
    int parts, spt;          // tasks per row block (and CTA), steps per task
    int tail_bytes, tail_words;
    int warps;               // warps that have a ring and take tasks (all sixteen stage x)
    int ring_at, sums_at, part_at;
    const uint16_t *x;
    const uint16_t *nr, *nw;
    float eps;
    uint16_t *nsum, *nnorm;
};

__device__ __forceinline__ uint32_t mm_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void mm_cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void mm_cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void mm_st_cluster(float *local, uint32_t rank, float v) {
    uint32_t remote;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

// MT (4 or 8) tokens of fragment storage; FUSE as in qmv_dp.cu (1: residual add + RMSNorm, 2: SwiGLU); CL: a cluster of CTAs
// divides the row's steps; G128: group size 128
template <int BITS, int FUSE, int MT, bool CL, bool G128>
__global__ void __launch_bounds__(kMmThreads, 1) qmv_mm_kernel(const MmParams p) {
    using S = MmShape<BITS>;
    constexpr int G = S::kGroups, PITCH = S::kPitch, DEPTH = 2;
    constexpr int WSLOT = 16 * PITCH;
    constexpr int FRAG = MT * 128;      // bytes of a group's fragments: two halves of MT x 4 lanes x 16
    constexpr int SUMS = MT * 8;        // of a pair of tokens: factors {a, b}, sums of x {a, b}
    constexpr int WPR = (G128 ? G / 2 : G) / 2;  // 32-bit words of scales (and of biases) per row and step: 4, 2 or 1
    extern __shared__ __align__(128) uint8_t mm_smem[];
    __shared__ float red[kMmWarps], inv_rms[8];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int g = lane >> 2, c = lane & 3;  // fragment row (A) or token (B), and quarter of a group
    const int splits = CL ? p.splits : 1, rank = CL ? static_cast<int>(mm_cluster_rank()) : 0;
    const int share = CL ? static_cast<int>(blockIdx.x) / splits : static_cast<int>(blockIdx.x);
    const int qb = share * p.base + min(share, p.extra), blocks = p.base + (share < p.extra ? 1 : 0);
    const int s0 = CL ? rank * p.steps / splits : 0, steps = CL ? (rank + 1) * p.steps / splits - s0 : p.steps;
    const int parts = CL ? (steps + p.spt - 1) / p.spt : p.parts;
    if (CL) mm_cluster_arrive();
    pdl_launch_dependents();
    const uint32_t frag = smem_u32(mm_smem), sums = frag + p.sums_at;
    float *part = reinterpret_cast<float *>(mm_smem + p.part_at);  // [rows of the share][splits][parts][MT], in the first CTA
    constexpr int SLOT = WSLOT + 16 * WPR * 8;  // scales, then biases: [16 rows][WPR words]
    const uint32_t ring = frag + p.ring_at + warp * DEPTH * SLOT;
    auto linear_of = [&](int q) { return (p.nseg > 2 && q >= p.q0[2]) ? 2 : (p.nseg > 1 && q >= p.q0[1]) ? 1 : 0; };

    // ---- the stream (see qmv_dp.cu)
    struct {
        int set, part, left, ragged;
        uint32_t slot;
        const uint8_t *w, *s, *b;
        uint32_t ow[4];
        int end;
    } ahead;
    const int pc = lane & 7, prow = lane >> 3;  // copy h: rows 4h + prow, piece pc
    auto open_ahead = [&]() {
        while (ahead.set >= blocks) {
            ahead.set -= blocks;
            ++ahead.part;
        }
        if (ahead.part >= parts) {
            ahead.left = 0;
            return;
        }
        const int q = qb + ahead.set, seg = linear_of(q), step = s0 + ahead.part * p.spt;
        ahead.left = min(p.spt, s0 + steps - step);
        ahead.ragged = p.tail_bytes && step + ahead.left == p.steps ? 1 : 0;
        const int row0 = (q - ((seg == 0) ? 0 : (seg == 1) ? p.q0[1] : p.q0[2])) * 16;
        ahead.end = ((seg == 0) ? p.n[0] : (seg == 1) ? p.n[1] : p.n[2]) - 1 - row0;
        ahead.w = ((seg == 0) ? p.w[0] : (seg == 1) ? p.w[1] : p.w[2]) + static_cast<size_t>(row0) * p.row_bytes + step * 128;
        const size_t go = (static_cast<size_t>(row0) * p.groups + step * 2 * WPR) * 2;
        ahead.s = reinterpret_cast<const uint8_t *>((seg == 0) ? p.s[0] : (seg == 1) ? p.s[1] : p.s[2]) + go;
        ahead.b = reinterpret_cast<const uint8_t *>((seg == 0) ? p.b[0] : (seg == 1) ? p.b[1] : p.b[2]) + go;
#pragma unroll
        for (int h = 0; h < 4; ++h) ahead.ow[h] = static_cast<uint32_t>(min(4 * h + prow, ahead.end) * p.row_bytes + pc * 16);
    };
    auto fetch = [&]() {
        if (ahead.left > 0) {
            const bool ragged = ahead.left == ahead.ragged;
            if (ragged) {
                const bool in = pc * 16 < p.tail_bytes;
#pragma unroll
                for (int h = 0; h < 4; ++h) mm_cp16z(ahead.slot + (4 * h + prow) * PITCH + pc * 16, ahead.w + (ahead.ow[h] - (in ? 0 : pc * 16)), in);
            } else {
#pragma unroll
                for (int h = 0; h < 4; ++h) mm_cp16(ahead.slot + (4 * h + prow) * PITCH + pc * 16, ahead.w + ahead.ow[h]);
            }
            // scales and biases: 16 rows x wpr words each (1, 2 or 4: a power of two)
            constexpr int WORDS = 16 * WPR;
#pragma unroll
            for (int i0 = 0; i0 < WORDS; i0 += 32) {
                const int i = i0 + lane, r = i / WPR, wd = i % WPR;
                if (WORDS < 32 && lane >= WORDS) break;
                const bool in = !ragged || wd < p.tail_words;
                const uint32_t o = static_cast<uint32_t>(min(r, ahead.end) * p.groups * 2 + (in ? wd * 4 : 0));
                mm_cp4z(ahead.slot + WSLOT + i * 4, ahead.s + o, in);
                mm_cp4z(ahead.slot + WSLOT + (WORDS + i) * 4, ahead.b + o, in);
            }
            ahead.w += 128;
            ahead.s += 4 * WPR;
            ahead.b += 4 * WPR;
            ahead.slot = ahead.slot == ring ? ring + SLOT : ring;
            if (--ahead.left == 0) {
                ahead.set += p.warps;
                open_ahead();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    ahead.set = warp;
    ahead.part = 0;
    ahead.slot = ring;
    ahead.left = 0;
    if (warp < p.warps) open_ahead();
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) fetch();

    // ---- B fragments.  An item is a lane's sixteen elements of a (group, token): pair q of the lane's packed words holds
    // elements (4-bit) 8 (q / 4) + q % 4 and + 4; (2-bit) q and q + 8, divided by the place 4^(q % 3); (8-bit) 4 (q / 2) + q % 2
    // and + 2.  Pairs 0..3 are half 0, pairs 4..7 half 1.
    pdl_wait();
    const int g0 = s0 * G, ng = min(steps * G, p.k / 64 - g0);  // groups of this CTA
    if constexpr (FUSE == 1) {
        // warps 2t, 2t + 1 (four tokens: 4t .. 4t + 3) sum the squares of token t, five chunks of loads in flight
        constexpr int WPT = kMmWarps / MT;
        const int t = warp / WPT;
        float acc = 0.f;
        if (t < p.m) {
            const uint4 *x4 = reinterpret_cast<const uint4 *>(p.x + static_cast<size_t>(t) * p.k), *r4 = reinterpret_cast<const uint4 *>(p.nr + static_cast<size_t>(t) * p.k);
            constexpr int U = 5;
            for (int i0 = (warp % WPT) * 32 + lane; i0 < p.k / 8; i0 += U * WPT * 32) {
                uint4 a[U], b[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int i = i0 + u * WPT * 32;
                    a[u] = i < p.k / 8 ? __ldg(x4 + i) : make_uint4(0, 0, 0, 0);
                    b[u] = i < p.k / 8 ? __ldg(r4 + i) : make_uint4(0, 0, 0, 0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, bw[4] = {b[u].x, b[u].y, b[u].z, b[u].w};
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t s2 = f32x2_to_bf16x2(__uint_as_float(aw[q] << 16) + __uint_as_float(bw[q] << 16),
                                                            __uint_as_float(aw[q] & 0xffff0000u) + __uint_as_float(bw[q] & 0xffff0000u));
                        const float f0 = __uint_as_float(s2 << 16), f1 = __uint_as_float(s2 & 0xffff0000u);
                        acc = fmaf(f0, f0, acc);
                        acc = fmaf(f1, f1, acc);
                    }
                }
            }
        }
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
        if (lane == 0) red[warp] = acc;
        __syncthreads();
        if (tid < p.m) {
            float tot = 0.f;
#pragma unroll
            for (int w = 0; w < WPT; ++w) tot += red[tid * WPT + w];
            inv_rms[tid] = 1.0f / sqrtf(tot / static_cast<float>(p.k) + p.eps);
        }
        __syncthreads();
    }
    // (whole warps: the four lanes of a (group, token) are neighbours and share its sums through shuffles)
    const int items = ng * p.m * 4, per_token = ng * 4;
    struct Item {
        bool in;
        int t, gl, cc;
        size_t at;
        uint4 v0, v1;
    };
    auto load = [&](int it) {
        Item q;
        q.in = it < items;
        q.t = q.in ? it / per_token : 0;
        const int u = q.in ? it - q.t * per_token : 0;
        q.gl = u >> 2;
        q.cc = u & 3;
        q.at = static_cast<size_t>(q.t) * p.k + static_cast<size_t>(g0 + q.gl) * 64 + q.cc * 16;
        const uint4 *src = reinterpret_cast<const uint4 *>(p.x + q.at);
        q.v0 = q.in ? __ldg(src) : make_uint4(0, 0, 0, 0);
        q.v1 = q.in ? __ldg(src + 1) : make_uint4(0, 0, 0, 0);
        return q;
    };
    auto stage = [&](const Item &item) {
        const bool in = item.in;
        const int t = item.t, gl = item.gl, cc = item.cc;
        const size_t at = item.at;
        const uint4 v0 = item.v0, v1 = item.v1;
        uint32_t e[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        if constexpr (FUSE != 0) {
            if (in) {
                const uint4 r0 = __ldg(reinterpret_cast<const uint4 *>(p.nr + at)), r1 = __ldg(reinterpret_cast<const uint4 *>(p.nr + at) + 1);
                const uint32_t rw[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
                if constexpr (FUSE == 2) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) e[q] = swiglu_bf16x2(e[q], rw[q]);
                } else {
                    const float inv = inv_rms[t];
                    const uint4 *nw4 = reinterpret_cast<const uint4 *>(p.nw + static_cast<size_t>(g0 + gl) * 64 + cc * 16);
                    const uint4 n0 = __ldg(nw4), n1 = __ldg(nw4 + 1);
                    const uint32_t nw[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
                    uint32_t sw[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        sw[q] = f32x2_to_bf16x2(__uint_as_float(e[q] << 16) + __uint_as_float(rw[q] << 16),
                                                __uint_as_float(e[q] & 0xffff0000u) + __uint_as_float(rw[q] & 0xffff0000u));
                        const uint32_t h = f32x2_to_bf16x2(__uint_as_float(sw[q] << 16) * inv, __uint_as_float(sw[q] & 0xffff0000u) * inv);
                        e[q] = f32x2_to_bf16x2(__uint_as_float(nw[q] << 16) * __uint_as_float(h << 16),
                                               __uint_as_float(nw[q] & 0xffff0000u) * __uint_as_float(h & 0xffff0000u));
                    }
                    if (share == 0) {
                        uint4 *to = reinterpret_cast<uint4 *>(p.nsum + at);
                        to[0] = make_uint4(sw[0], sw[1], sw[2], sw[3]);
                        to[1] = make_uint4(sw[4], sw[5], sw[6], sw[7]);
                    }
                }
                if (p.nnorm && share == 0) {
                    uint4 *to = reinterpret_cast<uint4 *>(p.nnorm + at);
                    to[0] = make_uint4(e[0], e[1], e[2], e[3]);
                    to[1] = make_uint4(e[4], e[5], e[6], e[7]);
                }
            }
        }
        mm_fragment<BITS, MT>(e, frag, sums, gl, t, cc, in);
    };
    // groups of a ragged last step that the row does not have: zeros (their codes and scales are zeros too)
    for (int i = tid; i < (steps * G - ng) * (FRAG + SUMS) / 8; i += kMmThreads) {
        const int gz = ng + i / ((FRAG + SUMS) / 8), o = (i % ((FRAG + SUMS) / 8)) * 8;
        const uint32_t to = o < FRAG ? frag + gz * FRAG + o : sums + gz * SUMS + (o - FRAG);
        asm volatile("st.shared.v2.u32 [%0], {%1, %1};" ::"r"(to), "r"(0) : "memory");
    }
    // (three items' loads in flight: a round trip to L2 costs as much as the conversion of six)
    for (int it = tid; it - lane < items; it += 3 * kMmThreads) {
        const Item i0 = load(it), i1 = load(it + kMmThreads), i2 = load(it + 2 * kMmThreads);
        stage(i0);
        if (it - lane + kMmThreads < items) stage(i1);
        if (it - lane + 2 * kMmThreads < items) stage(i2);
    }
    __syncthreads();
    if (CL) mm_cluster_wait();  // the first CTA of the cluster runs: its shared memory takes the others' partial sums

    // ---- the tasks of this warp
    const MmLift<BITS> lift;
    const uint32_t frag_lane = frag + ((g & (MT - 1)) * 4 + c) * 16, sums_lane = sums + (c & (MT / 2 - 1)) * 16;
    int set = warp, prt = 0;
    uint32_t at = ring;
    while (warp < p.warps) {
        while (set >= blocks) {
            set -= blocks;
            ++prt;
        }
        if (prt >= parts) break;
        float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};  // rows g, g + 8; tokens 2c, 2c + 1
        const int end = min((prt + 1) * p.spt, steps);
        for (int step = prt * p.spt; step < end; ++step) {
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            __syncwarp();
            mm_step<BITS, MT, G128>(at, frag_lane + step * (G * FRAG), sums_lane + step * (G * SUMS), g, c, lift, acc);
            __syncwarp();
            fetch();
            at = at == ring ? ring + SLOT : ring;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (2 * c + j < p.m) {
                    float *to = part + (((set * 16 + h * 8 + g) * splits + rank) * p.parts + prt) * MT + 2 * c + j;
                    if (CL) mm_st_cluster(to, 0, acc[h][j]);
                    else *to = acc[h][j];
                }
        set += p.warps;
    }
    if (CL) {
        mm_cluster_arrive();
        if (rank != 0) return;
        mm_cluster_wait();
    } else {
        __syncthreads();
    }

    // ---- sum of the parts in the order of k, store
    for (int i = tid; i < blocks * 16 * p.m; i += kMmThreads) {
        const int t = i / (blocks * 16), rr = i - t * (blocks * 16);
        const int q = qb + (rr >> 4), seg = linear_of(q);
        const int row = (q - ((seg == 0) ? 0 : (seg == 1) ? p.q0[1] : p.q0[2])) * 16 + (rr & 15);
        const int rows = (seg == 0) ? p.n[0] : (seg == 1) ? p.n[1] : p.n[2];
        if (row >= rows) continue;
        float tot = 0.f;
        for (int r = 0; r < splits; ++r) {
            const int cnt = CL ? ((r + 1) * p.steps / splits - r * p.steps / splits + p.spt - 1) / p.spt : p.parts;
            for (int k = 0; k < cnt; ++k) tot += part[((rr * splits + r) * p.parts + k) * MT + t];
        }
        uint16_t *y = (seg == 0) ? p.y[0] : (seg == 1) ? p.y[1] : p.y[2];
        y[static_cast<size_t>(t) * rows + row] = static_cast<uint16_t>(f32_to_bf16_bits(tot));
    }
}

struct MmPlan {
    int smem, grid;
};

// Clusters of `splits` CTAs that the current device runs at a time when a CTA takes a whole SM.
int cluster_limit(int splits) {
    static std::atomic<int> known[64][2];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int> &slot = known[dev & 63][splits == 2 ? 0 : 1];
    int v = slot.load(std::memory_order_relaxed);
    if (v > 0) return v;
    v = sm_count() / splits - 4;  // (where the query fails)
    if (allow_smem_of<qmv_mm_kernel<4, 0, 8, true, false>>() == LISA_OK) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(sm_count() / splits * splits);
        cfg.blockDim = dim3(kMmThreads);
        cfg.dynamicSmemBytes = max_smem_optin() - 2048;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = splits;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, qmv_mm_kernel<4, 0, 8, true, false>, &cfg) == cudaSuccess && n > 0) v = n;
        else cudaGetLastError();
    }
    slot.store(v, std::memory_order_relaxed);
    return v;
}

// CTAs per share of the row blocks, cut of their steps into tasks and shared memory, from n (all the linears of the launch),
// k and the tokens of fragment storage.
bool mm_make_plan(int64_t blocks, int64_t k, int group_size, int bits, int mt, MmParams &p, MmPlan &pl) {
    if ((bits != 2 && bits != 4 && bits != 8) || k % 64 != 0 || blocks > (1 << 24)) return false;
    if (group_size != 64 && (group_size != 128 || bits == 8)) return false;
    if ((k / group_size) % 2 != 0) return false;  // scales are copied in pairs
    p.k = static_cast<int>(k);
    p.groups = static_cast<int>(k / group_size);
    p.g128 = group_size == 128 ? 1 : 0;
    p.row_bytes = static_cast<int>(k * bits / 8);
    p.steps = (p.row_bytes + 127) / 128;
    const int g = 1024 / bits / 64;  // 64-k groups of a step
    const int words = (g >> p.g128) / 2;
    if (p.row_bytes % 128) {
        p.tail_bytes = p.row_bytes % 128;
        p.tail_words = p.groups / 2 - (p.steps - 1) * words;
    }
    const int pitch = bits == 2 ? 144 : bits == 4 ? 160 : 192;
    const int slot = 16 * pitch + 16 * words * 8;
    // Cut of k over a cluster of CTAs and over tasks, and the warps that take tasks, by the steps of the busiest warp.  x's
    // fragments have to fit beside the rings, which rows of much k force by more CTAs or by fewer warps (an SM with twelve
    // streaming warps runs about 13 % below one with sixteen, with eight 37 %); a cluster costs about a step per CTA.
    // Clusters only come as whole ones within a GPC: at most as many as fit at a time are launched (37 clusters of four
    // that run as two waves were the slower half of a 43 us launch).
    double best = 1e30;
    for (int splits = 1; splits <= 4 && splits <= p.steps; splits *= 2) {
        const int64_t shares = std::min<int64_t>(blocks, splits == 1 ? sm_count() : cluster_limit(splits));
        const int per = static_cast<int>((blocks + shares - 1) / shares), most = (p.steps + splits - 1) / splits;
        const int64_t frag = static_cast<int64_t>(most) * g;
        const int64_t sums_at = frag * mt * 128, ring_at = sums_at + ((frag * mt * 8 + 127) & ~127);
        for (int warps : {16, 12, 8}) {
            const double pace = warps == 16 ? 1.0 : warps == 12 ? 0.87 : 0.79;  // time of a step against sixteen warps
            for (int parts = 1; parts <= std::min(most, 64); ++parts) {
                const int spt = (most + parts - 1) / parts;
                if ((most + spt - 1) / spt != parts) continue;
                const int64_t part_at = ring_at + static_cast<int64_t>(warps) * 2 * slot;
                const int64_t bytes = part_at + static_cast<int64_t>(per) * 16 * splits * parts * mt * 4;
                if (frag >= (1 << 16) || bytes > max_smem_optin() - 2048) continue;
                const double cost = ((per * parts + warps - 1) / warps) * (spt + 0.1) * pace + 0.01 * parts + (splits > 1 ? splits : 0);
                if (cost < best) {
                    best = cost;
                    p.splits = splits;
                    p.warps = warps;
                    p.parts = parts;
                    p.spt = spt;
                    p.max_steps = most;
                    p.base = static_cast<int>(blocks / shares);
                    p.extra = static_cast<int>(blocks % shares);
                    p.sums_at = static_cast<int>(sums_at);
                    p.ring_at = static_cast<int>(ring_at);
                    p.part_at = static_cast<int>(part_at);
                    pl.smem = static_cast<int>(bytes);
                    pl.grid = static_cast<int>(shares) * splits;
                }
            }
        }
    }
    return best < 1e30;
}

bool mm_plan(int64_t blocks, int64_t k, int group_size, int bits, int mt, MmParams &p, MmPlan &pl) {
    struct Known {
        bool ok;
        MmParams p;
        MmPlan pl;
    };
    static thread_local PlanTable<Known> table;
    bool known;
    Known *e = table.find(blocks, k, (static_cast<int64_t>(current_device()) << 32) | (group_size << 16) | (bits << 8) | mt, known);
    if (!known) {
        e->p = {};
        e->ok = mm_make_plan(blocks, k, group_size, bits, mt, e->p, e->pl);
    }
    p = e->p;
    pl = e->pl;
    return e->ok;
}

template <int BITS, int FUSE, int MT, bool CL, bool G128>
int mm_launch_kernel(cudaStream_t stream, const MmParams &p, const MmPlan &pl, unsigned flags) {
    LISA_TRY((allow_smem_of<qmv_mm_kernel<BITS, FUSE, MT, CL, G128>>()));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pl.grid);
    cfg.blockDim = dim3(kMmThreads);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (CL) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = p.splits;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    if (flags & LISA_FLAG_PDL) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    LISA_CUDA_TRY(cudaLaunchKernelEx(&cfg, qmv_mm_kernel<BITS, FUSE, MT, CL, G128>, p));
    count_launch();
    return LISA_OK;
}

template <int BITS, int FUSE, int MT, bool CL>
int mm_launch_one(cudaStream_t stream, const MmParams &p, const MmPlan &pl, unsigned flags) {
    if constexpr (FUSE == 0 && BITS != 8) {
        if (p.g128) return mm_launch_kernel<BITS, FUSE, MT, CL, true>(stream, p, pl, flags);
    }
    return mm_launch_kernel<BITS, FUSE, MT, CL, false>(stream, p, pl, flags);
}

template <int BITS, int FUSE>
int mm_launch(cudaStream_t stream, const MmParams &p, const MmPlan &pl, int mt, unsigned flags) {
    if (mt == 4) return p.splits > 1 ? mm_launch_one<BITS, FUSE, 4, true>(stream, p, pl, flags) : mm_launch_one<BITS, FUSE, 4, false>(stream, p, pl, flags);
    return p.splits > 1 ? mm_launch_one<BITS, FUSE, 8, true>(stream, p, pl, flags) : mm_launch_one<BITS, FUSE, 8, false>(stream, p, pl, flags);
}

int64_t mm_blocks(int count, const int64_t *n) {
    int64_t q = 0;
    for (int i = 0; i < count; ++i) q += (n[i] + 15) / 16;
    return q;
}

}  // namespace

// Up to eight rows of x; k a multiple of 64 with an even number of groups; group size 64, and 128 for 2- and 4-bit; the fused
// forms for group size 64 and 2- and 4-bit.
bool qmv_mm_supported(int64_t m, int64_t k, int count, const int64_t *n, int group_size, int bits, bool fused) {
    if (m < 1 || m > 8 || count < 1 || count > kMmMaxSeg) return false;
    if (fused && (bits == 8 || group_size != 64)) return false;
    for (int i = 0; i < count; ++i)
        if (n[i] < 1 || n[i] > (1 << 26)) return false;
    MmParams p{};
    MmPlan pl;
    return mm_plan(mm_blocks(count, n), k, group_size, bits, m <= 4 ? 4 : 8, p, pl);
}

int qmv_mm(cudaStream_t stream, const void *x, int64_t m, int64_t k, int count, const uint32_t *const *w, const void *const *scales,
           const void *const *biases, const int64_t *n, int group_size, int bits, void *const *y, unsigned flags, const TcNormArgs *norm) {
    MmParams p{};
    MmPlan pl;
    const int mt = m <= 4 ? 4 : 8;
    if (m > 8 || !mm_plan(mm_blocks(count, n), k, group_size, bits, mt, p, pl)) return fail(LISA_ERR_UNSUPPORTED, "qmv_mm: shape not supported");
    p.m = static_cast<int>(m);
    p.nseg = count;
    int q = 0;
    for (int i = 0; i < count; ++i) {
        p.w[i] = reinterpret_cast<const uint8_t *>(w[i]);
        p.s[i] = reinterpret_cast<const uint16_t *>(scales[i]);
        p.b[i] = reinterpret_cast<const uint16_t *>(biases[i]);
        p.y[i] = reinterpret_cast<uint16_t *>(y[i]);
        p.n[i] = static_cast<int>(n[i]);
        p.q0[i] = q;
        q += static_cast<int>((n[i] + 15) / 16);
    }
    p.x = reinterpret_cast<const uint16_t *>(x);
    int fuse = 0;
    if (norm) {
        fuse = norm->weight ? 1 : 2;
        p.nr = reinterpret_cast<const uint16_t *>(norm->residual);
        p.nw = reinterpret_cast<const uint16_t *>(norm->weight);
        p.eps = norm->eps;
        p.nsum = reinterpret_cast<uint16_t *>(norm->sum);
        p.nnorm = reinterpret_cast<uint16_t *>(norm->normed);
    }
    if (bits == 4) return fuse == 1 ? mm_launch<4, 1>(stream, p, pl, mt, flags) : fuse == 2 ? mm_launch<4, 2>(stream, p, pl, mt, flags) : mm_launch<4, 0>(stream, p, pl, mt, flags);
    if (bits == 2) return fuse == 1 ? mm_launch<2, 1>(stream, p, pl, mt, flags) : fuse == 2 ? mm_launch<2, 2>(stream, p, pl, mt, flags) : mm_launch<2, 0>(stream, p, pl, mt, flags);
    return mm_launch<8, 0>(stream, p, pl, mt, flags);
}

}  // namespace lisa
