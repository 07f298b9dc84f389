// The routed-expert block for a handful of tokens on byte dot products (see qmv_dp.cu for the arithmetic and the streams of packed
// rows), two launches behind the router:
//   gate|up   act[slot, :] = swiglu(bf16(x . Wg[e]^T), bf16(x . Wu[e]^T))                  CTA = rows of one slot
//   down      out[t, :] = bf16(fold_j f32(bf16(act[t, j] . Wd[e_j]^T)) * w[t, j])          CTA = rows of one token
// What moe_gate_up_act and moe_down_combine compute (moe_decode.cu, with the reference's files), with their rounding points and
// their fold; like them it takes the activations as they are (four bytes each, see dp_core.cuh).
//
// At one token the block is latency, not bytes (21 MB of eight experts are 3.3 us at the copy rate; router, gate|up and down took
// 36 us one after another).  Both launches are dependent ones: gate|up converts x while the router runs and waits for nothing
// but the expert ids; it lets the down launch start once it has them, which then knows the router to be complete, reads the ids
// itself and has its weights in flight before it waits for the activations.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "dp_core.cuh"
#include "kernels.h"

namespace lisa {

namespace {

constexpr int kMdThreads = 512, kMdWarps = kMdThreads / 32, kMdMaxTopK = 32, kMdPlanes = 4;

struct MoeDpParams {
    const int32_t *idx;   // [tokens, top_k] expert ids and weights of the router
    const float *weights;
    const uint8_t *w[2];  // gate, up; or down
    const uint16_t *s[2], *b[2];
    const uint16_t *x;    // [tokens, k]; or the activations [tokens * top_k, k]
    uint16_t *y;          // [tokens * top_k, n]; or [tokens, n]
    int experts, top_k, n, k;
    int gshift, groups, row_bytes, scale_words, tail_bytes, tail_words;
    int steps, parts, spt;
    int ctas, base, extra;  // CTAs of a slot (token), octets of rows of a CTA (the first `extra` one more)
    int xf_at, ring_at, part_at;
};

template <int BITS, bool G32, bool DOWN>
__global__ void __launch_bounds__(kMdThreads, 2) moe_dp_kernel(const MoeDpParams p) {
    using S = DpShape<BITS, kMdPlanes>;
    using Take = DpTake<BITS, G32>;
    constexpr int XV = S::kXWords / 4, SUB = G32 ? 2 : 1, CB = S::kWords * 4, WSLOT = Take::kWSlot, SLOT = Take::kSlot, DEPTH = BITS == 2 ? 4 : 2;
    constexpr int MATS = DOWN ? 1 : 2;
    extern __shared__ __align__(128) uint8_t md_smem[];
    __shared__ float weight[kMdMaxTopK];
    __shared__ int sel[kMdMaxTopK];
    uint4 *xs = reinterpret_cast<uint4 *>(md_smem);               // [rows of x][steps][XV][8 lanes]
    float *xf = reinterpret_cast<float *>(md_smem + p.xf_at);     // [rows of x][steps * 8][1 + SUB]
    float *part = reinterpret_cast<float *>(md_smem + p.part_at);  // [sets][8 rows][parts]
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int sl = lane & 7, sub = lane >> 3;
    const int z = static_cast<int>(blockIdx.x) / p.ctas, cta = static_cast<int>(blockIdx.x) - z * p.ctas;
    const int token = DOWN ? z : z / p.top_k, slot_j = DOWN ? 0 : z - token * p.top_k;
    const int qb = cta * p.base + min(cta, p.extra), octets = p.base + (cta < p.extra ? 1 : 0);
    const int streams = DOWN ? p.top_k : 2;  // matrices per octet: the slots' down, or gate and up
    const int sets = octets * streams;       // a set is (octet, stream)
    auto convert_rows = [&](int xrows) {
        const uint16_t *xr = p.x + static_cast<size_t>(DOWN ? token * p.top_k : token) * p.k;
        const int nv = p.k / 8, nv_pad = p.steps * S::kCodes;  // vectors of a row; a multiple of 32 with the zeros behind it
        for (int i = tid; i < xrows * nv_pad; i += kMdThreads) {
            const int r = DOWN ? i / nv_pad : 0, v = i - r * nv_pad;
            const uint4 *src = reinterpret_cast<const uint4 *>(xr + static_cast<size_t>(r) * p.k);
            dp_convert<BITS, G32, kMdPlanes>(xs + static_cast<size_t>(r) * p.steps * XV * 8, xf + static_cast<size_t>(r) * p.steps * 8 * (1 + SUB), v,
                                  v < nv ? (DOWN ? __ldcg(src + v) : __ldg(src + v)) : make_uint4(0, 0, 0, 0));
        }
    };
    if (!DOWN) {
        convert_rows(1);  // x is older than the router
        pdl_wait();
    }
    if (tid < p.top_k) {
        const int e = __ldcg(p.idx + token * p.top_k + tid);
        sel[tid] = e >= 0 && e < p.experts ? e : -1;
        weight[tid] = DOWN ? __ldcg(p.weights + token * p.top_k + tid) : 0.f;
    }
    __syncthreads();
    pdl_launch_dependents();  // (behind the wait: a launch that starts now finds the router complete)

    // ---- the stream: a warp's ring of slots, a slot is one step of one set
    const uint32_t ring = smem_u32(md_smem) + p.ring_at + warp * (DEPTH * SLOT), ring_end = ring + DEPTH * SLOT;
    constexpr int H = CB / 8;
    const int pc = CB == 32 ? lane & 15 : sl, prow = CB == 32 ? lane >> 4 : sub;
    const int wpr = p.scale_words, srow = lane >> 2, sword = lane & 3 & (wpr - 1);
    struct {
        int set, part, left, ragged;
        uint32_t slot;
        const uint8_t *w, *s, *b;
        uint32_t ow[H], os;
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
        const int o = ahead.set / streams, m = ahead.set - o * streams, step = ahead.part * p.spt;
        const int e = max(DOWN ? sel[m] : sel[slot_j], 0);  // (an id outside the table: expert 0's weights, and zeros at the stores)
        const int mat = DOWN ? 0 : m;
        ahead.left = min(p.spt, p.steps - step);
        ahead.ragged = p.tail_bytes && step + ahead.left == p.steps ? 1 : 0;
        const int row0 = (qb + o) * 8, end = p.n - 1 - row0;
        const size_t row = static_cast<size_t>(e) * p.n + row0, g = (row * p.groups + step * 2 * wpr) * 2;
        ahead.w = (mat ? p.w[1] : p.w[0]) + row * p.row_bytes + step * (8 * CB);
        ahead.s = reinterpret_cast<const uint8_t *>(mat ? p.s[1] : p.s[0]) + g;
        ahead.b = reinterpret_cast<const uint8_t *>(mat ? p.b[1] : p.b[0]) + g;
#pragma unroll
        for (int h = 0; h < H; ++h) ahead.ow[h] = static_cast<uint32_t>(min(prow + h * (8 / H), end) * p.row_bytes + pc * 16);
        ahead.os = static_cast<uint32_t>(min(srow, end) * p.groups * 2 + sword * 4);
    };
    auto fetch = [&]() {
        if (ahead.left > 0) {
            if (ahead.left == ahead.ragged) {
                const bool in = pc * 16 < p.tail_bytes;
#pragma unroll
                for (int h = 0; h < H; ++h) cp_async16z(ahead.slot + lane * 16 + h * 512, ahead.w + (ahead.ow[h] - (in ? 0 : pc * 16)), in);
#pragma unroll
                for (int i = 0; i < SUB; ++i) {
                    const bool in_s = sword + 4 * i < p.tail_words;
                    const uint32_t o = ahead.os + (in_s ? 16 * i : -sword * 4);
                    cp_async4z(ahead.slot + WSLOT + i * 128 + lane * 4, ahead.s + o, in_s);
                    cp_async4z(ahead.slot + WSLOT + (SUB + i) * 128 + lane * 4, ahead.b + o, in_s);
                }
            } else {
#pragma unroll
                for (int h = 0; h < H; ++h) cp_async16(ahead.slot + lane * 16 + h * 512, ahead.w + ahead.ow[h]);
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
                ahead.set += kMdWarps;
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
    for (int i = 0; i < DEPTH; ++i) fetch();

    // ---- the down launch's activations, written by the gate|up launch
    if (DOWN) {
        pdl_wait();
        convert_rows(p.top_k);
    }
    __syncthreads();

    // ---- the tasks of this warp
    uint32_t mask[S::kFields];
#pragma unroll
    for (int f = 0; f < S::kFields; ++f) mask[f] = (BITS == 4 ? 0x0f0f0f0fu : 0x03030303u) << (f * BITS);
    const Take take(sl, sub, p.gshift);
    const uint32_t xs32 = smem_u32(xs) + sl * 16, xf32 = smem_u32(xf) + sl * (4 + 4 * SUB);
    int set = warp, prt = 0;
    uint32_t at = ring;
    while (true) {
        while (set >= sets) {
            set -= sets;
            ++prt;
        }
        if (prt >= p.parts) break;
        float acc0 = 0.f, acc1 = 0.f;
        const int xr = DOWN ? set % streams : 0;
        int step = prt * p.spt;
        const int end = min(step + p.spt, p.steps);
        uint32_t xp = xs32 + (xr * p.steps + step) * (XV * 128), fp = xf32 + (xr * p.steps + step) * (32 + 32 * SUB);
        for (; step < end; ++step, xp += XV * 128, fp += 32 + 32 * SUB) {
            asm volatile("cp.async.wait_group %0;" ::"n"(DEPTH - 1) : "memory");
            __syncwarp();
            uint32_t w[2][S::kWords], sc[2][SUB], bi[2][SUB];
            take(at, w, sc, bi);
            __syncwarp();
            fetch();
            at += SLOT;
            if (at == ring_end) at = ring;
            dp_chunk<BITS, G32, kMdPlanes>(w, sc, bi, xp, fp, mask, take.flip, acc0, acc1);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            float v = r ? acc1 : acc0;
#pragma unroll
            for (int off = 4; off >= 1; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
            if (sl == 0) part[(set * 8 + r * 4 + sub) * p.parts + prt] = v;
        }
        set += kMdWarps;
    }
    __syncthreads();

    // ---- sums in the order of k; SwiGLU, or the weighted fold over the slots
    for (int i = tid; i < octets * 8; i += kMdThreads) {
        const int o = i >> 3, r = i & 7, row = (qb + o) * 8 + r;
        if (row >= p.n) continue;
        auto total = [&](int m) {
            float t = 0.f;
            for (int k = 0; k < p.parts; ++k) t += part[((o * streams + m) * 8 + r) * p.parts + k];
            return t;
        };
        if constexpr (!DOWN) {
            p.y[static_cast<size_t>(z) * p.n + row] =
                sel[slot_j] < 0 ? 0 : static_cast<uint16_t>(swiglu_bf16x2(f32_to_bf16_bits(total(0)), f32_to_bf16_bits(total(MATS - 1))));
        } else {
            // fold of mlx_colsum_small_f32: ty = min(k, 8) strided partial sums, then total = part[j] + total
            const int ty = p.top_k < 8 ? p.top_k : 8;
            float fold[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) fold[q] = 0.f;
            for (int m = 0; m < p.top_k; ++m) {
                const float d = sel[m] < 0 ? 0.f : bf16_bits_to_f32(f32_to_bf16_bits(total(m)));
                const float v = __fmul_rn(d, weight[m]);
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (q == m % ty) fold[q] = __fadd_rn(v, fold[q]);
            }
            float t = fold[0];
#pragma unroll
            for (int q = 1; q < 8; ++q)
                if (q < ty) t = fold[q] + t;
            p.y[static_cast<size_t>(token) * p.n + row] = static_cast<uint16_t>(f32_to_bf16_bits(t));
        }
    }
}

// One launch's geometry: `zs` slots or tokens of n rows and k columns, `streams` matrices and `xrows` rows of x per octet.
bool md_plan(int64_t zs, int64_t n, int64_t k, int streams, int xrows, int group_size, int bits, MoeDpParams &p, int &smem) {
    if ((bits != 2 && bits != 4) || k % 64 != 0 || (k / group_size) % 2 != 0 || n < 1 || n > (1 << 24)) return false;
    if (group_size != 32 && group_size != 64 && group_size != 128) return false;
    p.n = static_cast<int>(n);
    p.k = static_cast<int>(k);
    const int chunks = static_cast<int>(k / 64);
    p.gshift = group_size == 32 ? 5 : group_size == 64 ? 6 : 7;
    p.groups = static_cast<int>(k / group_size);
    p.row_bytes = static_cast<int>(k * bits / 8);
    p.steps = (chunks + 7) / 8;
    p.scale_words = 256 / group_size;
    if (chunks % 8) {
        p.tail_bytes = p.row_bytes - (p.steps - 1) * 8 * (bits == 2 ? 16 : 32);
        p.tail_words = p.groups / 2 - (p.steps - 1) * p.scale_words;
    }
    const int octets = static_cast<int>((n + 7) / 8);
    p.ctas = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(octets, sm_count() / zs)));
    p.base = octets / p.ctas;
    p.extra = octets % p.ctas;
    const int per = (p.base + (p.extra ? 1 : 0)) * streams;
    double best = 1e30;
    for (int parts = 1; parts <= std::min(p.steps, 32); ++parts) {
        const int spt = (p.steps + parts - 1) / parts;
        if ((p.steps + spt - 1) / spt != parts) continue;
        const double cost = ((per * parts + kMdWarps - 1) / kMdWarps) * (spt + 0.15) + 0.01 * parts;
        if (cost < best) {
            best = cost;
            p.parts = parts;
            p.spt = spt;
        }
    }
    const int sub = group_size == 32 ? 2 : 1;
    const int64_t xs = static_cast<int64_t>(xrows) * p.steps * 8 * 64 * kMdPlanes, xf = static_cast<int64_t>(xrows) * p.steps * 8 * 4 * (1 + sub);
    if (xs > (1 << 20)) return false;
    p.xf_at = static_cast<int>(xs);
    p.ring_at = static_cast<int>((xs + xf + 127) & ~127);
    p.part_at = p.ring_at + kMdWarps * (bits == 2 ? 4 : 2) * (64 * (bits == 2 ? 16 : 32) + 256 * sub);
    const int64_t bytes = p.part_at + static_cast<int64_t>(per) * 8 * p.parts * 4;
    // (up to half of an SM's a CTA lets the down launch's weights come in beside the gate|up launch; more -- activations of eight slots of
    // 1792 -- still beat the kernels that read a slot at a time: 80 -> 25 us)
    if (bytes > max_smem_optin() - 4096) return false;
    smem = static_cast<int>(bytes);
    return true;
}

struct MdPlans {
    bool ok;
    MoeDpParams up, down;
    int up_smem, down_smem;
};

const MdPlans &md_plans(int64_t tokens, int top_k, int64_t hidden, int64_t inter, int group_size, int bits) {
    static thread_local PlanTable<MdPlans> table;
    bool known;
    MdPlans *e = table.find(hidden, inter, (tokens << 40) | (static_cast<int64_t>(current_device()) << 32) | (group_size << 16) | (bits << 8) | top_k, known);
    if (!known) {
        *e = {};
        e->ok = md_plan(tokens * top_k, inter, hidden, 2, 1, group_size, bits, e->up, e->up_smem) &&
                md_plan(tokens, hidden, inter, top_k, top_k, group_size, bits, e->down, e->down_smem);
    }
    return *e;
}

template <int BITS, bool G32>
int md_launch(cudaStream_t stream, const MoeDpParams &up, const MoeDpParams &down, const MdPlans &pl, int64_t tokens, int top_k) {
    LISA_TRY((allow_smem_of<moe_dp_kernel<BITS, G32, false>>()));
    LISA_TRY((allow_smem_of<moe_dp_kernel<BITS, G32, true>>()));
    LISA_TRY((launch_kernel(stream, static_cast<unsigned>(tokens * top_k * up.ctas), kMdThreads, pl.up_smem, LISA_FLAG_PDL, moe_dp_kernel<BITS, G32, false>, up)));
    LISA_TRY((launch_kernel(stream, static_cast<unsigned>(tokens * down.ctas), kMdThreads, pl.down_smem, LISA_FLAG_PDL, moe_dp_kernel<BITS, G32, true>, down)));
    count_launch(2);
    return LISA_OK;
}

}  // namespace

bool moe_dp_supported(int64_t tokens, int64_t experts, int top_k, int64_t hidden, int64_t inter, int group_size, int bits) {
    if (tokens < 1 || tokens > 128 || top_k < 1 || top_k > kMdMaxTopK || experts < 1 || experts > (1 << 20)) return false;
    if (hidden < 1 || inter < 1 || hidden > (1 << 20) || inter > (1 << 20)) return false;
    return md_plans(tokens, top_k, hidden, inter, group_size, bits).ok;
}

int moe_dp(cudaStream_t stream, const void *x, const int32_t *idx, const float *weights, int64_t tokens, int64_t experts, int top_k, int64_t hidden,
           int64_t inter, const uint32_t *const *w, const void *const *scales, const void *const *biases, int group_size, int bits, void *act, void *out) {
    const MdPlans &pl = md_plans(tokens, top_k, hidden, inter, group_size, bits);
    MoeDpParams up = pl.up, down = pl.down;
    for (MoeDpParams *p : {&up, &down}) {
        const int first = p == &up ? 0 : 2, count = p == &up ? 2 : 1;
        p->idx = idx;
        p->weights = weights;
        p->experts = static_cast<int>(experts);
        p->top_k = top_k;
        for (int i = 0; i < count; ++i) {
            p->w[i] = reinterpret_cast<const uint8_t *>(w[first + i]);
            p->s[i] = reinterpret_cast<const uint16_t *>(scales[first + i]);
            p->b[i] = reinterpret_cast<const uint16_t *>(biases[first + i]);
        }
    }
    up.x = reinterpret_cast<const uint16_t *>(x);
    up.y = reinterpret_cast<uint16_t *>(act);
    down.x = reinterpret_cast<const uint16_t *>(act);
    down.y = reinterpret_cast<uint16_t *>(out);
    const bool g32 = group_size == 32;
    if (bits == 4) return g32 ? md_launch<4, true>(stream, up, down, pl, tokens, top_k) : md_launch<4, false>(stream, up, down, pl, tokens, top_k);
    return g32 ? md_launch<2, true>(stream, up, down, pl, tokens, top_k) : md_launch<2, false>(stream, up, down, pl, tokens, top_k);
}

}  // namespace lisa
