// Split-KV ragged paged attention of grouped queries, for work items of up to 8 query rows per KV head (decode and short
// continuations, the rows being the (token, query head of the group) pairs): memory-bound, so the design goal is bytes in
// flight, from the first key on.
//
//   * A warp takes strips of 16 keys (8 KB at 128 dims) through a ring of its own: its first lane requests them by TMA
//     (SWIZZLE_128B boxes of 64 dims) straight from the pages, three strips ahead; no barrier of more than the warp until the end.
//     192 KB are in flight per SM.
//   * A lane reads from a strip what mma.sync wants it to hold: a sum over dims does not mind their order, so 16 bytes of a K row are
//     two k-steps' worth of B operand (Q is permuted alike), and 16 bytes of four V rows become eight n-tiles' by byte permutes
//     (the output dims are permuted back at the end). With the swizzle, and K's pieces 32 bytes apart, no two lanes of a
//     shared-memory access meet in a bank. (Loads per lane instead, into registers or by cp.async, kept the load/store unit
//     busier than the memory: 4.6 and 4.0 TB/s at 32 sequences x 32 heads x 1000 keys, where this has 6.1.)
//   * The tensor cores do the arithmetic at any group size: 8 of the MMA's 16 rows are query rows. The other 8 take what
//     rounding the weights to 16 bits leaves over, itself in 16 bits, so P V keeps the weights to 2^-16 and better in the same
//     instruction. fp16 would lose that, and at last the weight itself, below 2^-9, where its steps no longer shrink with the value:
//     sigmoid weights are that small. There the weights go in times 2^14 (they are 1 at most), and the outputs come back by it: to
//     2^-22 from 2^-17 on, no step above 2^-39. Scores, maxima, sums and outputs are fp32.
//   * KV range is split over gridDim.z CTAs; partial (O, m, l) go to a scratch buffer and the last CTA to finish (atomic ticket)
//     merges them: one launch, no separate combine kernel.
//
// Bound by HBM where there are keys enough, by a chain of dependent reads (item, page table, keys, merge) of some 6 us below.
// Measured on B200 (head_dim 128, bf16; before: 128-row tcgen05 tiles of the packed kernel):
//   8 heads of 8 : 64 x 250 keys 34.4 -> 19.7 us, 8 x 4096: 42.8 -> 27.3, 1 x 16384: 30.4 -> 17.6
//   4 heads of 4 : 8 x 600 keys 12.9 -> 8.3 us, 4 x 1024: 11.8 -> 7.5
// Dispatched for groups of 4 and 8 heads at 128 dims, whose kernel before had 16-bit weights. All others stay with attention_splitkv.cu,
// whose weights are fp32 throughout.
//
// Stands in for the external paged flash kernel the reference links
// (deepspeed/inference/v2/kernels/ragged_ops/blocked_flash/blocked_flash.cpp:21-101, flash.h:74).
#include <stdlib.h>
#include "hds_ptx.cuh"
#include "hds_host.cuh"
#include "../../../include/hds_b200.h"

namespace hds {

// Warps per CTA: 4, two CTAs per SM; or 8, one per SM, where there are no more CTAs than SMs (fewer splits to merge).
constexpr int kGroupRows = 8;      // query rows per item and KV head at most
constexpr int kGroupStrip = 16;    // keys a warp takes at a time; pages hold a multiple
__host__ __device__ constexpr int group_stages(int d) { return d == 128 ? 3 : 6; }
__host__ __device__ constexpr int group_slot_bytes(int d) { return 2 * kGroupStrip * d * 2; }      // K and V of a strip
__host__ __device__ constexpr int group_smem_bytes(int d, int w) { return w * group_stages(d) * group_slot_bytes(d) + 1024; }

struct GroupArgs {
    const void* q;
    void* out;
    const int32_t* block_tables;
    const hds_attn_item* items;
    int max_blocks_per_seq;
    int n_q_heads, n_kv_heads, block_size, bs_log2;
    int n_splits;
    float scale_log2;  // softmax scale * log2(e)
    int ws_rows;        // R of the scratch: 1 / 2 / 4 / 8, at least the rows of an item
    int32_t* counters;  // [n_items][n_kv_heads]
    float* ws_ml;       // [n_items][n_kv_heads][n_splits][R][2]
    float* ws_o;        // [n_items][n_kv_heads][n_splits][R][D]
    const float* alibi; // [n_q_heads] ALiBi slopes (natural-log units) or nullptr: score += slope * (key pos - query pos)
    int window;         // sliding-window attention: a query at position p sees keys (p - window, p]; 0 = unlimited
    int keep_first;     // with a window: the first keep_first positions stay visible to every later query
    int64_t out_ld;     // elements between the output rows of two tokens
    const float* sink;  // [n_q_heads] or nullptr: one more score (natural-log units) in every denominator
    const float* sigmoid_bias;  // [n_q_heads] or nullptr: keys weigh sigmoid(score + bias), no denominator
    const void* gate;   // nullptr, or rows (gate_ld apart) like out's whose sigmoid multiplies it
    int64_t gate_ld;
    float cap_log2, cap_k;      // cap_log2 > 0: bounded scores (softcap_log2; scores come scaled, in log2 units)
};

// a finished output value, behind the denominator (sink included) and the gate; m in log2 units
template <bool kBf16>
__device__ __forceinline__ float group_finish(const GroupArgs& a, float o, float l, float m, int64_t row, int head, int col) {
    if (a.sigmoid_bias == nullptr) {
        if (a.sink != nullptr) l += exp2f(a.sink[head] * 1.4426950408889634f - m);
        o /= l;
    }
    if (a.gate != nullptr) {
        const float g = load_scalar<kBf16>(a.gate, row * a.gate_ld + col);
        o /= 1.0f + exp2f(g * -1.4426950408889634f);
    }
    return o;
}

__device__ __forceinline__ float group_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

template <bool kBf16>
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if constexpr (kBf16)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Lane = 4 * g + t. Row g of the MMA is query row g; t picks two of every eight keys (as the rows of C and A have it), g the key of
// K (as the columns of B have it) and, for V, eight output dims. Every warp keeps its own running (max, sum, accumulator).
template <int D, bool kBf16, int W>
__global__ void __launch_bounds__(W * 32, W == 4 ? 2 : 1)
paged_attn_group_kernel(const __grid_constant__ CUtensorMap tmap_kv, const GroupArgs a) {
    constexpr int KC = D / 32;        // 16-byte pieces of a K row per lane
    constexpr int VC = D / 64;        // 16-byte pieces of a V row per lane
    constexpr int LD = D + 4;
    constexpr int ST = group_stages(D);
    constexpr float kUp = kBf16 ? 1.0f : 16384.0f;      // what a weight is multiplied by before it becomes 16 bits
    static_assert(kGroupRows * LD * 4 <= ST * group_slot_bytes(D), "a warp's outputs fit its ring");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[W][ST];
    __shared__ float mg_ml[W][kGroupRows][2];
    __shared__ int flag_s;

    pdl_enter();  // PDL: the next kernel may be scheduled; this one needs its predecessor's Q and KV writes
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int item_idx = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
    const hds_attn_item item = a.items[item_idx];
    const int G = a.n_q_heads / a.n_kv_heads;
    const int rows = min(item.n_q * G, kGroupRows);  // (the host allows no more)
    const int kv_len = item.pos0 + item.n_q;
    const int strips_total = (kv_len + kGroupStrip - 1) / kGroupStrip;
    // sliding window: strips that lie wholly before the first query's window are never loaded
    // (those of the kept first tokens are visited before them: live strip i is strip i, or i + skipped behind the kept ones)
    const int strip_first = a.window > 0 ? max(0, item.pos0 - a.window + 1) / kGroupStrip : 0;
    const int strips_keep = min((a.keep_first + kGroupStrip - 1) / kGroupStrip, strip_first);
    const int strips_skip = strip_first - strips_keep;
    const int strips_live = strips_total - strips_skip;
    const int per = (strips_live + a.n_splits - 1) / a.n_splits;
    const int eff_splits = (strips_live + per - 1) / per;
    if (split >= eff_splits) return;
    if (lane == 0) {
        if (warp == 0) prefetch_tmap(&tmap_kv);
        for (int i = 0; i < ST; ++i) mbar_init(&full[warp][i], 1);
        fence_barrier_init();
    }
    __syncwarp();
    const int s0 = split * per + warp, s1 = min(strips_live, split * per + per);

    // ---- my query row, pieces of 8 dims permuted as K's are ----
    const bool live = g < rows;
    const int r_tok = live ? g / G : 0, r_head = kvh * G + (live ? g % G : 0);
    const int q_pos = item.pos0 + r_tok;
    uint4 q[KC];
    {
        const char* qp = reinterpret_cast<const char*>(a.q) + ((static_cast<int64_t>(item.q_row0) + r_tok) * a.n_q_heads + r_head) * D * 2 + t * 32;
        const bool wide = (reinterpret_cast<uintptr_t>(a.q) & 15) == 0;
#pragma unroll
        for (int c = 0; c < KC; ++c) {
            const char* p = qp + (c >> 1) * 128 + (c & 1) * 16;
            if (!live) {
                q[c] = make_uint4(0u, 0u, 0u, 0u);
            } else if (wide) {
                q[c] = *reinterpret_cast<const uint4*>(p);
            } else {
                const uint16_t* h = reinterpret_cast<const uint16_t*>(p);
                q[c] = make_uint4(h[0] | (uint32_t)h[1] << 16, h[2] | (uint32_t)h[3] << 16, h[4] | (uint32_t)h[5] << 16, h[6] | (uint32_t)h[7] << 16);
            }
        }
    }
    const float slope = a.alibi ? a.alibi[r_head] * 1.4426950408889634f : 0.0f;
    const bool sigmoid = a.sigmoid_bias != nullptr;
    const float bias = sigmoid ? a.sigmoid_bias[r_head] * 1.4426950408889634f : 0.0f;

    const int32_t* table = a.block_tables + static_cast<int64_t>(item.seq) * a.max_blocks_per_seq;
    auto first_key = [&](int s) { return (s < strips_keep ? s : s + strips_skip) * kGroupStrip; };
    auto page_of = [&](int s) { return s < s1 ? table[first_key(s) >> a.bs_log2] : 0; };
    // a warp's ring of strips: 16 rows of 128 bytes per 64 dims, K's panels, then V's
    uint8_t* ring = smem + warp * ST * group_slot_bytes(D);
    auto load = [&](int s, int blk, int slot) {     // (one lane)
        uint8_t* dst = ring + slot * group_slot_bytes(D);
        const int krow = (((blk * 2) * a.n_kv_heads + kvh) << a.bs_log2) + (first_key(s) & (a.block_size - 1));
        const int vrow = krow + (a.n_kv_heads << a.bs_log2);
        mbar_expect_tx(&full[warp][slot], group_slot_bytes(D));
#pragma unroll
        for (int c = 0; c < VC; ++c) tma_load_2d(dst + c * 2048, &tmap_kv, &full[warp][slot], c * 64, krow, kEvictFirst);
#pragma unroll
        for (int c = 0; c < VC; ++c) tma_load_2d(dst + (VC + c) * 2048, &tmap_kv, &full[warp][slot], c * 64, vrow, kEvictFirst);
    };

    float m_run = sigmoid ? 0.0f : -INFINITY, l_run = 0.0f;   // (sigmoid weights have no maximum to be relative to); l_run: this lane's keys
    float acc[VC][8][4];
#pragma unroll
    for (int c = 0; c < VC; ++c)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[c][j][i] = 0.0f;

    int next_page = 0;
    if (lane == 0) {
        int pages[ST];
#pragma unroll
        for (int i = 0; i < ST; ++i) pages[i] = page_of(s0 + i * W);
#pragma unroll
        for (int i = 0; i < ST; ++i)
            if (s0 + i * W < s1) load(s0 + i * W, pages[i], i);
        next_page = page_of(s0 + ST * W);
    }
    int slot = 0;
    uint32_t phase = 0;
    for (int s = s0; s < s1; s += W) {
        const uint8_t* strip = ring + slot * group_slot_bytes(D);
        const int key0 = first_key(s);
        mbar_wait(&full[warp][slot], phase);
        // ---- scores of 16 keys: two chains per tile of 8 ----
        float sc[2][4], sd[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) sc[i][e] = sd[i][e] = 0.0f;
        }
#pragma unroll
        for (int c = 0; c < KC; ++c)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint4 k = *reinterpret_cast<const uint4*>(strip + (c >> 1) * 2048 + (g + 8 * i) * 128 + (((2 * t + (c & 1)) ^ g) << 4));
                mma_16816<kBf16>(sc[i], q[c].x, 0u, q[c].y, 0u, k.x, k.y);
                mma_16816<kBf16>(sd[i], q[c].z, 0u, q[c].w, 0u, k.z, k.w);
            }
        // ---- weights ----
        float p[4];
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = key0 + 2 * t + (i & 1) + 8 * (i >> 1);
            float x = (sc[i >> 1][i & 1] + sd[i >> 1][i & 1]) * a.scale_log2;
            if (a.cap_log2 > 0.0f) x = softcap_log2(x, a.cap_k, a.cap_log2);
            const bool ok = live && pos <= q_pos && (a.window <= 0 || pos > q_pos - a.window || pos < a.keep_first);
            p[i] = ok ? fmaf(slope, static_cast<float>(pos - q_pos), x) : -INFINITY;
            mx = fmaxf(mx, p[i]);
        }
        if (sigmoid) {
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = 1.0f / (1.0f + group_ex2(-(p[i] + bias)));
        } else {
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            const float m_new = fmaxf(m_run, mx);
            if (__any_sync(0xffffffffu, m_new > m_run)) {
                const float scale = m_run == -INFINITY ? 0.0f : group_ex2(m_run - m_new);
                l_run *= scale;
#pragma unroll
                for (int c = 0; c < VC; ++c)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[c][j][e] *= scale;
                m_run = m_new;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                p[i] = m_run == -INFINITY ? 0.0f : group_ex2(p[i] - m_run);
                l_run += p[i];
            }
        }
        // ---- O += P V: rounded weights in rows 0..7, what the rounding left in rows 8..15 ----
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] *= kUp;
        const uint32_t h0 = pack2<kBf16>(p[0], p[1]), h1 = pack2<kBf16>(p[2], p[3]);
        const uint32_t r0 = pack2<kBf16>(p[0] - unpack_lo<kBf16>(h0), p[1] - unpack_hi<kBf16>(h0));
        const uint32_t r1 = pack2<kBf16>(p[2] - unpack_lo<kBf16>(h1), p[3] - unpack_hi<kBf16>(h1));
#pragma unroll
        for (int c = 0; c < VC; ++c) {
            uint4 vr[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int key = 2 * t + (i & 1) + 8 * (i >> 1);
                vr[i] = *reinterpret_cast<const uint4*>(strip + (VC + c) * 2048 + key * 128 + ((g ^ (key & 7)) << 4));
                // rows past the last key may hold anything: no weight of zero makes that finite
                if (key0 + kGroupStrip > kv_len && key0 + key >= kv_len) vr[i] = make_uint4(0u, 0u, 0u, 0u);
            }
            const uint32_t w0[4] = {vr[0].x, vr[0].y, vr[0].z, vr[0].w}, w1[4] = {vr[1].x, vr[1].y, vr[1].z, vr[1].w};
            const uint32_t w2[4] = {vr[2].x, vr[2].y, vr[2].z, vr[2].w}, w3[4] = {vr[3].x, vr[3].y, vr[3].z, vr[3].w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t sel = (j & 1) ? 0x7632u : 0x5410u;
                mma_16816<kBf16>(acc[c][j], h0, r0, h1, r1, __byte_perm(w0[j >> 1], w1[j >> 1], sel), __byte_perm(w2[j >> 1], w3[j >> 1], sel));
            }
        }
        __syncwarp();       // (the slot has been read)
        if (lane == 0) {
            const int sn = s + ST * W;
            if (sn < s1) load(sn, next_page, slot);
            next_page = page_of(sn + W);
        }
        if (++slot == ST) {
            slot = 0;
            phase ^= 1;
        }
    }

    // ---- the warps' states through shared memory: each in its own ring, whose loads have all been waited for ----
    auto mg_o = [&](int w, int r) { return reinterpret_cast<float*>(smem + w * ST * group_slot_bytes(D)) + r * LD; };
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 1);
    l_run += __shfl_xor_sync(0xffffffffu, l_run, 2);
    if (live) {
        if (t == 0) {
            mg_ml[warp][g][0] = m_run;
            mg_ml[warp][g][1] = l_run;
        }
#pragma unroll
        for (int c = 0; c < VC; ++c)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                float4* d = reinterpret_cast<float4*>(mg_o(warp, g) + c * 64 + (2 * t + e) * 8);
                auto sum = [&](int j) { return (acc[c][j][e] + acc[c][j][e + 2]) * (1.0f / kUp); };
                d[0] = make_float4(sum(0), sum(1), sum(2), sum(3));
                d[1] = make_float4(sum(4), sum(5), sum(6), sum(7));
            }
    }
    __syncthreads();
    const int R = a.ws_rows;
    const int64_t unit = static_cast<int64_t>(item_idx) * a.n_kv_heads + kvh;
    const int64_t ws_base = unit * a.n_splits;
    auto finish4 = [&](int r, int dd, const float (&o)[4], float l, float mx) {
        const int64_t row = item.q_row0 + r / G;
        const int hd = kvh * G + r % G;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int col = hd * D + dd + i;
            store_scalar<kBf16>(a.out, row * a.out_ld + col, group_finish<kBf16>(a, o[i], l, mx, row, hd, col));
        }
    };
    for (int e = tid; e < rows * (D / 4); e += W * 32) {
        const int r = e / (D / 4), dd = (e % (D / 4)) * 4;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < W; ++w) mx = fmaxf(mx, mg_ml[w][r][0]);
        float o[4] = {0.f, 0.f, 0.f, 0.f}, l = 0.0f;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const float mw = mg_ml[w][r][0];
            const float wt = (mw == -INFINITY) ? 0.0f : group_ex2(mw - mx);
            const float4 x = *reinterpret_cast<const float4*>(mg_o(w, r) + dd);
            l = fmaf(wt, mg_ml[w][r][1], l);
            o[0] = fmaf(wt, x.x, o[0]); o[1] = fmaf(wt, x.y, o[1]); o[2] = fmaf(wt, x.z, o[2]); o[3] = fmaf(wt, x.w, o[3]);
        }
        if (eff_splits == 1) {
            finish4(r, dd, o, l, mx);
        } else {
            __stcg(reinterpret_cast<float4*>(a.ws_o + ((ws_base + split) * R + r) * D + dd), make_float4(o[0], o[1], o[2], o[3]));
            if (dd == 0) __stcg(reinterpret_cast<float2*>(a.ws_ml + ((ws_base + split) * R + r) * 2), make_float2(mx, l));
        }
    }
    if (eff_splits == 1) return;
    __threadfence();
    __syncthreads();
    if (tid == 0) flag_s = atomicAdd(&a.counters[unit], 1) == eff_splits - 1 ? 1 : 0;
    __syncthreads();
    if (flag_s == 0) return;
    __threadfence();
    // ---- last CTA of this (item, kv head): merge the splits ----
    for (int e = tid; e < rows * (D / 4); e += W * 32) {
        const int r = e / (D / 4), dd = (e % (D / 4)) * 4;
        float mx = -INFINITY, l = 0.0f, o[4] = {0.f, 0.f, 0.f, 0.f};
        for (int b = 0; b < eff_splits; b += 8) {     // eight splits' loads at once, whatever their number
            float2 ml[8];
            float4 x[8];
            float m = mx;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int64_t at = (ws_base + min(b + i, eff_splits - 1)) * R + r;
                ml[i] = __ldcg(reinterpret_cast<const float2*>(a.ws_ml + at * 2));
                x[i] = __ldcg(reinterpret_cast<const float4*>(a.ws_o + at * D + dd));
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (b + i >= eff_splits) ml[i] = make_float2(-INFINITY, 0.0f);
                m = fmaxf(m, ml[i].x);
            }
            const float old = mx == -INFINITY ? 0.0f : group_ex2(mx - m);
            l *= old;
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] *= old;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float w = ml[i].x == -INFINITY ? 0.0f : group_ex2(ml[i].x - m);
                l = fmaf(w, ml[i].y, l);
                o[0] = fmaf(w, x[i].x, o[0]); o[1] = fmaf(w, x[i].y, o[1]); o[2] = fmaf(w, x[i].z, o[2]); o[3] = fmaf(w, x[i].w, o[3]);
            }
            mx = m;
        }
        finish4(r, dd, o, l, mx);
    }
    if (tid == 0) a.counters[unit] = 0;
}

template <int D, bool kBf16, int W>
static int launch_group_w(const CUtensorMap& tm, const GroupArgs& a, int n_items, cudaStream_t s) {
    auto kern = paged_attn_group_kernel<D, kBf16, W>;
    static bool configured[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (!configured[dev & 63]) {
        HDS_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, group_smem_bytes(D, W)));
        configured[dev & 63] = true;
    }
    HDS_CHECK_CUDA(launch_kernel(kern, dim3(n_items, a.n_kv_heads, a.n_splits), dim3(W * 32), group_smem_bytes(D, W), s, tm, a));
    return HDS_OK;
}

template <int D, bool kBf16>
static int launch_group(const CUtensorMap& tm, const GroupArgs& a, int n_items, cudaStream_t s) {
    return static_cast<int64_t>(n_items) * a.n_kv_heads * a.n_splits <= sm_count() ? launch_group_w<D, kBf16, 8>(tm, a, n_items, s)
                                                                                   : launch_group_w<D, kBf16, 4>(tm, a, n_items, s);
}

}  // namespace hds

using namespace hds;

static inline int64_t align256(int64_t x) { return (x + 255) & ~int64_t(255); }

extern "C" int hds_paged_attention_group(const void* q, void* out, const void* kv_cache_layer, int64_t num_blocks,
                                         const int32_t* block_tables, int max_blocks_per_seq, const hds_attn_item* items, int n_items,
                                         int rows_per_item, int n_q_heads, int n_kv_heads, int head_dim, int block_size, int n_splits,
                                         float scale, void* workspace, int64_t workspace_bytes, int dtype, void* stream) {
    const float* alibi = attn_take_alibi();
    const int window = attn_take_window();
    const int keep_first = attn_take_keep_first();
    const int64_t out_ld = attn_take_out_stride();
    const AttnOptions opt = attn_take_options();
    HDS_REQUIRE(head_dim == 64 || head_dim == 128, "paged_attention_group: head_dim must be 64 or 128");
    HDS_REQUIRE(block_size == 16 || block_size == 32 || block_size == 64 || block_size == 128,
                "paged_attention_group: block_size must be 16/32/64/128");
    HDS_REQUIRE(n_kv_heads > 0 && n_q_heads % n_kv_heads == 0, "paged_attention_group: n_q_heads % n_kv_heads != 0");
    HDS_REQUIRE(rows_per_item >= 1 && rows_per_item <= kGroupRows, "paged_attention_group: at most 8 query rows per item");
    HDS_REQUIRE(n_splits >= 1 && n_splits <= 64, "paged_attention_group: n_splits in [1,64]");
    HDS_REQUIRE(dtype == 0 || dtype == 1, "paged_attention_group: dtype must be 0 (bf16) or 1 (fp16)");
    if (n_items == 0) return HDS_OK;
    // the scratch of the split-KV entry point: counters first (one size for all problems: they read zero at every launch), then (m, l), then O
    const int64_t need = hds_paged_attention_splitkv_workspace_bytes(n_items, n_q_heads, n_kv_heads, head_dim, n_splits, rows_per_item);
    if (n_splits > 1) HDS_REQUIRE(workspace != nullptr && workspace_bytes >= need, "paged_attention_group: workspace too small");
    GroupArgs a;
    memset(&a, 0, sizeof(a));
    a.q = q;
    a.out = out;
    a.block_tables = block_tables;
    a.items = items;
    a.max_blocks_per_seq = max_blocks_per_seq;
    a.n_q_heads = n_q_heads;
    a.n_kv_heads = n_kv_heads;
    a.block_size = block_size;
    a.bs_log2 = block_size == 16 ? 4 : block_size == 32 ? 5 : block_size == 64 ? 6 : 7;
    a.n_splits = n_splits;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.ws_rows = rows_per_item <= 1 ? 1 : rows_per_item <= 2 ? 2 : rows_per_item <= 4 ? 4 : 8;
    a.alibi = alibi;
    a.window = window;
    a.keep_first = window > 0 ? keep_first : 0;
    a.out_ld = out_ld > 0 ? out_ld : static_cast<int64_t>(n_q_heads) * head_dim;
    a.sink = opt.sink;
    a.sigmoid_bias = opt.sigmoid_bias;
    a.gate = opt.gate;
    a.gate_ld = opt.gate_ld;
    HDS_REQUIRE(opt.softcap == 0.0f || (alibi == nullptr && opt.sigmoid_bias == nullptr), "paged_attention_group: bounded scores without other terms");
    a.cap_log2 = opt.softcap * 1.4426950408889634f;
    a.cap_k = opt.softcap > 0.0f ? 2.0f / opt.softcap : 0.0f;
    const int64_t parts = static_cast<int64_t>(n_items) * n_kv_heads * n_splits * a.ws_rows;
    char* ws = reinterpret_cast<char*>(workspace);
    a.counters = reinterpret_cast<int32_t*>(ws);
    a.ws_ml = reinterpret_cast<float*>(ws + need - align256(parts * head_dim * 4) - align256(parts * 2 * 4));
    a.ws_o = reinterpret_cast<float*>(ws + need - align256(parts * head_dim * 4));
    CUtensorMap tm;
    const uint64_t rows = static_cast<uint64_t>(num_blocks) * 2 * n_kv_heads * block_size;
    const int rc = make_tmap_2d_16b(&tm, kv_cache_layer, head_dim, rows, static_cast<uint64_t>(head_dim) * 2, 64, kGroupStrip, dtype == 0);
    if (rc) return rc;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (head_dim == 128) return dtype == 0 ? launch_group<128, true>(tm, a, n_items, s) : launch_group<128, false>(tm, a, n_items, s);
    return dtype == 0 ? launch_group<64, true>(tm, a, n_items, s) : launch_group<64, false>(tm, a, n_items, s);
}
