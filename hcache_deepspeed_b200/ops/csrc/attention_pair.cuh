// Prefill attention of grouped queries, two heads of a KV group per CTA (included by attention_prefill.cu).
//
// One 128-row tile of queries leaves the tensor pipe idle while its softmax runs, and the softmax idle while its products run: the
// kernel with one head per CTA reaches 474 TFLOP/s at 16384 causal tokens. Two heads of the group see the same K and V tiles, so a
// CTA takes both: while one head's scores are weighed, the other's products run, and every tile is loaded once for the two.
//
//   warp 0    : TMA producer: Q of both heads, then K and V tiles of 128 keys, in the order of their use (K0 K1 V0 K2 V1 ...),
//               through one ring of five 32 KB slots
//   warp 1    : TMEM allocator + tcgen05.mma issuer. Per key tile and head: O += P V, then S = Q K^T of the next tile
//   warps 2-9 : softmax, four warps per head, one thread per query row (128 scores in registers, no exchange between threads).
//               P goes back to TMEM as 16-bit pairs, over the scores it came from, and is the A operand from there: the products of a
//               head are issued in order, so that the next scores overwrite P only when P V has read it, and their arrival tells
//               the softmax that O is stable (it rescales O in place, where the row maximum grew by more than 2^8)
//
// TMEM: S0 S1 O0 O1, 128 columns each: all 512.
// Bound by the tensor pipe and the exponentials, 2048 cycles each per key tile of both heads. Measured on B200 (bf16, 64 heads on 8):
// 8192 tokens behind 8192: 4421 -> 2702 us (1221 TFLOP/s); 8192 from the start: 1627 -> 1144 (962); 2048: 156 -> 125; 6 x 300: 75 -> 61.
#pragma once

namespace hds {

constexpr int kPairSlots = 5;
constexpr size_t kPairTile = 128 * 128 * 2;      // 128 rows x 128 dims of 16 bits: two 64-dim panels
constexpr size_t kPairSmemBytes = 2 * kPairTile + kPairSlots * kPairTile + 256 + 1024;

__device__ __forceinline__ uint64_t pack_f32x2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

template <bool kBf16, int kWeights>
__global__ void __launch_bounds__(kPfThreads, 1)
paged_attn_pair_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_kv, const PrefillArgs a) {
    constexpr bool kSigmoid = kWeights == PF_SIGMOID, kCapped = kWeights == PF_CAPPED;
    constexpr int D = 128, PANEL_BYTES = kPfTok * 128;
    constexpr uint32_t IDESC_QK = make_idesc_f16(128, kPfTok, kBf16, false, false);
    constexpr uint32_t IDESC_PV = make_idesc_f16(128, D, kBf16, false, true);  // B = V is MN-major

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* q_sm = smem;                          // [head][panel][128 x 64]
    uint8_t* ring = smem + 2 * kPairTile;
    uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kPairSlots * kPairTile);
    uint64_t* q_full = bars;
    uint64_t* full = bars + 1;
    uint64_t* empty = full + kPairSlots;
    uint64_t* s_full = empty + kPairSlots;   // [head] S of a tile is there (and P V of the tile before is done)
    uint64_t* p_full = s_full + 2;           // [head] P is there (and O rescaled)
    uint64_t* o_full = p_full + 2;           // [head] the last P V is done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);

    const uint32_t warp = warp_id(), lane = lane_id();
    pdl_enter();
    const int item_idx = static_cast<int>(gridDim.x - 1 - blockIdx.x);   // heaviest first, as in the one-head kernel
    const hds_attn_item item = a.items[item_idx];
    const int head0 = blockIdx.y * 2;
    const int kvh = head0 / (a.n_q_heads / a.n_kv_heads);
    const int kv_len = item.pos0 + item.n_q;
    const int tiles_total = (kv_len + kPfTok - 1) / kPfTok;
    const int tile_first = a.window > 0 ? max(0, item.pos0 - a.window + 1) / kPfTok : 0;
    const int tiles_keep = min((a.keep_first + kPfTok - 1) / kPfTok, tile_first);
    const int tiles_skip = tile_first - tiles_keep;
    const int n_tiles = tiles_total - tiles_skip;
    auto key_tile = [&](int ti) { return ti < tiles_keep ? ti : ti + tiles_skip; };
    // place of a tile in the producer's order
    auto seq_k = [](int ti) { return ti == 0 ? 0 : 2 * ti - 1; };
    auto seq_v = [&](int ti) { return ti == n_tiles - 1 ? 2 * n_tiles - 1 : 2 * ti + 2; };

    if (warp == 0 && lane == 0) {
        prefetch_tmap(&tmap_q);
        prefetch_tmap(&tmap_kv);
        mbar_init(q_full, 1);
        for (int i = 0; i < kPairSlots; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(&s_full[h], 1);
            mbar_init(&p_full[h], 4);
            mbar_init(&o_full[h], 1);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc<512>(tmem_slot);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(q_full, 2 * kPairTile);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                tma_load_2d(q_sm + i * PANEL_BYTES, &tmap_q, q_full, (head0 + (i >> 1)) * D + (i & 1) * 64, item.q_row0, kEvictFirst);
            const int32_t* table = a.block_tables + static_cast<int64_t>(item.seq) * a.max_blocks_per_seq;
            const int bs = a.block_size, bps = kPfTok / bs, last_blk_idx = (kv_len - 1) / bs;
            uint32_t slot = 0, phase = 0;
            auto load = [&](int ti, int which) {
                mbar_wait(&empty[slot], phase ^ 1);
                uint8_t* dst = ring + slot * kPairTile;
                mbar_expect_tx(&full[slot], kPairTile);
                for (int b = 0; b < bps; ++b) {
                    // past the end of the sequence its last page again: hidden later, but every V value stays finite
                    const int blk = table[min(key_tile(ti) * bps + b, last_blk_idx)];
                    const int row = ((blk * 2 + which) * a.n_kv_heads + kvh) * bs;
#pragma unroll
                    for (int p = 0; p < 2; ++p) tma_load_2d(dst + p * PANEL_BYTES + b * bs * 128, &tmap_kv, &full[slot], p * 64, row, kEvictNormal);
                }
                if (++slot == kPairSlots) {
                    slot = 0;
                    phase ^= 1;
                }
            };
            load(0, 0);
            for (int ti = 0; ti < n_tiles; ++ti) {
                if (ti + 1 < n_tiles) load(ti + 1, 0);
                load(ti, 1);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            auto wait_full = [&](int seq) { mbar_wait(&full[seq % kPairSlots], (seq / kPairSlots) & 1); };
            auto issue_qk = [&](int h, int seq) {
                const uint8_t* ktile = ring + (seq % kPairSlots) * kPairTile;
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const uint64_t dq = make_desc_kmajor_sw128(smem_u32(q_sm + (h * 2 + p) * PANEL_BYTES));
                    const uint64_t dk = make_desc_kmajor_sw128(smem_u32(ktile + p * PANEL_BYTES));
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_f16_ss(tmem_base + h * 128, dq + 2 * k, dk + 2 * k, IDESC_QK, (p > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(&s_full[h]);
            };
            mbar_wait(q_full, 0);
            wait_full(0);
            tc_fence_after();
            issue_qk(0, 0);
            issue_qk(1, 0);
            umma_commit(&empty[0]);
            for (int ti = 0; ti < n_tiles; ++ti) {
                const int sv = seq_v(ti), sk = seq_k(ti + 1);
                const bool more = ti + 1 < n_tiles;
                if (more) wait_full(sk);       // (it comes before V)
                wait_full(sv);
                const uint8_t* vtile = ring + (sv % kPairSlots) * kPairTile;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    mbar_wait(&p_full[h], ti & 1);
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < kPfTok / 16; ++kk)
                        umma_f16_ts(tmem_base + 256 + h * 128, tmem_base + h * 128 + kk * 8,
                                    make_desc_mnmajor_sw128(smem_u32(vtile + kk * 16 * 128), PANEL_BYTES), IDESC_PV, (ti > 0 || kk > 0) ? 1u : 0u);
                    if (h == 1) umma_commit(&empty[sv % kPairSlots]);
                    if (more) issue_qk(h, sk);
                    else umma_commit(&o_full[h]);
                }
                if (more) umma_commit(&empty[sk % kPairSlots]);
            }
        }
    } else {
        // ===================== softmax / output: one thread per query row =====================
        const uint32_t quad = warp & 3;              // TMEM lane quadrant this warp may touch
        const int h = (warp - 2) >> 2;
        const int r = quad * 32 + lane;
        const int head = head0 + h;
        const int q_pos = item.pos0 + r;
        const bool quad_live = static_cast<int>(quad * 32) < item.n_q;   // warp-uniform
        const uint32_t tmem_s = tmem_base + h * 128 + ((quad * 32u) << 16);
        const uint32_t tmem_o = tmem_s + 256;
        const float to_log2 = kCapped ? 1.0f : a.scale_log2;
        const float sig_bias = kSigmoid ? a.sigmoid_bias[head] * -1.4426950408889634f : 0.0f;
        constexpr float kRescaleThreshold = 8.0f;    // log2 units: probabilities stay below 2^8 against a stale max
        float m_run = kSigmoid ? 0.0f : -INFINITY, l_run = 0.0f;
        for (int ti = 0; ti < n_tiles; ++ti) {
            mbar_wait(&s_full[h], ti & 1);
            tc_fence_after();
            if (!quad_live) {
                if (lane == 0) mbar_arrive(&p_full[h]);
                continue;
            }
            const int tile0 = key_tile(ti) * kPfTok;
            const bool need_mask = tile0 + kPfTok - 1 > item.pos0 || (a.window > 0 && tile0 <= item.pos0 + item.n_q - 1 - a.window);
            uint32_t sr[128];
#pragma unroll
            for (int c = 0; c < 128; c += 32) tmem_ld_32x32(tmem_s + c, *reinterpret_cast<uint32_t(*)[32]>(&sr[c]));
            tmem_ld_wait();
            if constexpr (kCapped) {
#pragma unroll
                for (int j = 0; j < 128; ++j) sr[j] = __float_as_uint(softcap_log2(__uint_as_float(sr[j]), a.cap_k, a.cap_log2));
            }
            if (need_mask) {
                const int win_lo = a.window > 0 ? q_pos - a.window : -(1 << 30);   // keys at or before this position are hidden
#pragma unroll
                for (int j = 0; j < 128; ++j) {
                    const int kv_pos = tile0 + j;
                    if (!(kv_pos <= q_pos && kv_pos < kv_len && (kv_pos > win_lo || kv_pos < a.keep_first))) sr[j] = __float_as_uint(-INFINITY);
                }
            }
            if constexpr (kSigmoid) {
#pragma unroll
                for (int c = 0; c < 128; c += 64) {
                    uint32_t packed[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {     // (hidden keys: 1 / (1 + inf) = 0)
                        const float p0 = rcp_approx(1.0f + ex2_approx(fmaf(__uint_as_float(sr[c + 2 * j]), -a.scale_log2, sig_bias)));
                        const float p1 = rcp_approx(1.0f + ex2_approx(fmaf(__uint_as_float(sr[c + 2 * j + 1]), -a.scale_log2, sig_bias)));
                        packed[j] = pack2<kBf16>(p0, p1);
                    }
                    tmem_st_32x32(tmem_s + c / 2, packed);
                }
            } else {
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int j = 0; j < 128; j += 8)
#pragma unroll
                    for (int i = 0; i < 4; ++i) mx[i] = fmaxf(mx[i], fmaxf(__uint_as_float(sr[j + 2 * i]), __uint_as_float(sr[j + 2 * i + 1])));
                const float tmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                // lazy rescale: move the reference max only when it grew by more than the threshold
                const float m_cand = fmaxf(m_run, tmax * to_log2);
                const bool fresh = (m_run == -INFINITY);   // nothing accumulated for this row yet
                const bool grow = (m_cand > m_run + kRescaleThreshold) || (fresh && m_cand != -INFINITY);
                const float m_new = grow ? m_cand : m_run;
                const float alpha = (!grow || fresh) ? (grow ? 0.0f : 1.0f) : ex2_approx(m_run - m_new);
                const float m_sub = (m_new == -INFINITY) ? 0.0f : m_new;  // fully masked row: exp2(-inf - 0) = 0
                m_run = m_new;
                if (ti > 0 && __any_sync(0xffffffffu, grow && !fresh)) {     // (S has arrived: P V of the tile before is done)
                    const float f = grow && !fresh ? alpha : 1.0f;
#pragma unroll
                    for (int c = 0; c < D; c += 16) {
                        uint32_t orr[16];
                        tmem_ld_32x16(tmem_o + c, orr);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; ++j) orr[j] = __float_as_uint(__uint_as_float(orr[j]) * f);
                        tmem_st_32x16(tmem_o + c, orr);
                    }
                }
                const uint64_t k2 = pack_f32x2(to_log2, to_log2), m2 = pack_f32x2(-m_sub, -m_sub);
                uint64_t sum[2] = {0ull, 0ull};
#pragma unroll
                for (int c = 0; c < 128; c += 64) {
                    uint32_t packed[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        float x0, x1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(sr[c + 2 * j]), __uint_as_float(sr[c + 2 * j + 1])), k2, m2), x0, x1);
                        x0 = ex2_approx(x0);
                        x1 = ex2_approx(x1);
                        sum[j & 1] = add_f32x2(sum[j & 1], pack_f32x2(x0, x1));
                        packed[j] = pack2<kBf16>(x0, x1);
                    }
                    tmem_st_32x32(tmem_s + c / 2, packed);
                }
                float u0, u1;
                unpack_f32x2(add_f32x2(sum[0], sum[1]), u0, u1);
                l_run = l_run * alpha + (u0 + u1);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[h]);
        }
        mbar_wait(&o_full[h], 0);
        tc_fence_after();
        if (quad_live) {
            const float inv = r < item.n_q ? pf_row_factor<kSigmoid>(a, l_run, m_run, head) : 0.0f;
            const int64_t out_row = item.q_row0 + r;
#pragma unroll
            for (int c = 0; c < D; c += 32) {
                uint32_t orr[32];
                tmem_ld_32x32(tmem_o + c, orr);
                tmem_ld_wait();
                float o[32];
#pragma unroll
                for (int j = 0; j < 32; ++j) o[j] = __uint_as_float(orr[j]);
                if (r < item.n_q) {
#pragma unroll
                    for (int j = 0; j < 32; j += 8) pf_store8<kBf16>(a, o + j, inv, out_row, head * D + c + j);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<512>(tmem_base);
    }
}

}  // namespace hds
