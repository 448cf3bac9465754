// Weight-streaming tcgen05 GEMM for decode-size M (<= 64 tokens):  D[M,N] = X[M,K] * W[N,K]^T
//
// The operands are swapped relative to gemm_core.cuh: the 128 rows of the MMA are 128 output FEATURES (a
// 128 x 64 weight tile, K-major, straight from the [N, K] checkpoint layout) and the MMA's N side is the token
// tile (NT = 16 / 32 / 64 tokens). A 128 x NT x 16 tcgen05.mma costs NT/128 of the tensor-pipe time of the
// token-major 128 x 128 x 16 instruction for the same 4 KB of weights, so the tensor pipe stops being the limit
// of a skinny GEMM and the kernel is a pure HBM stream. To keep enough bytes in flight without a persistent
// schedule each CTA owns ONE (feature tile, K split) unit and 2-3 CTAs are resident per SM (4-5 stages of
// 16 KB weights each); prologue / epilogue of one CTA overlap the streaming of its neighbours.
//
//   warp 0   : TMA producer         warp 1 : TMEM alloc + MMA issuer        warps 2-5 : epilogue
//   accumulator: TMEM lanes = features, columns = tokens  ->  one epilogue thread owns one output feature
//
// Epilogues: store (+bias +act), gated (interleaved gate/up rows of W -> act(g)*u; the partner feature lives
// in the neighbouring lane), fp32 accumulate into the pending residual delta (split-K needs no meeting there).
// The K splits of a store / gated tile are a cluster (up to 8): each leaves its sums in its shared memory, behind the cluster's barrier
// CTA r adds up the tokens r, r + splits, ... of all of them and stores those. Through an fp32 scratch in global memory, with
// atomic sums and tickets, the end of a tile took 1 - 2 us more: one token, weights read from memory (300 MB of them in turn),
// 12288 x 4096 19.8 us so and 17.6 now, the gated 22016 x 4096 31.4 and 29.0 us (6.2 TB/s), 2048 x 2048 6.5 and 4.5.
//
// Role in the reference: the cuBLAS GEMMs of a decode step (core_ops/blas_kernels/blas.h:31-136) plus the
// bias / gated activation kernels that follow them.
#pragma once
#include "gemm_core.cuh"

namespace hds {

constexpr int kSkinnyBF = 128;  // features per CTA (MMA M)

// Grouped (experts): a few hundred units at most, so two CTAs per SM with as many stages as fit keep more bytes in flight than three
// with four each would when not all of them are there.
__host__ __device__ constexpr int skinny_stages(int nt, bool grouped = false) { return grouped ? (nt == 64 ? 4 : nt == 32 ? 5 : 6) : nt == 32 ? 5 : 4; }
__host__ __device__ constexpr int skinny_occupancy(int nt, bool grouped = false) { return nt == 16 && !grouped ? 3 : 2; }
__host__ __device__ constexpr size_t skinny_smem_bytes(int nt, bool grouped = false) {
    return static_cast<size_t>(skinny_stages(nt, grouped)) * (kSkinnyBF * kGemmBK * 2 + nt * kGemmBK * 2) + 256 + 1024;
}

// K splits of a decode GEMM of n_tiles feature tiles. Measured: fill the resident slots once;
// past one full wave of tiles, split until the waves are >= 80 % full (448 tiles of a 57344-wide MLP-1: 5.25 -> 5.66 TB/s at 4
// splits). At most 8, the size of a portable cluster; a count that the caller gives is held to that where the splits meet in one (`clusters`),
// and to the K blocks where they add up in memory. A cluster needs its slots in one GPC, so that some stay empty: where the splits
// meet in one, they fill no more than 87 % (96 tiles x 3 of 296 slots: 27.7 us at 17 tokens of 12288 x 4096, 20.4 us in 2). Past one
// wave clusters of more than 16 tokens are slower than the empty slots of a last wave (64 tokens, unsplit and in 2 or 3: 57344 x 8192 148.3
// and 170.3 us, 57344 x 2048 45.2 and 71.2, 50272 x 4096 77.3 and 82.4), but for long rows on a wave less than 60 % full (17 tokens of
// 43008 x 8192: 124.2 and 117.7).
inline int skinny_splits(int n_tiles, int kb_total, int nt, int want, int sms, bool clusters) {
    int splits = want;
    if (want <= 0) {
        const int slots = sms * skinny_occupancy(nt);
        splits = slots / n_tiles;
        if (clusters && n_tiles <= slots)
            while (splits > 1 && static_cast<int64_t>(n_tiles) * (splits < 8 ? splits : 8) * 100 > static_cast<int64_t>(slots) * 87) --splits;
        if (n_tiles > slots) {
            splits = 1;
            for (int s = 1; s <= 8; ++s) {
                const int64_t ctas = static_cast<int64_t>(n_tiles) * s;
                const int64_t waves = (ctas + slots - 1) / slots;
                if (ctas * 100 >= waves * slots * 80) {
                    splits = s;
                    break;
                }
            }
            const int64_t waves = (n_tiles + slots - 1) / slots;
            if (clusters && nt > 16 && !(kb_total >= 128 && static_cast<int64_t>(n_tiles) * 100 < waves * slots * 60)) splits = 1;
        }
        if (splits > kb_total / 4) splits = kb_total / 4;
    }
    if (splits > 8 && (clusters || want <= 0)) splits = 8;
    if (splits > kb_total) splits = kb_total;
    return splits < 1 ? 1 : splits;
}

struct SkinnyArgs {
    int M, N, K;
    int splits, kb_per_split;
    int act;
    float act_limit;    // ACT_SWIGLU_CLAMPED: the bound L
    void* out;          // EPI_STORE / EPI_GATED
    int64_t ldo;
    const void* bias;   // [N] I/O dtype, may be null
    float* accum;       // EPI_RED_F32: [M, ld_accum] fp32, accumulated with red.global.add
    int64_t ld_accum;
    const float* a_scale;  // fp8 operands only: per-token scales [M]
    const float* w_scale;  // fp8 operands only: per-feature scales [N]
    uint32_t idesc_or;     // fp8 kernels: operand-format bits for 6-bit (E3M2) weights, else 0
    uint32_t w_tx_bytes;   // bytes one weight-tile TMA load reports to the mbarrier (0 = the tile's shared-memory size)
    const int32_t* group_pad_off;  // kGrouped: expert e owns the rows [pad_off[e], pad_off[e + 1]) of X and of the output (none if empty),
    int n_groups;                  // the first M of them at most live, and the N weight rows from e * N on
    TpSync sync;           // tensor parallel: the producer acquires the peers' flags before its first activation load
                           // (sync.wait); the last CTA to retire releases the output to the peers (sync.signal)
};

template <int NT>
__device__ __forceinline__ void skinny_tmem_load(uint32_t taddr, float (&v)[NT]) {
    if constexpr (NT == 16) {
        uint32_t r[16];
        tmem_ld_32x16(taddr, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
    } else {
#pragma unroll
        for (int c = 0; c < NT; c += 32) {
            uint32_t r[32];
            tmem_ld_32x32(taddr + c, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[c + j] = __uint_as_float(r[j]);
        }
    }
}

// Final store of one feature column (this thread) for the live ones of the tokens t0, t0 + dt, ..., in rows row0 on. For the gated form
// the whole warp must call (shuffles): even lanes hold gate features, odd lanes the matching up features.
template <int NT, bool kBf16, bool kGated>
__device__ __forceinline__ void skinny_finalize(const SkinnyArgs& a, int n, uint32_t lane, float (&v)[NT], int t0 = 0, int dt = 1, int row0 = 0) {
    const bool live = n < a.N;
    const float b = (a.bias != nullptr && live) ? load_scalar<kBf16>(a.bias, n) : 0.0f;
#pragma unroll
    for (int t = 0; t < NT; ++t) v[t] += b;
    if constexpr (kGated) {
        // even lanes hold gate features (activated), odd lanes the matching up features (left as they are)
        if (a.act == ACT_SWIGLU_CLAMPED) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const float c = fminf(v[t], a.act_limit);
                v[t] = (lane & 1) ? fmaxf(c, -a.act_limit) + 1.0f : __fdividef(c, 1.0f + __expf(-kClampedGluAlpha * c));
            }
        } else {
            apply_act_vec<NT>(v, (lane & 1) ? static_cast<int>(ACT_IDENTITY) : a.act);
        }
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            const float partner = __shfl_xor_sync(0xffffffffu, v[t], 1);
            if (live && !(lane & 1) && t0 + t * dt < a.M)
                store_scalar<kBf16>(a.out, static_cast<int64_t>(row0 + t0 + t * dt) * a.ldo + (n >> 1), v[t] * partner);
        }
    } else {
        if (!live) return;
        apply_act_vec<NT>(v, a.act);
#pragma unroll
        for (int t = 0; t < NT; ++t)
            if (t0 + t * dt < a.M) store_scalar<kBf16>(a.out, static_cast<int64_t>(row0 + t0 + t * dt) * a.ldo + n, v[t]);
    }
}

// a float of CTA `cta` of the cluster, at the place where `p` is in this one
__device__ __forceinline__ float cluster_load(const float* p, uint32_t cta) {
    float v;
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %1, %2;\n\tld.shared::cluster.f32 %0, [ra];\n\t}\n"
                 : "=f"(v) : "r"(smem_u32(p)), "r"(cta) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// kFp8: both operands are E4M3 codes (a 128-byte row of a tile then holds 128 K-elements instead of 64, i.e. half the
// weight bytes per MAC); the accumulator is scaled by w_scale[feature] * a_scale[token] right after it leaves TMEM, so
// split-K partial sums and all three epilogues see real-valued numbers. kBf16 then names the OUTPUT / bias dtype.
// kGrouped: the experts of a decode step. A unit is (the i-th expert that has rows, feature tile); which experts these are is known
// to the routing kernels before it only, so nothing is requested ahead of them. Every expert's weights are streamed once: the
// token-major kernel's 256-wide tiles are too few for that (8 tokens x top 2 of 16 experts of 2048 x 2688: 35 us up and 26 us down,
// 3.6 TB/s).
// kMeet: the K splits of a store / gated tile, a cluster. A form of its own, because what it adds costs unsplit tiles up to 7 %.
template <int NT, int EPI, bool kBf16, bool kFp8 = false, bool kGrouped = false, bool kMeet = false>
__global__ void __launch_bounds__(kGemmThreads, skinny_occupancy(NT, kGrouped))
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const SkinnyArgs args) {
    constexpr int STAGES = skinny_stages(NT, kGrouped);
    constexpr uint32_t W_BYTES = kSkinnyBF * kGemmBK * 2;
    constexpr uint32_t X_BYTES = NT * kGemmBK * 2;
    constexpr uint32_t TMEM_COLS = NT < 32 ? 32 : NT;
    constexpr uint32_t IDESC = kFp8 ? make_idesc_f8(kSkinnyBF, NT) : make_idesc_f16(kSkinnyBF, NT, kBf16, false, false);
    constexpr int KB = kFp8 ? 2 * kGemmBK : kGemmBK;  // K-elements per 128-byte tile row
    static_assert(NT == 16 || NT == 32 || NT == 64, "token tile must be 16, 32 or 64");

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* smem_w = smem;
    uint8_t* smem_x = smem + STAGES * W_BYTES;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * (W_BYTES + X_BYTES));
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* tfull_bar = empty_bar + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull_bar + 1);

    const uint32_t warp = warp_id();
    const uint32_t lane = lane_id();
    const int n_tiles = (args.N + kSkinnyBF - 1) / kSkinnyBF;
    const int kb_total = (args.K + KB - 1) / KB;
    // (kGrouped: sp is the place of the expert; else the K split, whose CTAs are neighbours where they are a cluster)
    static_assert(!kMeet || (EPI != EPI_RED_F32 && !kGrouped), "the other forms have nothing to meet for");
    const int n_t = kMeet ? static_cast<int>(blockIdx.x) / args.splits : static_cast<int>(blockIdx.x) % n_tiles;
    const int sp = kMeet ? static_cast<int>(blockIdx.x) % args.splits : static_cast<int>(blockIdx.x) / n_tiles;
    const int kb0 = kGrouped ? 0 : sp * args.kb_per_split;
    const int kb1 = min(kb_total, kb0 + args.kb_per_split);
    const uint32_t w_tx = args.w_tx_bytes ? args.w_tx_bytes : W_BYTES;

    if (warp == 0 && lane == 0) {
        prefetch_tmap(&tmap_w);
        prefetch_tmap(&tmap_x);
        for (int i = 0; i < STAGES; ++i) {
            mbar_init(&full_bar[i], 1);
            mbar_init(&empty_bar[i], 1);
        }
        mbar_init(tfull_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc<TMEM_COLS>(tmem_slot);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    griddep_launch_dependents();
    int x_row = 0, w_row = n_t * kSkinnyBF;   // first row of the activations and of the weight tile
    if constexpr (kGrouped) {
        // every warp looks for the sp-th expert with rows (kb_per_split covers K: sp is not a split here)
        griddep_wait();
        int left = sp, e = -1;
        for (int e0 = 0; e0 < args.n_groups && e < 0; e0 += 32) {
            const int i = e0 + static_cast<int>(lane);
            const bool has = i < args.n_groups && args.group_pad_off[i + 1] > args.group_pad_off[i];
            const uint32_t m = __ballot_sync(0xffffffffu, has);
            if (left < __popc(m)) e = e0 + static_cast<int>(__fns(m, 0, left + 1));
            else left -= __popc(m);
        }
        if (e < 0) {      // fewer experts than units: the whole CTA leaves
            tc_fence_before();
            __syncthreads();
            if (warp == 1) {
                tc_fence_after();
                tmem_dealloc<TMEM_COLS>(tmem_base);
            }
            if (args.sync.signal) tp_signal_tail(args.sync, gridDim.x);
            return;
        }
        x_row = args.group_pad_off[e];
        w_row += e * args.N;
    }
    if (warp == 0) {
        if (lane == 0) {
            // Weights are never written by a kernel: the first STAGES weight tiles are requested BEFORE waiting for
            // the previous kernel (PDL), so HBM keeps streaming across the kernel boundary; the activation tiles
            // (produced by the predecessor) follow after the wait and complete the same stage barriers.
            const int pre = min(STAGES, kb1 - kb0);
            for (int i = 0; i < pre; ++i) {
                mbar_expect_tx(&full_bar[i], w_tx + X_BYTES);
                tma_load_2d(smem_w + i * W_BYTES, &tmap_w, &full_bar[i], (kb0 + i) * KB, w_row, kEvictFirst);
            }
            griddep_wait();
            if (args.sync.wait) {  // tensor parallel: the activations were all-gathered into this buffer by the peers
                tp_wait_thread(args.sync);
                fence_proxy_async_global();
            }
            for (int i = 0; i < pre; ++i)
                tma_load_2d(smem_x + i * X_BYTES, &tmap_x, &full_bar[i], (kb0 + i) * KB, x_row, kEvictLast);
            uint32_t stage = 0, phase = 1;  // the ring has been filled once
            for (int kb = kb0 + pre; kb < kb1; ++kb) {
                mbar_wait(&empty_bar[stage], phase ^ 1);
                mbar_expect_tx(&full_bar[stage], w_tx + X_BYTES);
                tma_load_2d(smem_x + stage * X_BYTES, &tmap_x, &full_bar[stage], kb * KB, x_row, kEvictLast);
                tma_load_2d(smem_w + stage * W_BYTES, &tmap_w, &full_bar[stage], kb * KB, w_row, kEvictFirst);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t stage = 0, phase = 0;
            for (int kb = kb0; kb < kb1; ++kb) {
                mbar_wait(&full_bar[stage], phase);
                tc_fence_after();
                const uint64_t dw = make_desc_kmajor_sw128(smem_u32(smem_w + stage * W_BYTES));
                const uint64_t dx = make_desc_kmajor_sw128(smem_u32(smem_x + stage * X_BYTES));
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // 32 bytes of K per instruction: 16 (16-bit) or 32 (fp8) elements
                    if constexpr (kFp8) umma_f8_ss(tmem_base, dw + 2 * k, dx + 2 * k, IDESC | args.idesc_or, (kb > kb0 || k > 0) ? 1u : 0u);
                    else umma_f16_ss(tmem_base, dw + 2 * k, dx + 2 * k, IDESC, (kb > kb0 || k > 0) ? 1u : 0u);
                }
                umma_commit(&empty_bar[stage]);
                if (++stage == STAGES) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            umma_commit(tfull_bar);
        }
    } else {
        const uint32_t quad = warp & 3;
        const int n = n_t * kSkinnyBF + static_cast<int>(quad * 32 + lane);
        griddep_wait();  // this warp writes global memory the previous kernel may still be reading
        mbar_wait(tfull_bar, 0);
        tc_fence_after();
        float v[NT];
        skinny_tmem_load<NT>(tmem_base + ((quad * 32u) << 16), v);
        if constexpr (kFp8) {
            const float sw = n < args.N ? __ldg(args.w_scale + n) : 0.0f;
#pragma unroll
            for (int t = 0; t < NT; ++t) v[t] *= sw * (t < args.M ? __ldg(args.a_scale + t) : 0.0f);
        }
        if constexpr (EPI == EPI_RED_F32) {
            if (n < args.N) {
                const float b = (args.bias != nullptr && sp == 0) ? load_scalar<kBf16>(args.bias, n) : 0.0f;
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    if (t < args.M) atomicAdd(args.accum + static_cast<int64_t>(t) * args.ld_accum + n, v[t] + b);
            }
        } else {
            constexpr bool kGated = EPI == EPI_GATED;
            if constexpr (!kMeet) {
                skinny_finalize<NT, kBf16, kGated>(args, n, lane, v, 0, 1, x_row);
            } else {      // (the stages are free: every product has been read out of them)
                float* part = reinterpret_cast<float*>(smem) + quad * 32 + lane;
#pragma unroll
                for (int t = 0; t < NT; ++t)
                    if (t < args.M) part[t * kSkinnyBF] = v[t];
            }
        }
    }
    if constexpr (kMeet) {
        __syncwarp();
        cluster_sync();       // every split's sums are there
        if (warp >= 2) {
            constexpr int C = 4;      // tokens at a time
            const uint32_t quad = warp & 3;
            const int n = n_t * kSkinnyBF + static_cast<int>(quad * 32 + lane);
            const float* part = reinterpret_cast<const float*>(smem) + quad * 32 + lane;
            for (int t0 = sp; t0 < args.M; t0 += C * args.splits) {
                float v[C] = {};
                for (int s = 0; s < args.splits; ++s)
#pragma unroll
                    for (int i = 0; i < C; ++i) v[i] += cluster_load(part + min(t0 + i * args.splits, args.M - 1) * kSkinnyBF, s);
                skinny_finalize<C, kBf16, EPI == EPI_GATED>(args, n, lane, v, t0, args.splits);
            }
        }
        __syncwarp();
        cluster_sync();       // nobody leaves while its sums are read
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc<TMEM_COLS>(tmem_base);
    }
    if (args.sync.signal) tp_signal_tail(args.sync, gridDim.x);
}

}  // namespace hds
