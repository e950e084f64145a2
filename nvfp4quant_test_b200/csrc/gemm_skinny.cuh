// Decode-sized kernel of the NVFP4 GEMM: weights on the MMA rows, K ranges across a thread-block cluster.
#pragma once

#include "gemm_pair.cuh"

namespace nvfp4 {
namespace gemm {

// =============================================================================================
// Skinny variant for decode-sized batches (M <= 128).  The roles of the operands are swapped: the 128 rows of
// the MMA are WEIGHT rows and its N dimension is the (padded) token count BT = 16 / 32 / 64 / 128, so the tensor
// cores spend BT/128 of the time a 128-row token tile of mostly padding would take and the kernel is a
// stream of the weights.  One CTA owns 128 weight rows and one K range; the K ranges of a tile are the CTAs
// of one thread-block cluster (1..8), which lets a shape with few weight tiles still pull from every SM.
// The partial accumulators are combined by a reduce-scatter through distributed shared memory: the token
// columns are dealt out to the ranks, every rank writes its partial tile to its own shared memory and sends
// each other rank the columns that rank owns with one bulk copy (cp.async.bulk shared::cta -> shared::cluster,
// completion counted on the receiver's mbarrier) into an area that nothing else uses; the owner adds the partials in ascending rank order, applies
// alpha and stores bf16.  One kernel, no workspace, and the result does not depend on timing.  Every copy has
// one destination CTA (no multicast).
// =============================================================================================
namespace skinny {

using pair::cluster_arrive;
using pair::cluster_ctarank;
using pair::cluster_sync_all;
using pair::cluster_wait;
using pair::map_to_cta;

constexpr int kMaxStages = 8;
constexpr int kBarrierBytes = 256;
constexpr int kSlack = 1024;   // a ring that starts at a rounded address of the launch measured 2 to 5 % faster than one at a fixed offset
// Stages of prepared weights that are requested ahead of the wait for the kernel before this one.  A CTA's copies are carried out in
// order: the token tile of the first stage, without which none is consumed and none is requested again, comes behind them all.
// Raw weights have none ahead and each stage's operands side by side; all weights of a ring of eight first, then the tokens: us, raw, 16
// x 14336 x 8192 15.23 -> 14.38, 1 x 14336 x 4096 9.99 -> 9.04, 16 x 16384 x 2048 7.62 -> 6.69, 4 x 11000 x 4096 9.46 -> 8.48; prepared, eight
// ahead / five, behind a product 14.09 / 13.78, 8.49 / 8.25, 6.48 / 6.29, 8.09 / 7.87, behind the quantizer 15.66 / 15.57, 10.00 / 9.47, 8.09 /
// 7.55, 9.26 / 9.20 (three 16.08, 9.90, 7.23, 9.71).
constexpr int kAhead = 5;
// TMEM: accumulator in columns 0..BT-1, then two scale sets of 32 columns

template <int BT>
struct SkinnyCfg {
    static constexpr int kWBytes = 128 * kBKBytes;     // 128 weight rows x 256 codes
    static constexpr int kXBytes = BT * kBKBytes;      // BT token rows x 256 codes
    static constexpr int kSfBytes = 2048;              // one 128-row scale group x 16 blocks, for each operand
    static constexpr int kStageBytes = kWBytes + kXBytes + 2 * kSfBytes;
    static constexpr int kSfCol = BT <= 64 ? 64 : 128; // scale set 0: weights +0..15, tokens +16..31; set 1: +32
    static constexpr int kTmemCols = BT <= 64 ? 128 : 256;
    static constexpr int kMaxStages = (BT <= 64) ? 8 : 6;
    static_assert(kStageBytes % 1024 == 0, "stage alignment for the 128-byte swizzle");
    static_assert(BT % 16 == 0 && BT >= 16 && BT <= 128, "token tile");
};

__device__ __forceinline__ void tc_ld_32x32b_x16(uint32_t taddr, uint32_t v[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}
// shared memory of this CTA -> shared memory of a CTA of the cluster; the bytes are counted on the receiver's barrier
__device__ __forceinline__ void bulk_copy_to_cta(uint32_t dst_cluster, uint32_t src_cta, uint32_t bytes, uint32_t bar_cluster) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster),
                 "r"(src_cta), "r"(bytes), "r"(bar_cluster)
                 : "memory");
}

// One launch may hold several products of equal M (a layer's q / k / v, or gate / up projections, or all of its matrices):
// the weight tiles of all of them are numbered through, and a CTA looks up whose tile it owns.  The launch's fixed costs
// (prologue, ramp-up and drain of the weight stream) are then paid once per group.
constexpr int kMaxGroup = 8;

struct SkinnyWeight {
    const uint8_t* sfw;   // weight scales
    const uint8_t* sfx;   // token scales (group 0 of the tiled layout)
    const float* alpha_x; // optional second factor of the output scale
    const float* alpha;   // output scale of this weight (times alpha_x when that is given)
    __nv_bfloat16* out;   // [M, N]
    int N, K;
    int k_tiles_per_rank;
    int ranks;            // K ranges of a tile: a power of two of the cluster's CTAs, or all of them
    int tiles;            // tiles of a cluster: its CTAs / ranks
    int rank_shift;       // a CTA's tile among the cluster's: its rank in the cluster >> rank_shift
    int64_t sf_group_stride;
    int cluster_end;      // clusters of this and all earlier weights of the group
};

// G: products the launch has room for; 1 for the usual case, whose parameters then stay small.
template <int G>
struct SkinnyParams {
    int M;
    int stages;
    int n_weights;
    int apart;            // one product only: the other ranks' partials have a place behind the ring
    int weights_ready;    // != 0: all weights are prepared weights (constant while in use): read them before griddep_wait()
    SkinnyWeight w[G];
};

template <int G>
struct SkinnyMaps {
    CUtensorMap m[G];        // one per weight: [N, K/2] bytes in boxes of 128 rows x 128 bytes
    CUtensorMap m_rest[G];   // and of the N % 128 last rows (see TileParams)
    CUtensorMap x[G];        // its activation: [M, K/2] bytes in boxes of M rows
};

template <int BT, int G>
__global__ void __launch_bounds__(kThreads)
skinny_kernel(const __grid_constant__ SkinnyMaps<G> maps, const __grid_constant__ SkinnyParams<G> p) {
    using C = SkinnyCfg<BT>;
    // Where the ranks' partials meet: behind the ring, or in it.  See the epilogue.
    const bool apart = G == 1 && p.apart;
    extern __shared__ uint8_t smem_raw[];
    // The kernel queued behind this one may be scheduled at once: ahead of its own wait it reads nothing but a
    // prepared (constant) weight, and that wait covers this kernel's completion.
    griddep_launch();
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - raw_addr);
    const int nstages = p.stages;
    uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + nstages * C::kStageBytes);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kMaxStages + s); };
    const uint32_t tfull_bar = bar_base + 8u * (2 * kMaxStages);
    const uint32_t recv_bar = bar_base + 8u * (2 * kMaxStages + 1);   // partials from the other ranks have landed
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * kMaxStages + 2);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    // Clusters run along x and are numbered through the weights of the group.  A cluster holds cluster / ranks weight tiles of
    // one weight, a tile's K ranges side by side.
    const uint32_t crank = cluster_ctarank();
    uint32_t cluster, cluster_id;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(cluster));
    asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(cluster_id));
    int gi = 0;
    if (G > 1)
        while (gi + 1 < p.n_weights && static_cast<int>(cluster_id) >= p.w[gi].cluster_end) ++gi;
    const uint32_t ranks = G > 1 ? static_cast<uint32_t>(p.w[gi].ranks) : cluster;
    const uint32_t sub = G > 1 ? crank >> p.w[gi].rank_shift : 0u;
    const uint32_t rank = crank - sub * ranks, first_peer = sub * ranks;
    const int nt = G > 1 ? (static_cast<int>(cluster_id) - (gi > 0 ? p.w[gi - 1].cluster_end : 0)) * p.w[gi].tiles + static_cast<int>(sub)
                         : static_cast<int>(cluster_id);
    const uint8_t *const sfw = p.w[gi].sfw, *const sfx = p.w[gi].sfx;
    const int N = p.w[gi].N, K = p.w[gi].K;
    const int w_rows = box_rows(N, nt, 128);   // 0 behind a weight's last tile
    const BoxMap w_map = box_map(w_rows, 128);
    const CUtensorMap* tmap_w = w_map == kRestMap ? &maps.m_rest[gi] : &maps.m[gi];
    const CUtensorMap* tmap_x = &maps.x[gi];
    const uint32_t operand_bytes = static_cast<uint32_t>(w_rows + p.M) * kBKBytes;
    const int64_t sf_group_stride = p.w[gi].sf_group_stride;
    // reduce-scatter: token column c belongs to rank c / cols_per_rank
    const uint32_t m_cols = static_cast<uint32_t>(min(p.M, BT));
    const uint32_t cols_per_rank = (m_cols + ranks - 1) / ranks;
    const uint32_t my_first = rank * cols_per_rank;
    const uint32_t my_cols = my_first < m_cols ? min(cols_per_rank, m_cols - my_first) : 0u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < nstages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        mbar_init(tfull_bar, 1);
        mbar_init(recv_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // (ranks - 1) senders x my columns x 128 rows x 4 bytes; armed before any rank can send
        if (ranks > 1 && my_cols > 0) mbar_expect_tx(recv_bar, (ranks - 1) * my_cols * 512u);
    }
    // Two phases of the cluster barrier: the barriers of all CTAs exist and are armed (waited for before the first copy to another
    // CTA), and all copies have landed (waited for at the end).
    if (apart && ranks > 1) {
        __syncwarp();
        cluster_arrive();
    }
    const int k_tiles = (K + kBK - 1) / kBK;
    const int kt_begin = static_cast<int>(rank) * p.w[gi].k_tiles_per_rank;
    // never 0 (the launcher leaves no K range empty), but for a CTA of a weight's last cluster behind its last tile: that one streams nothing, takes part in the
    // barriers and stores nothing (its rows lie beyond N)
    const int kcount = w_map != kNoMap ? max(0, min(k_tiles, kt_begin + p.w[gi].k_tiles_per_rank) - kt_begin) : 0;

    // Producer state (warp 0).  The first ring-full of copies is issued BEFORE the CTA-wide barrier of the prologue:
    // the copies need the mbarriers (initialised by this warp's thread 0 just above) but neither TMEM nor the other
    // warps, so the first HBM round trip overlaps the TMEM allocation and the barrier instead of following them.
    int p_stage = 0, p_next = 0;
    uint32_t p_phase = 0;
    bool p_ok = true;
    // copies of one stage, by the elected lane: the weight tile and its scales, the token tile and its scales
    auto copy_stage = [&](int stage, int kt, bool weights, bool tokens) {
        const uint32_t sf_bytes = 512u * min(4, (K - kt * kBK + 63) / 64);
        const uint32_t sbase = base + stage * C::kStageBytes;
        if (weights) {
            mbar_expect_tx(full_bar(stage), operand_bytes + 2 * sf_bytes);
            tma_load_2d(sbase, tmap_w, kt * kBKBytes, nt * 128, full_bar(stage));
        }
        if (tokens) tma_load_2d(sbase + C::kWBytes, tmap_x, kt * kBKBytes, 0, full_bar(stage));
        if (weights)
            bulk_load_1d(sbase + C::kWBytes + C::kXBytes, sfw + static_cast<int64_t>(nt) * sf_group_stride + static_cast<int64_t>(kt) * 2048,
                         sf_bytes, full_bar(stage));
        if (tokens)
            bulk_load_1d(sbase + C::kWBytes + C::kXBytes + C::kSfBytes, sfx + static_cast<int64_t>(kt) * 2048, sf_bytes, full_bar(stage));
    };
    auto produce = [&](int end) {
        const bool issuer = elect_one();
        for (; p_ok && p_next < end; ++p_next) {
            const int kt = kt_begin + p_next;
            if (!(p_ok = mbar_wait_warp(empty_bar(p_stage), p_phase ^ 1u, abort_flag, (7u << 24) | kt))) break;
            if (issuer) copy_stage(p_stage, kt, true, true);
            __syncwarp();
            if (++p_stage == nstages) {
                p_stage = 0;
                p_phase ^= 1u;
            }
        }
    };
    if (warp == 0) {
        __syncwarp();   // thread 0's barrier initialisation above, before any lane of this warp uses the barriers
        if (w_map != kNoMap && elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(tmap_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(tmap_x) : "memory");
        }
        // First ring-full.  The weights do not depend on whatever ran before this kernel on the stream, the token tile
        // and its scales (the quantizer's output) do: with a programmatic dependent launch up to kAhead stages' prepared weights go out
        // at once, the rest after griddep_wait().
        const int first = min(kcount, nstages);
        const bool issuer = elect_one();
        const int ahead = !p.weights_ready ? 0 : G > 1 ? first : min(first, kAhead);   // raw weight pointers may be the previous kernel's output too
        if (issuer)
            for (int i = 0; i < ahead; ++i) copy_stage(i, kt_begin + i, true, false);
        griddep_wait();
        if (issuer) {
            if (G > 1) {
                for (int i = 0; i < first; ++i) copy_stage(i, kt_begin + i, !p.weights_ready, true);
            } else {
                for (int i = 0; i < ahead; ++i) copy_stage(i, kt_begin + i, false, true);
                for (int i = ahead; i < first; ++i) copy_stage(i, kt_begin + i, true, true);
            }
        }
        __syncwarp();
        p_next = first;
        p_stage = first == nstages ? 0 : first;
        p_phase = first == nstages ? 1u : 0u;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t*>(tmem_slot))),
                     "r"(C::kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (warp >= 2) griddep_wait();   // the epilogue reads alpha (and writes out): only once the previous kernel is done

    if (warp == 0) {
        // ------------------------------------------------------------------ producer, stages after the first ring-full
        produce(kcount);
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const bool issuer = elect_one();
        constexpr uint32_t idesc = instr_desc<BT>();
        int stage = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int i = 0; i < kcount; ++i) {
            if (!(ok = mbar_wait_warp(full_bar(stage), phase, abort_flag, (8u << 24) | i))) break;
            tc_fence_after();
            const int kb_count = min(4, (K - (kt_begin + i) * kBK + 63) / 64);
            const uint32_t sbase = base + stage * C::kStageBytes;
            const uint32_t w_lo = ((sbase & 0x3ffffu) >> 4) | (1u << 16);
            const uint32_t x_lo = w_lo + (C::kWBytes >> 4);
            const uint32_t sfw_lo = ((sbase + C::kWBytes + C::kXBytes) & 0x3ffffu) >> 4;
            const uint32_t sfx_lo = sfw_lo + (C::kSfBytes >> 4);
            const uint32_t sfw_t = tmem_base + C::kSfCol + (i & 1) * 32;
            const uint32_t sfx_t = sfw_t + 16;
            if (issuer) {
                for (int kb = 0; kb < kb_count; ++kb) {
                    tc_cp_lohi(sfw_t + 4 * kb, sfw_lo + 32 * kb);
                    tc_cp_lohi(sfx_t + 4 * kb, sfx_lo + 32 * kb);
                }
                for (int kb = 0; kb < kb_count; ++kb)
                    tc_mma_lohi(tmem_base, w_lo + 2 * kb, x_lo + 2 * kb, idesc, sfw_t + 4 * kb, sfx_t + 4 * kb,
                                (i > 0 || kb > 0) ? 1u : 0u);
                tc_commit(empty_bar(stage));
            }
            __syncwarp();
            if (++stage == nstages) {
                stage = 0;
                phase ^= 1u;
            }
        }
        if (ok && issuer) tc_commit(tfull_bar);
        __syncwarp();
    }

    // ---------------------------------------------------------------------- epilogue
    // Thread (sub-partition sp, lane) of warps 2..5 owns weight row nt*128 + 32*sp + lane; TMEM column m of its
    // lane is the partial sum for token m.  Columns are handled 16 at a time to keep the register count low.
    const int sp = warp & 3;
    const int n_local = sp * 32 + lane;
    const int n = nt * 128 + n_local;
    bool have = false;
    if (warp >= 2) {
        bool ok = mbar_wait(tfull_bar, 0, abort_flag, (9u << 24) | nt);
        have = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        if (have) tc_fence_after();
    }
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(sp * 32) << 16);
    if (ranks == 1) {
        if (warp >= 2 && have) {
            const float alpha = load_alpha(p.w[gi].alpha, p.w[gi].alpha_x);
            __nv_bfloat16* const out = p.w[gi].out;
#pragma unroll 1
            for (int c = 0; c < BT / 16 && c * 16 < p.M; ++c) {
                uint32_t v[16];
                tc_ld_32x32b_x16(t_lane + c * 16, v);
                tc_ld_wait();
                if (n < N) {
#pragma unroll
                    for (int e = 0; e < 16; ++e)
                        if (c * 16 + e < p.M)
                            out[static_cast<int64_t>(c * 16 + e) * N + n] =
                                __float2bfloat16_rn(__fmul_rn(__uint_as_float(v[e]), alpha));
                }
            }
        }
    } else {
        // The ring is idle once the accumulator is complete (all copies landed and were consumed) and takes this rank's partial tile:
        // `part` [token column][128 rows] fp32.  `recv` [sending rank][owned column][128 rows] holds the other ranks' partials of the
        // columns that this one owns.
        //
        // With room for `recv` behind the barriers (`apart`) a rank sends as soon as it is done, whether or not the owner
        // still multiplies, and the cluster meets once, at the end.  us, with `recv` in the ring, behind a cluster barrier and with another
        // one after the exchange / this, prepared: 16 x 4096 x 4096 5.26 / 4.75, 1 x 4096 x 4096 5.08 / 4.56, 16 x 8192 x 8192 9.96 / 9.46,
        // raw 6.26 / 6.00, 5.87 / 5.73, 10.39 / 10.39, behind the quantizer 7.57 / 7.25, 6.65 / 6.15, 11.65 / 11.00.  (Partials stored straight
        // into the owner's shared memory, 4 bytes per lane, instead of bulk copies: 4 x 1024 x 8192 4.64 for 4.42, 48 x 7168 x 7168 10.64 for 9.92.)
        //
        // CTAs that share an SM hide one another's waits, and their rings have no stage to spare: where the room would cost one (see
        // launch_skinny_list) `recv` stays in the ring, as it does in launches of many products, three or four CTAs on an SM (the seven
        // matrices of a layer of hidden 5120, FFN 13824, 16 tokens, with their quantization: 34.5 us, 35.1 apart; 32 tokens 36.2 and 43.9).
        float* part = reinterpret_cast<float*>(aligned);
        const float* const recv = apart ? reinterpret_cast<const float*>(reinterpret_cast<uint8_t*>(bars) + kBarrierBytes) : part + BT * 128;
        if (warp >= 2 && have) {
#pragma unroll 1
            for (int c = 0; c < BT / 16 && c * 16 < p.M; ++c) {
                uint32_t v[16];
                tc_ld_32x32b_x16(t_lane + c * 16, v);
                tc_ld_wait();
#pragma unroll
                for (int e = 0; e < 16; ++e)
                    if (c * 16 + e < p.M) part[(c * 16 + e) * 128 + n_local] = __uint_as_float(v[e]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the bulk copies below read `part`
        }
        if (apart) {
            if (warp >= 2) {
                cluster_wait();
                asm volatile("bar.sync 2, 128;" ::: "memory");   // the four warps' rows are staged
            }
        } else {
            __syncwarp();
            cluster_sync_all();   // every rank has left its main loop: the `recv` areas may be written
        }
        if (warp == 2 && have && elect_one()) {
            for (uint32_t i = 1; i < ranks; ++i) {   // this rank's successor first
                const uint32_t o = rank + i < ranks ? rank + i : rank + i - ranks, first = o * cols_per_rank;
                if (first >= m_cols) continue;
                const uint32_t cols = min(cols_per_rank, m_cols - first);
                bulk_copy_to_cta(map_to_cta(smem_u32(recv + (rank * cols_per_rank) * 128), first_peer + o),
                                 smem_u32(part + first * 128), cols * 512u, map_to_cta(recv_bar, first_peer + o));
            }
        }
        __syncwarp();
        if (warp >= 2 && have && my_cols > 0) {
            const float alpha = load_alpha(p.w[gi].alpha, p.w[gi].alpha_x);
            bool ok = mbar_wait(recv_bar, 0, abort_flag, (10u << 24) | nt);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (apart) cluster_arrive();
            if (ok && n < N) {
                // this rank's own partial sits in `recv` terms at part[my_first ..]; eight columns at a time so that
                // the shared-memory loads of one rank's partials are in flight together
                const float* own = part + my_first * 128 + n_local;
                __nv_bfloat16* dst = p.w[gi].out + static_cast<int64_t>(my_first) * N + n;
                for (uint32_t c0 = 0; c0 < my_cols; c0 += 8) {
                    float acc[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc[j] = 0.0f;
                    for (uint32_t r = 0; r < ranks; ++r) {
                        const float* src = (r == rank) ? own : recv + (r * cols_per_rank) * 128 + n_local;
                        float v[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) v[j] = (c0 + j < my_cols) ? src[(c0 + j) * 128] : 0.0f;
#pragma unroll
                        for (int j = 0; j < 8; ++j) acc[j] = r == 0 ? v[j] : __fadd_rn(acc[j], v[j]);
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c0 + j < my_cols)
                            dst[static_cast<int64_t>(c0 + j) * N] = __float2bfloat16_rn(__fmul_rn(acc[j], alpha));
                }
            }
        } else if (apart && warp >= 2) {
            cluster_arrive();
        }
        __syncwarp();
        if (apart) {
            if (warp < 2) {   // the others have done this around the exchange
                cluster_wait();
                cluster_arrive();
            }
        } else {
            cluster_sync_all();   // no rank may leave while another still copies out of its `part`
        }
    }

    // ---------------------------------------------------------------------- teardown
    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::kTmemCols) : "memory");
    }
    if (apart && ranks > 1) {   // no rank may leave while another still copies out of its `part` or into its `recv`
        __syncwarp();
        cluster_wait();
    }
}

// Clusters of `ranks` CTAs that are resident at once with `per_sm` CTAs on an SM (cudaOccupancyMaxActiveClusters on a B200; a
// cluster lives in one GPC, so large ones leave SMs over: 15 clusters of eight at one CTA per SM, not 18).
static int resident_clusters(int ranks, int per_sm, int sms) {
    static const int kOn148[4][8] = {{148, 74, 45, 33, 26, 22, 15, 15},
                                     {296, 148, 93, 71, 56, 45, 37, 33},
                                     {444, 222, 142, 104, 82, 71, 56, 48},
                                     {592, 296, 187, 142, 112, 93, 78, 71}};
    return kOn148[per_sm - 1][ranks - 1] * sms / 148;
}

// K ranges per weight tile: the largest power of two that keeps every CTA of the grid resident at once (one per
// SM), with at least two K stages each and at most 8 (the portable cluster size); measured (us):
// - a K of few stages is not cut where the tiles are many already (4 x 8512 x 1536, 67 tiles of 6 stages: one range 4.9, two 5.5);
// - with small token tiles two CTAs fit on an SM, and where the K range is already cut, cutting it once more is faster
//   (16 x 8192 x 8192: 12.2 -> 11.4);
// - one range becomes two where the tiles leave a third of the SMs without one, too few streams for HBM (16 x 9728 x 12288, 76
//   tiles, 18.7 -> 15.8; at 92 tiles 2 to 9 % are left, at 112 tiles and K 8192 two are 5 % slower), and where a very long K
//   would leave the last of up to 1.4 tiles per SM alone (16 x 23040 x 12288 30.5 -> 28.6; K 8192: no gain);
// - cluster sizes that are not a power of two are slower (6144 x 4096: 3 ranges 11.9, 2 ranges 8.0).
static int choose_ranks(int n_tiles, int k_tiles, int sms, int forced, int bt) {
    int r = 1;
    if (forced > 0) {
        r = forced;
    } else {
        const bool few = k_tiles <= 8 && n_tiles >= 40;
        // 128 tokens need a ring that leaves room for one CTA per SM: there the GPCs' room for clusters counts (119 x 2164 x 8448,
        // 17 tiles: 18.8 us with eight ranges, whose 16th cluster waits for the first to finish, 10.6 with four)
        while (!few && r < 8 && n_tiles * (2 * r) <= sms && (bt <= 64 || n_tiles <= resident_clusters(2 * r, 1, sms))) r *= 2;
        if (bt <= 32 && r >= 2 && r < 8 && n_tiles * (2 * r) <= 2 * sms - 40 && k_tiles / (2 * r) >= 4) r *= 2;
        const bool thin = n_tiles * 8 <= sms * 5, tail = k_tiles >= 40 && n_tiles > sms && n_tiles * 10 <= sms * 14;
        if (bt <= 32 && r == 1 && k_tiles > 16 && (thin || tail)) r = 2;
    }
    if (r > 8) r = 8;
    while (r > 1 && r > k_tiles / 2) --r;
    return r;
}

// One weight of a grouped launch, as the host sees it.
struct SkinnyItem {
    const uint8_t* x;         // codes [M, K/2]
    const uint8_t* sfx;       // tiled scales
    const float* alpha_x;     // or NULL
    const uint8_t* w;         // codes [N, K/2]
    const uint8_t* sfw;       // tiled scales
    const float* alpha;
    __nv_bfloat16* out;       // [M, N]
    int64_t N, K;
    const WeightHandle* wh;   // prepared tensor maps, or NULL
};

// Ring depth: the deepest ring with which the whole grid is resident at once (as many CTAs per SM as that takes, at
// most what the TMEM columns allow), since a CTA that has to wait for a free SM starts its weight stream late.
template <int BT>
static int choose_stages(int clusters, int ranks, int sms, int recv_bytes, int& per_sm) {
    using C = SkinnyCfg<BT>;
    constexpr int kMaxPerSm = kTmemCols / C::kTmemCols;
    per_sm = 1;
    while (per_sm < kMaxPerSm && clusters > resident_clusters(ranks, per_sm, sms)) ++per_sm;
    // an SM has 233472 bytes of shared memory, of which 1 KiB per resident CTA is reserved; a CTA asks for its ring with
    // alignment slack, its barriers and the area of the other ranks' partials
    int stages = (233472 / per_sm - 1024 - kSlack - kBarrierBytes - recv_bytes) / C::kStageBytes;
    if (stages > C::kMaxStages) stages = C::kMaxStages;
    // with CTAs sharing an SM a fifth stage, which would still fit, measured slower than four (Llama-3-8B-shaped decode
    // chain of 32 layers at 1 / 16 tokens: 1.30 / 1.48 ms against 1.25 / 1.43; 16 x 28672 x 8192: 23.3 against 23.0 us)
    if (per_sm >= 2 && stages > 4) stages = 4;
    // a cluster's CTAs need room at the same time, which they find sooner beside the launch before them with six stages than with
    // eight (30 x 9000 x 5120, raw / prepared / behind the quantizer: 9.36 / 8.82 / 11.75 -> 9.10 / 8.40 / 10.35; 16 x 9216 x 4096 8.16 / 7.49 /
    // 8.96 -> 7.95 / 7.13 / 8.62); single CTAs gain 1-4 % with raw weights and lose 1-8 % behind the quantizer
    if (ranks > 1 && stages > 6) stages = 6;
    if (stages < 2) stages = 2;
    return stages;
}

// K ranges of products of different K, in clusters of four: each product's ranges by its own K, so that the longest tiles end
// with the others.  The ranges are the finest for which the CTAs still fit the GPU at once, 13 for 4 SMs: a second wave pays
// the kernel's whole latency again.  Where the shortest K is cut too, its many short ranges must leave room, 5 for 2 SMs (4
// tokens, hidden 1280, FFN 9984, K of 5 and 39 stages: 13.7 with 432 CTAs, 11.6 with 236).  A layer's seven matrices with their
// quantization, us, against the same number of ranges for all: hidden 4096, K / V 1024, FFN 14336, 1 token 26.2 -> 24.1, 16
// tokens 30.4 -> 28.1; 2048 / 512 / 8192, 4 tokens 17.6 -> 12.4; 3072 / 3072 / 8192, 3 tokens 24.5 -> 15.1; clusters of eight are
// no faster.
template <int G>
static int plan_mixed(SkinnyParams<G>& p, int n, int sms) {
    constexpr int kCluster = 4;
    for (int target = 2;; ++target) {
        int64_t ctas = 0;
        bool longer = false;   // a larger target would change something
        bool all_cut = true;
        for (int i = 0; i < n; ++i) {
            const int k = (p.w[i].K + kBK - 1) / kBK;
            int r = 1;
            while (r < kCluster && (k + r - 1) / r > target) r *= 2;
            while (r > 1 && (r - 1) * ((k + r - 1) / r) >= k) r /= 2;   // no empty range
            p.w[i].ranks = r;
            longer = longer || r > 1;
            all_cut = all_cut && r > 1;
            ctas += static_cast<int64_t>((p.w[i].N + 127) / 128) * r;
        }
        if (!longer || ctas * 4 <= static_cast<int64_t>(sms) * (all_cut ? 10 : 13)) return kCluster;
    }
}

// Items are in order of descending K (the longest tiles start first).
template <int BT, int G>
static int launch_skinny_list(int M, const SkinnyItem* items, int n_items, int forced_ranks, cudaStream_t stream) {
    using C = SkinnyCfg<BT>;
    SkinnyMaps<G> maps;
    SkinnyParams<G> p;
    int n_tiles = 0, st = NVFP4_OK;
    p.weights_ready = 1;
    for (int i = 0; i < n_items && st == NVFP4_OK; ++i) {
        const SkinnyItem& it = items[i];
        if (!it.wh) p.weights_ready = 0;
        if (it.wh) {
            maps.m[i] = it.wh->rows[WeightHandle::index(128)];
            maps.m_rest[i] = it.wh->rest[WeightHandle::index(128)];
        } else {
            st = make_operand_maps(&maps.m[i], &maps.m_rest[i], it.w, it.N, it.K / 2, 128);
        }
        if (i > 0 && it.x == items[i - 1].x && it.K == items[i - 1].K) maps.x[i] = maps.x[i - 1];
        else if (st == NVFP4_OK) st = make_operand_map(&maps.x[i], it.x, M, it.K / 2, M);
        n_tiles += static_cast<int>((it.N + 127) / 128);
        p.w[i].sfw = it.sfw;
        p.w[i].sfx = it.sfx;
        p.w[i].alpha = it.alpha;
        p.w[i].alpha_x = it.alpha_x;
        p.w[i].out = it.out;
        p.w[i].N = static_cast<int>(it.N);
        p.w[i].K = static_cast<int>(it.K);
        p.w[i].sf_group_stride = round_up_i64(it.K / 16, 4) * 128;
    }
    if (st != NVFP4_OK) return st;
    const DeviceInfo di = device_info();
    const int sms = di.sms;
    const int longest = (p.w[0].K + kBK - 1) / kBK, shortest = (p.w[n_items - 1].K + kBK - 1) / kBK;
    const bool mixed = longest != shortest;
    auto stages_of = [&](int i, int r) { return ((p.w[i].K + kBK - 1) / kBK + r - 1) / r; };
    // no empty K range: with every rank holding ceil(k / ranks) stages the last one must get some
    auto fits = [&](int i, int r) { return (r - 1) * stages_of(i, r) < (p.w[i].K + kBK - 1) / kBK; };
    int cluster;
    if (mixed && forced_ranks == 0) {
        cluster = plan_mixed(p, n_items, sms);
    } else {
        // one number of ranges for all: the largest that leaves none of any item empty.  (A smaller one need not fit where a larger
        // one did, 24 stages fit 6 ranges and 25 do not, so every item is asked again for each.)
        cluster = choose_ranks(n_tiles, shortest, sms, forced_ranks, BT);
        auto all_fit = [&](int r) {
            for (int i = 0; i < n_items; ++i)
                if (!fits(i, r)) return false;
            return true;
        };
        while (cluster > 1 && !all_fit(cluster)) --cluster;
        for (int i = 0; i < n_items; ++i) p.w[i].ranks = cluster;
    }
    int clusters = 0, per_rank = 1, max_ranks = 1;
    for (int i = 0; i < n_items; ++i) {
        const int tiles = static_cast<int>((items[i].N + 127) / 128), per = cluster / p.w[i].ranks;
        p.w[i].tiles = per;
        p.w[i].rank_shift = 31;   // one tile per cluster: the first
        if (per > 1)
            for (p.w[i].rank_shift = 0; 1 << p.w[i].rank_shift < p.w[i].ranks;) ++p.w[i].rank_shift;
        clusters += (tiles + per - 1) / per;
        p.w[i].cluster_end = clusters;
        p.w[i].k_tiles_per_rank = stages_of(i, p.w[i].ranks);
        if (p.w[i].k_tiles_per_rank > per_rank) per_rank = p.w[i].k_tiles_per_rank;
        if (p.w[i].ranks > max_ranks) max_ranks = p.w[i].ranks;
    }
    p.M = M;
    p.n_weights = n_items;
    int per_sm = 1;
    // Stages with `recv` bytes for the other ranks' partials behind the ring; without, the ring holds them beside this rank's own (the
    // size of `part` and a rounding).
    auto stages_with = [&](int recv) {
        int st = choose_stages<BT>(clusters, cluster, sms, recv, per_sm);
        if (st > per_rank) st = per_rank < 2 ? 2 : per_rank;
        while (max_ranks > 1 && (recv > 0 ? BT : 2 * BT + 8) * 512 > st * C::kStageBytes) ++st;
        return st;
    };
    int recv_bytes = 0;
    p.stages = stages_with(0);
    if (G == 1 && max_ranks > 1) {
        // ranks x owned columns x 128 rows behind the ring, unless CTAs that share an SM would lose a stage by it (us, in the ring / behind
        // it, prepared, raw, behind the quantizer: 19 x 20672 x 10624 24.4 / 25.2, 24.6 / 25.6, 26.0 / 27.1, 31 x 4288 x 14016 10.4 / 10.8, 10.9 /
        // 11.6, 13.4 / 14.0; over 115 random launches the ring is 2.0, 2.7 and 3.1 % ahead.  Over 4645 others it is 4.8, 2.7 and 3.4 % behind,
        // also where CTAs alone on their SM lose a stage, 965 of them: 1.9, 0.9 and 1.9 %.)
        const int columns = (M < BT ? M : BT) + max_ranks - 1, bytes = columns / max_ranks * max_ranks * 512, left = stages_with(bytes);
        if (per_sm < 2 || left >= p.stages) {
            p.stages = left;
            recv_bytes = bytes;
        }
    }
    p.apart = recv_bytes > 0;
    // Co-resident CTAs must never want more than the 512 TMEM columns of an SM between them (a CTA that waits in
    // tcgen05.alloc while its cluster peers wait for it is a deadlock).  Shared memory is what bounds co-residency, so
    // every CTA asks for at least the share of the SM's shared memory that matches its share of the TMEM columns
    // (1 KiB per CTA is reserved by the system): whatever mix of these kernels fits an SM then fits its TMEM too.
    constexpr int kMinSmem = 233472 / (kTmemCols / C::kTmemCols) - 1024;   // 128 columns: 57344 (4 CTAs), 256: 115712 (2)
    int smem = p.stages * C::kStageBytes + kSlack + kBarrierBytes + recv_bytes;
    if (smem < kMinSmem) smem = kMinSmem;
    static_assert(C::kMaxStages * C::kStageBytes + kSlack + kBarrierBytes <= kGemmDynSmemBytes, "ring does not fit");
    static_assert(2 * C::kStageBytes + kSlack + kBarrierBytes + (BT + 7) * 512 <= kGemmDynSmemBytes && BT * 512 <= 2 * C::kStageBytes, "partials do not fit");
    static bool attr_done[64] = {false};
    cudaError_t e = allow_full_smem(skinny_kernel<BT, G>, attr_done, di.device);
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * cluster, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    // programmatic dependent launch: this kernel may be scheduled while its predecessor on the stream is finishing
    // (it stops at griddep_wait() before touching anything the predecessor may have written)
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_dependent_launch ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, skinny_kernel<BT, G>, maps, p);
    return static_cast<int>(e);
}

template <int BT>
static int launch_skinny_group(int M, const SkinnyItem* items, int n_items, int forced_ranks, cudaStream_t stream) {
    if (n_items < 1 || n_items > kMaxGroup) return NVFP4_ERR_BAD_RANGE;
    return n_items == 1 ? launch_skinny_list<BT, 1>(M, items, 1, forced_ranks, stream)
                        : launch_skinny_list<BT, kMaxGroup>(M, items, n_items, forced_ranks, stream);
}

template <int BT>
static int launch_skinny(const GemmParams& g, int forced_ranks, cudaStream_t stream,
                         const WeightHandle* wh) {
    const SkinnyItem it = {g.a, g.sfa, g.alpha2, g.b, g.sfb, g.alpha, g.out, g.N, g.K, wh};
    return launch_skinny_group<BT>(g.M, &it, 1, forced_ranks, stream);
}

}  // namespace skinny

}  // namespace gemm
}  // namespace nvfp4
