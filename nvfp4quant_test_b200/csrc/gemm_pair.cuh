// CTA-pair kernels of the NVFP4 GEMM (cta_group::2, 256 x 128 / 256 x 192 / 256 x 256 output tiles).
#pragma once

#include "gemm_tile.cuh"

namespace nvfp4 {
namespace gemm {

// =============================================================================================
// Two-CTA variant (cta_group::2): a CTA pair owns a 256 x 256 output tile.  Each CTA loads its own
// 128 rows of A and HALF of the B tile (128 of the 256 weight rows); the pair's tensor cores read
// both halves, so B crosses L2 -> shared memory once per pair instead of once per CTA.  No
// multicast load is involved: every TMA copy has exactly one destination CTA.  The CTA with
// cluster rank 0 issues all MMAs; copies of both CTAs report to rank 0's "full" barrier
// (cp.async.bulk.tensor ... .cta_group::2), and tcgen05.commit signals the "empty" and
// "accumulator ready" barriers of both CTAs.
// =============================================================================================
namespace pair {

// Tile-width dependent constants of the pair kernel.  BN = 256: one accumulator (256 columns) per CTA.
// BN = 192 / 128: two accumulators (2 x BN columns), so the epilogue of one tile overlaps the MMAs of the next.
// BN = 128 (256 x 128 tiles) is for a few hundred tokens: twice the CTAs of the wider tiles on the weight stream,
// and each CTA still loads only half of the tile's weight rows.
template <int BN>
struct PairCfg {
    static constexpr int kAcc = (BN <= 192) ? 2 : 1;
    static constexpr int kABytes = 128 * kBKBytes;          // this CTA's 128 rows of A
    static constexpr int kBBytes = (BN / 2) * kBKBytes;     // this CTA's half of the B rows
    static constexpr int kSfaBytes = 2048;                  // scales of this CTA's A rows
    // 128-row scale groups that a B tile touches: a 128-wide one exactly one (with two loaded for it, us, before / after: 256 x 4096 x 14336
    // 15.08 / 14.71, 700 x 1500 x 14336 14.99 / 14.43, 300 x 1024 x 8192 9.86 / 9.54)
    static constexpr int kSfbGroups = BN == 128 ? 1 : 2;
    static constexpr int kSfbBytes = 2048 * kSfbGroups;
    static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
    // ring stages against staged output pieces per epilogue warp: as deep a ring as leaves one piece (256 x 192 tiles with 5
    // stages and two pieces: 5 % faster at K = 1024, 4 % slower at K = 8192)
    static constexpr int kStages = (BN == 128) ? 7 : (BN == 192) ? 6 : 5;
    static constexpr int kOutBufs = (BN == 256) ? 2 : 1;
    static constexpr int kEpilogueBytes = 4 * kOutBufs * kPieceBytes;
    static constexpr int kSmemBytes = kStages * kStageBytes + kEpilogueBytes + 256;
    static constexpr int kSfaCol = kAcc * BN;               // scale set 0; set 1 follows
    static constexpr int kSfbCol = kSfaCol + 16;
    static constexpr int kSfSetCols = 16 + 16 * kSfbGroups;
    static_assert(kSfaCol + 2 * kSfSetCols <= kTmemCols, "TMEM budget");
    static_assert(kStageBytes % 1024 == 0, "stage alignment for the 128-byte swizzle");
};

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
// every thread of the cluster arrives and waits in turn
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// tile load whose completion bytes are reported to a barrier that may live in the peer CTA
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(bar_cluster)
        : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"(static_cast<uint16_t>(3))
                 : "memory");
}
__device__ __forceinline__ void tc_cp_pair(uint32_t taddr, uint32_t lo) {
    asm volatile("{ .reg .b64 d; mov.b64 d, {%1, %2}; tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], d; }" ::"r"(taddr),
                 "r"(lo), "r"(kDescHiSf)
                 : "memory");
}
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc,
                                            uint32_t sfa_tmem, uint32_t sfb_tmem, uint32_t accumulate) {
    asm volatile(
        "{ .reg .pred p; .reg .b64 da, db; setp.ne.b32 p, %4, 0; mov.b64 da, {%1, %7}; mov.b64 db, {%2, %7};\n"
        "  tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], da, db, %3, [%5], [%6], p; }" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem), "r"(kDescHiSw128)
        : "memory");
}

// Operand maps and the work list of one launch over G products (G = 1: an ordinary GEMM).
template <int G>
struct PairParams {
    CUtensorMap a[G], b[G], sfa[G], sfb[G], out[G];
    GroupTable<G> g;
    int M;
    int raster_group;
    int weights_ready;   // see TileParams
};

template <int BN, int G>
__global__ void __launch_bounds__(kThreads, 1)
gemm_pair_kernel(const __grid_constant__ PairParams<G> p) {
    using C = PairCfg<BN>;
    extern __shared__ __align__(1024) uint8_t smem[];   // the 128-byte swizzle repeats every 1024 bytes
    // The kernel queued behind this one may be scheduled at once: ahead of its own wait it reads nothing but a
    // prepared (constant) weight, and that wait covers this kernel's completion.
    griddep_launch();
    uint8_t* const aligned = smem;
    const uint32_t base = smem_u32(aligned);
    uint64_t* bars = reinterpret_cast<uint64_t*>(aligned + C::kStages * C::kStageBytes + C::kEpilogueBytes);
    const uint32_t bar_base = smem_u32(bars);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (C::kStages + s); };
    auto tfull_bar = [&](int a) { return bar_base + 8u * (2 * C::kStages + a); };
    auto tempty_bar = [&](int a) { return bar_base + 8u * (2 * C::kStages + 2 + a); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 2 * C::kStages + 4);
    volatile uint32_t* abort_flag = tmem_slot + 1;

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();           // 0 = leader (issues the MMAs)
    const int pair_id = blockIdx.x >> 1;
    if (threadIdx.x == 0) trace_mark(1, 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full_bar(s), 1);    // leader's producer; bytes of both CTAs' copies land here
            mbar_init(empty_bar(s), 1);   // one tcgen05.commit
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 8);  // 4 epilogue warps of each CTA
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    // Two phases of the cluster barrier: the barriers of both CTAs exist (nothing is signalled across CTAs before), which is all that
    // the producers need; TMEM is allocated in both, which the other warps wait for as well while the first copies are on their way.
    cluster_arrive();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t*>(tmem_slot))),
                     "r"(kTmemCols)
                     : "memory");
        if (lane == 0) trace_mark(1, 1);
    }
    tc_fence_before();
    cluster_wait();
    if (threadIdx.x == 0) trace_mark(1, 9);
    cluster_arrive();
    if (warp != 0) cluster_wait();   // the producer warps wait at their end
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;   // meaningful in warps 1..5 only
    if (threadIdx.x == 0) trace_mark(1, 2);
    if (warp >= 2) griddep_wait();    // the epilogue reads alpha and writes the output: only after the previous kernel

    const int m_tiles = (p.M + 255) / 256;
    TileCursor<G> cur;
    cur.init(p.g, pair_id);
    // tile -> its item (cur.item), m tile and n tile
    auto locate = [&](int tile, int& mt, int& nt) {
        cur.seek(p.g, tile);
        const int n_tiles = (p.g.item[cur.item].N + BN - 1) / BN;
        tile_to_mn(tile - cur.first_tile, m_tiles, n_tiles, p.raster_group, mt, nt);
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ producer (both CTAs)
        {
            const bool issuer = elect_one();
            int mt = 0, nt = 0, k_tiles = 0;
            auto set_tile = [&](int tile) {
                locate(tile, mt, nt);
                k_tiles = (p.g.item[cur.item].K + kBK - 1) / kBK;
            };
            const uint32_t lead_full = map_to_cta(full_bar(0), 0);
            // weight half (B rows and their scales: independent of whatever ran before this kernel) and token half (A rows
            // and their scales) of a stage; the weight halves of the first ring-full are issued before griddep_wait(), if they are
            // prepared (raw: side by side with the tokens, see gemm_kernel)
            auto issue = [&](int st, int kt, bool weights, bool tokens) {
                const uint32_t bar = lead_full + 8u * st;
                const uint32_t sbase = base + st * C::kStageBytes;
                if (weights) {
                    if (rank == 0) mbar_expect_tx(full_bar(st), 2u * C::kStageBytes);
                    tma_load_2d_pair(sbase + C::kABytes, &p.b[cur.item], kt * kBKBytes, nt * BN + static_cast<int>(rank) * (BN / 2), bar);
                }
                if (tokens) tma_load_2d_pair(sbase, &p.a[cur.item], kt * kBKBytes, mt * 256 + static_cast<int>(rank) * 128, bar);
                if (weights) {
                    // scale tiles: x counts 8-byte elements (2048 B per K tile), y = 128-row group
#pragma unroll
                    for (int g = 0; g < C::kSfbGroups; ++g)
                        tma_load_2d_pair(sbase + C::kABytes + C::kBBytes + C::kSfaBytes + 2048 * g, &p.sfb[cur.item], kt * 256, (nt * BN) / 128 + g, bar);
                }
                if (tokens)
                    tma_load_2d_pair(sbase + C::kABytes + C::kBBytes, &p.sfa[cur.item], kt * 256, mt * 2 + static_cast<int>(rank), bar);
            };
            const bool any = cur.local < cur.total;
            if (any) set_tile(cur.local);
            if (issuer) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.a[cur.item]) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.b[cur.item]) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.sfa[cur.item]) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(&p.sfb[cur.item]) : "memory");
            }
            const int early = any ? min(k_tiles, C::kStages) : 0;   // stages requested without a wait
            if (issuer && p.weights_ready)
                for (int i = 0; i < early; ++i) issue(i, i, true, false);
            griddep_wait();
            if (issuer)
                for (int i = 0; i < early; ++i) issue(i, i, !p.weights_ready, true);
            __syncwarp();
            int stage = early == C::kStages ? 0 : early;
            uint32_t phase = early == C::kStages ? 1u : 0u;
            bool ok = true;
            for (int tile = cur.local; ok && tile < cur.total; tile += cur.workers) {
                int kt = early;
                if (tile != cur.local) {
                    set_tile(tile);
                    kt = 0;
                }
                for (; kt < k_tiles; ++kt) {
                    if (!(ok = mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag, (1u << 24) | kt))) break;
                    if (issuer) issue(stage, kt, true, true);
                    __syncwarp();
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer (leader only)
        if (rank == 0) {
            const bool issuer = elect_one();
            constexpr uint32_t idesc = (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) |
                                       (static_cast<uint32_t>(256 >> 4) << 24);
            int stage = 0;
            uint32_t phase = 0, acc_phase = 0;
            int acc = 0;
            bool ok = true;
            for (int tile = cur.local; ok && tile < cur.total; tile += cur.workers) {
                if (!(ok = mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag, (2u << 24) | 0xffff))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                // a 192-wide tile starts 0 or 64 rows into its first scale group: 64 rows = 2 TMEM columns
                int mt_unused, nt_of_tile;
                locate(tile, mt_unused, nt_of_tile);
                const int K = p.g.item[cur.item].K;
                const int k_tiles = (K + kBK - 1) / kBK;
                const uint32_t sfb_shift = (nt_of_tile * BN % 128) / 32;
                for (int kt = 0; kt < k_tiles; ++kt) {
                    if (!(ok = mbar_wait_warp(full_bar(stage), phase, abort_flag, (2u << 24) | kt))) break;
                    tc_fence_after();
                    const int kb_count = min(4, (K - kt * kBK + 63) / 64);
                    const uint32_t sbase = base + stage * C::kStageBytes;
                    const uint32_t a_lo = ((sbase & 0x3ffffu) >> 4) | (1u << 16);
                    const uint32_t b_lo = a_lo + (C::kABytes >> 4);
                    const uint32_t sfa_lo = ((sbase + C::kABytes + C::kBBytes) & 0x3ffffu) >> 4;
                    const uint32_t sfb_lo = sfa_lo + (C::kSfaBytes >> 4);
                    const uint32_t set = (kt & 1) * C::kSfSetCols;
                    const uint32_t sfa_t = tmem_base + C::kSfaCol + set;
                    const uint32_t sfb_t = tmem_base + C::kSfbCol + set;
                    const uint32_t first = kt > 0 ? 1u : 0u;
                    if (!issuer) {
                        // nothing to issue on this lane
                    } else if (kb_count == 4) {
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb) {
                            tc_cp_pair(sfa_t + 4 * kb, sfa_lo + 32 * kb);
#pragma unroll
                            for (int g = 0; g < C::kSfbGroups; ++g)
                                tc_cp_pair(sfb_t + 4 * C::kSfbGroups * kb + 4 * g, sfb_lo + 128 * g + 32 * kb);
                        }
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb)
                            tc_mma_pair(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa_t + 4 * kb, sfb_t + 4 * C::kSfbGroups * kb + sfb_shift,
                                        kb == 0 ? first : 1u);
                    } else {
                        for (int kb = 0; kb < kb_count; ++kb) {
                            tc_cp_pair(sfa_t + 4 * kb, sfa_lo + 32 * kb);
#pragma unroll
                            for (int g = 0; g < C::kSfbGroups; ++g)
                                tc_cp_pair(sfb_t + 4 * C::kSfbGroups * kb + 4 * g, sfb_lo + 128 * g + 32 * kb);
                        }
                        for (int kb = 0; kb < kb_count; ++kb)
                            tc_mma_pair(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa_t + 4 * kb, sfb_t + 4 * C::kSfbGroups * kb + sfb_shift,
                                        kb == 0 ? first : 1u);
                    }
                    if (issuer) tc_commit_pair(empty_bar(stage));   // frees this slot in both CTAs
                    __syncwarp();
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                if (issuer) tc_commit_pair(tfull_bar(acc));         // accumulators of both CTAs are complete
                __syncwarp();
                if (++acc == C::kAcc) {
                    acc = 0;
                    acc_phase ^= 1u;
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (both CTAs)
        const int sp = warp & 3;
        // staged output, behind the ring
        uint8_t* epilogue_stage = aligned + C::kStages * C::kStageBytes + sp * (C::kEpilogueBytes / 4);
        int out_turn = 0;
        int alpha_item = -1;
        float alpha = 0.0f;
        uint32_t acc_phase = 0;
        int acc = 0;
        bool ok = true;
        for (int tile = cur.local; ok && tile < cur.total; tile += cur.workers) {
            int mt, nt;
            locate(tile, mt, nt);
            const GemmItem& it = p.g.item[cur.item];
            const int N = it.N;
            if (cur.item != alpha_item) {
                alpha_item = cur.item;
                alpha = load_alpha(it.alpha, it.alpha2);
            }
            ok = mbar_wait(tfull_bar(acc), acc_phase, abort_flag, (3u << 24) | (tile & 0xffff));
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            tc_fence_after();
            store_accumulator<BN, C::kOutBufs>(tmem_base + (static_cast<uint32_t>(sp * 32) << 16) + acc * BN, it.out, &p.out[cur.item], p.M, N,
                                  mt * 256 + static_cast<int>(rank) * 128 + sp * 32, nt * BN, alpha, epilogue_stage, out_turn, [&] {
                                      tc_fence_before();
                                      __syncwarp();
                                      if (lane == 0) mbar_arrive_cluster(map_to_cta(tempty_bar(acc), 0));
                                  });
            if (++acc == C::kAcc) {
                acc = 0;
                acc_phase ^= 1u;
            }
        }
    }

    if (warp == 0) {
        __syncwarp();
        cluster_wait();
    }
    // the staged output has been read; the writes themselves are complete when the grid is
    if (warp >= 2 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
    if (lane == 0) trace_mark(1, warp == 0 ? 3 : warp == 1 ? 4 : 5);
    // ---------------------------------------------------------------------- teardown
    if (*abort_flag) {
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) trace_mark(1, 6);
    cluster_sync_all();   // neither CTA leaves while its partner may still signal or read it
    if (threadIdx.x == 0) trace_mark(1, 7);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
        if (lane == 0) trace_mark(1, 8);
    }
    // cta_group::2 allocation state spans both SMs of the pair.  If one CTA left right after its own dealloc, another
    // kernel's CTA could start on that SM and allocate while the partner's dealloc for the pair is still to come;
    // with several GEMM kernels running at once that left a later tcgen05.alloc waiting for ever.  Both CTAs
    // therefore stay until both deallocations have been issued.
    cluster_sync_all();
}

// Scale buffer as a 2-D array of 8-byte words: row = 128-row group, 2048 B (one K tile) per box.
static int make_scale_map(CUtensorMap* map, const void* ptr, int64_t groups, int64_t group_stride_bytes) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return NVFP4_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(group_stride_bytes / 8), static_cast<cuuint64_t>(groups)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(group_stride_bytes)};
    cuuint32_t box[2] = {256, 1};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? NVFP4_OK : NVFP4_ERR_UNSUPPORTED;
}

// One launch over the `n` products of `list` (1 <= n <= G), items of equal K next to one another, longest K first.
template <int BN, int G>
static int launch_pair_list(const GemmParams* list, const WeightHandle* const* wh, int n, cudaStream_t stream) {
    using C = PairCfg<BN>;
    static_assert(C::kSmemBytes <= kGemmDynSmemBytes, "ring does not fit");
    PairParams<G> q;
    q.M = list[0].M;
    const int m_tiles = (q.M + 255) / 256;
    q.raster_group = band_rows(list[0].raster_group, m_tiles);
    q.weights_ready = 1;
    for (int i = 0; i < n; ++i) {
        const GemmParams& p = list[i];
        int st = make_operand_map(&q.a[i], p.a, p.M, p.K / 2, 128);
        if (st == NVFP4_OK) st = make_scale_map(&q.sfa[i], p.sfa, p.sfa_groups, p.sf_group_stride);
        if (st == NVFP4_OK) st = make_output_map(&q.out[i], p.out, p.M, p.N);
        if (wh[i]) {
            q.b[i] = wh[i]->rows[WeightHandle::index(BN / 2)];
            q.sfb[i] = wh[i]->scales;
        } else {
            q.weights_ready = 0;
            if (st == NVFP4_OK) st = make_operand_map(&q.b[i], p.b, p.N, p.K / 2, BN / 2);
            if (st == NVFP4_OK) st = make_scale_map(&q.sfb[i], p.sfb, p.sfb_groups, p.sf_group_stride);
        }
        if (st != NVFP4_OK) return st;
    }
    const DeviceInfo di = device_info();
    const int pairs = fill_group_table<G>(q.g, list, n, m_tiles, BN, di.sms / 2);
    if (pairs == 0) return NVFP4_ERR_TOO_LARGE;
    static bool attr_done[64] = {false};
    cudaError_t e = allow_full_smem(gemm_pair_kernel<BN, G>, attr_done, di.device);
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * pairs, 1, 1);
    cfg.blockDim = dim3(kThreads, 1, 1);
    cfg.dynamicSmemBytes = kGemmDynSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // may start while its predecessor finishes
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = g_dependent_launch ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, gemm_pair_kernel<BN, G>, q);
    return static_cast<int>(e);
}

template <int BN>
static int launch_pair(const GemmParams& p, cudaStream_t stream, const WeightHandle* wh) {
    return launch_pair_list<BN, 1>(&p, &wh, 1, stream);
}

}  // namespace pair

}  // namespace gemm
}  // namespace nvfp4
