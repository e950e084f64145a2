// Tile kernels of the NVFP4 GEMM: one persistent CTA per SM, 128 x 64 / 128 x 128 / 128 x 256 output tiles.
#pragma once

#include "tc_ptx.cuh"
#include "tile_index.cuh"

namespace nvfp4 {
namespace gemm {

// Epilogue staging, per epilogue warp: a piece of 32 rows x 64 columns of bf16 for a TMA store, or half of one (with a word
// of padding per row) that is turned for rows TMA cannot write.
constexpr int kPieceBytes = 4096;
constexpr int kTurnPitch = 17;   // 32-bit words per row: conflict-free both ways
constexpr int kTurnBytes = 32 * kTurnPitch * 4;

template <int BN>
struct Cfg {
    static constexpr int kNG = (BN + 127) / 128;            // 128-row scale groups a B tile touches (a 64-row tile: half of one)
    static constexpr int kAcc = (BN <= 128) ? 2 : 1;        // accumulator buffers in TMEM
    static constexpr int kABytes = kBM * kBKBytes;          // 16 KiB
    static constexpr int kBBytes = BN * kBKBytes;
    static constexpr int kSfaBytes = 2048;                  // 128 rows x 16 blocks
    static constexpr int kSfbBytes = 2048 * kNG;
    static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
    // ring depth: as many stages as fit in shared memory (the bytes in flight per SM are what keeps HBM busy when
    // few CTAs stream a long K)
    static constexpr int kStages = (BN == 64) ? 7 : (BN == 128) ? 6 : 4;
    // no staged output pieces: the ring is worth more than they are (with 5 stages and two pieces 128 x 128 tiles gain 7 % at
    // K = 1088 and lose 5 % at K = 2880), so rows go out of the registers
    static constexpr int kEpilogueBytes = 4 * kTurnBytes;
    static constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*align*/ + 256 /*barriers*/ + kEpilogueBytes;

    // scale factors sit behind the accumulators, in two sets used by alternate K tiles so that the
    // copies for the next K tile do not have to wait for the MMAs still reading the current set
    static constexpr int kSfSetCols = 16 + 16 * kNG;
    static constexpr int kSfaCol = kAcc * BN;               // TMEM column of the A scales (set 0)
    static constexpr int kSfbCol = kSfaCol + 16;            // TMEM column of the B scales (set 0)
    static_assert(kSfaCol + 2 * kSfSetCols <= kTmemCols, "TMEM budget");
};

// One product, as the entry points see it.
struct GemmParams {
    const uint8_t* a;
    const uint8_t* b;
    const uint8_t* sfa;
    const uint8_t* sfb;
    const float* alpha;
    const float* alpha2;      // optional second factor: the output scale is alpha[0] * alpha2[0] (one fp32 multiplication)
    __nv_bfloat16* out;
    int M, N, K;
    int64_t sf_group_stride;  // bytes between consecutive 128-row scale groups = round_up(K/16, 4) * 128
    int sfa_groups, sfb_groups;  // 128-row groups present in each scale buffer
    // single-CTA kernel only: K is cut into k_splits ranges of k_tiles_per_split stages; with more than one range
    // each work item writes an fp32 partial tile to `partial` ([k_splits, M, N]) and a second kernel sums them.
    int k_splits, k_tiles_per_split;
    int k_rotate;             // != 0: each tile starts its K loop at a different stage (spreads requests for shared A rows)
    float* partial;
    int raster_group;         // m-tiles per band of the tile numbering (see tile_to_mn)
};

// One launch over several products (a layer's matrices at prefill): up to kMaxItems weights, each with its own activation,
// K, output scale and output, all with the same M.  Tiles are numbered through the items; items of equal K form a class,
// and every class has its own workers (CTAs or CTA pairs), because a tile's time is its K: with the workers dealt out by
// the host so that the longest class is as short as possible, a K = 14336 product runs beside K = 4096 ones without leaving
// SMs idle at the end (256 tokens, the seven matrices of a Llama-3-8B layer: one launch instead of seven on four streams).
constexpr int kMaxItems = 8;

struct GemmItem {
    const uint8_t* sfa;       // single-CTA kernel: scales are fetched by address
    const uint8_t* sfb;
    const float* alpha;
    const float* alpha2;
    __nv_bfloat16* out;
    int64_t sf_group_stride;
    int N, K;
    int sfb_groups;
    int tile_end;             // tiles of this and the earlier items of its class
};

// ---- epilogue -----------------------------------------------------------------------------------------------------
// A warp holds 32 rows of an accumulator, lane = row, and writes them as bf16(alpha * v).
//
// Written 16 bytes per lane straight from the registers, a store instruction touches 32 rows, half a sector of each: that
// bound every product whose K is short, and 2 bytes per lane where rows are no multiple of 16 bytes bound those at any K.
// Now, rows of a multiple of 16 bytes go out as TMA stores of 32 x 64 pieces (asynchronous, whole lines; pieces of 32 columns
// are 10 % slower; ragged edges clipped by the tensor map) or, where the ring leaves no room, 32 bytes per lane; other rows
// are turned through shared memory so that an instruction covers neighbours of one or two rows.  Measured (us): 4585 x 12864 x
// 2880 104 -> 82, 5644 x 16832 x 1088 140 -> 80, 8192^3 210 -> 198, 517 x 738 x 2240 22.7 -> 7.0, 2092 x 17604 x 6784 442 -> 115.

__device__ __forceinline__ uint32_t scaled_pair(uint32_t lo, uint32_t hi, float alpha) {
    const __nv_bfloat162 b2 = __floats2bfloat162_rn(__fmul_rn(__uint_as_float(lo), alpha), __fmul_rn(__uint_as_float(hi), alpha));
    return *reinterpret_cast<const uint32_t*>(&b2);
}

// 32 columns (16-byte chunks first .. first + 3 of a row) of a piece laid out for a TMA store with 128-byte swizzle.
__device__ __forceinline__ void stage_half(uint32_t piece, int first, float alpha, const uint32_t v[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(piece + lane * 128 + (((first + q) ^ (lane & 7)) << 4)),
                     "r"(scaled_pair(v[8 * q], v[8 * q + 1], alpha)), "r"(scaled_pair(v[8 * q + 2], v[8 * q + 3], alpha)),
                     "r"(scaled_pair(v[8 * q + 4], v[8 * q + 5], alpha)), "r"(scaled_pair(v[8 * q + 6], v[8 * q + 7], alpha))
                     : "memory");
}

// 32 columns from the registers, by way of `turn` where they do not start on 16-byte boundaries.
__device__ __forceinline__ void store_half(__nv_bfloat16* out, int M, int N, int row0, int col0, float alpha, const uint32_t v[32],
                                           uint32_t* turn) {
    const int lane = threadIdx.x & 31;
    uint32_t w[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) w[e] = scaled_pair(v[2 * e], v[2 * e + 1], alpha);
    if ((N & 7) == 0 && col0 + 32 <= N) {
        if (row0 + lane >= M) return;
        __nv_bfloat16* dst = out + static_cast<int64_t>(row0 + lane) * N + col0;
        if ((N & 15) == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
                asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + 16 * q), "r"(w[8 * q]),
                             "r"(w[8 * q + 1]), "r"(w[8 * q + 2]), "r"(w[8 * q + 3]), "r"(w[8 * q + 4]), "r"(w[8 * q + 5]),
                             "r"(w[8 * q + 6]), "r"(w[8 * q + 7])
                             : "memory");
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                *reinterpret_cast<uint4*>(dst + 8 * q) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
        }
        return;
    }
    __syncwarp();   // what was turned before has been read
#pragma unroll
    for (int e = 0; e < 16; ++e) turn[lane * kTurnPitch + e] = w[e];
    __syncwarp();
    const int cols = min(32, N - col0), rows = min(32, M - row0);
    if ((N & 1) == 0) {   // rows start on 4-byte boundaries (col0 is even): two rows per store
        const int c = lane & 15;
        if (2 * c < cols)
            for (int r = lane >> 4; r < rows; r += 2)
                *reinterpret_cast<uint32_t*>(out + static_cast<int64_t>(row0 + r) * N + col0 + 2 * c) = turn[r * kTurnPitch + c];
    } else if (lane < cols) {
        const uint16_t* half = reinterpret_cast<const uint16_t*>(turn) + lane;
        for (int r = 0; r < rows; ++r)
            reinterpret_cast<uint16_t*>(out)[static_cast<int64_t>(row0 + r) * N + col0 + lane] = half[r * kTurnPitch * 2];
    }
}

// One warp's 32 rows of an accumulator of BN columns.  The next 32 columns are on their way from TMEM while the current ones
// are rounded and stored, and `release` (the accumulator may be overwritten) runs as soon as the last ones have arrived.
// `turn` says which of the BUFS staged pieces is next; the caller waits for the last TMA stores before it returns.
template <int BN, int BUFS, class Release>
__device__ __forceinline__ void store_accumulator(uint32_t taddr, __nv_bfloat16* out, const CUtensorMap* map, int M, int N, int row0, int col0,
                                                  float alpha, uint8_t* stage, int& turn, Release release) {
    static_assert(BN % 64 == 0, "pieces of 64 columns");
    const bool tma = BUFS > 0 && (N & 7) == 0;
    const bool first_lane = (threadIdx.x & 31) == 0;
    uint32_t a[32], b[32];
    tc_ld_32x32b_x32(taddr, a);
#pragma unroll 1
    for (int c = 0; c < BN; c += 64) {
        const bool inside = row0 < M && col0 + c < N;
        const uint32_t piece = smem_u32(stage) + (BUFS > 1 ? turn : 0) * kPieceBytes;
        if (BUFS > 1 && ++turn == BUFS) turn = 0;
        tc_ld_wait();
        tc_ld_32x32b_x32(taddr + c + 32, b);
        if (tma) {
            if (first_lane) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(BUFS > 0 ? BUFS - 1 : 0) : "memory");
            __syncwarp();   // what was staged here before has been read
            stage_half(piece, 0, alpha, a);
        } else if (inside) {
            store_half(out, M, N, row0, col0 + c, alpha, a, reinterpret_cast<uint32_t*>(stage));
        }
        tc_ld_wait();
        if (c + 64 < BN) tc_ld_32x32b_x32(taddr + c + 64, a);
        else release();
        if (tma) {
            stage_half(piece, 4, alpha, b);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (first_lane) {
                if (inside)
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map), "r"(piece),
                                 "r"(col0 + c), "r"(row0)
                                 : "memory");
                asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
        } else if (inside && col0 + c + 32 < N) {
            store_half(out, M, N, row0, col0 + c + 32, alpha, b, reinterpret_cast<uint32_t*>(stage));
        }
    }
}

template <int G>
struct GroupTable {
    GemmItem item[G];
    int n_classes;
    int worker_end[G];        // workers of this and all earlier classes
    int item_end[G];          // items of this and all earlier classes
};

// Where a worker of a grouped launch stands: its class, and the item that its current tile belongs to.  Every role of a
// CTA walks the same tiles in the same order with a cursor of its own.
template <int G>
struct TileCursor {
    int local, workers, total, item, first_tile;
    __device__ __forceinline__ void init(const GroupTable<G>& g, int worker) {
        int c = 0;
        while (c + 1 < g.n_classes && worker >= g.worker_end[c]) ++c;
        const int begin = c > 0 ? g.worker_end[c - 1] : 0;
        local = worker - begin;
        workers = g.worker_end[c] - begin;
        item = c > 0 ? g.item_end[c - 1] : 0;
        total = g.item[g.item_end[c] - 1].tile_end;
        first_tile = 0;
    }
    // `tile` never decreases from call to call
    __device__ __forceinline__ void seek(const GroupTable<G>& g, int tile) {
        if constexpr (G > 1) while (tile >= g.item[item].tile_end) {
            first_tile = g.item[item].tile_end;
            ++item;
        }
    }
};

// Output scale of a launch: alpha[0], or alpha[0] * alpha2[0] rounded once (what a separate fp32 multiplication of the
// activation's and the weight's global scales gives).
__device__ __forceinline__ float load_alpha(const float* alpha, const float* alpha2) {
    // called behind griddep_wait(): the scales may be the work of the kernels before this one
    const float a = load_f32_after_wait(alpha);
    return alpha2 ? __fmul_rn(a, load_f32_after_wait(alpha2)) : a;
}

// Operand maps and the work list of one launch over G products (G = 1: an ordinary GEMM, whose K may be cut into ranges).
//
// A copy of a box that reaches beyond the matrix fills the rows outside with zeros, and takes longer over a row of zeros than over one
// that it fetches.  So a last tile that is not whole has a map of its own (`a_rest`, `b_rest`), whose box ends with the matrix.  The rows
// behind it in shared memory hold what was there before: bytes that are valid codes, for outputs that do not exist.  us, whole boxes /
// this, prepared: 128 x 64 tiles 17 x 6208 x 4224 10.1 / 5.9, 48 x 14336 x 4096 13.5 / 9.3, 150 x 3000 x 1024 3.45 / 3.15, 128 x 128 tiles 48 x 14336 x 4096 8.8 /
// 7.9.  (The pair kernels, which take larger launches, gain nothing by it and lose 1 to 3 % to the choice.)
template <int G>
struct TileParams {
    CUtensorMap a[G], b[G], a_rest[G], b_rest[G];
    GroupTable<G> g;
    int M;
    int k_splits, k_tiles_per_split, k_rotate;   // G = 1 only, see GemmParams
    float* partial;
    int raster_group;
    // != 0: every weight is a prepared weight, constant while launches with it are in flight, and may be read before
    // griddep_wait(); 0 (raw pointers): one may be the output of the kernel just before this one, like the tokens
    int weights_ready;
};

template <int BN, int G>
__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ TileParams<G> p) {
    using C = Cfg<BN>;
    extern __shared__ uint8_t smem_raw[];
    // The kernel queued behind this one may be scheduled at once: ahead of its own wait it reads nothing but a
    // prepared (constant) weight, and that wait covers this kernel's completion.
    griddep_launch();
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - raw_addr);
    // ring: [stage][A | B | SFA | SFB]; then barriers
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
    if (threadIdx.x == 0) trace_mark(0, 0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(tfull_bar(a), 1);
            mbar_init(tempty_bar(a), 4);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(const_cast<uint32_t*>(tmem_slot))),
                     "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        if (lane == 0) trace_mark(0, 1);
    }
    // The producer warp initialised the mbarriers itself (thread 0) and needs neither TMEM nor the other warps, so it
    // only ARRIVES on the prologue barrier and starts its copies at once; the first HBM round trip then overlaps the
    // TMEM allocation.  Warps 1..5 wait for the arrival (barrier initialisation, TMEM address).
    tc_fence_before();
    if (warp == 0) {
        __syncwarp();
        asm volatile("bar.arrive 1, %0;" ::"n"(kThreads) : "memory");
    } else {
        asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory");
    }
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;   // meaningful in warps 1..5 only
    if (threadIdx.x == 32) trace_mark(0, 2);
    if (warp >= 2) griddep_wait();    // alpha, and the output buffer, belong to whatever ran before: epilogue only after it

    const int m_tiles = (p.M + kBM - 1) / kBM;
    TileCursor<G> cur;
    cur.init(p.g, blockIdx.x);
    const int splits = G == 1 ? p.k_splits : 1;
    const int total_tiles = cur.total * splits;   // work items: (K range, n tile, m tile)
    // work item -> its product (cur.item), K range, m tile and n tile
    auto locate = [&](int tile, int& ks, int& mt, int& nt) {
        ks = splits > 1 ? tile / cur.total : 0;
        const int t2 = tile - ks * cur.total;
        cur.seek(p.g, t2);
        const int n_tiles = (p.g.item[cur.item].N + BN - 1) / BN;
        tile_to_mn(t2 - cur.first_tile, m_tiles, n_tiles, p.raster_group, mt, nt);
    };
    // stages of the current product's K range: first, count, and where the loop starts (see GemmParams::k_rotate)
    auto k_range = [&](int ks, int tile, int& kt_begin, int& kcount, int& rot) {
        const int k_tiles = (p.g.item[cur.item].K + kBK - 1) / kBK;
        kt_begin = splits > 1 ? ks * p.k_tiles_per_split : 0;
        kcount = (splits > 1 ? min(k_tiles, kt_begin + p.k_tiles_per_split) : k_tiles) - kt_begin;
        rot = G == 1 && p.k_rotate ? ((tile - ks * cur.total) * 5) % kcount : 0;
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ producer
        {
            const bool issuer = elect_one();
            // One lane requests four copies per stage, and how long it takes over them bounds these kernels (with the addresses, the K
            // range and the number of scale groups worked out for every stage, us: 128 x 64 tiles 128 x 4096 x 4096 7.27 -> 5.48, 512 x 4096 x
            // 4096 12.5 -> 9.7; 128 x 128 tiles 333 x 5000 x 2880 7.16 -> 6.28, 300 x 1024 x 8192 12.1 -> 9.3, 2048 x 4096 x 4096 24.9 -> 18.8).
            // So all that is constant over a tile is worked out once per tile.
            // The current tile: coordinates, K range (see k_range), its operands' maps, where its scales are.
            int ks, mt = 0, nt = 0, kt_begin = 0, kcount = 0, rot = 0, kt_last = 0;
            uint32_t last_bytes = 0, groups = 0, operand_bytes = 0;
            const CUtensorMap *map_a = &p.a[0], *map_b = &p.b[0];
            const uint8_t *sfa = nullptr, *sfb = nullptr;
            int64_t group_stride = 0;
            auto set_tile = [&](int tile) {
                locate(tile, ks, mt, nt);
                k_range(ks, tile, kt_begin, kcount, rot);
                const GemmItem& it = p.g.item[cur.item];
                const int a_rows = box_rows(p.M, mt, kBM), b_rows = box_rows(it.N, nt, BN);
                map_a = box_map(a_rows, kBM) == kRestMap ? &p.a_rest[cur.item] : &p.a[cur.item];
                map_b = box_map(b_rows, BN) == kRestMap ? &p.b_rest[cur.item] : &p.b[cur.item];
                operand_bytes = static_cast<uint32_t>(a_rows + b_rows) * kBKBytes;
                group_stride = it.sf_group_stride;
                const int grp0 = BN == 64 ? (nt >> 1) : nt * C::kNG;   // first 128-row scale group of this B tile
                groups = static_cast<uint32_t>(min(C::kNG, it.sfb_groups - grp0));
                sfa = it.sfa + static_cast<int64_t>(mt) * group_stride;
                sfb = it.sfb + static_cast<int64_t>(grp0) * group_stride;
                kt_last = (it.K + kBK - 1) / kBK - 1;
                last_bytes = 512u * static_cast<uint32_t>((it.K - kt_last * kBK + 63) / 64);   // 64-element K blocks of the last stage
            };
            // Stage copies come in two halves: the weight half (B tile and its scales) of a prepared weight depends on nothing that ran
            // before this kernel, the token half (A tile and its scales) may be the previous kernel's output.  The
            // weight halves of the first ring-full go out before griddep_wait(), so that with a programmatic dependent
            // launch the weight stream starts while the previous kernel is still finishing.  A raw weight has to
            // wait itself, and its first ring-full goes side by side with the tokens: copies are carried out in order, and behind a ring-full
            // of weights the first stage's tokens come late (us, 100 x 14336 x 4096 10.01 -> 8.87, 150 x 3000 x 1024 4.22 -> 3.62, 1000 x 2048 x
            // 2048 6.05 -> 5.54).
            auto issue = [&](int st, int kt, bool weights, bool tokens) {
                const uint32_t sf_bytes = kt == kt_last ? last_bytes : 2048u;
                const uint32_t sbase = base + st * C::kStageBytes;
                const int64_t sf_at = static_cast<int64_t>(kt) * 2048;
                if (weights) {
                    mbar_expect_tx(full_bar(st), operand_bytes + sf_bytes * (1 + groups));
                    tma_load_2d(sbase + C::kABytes, map_b, kt * kBKBytes, nt * BN, full_bar(st));
                }
                if (tokens) tma_load_2d(sbase, map_a, kt * kBKBytes, mt * kBM, full_bar(st));
                if (weights) {
                    bulk_load_1d(sbase + C::kABytes + C::kBBytes + C::kSfaBytes, sfb + sf_at, sf_bytes, full_bar(st));
                    if (C::kNG > 1 && groups > 1)
                        bulk_load_1d(sbase + C::kABytes + C::kBBytes + C::kSfaBytes + 2048, sfb + group_stride + sf_at, sf_bytes, full_bar(st));
                }
                if (tokens) bulk_load_1d(sbase + C::kABytes + C::kBBytes, sfa + sf_at, sf_bytes, full_bar(st));
            };
            const bool any = cur.local < total_tiles;
            if (any) set_tile(cur.local);
            if (any && issuer) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(map_a) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(map_b) : "memory");
            }
            const int early = any && !(G == 1 && p.k_rotate) ? min(kcount, C::kStages) : 0;   // stages requested without a wait
            if (issuer && p.weights_ready)
                for (int i = 0; i < early; ++i) issue(i, kt_begin + i, true, false);
            griddep_wait();
            if (issuer)
                for (int i = 0; i < early; ++i) issue(i, kt_begin + i, !p.weights_ready, true);
            __syncwarp();
            int stage = early == C::kStages ? 0 : early;
            uint32_t phase = early == C::kStages ? 1u : 0u;
            bool ok = true;
            for (int tile = cur.local; ok && tile < total_tiles; tile += cur.workers) {
                int i = early;
                if (tile != cur.local) {
                    set_tile(tile);
                    i = 0;
                }
                int kt = kt_begin + i + rot;
                for (; i < kcount; ++i) {
                    if (!(ok = mbar_wait_warp(empty_bar(stage), phase ^ 1u, abort_flag, (1u << 24) | kt))) break;
                    if (issuer) issue(stage, kt, true, true);
                    __syncwarp();
                    if (++kt == kt_begin + kcount) kt = kt_begin;
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        {
            const bool issuer = elect_one();
            constexpr uint32_t idesc = instr_desc<BN>();
            int stage = 0;
            uint32_t phase = 0;
            int acc = 0;
            uint32_t acc_phase = 0;
            bool ok = true;
            for (int tile = cur.local; ok && tile < total_tiles; tile += cur.workers) {
                if (!(ok = mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u, abort_flag, (2u << 24) | 0xffff))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * BN;
                int ks, mt, nt, kt_begin, kcount, rot;
                locate(tile, ks, mt, nt);
                k_range(ks, tile, kt_begin, kcount, rot);
                const int K = p.g.item[cur.item].K;
                // a 64-row B tile is one half of a 128-row scale group: rows 64..127 sit two TMEM columns further on
                const uint32_t sfb_half = BN == 64 ? 2u * (nt & 1) : 0u;
                int kt = kt_begin + rot;
                for (int i = 0; i < kcount; ++i) {
                    if (!(ok = mbar_wait_warp(full_bar(stage), phase, abort_flag, (2u << 24) | kt))) break;
                    tc_fence_after();
                    const int kb_count = min(4, (K - kt * kBK + 63) / 64);
                    const uint32_t sbase = base + stage * C::kStageBytes;
                    const uint32_t a_lo = ((sbase & 0x3ffffu) >> 4) | (1u << 16);
                    const uint32_t b_lo = a_lo + (C::kABytes >> 4);
                    const uint32_t sfa_lo = ((sbase + C::kABytes + C::kBBytes) & 0x3ffffu) >> 4;
                    const uint32_t sfb_lo = sfa_lo + (C::kSfaBytes >> 4);
                    const uint32_t set = (i & 1) * C::kSfSetCols;
                    const uint32_t sfa_t = tmem_base + C::kSfaCol + set;
                    const uint32_t sfb_t = tmem_base + C::kSfbCol + set;
                    const uint32_t sfb_use = sfb_t + sfb_half;
                    const uint32_t first = i > 0 ? 1u : 0u;
                    if (!issuer) {
                        // nothing to issue on this lane
                    } else if (kb_count == 4) {
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb) {
                            tc_cp_lohi(sfa_t + 4 * kb, sfa_lo + 32 * kb);
#pragma unroll
                            for (int g = 0; g < C::kNG; ++g)
                                tc_cp_lohi(sfb_t + 4 * C::kNG * kb + 4 * g, sfb_lo + 128 * g + 32 * kb);
                        }
#pragma unroll
                        for (int kb = 0; kb < 4; ++kb)   // 32 bytes of K per instruction: start address + 2 (x16 B)
                            tc_mma_lohi(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa_t + 4 * kb, sfb_use + 4 * C::kNG * kb,
                                        kb == 0 ? first : 1u);
                    } else {
                        for (int kb = 0; kb < kb_count; ++kb) {
                            tc_cp_lohi(sfa_t + 4 * kb, sfa_lo + 32 * kb);
                            for (int g = 0; g < C::kNG; ++g)
                                tc_cp_lohi(sfb_t + 4 * C::kNG * kb + 4 * g, sfb_lo + 128 * g + 32 * kb);
                        }
                        for (int kb = 0; kb < kb_count; ++kb)
                            tc_mma_lohi(d_tmem, a_lo + 2 * kb, b_lo + 2 * kb, idesc, sfa_t + 4 * kb, sfb_use + 4 * C::kNG * kb,
                                        kb == 0 ? first : 1u);
                    }
                    if (issuer) tc_commit(empty_bar(stage));  // slot reusable once these MMAs have read it
                    __syncwarp();
                    if (++kt == kt_begin + kcount) kt = kt_begin;
                    if (++stage == C::kStages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok) break;
                if (issuer) tc_commit(tfull_bar(acc));  // accumulator complete
                __syncwarp();
                if (++acc == C::kAcc) {
                    acc = 0;
                    acc_phase ^= 1u;
                }
            }
        }
    } else {
        // ------------------------------------------------------------------ epilogue (warps 2..5)
        const int sp = warp & 3;  // TMEM sub-partition this warp may read: lanes 32*sp .. 32*sp+31
        // staged output, behind the ring
        uint8_t* epilogue_stage = aligned + C::kStages * C::kStageBytes + sp * (C::kEpilogueBytes / 4);
        int out_turn = 0;
        int alpha_item = -1;
        float alpha = 0.0f;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int tile = cur.local; ok && tile < total_tiles; tile += cur.workers) {
            int ks, mt, nt;
            locate(tile, ks, mt, nt);
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
            const int row0 = mt * kBM + sp * 32;
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(sp * 32) << 16) + acc * BN;
            auto release = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(tempty_bar(acc));
            };
            if (splits == 1) {
                store_accumulator<BN, 0>(taddr, it.out, nullptr, p.M, N, row0, nt * BN, alpha, epilogue_stage, out_turn, release);
            } else {
                // fp32 partials of this K range; alpha and the bf16 rounding happen in the reduction kernel
#pragma unroll 1
                for (int c = 0; c < BN / 32; ++c) {
                    uint32_t v[32];
                    tc_ld_32x32b_x32(taddr + c * 32, v);
                    tc_ld_wait();
                    const int col0 = nt * BN + c * 32;
                    if (row0 + lane >= p.M || col0 >= N) continue;
                    float* prow = p.partial + (static_cast<int64_t>(ks) * p.M + row0 + lane) * N + col0;
                    if ((N % 4) == 0 && col0 + 32 <= N) {
#pragma unroll
                        for (int q = 0; q < 8; ++q)
                            *reinterpret_cast<uint4*>(prow + 4 * q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                    } else {
                        for (int e = 0; e < 32; ++e)
                            if (col0 + e < N) prow[e] = __uint_as_float(v[e]);
                    }
                }
                release();
            }
            if (++acc == C::kAcc) {
                acc = 0;
                acc_phase ^= 1u;
            }
        }
    }

    if (lane == 0) trace_mark(0, warp == 0 ? 3 : warp == 1 ? 4 : 5);
    // ---------------------------------------------------------------------- teardown
    if (*abort_flag) {
        // give any bulk copy still in flight time to land before shared memory is released
        const uint64_t t0 = global_timer_ns();
        while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) trace_mark(0, 6);
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
        if (lane == 0) trace_mark(0, 8);
    }
}

// out[m, n] = bf16(alpha * sum over K ranges of partial[s][m][n]); ranges are added in ascending order.
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ partial, const float* alpha_ptr,
                                                            const float* alpha2_ptr, __nv_bfloat16* __restrict__ out,
                                                            int64_t mn, int splits) {
    const float alpha = load_alpha(alpha_ptr, alpha2_ptr);
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < mn; i += static_cast<int64_t>(gridDim.x) * 256) {
        float acc = partial[i];
        for (int s = 1; s < splits; ++s) acc = __fadd_rn(acc, partial[static_cast<int64_t>(s) * mn + i]);
        out[i] = __float2bfloat16_rn(__fmul_rn(acc, alpha));
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// [rows, k_bytes] row-major byte matrix, box = 128 bytes x box_rows, 128-byte swizzle, zero fill.
static int make_operand_map(CUtensorMap* map, const void* ptr, int64_t rows, int64_t k_bytes, int box_rows) {
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return NVFP4_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(k_bytes), static_cast<cuuint64_t>(rows)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(k_bytes)};
    cuuint32_t box[2] = {static_cast<cuuint32_t>(kBKBytes), static_cast<cuuint32_t>(box_rows)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? NVFP4_OK : NVFP4_ERR_UNSUPPORTED;
}

// The output [M, N] bf16 in pieces of 32 rows x 64 columns; only for rows of a multiple of 16 bytes (else left undefined).
static int make_output_map(CUtensorMap* map, void* ptr, int64_t M, int64_t N) {
    if (N % 8) return NVFP4_OK;
    EncodeTiledFn enc = encode_tiled_fn();
    if (!enc) return NVFP4_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(M)};
    cuuint64_t strides[1] = {static_cast<cuuint64_t>(N * 2)};
    cuuint32_t box[2] = {64, 32};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? NVFP4_OK : NVFP4_ERR_UNSUPPORTED;
}

// Per-device facts the launchers need on every call, looked up once per device.

struct DeviceInfo {
    int device;
    int sms;
};
static DeviceInfo device_info() {
    static int sm_count[64] = {0};
    DeviceInfo d{0, 148};
    if (cudaGetDevice(&d.device) != cudaSuccess || d.device < 0 || d.device >= 64) return d;
    if (sm_count[d.device] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d.device) == cudaSuccess && v > 0) sm_count[d.device] = v;
    }
    if (sm_count[d.device] > 0) d.sms = sm_count[d.device];
    return d;
}
// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) is per device and sticky: once per (kernel, device) is enough.
template <class Kernel>
static cudaError_t allow_full_smem(Kernel kernel, bool* done_per_device, int device) {
    if (device >= 0 && device < 64 && done_per_device[device]) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmDynSmemBytes);
    if (e == cudaSuccess && device >= 0 && device < 64) done_per_device[device] = true;
    return e;
}

// A weight matrix prepared once for many GEMM calls: its tensor maps for every tile height the kernels use.
struct WeightHandle {
    uint32_t magic;
    int device;
    const uint8_t* b;
    const uint8_t* sfb;
    int64_t N, K;
    CUtensorMap rows[4], rest[4];   // operand maps by box height (kHeights), and of a last box that is not whole (N % height rows, if any)
    CUtensorMap scales;             // scale groups as rows of 8-byte words (pair kernels)
    static constexpr int kHeights[4] = {64, 96, 128, 256};
    static constexpr int index(int height) { return height == 64 ? 0 : height == 96 ? 1 : height == 128 ? 2 : 3; }
};
// Maps of a [rows, k_bytes] operand in boxes of `height` rows: of whole ones and of the rows % height last rows, each where there are
// any.  (Encoding one takes the host a while, and a launch of a few microseconds does not hide it.)
static int make_operand_maps(CUtensorMap* whole, CUtensorMap* rest, const void* ptr, int64_t rows, int64_t k_bytes, int height) {
    int st = NVFP4_OK;
    if (has_map(rows, height, kWholeMap)) st = make_operand_map(whole, ptr, rows, k_bytes, height);
    if (st == NVFP4_OK && has_map(rows, height, kRestMap)) st = make_operand_map(rest, ptr, rows, k_bytes, static_cast<int>(rows % height));
    return st;
}
// A weight's maps for a launch: the prepared ones, or encoded now.
static int weight_maps(CUtensorMap* whole, CUtensorMap* rest, const GemmParams& p, const WeightHandle* wh, int height) {
    if (!wh) return make_operand_maps(whole, rest, p.b, p.N, p.K / 2, height);
    const int i = WeightHandle::index(height);
    if (has_map(p.N, height, kWholeMap)) *whole = wh->rows[i];
    if (has_map(p.N, height, kRestMap)) *rest = wh->rest[i];
    return NVFP4_OK;
}
constexpr uint32_t kWeightMagic = 0x4e56463u;

// Fills the work list for `workers` CTAs (or CTA pairs) and returns how many are used (0: too few for the classes, or more
// tiles than a launch can number).
// A class is a run of items of equal K.  With one class every worker takes tiles of it; with several the smallest makespan
// T (in K stages) is searched for which the classes' workers, ceil(tiles / floor(T / k)) each, fit.
template <int G>
static int fill_group_table(GroupTable<G>& g, const GemmParams* list, int n, int m_tiles, int bn, int workers) {
    int64_t tiles[G], k[G], stages = 0, longest = 0;
    g.n_classes = 0;
    for (int i = 0; i < n; ++i) {
        const GemmParams& p = list[i];
        GemmItem& it = g.item[i];
        it.sfa = p.sfa;
        it.sfb = p.sfb;
        it.alpha = p.alpha;
        it.alpha2 = p.alpha2;
        it.out = p.out;
        it.sf_group_stride = p.sf_group_stride;
        it.N = p.N;
        it.K = p.K;
        it.sfb_groups = p.sfb_groups;
        const bool same = i > 0 && list[i - 1].K == p.K;
        if (!same) {
            k[g.n_classes] = (p.K + kBK - 1) / kBK;
            tiles[g.n_classes++] = 0;
        }
        const int c = g.n_classes - 1;
        const int64_t mine = static_cast<int64_t>(m_tiles) * ((p.N + bn - 1) / bn);
        tiles[c] += mine;
        stages += mine * k[c];
        if (k[c] > longest) longest = k[c];
        if (tiles[c] > kMaxTiles) return 0;
        it.tile_end = static_cast<int>(tiles[c]);
        g.item_end[c] = i + 1;
    }
    if (g.n_classes == 1) {
        const int64_t all = tiles[0] * (G == 1 ? list[0].k_splits : 1);
        if (all > kMaxTiles) return 0;
        return g.worker_end[0] = static_cast<int>(all < workers ? all : workers);
    }
    if (workers < g.n_classes) return 0;
    int64_t T = (stages + workers - 1) / workers;
    if (T < longest) T = longest;
    for (;;) {
        int64_t used = 0, next = INT64_MAX;
        for (int c = 0; c < g.n_classes; ++c) {
            const int64_t per = T / k[c];
            used += (tiles[c] + per - 1) / per;
            g.worker_end[c] = static_cast<int>(used);
            if ((per + 1) * k[c] < next) next = (per + 1) * k[c];
        }
        if (used <= workers) return static_cast<int>(used);
        T = next;
    }
}

// Time of the busiest worker, at so much per K stage of its first tile, of the others, and per tile that follows another.
template <int G>
static double list_makespan(const GroupTable<G>& g, const GemmParams* list, double first_stage, double stage, double epilogue) {
    double longest = 0.0;
    for (int c = 0; c < g.n_classes; ++c) {
        const int workers = g.worker_end[c] - (c > 0 ? g.worker_end[c - 1] : 0);
        const int last = g.item_end[c] - 1;
        const int tiles = (g.item[last].tile_end + workers - 1) / workers, k = (list[last].K + kBK - 1) / kBK;
        const double mine = k * first_stage + (tiles - 1) * (k * stage + epilogue);
        if (mine > longest) longest = mine;
    }
    return longest;
}

// One launch over the `n` products of `list` (1 <= n <= G), items of equal K next to one another, longest K first.
template <int BN, int G>
static int launch_list(const GemmParams* list, const WeightHandle* const* wh, int n, cudaStream_t stream) {
    using C = Cfg<BN>;
    static_assert(C::kSmemBytes <= kGemmDynSmemBytes, "ring does not fit");
    const GemmParams& p0 = list[0];
    TileParams<G> q;
    q.M = p0.M;
    q.k_splits = p0.k_splits;
    q.k_tiles_per_split = p0.k_tiles_per_split;
    q.k_rotate = p0.k_rotate;
    q.partial = p0.partial;
    const int m_tiles = (q.M + kBM - 1) / kBM;
    q.raster_group = band_rows(p0.raster_group, m_tiles);
    q.weights_ready = 1;
    for (int i = 0; i < n; ++i) {
        const GemmParams& p = list[i];
        if (!wh[i]) q.weights_ready = 0;
        int st = NVFP4_OK;
        if (i > 0 && p.a == list[i - 1].a && p.K == list[i - 1].K) {   // products of one activation share its maps
            q.a[i] = q.a[i - 1];
            q.a_rest[i] = q.a_rest[i - 1];
        } else {
            st = make_operand_maps(&q.a[i], &q.a_rest[i], p.a, p.M, p.K / 2, kBM);
        }
        if (st == NVFP4_OK) st = weight_maps(&q.b[i], &q.b_rest[i], p, wh[i], BN);
        if (st != NVFP4_OK) return st;
    }
    const DeviceInfo di = device_info();
    const int grid = fill_group_table<G>(q.g, list, n, m_tiles, BN, di.sms);
    if (grid == 0) return NVFP4_ERR_TOO_LARGE;
    static bool attr_done[64] = {false};
    cudaError_t e = allow_full_smem(gemm_kernel<BN, G>, attr_done, di.device);
    if (e != cudaSuccess) return static_cast<int>(e);
    e = launch_dependent(gemm_kernel<BN, G>, dim3(grid), dim3(kThreads), kGemmDynSmemBytes, stream, q);
    if (e != cudaSuccess || G > 1 || p0.k_splits == 1) return static_cast<int>(e);
    const int64_t mn = static_cast<int64_t>(p0.M) * p0.N;
    int64_t rblocks = (mn + 255) / 256;
    if (rblocks > 148 * 8) rblocks = 148 * 8;
    splitk_reduce_kernel<<<static_cast<unsigned>(rblocks), 256, 0, stream>>>(p0.partial, p0.alpha, p0.alpha2, p0.out, mn, p0.k_splits);
    return static_cast<int>(cudaGetLastError());
}

template <int BN>
static int launch(const GemmParams& p, cudaStream_t stream, const WeightHandle* wh) {
    return launch_list<BN, 1>(&p, &wh, 1, stream);
}

}  // namespace gemm
}  // namespace nvfp4
