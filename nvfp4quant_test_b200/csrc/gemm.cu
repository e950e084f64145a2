// NVFP4 block-scaled GEMM for sm_100a:
//   out[M, N] (bf16) = alpha * sum_k dq(a)[m, k] * dq(b)[n, k]
// with a, b packed E2M1 (K-major) and one UE4M3 scale per 16 elements stored in the
// 128x4-tiled layout the quantizer writes.  Replaces vllm's cutlass_scaled_fp4_mm
// (vllm/_custom_ops.py:741-752), the consumer efsotr/nvfp4quant_test names at README.md:68.
//
// Structure (one persistent CTA per SM, 192 threads):
//   warp 0      producer: TMA tile loads of A / B (128-byte swizzle) and bulk copies of the
//               scale tiles into a shared-memory ring (6 stages with 128-wide tiles, 4 with 256-wide); what is constant over a tile
//               is worked out once per tile, and the first ring-full is requested without a wait
//   warp 1      MMA issuer: tcgen05.cp scale tiles smem -> TMEM, then
//               tcgen05.mma.kind::mxf4nvf4.block_scale (K = 64 per instruction) into a TMEM
//               accumulator; tcgen05.commit releases ring slots / publishes the accumulator
//   warps 2-5   epilogue: tcgen05.ld the accumulator, * alpha, -> bf16, store
// No cluster multicast is used anywhere.  Every barrier wait is bounded: on expiry the kernel
// records a status word and every role leaves its loop, so a fault in the pipeline logic
// surfaces as an error code rather than a hung device.
//
// Launches are programmatic dependent launches (see common.cuh): a kernel lets the one queued behind it be scheduled from its
// first instruction and itself waits before it touches anything an earlier kernel may have written; a prepared weight is a
// constant by contract and is streamed ahead of that wait.  nvfp4_gemm_launch_grouped multiplies one activation with several
// prepared weights in one launch of the decode-sized kernel.
//
// This file holds the C entry points and the kernel choice; the kernels live in gemm_tile.cuh (one CTA per tile),
// gemm_pair.cuh (CTA pairs, cta_group::2) and gemm_skinny.cuh (decode-sized batches, K ranges across a cluster),
// all on the PTX wrappers of tc_ptx.cuh.  One translation unit, so that there is one status word.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>
#include <utility>

#include "gemm_tile.cuh"
#include "gemm_pair.cuh"
#include "gemm_skinny.cuh"
#include "gemm_peak.cuh"

static int g_gemm_force_path = 0;
constexpr int64_t kSkinnyMaxM = 128;   // what the skinny kernel accepts
static int g_gemm_force_splits = 0;    // 0 = by shape
static int g_gemm_force_rotate = -1;   // -1 = by shape
static int g_gemm_raster_group = 0;    // 0 = default

// K ranges for the single-CTA kernel.  Measured on B200 (M <= 128, K = 8192): cutting K never paid, the fixed
// cost of a second kernel and of the partial tiles outweighs the extra SMs, so the default is one range and the
// feature stays available through nvfp4_gemm_tune for shapes with very few tiles and very long K.
static int choose_k_splits(int64_t, int64_t, int64_t K) {
    if (g_gemm_force_splits <= 0) return 1;
    const int64_t k_tiles = (K + 255) / 256;
    return static_cast<int>(g_gemm_force_splits < k_tiles ? g_gemm_force_splits : k_tiles);
}

extern "C" size_t nvfp4_gemm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int splits = choose_k_splits(M, N, K);
    return splits > 1 ? static_cast<size_t>(splits) * static_cast<size_t>(M) * static_cast<size_t>(N) * sizeof(float) : 0;
}

// Testing hook: m-tiles per band of the tile numbering (0 = default).
extern "C" int nvfp4_gemm_tune_raster(int group) {
    if (group < 0 || group > 4096) return NVFP4_ERR_BAD_ENUM;
    g_gemm_raster_group = group;
    return NVFP4_OK;
}

// Testing hook: 0 = launch the library's kernels (GEMM, quantizer, global scale) without the programmatic-dependent-launch
// attribute, 1 = with (default).
extern "C" int nvfp4_gemm_tune_pdl(int enabled) {
    nvfp4::g_dependent_launch = enabled ? 1 : 0;
    return NVFP4_OK;
}

// Testing hook: K ranges (0 = by shape) and K-loop rotation (-1 = by shape, 0 = off, 1 = on) of the single-CTA kernel.
extern "C" int nvfp4_gemm_tune(int k_splits, int k_rotate) {
    if (k_splits < 0 || k_splits > 16 || k_rotate < -1 || k_rotate > 1) return NVFP4_ERR_BAD_ENUM;
    g_gemm_force_splits = k_splits;
    g_gemm_force_rotate = k_rotate;
    return NVFP4_OK;
}

// Testing hook: 0 = choose the kernel by shape, 1 = 128x128 tiles, 2 = 128x256 tiles, 3 = CTA-pair 256x256 tiles,
// 4 = CTA-pair 256x192 tiles with two accumulators, 5 = skinny kernel (M <= 128; nvfp4_gemm_tune's k_splits then
// sets its K ranges per weight tile; larger M falls back to the choice by shape), 6 = 128x64 tiles,
// 7 = CTA-pair 256x128 tiles.
extern "C" int nvfp4_gemm_force_path(int path) {
    if (path < 0 || path > 7) return NVFP4_ERR_BAD_ENUM;
    g_gemm_force_path = path;
    return NVFP4_OK;
}

// Measured kernel choice (generated file, see its first lines): {M, N, K, path} for a grid of shapes on a 148-SM B200.
struct PlanRow {
    int M, N, K, path;
};
static const PlanRow kPlanTable[] = {
#include "gemm_plan_table.inc"
};
// Fastest measured kernel for (N, K) at the smallest tabulated M >= the launch's M; 0 when the shape is not tabulated.
static int table_path(int64_t M, int64_t N, int64_t K) {
    int64_t best_m = INT64_MAX;
    int path = 0;
    for (const PlanRow& r : kPlanTable)
        if (r.N == N && r.K == K && r.M >= M && r.M < best_m) {
            best_m = r.M;
            path = r.path;
        }
    return path;
}

// Microseconds of one launch, by kernel.  A K stage takes as long as it does alone or as the fetches of all SMs at work let it, tiles go
// over the SMs in waves, and a wave takes the longer of its stages and its share of the weights, tokens and output at the rate the
// kernel streams them.  The constants are a fit to 25000 random products (1 .. 8192 tokens, pairs from 129 on, N 512 .. 28672, a sixth of
// them no multiple of 8, K 1024 .. 14336) and 13000 launches over the products of a decoder layer, or its q / k / v, or gate / up (17 .. 1024
// tokens), launches back to back and weights from HBM every time: rms error 5-10 %.  How far the kernel chosen is behind the fastest one on
// average, over 15700 other products: back to back up to 32 tokens 0.5 %, 33 to 128 0.7, 129 to 512 0.3, up to 1024 0.7, more 1.2; behind the quantizer
// 0.4, 1.0, 0.9, 0.6, 0.6.  (By the fit to waves and one time per stage that this one replaces 1.5 %, 1.8 % where N is no multiple of 8, and
// up to 20 % behind the choice before that one: 190 x 28288 x 10304, 1432 x 2266 x 13824, 30 x 12797 x 1024.)
struct TileCost {
    int path, rows, cols, pair;
    // us: a launch, and with a whole tile's tokens; a K stage alone; relative to it, one behind a worker's first tile; us: an epilogue that
    // the next tile waits for, in a list and in many waves of one product (128x128 tiles with a K of less than 1900 fell 8 to 16 % short there by
    // the other: 2000 x 23616 x 1472); relative to it, one at the end of a last wave that is not full
    double launch, tokens, stage, later, epilogue, wave_epilogue, last_epilogue;
    // KB per us: operands of all SMs, streamed bytes; relative to their bytes: output, and in pairs a box's rows of zeros
    double fabric, memory, out_weight, empty_rows;
    // us, where the rows of the output are no multiple of 16 bytes: a launch, a tile
    double ragged_launch, ragged_tile;
};
static const TileCost kTileCosts[] = {
    {1, 128, 128, 0, 2.21, 0.88, 0.214, 0.893, 0.35, 0.50, 1.02, 19342, 6567, 1.00, 0.00, 1.10, 0.79},
    {2, 128, 256, 0, 2.31, 1.45, 0.352, 0.926, 1.41, 1.41, 1.04, 20034, 5881, 1.00, 0.00, 2.15, 1.84},
    {3, 256, 256, 1, 4.88, 0.09, 0.287, 0.828, 2.04, 2.04, 0.64, 14042, 6849, 1.64, 0.90, 2.48, 2.60},
    {4, 256, 192, 1, 4.29, 0.64, 0.228, 0.768, 1.19, 1.19, 0.41, 14572, 7654, 1.89, 0.43, 1.61, 1.58},
    {6, 128, 64, 0, 1.97, 0.51, 0.205, 0.876, 0.45, 0.45, 1.22, 23086, 6200, 1.52, 0.00, 0.65, 0.14},
    {7, 256, 128, 1, 3.75, 0.61, 0.188, 0.705, 0.95, 0.95, 0.53, 15500, 8378, 2.78, 0.65, 1.13, 1.09}};

// A launch whose workers take several tiles each, products of one K: what is queued behind it does not get in while the last ones
// end (2 x 14336 x 4096, 32 tokens, behind the quantizer: 128x128 tiles, 224 of them, 17.3 us, the decode-sized kernel 14.8; back to
// back 13.5 and 13.0).
constexpr double kTail = 0.8;

// Of two things that go on at the same time; they are in one another's way where both take about as long.
static double longer(double a, double b) {
    const double a2 = a * a, b2 = b * b;
    return std::sqrt(std::sqrt(a2 * a2 + b2 * b2));
}
// A K stage with `active` workers at it, tiles of `cols` columns on average.
static double stage_time(const TileCost& c, int64_t M, double cols, double active) {
    const double rows = static_cast<double>(M) / static_cast<double>((M + c.rows - 1) / c.rows);
    const double kbytes = (rows + (c.pair ? c.empty_rows * (c.rows - rows) : 0.0) + cols) * 0.128 + 4.0;   // operands, scales
    return longer(c.stage, kbytes * active / c.fabric);
}
static double launch_time(const TileCost& c, int64_t M, bool ragged) {
    return c.launch + c.tokens * std::min(static_cast<double>(M) / 128.0, 1.0) + (ragged ? c.ragged_launch : 0.0);
}
static double streamed_kbytes(const TileCost& c, int64_t M, int64_t N, int64_t K) {
    return (static_cast<double>(M + N) * static_cast<double>(K) * 9.0 / 16.0 + c.out_weight * 2.0 * static_cast<double>(M) * static_cast<double>(N)) / 1000.0;
}

static double tile_time(const TileCost& c, int64_t M, int64_t N, int64_t K, int sms) {
    const double workers = c.pair ? (sms > 1 ? sms / 2 : 1) : sms;
    const double n_tiles = static_cast<double>((N + c.cols - 1) / c.cols), tiles = static_cast<double>((M + c.rows - 1) / c.rows) * n_tiles;
    const double k = static_cast<double>((K + 255) / 256), cols = static_cast<double>(N) / n_tiles;
    const bool ragged = N % 8 != 0;
    const double share = streamed_kbytes(c, M, N, K) / tiles / c.memory, epilogue = c.wave_epilogue + (ragged ? c.ragged_tile : 0.0);
    const double full = std::floor(tiles / workers), rest = tiles - full * workers, first = std::min(tiles, workers);
    double t = launch_time(c, M, ragged) + longer(k * stage_time(c, M, cols, first), share * first);
    if (full > 1.0) t += (full - 1.0) * longer(k * c.later * stage_time(c, M, cols, workers) + epilogue, share * workers);
    if (tiles > workers) t += kTail;
    if (full > 0.0 && rest > 0.0) t += longer(k * c.later * stage_time(c, M, cols, rest) + epilogue * c.last_epilogue, share * rest);
    return t;
}

// A row's kernel was fastest at the row's M; how the tiles fill the waves at the launch's own M may favour another (600 x 7168 x 8192
// would take the 1024-token row's 256x256 tiles in two waves, 27 us, and takes 128x256 ones in one, 17).  The model errs by less than this
// on every row of the table, so that a row holds at its own size.
constexpr double kRowMargin = 1.18;

// The decode-sized kernel: the stages of its K ranges, with the fetches of up to two CTAs an SM, or the stream of the weights; the
// exchange of partials; and an epilogue that grows with the tokens.  Fit to 13900 random products of up to 128 tokens, rms error
// 6 %.
static double skinny_time(int64_t M, int64_t K, int n_tiles, int ranks) {
    const double m = static_cast<double>(M), n = 128.0 * n_tiles;
    const int k_tiles = static_cast<int>((K + 255) / 256);
    const double stage = longer(0.284, (16.384 + 0.128 * m + 4.096) * std::min(1.0 * n_tiles * ranks, 296.0) / 10417.0);
    return 2.06 + (ranks > 1 ? 0.98 : 0.0) + 0.0316 * m +
           longer((k_tiles + ranks - 1) / ranks * stage, (m + n) * static_cast<double>(K) * 9.0 / 16000.0 / 6264.0);
}
// Whether it is chosen, against the time of the best tile or pair kernel.  How far the kernel chosen is behind the fastest one on average,
// over 7300 random products of up to 128 tokens, prepared back to back / raw / behind the quantizer, %: up to 16 tokens 0.5 / 0.2 / 0.4, 17 to
// 32 0.8 / 0.3 / 0.8 (without the factor 1.0 / 0.3 / 1.2), 33 to 64 0.8 / 0.2 / 1.5 (with it 1.4 / 0.6 / 1.8), 65 to 128 0.6 / 0.2 / 1.5.  Always in
// this kernel, up to 16 tokens 3.4 to 4.4 / 3.6 to 4.8 / 1.7 to 2.8, 17 to 32 10 / 11 / 7.
static bool skinny_ahead(int64_t M, double skinny, double tiles) { return skinny < (M <= 32 ? 1.06 : 1.0) * tiles; }
// Its K ranges for so many weight tiles: none of them empty.
static int skinny_ranges(int64_t M, int n_tiles, int k_tiles, int sms, int forced) {
    const int bt = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
    const int ranks = nvfp4::gemm::skinny::choose_ranks(n_tiles, k_tiles, sms, forced, bt), per = (k_tiles + ranks - 1) / ranks;
    return (k_tiles + per - 1) / per;
}

// Kernel choice for one shape: host arithmetic only.  *path: 1 = 128x128 tiles, 2 = 128x256, 3 = pair 256x256,
// 4 = pair 256x192, 5 = skinny, 6 = 128x64, 7 = pair 256x128; *k_ranges: cluster size of the skinny kernel (1 for the others).
static void plan_gemm(int64_t M, int64_t N, int64_t K, int sms, int k_splits, int* path_out, int* ranges_out) {
    const int k_tiles = static_cast<int>((K + 255) / 256);
    const int n_tiles = static_cast<int>((N + 127) / 128);
    int best = 0;
    double best_time = 0.0;
    for (const TileCost& c : kTileCosts) {
        if (c.pair && (M <= 128 || N <= 128)) continue;   // half of the pair would have no rows: never the fastest
        const double t = tile_time(c, M, N, K, sms);
        if (best == 0 || t < best_time) {
            best = c.path;
            best_time = t;
        }
    }
    // Decode-sized batches: weight rows on the MMA's 128 rows, tokens on its N dimension, K ranges across a cluster.
    const bool decode = M <= kSkinnyMaxM && (g_gemm_force_path == 5 || (g_gemm_force_path == 0 && g_gemm_force_splits == 0));
    const int ranges = decode ? skinny_ranges(M, n_tiles, k_tiles, sms, g_gemm_force_path == 5 ? g_gemm_force_splits : 0) : 1;
    const double decode_time = decode ? skinny_time(M, K, n_tiles, ranges) : 0.0;
    if (decode && skinny_ahead(M, decode_time, best_time)) {
        best = 5;
        best_time = decode_time;
    }
    int path = g_gemm_force_path == 5 && !decode ? 0 : g_gemm_force_path;   // 0 = choose by shape
    // shapes of the measured table (on the GPU it was measured on) take the kernel that was fastest there
    if (path == 0 && k_splits == 1 && sms == 148) {
        path = table_path(M, N, K);
        if (path == 5 && (!decode || decode_time > kRowMargin * best_time)) path = 0;
        for (const TileCost& c : kTileCosts)
            if (c.path == path && tile_time(c, M, N, K, sms) > kRowMargin * best_time) path = 0;
    }
    if (path == 0) path = best;
    if (k_splits > 1 && path != 1 && path != 2 && path != 5 && path != 6) path = 1;
    *path_out = path;
    *ranges_out = path == 5 ? ranges : 1;
}

// Testing hook: the kernel nvfp4_gemm_launch would pick for this shape on a GPU with `sms` SMs (under the current
// force / tune settings).  No GPU is touched.
extern "C" int nvfp4_gemm_plan(int64_t M, int64_t N, int64_t K, int sms, int* path, int* k_ranges) {
    if (!path || !k_ranges) return NVFP4_ERR_NULL_POINTER;
    if (M <= 0 || N <= 0 || K <= 0 || (K % 64) != 0 || sms <= 0) return NVFP4_ERR_BAD_SHAPE;
    plan_gemm(M, N, K, sms, choose_k_splits(M, N, K), path, k_ranges);
    return NVFP4_OK;
}

// Fills one product's parameters; an NVFP4_ERR_* where an argument is wrong.  M, N > 0 are checked by the caller.
static int gemm_params(nvfp4::gemm::GemmParams& p, const uint8_t* a, const uint8_t* b, const uint8_t* sfa, const uint8_t* sfb,
                       const float* alpha, const float* alpha2, void* out_bf16, int64_t M, int64_t N, int64_t K) {
    using namespace nvfp4;
    if (M > 0x7fffff00LL || N > 0x7fffff00LL || K > 0x7fffff00LL) return NVFP4_ERR_TOO_LARGE;
    if (!a || !b || !sfa || !sfb || !alpha || !out_bf16) return NVFP4_ERR_NULL_POINTER;
    if (K == 0) return NVFP4_ERR_BAD_SHAPE;
    if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(b) & 15) ||
        (reinterpret_cast<uintptr_t>(sfa) & 15) || (reinterpret_cast<uintptr_t>(sfb) & 15) ||
        (reinterpret_cast<uintptr_t>(out_bf16) & 15) || (reinterpret_cast<uintptr_t>(alpha) & 3) ||
        (reinterpret_cast<uintptr_t>(alpha2) & 3))
        return NVFP4_ERR_MISALIGNED;
    p.a = a;
    p.b = b;
    p.sfa = sfa;
    p.sfb = sfb;
    p.alpha = alpha;
    p.alpha2 = alpha2;
    p.out = static_cast<__nv_bfloat16*>(out_bf16);
    p.M = static_cast<int>(M);
    p.N = static_cast<int>(N);
    p.K = static_cast<int>(K);
    p.sf_group_stride = round_up_i64(K / 16, 4) * 128;
    p.sfa_groups = static_cast<int>((M + 127) / 128);
    p.sfb_groups = static_cast<int>((N + 127) / 128);
    p.k_splits = choose_k_splits(M, N, K);
    const int k_tiles_total = static_cast<int>((K + 255) / 256);
    p.k_tiles_per_split = (k_tiles_total + p.k_splits - 1) / p.k_splits;
    p.k_splits = (k_tiles_total + p.k_tiles_per_split - 1) / p.k_tiles_per_split;   // no empty range
    p.k_rotate = g_gemm_force_rotate > 0 ? 1 : 0;
    p.partial = nullptr;
    // default: one band over all m-tiles (band sizes 1..16 measured within noise of it on B200)
    p.raster_group = g_gemm_raster_group > 0 ? g_gemm_raster_group : (1 << 20);
    return NVFP4_OK;
}

static int gemm_launch_impl(const uint8_t* a, const uint8_t* b, const uint8_t* sfa, const uint8_t* sfb,
                            const float* alpha, void* out_bf16, int64_t M, int64_t N, int64_t K, void* workspace,
                            size_t workspace_bytes, void* stream, const nvfp4::gemm::WeightHandle* wh,
                            const float* alpha2 = nullptr) {
    using namespace nvfp4;
    if (M < 0 || N < 0 || K < 0 || (K % 64) != 0) return NVFP4_ERR_BAD_SHAPE;
    if (M == 0 || N == 0) return NVFP4_OK;
    gemm::GemmParams p;
    const int bad = gemm_params(p, a, b, sfa, sfb, alpha, alpha2, out_bf16, M, N, K);
    if (bad != NVFP4_OK) return bad;
    p.partial = static_cast<float*>(workspace);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int sms = gemm::device_info().sms;
    int path = 0, ranges = 1;
    plan_gemm(M, N, K, sms, p.k_splits, &path, &ranges);
    if (path == 5) {
        const int forced = g_gemm_force_path == 5 ? g_gemm_force_splits : 0;
        if (M <= 16) return gemm::skinny::launch_skinny<16>(p, forced, s, wh);
        if (M <= 32) return gemm::skinny::launch_skinny<32>(p, forced, s, wh);
        if (M <= 64) return gemm::skinny::launch_skinny<64>(p, forced, s, wh);
        return gemm::skinny::launch_skinny<128>(p, forced, s, wh);
    }
    if (p.k_splits > 1) {
        const size_t need = static_cast<size_t>(p.k_splits) * static_cast<size_t>(M) * static_cast<size_t>(N) * sizeof(float);
        if (!workspace || workspace_bytes < need) return NVFP4_ERR_WORKSPACE;
        if (reinterpret_cast<uintptr_t>(workspace) & 15) return NVFP4_ERR_MISALIGNED;
    }
    if (path == 3) return gemm::pair::launch_pair<256>(p, s, wh);
    if (path == 4) return gemm::pair::launch_pair<192>(p, s, wh);
    if (path == 7) return gemm::pair::launch_pair<128>(p, s, wh);
    if (path == 2) return gemm::launch<256>(p, s, wh);
    if (path == 6) return gemm::launch<64>(p, s, wh);
    return gemm::launch<128>(p, s, wh);
}

// Kernel of a launch over several products (sorted by K), and its time: the tile costs of plan_gemm over the busiest worker's tiles.  0 =
// launch them one by one (K ranges are forced, or a kernel that has no form for lists).  How far the kernel chosen is behind the fastest
// one on average, back to back / behind the quantizer, %: layers up to 128 tokens 0.0 / 1.2, 129 to 256 0.2 / 0.3, more 0.3 / 0.2; q / k / v up to 128 0.0 /
// 1.0, more 0.3 / 1.0; gate / up 33 to 128 2.0 / 1.2, more 0.8 / 0.6.  (By the makespan at one time per stage, 128x64 tiles weighed 1.3 and 256x256
// pairs 1.1, which this replaces, back to back: layers 65 to 128 tokens 2.2, 129 to 256 2.4, more 0.6; q / k / v 2 to 13; gate / up 1 to 2.)
static int plan_list(const nvfp4::gemm::GemmParams* list, int n, int sms, double* time) {
    using namespace nvfp4::gemm;
    *time = 0.0;
    if (g_gemm_force_splits != 0) return 0;
    if (g_gemm_force_path != 0) return g_gemm_force_path == 5 ? 0 : g_gemm_force_path;
    const int64_t M = list[0].M;
    int path = 0;
    for (const TileCost& c : kTileCosts) {
        // one token tile: the second CTA of a pair has no rows (Llama-3-8B layer, 128 tokens: 24.8 us with 128x128 tiles, 29.0
        // with 256x192, 30.1 with 256x256)
        if (c.pair && M <= 128) continue;
        const int workers = c.pair ? sms / 2 : sms;
        GroupTable<kMaxItems> g;
        const int used = fill_group_table<kMaxItems>(g, list, n, static_cast<int>((M + c.rows - 1) / c.rows), c.cols, workers);
        if (used == 0) continue;
        double kbytes = 0.0, columns = 0.0, n_tiles = 0.0;
        bool ragged = false;
        for (int i = 0; i < n; ++i) {
            kbytes += streamed_kbytes(c, M, list[i].N, list[i].K);
            columns += list[i].N;
            n_tiles += static_cast<double>((static_cast<int64_t>(list[i].N) + c.cols - 1) / c.cols);
            ragged = ragged || list[i].N % 8 != 0;
        }
        const double cols = columns / n_tiles;
        const double span = list_makespan(g, list, stage_time(c, M, cols, used), c.later * stage_time(c, M, cols, workers),
                                          c.epilogue + (ragged ? c.ragged_tile : 0.0));
        const bool tail = g.n_classes == 1 && g.item[n - 1].tile_end > workers;
        const double t = launch_time(c, M, ragged) + longer(span, kbytes / c.memory) + (tail ? kTail : 0.0);
        if (path == 0 || t < *time) {
            *time = t;
            path = c.path;
        }
    }
    return path;
}

// Whether products of equal K go out in the decode-sized kernel: as one product of all their weight tiles, against one launch over
// the list.  Behind the faster of the two on average, by this / always in the decode-sized kernel / always as a list, over 4500 random
// groups back to back, %: q / k / v, up to 16 tokens 0.8 / 18 / 0.8, 17 to 32 0.2 / 29 / 0.2, 33 to 64 0.0 / 50 / 0.0; gate / up 0.7 / 3.2 / 5.4, 0.7 / 8.8 /
// 2.2, 2.3 / 22 / 0.7.
static bool group_in_skinny(const nvfp4::gemm::GemmParams* list, int n, int sms) {
    using namespace nvfp4::gemm;
    const int64_t M = list[0].M, K = list[0].K;
    if (M > kSkinnyMaxM) return false;
    if (g_gemm_force_path != 0 || g_gemm_force_splits != 0) return g_gemm_force_path == 5;
    if (n > kMaxItems) n = kMaxItems;
    double t = 0.0;
    if (plan_list(list, n, sms, &t) == 0) return true;
    int64_t n_tiles = 0;
    for (int i = 0; i < n; ++i) n_tiles += (static_cast<int64_t>(list[i].N) + 127) / 128;
    const int tiles = static_cast<int>(n_tiles);
    return skinny_ahead(M, skinny_time(M, K, tiles, skinny_ranges(M, tiles, static_cast<int>((K + 255) / 256), sms, 0)), t);
}

// Several products of equal M in as few launches as the tile kernels allow.
static int gemm_launch_list(nvfp4::gemm::GemmParams* list, const nvfp4::gemm::WeightHandle** wh, int n, void* stream) {
    using namespace nvfp4::gemm;
    // longest K first (insertion sort, stable): equal K end up next to one another
    for (int i = 1; i < n; ++i)
        for (int j = i; j > 0 && list[j].K > list[j - 1].K; --j) {
            std::swap(list[j], list[j - 1]);
            std::swap(wh[j], wh[j - 1]);
        }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    for (int first = 0; first < n; first += kMaxItems) {
        const int m = n - first < kMaxItems ? n - first : kMaxItems;
        const GemmParams* l = list + first;
        const WeightHandle* const* w = wh + first;
        double t = 0.0;
        const int path = m > 1 ? plan_list(l, m, device_info().sms, &t) : 0;
        int st = NVFP4_OK;
        if (path == 1) st = launch_list<128, kMaxItems>(l, w, m, s);
        else if (path == 2) st = launch_list<256, kMaxItems>(l, w, m, s);
        else if (path == 6) st = launch_list<64, kMaxItems>(l, w, m, s);
        else if (path == 7) st = pair::launch_pair_list<128, kMaxItems>(l, w, m, s);
        else if (path == 4) st = pair::launch_pair_list<192, kMaxItems>(l, w, m, s);
        else if (path == 3) st = pair::launch_pair_list<256, kMaxItems>(l, w, m, s);
        else
            for (int i = 0; i < m && st == NVFP4_OK; ++i)
                st = gemm_launch_impl(l[i].a, l[i].b, l[i].sfa, l[i].sfb, l[i].alpha, l[i].out, l[i].M, l[i].N, l[i].K, nullptr, 0, stream,
                                      w[i], l[i].alpha2);
        if (st != NVFP4_OK) return st;
    }
    return NVFP4_OK;
}

extern "C" int nvfp4_gemm_launch(const uint8_t* a, const uint8_t* b, const uint8_t* sfa, const uint8_t* sfb,
                                 const float* alpha, void* out_bf16, int64_t M, int64_t N, int64_t K, void* workspace,
                                 size_t workspace_bytes, void* stream) {
    return gemm_launch_impl(a, b, sfa, sfb, alpha, out_bf16, M, N, K, workspace, workspace_bytes, stream, nullptr);
}

// A weight matrix used by many GEMM calls (a model's linear layer): its tensor maps are encoded once here instead
// of on every launch.  The handle is a small host object; it refers to `b` / `sfb`, which the caller keeps alive and
// unchanged in place (their contents may change, their addresses and shape may not) until nvfp4_gemm_release.
extern "C" int nvfp4_gemm_prepare(const uint8_t* b, const uint8_t* sfb, int64_t N, int64_t K, void** handle_out) {
    using namespace nvfp4;
    if (!handle_out) return NVFP4_ERR_NULL_POINTER;
    *handle_out = nullptr;
    if (N <= 0 || K <= 0 || (K % 64) != 0) return NVFP4_ERR_BAD_SHAPE;
    if (N > 0x7fffff00LL || K > 0x7fffff00LL) return NVFP4_ERR_TOO_LARGE;
    if (!b || !sfb) return NVFP4_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(b) & 15) || (reinterpret_cast<uintptr_t>(sfb) & 15)) return NVFP4_ERR_MISALIGNED;
    gemm::WeightHandle* h = new (std::nothrow) gemm::WeightHandle();
    if (!h) return NVFP4_ERR_UNSUPPORTED;
    h->magic = gemm::kWeightMagic;
    h->device = gemm::device_info().device;
    h->b = b;
    h->sfb = sfb;
    h->N = N;
    h->K = K;
    int st = NVFP4_OK;
    for (int i = 0; i < 4 && st == NVFP4_OK; ++i) {
        const int height = gemm::WeightHandle::kHeights[i];
        st = gemm::make_operand_maps(&h->rows[i], &h->rest[i], b, N, K / 2, height);
        // the pair kernels' boxes are whole ones, whatever N is
        if (st == NVFP4_OK && !gemm::has_map(N, height, gemm::kWholeMap)) st = gemm::make_operand_map(&h->rows[i], b, N, K / 2, height);
    }
    if (st == NVFP4_OK)
        st = gemm::pair::make_scale_map(&h->scales, sfb, (N + 127) / 128, round_up_i64(K / 16, 4) * 128);
    if (st != NVFP4_OK) {
        delete h;
        return st;
    }
    *handle_out = h;
    return NVFP4_OK;
}

extern "C" int nvfp4_gemm_release(void* handle) {
    auto* h = static_cast<nvfp4::gemm::WeightHandle*>(handle);
    if (!h) return NVFP4_OK;
    if (h->magic != nvfp4::gemm::kWeightMagic) return NVFP4_ERR_BAD_ENUM;
    h->magic = 0;
    delete h;
    return NVFP4_OK;
}

// out[M, N] = alpha * dq(a) dq(weight)^T with a prepared weight: the same kernels and bits as nvfp4_gemm_launch.
extern "C" int nvfp4_gemm_launch_prepared(void* handle, const uint8_t* a, const uint8_t* sfa, const float* alpha,
                                          void* out_bf16, int64_t M, void* workspace, size_t workspace_bytes, void* stream) {
    auto* h = static_cast<const nvfp4::gemm::WeightHandle*>(handle);
    if (!h) return NVFP4_ERR_NULL_POINTER;
    if (h->magic != nvfp4::gemm::kWeightMagic) return NVFP4_ERR_BAD_ENUM;
    if (h->device != nvfp4::gemm::device_info().device) return NVFP4_ERR_UNSUPPORTED;   // prepared on another device
    return gemm_launch_impl(a, h->b, sfa, h->sfb, alpha, out_bf16, M, h->N, h->K, workspace, workspace_bytes, stream, h);
}

// Products of equal M in launches of the decode-sized kernel, kMaxGroup at a time.
static int launch_skinny_items(int M, const nvfp4::gemm::skinny::SkinnyItem* items, int n, cudaStream_t s) {
    using namespace nvfp4::gemm::skinny;
    const int forced = g_gemm_force_path == 5 ? g_gemm_force_splits : 0;
    for (int first = 0; first < n; first += kMaxGroup) {
        const int c = n - first < kMaxGroup ? n - first : kMaxGroup;
        const int st = M <= 16   ? launch_skinny_group<16>(M, items + first, c, forced, s)
                       : M <= 32 ? launch_skinny_group<32>(M, items + first, c, forced, s)
                       : M <= 64 ? launch_skinny_group<64>(M, items + first, c, forced, s)
                                 : launch_skinny_group<128>(M, items + first, c, forced, s);
        if (st != NVFP4_OK) return st;
    }
    return NVFP4_OK;
}

// One activation against several prepared weights of equal K, e.g. a layer's q / k / v projections:
//   outs[i][M, N_i] = alpha_w[i][0] * alpha_a[0] * dq(a) dq(weight_i)^T      (alpha_a may be NULL: factor 1)
// One launch per 8 weights: of the decode-sized kernel at batches and shapes it is chosen for, of a tile or pair kernel
// over the list of products otherwise.  Each output has the bits nvfp4_gemm_launch_prepared gives for the same weight with
// alpha = alpha_w[i][0] * alpha_a[0] whenever the K ranges per tile agree (they are chosen from the group's total tile count).
extern "C" int nvfp4_gemm_launch_grouped(void* const* handles, int n_weights, const uint8_t* a, const uint8_t* sfa,
                                         const float* alpha_a, const float* const* alpha_w, void* const* outs_bf16,
                                         int64_t M, void* stream) {
    using namespace nvfp4;
    if (n_weights < 0 || n_weights > 64) return NVFP4_ERR_BAD_RANGE;
    if (n_weights == 0) return NVFP4_OK;
    if (!handles || !alpha_w || !outs_bf16) return NVFP4_ERR_NULL_POINTER;
    if (M < 0) return NVFP4_ERR_BAD_SHAPE;
    const int device = gemm::device_info().device;
    int64_t K = 0, n_total = 0;
    for (int i = 0; i < n_weights; ++i) {
        auto* h = static_cast<const gemm::WeightHandle*>(handles[i]);
        if (!h || !alpha_w[i] || !outs_bf16[i]) return NVFP4_ERR_NULL_POINTER;
        if (h->magic != gemm::kWeightMagic) return NVFP4_ERR_BAD_ENUM;
        if (h->device != device) return NVFP4_ERR_UNSUPPORTED;
        if (i == 0) K = h->K;
        else if (h->K != K) return NVFP4_ERR_BAD_SHAPE;
        if ((reinterpret_cast<uintptr_t>(outs_bf16[i]) & 15) || (reinterpret_cast<uintptr_t>(alpha_w[i]) & 3))
            return NVFP4_ERR_MISALIGNED;
        n_total += (h->N + 127) / 128 * 128;
    }
    if (M == 0) return NVFP4_OK;
    if (!a || !sfa) return NVFP4_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(a) & 15) || (reinterpret_cast<uintptr_t>(sfa) & 15) ||
        (reinterpret_cast<uintptr_t>(alpha_a) & 3))
        return NVFP4_ERR_MISALIGNED;
    if (M > 0x7fffff00LL || n_total > 0x7fffff00LL) return NVFP4_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    gemm::GemmParams list[64];
    const gemm::WeightHandle* wh[64];
    for (int i = 0; i < n_weights; ++i) {
        wh[i] = static_cast<const gemm::WeightHandle*>(handles[i]);
        const int st = gemm_params(list[i], a, wh[i]->b, sfa, wh[i]->sfb, alpha_w[i], alpha_a, outs_bf16[i], M, wh[i]->N, K);
        if (st != NVFP4_OK) return st;
    }
    if (n_weights > 1 && group_in_skinny(list, n_weights, gemm::device_info().sms)) {
        gemm::skinny::SkinnyItem items[64];
        for (int i = 0; i < n_weights; ++i)
            items[i] = {a, sfa, alpha_a, wh[i]->b, wh[i]->sfb, alpha_w[i], static_cast<__nv_bfloat16*>(outs_bf16[i]), wh[i]->N, K, wh[i]};
        return launch_skinny_items(static_cast<int>(M), items, n_weights, s);
    }
    return gemm_launch_list(list, wh, n_weights, stream);
}

// Several products of equal M, each with its own activation: the matrices of a layer whose inputs are all at hand.
extern "C" int nvfp4_gemm_launch_multi(const nvfp4_gemm_item* items, int n_items, int64_t M, void* stream) {
    using namespace nvfp4;
    if (n_items < 0 || n_items > 64) return NVFP4_ERR_BAD_RANGE;
    if (n_items == 0) return NVFP4_OK;
    if (!items) return NVFP4_ERR_NULL_POINTER;
    if (M < 0) return NVFP4_ERR_BAD_SHAPE;
    const int device = gemm::device_info().device;
    gemm::GemmParams list[64];
    const gemm::WeightHandle* wh[64];
    for (int i = 0; i < n_items; ++i) {
        const nvfp4_gemm_item& it = items[i];
        wh[i] = static_cast<const gemm::WeightHandle*>(it.weight);
        if (!wh[i]) return NVFP4_ERR_NULL_POINTER;
        if (wh[i]->magic != gemm::kWeightMagic) return NVFP4_ERR_BAD_ENUM;
        if (wh[i]->device != device) return NVFP4_ERR_UNSUPPORTED;
        if (M == 0) continue;
        const int st = gemm_params(list[i], it.a, wh[i]->b, it.sfa, wh[i]->sfb, it.alpha_w, it.alpha_a, it.out_bf16, M, wh[i]->N, wh[i]->K);
        if (st != NVFP4_OK) return st;
    }
    if (M == 0) return NVFP4_OK;
    // With different K, beyond 32 tokens (where the decode-sized kernel's token tile doubles and two CTAs an SM have room for) one
    // launch of a tile kernel over the list takes over.  A layer's seven products, us, tile kernel / decode-sized kernel, hidden
    // 4096, K / V 1024, FFN 14336: 24 tokens 23.2 / 23.2, 32 23.2 / 23.5; 2048 / 512 / 8192: 10.6 / 8.8, 10.5 / 9.0; over 730 random layers of 17
    // to 32 tokens the tile kernel is 8.5 % behind, over 1470 of 33 to 64 the decode-sized one 21 %.
    bool mixed = false;
    for (int i = 1; i < n_items; ++i) mixed = mixed || list[i].K != list[0].K;
    const bool forced = g_gemm_force_path != 0 || g_gemm_force_splits != 0;
    const bool decode = mixed || forced ? M <= (mixed ? 32 : 64) && (g_gemm_force_path == 0 || g_gemm_force_path == 5)
                                        : group_in_skinny(list, n_items, gemm::device_info().sms);
    if (n_items == 1 || !decode) return gemm_launch_list(list, wh, n_items, stream);
    // decode-sized: one launch of the decode-sized kernel per 8 products, longest K first
    gemm::skinny::SkinnyItem s_items[64];
    for (int i = 0; i < n_items; ++i) {
        const gemm::GemmParams& p = list[i];
        const gemm::skinny::SkinnyItem it = {p.a, p.sfa, p.alpha2, p.b, p.sfb, p.alpha, p.out, p.N, p.K, wh[i]};
        int j = i;
        for (; j > 0 && s_items[j - 1].K < it.K; --j) s_items[j] = s_items[j - 1];
        s_items[j] = it;
    }
    return launch_skinny_items(static_cast<int>(M), s_items, n_items, static_cast<cudaStream_t>(stream));
}

extern "C" int nvfp4_gemm_last_status(void* stream, uint32_t* status_host) {
    if (!status_host) return NVFP4_ERR_NULL_POINTER;
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return static_cast<int>(e);
    uint32_t zero = 0;
    e = cudaMemcpyFromSymbol(status_host, nvfp4::gemm::g_gemm_status, sizeof(uint32_t));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (*status_host != 0) e = cudaMemcpyToSymbol(nvfp4::gemm::g_gemm_status, &zero, sizeof(uint32_t));
    return static_cast<int>(e);
}


// Tensor-pipe rate probe: `stages` x 4 block-scaled FP4 MMAs per SM on operands resident in shared memory; time the
// launch with events on `stream`.  pair == 0: one CTA per SM, M = 128, N = 256, K = 64 per instruction; pair != 0:
// a CTA pair (cta_group::2) per two SMs, M = 256, N = 256, K = 64 per instruction -- the form the large-shape
// kernels use; pair == 2 (testing hook): the pair == 0 kernel with its last tcgen05.commit left out, so that its
// final wait ends at the wait limit and the status word is set (nothing faults, TMEM is freed).  Work done either way: *sms_out * stages * 4 * 2 * 128 * 256 * 64 flop (*sms_out = SMs used).
// Bounded: stages <= 1 << 20.
extern "C" int nvfp4_gemm_peak_probe(int stages, int pair_mode, int* sms_out, void* stream) {
    using namespace nvfp4::gemm;
    if (stages <= 0 || stages > (1 << 20)) return NVFP4_ERR_BAD_RANGE;
    if (pair_mode < 0 || pair_mode > 2) return NVFP4_ERR_BAD_ENUM;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return static_cast<int>(e);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (pair_mode != 1) {
        e = cudaFuncSetAttribute(peak::fp4_peak_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmDynSmemBytes);
        if (e != cudaSuccess) return static_cast<int>(e);
        if (sms_out) *sms_out = sms;
        // whole SM: it takes all TMEM columns
        peak::fp4_peak_kernel<<<sms, peak::kPeakThreads, kGemmDynSmemBytes, s>>>(stages, pair_mode == 2 ? 1 : 0);
        return static_cast<int>(cudaGetLastError());
    }
    e = cudaFuncSetAttribute(peak::fp4_peak_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGemmDynSmemBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    const int ctas = sms / 2 * 2;
    if (sms_out) *sms_out = ctas;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(peak::kPeakThreads, 1, 1);
    cfg.dynamicSmemBytes = kGemmDynSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return static_cast<int>(cudaLaunchKernelEx(&cfg, peak::fp4_peak_pair_kernel, stages));
}

// Testing hook: the limit (nanoseconds, 1 us .. 10 s) after which a wait inside the GEMM kernels of the current device
// gives up and records a status word; 0 restores the default of 2 s.  Synchronous (it copies to a device symbol).
extern "C" int nvfp4_gemm_set_wait_limit_ns(uint64_t ns) {
    if (ns == 0) ns = nvfp4::gemm::kWaitLimitNs;
    if (ns < 1000ull || ns > 10000000000ull) return NVFP4_ERR_BAD_RANGE;
    return static_cast<int>(cudaMemcpyToSymbol(nvfp4::gemm::g_gemm_wait_limit_ns, &ns, sizeof(ns)));
}

#ifdef NVFP4_GEMM_TRACE
// Debugging builds only: device buffer of 64 counters the kernels add their progress marks to (NULL = off).
extern "C" int nvfp4_gemm_set_trace(uint32_t* counters) {
    return static_cast<int>(cudaMemcpyToSymbol(nvfp4::gemm::g_gemm_trace, &counters, sizeof(counters)));
}
#endif
