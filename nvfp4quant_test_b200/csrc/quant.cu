// NVFP4 quantizer for sm_100a: ScaleSweep (unweighted and importance-weighted)
// and the amax baseline, one kernel family.
//
// Behaviour follows efsotr/nvfp4quant_test:
//   kernels/kernel_ScaleSweep_MSE.py:271-377  (unweighted sweep, RNE base, -3..+7)
//   kernels/kernel_ScaleSweep.py:290-416      (weighted sweep, floor base, -8..+7)
// and, for the amax variant, the NVFP4 recipe of vllm's scaled_fp4_quant.
//
// Bit-exactness rules kept here: fp32 everywhere with explicit round-to-nearest
// operations (no contraction), `1/scale` through div.full.f32, squared errors
// accumulated as one serial FMA chain over elements 0..15 (unweighted) or as the
// fixed pairwise tree (weighted), candidates visited in ascending raw order with
// a strict `<` (or in descending order with `<=`), so the lowest raw code wins ties.
// The weighted sweep leaves out candidates that provably cannot win (sweep_weighted).
//
// Mapping: one 16-element block per thread; a warp covers 32 consecutive blocks
// of one row (1 KiB of bf16).  Three interchangeable loop bodies give identical
// bytes: the scalar transcription (1), one candidate per trip with packed
// multiplies and the mixed-precision subtract (2), and the default: two
// candidates per trip whose FMA chains share one f32x2 instruction (each lane of
// a packed instruction is an independent IEEE operation).
//
// Bodies 3 and 5 to 9 are the default loop over different grids: 3, 5 and 9 number the slots of the real rows through (5 in
// CTAs of 256 threads with the loop rolled, for large ragged unweighted 16-bit tensors; 9 in small CTAs, for a few tokens), 6 the
// warps of rows, 7 and 8 have a two-dimensional grid, a row's chunks by a row's CTAs (8 for rows of whole chunks: sweeps of tensors
// without any padding, without predicates, and amax).
//
// Body 4 is the default loop with the tensor-wide global scale (helper.py:96-100: amax / (6 * fp8_max) and its reciprocal)
// computed inside the same launch: every thread keeps its block in registers, the CTAs combine their maxima
// through a scratch word and wait for one another (cooperative launch: all CTAs are resident; the wait is bounded
// by the global timer), then the sweep runs as usual.  x is read from HBM once and one launch replaces two; the
// tensor must fit the resident grid (about 3 M elements on a B200).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace nvfp4 {
namespace {

constexpr int kThreads = 256;
// The sweeps' bodies 3, 7 and 8 run in CTAs of 128 threads with up to 72 registers (7 CTAs, 28 warps per SM).  A large
// sweep takes the same time with anything from 20 to 48 warps per SM (8192 x 8192, us, unweighted / weighted with all its candidates: 256 threads
// at 40 registers 110.4 / 237, at 64 114.4 / 191; 128 threads at 96 registers 110.7 / 193, at 72 110.5 / 190.5): instruction
// issue (79 % of the active cycles unweighted, 73 % weighted) and the FMA and ALU pipes (61 and 63 %, 72 and 48 %) bound it together,
// not latency.  Below a few hundred tokens latency does, and there more registers
// (independent work in flight per warp) and smaller CTAs (an even spread over the SMs) decide: 256 x 8192 7.2 -> 4.9 us
// unweighted and 9.1 -> 7.9 weighted against 256 threads at 40 and 64 registers, 128 x 8192 5.4 -> 3.3 and 7.0 -> 5.1.
constexpr int kSweepThreads = 128;
constexpr int kSweepMinBlocks = 7;
// Body 9 (few tokens): CTAs of 64 threads with up to 128 registers.  A warp's sweep is ~750 instructions; the smallest CTAs
// spread the blocks over the most SMs.
constexpr int kSmallThreads = 64;
// Real 16-element blocks up to which body 9 is the default, for rows of whole chunks (against body 7) and for others
// (against body 3).  Measured in a chain of launches (us, body 9 / the other): whole chunks, unweighted 4 x 8192 1.92 / 2.03,
// 32 x 8192 2.10 / 3.23, 96 x 4096 2.48 / 3.00, 40 x 8192 3.28 / 3.06, 128 x 8192 3.52 / 3.14; weighted 32 x 8192 2.90 / 5.23,
// 40 x 8192 3.52 / 4.73, 48 x 8192 5.69 / 4.91, 128 x 8192 6.30 / 5.33.  Ragged rows, unweighted 77 x 5104 2.86 / 3.69, 300 x
// 5104 4.85 / 5.05, 200 x 10000 5.52 / 5.09; weighted 150 x 5104 6.29 / 7.98, 500 x 10000 17.47 / 17.60.  (Against body 6 or 7
// on ragged rows the weighted line is the unweighted one: 120000 blocks 8.5 / 8.5, 250000 15.2 / 14.7.)
constexpr int64_t kSmallBlocks = 24576;
constexpr int64_t kSmallBlocksRagged = 98304;
constexpr int64_t kSmallBlocksRaggedWeighted = 327680;
// Real blocks from which body 5 takes the place of 3 (unweighted, 16-bit), us bodies 3 / 5: 300000 blocks, 2325 x 2064 10.69 / 10.94;
// 400000, 1111 x 5760 13.76 / 13.50; 1500000, 7575 x 3168 45.99 / 44.97; 3700000, 8191 x 7216 110.1 / 107.5.  fp32 gains nothing.
constexpr int64_t kLargeBlocksRagged = 393216;
__host__ __device__ constexpr int block_threads(int variant, int impl) {
    return impl == 9 ? kSmallThreads : (variant != NVFP4_VARIANT_AMAX && (impl == 3 || impl == 6 || impl == 7 || impl == 8 || impl == 10)) ? kSweepThreads : kThreads;
}
// The reference's windows: 11 candidates, unweighted; 16 from eight below the base, weighted.  The unrolled sweeps are compiled for these.
constexpr int kWindow = 11, kWindowWeighted = 16, kWeightedLower = -8;
__host__ __device__ constexpr bool own_window(int variant, int lower, int ncand) {
    return variant == NVFP4_VARIANT_WEIGHTED ? lower == kWeightedLower && ncand == kWindowWeighted : ncand == kWindow;
}
constexpr int min_blocks(int variant, int impl) {
    if (impl == 9) return 8;
    if (impl == 10) return 4;
    if (block_threads(variant, impl) == kSweepThreads) return kSweepMinBlocks;
    return variant == NVFP4_VARIANT_WEIGHTED ? 4 : 5;
}

constexpr int kMaxChain = 4;   // tensors per launch of the chain

struct QuantParams {
    const void* x;
    const float* importance;
    const float* gs_inv;
    uint8_t* codes;
    uint8_t* scales;
    int64_t m, n;
    int64_t bin, bout;      // 16-element blocks per input / output row
    int64_t width, rows;    // slot grid: scale columns / rows that get written
    int64_t k_pad;          // padded scale columns (swizzled layout)
    int64_t total;          // rows * width
    uint32_t div_mul, div_shift;  // division by width: see set_row_div
    int lower, ncand;
    int swizzled;
    int early;              // != 0: kernels behind this one may be scheduled while it runs (see the kernel's first lines)
    // fused global-scale variant only
    float fp8_max;
    float* gs_out;          // [2]: global scale, its reciprocal
    uint32_t* fused_scratch;  // [4]: running maximum, arrivals, readers, unused; zero between calls
};

// n / d for n < 2^31, as (n * ceil(2^(32 + shift) / d)) >> (32 + shift) with 2^shift < d <= 2^(shift + 1): the rounding of the
// multiplier is e / d with e < d and adds n * e / (d * 2^(32 + shift)) < n / 2^(32 + shift) to the quotient, less than the 1 / d that
// its fraction is at least away from the next integer because n * e < 2^31 * 2^(shift + 1).  d: the width, or the warps of a row (body 6).
inline void set_row_div(QuantParams& p, int64_t d) {
    p.div_mul = p.div_shift = 0;
    if (d <= 1 || d > 0x7fffffffLL) return;
    while ((2ll << p.div_shift) < d) ++p.div_shift;
    p.div_mul = static_cast<uint32_t>(((1ull << (32 + p.div_shift)) + d - 1) / d);
}
__device__ __forceinline__ uint32_t row_div(const QuantParams& p, uint32_t n) {
    return p.div_mul == 0 ? n : __umulhi(n, p.div_mul) >> p.div_shift;
}

__device__ uint32_t g_quant_status;   // 0 = ok; 1 = the grid-wide wait of the fused kernel gave up
constexpr uint64_t kFusedWaitLimitNs = 2000000000ull;
__device__ uint64_t g_fused_wait_limit_ns = kFusedWaitLimitNs;   // settable from the host (nvfp4_quant_fused_set_wait_limit_ns)

template <int DT>
__device__ __forceinline__ void load16(const void* base, int64_t elem, float v[16]);

template <>
__device__ __forceinline__ void load16<NVFP4_DT_BF16>(const void* base, int64_t elem, float v[16]) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + elem);
    uint4 a = __ldg(p), b = __ldg(p + 1);
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}

template <>
__device__ __forceinline__ void load16<NVFP4_DT_F16>(const void* base, int64_t elem, float v[16]) {
    const uint4* p = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(base) + elem);
    uint4 a = __ldg(p), b = __ldg(p + 1);
    uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
        v[2 * i] = f.x;
        v[2 * i + 1] = f.y;
    }
}

template <>
__device__ __forceinline__ void load16<NVFP4_DT_F32>(const void* base, int64_t elem, float v[16]) {
    const float4* p = reinterpret_cast<const float4*>(static_cast<const float*>(base) + elem);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float4 f = __ldg(p + i);
        v[4 * i] = f.x;
        v[4 * i + 1] = f.y;
        v[4 * i + 2] = f.z;
        v[4 * i + 3] = f.w;
    }
}

__device__ __forceinline__ float max_abs16(const float v[16]) {
    float m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = fmaxf(fabsf(v[2 * i]), fabsf(v[2 * i + 1]));
    return fmaxf(fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])), fmaxf(fmaxf(m[4], m[5]), fmaxf(m[6], m[7])));
}

// Candidate table: entry k describes raw code table_raw(k), so a sweep that starts at tab[first + kTabPad] reads consecutive
// entries and needs no per-candidate clamping.  .x = .y = 1/s (div.full.f32), .z = s*s, .w = s*s of entry k + 1: a trip's two
// factors are a register pair as they are loaded.
constexpr int kTabPad = 64;
constexpr int kTabSize = 256;
__device__ __forceinline__ uint32_t table_raw(int k) { return static_cast<uint32_t>(min(max(k - kTabPad, 1), 126)); }

// ---- scalar transcription: one candidate at a time --------------------------------------
template <bool WEIGHTED>
__device__ __forceinline__ uint32_t sweep_scalar(const float v[16], const float w[16], int first_idx, int ncand,
                                                 const float4* tab) {
    float best = __int_as_float(0x7f800000);
    uint32_t best_raw = 0;
#pragma unroll 1
    for (int i = 0; i < ncand; ++i) {
        const float4 e4 = tab[first_idx + i];
        const float2 e = make_float2(e4.x, e4.z);
        const uint32_t raw = table_raw(first_idx + i);
        float err;
        if (!WEIGHTED) {
            float acc = 0.0f;
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float x0 = __fmul_rn(v[2 * p], e.x), x1 = __fmul_rn(v[2 * p + 1], e.x), q0, q1;
                e2m1_round_pair(x0, x1, q0, q1);
                float d0 = __fsub_rn(q0, x0), d1 = __fsub_rn(q1, x1);
                acc = __fmaf_rn(d0, d0, acc);  // fma(d, d, +0) == mul.rn(d, d) for the first term
                acc = __fmaf_rn(d1, d1, acc);
            }
            err = __fmul_rn(acc, e.y);
        } else {
            float pe[8];
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float x0 = __fmul_rn(v[2 * p], e.x), x1 = __fmul_rn(v[2 * p + 1], e.x), q0, q1;
                e2m1_round_pair(x0, x1, q0, q1);
                float d0 = __fsub_rn(q0, x0), d1 = __fsub_rn(q1, x1);
                float a = __fmul_rn(__fmul_rn(d0, d0), w[2 * p]);
                pe[p] = __fmaf_rn(__fmul_rn(d1, d1), w[2 * p + 1], a);
            }
            float t = __fadd_rn(__fadd_rn(__fadd_rn(pe[0], pe[1]), __fadd_rn(pe[2], pe[3])),
                                __fadd_rn(__fadd_rn(pe[4], pe[5]), __fadd_rn(pe[6], pe[7])));
            err = __fmul_rn(t, e.y);
        }
        if (err < best) {
            best = err;
            best_raw = raw;
        }
    }
    return best_raw;
}

// ---- paired: two candidates per loop trip; element pairs share the multiply and both
// conversions, the difference uses the mixed-precision subtract (f16 grid value minus fp32 x,
// one full-rate instruction, exact like cvt + sub), and the two candidates' accumulations
// share one f32x2 instruction -------------------------------------------------------------
__device__ __forceinline__ void e2m1_diff_pair(uint64_t x2, float& d0, float& d1) {
    asm("{ .reg .b8 b; .reg .b32 h; .reg .b16 lo, hi; .reg .f32 x0, x1;\n"
        "  mov.b64 {x0, x1}, %2;\n"
        "  cvt.rn.satfinite.e2m1x2.f32 b, x1, x0;\n"
        "  cvt.rn.f16x2.e2m1x2 h, b;\n"
        "  mov.b32 {lo, hi}, h;\n"
        "  sub.rn.f32.f16 %0, lo, x0;\n"
        "  sub.rn.f32.f16 %1, hi, x1; }"
        : "=f"(d0), "=f"(d1)
        : "l"(x2));
}

// Both lanes' sums of a trip: candidate a in the low lane, b in the high lane.
__device__ __forceinline__ uint64_t trip_sum(const uint64_t vp[8], uint64_t inv_a, uint64_t inv_b) {
    uint64_t acc2 = 0;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        float a0, a1, b0, b1;
        e2m1_diff_pair(mul_f32x2(vp[p], inv_a), a0, a1);
        e2m1_diff_pair(mul_f32x2(vp[p], inv_b), b0, b1);
        const uint64_t d0 = pack_f32x2(a0, b0), d1 = pack_f32x2(a1, b1);
        acc2 = fma_f32x2(d0, d0, acc2);
        acc2 = fma_f32x2(d1, d1, acc2);
    }
    return acc2;
}
__device__ __forceinline__ uint64_t trip_sum_weighted(const uint64_t vp[8], const float w[16], uint64_t inv_a, uint64_t inv_b) {
    uint64_t pe[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        float a0, a1, b0, b1;
        e2m1_diff_pair(mul_f32x2(vp[p], inv_a), a0, a1);
        e2m1_diff_pair(mul_f32x2(vp[p], inv_b), b0, b1);
        const uint64_t d0 = pack_f32x2(a0, b0), d1 = pack_f32x2(a1, b1);
        const uint64_t t = mul_f32x2(mul_f32x2(d0, d0), pack_f32x2(w[2 * p], w[2 * p]));
        pe[p] = fma_f32x2(mul_f32x2(d1, d1), pack_f32x2(w[2 * p + 1], w[2 * p + 1]), t);
    }
    return add_f32x2(add_f32x2(add_f32x2(pe[0], pe[1]), add_f32x2(pe[2], pe[3])),
                     add_f32x2(add_f32x2(pe[4], pe[5]), add_f32x2(pe[6], pe[7])));
}
// One candidate alone (an odd count's last one).
template <bool WEIGHTED>
__device__ __forceinline__ float single_sum(const uint64_t vp[8], const float w[16], uint64_t inv2) {
    if (!WEIGHTED) {
        float acc = 0.0f;
#pragma unroll
        for (int p = 0; p < 8; ++p) {
            float d0, d1;
            e2m1_diff_pair(mul_f32x2(vp[p], inv2), d0, d1);
            acc = __fmaf_rn(d0, d0, acc);
            acc = __fmaf_rn(d1, d1, acc);
        }
        return acc;
    }
    float pe[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        float d0, d1;
        e2m1_diff_pair(mul_f32x2(vp[p], inv2), d0, d1);
        const float a = __fmul_rn(__fmul_rn(d0, d0), w[2 * p]);
        pe[p] = __fmaf_rn(__fmul_rn(d1, d1), w[2 * p + 1], a);
    }
    return __fadd_rn(__fadd_rn(__fadd_rn(pe[0], pe[1]), __fadd_rn(pe[2], pe[3])),
                     __fadd_rn(__fadd_rn(pe[4], pe[5]), __fadd_rn(pe[6], pe[7])));
}

// NC > 0: the candidate count is the compile-time constant NC and the trips are unrolled (the table index and the
// loop control leave the instruction stream); NC = 0: `ncand` at run time, one rolled loop.
// A trip keeps the least error so far (one three-way minimum, which passes over NaN), its own index if that fell, and its first
// candidate's error, by which the winner of the pair is told at the end.
// (Two compares, two error and two code selects per trip before, and the factors packed: us, 8192 x 8192 111.2 -> 109.7, 1024 x 8192
// 15.74 -> 15.50, 3000 x 5104 28.82 -> 28.23.)
template <int NC = 0>
__device__ __forceinline__ uint32_t sweep_paired(const float v[16], int first_idx, int ncand_rt, const float4* tab) {
    const int ncand = NC > 0 ? NC : ncand_rt;
    uint64_t vp[8];  // (v[2p], v[2p+1])
#pragma unroll
    for (int p = 0; p < 8; ++p) vp[p] = pack_f32x2(v[2 * p], v[2 * p + 1]);
    float best = __int_as_float(0x7f800000), err_first = 0.0f;
    int pos = -2;   // of the best trip's first candidate; below 0: no error was comparable
    auto trip = [&](int i) {
        const float4 ea = tab[first_idx + i];
        const float2 eb = *reinterpret_cast<const float2*>(tab + first_idx + i + 1);
        float err_a, err_b;
        unpack_f32x2(mul_f32x2(trip_sum(vp, pack_f32x2(ea.x, ea.y), pack_f32x2(eb.x, eb.y)), pack_f32x2(ea.z, ea.w)), err_a, err_b);
        const float least = fminf(fminf(best, err_a), err_b);
        if (least < best) {
            pos = i;
            err_first = err_a;
        }
        best = least;
    };
    if (NC > 0) {
#pragma unroll
        for (int i = 0; i + 1 < NC; i += 2) trip(i);
    } else {
#pragma unroll 1
        for (int i = 0; i + 1 < ncand; i += 2) trip(i);
    }
    pos += err_first == best ? 0 : 1;
    if (ncand & 1) {
        const float4 e4 = tab[first_idx + ncand - 1];
        const float err = __fmul_rn(single_sum<false>(vp, nullptr, pack_f32x2(e4.x, e4.y)), e4.z);
        if (err < best) pos = ncand - 1;
    }
    return pos < 0 ? 0u : table_raw(first_idx + pos);
}

// Lanes of a warp that may still need smaller scales at the first test: by the bound with the least weight of each block, for the
// bound with the largest element's own weight to be tried; by that one, for the tests to go on.
constexpr int kLookupLanes = 28, kWorthLanes = 10;

// The weighted sweep, from the largest scale down: `<=` against a finite start chooses what `<` against infinity chooses
// upwards, the lowest raw code of the least comparable error.
//
// The window reaches eight codes below the floor code of amax / 6, where the block's largest element saturates (6 s < amax) and
// its error alone soon exceeds what a larger scale gave.  A candidate's error is at least that of one saturated element: with
// y = RN(amax * (1/s)) >= 6, d = RN(6 - y) is that element's difference, every operation of the tree is monotone in d^2 for
// weights >= 0, and so err >= RN(RN(RN(d * d) * w) * s^2), in the kernel's own roundings, for the element's weight or any smaller
// one.  Strictly above the least error so far, the candidate cannot win (equality is kept).  Neither can a smaller scale: amax -
// 6 s grows by at least 6 s / 16 >= y s / 2731 for y <= 1024, far more than the roundings, while the product with s^2 stays normal
// (least error >= 1e-30).  A lane whose candidates have come down to raw code 1 has seen the rest.  When all lanes of a warp are
// done, it stops.  Where the weights of a block lie within a few per cent of one another, ten of the sixteen candidates are evaluated;
// with spread weights the largest element's own weight takes the place of the least one, and a warp whose lanes have too many
// candidates left (see the constants above) tests no further.  Importances that differ by a factor of five within a block and more
// gain nothing and pay for the first test.  us, sixteen candidates / this, 8192 x 8192: weights within 3 % 191.1 / 134.9; log-normal ones,
// sigma 0.3 191.3 / 145.0, 0.6 191.5 / 159.8, 1 191.6 / 188.0, 1.5 191.7 / 196.5, 3 191.6 / 196.5; 1 % of the channels a hundred times the
// others' 191.4 / 156.9, one in sixteen 191.6 / 190.1; 3000 x 5104, within 3 % 46.5 / 34.6, sigma 2 46.5 / 47.9, 1024 x 4096 14.1 / 10.6, 14.1 /
// 14.3.  (With the trips that are left in a loop where the tests do not pay, and the largest element always looked up: sigma 1 189.5,
// sigma 2 204.4, one channel in sixteen 194.2.  Without any test, the trips unrolled: 191.9.)
template <int NC = 0>
__device__ __forceinline__ uint32_t sweep_weighted(const float v[16], const float w[16], float w_min, float amax, int first_idx, int ncand_rt,
                                                   int lower_rt, const float4* tab) {
    const int ncand = NC > 0 ? NC : ncand_rt;
    const int lower = NC > 0 ? kWeightedLower : lower_rt;
    uint64_t vp[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) vp[p] = pack_f32x2(v[2 * p], v[2 * p + 1]);
    float best = __int_as_float(0x7f7fffff), err_first = 0.0f;
    int pos = -2;
    auto trip = [&](int i) {
        const float4 ea = tab[first_idx + i];
        const float2 eb = *reinterpret_cast<const float2*>(tab + first_idx + i + 1);
        float err_a, err_b;
        unpack_f32x2(mul_f32x2(trip_sum_weighted(vp, w, pack_f32x2(ea.x, ea.y), pack_f32x2(eb.x, eb.y)), pack_f32x2(ea.z, ea.w)), err_a, err_b);
        const float least = fminf(err_a, err_b);
        if (least <= best) {
            best = least;
            pos = i;
            err_first = err_a;
        }
    };
    // Down to two codes below the base every trip is needed by some lane of nearly every warp, and is not tested.
    constexpr int kTested = -3 - kWeightedLower;
    constexpr int kFirstTested = kTested - 1 - ((NC + kTested + 1) & 1);   // counts down from NC - 2 in twos
    const int tested = NC > 0 ? kTested : min(-3 - lower, ncand - 3);
    int i = ncand - 2;
    if (NC > 0) {
#pragma unroll 2
        for (; i >= tested; i -= 2) trip(i);
    } else {
#pragma unroll 1
        for (; i >= 0 && i >= tested; i -= 2) trip(i);
    }
    float w_bound = w_min;
    bool first = true;
#pragma unroll 1
    for (; i >= 0; i -= 2) {
        const float4 e = tab[first_idx + i + 1];   // the trip's larger scale
        const float y = __fmul_rn(amax, e.x), d = __fsub_rn(6.0f, y), dd = __fmul_rn(d, d);
        const bool last_code = first_idx + i + 2 <= kTabPad + 1;
        const bool bounded = w_min >= 0.0f && y >= 6.0f && y <= 1024.0f && best >= 1e-30f;
        auto undecided = [&] { return __ballot_sync(0xffffffffu, !(last_code || (bounded && __fmul_rn(__fmul_rn(dd, w_bound), e.z) > best))); };
        uint32_t lanes = undecided();
        if (lanes == 0) break;
        if (first) {
            first = false;
            if (__popc(lanes) <= kLookupLanes) {
#pragma unroll
                for (int j = 0; j < 16; ++j) w_bound = fabsf(v[j]) == amax ? w[j] : w_bound;
                lanes = undecided();
                if (lanes == 0) break;
            }
            if (__popc(lanes) > kWorthLanes) {   // the rest untested
                if (NC > 0) {
#pragma unroll
                    for (int k = kFirstTested; k >= 0; k -= 2) trip(k);
                    i = NC & 1 ? -1 : -2;
                } else {
#pragma unroll 1
                    for (; i >= 0; i -= 2) trip(i);
                }
                break;
            }
        }
        trip(i);
    }
    pos += err_first == best ? 0 : 1;
    if ((ncand & 1) && i == -1) {
        const float4 e4 = tab[first_idx];
        const float err = __fmul_rn(single_sum<true>(vp, w, pack_f32x2(e4.x, e4.y)), e4.z);
        if (err <= best) pos = 0;
    }
    return pos < 0 ? 0u : table_raw(first_idx + pos);
}

// ---- one candidate per trip, element pairs share the multiply, scalar FMA chain ----------------
template <bool WEIGHTED>
__device__ __forceinline__ uint32_t sweep_single(const float v[16], const float w[16], int first_idx, int ncand,
                                                 const float4* tab) {
    uint64_t vp[8];
#pragma unroll
    for (int p = 0; p < 8; ++p) vp[p] = pack_f32x2(v[2 * p], v[2 * p + 1]);
    float best = __int_as_float(0x7f800000);
    uint32_t best_raw = 0;
#pragma unroll 1
    for (int i = 0; i < ncand; ++i) {
        const float4 e4 = tab[first_idx + i];
        const float2 e = make_float2(e4.x, e4.z);
        const uint32_t raw = table_raw(first_idx + i);
        const uint64_t inv2 = pack_f32x2(e4.x, e4.y);
        float err;
        if (!WEIGHTED) {
            float acc = 0.0f;
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float d0, d1;
                e2m1_diff_pair(mul_f32x2(vp[p], inv2), d0, d1);
                acc = __fmaf_rn(d0, d0, acc);
                acc = __fmaf_rn(d1, d1, acc);
            }
            err = __fmul_rn(acc, e.y);
        } else {
            float pe[8];
#pragma unroll
            for (int p = 0; p < 8; ++p) {
                float d0, d1;
                e2m1_diff_pair(mul_f32x2(vp[p], inv2), d0, d1);
                const float a = __fmul_rn(__fmul_rn(d0, d0), w[2 * p]);
                pe[p] = __fmaf_rn(__fmul_rn(d1, d1), w[2 * p + 1], a);
            }
            const float t = __fadd_rn(__fadd_rn(__fadd_rn(pe[0], pe[1]), __fadd_rn(pe[2], pe[3])),
                                      __fadd_rn(__fadd_rn(pe[4], pe[5]), __fadd_rn(pe[6], pe[7])));
            err = __fmul_rn(t, e.y);
        }
        if (err < best) {
            best = err;
            best_raw = raw;
        }
    }
    return best_raw;
}

// Largest magnitude of `nvec` 16-byte vectors as an fp32 bit pattern, by the whole CTA (what global_scale_kernel computes).
template <int DT, int T>
__device__ __forceinline__ uint32_t cta_amax_bits(const uint4* x, uint32_t nvec) {
    constexpr int kBatch = 16;   // loads in flight per thread
    uint32_t acc = 0;
    for (uint32_t i = threadIdx.x; i < nvec; i += kBatch * T) {
        uint4 q[kBatch];
#pragma unroll
        for (int b = 0; b < kBatch; ++b) q[b] = i + b * T < nvec ? __ldg(x + i + b * T) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int b = 0; b < kBatch; ++b) {
            if (DT == NVFP4_DT_F32)
                acc = max(acc, max(max(q[b].x & 0x7fffffffu, q[b].y & 0x7fffffffu), max(q[b].z & 0x7fffffffu, q[b].w & 0x7fffffffu)));
            else
                acc = __vmaxu2(acc, __vmaxu2(__vmaxu2(q[b].x & 0x7fff7fffu, q[b].y & 0x7fff7fffu),
                                             __vmaxu2(q[b].z & 0x7fff7fffu, q[b].w & 0x7fff7fffu)));
        }
    }
    uint32_t bits = acc;
    if (DT != NVFP4_DT_F32) {
        const uint32_t h = max(acc & 0xffffu, acc >> 16);
        bits = DT == NVFP4_DT_BF16 ? h << 16 : __float_as_uint(__half2float(__ushort_as_half(static_cast<unsigned short>(h))));
    }
    bits = __reduce_max_sync(0xffffffffu, bits);
    __shared__ uint32_t warp_max[T / 32];
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T / 32; ++i) bits = max(bits, warp_max[i]);
    return bits;
}

// Several tensors in one launch (a layer's activations): CTAs are numbered through the tensors.  (The body stands in the
// kernel, for one tensor and several: as an inlined function the compiler scheduled the sweep worse, 8192 x 8192 110.9 -> 112.4 us.)
struct MultiParams {
    QuantParams q[kMaxChain];
    uint32_t cta_end[kMaxChain];
};
// This CTA's tensor, and its number `bx` of the tensor's `ctas`.
__device__ __forceinline__ const QuantParams& tensor_of(const QuantParams& a, uint32_t& bx, uint32_t& ctas) {
    bx = blockIdx.x;
    ctas = gridDim.x;
    return a;
}
__device__ __forceinline__ const QuantParams& tensor_of(const MultiParams& a, uint32_t& bx, uint32_t& ctas) {
    int i = 0;
    while (blockIdx.x >= a.cta_end[i]) ++i;
    const uint32_t begin = i > 0 ? a.cta_end[i - 1] : 0;
    bx = blockIdx.x - begin;
    ctas = a.cta_end[i] - begin;
    return a.q[i];
}

template <int DT, int VARIANT, int IMPL, class Args>
__global__ void __launch_bounds__(block_threads(VARIANT, IMPL), min_blocks(VARIANT, IMPL))
quant_kernel(const __grid_constant__ Args args) {
    uint32_t bx, ctas;
    const QuantParams& p = tensor_of(args, bx, ctas);
    constexpr int T = block_threads(VARIANT, IMPL);   // threads per CTA
    static_assert(kTabSize % T == 0, "every thread builds the same number of table entries");
    __shared__ float4 tab[kTabSize];
    constexpr bool FUSED = IMPL == 4;
    constexpr bool OWN_SCALE = IMPL == 10;   // every CTA takes the global scale of the whole (small) tensor itself
    static_assert(!FUSED || VARIANT != NVFP4_VARIANT_AMAX, "the fused variant covers the two sweeps");
    // Launched as a programmatic dependent: the input, the global scale and the output buffers may still be in use by
    // the kernel before this one on the stream, so everything waits.  The kernel BEHIND this one may be scheduled right
    // away, even before that wait is over: whatever it does ahead of its own wait (a GEMM streams a prepared, constant
    // weight) depends on neither this kernel nor the ones before it, and its wait covers this kernel's completion,
    // which in turn comes after this wait.  That does not hold where this kernel writes such a weight: then (early == 0)
    // nothing behind it starts before it is complete, not even a GEMM two launches on, which without this could be let in by
    // a short kernel between them while this one still runs.
    if (p.early) griddep_launch();
    if (!FUSED) griddep_wait();
    // everything the kernel before this one may have written is read through pointers taken behind the wait
    const void* const x_in = after_wait(p.x);
    const float* const importance_in = after_wait(p.importance);
    float gs_inv = FUSED || OWN_SCALE ? 0.0f : load_f32_after_wait(p.gs_inv);
    // Two-dimensional grid: blockIdx.x is the row, blockIdx.y the column chunk.  The row is then uniform over the CTA, so
    // the division below, the row part of the addresses and most of the tiled scale offset leave the per-thread
    // instruction stream (8192 x 8192 sweep: 126 us numbered through, 112 us with this grid).
    constexpr bool GRID2D = IMPL == 7 || IMPL == 8;
    constexpr bool WHOLE = IMPL == 8 && VARIANT != NVFP4_VARIANT_AMAX;
    constexpr bool CHUNKS = IMPL == 8;   // rows of whole chunks: every column is in range
    constexpr bool FLAT = IMPL == 3 || IMPL == 5 || IMPL == 9 || IMPL == 10;   // real rows' slots numbered through, then CTAs that fill the padding rows
    const int64_t id = GRID2D ? 0 : static_cast<int64_t>(bx) * T + threadIdx.x;
    const int64_t slots = FLAT ? p.m * p.width : p.total;
    constexpr bool WARPS = IMPL == 6;               // a row's columns by whole warps, numbered through the rows
    const uint32_t row_warps = static_cast<uint32_t>((p.width + 31) >> 5);
    const uint32_t warps = static_cast<uint32_t>(p.m) * row_warps;
    bool in_range = GRID2D ? true : id < slots;
    int64_t row = 0, col = 0;
    if (GRID2D) {
        row = bx;
        col = static_cast<int64_t>(blockIdx.y) * T + threadIdx.x;
        if (!CHUNKS) in_range = col < p.width;
    } else if (WARPS) {
        const uint32_t w = bx * (T / 32) + __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
        const uint32_t r32 = row_div(p, w);
        row = r32;
        col = (w - r32 * row_warps) * 32u + (threadIdx.x & 31u);
        in_range = w < warps && col < p.width;
    } else if (in_range) {
        if (p.total <= 0x7fffffffLL) {
            const uint32_t r32 = row_div(p, static_cast<uint32_t>(id));
            row = r32;
            col = static_cast<uint32_t>(id) - r32 * static_cast<uint32_t>(p.width);
        } else {
            row = id / p.width;
            col = id - row * p.width;
        }
    }
    const bool valid = WHOLE ? true : (in_range && row < p.m && col < p.bout);
    if (IMPL == 7 && row >= p.m) {   // a padding row of the tiled scale layout: zero words, nothing else
        if (in_range && (threadIdx.x & 3) == 0) *reinterpret_cast<uint32_t*>(p.scales + swizzled_scale_offset(row, col, p.k_pad)) = 0u;
        return;
    }
    const uint32_t real_ctas = WARPS ? (warps + T / 32 - 1) / (T / 32) : FLAT ? static_cast<uint32_t>((slots + T - 1) / T) : 0u;
    if ((FLAT || WARPS) && bx >= real_ctas) {
        // A CTA behind the real rows' slots.  The rows m .. rows-1 of the tiled scale layout (127 of 128 for one token)
        // hold no data; these CTAs write their zero scale bytes, four 32-bit words (of four columns each) per thread,
        // and leave before the candidate table is built.  (Rows beyond m exist only in the tiled layout, whose width is
        // a multiple of 4; the launcher sizes this part of the grid, and at most 127 rows are padding.)
        const uint32_t words_per_row = static_cast<uint32_t>(p.width >> 2);
        const uint32_t words = static_cast<uint32_t>(p.rows - p.m) * words_per_row;
        const uint32_t fill_threads = (ctas - real_ctas) * T;
        for (uint32_t wi = (bx - real_ctas) * T + threadIdx.x; wi < words; wi += fill_threads) {
            const uint32_t r = wi / words_per_row;
            const uint32_t c = (wi - r * words_per_row) * 4u;
            *reinterpret_cast<uint32_t*>(p.scales + swizzled_scale_offset(p.m + r, c, p.k_pad)) = 0u;
        }
        return;
    }

    float v[16], w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        v[j] = 0.0f;
        w[j] = 0.0f;
    }
    if (WHOLE || (valid && col < p.bin)) {
        load16<DT>(x_in, row * p.n + col * kBlock, v);
        if (VARIANT == NVFP4_VARIANT_WEIGHTED) load16<NVFP4_DT_F32>(importance_in, col * kBlock, w);
    }

    if constexpr (OWN_SCALE) {
        const uint32_t nvec = static_cast<uint32_t>(p.m * p.n / (DT == NVFP4_DT_F32 ? 4 : 8));
        const float amax_x = __uint_as_float(cta_amax_bits<DT, T>(static_cast<const uint4*>(x_in), nvec));
        const float gs = __fmul_rn(amax_x, __fdiv_rn(1.0f, __fmul_rn(6.0f, p.fp8_max)));
        gs_inv = __fdiv_rn(1.0f, gs);
        if (bx == 0 && threadIdx.x == 0) {
            p.gs_out[0] = gs;
            p.gs_out[1] = gs_inv;
        }
    }

    // The global scale and the block's elements were requested above; the candidate table is built while they are
    // on their way (at small batch sizes nothing else hides a trip to memory).  The amax variant needs no table: its
    // one multiplier per block is two reciprocals away from the scale byte, and without the table there is no
    // CTA-wide barrier between the loads and their use.
    if (VARIANT != NVFP4_VARIANT_AMAX) {
#pragma unroll
        for (int t = threadIdx.x; t < kTabSize; t += T) {   // one entry per thread with 256 threads, four with 64
            const float s = e4m3_to_f32(table_raw(t)), s_next = e4m3_to_f32(table_raw(t + 1));
            float4 e;
            e.x = e.y = div_full(1.0f, s);
            e.z = __fmul_rn(s, s);
            e.w = __fmul_rn(s_next, s_next);
            tab[t] = e;
        }
        __syncthreads();
    }

    if (FUSED) {
        // tensor-wide maximum on fp32 magnitude bit patterns (a NaN pattern is larger than +inf, as torch's max wants)
        __shared__ uint32_t warp_max[kThreads / 32];
        __shared__ float gs_inv_shared;
        uint32_t bits = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) bits = max(bits, __float_as_uint(v[j]) & 0x7fffffffu);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) bits = max(bits, __shfl_xor_sync(0xffffffffu, bits, o));
        if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t b = 0;
            for (int i = 0; i < kThreads / 32; ++i) b = max(b, warp_max[i]);
            volatile uint32_t* sc = p.fused_scratch;
            atomicMax(p.fused_scratch, b);
            __threadfence();
            // scratch[3] != 0 is a testing hook: CTA 0 then withholds its arrival, so that every wait below runs into
            // the limit and the error path (status word, no hang) can be exercised
            if (!(blockIdx.x == 0 && sc[3] != 0u)) atomicAdd(p.fused_scratch + 1, 1u);
            // every CTA of a cooperative launch is resident, so the others will arrive; bounded all the same
            uint64_t t0 = 0;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
            while (sc[1] < gridDim.x) {
                uint64_t t1;
                asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
                if (t1 - t0 > g_fused_wait_limit_ns) {
                    atomicExch(&g_quant_status, 1u);
                    break;
                }
                __nanosleep(64);
            }
            __threadfence();
            const float amax = __uint_as_float(sc[0]);
            const float inv_den = __fdiv_rn(1.0f, __fmul_rn(6.0f, p.fp8_max));
            const float gs = __fmul_rn(amax, inv_den);
            const float gsi = __fdiv_rn(1.0f, gs);
            gs_inv_shared = gsi;
            __threadfence();
            // the last CTA to have read the maximum publishes the result and leaves the scratch zeroed
            if (atomicAdd(p.fused_scratch + 2, 1u) == gridDim.x - 1) {
                p.gs_out[0] = gs;
                p.gs_out[1] = gsi;
                sc[0] = 0u;
                sc[1] = 0u;
                sc[2] = 0u;
            }
        }
        __syncthreads();
        gs_inv = gs_inv_shared;
    }

    uint32_t sbyte = 0;
    float inv = 0.0f;
    // A warp with nothing but padding columns or threads behind the last slot has nothing to sweep.  (Body 6 has next to none of
    // these and is 0.5 % faster without the vote, the weighted body 3 up to 3 %, body 5 2.5 %; the unweighted body 3 is slower without
    // it.)  Amax has little to skip: 16-bit 7575 x 3168 13.1 us with the vote, 11.9 without; fp32, whose warps wait for twice the
    // bytes, 17.6 and 18.3.
    constexpr bool VOTE = VARIANT == NVFP4_VARIANT_AMAX ? FLAT && DT == NVFP4_DT_F32
                                                        : IMPL == 7 || (FLAT && IMPL != 5 && !(IMPL == 3 && VARIANT == NVFP4_VARIANT_WEIGHTED));
    if (VOTE && !__any_sync(0xffffffffu, valid)) {
        // nothing
    } else if (VARIANT == NVFP4_VARIANT_AMAX) {
        const float amax = max_abs16(v);
        const float sf = __fmul_rn(gs_inv, __fmul_rn(amax, rcp_approx_ftz(6.0f)));
        sbyte = f32_to_e4m3(sf);
        const uint32_t raw = sbyte & 0x7fu;
        inv = (raw == 0) ? 0.0f : rcp_approx_ftz(__fmul_rn(e4m3_to_f32(raw), rcp_approx_ftz(gs_inv)));
    } else {
        const uint64_t gs2 = pack_f32x2(gs_inv, gs_inv);
#pragma unroll
        for (int q = 0; q < 8; ++q)   // packed multiply: each lane is the same IEEE product as a scalar mul.rn
            unpack_f32x2(mul_f32x2(pack_f32x2(v[2 * q], v[2 * q + 1]), gs2), v[2 * q], v[2 * q + 1]);
        const float amax = max_abs16(v);
        const float base_scale = __fmul_rn(amax, __uint_as_float(0x3E2AAAABu));  // fp32(1/6)
        const uint32_t base_fp8 = f32_to_e4m3(base_scale);
        int base_raw = static_cast<int>(base_fp8);
        if (VARIANT == NVFP4_VARIANT_WEIGHTED) base_raw -= (e4m3_to_f32(base_fp8) > base_scale) ? 1 : 0;
        constexpr bool W = VARIANT == NVFP4_VARIANT_WEIGHTED;
        // clamping the start once is enough: with it below -kTabPad every candidate is raw 1, above 127 every one 126
        const int first_idx = min(max(base_raw + p.lower, -kTabPad), 127) + kTabPad;
        if constexpr (IMPL == 1) {
            sbyte = sweep_scalar<W>(v, w, first_idx, p.ncand, tab);
        } else if constexpr (IMPL == 2) {
            sbyte = sweep_single<W>(v, w, first_idx, p.ncand, tab);
        } else {
            // the reference's own windows are compiled in, unrolled
            constexpr int NC = W ? kWindowWeighted : kWindow;
            const bool compiled = WHOLE || ((IMPL == 7 || (FLAT && IMPL != 5) || WARPS) && own_window(VARIANT, p.lower, p.ncand));
            if constexpr (W) {
                float w_min = w[0];
#pragma unroll
                for (int j = 1; j < 16; ++j) w_min = fminf(w_min, w[j]);
                sbyte = compiled ? sweep_weighted<NC>(v, w, w_min, amax, first_idx, p.ncand, p.lower, tab)
                                 : sweep_weighted<>(v, w, w_min, amax, first_idx, p.ncand, p.lower, tab);
            } else {
                sbyte = compiled ? sweep_paired<NC>(v, first_idx, p.ncand, tab) : sweep_paired<>(v, first_idx, p.ncand, tab);
            }
        }
        // sbyte is 0 only when no candidate had a comparable (non-NaN, < inf) error: 1/0 as the reference computes it
        inv = (sbyte == 0) ? div_full(1.0f, 0.0f) : tab[sbyte + kTabPad].x;
    }

    if (valid) {
        const uint64_t inv2 = pack_f32x2(inv, inv);
        float x[16];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            unpack_f32x2(mul_f32x2(pack_f32x2(v[2 * q], v[2 * q + 1]), inv2), x[2 * q], x[2 * q + 1]);
        const uint32_t lo = f32x8_to_e2m1x8(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]);
        const uint32_t hi = f32x8_to_e2m1x8(x[8], x[9], x[10], x[11], x[12], x[13], x[14], x[15]);
        *reinterpret_cast<uint2*>(p.codes + (row * p.bout + col) * 8) = make_uint2(lo, hi);
    } else {
        sbyte = 0;  // padding rows / columns of the scale buffer read as zero scales
    }

    // Scale store.  With width % 4 == 0 (always true for the swizzled layout) lanes
    // 4q..4q+3 hold four consecutive blocks of one row: merge them into one 32-bit store.
    if ((p.width & 3) == 0) {
        const uint32_t lane = threadIdx.x & 31;
        uint32_t word = sbyte << (8 * (lane & 3));
        word |= __shfl_xor_sync(0xffffffffu, word, 1);
        word |= __shfl_xor_sync(0xffffffffu, word, 2);
        if (in_range && (lane & 3) == 0) {
            const int64_t off = p.swizzled ? swizzled_scale_offset(row, col, p.k_pad) : row * p.width + col;
            *reinterpret_cast<uint32_t*>(p.scales + off) = word;
        }
    } else if (in_range) {
        p.scales[row * p.width + col] = static_cast<uint8_t>(sbyte);
    }
}

// Grid of the bodies that number the real rows' slots (or warps of rows) through: CTAs for those, then CTAs that zero the padding rows' scale
// words (4 words per thread).
int64_t flat_ctas(const QuantParams& p, int T, bool warps) {
    const int64_t pad_words = (p.rows - p.m) * (p.width >> 2);
    if (pad_words > 0x7fffffffLL) return INT64_MAX;   // at most 127 rows: a width beyond 2^26 columns
    const int64_t slots = warps ? p.m * ((p.width + 31) / 32 * 32) : p.m * p.width;
    return (slots + T - 1) / T + (pad_words + 4 * T - 1) / (4 * T);
}
template <int DT, int VARIANT, int IMPL>
cudaError_t launch_flat(const QuantParams& p, cudaStream_t stream) {
    constexpr int T = block_threads(VARIANT, IMPL);
    const int64_t grid = flat_ctas(p, T, IMPL == 6);
    if (grid > 0x7fffffffLL) return cudaErrorInvalidValue;
    return launch_dependent(quant_kernel<DT, VARIANT, IMPL, QuantParams>, static_cast<unsigned>(grid), dim3(T), 0, stream, p);
}

// The grid of rows that are no whole chunks of T blocks: the slots numbered through (3) keeps every thread busy but divides
// per thread, a row by whole warps (6) or by whole CTAs (7) leaves the last one partly idle; 7 divides nothing, 6 once per warp.
// By the idle part; us, bodies 3 / 6 / 7, bf16, 1500000 blocks: unweighted, rows of 498 45.6 / 44.4 / 43.9, 575 45.5 / 43.3 /
// 44.0, 643 45.5 / 45.0 / 45.7, 90 46.5 / 45.9 / 47.7 (not tiled,
// where the address is cheap, 44.2 / 45.0 / 46.3); weighted, 498 73.9 / 73.7 / 73.2, 643 73.8 / 74.7 / 75.3; amax, 200000 blocks, rows of 200
// 2.95 / 2.82 / 2.69, 564 3.07 / 2.88 / 2.62, 1500000, 200 11.9 / 12.2 / 12.1, 320 11.8 / 11.3 / 13.4, 716 11.7 / 11.4 / 11.2, 4000000, 836
// 30.5 / 29.4 / 31.0, 500 29.7 / 29.4 / 28.9.  Fp32 amax is bound by its loads: the grid without an idle thread is ahead (4000000, 836
// 43.3 / 43.8 / 46.3) but for a short launch, which its division delays (60000, 512 2.88 / 2.50 / 2.93, 716 3.33 / 3.14 / 3.33).
int ragged_body(int variant, bool fp32, int64_t blocks, int64_t width, bool tiled, int T) {
    const int64_t idle_warp = (width + 31) / 32 * 32 - width, idle_cta = (width + T - 1) / T * T - width;
    if (variant == NVFP4_VARIANT_AMAX && fp32) return blocks >= 131072 ? 3 : 6;
    if (variant == NVFP4_VARIANT_AMAX)
        return idle_cta * (blocks < 524288 ? 2 : 8) <= width ? 7 : idle_warp * 10 <= width ? 6 : 3;
    if (idle_warp * (variant == NVFP4_VARIANT_WEIGHTED ? 32 : tiled ? 17 : 20) > width) return 3;
    return idle_cta == idle_warp ? 7 : 6;
}
template <int DT, int VARIANT>
cudaError_t launch_impl(int impl, const QuantParams& p, cudaStream_t stream) {
    constexpr bool kSweep = VARIANT != NVFP4_VARIANT_AMAX;
    constexpr int T = block_threads(VARIANT, 7);
    if (impl == 1 || impl == 2) {
        const unsigned grid = static_cast<unsigned>((p.total + kThreads - 1) / kThreads);
        return impl == 1 ? launch_dependent(quant_kernel<DT, VARIANT, 1, QuantParams>, grid, dim3(kThreads), 0, stream, p)
                         : launch_dependent(quant_kernel<DT, VARIANT, 2, QuantParams>, grid, dim3(kThreads), 0, stream, p);
    }
    const bool chunks = p.width % T == 0;
    int body = impl;
    const int64_t blocks = p.m * p.bout;
    constexpr bool kFp32 = DT == NVFP4_DT_F32;
    if (impl == 0 || impl == 8) body = chunks && !(!kSweep && kFp32 && blocks >= 131072) ? 7 : ragged_body(VARIANT, kFp32, blocks, p.width, p.swizzled != 0, T);
    if (impl == 0 && kSweep) {
        const int64_t small = chunks ? kSmallBlocks : VARIANT == NVFP4_VARIANT_WEIGHTED && body == 3 ? kSmallBlocksRaggedWeighted : kSmallBlocksRagged;
        if (blocks <= small) body = 9;
        if (body == 3 && VARIANT == NVFP4_VARIANT_MSE && !kFp32 && blocks >= kLargeBlocksRagged) body = 5;
    }
    if (body == 7 && ((p.width + T - 1) / T > 65535 || p.rows > 0x7fffffffLL)) body = 3;
    if (body == 6 && p.m * ((p.width + 31) / 32) > 0x7fffffffLL) body = 3;
    if (body == 9) return launch_flat<DT, VARIANT, 9>(p, stream);
    if (body == 6) {
        QuantParams q = p;
        set_row_div(q, (p.width + 31) / 32);
        return launch_flat<DT, VARIANT, 6>(q, stream);
    }
    if (body == 7) {
        const dim3 grid2(static_cast<unsigned>(p.rows), static_cast<unsigned>((p.width + T - 1) / T));
        // no padding anywhere: every slot of the scale layout is a real block
        const bool whole = chunks && p.rows == p.m && p.bin == p.bout && p.bout == p.width && own_window(VARIANT, p.lower, p.ncand);
        if constexpr (!kSweep)
            if (chunks && impl != 7) return launch_dependent(quant_kernel<DT, VARIANT, 8, QuantParams>, grid2, dim3(T), 0, stream, p);
        if constexpr (kSweep)
            if (whole && impl != 7) return launch_dependent(quant_kernel<DT, VARIANT, 8, QuantParams>, grid2, dim3(T), 0, stream, p);
        return launch_dependent(quant_kernel<DT, VARIANT, 7, QuantParams>, grid2, dim3(T), 0, stream, p);
    }
    if constexpr (VARIANT == NVFP4_VARIANT_MSE && !kFp32)
        if (body == 5) return launch_flat<DT, VARIANT, 5>(p, stream);
    return launch_flat<DT, VARIANT, 3>(p, stream);
}

template <int DT>
cudaError_t launch_variant(int variant, int impl, const QuantParams& p, cudaStream_t stream) {
    switch (variant) {
        case NVFP4_VARIANT_MSE: return launch_impl<DT, NVFP4_VARIANT_MSE>(impl, p, stream);
        case NVFP4_VARIANT_WEIGHTED: return launch_impl<DT, NVFP4_VARIANT_WEIGHTED>(impl, p, stream);
        default: return launch_impl<DT, NVFP4_VARIANT_AMAX>(impl, p, stream);
    }
}

}  // namespace
}  // namespace nvfp4

namespace nvfp4 {
namespace {
// Checks one tensor's arguments and fills its parameters.  NVFP4_OK with p.total == 0: nothing to do.  `gs_inv` is required
// here; the chain passes the pair its first kernel writes.
int fill_params(QuantParams& p, int variant, const void* x, int x_dtype, const float* importance, const float* gs_inv, uint8_t* codes,
                uint8_t* scales, int64_t m, int64_t n, int64_t padded_n, int lower, int upper, int swizzled) {
    if (variant < NVFP4_VARIANT_MSE || variant > NVFP4_VARIANT_AMAX) return NVFP4_ERR_BAD_ENUM;
    if (x_dtype < NVFP4_DT_BF16 || x_dtype > NVFP4_DT_F32) return NVFP4_ERR_BAD_ENUM;
    if (m < 0 || n < 0 || (n % kBlock) != 0 || (padded_n % kBlock) != 0 || padded_n < n) return NVFP4_ERR_BAD_SHAPE;
    if (variant != NVFP4_VARIANT_AMAX && (upper < lower || upper - lower + 1 > 64)) return NVFP4_ERR_BAD_RANGE;
    p.m = m;
    p.n = n;
    p.bin = n / kBlock;
    p.bout = padded_n / kBlock;
    p.k_pad = round_up_i64(p.bout, 4);
    p.swizzled = swizzled ? 1 : 0;
    p.width = swizzled ? p.k_pad : p.bout;
    p.rows = swizzled ? round_up_i64(m, 128) : m;
    p.total = p.rows * p.width;
    set_row_div(p, p.width);
    if (p.total == 0) return NVFP4_OK;
    if ((p.total + kThreads - 1) / kThreads > 0x7fffffffLL) return NVFP4_ERR_TOO_LARGE;
    if (!gs_inv || !codes || !scales || (!x && m * n > 0)) return NVFP4_ERR_NULL_POINTER;
    if (variant == NVFP4_VARIANT_WEIGHTED && !importance && n > 0) return NVFP4_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(codes) & 7) ||
        (reinterpret_cast<uintptr_t>(gs_inv) & 3))
        return NVFP4_ERR_MISALIGNED;
    if (swizzled && (reinterpret_cast<uintptr_t>(scales) & 3)) return NVFP4_ERR_MISALIGNED;
    if (!swizzled && (p.width & 3) == 0 && (reinterpret_cast<uintptr_t>(scales) & 3)) return NVFP4_ERR_MISALIGNED;
    if (variant == NVFP4_VARIANT_WEIGHTED && (reinterpret_cast<uintptr_t>(importance) & 15)) return NVFP4_ERR_MISALIGNED;
    p.x = x;
    p.importance = importance;
    p.gs_inv = gs_inv;
    p.codes = codes;
    p.scales = scales;
    p.lower = lower;
    p.ncand = (variant == NVFP4_VARIANT_AMAX) ? 0 : upper - lower + 1;
    p.early = 1;
    p.fp8_max = 0.0f;
    p.gs_out = nullptr;
    p.fused_scratch = nullptr;
    return NVFP4_OK;
}
}  // namespace
}  // namespace nvfp4

static int quant_launch(int impl, int early, int variant, const void* x, int x_dtype, const float* importance, const float* gs_inv,
                        uint8_t* codes, uint8_t* scales, int64_t m, int64_t n, int64_t padded_n, int lower, int upper, int swizzled,
                        void* stream) {
    using namespace nvfp4;
    if (impl < 0 || impl > 9 || impl == 4) return NVFP4_ERR_BAD_ENUM;
    QuantParams p;
    const int st = fill_params(p, variant, x, x_dtype, importance, gs_inv, codes, scales, m, n, padded_n, lower, upper, swizzled);
    if (st != NVFP4_OK || p.total == 0) return st;
    p.early = early;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t err;
    switch (x_dtype) {
        case NVFP4_DT_BF16: err = launch_variant<NVFP4_DT_BF16>(variant, impl, p, s); break;
        case NVFP4_DT_F16: err = launch_variant<NVFP4_DT_F16>(variant, impl, p, s); break;
        default: err = launch_variant<NVFP4_DT_F32>(variant, impl, p, s); break;
    }
    return static_cast<int>(err);
}

extern "C" int nvfp4_quant_launch_impl(int impl, int variant, const void* x, int x_dtype, const float* importance,
                                       const float* gs_inv, uint8_t* codes, uint8_t* scales, int64_t m, int64_t n,
                                       int64_t padded_n, int lower, int upper, int swizzled, void* stream) {
    return quant_launch(impl, 1, variant, x, x_dtype, importance, gs_inv, codes, scales, m, n, padded_n, lower, upper, swizzled, stream);
}

// nvfp4_quant_launch into buffers that a prepared weight may refer to.
extern "C" int nvfp4_quant_launch_in_place(int variant, const void* x, int x_dtype, const float* importance, const float* gs_inv,
                                           uint8_t* codes, uint8_t* scales, int64_t m, int64_t n, int64_t padded_n, int lower,
                                           int upper, int swizzled, void* stream) {
    return quant_launch(0, 0, variant, x, x_dtype, importance, gs_inv, codes, scales, m, n, padded_n, lower, upper, swizzled, stream);
}

namespace nvfp4 {
namespace {
template <int DT, int VARIANT>
cudaError_t launch_fused(const QuantParams& p, int sms, cudaStream_t stream, bool* too_large) {
    const int64_t grid = (p.total + kThreads - 1) / kThreads;
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, quant_kernel<DT, VARIANT, 4, QuantParams>, kThreads, 0);
    if (e != cudaSuccess) return e;
    if (grid > static_cast<int64_t>(per_sm) * sms) {
        *too_large = true;
        return cudaSuccess;
    }
    QuantParams q = p;
    void* args[] = {&q};
    return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(quant_kernel<DT, VARIANT, 4, QuantParams>),
                                       dim3(static_cast<unsigned>(grid)), dim3(kThreads), args, 0, stream);
}
template <int DT>
cudaError_t launch_fused_variant(int variant, const QuantParams& p, int sms, cudaStream_t stream, bool* too_large) {
    if (variant == NVFP4_VARIANT_MSE) return launch_fused<DT, NVFP4_VARIANT_MSE>(p, sms, stream, too_large);
    return launch_fused<DT, NVFP4_VARIANT_WEIGHTED>(p, sms, stream, too_large);
}
}  // namespace
}  // namespace nvfp4

namespace nvfp4 {
namespace {
// Tensors of up to this many bytes take their global scale inside the quantizer: every CTA reads the whole tensor (from L2,
// 16 loads per thread in flight at once) instead of waiting for a kernel before it.  One launch instead of two: chain of
// launches, 1 x 4096 bf16 3.2 -> 2.4 us, 4 x 8192 (64 KiB) 4.8 -> 3.5, 16 x 4096 (128 KiB) 5.0 -> 4.8, but 16 x 8192 5.4 -> 8.0.
// A quantization on its own is bound by the host up to there (5 x 13024 from Python, 127 KiB: 5.8 us with one launch, 7.6 with two).
// With products behind it the pass over all of the tensor delays them more than a launch does from 64 KiB on: a Llama-3-8B-shaped layer
// as four quantizers and the products with each, 8 tokens 51.7 us, 12 tokens 54.6 with two launches and 56.8 with one, 16 tokens 57.9
// and 62.8; launched eagerly, 16 tokens 62.6 and 65.7.
constexpr int64_t kOwnScaleBytes = 131072;        // nvfp4_quant_chain_launch
constexpr int64_t kOwnScaleBytesLayer = 65536;    // nvfp4_quant_chain_multi_launch: a layer's activations
// Several tensors with up to this many blocks in all share their launches, slots numbered through; beyond it the
// two-dimensional grids of separate launches gain more than the launches cost.
constexpr int64_t kMultiBlocks = 524288;
constexpr int64_t kMultiSmallBlocks = 98304;   // as kSmallBlocksRagged

template <int DT, int VARIANT, int IMPL>
cudaError_t launch_multi(const QuantParams* q, int n, cudaStream_t stream) {
    constexpr int T = block_threads(VARIANT, IMPL);
    if (n == 1) return launch_flat<DT, VARIANT, IMPL>(q[0], stream);
    MultiParams mp;
    int64_t end = 0;
    for (int i = 0; i < n; ++i) {
        mp.q[i] = q[i];
        end += flat_ctas(q[i], T, false);
        mp.cta_end[i] = static_cast<uint32_t>(end);
    }
    return launch_dependent(quant_kernel<DT, VARIANT, IMPL, MultiParams>, dim3(static_cast<unsigned>(end)), dim3(T), 0, stream, mp);
}

// The quantizer half of a chain over n tensors of one variant (n > 1, or own_scale).
template <int DT>
cudaError_t launch_chain(int variant, bool own_scale, bool small, const QuantParams* q, int n, cudaStream_t s) {
    if (variant == NVFP4_VARIANT_MSE)
        return own_scale ? launch_multi<DT, NVFP4_VARIANT_MSE, 10>(q, n, s)
               : small   ? launch_multi<DT, NVFP4_VARIANT_MSE, 9>(q, n, s)
                         : launch_multi<DT, NVFP4_VARIANT_MSE, 3>(q, n, s);
    return own_scale ? launch_multi<DT, NVFP4_VARIANT_WEIGHTED, 10>(q, n, s)
           : small   ? launch_multi<DT, NVFP4_VARIANT_WEIGHTED, 9>(q, n, s)
                     : launch_multi<DT, NVFP4_VARIANT_WEIGHTED, 3>(q, n, s);
}
}  // namespace
}  // namespace nvfp4

// Global scale, then the quantizer with that scale, of up to kMaxChain tensors per launch: what get_nvfp4_global_scale
// followed by scalesweep_*_quant_out do (helper.py:96-100, bench.py:57-67 of the reference), for callers that pay per
// launch and per host call (an eager decode loop).  Bytes equal the separate calls.
static int chain_launch(int64_t own_scale_bytes, int variant, int x_dtype, float fp8_max, const nvfp4_chain_item* items, int n_items,
                        int lower, int upper, int swizzled, void* stream) {
    using namespace nvfp4;
    if (n_items < 0 || n_items > 64) return NVFP4_ERR_BAD_RANGE;
    if (n_items == 0) return NVFP4_OK;
    if (!items) return NVFP4_ERR_NULL_POINTER;
    if (!(fp8_max > 0.0f)) return NVFP4_ERR_BAD_RANGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    for (int first = 0; first < n_items; first += kMaxChain) {
        const int n = n_items - first < kMaxChain ? n_items - first : kMaxChain;
        const nvfp4_chain_item* it = items + first;
        QuantParams q[kMaxChain];
        GsItem gs[kMaxChain];
        bool own_scale = variant != NVFP4_VARIANT_AMAX;
        int64_t blocks = 0;
        for (int i = 0; i < n; ++i) {
            if (it[i].m <= 0 || it[i].n <= 0) return NVFP4_ERR_BAD_SHAPE;   // an empty tensor has no maximum
            if (!it[i].gs_out) return NVFP4_ERR_NULL_POINTER;
            gs[i] = GsItem{it[i].x, it[i].m * it[i].n, it[i].gs_out, it[i].scratch};
            int st = check_global_scale(gs[i], x_dtype);
            if (st == NVFP4_OK)
                st = fill_params(q[i], variant, it[i].x, x_dtype, it[i].importance, it[i].gs_out + 1, it[i].codes, it[i].scales, it[i].m,
                                 it[i].n, it[i].padded_n, lower, upper, swizzled);
            if (st != NVFP4_OK) return st;
            q[i].fp8_max = fp8_max;
            q[i].gs_out = it[i].gs_out;
            blocks += q[i].m * q[i].width;
            own_scale = own_scale && it[i].m * it[i].n * (x_dtype == NVFP4_DT_F32 ? 4 : 2) <= own_scale_bytes;
        }
        const bool together = own_scale || (n > 1 && variant != NVFP4_VARIANT_AMAX && blocks <= kMultiBlocks);
        if (!own_scale) {
            const int st = launch_global_scales(gs, together ? n : 1, x_dtype, fp8_max, s);
            if (st != NVFP4_OK) return st;
        }
        if (together) {
            const bool small = blocks <= kMultiSmallBlocks;
            cudaError_t e;
            switch (x_dtype) {
                case NVFP4_DT_BF16: e = launch_chain<NVFP4_DT_BF16>(variant, own_scale, small, q, n, s); break;
                case NVFP4_DT_F16: e = launch_chain<NVFP4_DT_F16>(variant, own_scale, small, q, n, s); break;
                default: e = launch_chain<NVFP4_DT_F32>(variant, own_scale, small, q, n, s); break;
            }
            if (e != cudaSuccess) return static_cast<int>(e);
            continue;
        }
        for (int i = 0; i < n; ++i) {
            int st = i > 0 ? launch_global_scales(gs + i, 1, x_dtype, fp8_max, s) : NVFP4_OK;
            if (st == NVFP4_OK)
                st = nvfp4_quant_launch(variant, it[i].x, x_dtype, it[i].importance, it[i].gs_out + 1, it[i].codes, it[i].scales, it[i].m,
                                        it[i].n, it[i].padded_n, lower, upper, swizzled, stream);
            if (st != NVFP4_OK) return st;
        }
    }
    return NVFP4_OK;
}

extern "C" int nvfp4_quant_chain_multi_launch(int variant, int x_dtype, float fp8_max, const nvfp4_chain_item* items, int n_items,
                                              int lower, int upper, int swizzled, void* stream) {
    return chain_launch(nvfp4::kOwnScaleBytesLayer, variant, x_dtype, fp8_max, items, n_items, lower, upper, swizzled, stream);
}

extern "C" int nvfp4_quant_chain_launch(int variant, const void* x, int x_dtype, const float* importance, float fp8_max,
                                        float* gs_out, uint32_t* scratch, uint8_t* codes, uint8_t* scales, int64_t m,
                                        int64_t n, int64_t padded_n, int lower, int upper, int swizzled, void* stream) {
    const nvfp4_chain_item item = {x, importance, gs_out, scratch, codes, scales, m, n, padded_n};
    if (m <= 0 || n <= 0) return NVFP4_ERR_BAD_SHAPE;
    return chain_launch(nvfp4::kOwnScaleBytes, variant, x_dtype, fp8_max, &item, 1, lower, upper, swizzled, stream);
}

extern "C" int nvfp4_quant_fused_launch(int variant, const void* x, int x_dtype, const float* importance, float fp8_max,
                                        float* gs_out, uint32_t* scratch, uint8_t* codes, uint8_t* scales, int64_t m,
                                        int64_t n, int64_t padded_n, int lower, int upper, int swizzled, void* stream) {
    using namespace nvfp4;
    if (variant != NVFP4_VARIANT_MSE && variant != NVFP4_VARIANT_WEIGHTED) return NVFP4_ERR_BAD_ENUM;
    if (!(fp8_max > 0.0f)) return NVFP4_ERR_BAD_RANGE;
    QuantParams p;
    const int st = fill_params(p, variant, x, x_dtype, importance, gs_out, codes, scales, m, n, padded_n, lower, upper, swizzled);
    if (st != NVFP4_OK) return st;
    if (p.total == 0 || m * n == 0) return NVFP4_ERR_BAD_SHAPE;   // an empty tensor has no maximum
    if (!scratch) return NVFP4_ERR_NULL_POINTER;
    if (reinterpret_cast<uintptr_t>(scratch) & 3) return NVFP4_ERR_MISALIGNED;
    p.fp8_max = fp8_max;
    p.gs_out = gs_out;
    p.fused_scratch = scratch;
    int dev = 0, sms = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) return NVFP4_ERR_UNSUPPORTED;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    bool too_large = false;
    cudaError_t err;
    switch (x_dtype) {
        case NVFP4_DT_BF16: err = launch_fused_variant<NVFP4_DT_BF16>(variant, p, sms, s, &too_large); break;
        case NVFP4_DT_F16: err = launch_fused_variant<NVFP4_DT_F16>(variant, p, sms, s, &too_large); break;
        default: err = launch_fused_variant<NVFP4_DT_F32>(variant, p, sms, s, &too_large); break;
    }
    if (too_large) return NVFP4_ERR_TOO_LARGE;
    return static_cast<int>(err);
}

extern "C" int nvfp4_quant_fused_last_status(void* stream, uint32_t* status_host) {
    if (!status_host) return NVFP4_ERR_NULL_POINTER;
    cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
    if (e != cudaSuccess) return static_cast<int>(e);
    e = cudaMemcpyFromSymbol(status_host, nvfp4::g_quant_status, sizeof(uint32_t));
    if (e != cudaSuccess) return static_cast<int>(e);
    if (*status_host != 0) {
        const uint32_t zero = 0;
        e = cudaMemcpyToSymbol(nvfp4::g_quant_status, &zero, sizeof(uint32_t));
    }
    return static_cast<int>(e);
}

extern "C" int nvfp4_quant_launch(int variant, const void* x, int x_dtype, const float* importance,
                                  const float* gs_inv, uint8_t* codes, uint8_t* scales, int64_t m, int64_t n,
                                  int64_t padded_n, int lower, int upper, int swizzled, void* stream) {
    return nvfp4_quant_launch_impl(0, variant, x, x_dtype, importance, gs_inv, codes, scales, m, n, padded_n, lower,
                                   upper, swizzled, stream);
}

// Testing hook: the limit (nanoseconds, 1 us .. 10 s) of the fused kernel's grid-wide wait on the current device;
// 0 restores the default of 2 s.  Synchronous.
extern "C" int nvfp4_quant_fused_set_wait_limit_ns(uint64_t ns) {
    if (ns == 0) ns = nvfp4::kFusedWaitLimitNs;
    if (ns < 1000ull || ns > 10000000000ull) return NVFP4_ERR_BAD_RANGE;
    return static_cast<int>(cudaMemcpyToSymbol(nvfp4::g_fused_wait_limit_ns, &ns, sizeof(ns)));
}
