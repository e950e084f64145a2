// Per-input-channel squared L2 norm of an activation batch: out[j] = sum_i x[i, j]^2 (fp32).
//
// This is the importance vector the reference feeds to the weighted quantizer ("the importance scores for
// weight tensors are based on the activation input-channel square norm, and vice versa", README.md:11 of
// efsotr/nvfp4quant_test; its driver script is not published, torch's `(x.float() ** 2).sum(0)` is the
// obvious spelling).  One pass over x; the summation order is fixed (rows strided by 64 per thread in ascending
// order, then a fixed binary tree over the 64 row groups), so the result is reproducible run to run.  A CTA owns
// 16 columns, so an 8192-column batch runs on 512 CTAs.  What bounds it: the latency of a thread's loads, one batch after another,
// as long as the CTAs leave SMs idle, and HBM from about 8192 columns on.  So the fewer CTAs share an SM, the more loads a thread
// has in flight, and the rows left over are one batch too, not a row at a time.  See launch_sqnorm for what each form measured.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace nvfp4 {
namespace {

constexpr int kSqThreads = 256;   // 64 row groups x 4 lanes
constexpr int kSqLanes = 4;       // lanes side by side on one row segment
constexpr int kSqGroups = kSqThreads / kSqLanes;
constexpr int kSqCols = 4 * kSqLanes;   // columns per CTA: 4 per lane (32 bytes of bf16 per row: one DRAM sector)
constexpr unsigned kSqSms = 148;  // of a B200; another count only makes the choice of a form coarser
constexpr unsigned kSqEarlyCtas = 128;   // CTAs up to which the next kernel is let in at once

// Four consecutive elements as they are stored.  The loads are volatile: left to itself the compiler sinks them to their uses, and
// about eight were in flight whatever the batch.
template <int DT>
struct Quad {
    static constexpr int kWords = DT == NVFP4_DT_F32 ? 4 : 2;
    uint32_t w[kWords];
    __device__ __forceinline__ void load(const char* p) {
        if constexpr (DT == NVFP4_DT_F32)
            asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "l"(p));
        else
            asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];" : "=r"(w[0]), "=r"(w[1]) : "l"(p));
    }
    __device__ __forceinline__ void add_squares(float acc[4]) const {
        float v[4];
        if constexpr (DT == NVFP4_DT_F32) {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = __uint_as_float(w[k]);
        } else if constexpr (DT == NVFP4_DT_BF16) {
            v[0] = __uint_as_float(w[0] << 16); v[1] = __uint_as_float(w[0] & 0xffff0000u);
            v[2] = __uint_as_float(w[1] << 16); v[3] = __uint_as_float(w[1] & 0xffff0000u);
        } else {
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w[0]));
            const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w[1]));
            v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = __fmaf_rn(v[k], v[k], acc[k]);
    }
};

// The last `left` <= W rows of a thread in one batch, of the smallest power of two that holds them: in the places beyond them the last
// row once more, left out of the sum.
template <int DT, int W>
__device__ __forceinline__ void add_rest(const char* p, int64_t step, int left, float acc[4]) {
    if constexpr (W > 1) {
        if (left <= W / 2) {
            add_rest<DT, W / 2>(p, step, left, acc);
            return;
        }
    }
    if (left <= 0) return;
    Quad<DT> q[W];
#pragma unroll
    for (int u = 0; u < W; ++u) q[u].load(p + min(u, left - 1) * step);
#pragma unroll
    for (int u = 0; u < W; ++u)
        if (u < left) q[u].add_squares(acc);
}

// U loads in flight per thread, kCtas CTAs per SM.
template <int DT, int U, int kCtas>
__global__ void __launch_bounds__(kSqThreads, kCtas) channel_sqnorm_kernel(const void* x, int64_t m, int64_t n, int64_t ld,
                                                                           float* out) {
    // A programmatic dependent launch like the library's others: everything waits.  The kernel behind this one is let in at once only
    // where this one leaves SMs free.  Beside more CTAs, those of another importance crowd on the SMs with room and stay there:
    // back to back, bf16, eight loads a thread, us, let in late / at once: 300 x 1040 2.4 / 2.0, 4096 x 1024 (64 CTAs) 8.6 / 8.1, 2048 x 4096 (256) 6.3 / 7.7,
    // 4096 x 8192 (512) 14.4 / 17.1, 8192 x 8192 26.0 / 29.2.
    if (gridDim.x <= kSqEarlyCtas) griddep_launch();
    griddep_wait();
    x = after_wait(x);
    const int lane = threadIdx.x % kSqLanes, rg = threadIdx.x / kSqLanes;
    const int64_t col = static_cast<int64_t>(blockIdx.x) * kSqCols + lane * 4;
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (col < n) {   // n % 4 == 0 is required, so a lane's 4 columns are all inside or all outside
        constexpr int kBytes = DT == NVFP4_DT_F32 ? 4 : 2;
        const int64_t step = ld * (kSqGroups * kBytes);   // from a thread's row to its next
        const char* p = static_cast<const char*>(x) + (rg * ld + col) * kBytes;
        // rows rg, rg + 64, ... in ascending order; U loads are issued before the first is consumed
        int64_t left = (m - rg + kSqGroups - 1) / kSqGroups;
        for (; left >= U; left -= U, p += U * step) {
            Quad<DT> q[U];
#pragma unroll
            for (int u = 0; u < U; ++u) q[u].load(p + u * step);
#pragma unroll
            for (int u = 0; u < U; ++u) q[u].add_squares(acc);
        }
        add_rest<DT, U>(p, step, static_cast<int>(left), acc);
    }
    // fixed binary tree over the 64 row groups
    __shared__ float part[kSqGroups][kSqCols];
#pragma unroll
    for (int k = 0; k < 4; ++k) part[rg][lane * 4 + k] = acc[k];
    __syncthreads();
    for (int half = kSqGroups / 2; half >= 1; half >>= 1) {
        for (int idx = threadIdx.x; idx < half * kSqCols; idx += kSqThreads) {
            const int g = idx / kSqCols, c = idx - g * kSqCols;
            part[g][c] = __fadd_rn(part[g][c], part[g + half][c]);
        }
        __syncthreads();
    }
    if (threadIdx.x < kSqCols) {
        const int64_t oc = static_cast<int64_t>(blockIdx.x) * kSqCols + threadIdx.x;
        if (oc < n) out[oc] = part[0][threadIdx.x];
    }
}

// The form by the CTAs an SM gets: up to eight, all of a launch are resident at once in each of them.
// Up to 256 rows (four loads a thread) registers held back for more only keep the next launch's CTAs out.  us, one row at a time beyond the
// last full batch of eight as before / now, 16-bit: 4096 x 1072 7.7 / 6.4, 4013 x 1072 9.3 / 6.3, 4096 x 2048 8.4 / 6.8, 4096 x 4096
// 9.4 / 7.9, 2000 x 5120 7.8 / 6.2, 500 x 8192 5.6 / 4.0, 4096 x 8192 13.7 / 13.7, 4096 x 14336 24.1 / 22.1 (5.3 TB/s by reads); f32: 4096 x
// 1072 12.1 / 6.5, 4096 x 4096 15.2 / 11.6, 4096 x 5120 16.6 / 14.3, 4096 x 8192 21.7 / 21.5, 4096 x 14336 41.3 / 37.5 (6.3 TB/s).  The lines lie where the
// forms cross: 4096 x 4800 in 16 bits, 32 / 16 / 8 loads: 11.1 / 9.9 / 10.0, in f32, 16 / 8 (three CTAs) / 8 (six): 16.2 / 13.3 / 15.6; 4096 x 12288,
// 16 bits, six / eight CTAs 21.6 / 19.8.
template <int DT>
int launch_sqnorm(const void* x, int64_t m, int64_t n, int64_t ld, float* out, unsigned grid, cudaStream_t s) {
    constexpr bool kWide = DT == NVFP4_DT_F32;
    const unsigned per_sm = (grid + kSqSms - 1) / kSqSms;
    if (m <= 256 || per_sm > 5)
        return static_cast<int>(launch_dependent(channel_sqnorm_kernel<DT, kWide ? 4 : 8, 8>, grid, kSqThreads, 0, s, x, m, n, ld, out));
    if (per_sm <= 2)
        return static_cast<int>(launch_dependent(channel_sqnorm_kernel<DT, kWide ? 16 : 32, 2>, grid, kSqThreads, 0, s, x, m, n, ld, out));
    if (kWide && per_sm == 3)
        return static_cast<int>(launch_dependent(channel_sqnorm_kernel<DT, 8, 3>, grid, kSqThreads, 0, s, x, m, n, ld, out));
    return static_cast<int>(launch_dependent(channel_sqnorm_kernel<DT, 8, 6>, grid, kSqThreads, 0, s, x, m, n, ld, out));
}

}  // namespace
}  // namespace nvfp4

extern "C" int nvfp4_channel_sqnorm_launch_strided(const void* x, int x_dtype, int64_t m, int64_t n, int64_t ld, float* out,
                                                   void* stream) {
    using namespace nvfp4;
    if (x_dtype < NVFP4_DT_BF16 || x_dtype > NVFP4_DT_F32) return NVFP4_ERR_BAD_ENUM;
    if (m < 0 || n < 0 || (n % 4) != 0 || ld < n) return NVFP4_ERR_BAD_SHAPE;
    if (n == 0) return NVFP4_OK;
    if (!out || (!x && m > 0)) return NVFP4_ERR_NULL_POINTER;
    // a lane reads 4 consecutive elements (8 or 16 bytes) of a row: the row pitch keeps those pieces aligned
    if ((ld % 4) != 0) return NVFP4_ERR_BAD_SHAPE;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(out) & 3)) return NVFP4_ERR_MISALIGNED;
    const int64_t blocks = (n + kSqCols - 1) / kSqCols;
    if (blocks > 0x7fffffffLL) return NVFP4_ERR_TOO_LARGE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const unsigned g = static_cast<unsigned>(blocks);
    switch (x_dtype) {
        case NVFP4_DT_BF16: return launch_sqnorm<NVFP4_DT_BF16>(x, m, n, ld, out, g, s);
        case NVFP4_DT_F16: return launch_sqnorm<NVFP4_DT_F16>(x, m, n, ld, out, g, s);
        default: return launch_sqnorm<NVFP4_DT_F32>(x, m, n, ld, out, g, s);
    }
}

extern "C" int nvfp4_channel_sqnorm_launch(const void* x, int x_dtype, int64_t m, int64_t n, float* out, void* stream) {
    return nvfp4_channel_sqnorm_launch_strided(x, x_dtype, m, n, n, out, stream);
}
