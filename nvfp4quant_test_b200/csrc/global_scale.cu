// Tensor-wide NVFP4 global scale: gs = amax|x| / (6 * fp8_max), gs_inv = 1 / gs.
//
// Follows helper.py:96-100 of efsotr/nvfp4quant_test (get_nvfp4_global_scale) as torch
// evaluates it on a CUDA tensor: a fp32 tensor divided by a host scalar is multiplied by
// the fp32 reciprocal of that scalar, and `.reciprocal()` is an IEEE fp32 division.
//
// One pass over x with 16-byte loads.  The maximum is taken on the magnitude BIT PATTERNS
// (sign cleared, unsigned compare): for non-negative floats that order equals the numeric
// order, and a NaN pattern is larger than +inf, so NaN propagates the way torch's max does.
// Blocks combine through a 2-word scratch (running maximum, arrival counter); the last
// block to arrive publishes the result and leaves the scratch zeroed for the next call.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"

namespace nvfp4 {
namespace {

constexpr int kGsThreads = 256;
constexpr int kGsLoads = 8;   // 16-byte loads in flight per thread

__device__ __forceinline__ uint32_t umax2x16(uint32_t a, uint32_t b) { return __vmaxu2(a, b); }

template <int G>
struct GsParams {
    GsItem item[G];
    unsigned cta_end[G];   // CTAs of this and all earlier tensors
    float fp8_max;
};

template <int DT, int G>
__global__ void __launch_bounds__(kGsThreads) global_scale_kernel(const __grid_constant__ GsParams<G> p) {
    // launched as a programmatic dependent: x, the scratch words and `out` belong to the kernel before this one until
    // it has finished.  The kernel behind this one (the quantizer, which waits before it touches anything) may be
    // scheduled at once.
    griddep_launch();
    griddep_wait();
    int gi = 0;
    if (G > 1) while (blockIdx.x >= p.cta_end[gi]) ++gi;
    const unsigned first = gi > 0 ? p.cta_end[gi - 1] : 0, bx = blockIdx.x - first, ctas = p.cta_end[gi] - first;
    const void* x = p.item[gi].x;
    const int64_t numel = p.item[gi].numel;
    float* const out = p.item[gi].out;
    uint32_t* const scratch = p.item[gi].scratch;
    constexpr int kPerVec = (DT == NVFP4_DT_F32) ? 4 : 8;
    const int64_t nvec = numel / kPerVec;
    x = after_wait(x);   // loads of x stay behind the wait
    const uint4* xv = static_cast<const uint4*>(x);
    uint32_t acc = 0;
    auto fold = [&](const uint4& q) {
        if (DT == NVFP4_DT_F32) {
            acc = max(acc, max(max(q.x & 0x7fffffffu, q.y & 0x7fffffffu), max(q.z & 0x7fffffffu, q.w & 0x7fffffffu)));
        } else {
            acc = umax2x16(acc, umax2x16(umax2x16(q.x & 0x7fff7fffu, q.y & 0x7fff7fffu),
                                         umax2x16(q.z & 0x7fff7fffu, q.w & 0x7fff7fffu)));
        }
    };
    // Chunks of 32 KiB: eight independent 16-byte loads in flight per thread, one contiguous piece per CTA and round (with the
    // grid's width between a thread's loads, 8192 x 8192 bf16 took 23.6 us, now 21.5).
    constexpr int64_t kChunk = static_cast<int64_t>(kGsThreads) * kGsLoads;
    for (int64_t c = bx * kChunk; c < nvec; c += static_cast<int64_t>(ctas) * kChunk) {
        const uint4* const at = xv + c + threadIdx.x;
        uint4 q[kGsLoads];
        if (c + kChunk <= nvec) {
#pragma unroll
            for (int u = 0; u < kGsLoads; ++u) q[u] = __ldg(at + u * kGsThreads);
        } else {   // slots past the end read as zeros, which never raise a maximum of magnitudes
#pragma unroll
            for (int u = 0; u < kGsLoads; ++u)
                q[u] = c + u * kGsThreads + threadIdx.x < nvec ? __ldg(at + u * kGsThreads) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int u = 0; u < kGsLoads; ++u) fold(q[u]);
    }
    // ragged tail (numel not a multiple of the vector width): first threads of block 0
    if (bx == 0) {
        const int64_t t = nvec * kPerVec + threadIdx.x;
        if (t < numel) {
            if (DT == NVFP4_DT_F32) acc = max(acc, static_cast<const uint32_t*>(x)[t] & 0x7fffffffu);
            else acc = umax2x16(acc, static_cast<const uint16_t*>(x)[t] & 0x7fffu);
        }
    }
    uint32_t bits;  // fp32 magnitude pattern of this thread's maximum
    if (DT == NVFP4_DT_F32) {
        bits = acc;
    } else {
        const uint32_t h = max(acc & 0xffffu, acc >> 16);
        if (DT == NVFP4_DT_BF16) bits = h << 16;
        else bits = __float_as_uint(__half2float(__ushort_as_half(static_cast<unsigned short>(h))));
    }
    bits = __reduce_max_sync(0xffffffffu, bits);
    __shared__ uint32_t warp_max[kGsThreads / 32];
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = bits;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t b = 0;
#pragma unroll
        for (int i = 0; i < kGsThreads / 32; ++i) b = max(b, warp_max[i]);
        // a one-block grid (activations of a few tokens) has its maximum already: no trip through the scratch words,
        // whose three dependent atomics would cost more than the rest of the kernel
        bool last = ctas == 1;
        uint32_t mx = b;
        if (!last) {
            atomicMax(&scratch[0], b);
            __threadfence();
            const uint32_t ticket = atomicAdd(&scratch[1], 1u);
            last = ticket == ctas - 1;
            if (last) {
                __threadfence();
                mx = atomicExch(&scratch[0], 0u);
                scratch[1] = 0u;
            }
        }
        if (last) {
            const float amax = __uint_as_float(mx);
            const float inv_den = __fdiv_rn(1.0f, __fmul_rn(6.0f, p.fp8_max));
            const float gs = __fmul_rn(amax, inv_den);
            out[0] = gs;
            out[1] = __fdiv_rn(1.0f, gs);
        }
    }
}

// CTAs for one tensor: one per chunk, at most five per SM (8192 x 8192 bf16, us: two 22.3, three 24.8, four 23.0, five 21.5 =
// 6.2 TB/s, six 22.2; 512-thread CTAs, three per SM and four loads each, 23.6; 128 x 8192 3.8 -> 2.9).  A tensor of one chunk
// stays in one CTA, which needs no atomics.
int64_t gs_ctas(int64_t numel, int x_dtype, int sms) {
    const int64_t nvec = numel / (x_dtype == NVFP4_DT_F32 ? 4 : 8), chunk = kGsThreads * kGsLoads;
    const int64_t blocks = std::min((nvec + chunk - 1) / chunk, static_cast<int64_t>(sms) * 5);
    return blocks < 1 ? 1 : blocks;
}

template <int G>
cudaError_t launch_group(const GsItem* items, int n, int x_dtype, float fp8_max, int sms, cudaStream_t s) {
    GsParams<G> p;
    p.fp8_max = fp8_max;
    unsigned end = 0;
    for (int i = 0; i < n; ++i) {
        p.item[i] = items[i];
        p.cta_end[i] = end += static_cast<unsigned>(gs_ctas(items[i].numel, x_dtype, sms));
    }
    const dim3 grid(end), block(kGsThreads);
    switch (x_dtype) {
        case NVFP4_DT_BF16: return launch_dependent(global_scale_kernel<NVFP4_DT_BF16, G>, grid, block, 0, s, p);
        case NVFP4_DT_F16: return launch_dependent(global_scale_kernel<NVFP4_DT_F16, G>, grid, block, 0, s, p);
        default: return launch_dependent(global_scale_kernel<NVFP4_DT_F32, G>, grid, block, 0, s, p);
    }
}

}  // namespace

int check_global_scale(const GsItem& item, int x_dtype) {
    if (x_dtype < NVFP4_DT_BF16 || x_dtype > NVFP4_DT_F32) return NVFP4_ERR_BAD_ENUM;
    if (item.numel < 0) return NVFP4_ERR_BAD_SHAPE;
    if (!item.out || !item.scratch || (!item.x && item.numel > 0)) return NVFP4_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(item.x) & 15) || (reinterpret_cast<uintptr_t>(item.out) & 3) ||
        (reinterpret_cast<uintptr_t>(item.scratch) & 3))
        return NVFP4_ERR_MISALIGNED;
    return NVFP4_OK;
}

int launch_global_scales(const GsItem* items, int n, int x_dtype, float fp8_max, cudaStream_t stream) {
    static int sm_count[64] = {0};
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        if (sm_count[dev] == 0) cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev);
        if (sm_count[dev] > 0) sms = sm_count[dev];
    }
    return static_cast<int>(n == 1 ? launch_group<1>(items, n, x_dtype, fp8_max, sms, stream)
                                   : launch_group<4>(items, n, x_dtype, fp8_max, sms, stream));
}

}  // namespace nvfp4

extern "C" int nvfp4_global_scale_launch(const void* x, int x_dtype, int64_t numel, float fp8_max, float* out,
                                         uint32_t* scratch, void* stream) {
    const nvfp4::GsItem item = {x, numel, out, scratch};
    const int st = nvfp4::check_global_scale(item, x_dtype);
    return st != NVFP4_OK ? st : nvfp4::launch_global_scales(&item, 1, x_dtype, fp8_max, static_cast<cudaStream_t>(stream));
}
