// The way back from a quantized tensor: packed E2M1 codes and E4M3 block scales to fp32, and scale bytes between the
// 128x4-tiled and the row-major layout.
//
// Behaviour follows efsotr/nvfp4quant_test: helper.py:103-147 (dequantize_base: (code * block scale) * global scale in
// fp32) and kernels/kernel_vllm.py:29-70 (swizzle / unswizzle).
#include <cuda_fp16.h>

#include "common.cuh"

namespace nvfp4 {
namespace {

constexpr int kDqThreads = 256;
constexpr int kDqUnroll = 4;    // 8-element groups per thread, a block's width apart: their loads are in flight together

// Two E2M1 codes -> two fp16 values (exact).
__device__ __forceinline__ __half2 e2m1x2_to_half2(uint32_t byte) {
    uint32_t h;
    asm("{ .reg .b8 b, z1, z2, z3; mov.b32 {b, z1, z2, z3}, %1; cvt.rn.f16x2.e2m1x2 %0, b; }" : "=r"(h) : "r"(byte));
    return *reinterpret_cast<__half2*>(&h);
}

__device__ __forceinline__ void store8(float* p, const float v[8]) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                 "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
}

// out[i] = (code * block scale) * global scale, or the bare code values (SCALED = false).
//
// Bound by the fp32 stores: 4.5625 bytes per element, 4 of them written.  A thread takes 8 elements, one 32-bit word of
// codes in and one 32-byte store out, so every store instruction of a warp is 1 KiB of whole sectors (16-byte stores of
// 16 consecutive elements per thread would touch each sector twice).  code * scale has at most 6 significant bits and is
// exact in fp16, so the product is one packed half multiplication and the only rounding is that of the global scale.
// Scales to row-major plus this kernel, 4096 x 14336: 45.5 us = 5.9 TB/s (the chain of torch operations with its int64
// index temporaries: 1032 us).
template <bool SCALED>
__global__ void __launch_bounds__(kDqThreads) dequant_kernel(const uint32_t* codes, const uint8_t* scales, const float* gs, float* out,
                                                             int64_t groups) {
    griddep_launch();
    griddep_wait();
    codes = after_wait(codes);
    scales = after_wait(scales);
    const float g = SCALED ? load_f32_after_wait(gs) : 1.0f;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * (kDqThreads * kDqUnroll) + threadIdx.x;
    uint32_t w[kDqUnroll], sb[kDqUnroll];
#pragma unroll
    for (int u = 0; u < kDqUnroll; ++u) {
        const int64_t i = first + u * kDqThreads;
        w[u] = i < groups ? __ldg(codes + i) : 0u;
        sb[u] = SCALED && i < groups ? __ldg(scales + (i >> 1)) : 0u;   // two groups share a block of 16
    }
#pragma unroll
    for (int u = 0; u < kDqUnroll; ++u) {
        const int64_t i = first + u * kDqThreads;
        if (i >= groups) break;
        const __half2 s = __float2half2_rn(SCALED ? e4m3_to_f32(sb[u]) : 1.0f);
        float v[8];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const __half2 q = e2m1x2_to_half2((w[u] >> (8 * b)) & 0xffu);
            const float2 f = __half22float2(SCALED ? __hmul2(q, s) : q);
            v[2 * b] = SCALED ? __fmul_rn(f.x, g) : f.x;
            v[2 * b + 1] = SCALED ? __fmul_rn(f.y, g) : f.y;
        }
        store8(out + i * 8, v);
    }
}

// Scale bytes between the tiled layout and row-major [m, k].
//
// A thread owns one 16-byte piece of a tile: four columns of the rows r, r + 32, r + 64, r + 96.  Eight neighbouring lanes
// take the same rows of eight tiles side by side and four such groups take consecutive r, so that a warp moves 64
// consecutive bytes per tile on the tiled side and 32 consecutive bytes per row on the other: whole sectors both ways.
template <bool TO_TILED>
__global__ void __launch_bounds__(kDqThreads) scale_layout_kernel(const uint8_t* src, uint8_t* dst, int64_t m, int64_t k, int64_t k_pad) {
    griddep_launch();
    griddep_wait();
    src = after_wait(src);
    const int64_t col4 = static_cast<int64_t>(blockIdx.x) * 8 + (threadIdx.x & 7);   // tile column
    const int r = threadIdx.x >> 3;                                                  // row of the tile's first quarter
    const int64_t row0 = static_cast<int64_t>(blockIdx.y) * 128 + r;
    if (col4 * 4 >= k_pad) return;
    const int64_t tiled = static_cast<int64_t>(blockIdx.y) * (k_pad * 128) + col4 * 512 + r * 16;
    const int cols = static_cast<int>(min(static_cast<int64_t>(4), k - col4 * 4));   // >= 1: k_pad rounds k up to 4
    const bool words = (k & 3) == 0;
    uint32_t w[4];
    if (TO_TILED) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t row = row0 + 32 * j;
            w[j] = 0u;   // padding rows and columns are zero
            if (row < m) {
                const uint8_t* p = src + row * k + col4 * 4;
                if (words) w[j] = __ldg(reinterpret_cast<const uint32_t*>(p));
                else
                    for (int c = 0; c < cols; ++c) w[j] |= static_cast<uint32_t>(__ldg(p + c)) << (8 * c);
            }
        }
        *reinterpret_cast<uint4*>(dst + tiled) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(src + tiled));
        w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t row = row0 + 32 * j;
            if (row >= m) continue;
            uint8_t* p = dst + row * k + col4 * 4;
            if (words) *reinterpret_cast<uint32_t*>(p) = w[j];
            else
                for (int c = 0; c < cols; ++c) p[c] = static_cast<uint8_t>(w[j] >> (8 * c));
        }
    }
}

}  // namespace
}  // namespace nvfp4

extern "C" int nvfp4_dequant_launch(const uint8_t* codes, const uint8_t* scales, const float* gs, float* out, int64_t m, int64_t n,
                                    void* stream) {
    using namespace nvfp4;
    const bool scaled = scales != nullptr;
    if (m < 0 || n < 0 || (n % (scaled ? kBlock : 8)) != 0) return NVFP4_ERR_BAD_SHAPE;
    if (m == 0 || n == 0) return NVFP4_OK;
    if (!codes || !out || (scaled && !gs)) return NVFP4_ERR_NULL_POINTER;
    if ((reinterpret_cast<uintptr_t>(codes) & 3) || (reinterpret_cast<uintptr_t>(out) & 31) || (reinterpret_cast<uintptr_t>(gs) & 3))
        return NVFP4_ERR_MISALIGNED;
    const int64_t groups = m * n / 8;
    const int64_t blocks = (groups + kDqThreads * kDqUnroll - 1) / (kDqThreads * kDqUnroll);
    if (blocks > 0x7fffffffLL) return NVFP4_ERR_TOO_LARGE;
    const dim3 grid(static_cast<unsigned>(blocks)), block(kDqThreads);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint32_t* words = reinterpret_cast<const uint32_t*>(codes);
    if (scaled) return static_cast<int>(launch_dependent(dequant_kernel<true>, grid, block, 0, s, words, scales, gs, out, groups));
    return static_cast<int>(launch_dependent(dequant_kernel<false>, grid, block, 0, s, words, scales, gs, out, groups));
}

extern "C" int nvfp4_scale_layout_launch(const uint8_t* src, uint8_t* dst, int64_t m, int64_t k, int to_tiled, void* stream) {
    using namespace nvfp4;
    if (m < 0 || k < 0) return NVFP4_ERR_BAD_SHAPE;
    if (m == 0 || k == 0) return NVFP4_OK;
    if (!src || !dst) return NVFP4_ERR_NULL_POINTER;
    const uintptr_t tiled = reinterpret_cast<uintptr_t>(to_tiled ? dst : src), linear = reinterpret_cast<uintptr_t>(to_tiled ? src : dst);
    if ((tiled & 15) || ((k & 3) == 0 && (linear & 3))) return NVFP4_ERR_MISALIGNED;
    const int64_t k_pad = round_up_i64(k, 4), bands = (m + 127) / 128, chunks = (k_pad / 4 + 7) / 8;
    if (bands > 65535 || chunks > 0x7fffffffLL) return NVFP4_ERR_TOO_LARGE;
    const dim3 grid(static_cast<unsigned>(chunks), static_cast<unsigned>(bands)), block(kDqThreads);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (to_tiled) return static_cast<int>(launch_dependent(scale_layout_kernel<true>, grid, block, 0, s, src, dst, m, k, k_pad));
    return static_cast<int>(launch_dependent(scale_layout_kernel<false>, grid, block, 0, s, src, dst, m, k, k_pad));
}
