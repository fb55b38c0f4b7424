// kv_unet_kernels.cuh -- the U-Net's 3x3x3 convolution on warp-level tensor
// cores (BF16 storage, FP32 accumulation), channels-last layout [D][H][W][C]:
// the single-layer operator's kernel for channel counts and alignments that
// the tcgen05 kernel (kv_conv_tc.cuh) does not cover, and its check.
//
// Implicit GEMM (mma.sync m16n8k16, BF16 x BF16 -> FP32): M = voxels, N =
// output channels, K = 27 x input channels; a warp owns 16 consecutive voxels
// of one row and all of its output channels (up to 64), the A fragments come
// straight from the channels-last activations (32-bit loads of channel pairs),
// the B fragments from the [Cout][27][Cin] weights.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

namespace unet {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ uint32_t ld32(const bf16 *p) {
    return __ldg(reinterpret_cast<const unsigned int *>(p));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 3x3x3 convolution, zero padding, optional concatenated second input
// (channels [0,c1) from in1, [c1,c1+c2) from in2), output channels
// [n_off, n_off + 8*NT) of a tensor with c_out_total channels.
// Requires W % 16 == 0, c1 % 16 == 0, c2 % 16 == 0.
template <int NT, bool RELU>
__global__ void __launch_bounds__(128) conv3_fwd(const bf16 *__restrict__ in1, int c1,
                                                 const bf16 *__restrict__ in2, int c2,
                                                 const bf16 *__restrict__ w, const float *__restrict__ bias,
                                                 bf16 *__restrict__ out, int c_out_total, int n_off, int D,
                                                 int H, int W) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long m0 = ((long long)blockIdx.x * 4 + warp) * 16;
    const long long nvox = (long long)D * H * W;
    if (m0 >= nvox) return;
    const int x0 = (int)(m0 % W);
    const long long zy = m0 / W;
    const int y = (int)(zy % H), z = (int)(zy / H);
    const int g = lane >> 2, t = lane & 3;
    const int cin = c1 + c2;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    for (int tap = 0; tap < 27; ++tap) {
        const int zz = z + tap / 9 - 1, yy = y + (tap / 3) % 3 - 1, dx = tap % 3 - 1;
        const bool zy_in = (unsigned)zz < (unsigned)D && (unsigned)yy < (unsigned)H;
        const int xa = x0 + g + dx, xb = xa + 8;
        const bool ina = zy_in && (unsigned)xa < (unsigned)W;
        const bool inb = zy_in && (unsigned)xb < (unsigned)W;
        const long long va = ((long long)zz * H + yy) * W + xa;
        for (int cc = 0; cc < cin; cc += 16) {
            const bf16 *src = cc < c1 ? in1 : in2;
            const int cs = cc < c1 ? c1 : c2;
            const int co = (cc < c1 ? cc : cc - c1) + 2 * t;
            const uint32_t a0 = ina ? ld32(src + va * cs + co) : 0u;
            const uint32_t a1 = inb ? ld32(src + (va + 8) * cs + co) : 0u;
            const uint32_t a2 = ina ? ld32(src + va * cs + co + 8) : 0u;
            const uint32_t a3 = inb ? ld32(src + (va + 8) * cs + co + 8) : 0u;
            const bf16 *wk = w + (size_t)tap * cin + cc + 2 * t;
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const bf16 *wr = wk + (size_t)(n_off + n * 8 + g) * 27 * cin;
                mma_bf16(acc[n], a0, a1, a2, a3, ld32(wr), ld32(wr + 8));
            }
        }
    }
#pragma unroll
    for (int n = 0; n < NT; ++n) {
        const int oc = n_off + n * 8 + 2 * t;
        const float b0 = bias ? bias[oc] : 0.f, b1 = bias ? bias[oc + 1] : 0.f;
        float v0 = acc[n][0] + b0, v1 = acc[n][1] + b1, v2 = acc[n][2] + b0, v3 = acc[n][3] + b1;
        if (RELU) {
            v0 = fmaxf(v0, 0.f);
            v1 = fmaxf(v1, 0.f);
            v2 = fmaxf(v2, 0.f);
            v3 = fmaxf(v3, 0.f);
        }
        *reinterpret_cast<__nv_bfloat162 *>(out + (m0 + g) * c_out_total + oc) = __floats2bfloat162_rn(v0, v1);
        *reinterpret_cast<__nv_bfloat162 *>(out + (m0 + g + 8) * c_out_total + oc) = __floats2bfloat162_rn(v2, v3);
    }
}

}  // namespace unet
