// kv_unet.cu -- learned warm start: a small 3D U-Net (4 levels, 16/32/64/128
// channels, 3x3x3 convolutions, BF16 weights and activations, FP32
// accumulation) that maps a shift-and-add volume to an MLEM initial estimate,
// with its own training step (backpropagation + Adam).  No reference
// counterpart.
//
// Network (channels-last BF16 activations, D x H x W voxels, W % 128 == 0 for
// the 16-voxel rows of the coarsest level):
//   a0 = relu(conv(x: 1 -> 16))      e1 = relu(conv(a0: 16 -> 16))
//   a2 = relu(conv(pool(e1) -> 32))  e2 = relu(conv(a2: 32 -> 32))
//   a4 = relu(conv(pool(e2) -> 64))  e3 = relu(conv(a4: 64 -> 64))
//   a6 = relu(conv(pool(e3) -> 128)) b  = relu(conv(a6: 128 -> 128))
//   a8 = relu(conv(up(b) ++ e3 -> 64))   d3 = relu(conv(a8 -> 64))
//   a10 = relu(conv(up(d3) ++ e2 -> 32)) d2 = relu(conv(a10 -> 32))
//   a12 = relu(conv(up(d2) ++ e1 -> 16)) d1 = relu(conv(a12 -> 16))
//   y = x + conv1x1(d1: 16 -> 1)     (FP32 output)
// pool = 2x2x2 average, up = nearest x2, ++ = channel concatenation (read in
// place by the convolution, never copied).
#include "kv_conv_tc.cuh"
#include "kv_internal.h"
#include "kv_unet_kernels.cuh"
#include "kv_wgrad_tc.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>

using unet::bf16;

namespace {

// ---------------------------------------------------------------- kernels

// Eight BF16 channels as one 16-byte access; every per-channel kernel below
// moves them so (scalar BF16 accesses kept these passes at a third of the
// memory rate).
struct __align__(16) Bf8 {
    __nv_bfloat162 v[4];
};

__device__ __forceinline__ Bf8 ld8(const bf16 *p) {
    const uint4 u = __ldg(reinterpret_cast<const uint4 *>(p));
    return *reinterpret_cast<const Bf8 *>(&u);
}

__device__ __forceinline__ void st8(bf16 *p, const Bf8 &b) {
    *reinterpret_cast<uint4 *>(p) = *reinterpret_cast<const uint4 *>(&b);
}

__device__ __forceinline__ void unpack8(const Bf8 &b, float (&f)[8]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 t = __bfloat1622float2(b.v[j]);
        f[2 * j] = t.x;
        f[2 * j + 1] = t.y;
    }
}

__device__ __forceinline__ Bf8 pack8(const float (&f)[8]) {
    Bf8 b;
#pragma unroll
    for (int j = 0; j < 4; ++j) b.v[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
    return b;
}

// First layer, 1 -> 16 channels in FP32.  432 multiply-adds a voxel bound it
// (0.39 ms of FP32 issue at 128 x 512 x 512 voxels, 0.18 ms of memory), so a
// thread computes kFirstRows voxels of consecutive y in packed arithmetic: the
// weights, in shared memory, are read once for all of them, and their rows
// overlap.  One voxel a thread with the weights in global memory took 2.19 ms;
// four rows 0.79 (0.94 with scalar fmaf), two rows, which leave registers for
// more warps, and 32-byte stores 0.75.  Blocks of 128 x.
constexpr int kFirstRows = 2;

__global__ void __launch_bounds__(128) conv_first_fwd(const float *__restrict__ x, const float *__restrict__ w /*[16][27]*/,
                                                      const float *__restrict__ b, bf16 *__restrict__ out, int D, int H,
                                                      int W) {
    __shared__ __align__(16) float ws[27][16];
    __shared__ __align__(16) float bs[16];
    for (int i = threadIdx.x; i < 432; i += blockDim.x) ws[i % 27][i / 27] = w[i];
    if (threadIdx.x < 16) bs[threadIdx.x] = b[threadIdx.x];
    __syncthreads();
    const int xx = blockIdx.x * 128 + threadIdx.x;   // W % 128 == 0, H % 8 == 0
    const int rows = H / kFirstRows;
    for (long long zy = blockIdx.y; zy < (long long)D * rows; zy += gridDim.y) {
        const int z = (int)(zy / rows), y0 = (int)(zy % rows) * kFirstRows;
        // two channels a register pair: fma.rn.f32x2 rounds each half as fmaf does and takes one issue slot for both
        unsigned long long acc[kFirstRows][8];
#pragma unroll
        for (int r = 0; r < kFirstRows; ++r)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[r][c] = *reinterpret_cast<const unsigned long long *>(&bs[2 * c]);
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            const int zz = z + dz - 1;
            unsigned long long in[kFirstRows + 2][3];
#pragma unroll
            for (int r = 0; r < kFirstRows + 2; ++r)
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    const int yy = y0 + r - 1, x2 = xx + dx - 1;
                    const bool ok = (unsigned)zz < (unsigned)D && (unsigned)yy < (unsigned)H && (unsigned)x2 < (unsigned)W;
                    const float f = ok ? __ldg(x + ((size_t)zz * H + yy) * W + x2) : 0.f;
                    asm("mov.b64 %0, {%1, %1};" : "=l"(in[r][dx]) : "f"(f));
                }
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                unsigned long long wv[8];
#pragma unroll
                for (int c = 0; c < 8; c += 2)
                    *reinterpret_cast<ulonglong2 *>(wv + c) = *reinterpret_cast<const ulonglong2 *>(&ws[dz * 9 + t][2 * c]);
#pragma unroll
                for (int r = 0; r < kFirstRows; ++r)
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[r][c]) : "l"(wv[c]), "l"(in[r + t / 3][t % 3]));
            }
        }
#pragma unroll
        for (int r = 0; r < kFirstRows; ++r) {
            bf16 *dst = out + (((size_t)z * H + y0 + r) * W + xx) * 16;
            Bf8 o[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float f[8];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(f[2 * c]), "=f"(f[2 * c + 1]) : "l"(acc[r][4 * h + c]));
                    f[2 * c] = fmaxf(f[2 * c], 0.f);
                    f[2 * c + 1] = fmaxf(f[2 * c + 1], 0.f);
                }
                o[h] = pack8(f);
            }
            convtc::st32(dst, *reinterpret_cast<const uint4 *>(&o[0]), *reinterpret_cast<const uint4 *>(&o[1]));
        }
    }
}

// Sums v over the block (blockDim.x threads, a multiple of 32, at most 512) and adds the total to *dst.
__device__ __forceinline__ void block_add(float v, float *dst, float *sh /* [16] */) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += sh[i];
        atomicAdd(dst, t);
    }
}

// dW0[c][tap] += sum_v dpre[v][c] * x[v + tap] for the nine taps of one dz (blockIdx.y) and eight channels
// (blockIdx.z): 72 sums a thread in packed FP32, over four voxels of consecutive y at a time, whose 18 x values and
// four 16-byte gradients are all in flight together.  All 16 channels of one voxel a thread (250 registers, one block
// a SM, a load latency a voxel) took 341 us at 128 x 256 x 128 voxels, one tap a pass 1244; this takes 167.  The bias
// gradient comes with dz = 1.
__global__ void __launch_bounds__(256, 2) conv_first_wgrad(const float *__restrict__ x, const bf16 *__restrict__ dpre,
                                                           float *__restrict__ dw, float *__restrict__ db, int D, int H,
                                                           int W) {
    __shared__ float part[8][9][8];
    const int dz = blockIdx.y, c0 = 8 * blockIdx.z, h4 = H / 4;   // H % 8 == 0
    const long long n = (long long)D * h4 * W;
    unsigned long long acc[9][4];
    float accb[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) accb[c] = 0.f;
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[t][c] = 0ull;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const int xx = (int)(v % W);
        const long long zy = v / W;
        const int y0 = (int)(zy % h4) * 4, z = (int)(zy / h4), zz = z + dz - 1;
        Bf8 g[4];
        float in[6][3];
#pragma unroll
        for (int r = 0; r < 4; ++r) g[r] = ld8(dpre + (((size_t)z * H + y0 + r) * W + xx) * 16 + c0);
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                const int yy = y0 + r - 1, x2 = xx + dx - 1;
                const bool ok = (unsigned)zz < (unsigned)D && (unsigned)yy < (unsigned)H && (unsigned)x2 < (unsigned)W;
                in[r][dx] = ok ? __ldg(x + ((size_t)zz * H + yy) * W + x2) : 0.f;
            }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            unsigned long long gp[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 f = __bfloat1622float2(g[r].v[c]);
                if (dz == 1) {
                    accb[2 * c] += f.x;
                    accb[2 * c + 1] += f.y;
                }
                asm("mov.b64 %0, {%1, %2};" : "=l"(gp[c]) : "f"(f.x), "f"(f.y));
            }
#pragma unroll
            for (int t = 0; t < 9; ++t) {
                unsigned long long xv;
                asm("mov.b64 %0, {%1, %1};" : "=l"(xv) : "f"(in[r + t / 3][t % 3]));
#pragma unroll
                for (int c = 0; c < 4; ++c) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[t][c]) : "l"(gp[c]), "l"(xv));
            }
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto warp_sum = [](float f) {
        for (int o = 16; o > 0; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
        return f;
    };
#pragma unroll
    for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            float a, b;
            asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(acc[t][c]));
            a = warp_sum(a);
            b = warp_sum(b);
            if (lane == 0) {
                part[warp][t][2 * c] = a;
                part[warp][t][2 * c + 1] = b;
            }
        }
    __syncthreads();
    if (threadIdx.x < 72) {
        const int t = threadIdx.x / 8, c = threadIdx.x % 8;
        float f = 0.f;
        for (int i = 0; i < 8; ++i) f += part[i][t][c];
        atomicAdd(dw + (c0 + c) * 27 + dz * 9 + t, f);
    }
    if (dz != 1) return;
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const float f = warp_sum(accb[c]);
        if (lane == 0) part[warp][0][c] = f;
    }
    __syncthreads();
    if (threadIdx.x < 8) {
        float f = 0.f;
        for (int i = 0; i < 8; ++i) f += part[i][0][threadIdx.x];
        atomicAdd(db + c0 + threadIdx.x, f);
    }
}

// loss partials: sum (y - t)^2 per block; dy = 2 (y - t) / n.  A NaN target
// marks a voxel without a target: it adds nothing to the loss or gradient.
__global__ void mse_loss(const float *__restrict__ y, const float *__restrict__ t, float *__restrict__ dy, long long n,
                         double *__restrict__ partials) {
    double s = 0.0;
    const float scale = 2.f / (float)n;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const float tv = t[v];
        if (tv != tv) {
            dy[v] = 0.f;
            continue;
        }
        const float d = y[v] - tv;
        s += (double)d * (double)d;
        dy[v] = scale * d;
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    __shared__ double sh[32];
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += sh[i];
        partials[blockIdx.x] = tot;
    }
}

__global__ void __launch_bounds__(256) sum_loss(const double *__restrict__ partials, int nb, long long n,
                                                float *__restrict__ out) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int i = threadIdx.x; i < nb; i += 256) s += partials[i];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[0] = (float)(sh[0] / (double)n);
}

// backward of the output layer: dh[v][c] = w[c] dy[v] where h > 0 (the ReLU of the layer before), else 0; dw[c] += sum
// dy h; db += sum dy
__global__ void __launch_bounds__(256) conv_out_bwd(const bf16 *__restrict__ h, const float *__restrict__ dy,
                                                    const float *__restrict__ w, bf16 *__restrict__ dh,
                                                    float *__restrict__ dw, float *__restrict__ db, long long n) {
    __shared__ float sh[16];
    float acc[16], wv[16], accb = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        acc[c] = 0.f;
        wv[c] = w[c];
    }
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const float g = dy[v];
        accb += g;
        Bf8 o[2];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            float hv[8], d[8];
            unpack8(ld8(h + v * 16 + 8 * q), hv);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                acc[8 * q + c] = fmaf(g, hv[c], acc[8 * q + c]);
                d[c] = hv[c] > 0.f ? wv[8 * q + c] * g : 0.f;
            }
            o[q] = pack8(d);
        }
        convtc::st32(dh + v * 16, *reinterpret_cast<const uint4 *>(&o[0]), *reinterpret_cast<const uint4 *>(&o[1]));
    }
#pragma unroll
    for (int c = 0; c < 16; ++c) block_add(acc[c], dw + c, sh);
    block_add(accb, db, sh);
}

// 2x2x2 average pool (channels-last), out dims D/2 x H/2 x W/2
__global__ void avgpool_fwd(const bf16 *__restrict__ in, bf16 *__restrict__ out, int D, int H, int W, int C) {
    const int d2 = D / 2, h2 = H / 2, w2 = W / 2, c8 = C / 8;
    const long long n = (long long)d2 * h2 * w2 * c8;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(e % c8) * 8;
        const long long v = e / c8;
        const int x = (int)(v % w2);
        const long long zy = v / w2;
        const int y = (int)(zy % h2), z = (int)(zy / h2);
        float s[8] = {};
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const long long src = ((long long)(2 * z + (k >> 2)) * H + (2 * y + ((k >> 1) & 1))) * W + 2 * x + (k & 1);
            float f[8];
            unpack8(ld8(in + src * C + c), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += f[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] *= 0.125f;
        st8(out + v * C + c, pack8(s));
    }
}

// de[v][c] = (relu mask) * (dp[parent(v)][c] / 8 + dcat[v][c_off + c]) -- the gradient of an encoder output
// e = relu(...) from its pool and its skip connection, already masked by e > 0
__global__ void pool_bwd_skip_mask(const bf16 *__restrict__ dp, const bf16 *__restrict__ dcat, int ccat, int c_off,
                                   const bf16 *__restrict__ e, bf16 *__restrict__ de, int D, int H, int W, int C) {
    const int c8 = C / 8;
    const long long n = (long long)D * H * W * c8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i % c8) * 8;
        const long long v = i / c8;
        const int x = (int)(v % W);
        const long long zy = v / W;
        const int y = (int)(zy % H), z = (int)(zy / H);
        const long long pv = ((long long)(z / 2) * (H / 2) + y / 2) * (W / 2) + x / 2;
        float p[8], k[8], m[8];
        unpack8(ld8(dp + pv * C + c), p);
        unpack8(ld8(dcat + v * ccat + c_off + c), k);
        unpack8(ld8(e + v * C + c), m);
#pragma unroll
        for (int j = 0; j < 8; ++j) p[j] = m[j] > 0.f ? 0.125f * p[j] + k[j] : 0.f;
        st8(de + v * C + c, pack8(p));
    }
}

// nearest x2 upsampling (channels-last): out D x H x W from in D/2 x H/2 x W/2; a thread writes the four children of one
// x, so that a warp writes consecutive voxels
__global__ void upsample_fwd(const bf16 *__restrict__ in, bf16 *__restrict__ out, int D, int H, int W, int C) {
    const int c8 = C / 8, w2 = W / 2, h2 = H / 2;
    const long long n = (long long)(D / 2) * h2 * W * c8;   // a thread: one x, the four (z, y) children
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(e % c8) * 8;
        const long long v = e / c8;
        const int x = (int)(v % W);
        const long long zy = v / W;
        const int y = (int)(zy % h2), z = (int)(zy / h2);
        const Bf8 val = ld8(in + (((long long)z * h2 + y) * w2 + x / 2) * C + c);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            st8(out + (((long long)(2 * z + (k >> 1)) * H + 2 * y + (k & 1)) * W + x) * C + c, val);
    }
}

// gradient through up(): dlow[p][c] = sum of the 8 children dcat[child][c] (channels [0,C) of a
// tensor with ccat channels), then masked by the relu output `a` of the low level
__global__ void upsample_bwd_mask(const bf16 *__restrict__ dcat, int ccat, const bf16 *__restrict__ a,
                                  bf16 *__restrict__ dlow, int D, int H, int W, int C) {
    // D, H, W: the low (half) resolution
    const int c8 = C / 8;
    const long long n = (long long)D * H * W * c8;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const int c = (int)(i % c8) * 8;
        const long long v = i / c8;
        const int x = (int)(v % W);
        const long long zy = v / W;
        const int y = (int)(zy % H), z = (int)(zy / H);
        float s[8] = {}, m[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const long long ch = ((long long)(2 * z + (k >> 2)) * (2 * H) + (2 * y + ((k >> 1) & 1))) * (2 * W) + 2 * x + (k & 1);
            float f[8];
            unpack8(ld8(dcat + ch * ccat + c), f);
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] += f[j];
        }
        unpack8(ld8(a + v * C + c), m);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (!(m[j] > 0.f)) s[j] = 0.f;
        st8(dlow + v * C + c, pack8(s));
    }
}

// db[c] += sum_v g[v][c].  A thread keeps eight channels (the stride is a multiple of C / 8) and sums them in
// registers; C is 16, 32, 64 or 128.  Shared-memory atomics for every element took 0.96 ms over the thirteen layers
// at 128 x 256 x 128 voxels.
__global__ void __launch_bounds__(256) bias_grad(const bf16 *__restrict__ g, float *__restrict__ db, long long nvox, int C) {
    __shared__ float sb[8][128];
    const int c8 = C / 8;
    const long long n = nvox * c8, stride = (long long)gridDim.x * blockDim.x;
    float s[8] = {};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride) {
        float f[8];
        unpack8(ld8(g + i * 8), f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        for (int o = 16; o >= c8; o >>= 1) s[j] += __shfl_xor_sync(0xffffffffu, s[j], o);
        if (lane < c8) sb[warp][lane * 8 + j] = s[j];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        float t = 0.f;
        for (int w = 0; w < 8; ++w) t += sb[w][c];
        atomicAdd(db + c, t);
    }
}

// Wt[ci][26 - tap][co] = W[co][tap][ci]: backward-data weights of every layer in one launch (blockIdx.y: layer)
struct FlipTable {
    int w[13], cout[13], cin[13];
};

__global__ void flip_transpose(const bf16 *__restrict__ pw, bf16 *__restrict__ pwt, FlipTable T) {
    const int l = blockIdx.y, cout = T.cout[l], cin = T.cin[l], n = cout * 27 * cin;
    const bf16 *w = pw + T.w[l];
    bf16 *wt = pwt + T.w[l];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int co = i % cout, t = (i / cout) % 27, ci = i / (27 * cout);
        wt[i] = w[((size_t)co * 27 + (26 - t)) * cin + ci];
    }
}

// Adam on the FP32 master parameters; refreshes the BF16 copies
__global__ void adam_step(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                          float *__restrict__ v, bf16 *__restrict__ pb, size_t n, float lr, float b1, float b2,
                          float eps, const float *__restrict__ corr /* 1 - b1^t, 1 - b2^t */) {
    const float c1 = corr[0], c2 = corr[1];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
        p[i] = pi;
        pb[i] = __float2bfloat16_rn(pi);
    }
}

__global__ void to_bf16(const float *__restrict__ in, bf16 *__restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = __float2bfloat16_rn(in[i]);
}

}  // namespace

// ------------------------------------------------------------------ model

struct kv_unet {
    kv_ctx *ctx = nullptr;
    // parameter layout
    struct Conv {
        int c1, c2, cout;
        size_t w, b;   // offsets into the flat parameter buffer
    };
    Conv conv[14];
    size_t w_first = 0, b_first = 0, w_out = 0, b_out = 0, nparams = 0;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;   // FP32 master, grads, Adam moments
    bf16 *pb = nullptr;                                             // BF16 copy of the parameters
    bf16 *wt = nullptr;                                             // flipped / transposed weights
    long long step = 0;
    // activation workspace for one shape
    int D = 0, H = 0, W = 0;
    bool with_grads = false;
    std::vector<void *> bufs;
    bf16 *act[24] = {};
    bf16 *grad[24] = {};
    float *x = nullptr, *t = nullptr, *y = nullptr, *dy = nullptr, *loss = nullptr;
    double *partials = nullptr;
    float *corr = nullptr;                                          // Adam bias corrections (device)
    int *tc_status = nullptr;                                       // tensor-core convolution wait status
    cudaGraphExec_t train_graph = nullptr;
    float graph_lr = 0.f;
};

namespace {

enum {
    A0, E1, P1, A2, E2, P2, A4, E3, P3, A6, B, U3, A8, D3, U2, A10, D2, U1, A12, D1, CAT3, CAT2, CAT1, NACT
};

int grid_n(kv_ctx *ctx, long long n, int block = 256) {
    long long g = (n + block - 1) / block, cap = (long long)ctx->sm_count * 16;
    return (int)(g < cap ? (g < 1 ? 1 : g) : cap);
}

void free_workspace(kv_unet *u) {
    if (u->train_graph) cudaGraphExecDestroy(u->train_graph);
    u->train_graph = nullptr;
    for (void *b : u->bufs) cudaFree(b);
    u->bufs.clear();
    for (int i = 0; i < 24; ++i) u->act[i] = u->grad[i] = nullptr;
    u->x = u->t = u->y = u->dy = u->loss = nullptr;
    u->partials = nullptr;
    u->D = u->H = u->W = 0;
}

kv_status alloc(kv_unet *u, void **p, size_t bytes) {
    if (cudaMalloc(p, bytes) != cudaSuccess) {
        cudaGetLastError();
        return kv_fail(u->ctx, KV_ERR_OOM, "U-Net workspace (%zu bytes)", bytes);
    }
    u->bufs.push_back(*p);
    return KV_OK;
}

// channel count and resolution level (0 = full) of each activation
void act_shape(int i, int &c, int &lvl) {
    static const int C[NACT] = {16, 16, 16, 32, 32, 32, 64, 64, 64, 128, 128, 128, 64, 64, 64, 32, 32, 32, 16, 16, 192, 96, 48};
    static const int L[NACT] = {0, 0, 1, 1, 1, 2, 2, 2, 3, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0, 2, 1, 0};
    c = C[i];
    lvl = L[i];
}

kv_status ensure_workspace(kv_unet *u, int D, int H, int W, bool grads) {
    if (u->D == D && u->H == H && u->W == W && (u->with_grads || !grads)) return KV_OK;
    free_workspace(u);
    if (D % 8 || H % 8 || W % 128)
        return kv_fail(u->ctx, KV_ERR_INVALID_ARG, "U-Net input must be D, H multiples of 8 and W of 128 (got %d x %d x %d)",
                       D, H, W);
    const long long n0 = (long long)D * H * W;
    for (int i = 0; i < NACT; ++i) {
        int c, l;
        act_shape(i, c, l);
        const long long nv = n0 >> (3 * l);
        if (i >= CAT3 && !grads) continue;   // concatenation gradients: training only
        KV_TRY(alloc(u, (void **)&u->act[i], (size_t)nv * c * sizeof(bf16)));
        if (grads) KV_TRY(alloc(u, (void **)&u->grad[i], (size_t)nv * c * sizeof(bf16)));
    }
    KV_TRY(alloc(u, (void **)&u->x, n0 * sizeof(float)));
    KV_TRY(alloc(u, (void **)&u->y, n0 * sizeof(float)));
    if (grads) {
        KV_TRY(alloc(u, (void **)&u->t, n0 * sizeof(float)));
        KV_TRY(alloc(u, (void **)&u->dy, n0 * sizeof(float)));
        KV_TRY(alloc(u, (void **)&u->loss, sizeof(float) * 4));
        KV_TRY(alloc(u, (void **)&u->partials, sizeof(double) * 4096));
    }
    u->D = D;
    u->H = H;
    u->W = W;
    u->with_grads = grads;
    return KV_OK;
}

// forward or backward-data convolution of one layer
kv_status conv3(kv_unet *u, int layer, const bf16 *in1, const bf16 *in2, bf16 *out, int lvl, bool weights_t,
                const bf16 *mask = nullptr, const convtc::Head *head = nullptr) {
    const kv_unet::Conv &L = u->conv[layer];
    kv_ctx *ctx = u->ctx;
    const int D = u->D >> lvl, H = u->H >> lvl, W = u->W >> lvl;
    // forward: in1 (c1) ++ in2 (c2) -> cout with W; backward-data: in1 = dPre (cout) -> c1 + c2 with Wt
    const int c1 = weights_t ? L.cout : L.c1, c2 = weights_t ? 0 : L.c2;
    const int cout = weights_t ? L.c1 + L.c2 : L.cout;
    const bf16 *w = weights_t ? u->wt + L.w : u->pb + L.w;
    const float *bias = weights_t ? nullptr : u->p + L.b;
    LaunchTimer lt(ctx, weights_t ? "unet_conv_dgrad" : "unet_conv_fwd");
    // tcgen05 / TMA implicit GEMM (kv_conv_tc.cuh); covers every level of every volume the network takes
    const char *why = convtc::launch(in1, c1, in2, c2, w, bias, !weights_t, mask, head, out, cout, D, H, W, false,
                                     u->tc_status, ctx->sm_count, ctx->stream);
    if (why != nullptr) return kv_fail(ctx, KV_ERR_UNSUPPORTED, "tensor-core convolution: %s", why);
    KV_CHECK_LAUNCH(ctx, "unet conv3 (tcgen05)");
    return KV_OK;
}

kv_status wgrad(kv_unet *u, int layer, const bf16 *dpre, const bf16 *in1, const bf16 *in2, int lvl) {
    const kv_unet::Conv &L = u->conv[layer];
    kv_ctx *ctx = u->ctx;
    const int D = u->D >> lvl, H = u->H >> lvl, W = u->W >> lvl;
    const long long nvox = (long long)D * H * W;
    {
        LaunchTimer lt(ctx, "unet_conv_wgrad");
        const char *why = wgradtc::launch(dpre, L.cout, in1, L.c1, in2, L.c2, u->g + L.w, D, H, W, u->tc_status,
                                          ctx->sm_count, ctx->stream);
        if (why != nullptr) return kv_fail(ctx, KV_ERR_UNSUPPORTED, "weight gradient: %s", why);
    }
    {
        LaunchTimer lb(ctx, "unet_bias_grad");
        bias_grad<<<std::min(grid_n(ctx, nvox * (L.cout / 8)), 4 * ctx->sm_count), 256, 0, ctx->stream>>>(dpre, u->g + L.b, nvox, L.cout);
    }
    KV_CHECK_LAUNCH(ctx, "unet wgrad");
    return KV_OK;
}

kv_status forward(kv_unet *u, bool keep) {
    kv_ctx *ctx = u->ctx;
    const int D = u->D, H = u->H, W = u->W;
    const long long n0 = (long long)D * H * W;
    bf16 **a = u->act;
    {
        LaunchTimer lt(ctx, "unet_conv_first");
        conv_first_fwd<<<dim3(W / 128, (unsigned)std::min<long long>((long long)D * (H / kFirstRows), 65535)), 128, 0, ctx->stream>>>(u->x, u->p + u->w_first, u->p + u->b_first, a[A0], D, H, W);
    }
    KV_TRY(conv3(u, 0, a[A0], nullptr, a[E1], 0, false));
    avgpool_fwd<<<grid_n(ctx, (n0 >> 3) * 2), 256, 0, ctx->stream>>>(a[E1], a[P1], D, H, W, 16);
    KV_TRY(conv3(u, 1, a[P1], nullptr, a[A2], 1, false));
    KV_TRY(conv3(u, 2, a[A2], nullptr, a[E2], 1, false));
    avgpool_fwd<<<grid_n(ctx, (n0 >> 6) * 4), 256, 0, ctx->stream>>>(a[E2], a[P2], D >> 1, H >> 1, W >> 1, 32);
    KV_TRY(conv3(u, 3, a[P2], nullptr, a[A4], 2, false));
    KV_TRY(conv3(u, 4, a[A4], nullptr, a[E3], 2, false));
    avgpool_fwd<<<grid_n(ctx, (n0 >> 9) * 8), 256, 0, ctx->stream>>>(a[E3], a[P3], D >> 2, H >> 2, W >> 2, 64);
    KV_TRY(conv3(u, 5, a[P3], nullptr, a[A6], 3, false));
    KV_TRY(conv3(u, 6, a[A6], nullptr, a[B], 3, false));
    upsample_fwd<<<grid_n(ctx, (n0 >> 8) * 16), 256, 0, ctx->stream>>>(a[B], a[U3], D >> 2, H >> 2, W >> 2, 128);
    KV_TRY(conv3(u, 7, a[U3], a[E3], a[A8], 2, false));
    KV_TRY(conv3(u, 8, a[A8], nullptr, a[D3], 2, false));
    upsample_fwd<<<grid_n(ctx, (n0 >> 5) * 8), 256, 0, ctx->stream>>>(a[D3], a[U2], D >> 1, H >> 1, W >> 1, 64);
    KV_TRY(conv3(u, 9, a[U2], a[E2], a[A10], 1, false));
    KV_TRY(conv3(u, 10, a[A10], nullptr, a[D2], 1, false));
    upsample_fwd<<<grid_n(ctx, (n0 >> 2) * 4), 256, 0, ctx->stream>>>(a[D2], a[U1], D, H, W, 32);
    KV_TRY(conv3(u, 11, a[U1], a[E1], a[A12], 0, false));
    // the output layer reads the last layer's voxels where they are computed; D1 itself is kept for the backward pass
    const convtc::Head head{u->p + u->w_out, u->p + u->b_out, u->x, u->y};
    KV_TRY(conv3(u, 12, a[A12], nullptr, keep ? a[D1] : nullptr, 0, false, nullptr, &head));
    KV_CHECK_LAUNCH(ctx, "unet forward");
    return KV_OK;
}

// backward of a conv + relu layer whose output gradient (already masked by
// the layer's relu) is dpre: weight / bias gradients and the input gradient
// into dx, zero where `mask` (the relu output it is the gradient of, when in1 is one) is not positive
kv_status conv_backward(kv_unet *u, int layer, const bf16 *dpre, const bf16 *in1, const bf16 *in2, bf16 *dx, int lvl,
                        const bf16 *mask = nullptr) {
    KV_TRY(wgrad(u, layer, dpre, in1, in2, lvl));
    return conv3(u, layer, dpre, nullptr, dx, lvl, true, mask);
}

kv_status backward(kv_unet *u) {
    kv_ctx *ctx = u->ctx;
    const int D = u->D, H = u->H, W = u->W;
    const long long n0 = (long long)D * H * W;
    bf16 **a = u->act, **g = u->grad;
    // weights for the backward-data convolutions
    FlipTable flip;
    for (int l = 0; l < 13; ++l) {
        flip.w[l] = (int)u->conv[l].w;
        flip.cout[l] = u->conv[l].cout;
        flip.cin[l] = u->conv[l].c1 + u->conv[l].c2;
    }
    flip_transpose<<<dim3(4 * ctx->sm_count / 13 + 1, 13), 256, 0, ctx->stream>>>(u->pb, u->wt, flip);
    // output layer
    conv_out_bwd<<<std::min(grid_n(ctx, n0), 4 * ctx->sm_count), 256, 0, ctx->stream>>>(a[D1], u->dy, u->p + u->w_out, g[D1], u->g + u->w_out,
                                                           u->g + u->b_out, n0);
    // level 0 decoder
    KV_TRY(conv_backward(u, 12, g[D1], a[A12], nullptr, g[A12], 0, a[A12]));
    KV_TRY(conv_backward(u, 11, g[A12], a[U1], a[E1], g[CAT1], 0));      // 48 ch: up(d2) 32 ++ e1 16
    upsample_bwd_mask<<<grid_n(ctx, (n0 >> 3) * 4), 256, 0, ctx->stream>>>(g[CAT1], 48, a[D2], g[D2], D >> 1, H >> 1, W >> 1, 32);
    // level 1 decoder
    KV_TRY(conv_backward(u, 10, g[D2], a[A10], nullptr, g[A10], 1, a[A10]));
    KV_TRY(conv_backward(u, 9, g[A10], a[U2], a[E2], g[CAT2], 1));       // 96 ch: up(d3) 64 ++ e2 32
    upsample_bwd_mask<<<grid_n(ctx, (n0 >> 6) * 8), 256, 0, ctx->stream>>>(g[CAT2], 96, a[D3], g[D3], D >> 2, H >> 2, W >> 2, 64);
    // level 2 decoder
    KV_TRY(conv_backward(u, 8, g[D3], a[A8], nullptr, g[A8], 2, a[A8]));
    KV_TRY(conv_backward(u, 7, g[A8], a[U3], a[E3], g[CAT3], 2));        // 192 ch: up(b) 128 ++ e3 64
    upsample_bwd_mask<<<grid_n(ctx, (n0 >> 9) * 16), 256, 0, ctx->stream>>>(g[CAT3], 192, a[B], g[B], D >> 3, H >> 3, W >> 3, 128);
    // bottleneck
    KV_TRY(conv_backward(u, 6, g[B], a[A6], nullptr, g[A6], 3, a[A6]));
    KV_TRY(conv_backward(u, 5, g[A6], a[P3], nullptr, g[P3], 3));
    pool_bwd_skip_mask<<<grid_n(ctx, (n0 >> 6) * 8), 256, 0, ctx->stream>>>(g[P3], g[CAT3], 192, 128, a[E3], g[E3],
                                                                             D >> 2, H >> 2, W >> 2, 64);
    // level 2 encoder
    KV_TRY(conv_backward(u, 4, g[E3], a[A4], nullptr, g[A4], 2, a[A4]));
    KV_TRY(conv_backward(u, 3, g[A4], a[P2], nullptr, g[P2], 2));
    pool_bwd_skip_mask<<<grid_n(ctx, (n0 >> 3) * 4), 256, 0, ctx->stream>>>(g[P2], g[CAT2], 96, 64, a[E2], g[E2],
                                                                             D >> 1, H >> 1, W >> 1, 32);
    // level 1 encoder
    KV_TRY(conv_backward(u, 2, g[E2], a[A2], nullptr, g[A2], 1, a[A2]));
    KV_TRY(conv_backward(u, 1, g[A2], a[P1], nullptr, g[P1], 1));
    pool_bwd_skip_mask<<<grid_n(ctx, n0 * 2), 256, 0, ctx->stream>>>(g[P1], g[CAT1], 48, 32, a[E1], g[E1], D, H, W, 16);
    // level 0 encoder
    KV_TRY(conv_backward(u, 0, g[E1], a[A0], nullptr, g[A0], 0, a[A0]));
    {
        // one round of resident blocks over the six (dz, channel half) passes
        dim3 grid(std::min(grid_n(ctx, n0 / 4), std::max(1, ctx->sm_count / 3)), 3, 2);
        conv_first_wgrad<<<grid, 256, 0, ctx->stream>>>(u->x, g[A0], u->g + u->w_first, u->g + u->b_first, D, H, W);
    }
    KV_CHECK_LAUNCH(ctx, "unet backward");
    return KV_OK;
}

kv_status loss_and_grad(kv_unet *u) {
    kv_ctx *ctx = u->ctx;
    const long long n0 = (long long)u->D * u->H * u->W;
    const int nb = grid_n(ctx, n0) > 4096 ? 4096 : grid_n(ctx, n0);
    mse_loss<<<nb, 256, 0, ctx->stream>>>(u->y, u->t, u->dy, n0, u->partials);
    sum_loss<<<1, 256, 0, ctx->stream>>>(u->partials, nb, n0, u->loss);
    KV_CHECK_LAUNCH(ctx, "unet loss");
    return KV_OK;
}

kv_status train_body(kv_unet *u, float lr, bool apply) {
    kv_ctx *ctx = u->ctx;
    KV_TRY(forward(u, true));
    KV_TRY(loss_and_grad(u));
    KV_CHECK_CUDA(ctx, cudaMemsetAsync(u->g, 0, u->nparams * sizeof(float), ctx->stream));
    KV_TRY(backward(u));
    if (apply) {
        adam_step<<<grid_n(ctx, (long long)u->nparams), 256, 0, ctx->stream>>>(u->p, u->g, u->m, u->v, u->pb, u->nparams, lr,
                                                                             0.9f, 0.999f, 1e-8f, u->corr);
        KV_CHECK_LAUNCH(ctx, "adam");
    }
    return KV_OK;
}

kv_status copy_in(kv_unet *u, float *dst, const float *src, size_t n, kv_mem mem) {
    KV_CHECK_CUDA(u->ctx, cudaMemcpyAsync(dst, src, n * sizeof(float),
                                          mem == KV_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice,
                                          u->ctx->stream));
    return KV_OK;
}

}  // namespace

// ------------------------------------------------------------------ C ABI

extern "C" kv_status kv_unet_create(kv_ctx *ctx, uint64_t seed, kv_unet **out) {
    if (ctx == nullptr || out == nullptr) return KV_ERR_INVALID_ARG;
    *out = nullptr;
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    kv_unet *u = new (std::nothrow) kv_unet;
    if (u == nullptr) return KV_ERR_OOM;
    u->ctx = ctx;
    ctx->plans += 1;   // the network keeps the context alive like a plan
    const int spec[14][3] = {{16, 0, 16},  {16, 0, 32},   {32, 0, 32},  {32, 0, 64},  {64, 0, 64},
                             {64, 0, 128}, {128, 0, 128}, {128, 64, 64}, {64, 0, 64}, {64, 32, 32},
                             {32, 0, 32},  {32, 16, 16},  {16, 0, 16},   {0, 0, 0}};
    size_t off = 0;
    u->w_first = off;
    off += 16 * 27;
    u->b_first = off;
    off += 16;
    for (int l = 0; l < 14; ++l) {
        u->conv[l] = {spec[l][0], spec[l][1], spec[l][2], 0, 0};
        if (spec[l][2] == 0) continue;
        u->conv[l].w = off;
        off += (size_t)spec[l][2] * 27 * (spec[l][0] + spec[l][1]);
        u->conv[l].b = off;
        off += spec[l][2];
        off = (off + 7) & ~(size_t)7;   // keep every weight block 16-byte aligned in BF16
    }
    u->w_out = off;
    off += 16;
    u->b_out = off;
    off += 8;
    u->nparams = off;
    // He initialisation (normal, std sqrt(2 / fan_in)); zero biases; the output
    // layer starts at zero so the untrained network returns its input
    std::vector<float> h(off, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](size_t o, size_t n, int fan_in) {
        std::normal_distribution<float> nd(0.f, std::sqrt(2.f / (float)fan_in));
        for (size_t i = 0; i < n; ++i) h[o + i] = nd(rng);
    };
    fill(u->w_first, 16 * 27, 27);
    for (int l = 0; l < 13; ++l) {
        const auto &L = u->conv[l];
        fill(L.w, (size_t)L.cout * 27 * (L.c1 + L.c2), 27 * (L.c1 + L.c2));
    }
    kv_status s = KV_OK;
    if (cudaMalloc((void **)&u->p, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&u->g, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&u->m, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&u->v, off * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&u->pb, off * sizeof(bf16)) != cudaSuccess ||
        cudaMalloc((void **)&u->wt, off * sizeof(bf16)) != cudaSuccess ||
        cudaMalloc((void **)&u->corr, 4 * sizeof(float)) != cudaSuccess ||
        cudaMalloc((void **)&u->tc_status, sizeof(int)) != cudaSuccess) {
        s = kv_fail(ctx, KV_ERR_OOM, "U-Net parameters");
    } else {
        cudaMemcpy(u->p, h.data(), off * sizeof(float), cudaMemcpyHostToDevice);
        cudaMemset(u->m, 0, off * sizeof(float));
        cudaMemset(u->v, 0, off * sizeof(float));
        cudaMemset(u->tc_status, 0, sizeof(int));
        to_bf16<<<grid_n(ctx, (long long)off), 256, 0, ctx->stream>>>(u->p, u->pb, off);
        if (cudaStreamSynchronize(ctx->stream) != cudaSuccess) s = kv_fail(ctx, KV_ERR_CUDA, "U-Net init");
    }
    if (s != KV_OK) {
        kv_unet_destroy(u);
        return s;
    }
    *out = u;
    return KV_OK;
}

extern "C" kv_status kv_unet_destroy(kv_unet *u) {
    if (u == nullptr) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    free_workspace(u);
    cudaFree(u->p);
    cudaFree(u->g);
    cudaFree(u->m);
    cudaFree(u->v);
    cudaFree(u->pb);
    cudaFree(u->wt);
    cudaFree(u->corr);
    cudaFree(u->tc_status);
    delete u;
    kv_ctx_release_ref(ctx);
    return KV_OK;
}

extern "C" size_t kv_unet_num_params(const kv_unet *u) { return u ? u->nparams : 0; }

namespace {
// Reads (and clears) the tensor-core convolution's wait status: non-zero when
// one of its bounded pipeline waits gave up.  Synchronises the stream.
kv_status tc_check(kv_unet *u) {
    kv_ctx *ctx = u->ctx;
    int h = 0;
    KV_CHECK_CUDA(ctx, cudaMemcpyAsync(&h, u->tc_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (h != 0) {
        cudaMemset(u->tc_status, 0, sizeof(int));
        return kv_fail(ctx, KV_ERR_TIMEOUT, "tensor-core convolution: pipeline wait %d timed out", h);
    }
    return KV_OK;
}
}  // namespace

extern "C" kv_status kv_unet_forward(kv_unet *u, const float *in, float *out, int32_t D, int32_t H, int32_t W,
                                     kv_mem mem) {
    if (u == nullptr || in == nullptr || out == nullptr) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    KV_TRY(ensure_workspace(u, D, H, W, false));
    const size_t n = (size_t)D * H * W;
    KV_TRY(copy_in(u, u->x, in, n, mem));
    KV_TRY(forward(u, false));
    KV_CHECK_CUDA(ctx, cudaMemcpyAsync(out, u->y, n * sizeof(float),
                                       mem == KV_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, ctx->stream));
    return tc_check(u);
}

// One Adam step on (input, target); loss = mean squared error before the step.
// The step (forward, loss, backward, update) runs as a CUDA graph captured on
// the first call for a given shape and learning rate.
extern "C" kv_status kv_unet_train_step(kv_unet *u, const float *in, const float *target, int32_t D, int32_t H,
                                        int32_t W, float lr, float *loss, kv_mem mem) {
    if (u == nullptr || in == nullptr || target == nullptr) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    KV_TRY(ensure_workspace(u, D, H, W, true));
    const size_t n = (size_t)D * H * W;
    KV_TRY(copy_in(u, u->x, in, n, mem));
    KV_TRY(copy_in(u, u->t, target, n, mem));
    // Adam bias corrections of this step go to device memory, so the captured
    // step stays valid from one step to the next
    const float corr[2] = {1.f - powf(0.9f, (float)(u->step + 1)), 1.f - powf(0.999f, (float)(u->step + 1))};
    KV_CHECK_CUDA(ctx, cudaMemcpyAsync(u->corr, corr, sizeof corr, cudaMemcpyHostToDevice, ctx->stream));
    if (ctx->timing) {
        KV_TRY(train_body(u, lr, true));          // traced: plain launches
    } else {
        if (u->train_graph == nullptr || u->graph_lr != lr) {
            if (u->train_graph) {
                KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
                cudaGraphExecDestroy(u->train_graph);
                u->train_graph = nullptr;
            }
            cudaStream_t user = ctx->stream;
            ctx->stream = ctx->own_stream;
            KV_CHECK_CUDA(ctx, cudaStreamBeginCapture(ctx->own_stream, cudaStreamCaptureModeThreadLocal));
            kv_status st = train_body(u, lr, true);
            cudaGraph_t graph = nullptr;
            cudaError_t e = cudaStreamEndCapture(ctx->own_stream, &graph);
            ctx->stream = user;
            if (st != KV_OK) {
                if (graph) cudaGraphDestroy(graph);
                return st;
            }
            if (e != cudaSuccess) return kv_fail(ctx, KV_ERR_CUDA, "train step capture: %s", cudaGetErrorString(e));
            e = cudaGraphInstantiate(&u->train_graph, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) {
                u->train_graph = nullptr;
                return kv_fail(ctx, KV_ERR_CUDA, "train step instantiate: %s", cudaGetErrorString(e));
            }
            u->graph_lr = lr;
        }
        KV_CHECK_CUDA(ctx, cudaGraphLaunch(u->train_graph, ctx->stream));
    }
    u->step += 1;
    if (loss) KV_CHECK_CUDA(ctx, cudaMemcpyAsync(loss, u->loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    return tc_check(u);
}

// Loss and FP32 parameter gradients (no update), for gradient checks.
extern "C" kv_status kv_unet_gradients(kv_unet *u, const float *in, const float *target, int32_t D, int32_t H,
                                       int32_t W, float *loss, float *grads, kv_mem mem) {
    if (u == nullptr || in == nullptr || target == nullptr || grads == nullptr) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    KV_TRY(ensure_workspace(u, D, H, W, true));
    const size_t n = (size_t)D * H * W;
    KV_TRY(copy_in(u, u->x, in, n, mem));
    KV_TRY(copy_in(u, u->t, target, n, mem));
    KV_TRY(train_body(u, 0.f, false));
    KV_CHECK_CUDA(ctx, cudaMemcpyAsync(grads, u->g, u->nparams * sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    if (loss) KV_CHECK_CUDA(ctx, cudaMemcpyAsync(loss, u->loss, sizeof(float), cudaMemcpyDeviceToHost, ctx->stream));
    return tc_check(u);
}

// State = parameters, Adam first and second moments (3 * num_params floats)
// and the step count, for checkpoints.
extern "C" kv_status kv_unet_get_state(const kv_unet *u, float *state, int64_t *step) {
    if (u == nullptr || state == nullptr) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    KV_CHECK_CUDA(ctx, cudaMemcpy(state, u->p, u->nparams * sizeof(float), cudaMemcpyDeviceToHost));
    KV_CHECK_CUDA(ctx, cudaMemcpy(state + u->nparams, u->m, u->nparams * sizeof(float), cudaMemcpyDeviceToHost));
    KV_CHECK_CUDA(ctx, cudaMemcpy(state + 2 * u->nparams, u->v, u->nparams * sizeof(float), cudaMemcpyDeviceToHost));
    if (step) *step = u->step;
    return KV_OK;
}

extern "C" kv_status kv_unet_set_state(kv_unet *u, const float *state, int64_t step) {
    if (u == nullptr || state == nullptr || step < 0) return KV_ERR_INVALID_ARG;
    kv_ctx *ctx = u->ctx;
    KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    KV_CHECK_CUDA(ctx, cudaMemcpy(u->p, state, u->nparams * sizeof(float), cudaMemcpyHostToDevice));
    KV_CHECK_CUDA(ctx, cudaMemcpy(u->m, state + u->nparams, u->nparams * sizeof(float), cudaMemcpyHostToDevice));
    KV_CHECK_CUDA(ctx, cudaMemcpy(u->v, state + 2 * u->nparams, u->nparams * sizeof(float), cudaMemcpyHostToDevice));
    to_bf16<<<grid_n(ctx, (long long)u->nparams), 256, 0, ctx->stream>>>(u->p, u->pb, u->nparams);
    KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    u->step = step;
    return KV_OK;
}

// One 3x3x3 convolution of the network's kind on caller buffers (device
// pointers, BF16 bit patterns): the operator behind every U-Net layer, for
// callers and tests that need a single layer.  kernel: 0 = the tensor-core
// (tcgen05 / TMA) kernel where it covers the call, else mma.sync; 1 = tcgen05
// only, for volumes of whole 128-voxel tiles; 2 = mma.sync only.
extern "C" kv_status kv_conv3_bf16(kv_ctx *ctx, const uint16_t *in1, int32_t c1, const uint16_t *in2, int32_t c2,
                                   const uint16_t *w, const float *bias, int32_t relu, uint16_t *out, int32_t cout,
                                   int32_t D, int32_t H, int32_t W, int32_t kernel) {
    if (ctx == nullptr) return KV_ERR_INVALID_ARG;
    if (in1 == nullptr || w == nullptr || out == nullptr || (c2 > 0 && in2 == nullptr))
        return kv_fail(ctx, KV_ERR_INVALID_ARG, "kv_conv3_bf16: null buffer");
    if (D <= 0 || H <= 0 || W <= 0 || c1 <= 0 || c2 < 0 || cout <= 0 || kernel < 0 || kernel > 2)
        return kv_fail(ctx, KV_ERR_INVALID_ARG, "kv_conv3_bf16: bad sizes or kernel choice");
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const bf16 *a = reinterpret_cast<const bf16 *>(in1), *b = reinterpret_cast<const bf16 *>(in2);
    const bf16 *wb = reinterpret_cast<const bf16 *>(w);
    bf16 *o = reinterpret_cast<bf16 *>(out);
    const bool tiles = convtc::tile_shape(D, H, W);
    if (kernel == 1 && !tiles)
        return kv_fail(ctx, KV_ERR_UNSUPPORTED, "kv_conv3_bf16: the volume is not a whole number of 128-voxel tiles");
    // volumes that are not whole tiles, of the widths that mma.sync takes, take the tensor-core kernel too where it
    // covers the call, else mma.sync; the two sum in the same order, with equal bits
    if (kernel != 2 && (tiles || W % 16 == 0)) {
        const char *why = convtc::launch(a, c1, c2 ? b : nullptr, c2, wb, bias, relu != 0, nullptr, nullptr, o, cout, D, H, W,
                                         true, ctx->d_status, ctx->sm_count, ctx->stream);
        if (why == nullptr) {
            KV_CHECK_LAUNCH(ctx, "kv_conv3_bf16 (tcgen05)");
            return KV_OK;
        }
        if (tiles) return kv_fail(ctx, KV_ERR_UNSUPPORTED, "tensor-core convolution: %s", why);
    }
    if (W % 16 != 0 || c1 % 16 != 0 || c2 % 16 != 0 || cout % 16 != 0)
        return kv_fail(ctx, KV_ERR_UNSUPPORTED, "kv_conv3_bf16: mma.sync needs W, channels multiples of 16");
    const long long nvox = (long long)D * H * W;
    const int blocks = (int)((nvox / 16 + 3) / 4);
    for (int n0 = 0; n0 < cout; n0 += 64) {
        const int nc = cout - n0 < 64 ? cout - n0 : 64;
        const bool rl = relu != 0;
        switch (nc) {
        case 16: rl ? unet::conv3_fwd<2, true><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W)
                    : unet::conv3_fwd<2, false><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W); break;
        case 32: rl ? unet::conv3_fwd<4, true><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W)
                    : unet::conv3_fwd<4, false><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W); break;
        case 48: rl ? unet::conv3_fwd<6, true><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W)
                    : unet::conv3_fwd<6, false><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W); break;
        default: rl ? unet::conv3_fwd<8, true><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W)
                    : unet::conv3_fwd<8, false><<<blocks, 128, 0, ctx->stream>>>(a, c1, b, c2, wb, bias, o, cout, n0, D, H, W); break;
        }
    }
    KV_CHECK_LAUNCH(ctx, "kv_conv3_bf16 (mma.sync)");
    return KV_OK;
}
