// kv_misc.cu -- shift-and-add, phantom rasteriser and elementwise kernels.
#include "kv_internal.h"
#include "kv_exact_common.cuh"
#include "kv_tma.cuh"

#include <algorithm>
#include <cmath>

namespace {

// Shift-and-add (recons::ShiftAndAdd, Reconstructors.h:263-379):
// out[k][v][u] = (1/P) * sum_i in[i][v + t_ki][u], zero outside the ROI.
// The reference sums the weighted views in double (vtkImageWeightedSum); here
// the views are summed exactly enough with a float-float (TwoSum) accumulator
// and the mean is formed in double before rounding to float.
// Block: 32 columns x 8 rows; each thread loops over a batch of slices so that
// consecutive slices, whose shifts differ by a few rows, hit the same lines.
__global__ void __launch_bounds__(256) saa_kernel(int nu, int nv, int nz, int P,
                                                  const int32_t *__restrict__ shift,
                                                  const float *__restrict__ proj,
                                                  float *__restrict__ out, int kb) {
    extern __shared__ int32_t sh_shift[];
    const int u = blockIdx.x * 32 + threadIdx.x;
    const int v = blockIdx.y * blockDim.y + threadIdx.y;
    const int k0 = blockIdx.z * kb, k1 = min(nz, k0 + kb);
    for (int t = threadIdx.y * 32 + threadIdx.x; t < (k1 - k0) * P; t += blockDim.x * blockDim.y)
        sh_shift[t] = shift[(size_t)k0 * P + t];
    __syncthreads();
    if (u >= nu || v >= nv) return;
    const double w = 1.0 / (double)P;
    for (int k = k0; k < k1; ++k) {
        float hi = 0.f, lo = 0.f;
        const int32_t *sk = sh_shift + (size_t)(k - k0) * P;
        for (int i = 0; i < P; ++i) {
            const int r = v + sk[i];
            if (r >= 0 && r < nv) {
                const float x = __ldg(proj + ((size_t)i * nv + r) * nu + u);
                const float s = hi + x;                       // TwoSum(hi, x)
                const float bp = s - hi;
                const float err = (hi - (s - bp)) + (x - bp);
                hi = s;
                lo += err;
            }
        }
        out[((size_t)k * nv + v) * nu + u] = (float)(((double)hi + (double)lo) * w);
    }
}

// The same sums with each view's rows staged in shared memory.  A block
// covers 32 detector columns x kSaaRows rows x KS slices; for every
// view one thread loads, by TMA, the band of that view's rows the block's
// shifted rows reach (kSaaRows + the largest spread of the block's shifts;
// rows outside the detector read zeros, which is the reference's zero
// padding) into a ring of shared-memory stages, and every thread adds its
// kSaaRows / 8 x KS outputs' rows from the band.  Views are added in
// the same order with the same TwoSum as saa_kernel, and a row outside the
// detector adds an exact zero, so the two kernels agree bit for bit.
//
// Seven FP32 additions per row and slice bound it (60 views of 2048 x 2048
// into 128 slices: 2.3e11, 6.0 ms of the FP32 pipes).  Two columns a lane in
// packed additions (each half rounds as the scalar one), eight slices a staged
// band, two views a barrier and the slices' places in the band computed before
// the loop: 18.4 -> 10.2 ms there.  Where eight slices' spread does not fit,
// four.
constexpr int kSaaRows = 32, kSaaStages = 4;
constexpr uint32_t kSaaWaitPolls = 1u << 22;

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long r, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a - b as b * -1 + a, rounded once: the packed multiply-add is native, the packed subtraction was not (10 instead of 5
// instructions a row and slice)
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(b), "l"(0xbf800000bf800000ull), "l"(a));
    return r;
}

template <int KS>
__global__ void __launch_bounds__(256, 2) saa_band_kernel(const __grid_constant__ CUtensorMap pmap, int nu, int nv,
                                                          int nz, int P, const int32_t *__restrict__ shift,
                                                          float *__restrict__ out, int nb, uint32_t stage_stride,
                                                          int wide, int *status) {
    constexpr int kPairs = kSaaRows / 16;   // a half warp a row, two columns a lane
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t full[kSaaStages];
    unsigned char *base = smem + ((128u - (kvtma::smem_u32(smem) & 127u)) & 127u);
    int *off = reinterpret_cast<int *>(base + kSaaStages * stage_stride);    // [P][KS]: bytes into the band
    int *first = off + KS * P;                                               // [P]: the band's first row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = blockIdx.x * 32, v0 = blockIdx.y * kSaaRows, k0 = blockIdx.z * KS;
    const int kn = min(KS, nz - k0);
    // Where in its band each (view, slice) starts, once: in the loop a slice costs an address and its seven additions
    // (shifts, band checks and addresses there were half its instructions).  A start outside the band is never
    // expected; it is recorded and the block ends.
    int err = 0;
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        int t[KS], tmin = shift[(size_t)k0 * P + p];
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            t[kk] = shift[(size_t)(k0 + min(kk, kn - 1)) * P + p];   // slices past the last repeat it
            tmin = min(tmin, t[kk]);
        }
        first[p] = v0 + tmin;
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            off[p * KS + kk] = (t[kk] - tmin) * 128;
            if (t[kk] - tmin > nb - kSaaRows) err = 4;
        }
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kSaaStages; ++s) kvtma::mbar_init(&full[s], 1);
        kvtma::fence_mbar_init();
    }
    if (__syncthreads_or(err)) {
        if (err) atomicOr(status, err);
        return;
    }
    const uint32_t band_bytes = 32u * (uint32_t)nb * 4u;
    auto issue = [&](int i, int st) {
        kvtma::fence_proxy_async_smem();
        kvtma::mbar_arrive_expect_tx(&full[st], band_bytes);
        kvtma::tma_load_3d(kvtma::smem_u32(base + (size_t)st * stage_stride), &pmap, &full[st], u0, first[i], i);
    };
    if (threadIdx.x == 0)
        for (int i = 0; i < kSaaStages && i < P; ++i) issue(i, i);
    __syncthreads();
    const int row0 = 2 * warp + (lane >> 4), col0 = 2 * (lane & 15);
    unsigned long long hi[kPairs][KS], lo[kPairs][KS];   // rows 16 m + row0, columns col0 and col0 + 1
#pragma unroll
    for (int m = 0; m < kPairs; ++m)
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) hi[m][kk] = lo[m][kk] = 0ull;
    int i = 0;
    // one view's rows into sums a -> b: two register sets, so that the new sums need no move into the old ones' place
    auto add_view = [&](int view, int st, unsigned long long (&a)[kPairs][KS], unsigned long long (&b)[kPairs][KS]) {
        const unsigned char *band = base + (size_t)st * stage_stride + (row0 * 32 + col0) * 4;
        int o[KS];
#pragma unroll
        for (int kk = 0; kk < KS; kk += 4) {
            const int4 v = *reinterpret_cast<const int4 *>(off + view * KS + kk);
            o[kk] = v.x;
            o[kk + 1] = v.y;
            o[kk + 2] = v.z;
            o[kk + 3] = v.w;
        }
#pragma unroll
        for (int kk = 0; kk < KS; ++kk) {
            const unsigned char *row = band + o[kk];
#pragma unroll
            for (int m = 0; m < kPairs; ++m) {
                const unsigned long long x = *reinterpret_cast<const unsigned long long *>(row + 16 * m * 128);
                b[m][kk] = add2(a[m][kk], x);                           // TwoSum(a, x)
                const unsigned long long bp = sub2(b[m][kk], a[m][kk]);
                const unsigned long long e = add2(sub2(a[m][kk], sub2(b[m][kk], bp)), sub2(x, bp));
                lo[m][kk] = add2(lo[m][kk], e);
            }
        }
    };
    for (; i < P; i += 2) {   // two views a barrier
        const int st = i % kSaaStages;
        const bool two = i + 1 < P;
        if (!kvtma::mbar_wait_bounded(&full[st], (uint32_t)(i / kSaaStages) & 1u, kSaaWaitPolls)) err |= 1;
        if (two && !kvtma::mbar_wait_bounded(&full[st + 1], (uint32_t)(i / kSaaStages) & 1u, kSaaWaitPolls)) err |= 1;
        if (err == 0) {
            unsigned long long mid[kPairs][KS];
            add_view(i, st, hi, mid);
            if (two) {
                add_view(i + 1, st + 1, mid, hi);
            } else {
#pragma unroll
                for (int m = 0; m < kPairs; ++m)
#pragma unroll
                    for (int kk = 0; kk < KS; ++kk) hi[m][kk] = mid[m][kk];
            }
        }
        if (__syncthreads_or(err)) break;
        if (threadIdx.x == 0) {
            if (i + kSaaStages < P) issue(i + kSaaStages, st);
            if (i + 1 + kSaaStages < P) issue(i + 1 + kSaaStages, st + 1);
        }
    }
    if (i < P) {   // failed: record, let the loads in flight land, leave
        if (err) atomicOr(status, err);
        if (threadIdx.x == 0)
            for (int j = i; j < min(P, i + kSaaStages); ++j)
                kvtma::mbar_wait_bounded(&full[j % kSaaStages], (uint32_t)(j / kSaaStages) & 1u, kSaaWaitPolls);
        return;
    }
    const int u = u0 + col0;   // nu is a multiple of 4 here
    if (u >= nu) return;
    const double w = 1.0 / (double)P;
#pragma unroll
    for (int kk = 0; kk < KS; ++kk) {
        if (kk >= kn) break;
#pragma unroll
        for (int m = 0; m < kPairs; ++m) {
            const int v = v0 + row0 + 16 * m;
            if (v >= nv) continue;
            float h[2], l[2];
            unpack2(hi[m][kk], h[0], h[1]);
            unpack2(lo[m][kk], l[0], l[1]);
            const float2 o = make_float2((float)(((double)h[0] + (double)l[0]) * w), (float)(((double)h[1] + (double)l[1]) * w));
            float *dst = out + ((size_t)(k0 + kk) * nv + v) * nu + u;
            if (wide) {
                *reinterpret_cast<float2 *>(dst) = o;
            } else {
                dst[0] = o.x;
                dst[1] = o.y;
            }
        }
    }
}

// The learned warm start's elementwise steps.
// ratio = a1 > 0 ? p / a1 : 0, and per block the FP64 sums of (a1 - p)^2 and
// p^2 (the uniform start's data residual: its forward projection is a1).
__global__ void __launch_bounds__(256) warm_ratio_kernel(const float *__restrict__ p, const float *__restrict__ a1,
                                                         float *__restrict__ ratio, size_t n, double *partials) {
    double d0 = 0.0, d1 = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float pv = p[i], av = a1[i];
        ratio[i] = av > 0.f ? pv / av : 0.f;
        const double d = (double)av - (double)pv;
        d0 += d * d;
        d1 += (double)pv * (double)pv;
    }
    for (int o = 16; o > 0; o >>= 1) {
        d0 += __shfl_xor_sync(0xffffffffu, d0, o);
        d1 += __shfl_xor_sync(0xffffffffu, d1, o);
    }
    __shared__ double red[2][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        red[0][warp] = d0;
        red[1][warp] = d1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0.0, s1 = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            s0 += red[0][w];
            s1 += red[1][w];
        }
        partials[2 * blockIdx.x] = s0;
        partials[2 * blockIdx.x + 1] = s1;
    }
}

// out[0..1] = the sums of the per-block partial pairs (one block, fixed order)
__global__ void sum_pairs_kernel(const double *partials, int nblocks, double *out) {
    __shared__ double sh[2][256];
    double s0 = 0.0, s1 = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        s0 += partials[2 * b];
        s1 += partials[2 * b + 1];
    }
    sh[0][threadIdx.x] = s0;
    sh[1][threadIdx.x] = s1;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + w];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = sh[0][0];
        out[1] = sh[1][0];
    }
}

// out = sens > 0 ? b / sens (in FP64, rounded once) : 0
__global__ void warm_normalize_kernel(const float *__restrict__ b, const double *__restrict__ sens,
                                      float *__restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const double sv = sens[i];
        out[i] = sv > 0.0 ? (float)((double)b[i] / sv) : 0.f;
    }
}

// out = seen ? max(net, eps) : max(saa, eps)
__global__ void warm_fill_kernel(const float *__restrict__ net, const float *__restrict__ saa,
                                 const uint8_t *__restrict__ seen, float eps, float *__restrict__ out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = fmaxf(seen[i] ? net[i] : saa[i], eps);
}

__global__ void fill_kernel(float *p, size_t n, float v) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        p[i] = v;
}

template <typename T>
__global__ void to_storage_kernel(const float *in, T *out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        Store<T>::st(out + i, in[i]);
}

template <typename T>
__global__ void from_storage_kernel(const T *in, float *out, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        out[i] = Store<T>::ld_rw(in + i);
}

// Ellipsoid phantom sampled at voxel centres.  params: n rows of 16 floats =
// centre[3], semi-axes[3], M[9] (local = M (q - c)), density.  The float
// operations and their order are fixed (explicit round-to-nearest
// intrinsics), so the result is bit-identical on every build.
__global__ void __launch_bounds__(256) phantom_kernel(int nx, int ny, int nz, float dx, float dy,
                                                      float dz, const float *__restrict__ params,
                                                      int n, float *__restrict__ vol) {
    extern __shared__ float sp[];
    for (int t = threadIdx.x; t < 16 * n; t += blockDim.x) sp[t] = params[t];
    __syncthreads();
    const size_t plane = (size_t)nx * ny, total = plane * nz;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int z = (int)(idx / plane);
        const size_t rem = idx % plane;
        const int y = (int)(rem / nx), x = (int)(rem % nx);
        const float q0 = __fsub_rn(__fmul_rn(__fadd_rn((float)x, 0.5f), dx), __fmul_rn(__fmul_rn(0.5f, (float)nx), dx));
        const float q1 = __fsub_rn(__fmul_rn(__fadd_rn((float)y, 0.5f), dy), __fmul_rn(__fmul_rn(0.5f, (float)ny), dy));
        const float q2 = __fsub_rn(__fmul_rn(__fadd_rn((float)z, 0.5f), dz), __fmul_rn(__fmul_rn(0.5f, (float)nz), dz));
        float val = 0.f;
        for (int e = 0; e < n; ++e) {
            const float *p = sp + 16 * e;
            const float r0 = __fsub_rn(q0, p[0]), r1 = __fsub_rn(q1, p[1]), r2 = __fsub_rn(q2, p[2]);
            const float l0 = __fadd_rn(__fadd_rn(__fmul_rn(p[6], r0), __fmul_rn(p[7], r1)), __fmul_rn(p[8], r2));
            const float l1 = __fadd_rn(__fadd_rn(__fmul_rn(p[9], r0), __fmul_rn(p[10], r1)), __fmul_rn(p[11], r2));
            const float l2 = __fadd_rn(__fadd_rn(__fmul_rn(p[12], r0), __fmul_rn(p[13], r1)), __fmul_rn(p[14], r2));
            const float t0 = __fdiv_rn(l0, p[3]), t1 = __fdiv_rn(l1, p[4]), t2 = __fdiv_rn(l2, p[5]);
            const float s = __fadd_rn(__fadd_rn(__fmul_rn(t0, t0), __fmul_rn(t1, t1)), __fmul_rn(t2, t2));
            if (s <= 1.f) val = __fadd_rn(val, p[15]);
        }
        vol[idx] = val;
    }
}

// FP64 reduction of {sum (q-p)^2, sum p^2, sum p log q - q} over n rays:
// grid-stride per-thread sums, one partial triple per block, then a single
// block adds the partials in a fixed order (deterministic).
__global__ void __launch_bounds__(256) residual_partials_kernel(const float *__restrict__ q,
                                                                const float *__restrict__ p, size_t n,
                                                                double *__restrict__ partials) {
    double d0 = 0.0, d1 = 0.0, d2 = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float qi = q[i], pi = p[i];
        const double dq = (double)qi - (double)pi;
        d0 += dq * dq;
        d1 += (double)pi * (double)pi;
        d2 += (qi > 0.f ? (double)pi * (double)logf(qi) : 0.0) - (double)qi;
    }
    for (int o = 16; o > 0; o >>= 1) {
        d0 += __shfl_xor_sync(0xffffffffu, d0, o);
        d1 += __shfl_xor_sync(0xffffffffu, d1, o);
        d2 += __shfl_xor_sync(0xffffffffu, d2, o);
    }
    __shared__ double sh[3][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { sh[0][warp] = d0; sh[1][warp] = d1; sh[2][warp] = d2; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s0 = 0.0, s1 = 0.0, s2 = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { s0 += sh[0][w]; s1 += sh[1][w]; s2 += sh[2][w]; }
        partials[3 * blockIdx.x] = s0;
        partials[3 * blockIdx.x + 1] = s1;
        partials[3 * blockIdx.x + 2] = s2;
    }
}

__global__ void sum_partials_kernel(const double *__restrict__ partials, int nblocks, double *__restrict__ out) {
    __shared__ double sh[3][256];
    double s0 = 0.0, s1 = 0.0, s2 = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
        s0 += partials[3 * b];
        s1 += partials[3 * b + 1];
        s2 += partials[3 * b + 2];
    }
    sh[0][threadIdx.x] = s0;
    sh[1][threadIdx.x] = s1;
    sh[2][threadIdx.x] = s2;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + w];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + w];
            sh[2][threadIdx.x] += sh[2][threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) { out[0] = sh[0][0]; out[1] = sh[1][0]; out[2] = sh[2][0]; }
}

int grid_for(const kv_ctx *ctx, size_t n, int block) {
    size_t g = (n + block - 1) / block;
    size_t cap = (size_t)ctx->sm_count * 8;
    if (cap == 0) cap = 1024;
    return (int)(g < cap ? (g == 0 ? 1 : g) : cap);
}

}  // namespace

// Ramp filtering of the projections along v (the tube's sweep direction)
// for the filtered backprojection: out[p][v][u] = Ls(u, v) * sum_{|k|<=K}
// h[|k|] * in[p][v-k][u], zero outside the detector; Ls, the ray's length in a
// slice, is the scaling the backprojector's input carries.  h is the
// Shepp-Logan kernel h[n] = -2 / (pi^2 (4 n^2 - 1)) in pixel units (L. A.
// Shepp, B. F. Logan, IEEE Trans. Nucl. Sci. 21, 1974), truncated at |n| <= K
// and passed by value.  A block holds 32 columns and 64 output rows; the 64 +
// 2K input rows it needs are staged in shared memory (zeros outside the
// detector), and each thread sums the symmetric taps pairwise in FP32.
//
// With one output a thread at a time every tap took two shared-memory reads
// for an add and a multiply-add, and shared memory bounded it.  A thread keeps
// eight consecutive rows: eight taps need 15 rows above and 15 below, seven of
// which it has from the taps before, so 16 reads serve 64 tap sums, and two
// adjacent columns, in packed arithmetic (the same roundings).  25 views
// of 1024 x 1024, K = 128: 780 us, and 127 us for a separate scaling pass, ->
// 258 us together.
namespace {

struct RampTaps {
    float h[KV_FBP_MAX_HALF_TAPS + 1];
};

constexpr int kRampRows = 64, kRampR = 8;   // rows of a block, of a thread
constexpr int kRampCols = 32;               // columns of a block, two a thread

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__global__ void __launch_bounds__(128) ramp_v_kernel(const float *__restrict__ in, float *__restrict__ out, int nu,
                                                     int nv, int K, int wide, const RampTaps taps, const ExactTables T) {
    extern __shared__ __align__(16) float tile[];   // [kRampRows + 2K][kRampCols]
    constexpr int kStep = kRampCols / 2;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int p = blockIdx.z, uc = blockIdx.x * kRampCols;
    const int v0 = blockIdx.y * kRampRows;
    const size_t base = (size_t)p * nv * nu;
    const int rows = kRampRows + 2 * K;
    // all rows in flight at once (asynchronous copies; size 0 writes zeros): 16 bytes where the detector's rows allow
    // it, else 4
    const uint32_t sm = kvtma::smem_u32(tile);
    if (wide) {
        for (int e = threadIdx.x; e < rows * (kRampCols / 4); e += 128) {
            const int r = e / (kRampCols / 4), q = e % (kRampCols / 4) * 4, v = v0 - K + r;
            const bool live = v >= 0 && v < nv && uc + q < nu;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sm + (uint32_t)(r * kRampCols + q) * 4u),
                         "l"(live ? in + base + (size_t)v * nu + uc + q : in), "r"(live ? 16 : 0)
                         : "memory");
        }
    } else {
        for (int e = threadIdx.x; e < rows * kRampCols; e += 128) {
            const int r = e / kRampCols, q = e % kRampCols, v = v0 - K + r;
            const bool live = v >= 0 && v < nv && uc + q < nu;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(sm + (uint32_t)(r * kRampCols + q) * 4u),
                         "l"(live ? in + base + (size_t)v * nu + uc + q : in), "r"(live ? 4 : 0)
                         : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const int o = ty * kRampR, u = uc + 2 * tx;
    if (u >= nu || v0 + o >= nv) return;
    // columns u, u + 1 of the thread's first output row, one 64-bit word a row
    const unsigned long long *c = reinterpret_cast<const unsigned long long *>(tile) + (o + K) * kStep + tx;
    unsigned long long acc[kRampR], lo[2 * kRampR - 1], hi[2 * kRampR - 1];
    const unsigned long long h0 = pack2(taps.h[0], taps.h[0]);
#pragma unroll
    for (int j = 0; j < kRampR; ++j)
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(acc[j]) : "l"(h0), "l"(c[j * kStep]));
#pragma unroll
    for (int j = 0; j < kRampR - 1; ++j) {
        lo[j] = c[j * kStep];
        hi[j + kRampR] = c[(j + 1) * kStep];
    }
    int k0 = 0;
    for (; k0 + kRampR <= K; k0 += kRampR) {
        // taps k0 + 1 .. k0 + 8: rows -k0 - 8 .. -k0 + 6 (lo) and k0 + 1 .. k0 + 15 (hi)
#pragma unroll
        for (int j = 0; j < kRampR - 1; ++j) {
            lo[j + kRampR] = lo[j];
            hi[j] = hi[j + kRampR];
        }
#pragma unroll
        for (int j = 0; j < kRampR; ++j) {
            lo[j] = c[(j - k0 - kRampR) * kStep];
            hi[j + kRampR - 1] = c[(k0 + kRampR + j) * kStep];
        }
#pragma unroll
        for (int k = 1; k <= kRampR; ++k) {
            const unsigned long long h = pack2(taps.h[k0 + k], taps.h[k0 + k]);
#pragma unroll
            for (int j = 0; j < kRampR; ++j) acc[j] = fma2(h, add2(lo[j + kRampR - k], hi[j + k - 1]), acc[j]);
        }
    }
    for (int k = k0 + 1; k <= K; ++k) {
        const unsigned long long h = pack2(taps.h[k], taps.h[k]);
#pragma unroll
        for (int j = 0; j < kRampR; ++j) acc[j] = fma2(h, add2(c[(j - k) * kStep], c[(j + k) * kStep]), acc[j]);
    }
    const float4 vi = T.vinfo[p];
    const float ax0 = T.xt[(size_t)p * nu + u].w, ax1 = u + 1 < nu ? T.xt[(size_t)p * nu + u + 1].w : 0.f;
#pragma unroll
    for (int j = 0; j < kRampR; ++j) {
        const int v = v0 + o + j;
        if (v >= nv) break;
        const float ay = T.yt[(size_t)p * nv + v].w;
        float a0, a1;
        unpack2(acc[j], a0, a1);
        float *dst = out + base + (size_t)v * nu + u;
        dst[0] = __fmul_rn(a0, ray_factor(ax0, ay, vi));
        if (u + 1 < nu) dst[1] = __fmul_rn(a1, ray_factor(ax1, ay, vi));
    }
}

}  // namespace

kv_status ramp_filter_launch(kv_plan *plan, const float *in, float *out, int half_taps) {
    const kv_geometry &g = plan->g;
    RampTaps taps;
    for (int n = 0; n <= half_taps; ++n)
        taps.h[n] = (float)(-2.0 / (M_PI * M_PI * (4.0 * (double)n * n - 1.0)));
    const size_t smem = (size_t)(kRampRows + 2 * half_taps) * kRampCols * sizeof(float);
    KV_CHECK_CUDA(plan->ctx, cudaFuncSetAttribute(ramp_v_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)smem));
    const int wide = g.nu % 4 == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
    dim3 grid((g.nu + kRampCols - 1) / kRampCols, (g.nv + kRampRows - 1) / kRampRows, g.n_views);
    LaunchTimer lt(plan->ctx, "ramp_v");
    ramp_v_kernel<<<grid, 128, smem, plan->ctx->stream>>>(in, out, g.nu, g.nv, half_taps, wide, taps, plan->ex);
    KV_CHECK_LAUNCH(plan->ctx, "ramp_v_kernel");
    return KV_OK;
}

namespace {

// Rows of the band a block of the staged kernel needs: kSaaRows + the
// largest spread of one block's shifts over its ks slices, for any view.
int saa_band_rows(const kv_geometry &g, const int32_t *sh, int ks) {
    int span = 0;
    for (int k0 = 0; k0 < g.nz; k0 += ks)
        for (int i = 0; i < g.n_views; ++i) {
            int lo = sh[(size_t)k0 * g.n_views + i], hi = lo;
            for (int k = k0 + 1; k < std::min(g.nz, k0 + ks); ++k) {
                lo = std::min(lo, sh[(size_t)k * g.n_views + i]);
                hi = std::max(hi, sh[(size_t)k * g.n_views + i]);
            }
            span = std::max(span, hi - lo);
        }
    return kSaaRows + span;
}

// The staged kernel with KS slices a block; false where its band does not fit.
template <int KS>
bool saa_band_launch(kv_plan *plan, const int32_t *d_shift, const int32_t *h_shift, const float *proj, float *out,
                     size_t smem_limit, kv_status *status) {
    const kv_geometry &g = plan->g;
    kv_ctx *ctx = plan->ctx;
    const int nb = saa_band_rows(g, h_shift, KS);
    const uint32_t stride = (uint32_t)((32u * nb * 4u + 127u) / 128u * 128u);
    const size_t smem = (size_t)kSaaStages * stride + (size_t)(KS + 1) * g.n_views * sizeof(int32_t) + 128;
    if (nb > 256 || smem > smem_limit) return false;
    CUtensorMap map;
    cuuint64_t dims[3] = {(cuuint64_t)g.nu, (cuuint64_t)g.nv, (cuuint64_t)g.n_views};
    cuuint64_t strides[2] = {(cuuint64_t)g.nu * 4, (cuuint64_t)g.nu * g.nv * 4};
    cuuint32_t box[3] = {32, (cuuint32_t)nb, 1};
    cuuint32_t es[3] = {1, 1, 1};
    if (kvtma::encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(proj), dims, strides, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    *status = [&]() -> kv_status {
        KV_CHECK_CUDA(ctx, cudaFuncSetAttribute(saa_band_kernel<KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        dim3 grid((g.nu + 31) / 32, (g.nv + kSaaRows - 1) / kSaaRows, (g.nz + KS - 1) / KS);
        LaunchTimer lt(ctx, "saa");
        saa_band_kernel<KS><<<grid, 256, smem, ctx->stream>>>(map, g.nu, g.nv, g.nz, g.n_views, d_shift, out, nb, stride,
                                                              reinterpret_cast<uintptr_t>(out) % 8 == 0, ctx->d_status);
        KV_CHECK_LAUNCH(ctx, "saa_band_kernel");
        return KV_OK;
    }();
    return true;
}

}  // namespace

kv_status saa_launch(kv_plan *plan, const int32_t *d_shift, const int32_t *h_shift, const float *proj, float *out) {
    const kv_geometry &g = plan->g;
    kv_ctx *ctx = plan->ctx;
    // the staged kernel where its band fits and TMA can address the stack; eight slices a block where two blocks
    // stay resident.  Four slices as far as shared memory goes: the direct kernel, next, is slower and takes 1536 views
    if ((g.nu * 4) % 16 == 0 && reinterpret_cast<uintptr_t>(proj) % 16 == 0 && kvtma::encoder() != nullptr) {
        kv_status s = KV_OK;
        if (saa_band_launch<8>(plan, d_shift, h_shift, proj, out, 100 * 1024, &s) ||
            saa_band_launch<4>(plan, d_shift, h_shift, proj, out, 208 * 1024, &s))
            return s;
    }
    const int kb = 8;
    dim3 block(32, 8), grid((g.nu + 31) / 32, (g.nv + 7) / 8, (g.nz + kb - 1) / kb);
    size_t smem1 = (size_t)kb * g.n_views * sizeof(int32_t);
    if (smem1 > 48 * 1024) return kv_fail(ctx, KV_ERR_UNSUPPORTED, "shift-and-add: too many views");
    LaunchTimer lt(ctx, "saa");
    saa_kernel<<<grid, block, smem1, ctx->stream>>>(g.nu, g.nv, g.nz, g.n_views, d_shift, proj, out, kb);
    KV_CHECK_LAUNCH(ctx, "saa_kernel");
    return KV_OK;
}

kv_status fill_launch(kv_ctx *ctx, float *p, size_t n, float v) {
    LaunchTimer lt(ctx, "fill");
    fill_kernel<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(p, n, v);
    KV_CHECK_LAUNCH(ctx, "fill_kernel");
    return KV_OK;
}

kv_status convert_launch(kv_ctx *ctx, const float *in, void *out, size_t n, kv_storage s) {
    int gb = grid_for(ctx, n, 256);
    LaunchTimer lt(ctx, "to_storage");
    if (s == KV_STORAGE_BF16) to_storage_kernel<__nv_bfloat16><<<gb, 256, 0, ctx->stream>>>(in, (__nv_bfloat16 *)out, n);
    else if (s == KV_STORAGE_F16) to_storage_kernel<__half><<<gb, 256, 0, ctx->stream>>>(in, (__half *)out, n);
    else to_storage_kernel<float><<<gb, 256, 0, ctx->stream>>>(in, (float *)out, n);
    KV_CHECK_LAUNCH(ctx, "to_storage_kernel");
    return KV_OK;
}

kv_status convert_back_launch(kv_ctx *ctx, const void *in, float *out, size_t n, kv_storage s) {
    int gb = grid_for(ctx, n, 256);
    LaunchTimer lt(ctx, "from_storage");
    if (s == KV_STORAGE_BF16) from_storage_kernel<__nv_bfloat16><<<gb, 256, 0, ctx->stream>>>((const __nv_bfloat16 *)in, out, n);
    else if (s == KV_STORAGE_F16) from_storage_kernel<__half><<<gb, 256, 0, ctx->stream>>>((const __half *)in, out, n);
    else from_storage_kernel<float><<<gb, 256, 0, ctx->stream>>>((const float *)in, out, n);
    KV_CHECK_LAUNCH(ctx, "from_storage_kernel");
    return KV_OK;
}

kv_status phantom_launch(kv_ctx *ctx, int nx, int ny, int nz, float dx, float dy, float dz,
                         const float *d_params, int n, float *vol) {
    size_t smem = (size_t)16 * n * sizeof(float);
    if (smem > 200 * 1024) return kv_fail(ctx, KV_ERR_INVALID_ARG, "phantom: too many ellipsoids");
    if (smem > 48 * 1024)
        KV_CHECK_CUDA(ctx, cudaFuncSetAttribute(phantom_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    size_t total = (size_t)nx * ny * nz;
    LaunchTimer lt(ctx, "phantom");
    phantom_kernel<<<grid_for(ctx, total, 256), 256, smem, ctx->stream>>>(nx, ny, nz, dx, dy, dz, d_params, n, vol);
    KV_CHECK_LAUNCH(ctx, "phantom_kernel");
    return KV_OK;
}

kv_status residual_reduce_launch(kv_ctx *ctx, const float *q, const float *p, size_t n, double *red) {
    const int nblocks = ctx->sm_count > 0 ? ctx->sm_count * 4 : 512;
    double *partials = nullptr;
    KV_CHECK_CUDA(ctx, cudaMallocAsync((void **)&partials, (size_t)nblocks * 3 * sizeof(double), ctx->stream));
    {
        LaunchTimer lt(ctx, "residual_partials");
        residual_partials_kernel<<<nblocks, 256, 0, ctx->stream>>>(q, p, n, partials);
    }
    {
        LaunchTimer lt(ctx, "sum_partials");
        sum_partials_kernel<<<1, 256, 0, ctx->stream>>>(partials, nblocks, red);
    }
    cudaError_t e = cudaGetLastError();
    cudaFreeAsync(partials, ctx->stream);
    if (e != cudaSuccess) return kv_fail(ctx, KV_ERR_CUDA, "residual reduction: %s", cudaGetErrorString(e));
    return KV_OK;
}

// ---------------------------------------------------------------------------
// The learned warm start's elementwise steps (device buffers)
// ---------------------------------------------------------------------------

extern "C" kv_status kv_warm_ratio(kv_ctx *ctx, const float *p, const float *a1, float *ratio, size_t n,
                                   double *uniform_residual) {
    if (ctx == nullptr) return KV_ERR_INVALID_ARG;
    if (p == nullptr || a1 == nullptr || ratio == nullptr || n == 0)
        return kv_fail(ctx, KV_ERR_INVALID_ARG, "kv_warm_ratio: null buffer or empty");
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    const int blocks = grid_for(ctx, n, 256);
    double *partials = nullptr;
    KV_CHECK_CUDA(ctx, cudaMallocAsync((void **)&partials, 2 * sizeof(double) * blocks, ctx->stream));
    {
        LaunchTimer lt(ctx, "warm_ratio");
        warm_ratio_kernel<<<blocks, 256, 0, ctx->stream>>>(p, a1, ratio, n, partials);
        sum_pairs_kernel<<<1, 256, 0, ctx->stream>>>(partials, blocks, ctx->d_red);
    }
    cudaError_t e = cudaGetLastError();
    cudaFreeAsync(partials, ctx->stream);
    if (e != cudaSuccess) return kv_fail(ctx, KV_ERR_CUDA, "kv_warm_ratio: %s", cudaGetErrorString(e));
    if (uniform_residual != nullptr) {
        double h[2];
        KV_CHECK_CUDA(ctx, cudaMemcpyAsync(h, ctx->d_red, sizeof h, cudaMemcpyDeviceToHost, ctx->stream));
        KV_CHECK_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        *uniform_residual = h[1] > 0.0 ? std::sqrt(h[0] / h[1]) : std::sqrt(h[0]);
    }
    return KV_OK;
}

extern "C" kv_status kv_warm_normalize(kv_ctx *ctx, const float *b, const double *sens, float *out, size_t n) {
    if (ctx == nullptr) return KV_ERR_INVALID_ARG;
    if (b == nullptr || sens == nullptr || out == nullptr || n == 0)
        return kv_fail(ctx, KV_ERR_INVALID_ARG, "kv_warm_normalize: null buffer or empty");
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    LaunchTimer lt(ctx, "warm_normalize");
    warm_normalize_kernel<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(b, sens, out, n);
    KV_CHECK_LAUNCH(ctx, "warm_normalize_kernel");
    return KV_OK;
}

extern "C" kv_status kv_warm_fill(kv_ctx *ctx, const float *net, const float *saa, const uint8_t *seen, float eps,
                                  float *out, size_t n) {
    if (ctx == nullptr) return KV_ERR_INVALID_ARG;
    if (net == nullptr || saa == nullptr || seen == nullptr || out == nullptr || n == 0)
        return kv_fail(ctx, KV_ERR_INVALID_ARG, "kv_warm_fill: null buffer or empty");
    KV_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
    LaunchTimer lt(ctx, "warm_fill");
    warm_fill_kernel<<<grid_for(ctx, n, 256), 256, 0, ctx->stream>>>(net, saa, seen, eps, out, n);
    KV_CHECK_LAUNCH(ctx, "warm_fill_kernel");
    return KV_OK;
}
