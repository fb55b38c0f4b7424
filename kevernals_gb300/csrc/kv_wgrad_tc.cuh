// kv_wgrad_tc.cuh -- weight gradient of the 3x3x3 convolution on the
// Blackwell tensor cores (tcgen05.mma, both operands MN-major).
//
//   dW[co][tap][ci] = sum over voxels v of dY[v - tap][co] * X[v][ci]
//
// A GEMM whose K runs over voxels.  With 16 channels a side one product per
// tap would leave M = 64 three quarters empty and read every tensor 27 times,
// so the taps fill the tile: operands are 16-channel segments of a plane in
// shared memory, one 32-byte row per voxel, and the segments' "next 16 rows
// of M (or N)" stride is set to a shift instead of to other channels:
//   M = 64:  dY at rows y - 1 (dy = 2), y (1), y + 1 (0) and an unused fourth,
//            16 output channels each;
//   N = 48:  X at columns x - 1 (dx = 0), x, x + 1, 16 input channels each;
// one MMA of 16 voxels of a row adds to nine taps, and three accumulators per
// (16 out, 16 in) channel pair (dz = 0, 1, 2) hold all 27.  A CTA owns 16
// output channels and up to three input segments (nine accumulators, 432 TMEM
// columns) and marches along z over its share of (column, plane) units; X
// planes pass through a ring of two, dY planes through a ring of four (each
// meets the X planes above, at and below it).
//
// FP32 sums in TMEM are cut every 256 MMAs (4096 voxels) and added to the FP32
// gradient: a longer run would add more truncation than the mma.sync kernel's,
// which this one replaces, had.
//
// What bounds it: an MMA reads 64 + 48 rows of 32 bytes from shared memory (28
// cycles at 128 B a cycle) for 24 cycles of arithmetic.  Measured on a GB300,
// the thirteen layers at 128 x 256 x 128 voxels: 13.5 ms with mma.sync, one tap
// a CTA, -> 1.24 ms (0.54 TFLOP, 440 TFLOP/s).
//
// Along x and y a voxel outside the volume enters as zero: X's halo columns, dY's
// halo rows.  Along z planes outside are not visited.  So a non-finite activation
// in a border row, or gradient in a border column, also reaches the taps that
// pair it with the outside; other border values do not.
//
// Warp roles (256 threads): warp 0 issues the TMA loads, warps 1-3 the MMAs of
// dz = 0, 1, 2, warps 4-7 read the accumulators out.  Every wait is bounded,
// as in kv_conv_tc.cuh.
#pragma once

#include "kv_conv_tc.cuh"

namespace wgradtc {

using namespace convtc;

constexpr int kWThreads = 256;
constexpr int kXStages = 2, kYStages = 4;
constexpr int kMaxNC = 3;         // input segments of a CTA
constexpr int kShifts = 3;        // N atoms
constexpr int kN = kShifts * kSeg;
constexpr int kFlush = 256;       // MMAs into one accumulator before it is read out

struct WParams {
    int nco, ngroups;             // output segments; groups of input segments
    int nc;                       // input segments of the largest group
    int nseg, nseg1;              // input segments; the first nseg1 come from the first tensor
    int D, H, W, BW, BY, tiles_x, pitch_x;
    long long units;              // columns x planes
    int flush;                    // planes between read-outs
    uint32_t x_bytes, y_bytes;    // one segment of an X plane, one dY plane (rounded up to 1024)
    uint32_t x_tx, y_tx;          // bytes their loads deliver
    uint32_t y_off;               // first byte of the dY ring
    uint32_t tmem_cols;
    int cin;
    float *dw;                    // [cout][27][cin], added to
    int *status;
};

// Descriptor of an MN-major tile of 32-byte rows (16 channels of one voxel) with the 32-byte swizzle: `next` = bytes
// to the next 16 rows of M or N (leading byte offset), 8 voxels to the next 8 of K (stride byte offset).
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr, uint32_t next) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((next >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((8u * kRow) >> 4) << 32) | (1ull << 46) | (6ull << 61);
}

__device__ __forceinline__ void tc_mma2(uint32_t tmem_d, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                        uint32_t idesc) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, 1, 0;\n mov.b64 a, {%1, %2};\n mov.b64 b, {%3, %4};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p;\n}\n" ::"r"(tmem_d),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc)
        : "memory");
}

__global__ void __launch_bounds__(kWThreads, 1)
    wgrad_march_kernel(const __grid_constant__ CUtensorMap map_x0, const __grid_constant__ CUtensorMap map_x1,
                       const __grid_constant__ CUtensorMap map_y, const __grid_constant__ WParams P) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t x_full[kXStages], x_empty[kXStages], y_full[kYStages], y_empty[kYStages],
        acc_full, acc_empty, drain_bar[3];
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;
    __shared__ unsigned long long x_issued_sh, y_issued_sh;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int i = 0; i < kXStages; ++i) {
            mbar_init(&x_full[i], 1);
            mbar_init(&x_empty[i], 3);
        }
        for (int i = 0; i < kYStages; ++i) {
            mbar_init(&y_full[i], 1);
            mbar_init(&y_empty[i], 3);
        }
        mbar_init(&acc_full, 3);
        mbar_init(&acc_empty, 4);
        for (int i = 0; i < 3; ++i) mbar_init(&drain_bar[i], 1);
        x_issued_sh = 0;
        y_issued_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_base_sh)),
                     "r"(P.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_sh;
    if (warp >= 4) {   // every accumulator starts at zero
        for (uint32_t c = 0; c < P.tmem_cols; c += 16) tc_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c);
        tc_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();

    // this CTA's channels and its range of (column, plane) units
    const int ncombo = P.nco * P.ngroups, combo = (int)blockIdx.x % ncombo;
    const int co = combo / P.ngroups, grp = combo % P.ngroups;
    const int s_begin = grp * P.nseg / P.ngroups, nc = (grp + 1) * P.nseg / P.ngroups - s_begin;
    const long long part = (long long)blockIdx.x / ncombo, parts = (long long)gridDim.x / ncombo;
    const long long u_begin = P.units * part / parts, u_end = P.units * (part + 1) / parts;

    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer
        if (lane == 0) {
            uint32_t xs = 0, xphase = 0, ys = 0, yphase = 0;
            bool ok = true;
            for (long long u = u_begin; u < u_end && ok;) {
                const int col = (int)(u / P.D), zs = (int)(u % P.D);
                const int ze = (int)(u_end - u < P.D - zs ? zs + (u_end - u) : P.D);
                const int x0 = (col % P.tiles_x) * P.BW, y0 = (col / P.tiles_x) * P.BY;
                int zy = max(zs - 1, 0);
                for (int z = zs; z < ze && ok; ++z) {
                    for (; zy <= min(z + 1, P.D - 1); ++zy) {
                        if (!mbar_wait(&y_empty[ys], yphase ^ 1u, &abort_flag, P.status, 11)) { ok = false; break; }
                        mbar_arrive_expect_tx(&y_full[ys], P.y_tx);
                        tma_load_4d(base + P.y_off + ys * P.y_bytes, &map_y, &y_full[ys], co * kSeg, x0, y0 - 1, zy);
                        ++y_issued_sh;
                        if (++ys == kYStages) { ys = 0; yphase ^= 1u; }
                    }
                    if (!ok || !mbar_wait(&x_empty[xs], xphase ^ 1u, &abort_flag, P.status, 12)) { ok = false; break; }
                    mbar_arrive_expect_tx(&x_full[xs], P.x_tx * (uint32_t)nc);
                    for (int s = 0; s < nc; ++s) {
                        const int g = s_begin + s;
                        tma_load_4d(base + (xs * (uint32_t)P.nc + (uint32_t)s) * P.x_bytes, g < P.nseg1 ? &map_x0 : &map_x1,
                                    &x_full[xs], (g < P.nseg1 ? g : g - P.nseg1) * kSeg, x0 - 1, y0, z);
                    }
                    ++x_issued_sh;
                    if (++xs == kXStages) { xs = 0; xphase ^= 1u; }
                }
                u += ze - zs;
            }
        }
    } else if (warp < 4) {
        // ---------------------------------------------------------- MMA issuers: X plane z with dY plane z + 1 - dz
        const int dz = warp - 1;
        // kind::f16: FP32 accumulator, BF16 A and B, both MN-major (bits 15, 16), N >> 3 at 17-22, M >> 4 at 24-28
        constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) |
                                    ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(64 >> 4) << 24);
        const uint32_t ubase = __shfl_sync(0xffffffffu, base, 0), utmem = __shfl_sync(0xffffffffu, tmem, 0);
        const uint64_t da = smem_desc_mn(ubase + P.y_off, (uint32_t)P.BW * kRow), db = smem_desc_mn(ubase, kRow);
        const uint32_t a_lo = (uint32_t)da, a_hi = (uint32_t)(da >> 32), b_lo = (uint32_t)db, b_hi = (uint32_t)(db >> 32);
        const uint32_t x_seg = P.x_bytes >> 4;
        auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
            return __all_sync(0xffffffffu, mbar_wait(bar, parity, &abort_flag, P.status, code));
        };
        uint32_t xs = 0, xphase = 0, ys = 0, yphase = 0, acc_phase = 0;
        int since = 0;
        bool ok = true;
        // a dY plane of the ring: waits for it, optionally with MMAs, then frees it
        auto next_y = [&]() {
            tc_commit(&y_empty[ys]);
            if (++ys == kYStages) { ys = 0; yphase ^= 1u; }
        };
        for (long long u = u_begin; u < u_end && ok;) {
            const int col = (int)(u / P.D), zs = (int)(u % P.D);
            const int ze = (int)(u_end - u < P.D - zs ? zs + (u_end - u) : P.D);
            const int rows = min(P.BY, P.H - (col / P.tiles_x) * P.BY), runs = P.BW / 16;
            const int y_last = min(ze, P.D - 1);
            int zy = max(zs - 1, 0);
            for (int z = zs; z < ze && ok; ++z) {
                const int zo = z + 1 - dz;
                for (; zy <= y_last && zy < zo; ++zy) {   // planes this dz does not use
                    if (!wait(&y_full[ys], yphase, 13)) { ok = false; break; }
                    next_y();
                }
                if (!ok || !wait(&x_full[xs], xphase, 14)) { ok = false; break; }
                if (zo >= 0 && zo < P.D) {
                    if (!wait(&y_full[ys], yphase, 15)) { ok = false; break; }
                    tc_fence_after();
                    for (int r = 0; r < rows; ++r) {
                        const uint32_t a = a_lo + ((ys * P.y_bytes) >> 4) + (uint32_t)(r * P.BW) * (kRow >> 4);
                        const uint32_t b =
                            b_lo + ((xs * (uint32_t)P.nc * P.x_bytes) >> 4) + (uint32_t)(r * P.pitch_x) * (kRow >> 4);
                        const uint32_t d = utmem + (uint32_t)(dz * kN);
                        if (elect_one()) {
                            for (int c = 0; c < runs; ++c)
                                for (int s = 0; s < nc; ++s)
                                    tc_mma2(d + (uint32_t)(s * 3 * kN), a + (uint32_t)c * (16 * kRow >> 4), a_hi,
                                            b + (uint32_t)c * (16 * kRow >> 4) + (uint32_t)s * x_seg, b_hi, kIdesc);
                        }
                        __syncwarp();
                    }
                    next_y();
                    ++zy;
                }
                tc_commit(&x_empty[xs]);
                if (++xs == kXStages) { xs = 0; xphase ^= 1u; }
                if (++since == P.flush || u + (z - zs) + 1 == u_end) {
                    since = 0;
                    tc_commit(&acc_full);
                    if (!wait(&acc_empty, acc_phase, 16)) { ok = false; break; }
                    tc_fence_after();
                    acc_phase ^= 1u;
                }
            }
            for (; ok && zy <= y_last; ++zy) {
                if (!wait(&y_full[ys], yphase, 13)) { ok = false; break; }
                next_y();
            }
            u += ze - zs;
        }
        tc_commit(&drain_bar[dz]);
        volatile int never = 0;
        mbar_wait(&drain_bar[dz], 0, &never, P.status, 17);
    } else {
        // ---------------------------------------------------------- read-out (warps 4-7): M rows 16 q .. + 15 lie in
        // TMEM lanes 32 q .. + 15; quarter q holds dy = 2 - q
        const int q = warp & 3;
        uint32_t acc_phase = 0;
        for (long long u = u_begin; u < u_end;) {
            const bool got = mbar_wait(&acc_full, acc_phase, &abort_flag, P.status, 18);
            if (!__all_sync(0xffffffffu, got)) break;
            acc_phase ^= 1u;
            tc_fence_after();
            for (int s = 0; s < nc; ++s)
                for (int dz = 0; dz < 3; ++dz) {
                    const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((s * 3 + dz) * kN);
                    uint32_t v[kShifts][16];
#pragma unroll
                    for (int dx = 0; dx < kShifts; ++dx) tc_ld16(ta + (uint32_t)(dx * 16), v[dx]);
                    tc_wait_ld();
#pragma unroll
                    for (int dx = 0; dx < kShifts; ++dx) tc_zero16(ta + (uint32_t)(dx * 16));
                    if (q < 3 && lane < 16) {
                        float *dst = P.dw + ((size_t)(co * kSeg + lane) * 27 + dz * 9 + (2 - q) * 3) * P.cin +
                                     (s_begin + s) * kSeg;
#pragma unroll
                        for (int dx = 0; dx < kShifts; ++dx)
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                atomicAdd(reinterpret_cast<float4 *>(dst + (size_t)dx * P.cin) + j,
                                          make_float4(__uint_as_float(v[dx][4 * j]), __uint_as_float(v[dx][4 * j + 1]),
                                                      __uint_as_float(v[dx][4 * j + 2]),
                                                      __uint_as_float(v[dx][4 * j + 3])));
                    }
                    __syncwarp();
                }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty);
            u += u_end - u < P.flush ? u_end - u : P.flush;
        }
    }

    // wind down: every role has left its loop (all waits are bounded)
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag) {
        volatile int never = 0;   // loads still in flight: at most the last ones into each buffer
        for (unsigned long long i = x_issued_sh > kXStages ? x_issued_sh - kXStages : 0; i < x_issued_sh; ++i)
            mbar_wait(&x_full[i % kXStages], (uint32_t)((i / kXStages) & 1u), &never, P.status, 19);
        for (unsigned long long i = y_issued_sh > kYStages ? y_issued_sh - kYStages : 0; i < y_issued_sh; ++i)
            mbar_wait(&y_full[i % kYStages], (uint32_t)((i / kYStages) & 1u), &never, P.status, 19);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P.tmem_cols)
                     : "memory");
    }
}

// Adds the weight gradient of one convolution (input in1 (c1 channels) ++ in2 (c2), output gradient dy (cout)) to dw.
// Returns a message on a configuration this kernel does not cover (nullptr: launched).
inline const char *launch(const __nv_bfloat16 *dy, int cout, const __nv_bfloat16 *in1, int c1,
                          const __nv_bfloat16 *in2, int c2, float *dw, int D, int H, int W, int *status, int sm_count,
                          cudaStream_t stream) {
    if (encoder() == nullptr) return "cuTensorMapEncodeTiled is not available";
    if (c1 % kSeg || c2 % kSeg || cout % kSeg || W % 16) return "channels and W must be multiples of 16";
    WParams P{};
    P.nco = cout / kSeg;
    P.nseg = (c1 + c2) / kSeg;
    P.nseg1 = c1 / kSeg;
    P.ngroups = (P.nseg + kMaxNC - 1) / kMaxNC;
    P.D = D;
    P.H = H;
    P.W = W;
    P.cin = c1 + c2;
    P.dw = dw;
    P.status = status;
    int BW = std::min(W, 128);
    while (W % BW) BW -= 16;
    P.BW = BW;
    P.tiles_x = W / BW;
    P.pitch_x = BW + 2;
    const int ncombo = P.nco * P.ngroups, parts = std::max(1, sm_count / ncombo);
    const int nc = (P.nseg + P.ngroups - 1) / P.ngroups;
    P.nc = nc;
    // rows of a column: the least estimated time of the busiest CTA (28 cycles an MMA, loads at 32 B a cycle, 800
    // cycles of waits a plane, two more dY planes at the ends of its share)
    double best = 1e300;
    size_t smem = 0;
    long long grid = 0;
    for (int BY = 1; BY <= std::min(H, 253); ++BY) {
        const uint32_t xb = align1k((uint32_t)(BY * P.pitch_x * kRow)), yb = align1k((uint32_t)((BY + 3) * BW * kRow));
        const size_t need = (size_t)kXStages * nc * xb + (size_t)kYStages * yb + 1024;
        if (need > 224 * 1024) break;
        const long long units = (long long)P.tiles_x * ((H + BY - 1) / BY) * D;
        const double mma = 28.0 * 3 * nc * BY * (BW / 16), load = (nc * (double)xb + yb) / 32.0;
        const double total = (std::max(mma, load) + 800.0) * (double)((units + parts - 1) / parts) + 4.0 * yb / 32.0;
        if (total >= best) continue;
        best = total;
        P.BY = BY;
        P.units = units;
        P.x_bytes = xb;
        P.y_bytes = yb;
        P.x_tx = (uint32_t)(BY * P.pitch_x * kRow);
        P.y_tx = (uint32_t)((BY + 3) * BW * kRow);
        P.y_off = (uint32_t)(kXStages * nc) * xb;
        P.flush = std::max(1, kFlush / (BY * (BW / 16)));
        grid = std::min<long long>(parts, units) * ncombo;
        smem = need;
    }
    if (smem == 0) return "no tile shape for this volume";
    P.tmem_cols = nc == 1 ? 256 : 512;
    CUtensorMap x0, x1, y;
    if (!encode_act(&x0, in1, c1, D, H, W, P.pitch_x, P.BY) ||
        !encode_act(&x1, c2 ? in2 : in1, c2 ? c2 : c1, D, H, W, P.pitch_x, P.BY) ||
        !encode_act(&y, dy, cout, D, H, W, BW, P.BY + 3))
        return "activation tensor map rejected";
    if (cudaFuncSetAttribute(wgrad_march_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return "shared memory request rejected";
    wgrad_march_kernel<<<(unsigned)grid, kWThreads, smem, stream>>>(x0, x1, y, P);
    return nullptr;
}

}  // namespace wgradtc
