// kv_conv_tc.cuh -- 3x3x3 convolution as an implicit GEMM on the Blackwell
// tensor cores: TMA tile loads into swizzled shared memory, tcgen05.mma with
// the accumulators in tensor memory (TMEM), tcgen05.ld epilogue.
//
// GEMM view (channels-last activations [D][H][W][C], BF16): M = voxels, N =
// output channels, K = 27 taps x input channels.
//
// What bounds it and why it is cut this way.  A tile load per tap reads every
// activation 27 times through L2, and an MMA of N = 16 output channels reads
// 128 rows of A from shared memory (32 cycles at 128 B a cycle) for 8 cycles
// of arithmetic.  So a CTA marches along z over a column of the volume
// (BW x BY voxels, x by y): each input plane is loaded once, with a halo of
// one voxel, 16 channels at a time, and
//   * the nine (dy, dx) taps are the same shared-memory tile read from
//     another first row: a voxel is one 32-byte row, rows lie BW + 2 to the
//     next y, so a tap is a row offset of the operand's start address;
//   * the three dz taps are stacked along N: plane z times [W(dz=0) W(dz=1)
//     W(dz=2)] is added to the accumulators of the output planes z + 1, z and
//     z - 1 with one read of A.  Each 128-voxel sub-tile keeps three
//     accumulators (slots) in TMEM; output plane z uses slot (-z) mod 3, so the
//     three lie in the order of dz, cyclically.  Where the cycle wraps the MMA
//     is split in two, or, where shared memory allows it, the weights are kept
//     as five groups dz = 0 1 2 0 1 and the MMA starts at the rotated one.
// An output plane is finished with dz = 2, read out, and its slot zeroed for
// the plane three further on: every MMA accumulates.  Sums run over dz, then
// (dy, dx), then 16-channel segments -- the tap order of the mma.sync kernel,
// with equal bits -- so a plane's segments are all in shared memory at once.
// Planes outside the volume are not loaded; a weight that is not finite would
// have made their zeros NaN, which a variant's epilogue adds (z_border; 1 % of the
// network's time, which does without: its outputs are lost then anyway).
// The weights stay there for the CTA's life where they fit beside the plane
// buffers; else they stream through a ring, one (dy, dx) of up to four
// segments at a time, each piece used for every sub-tile.
//
// M = 128 rows are 128 consecutive voxels of the padded plane: either one y
// row (BW = 128; sub-tile t = row t) or, where the volume is narrower,
// consecutive rows with their halo columns in between, whose results are not
// stored.  The host takes the shape with the least estimated time.
//
// Measured on a GB300, against a kernel that loaded one tile per tap and
// issued one N = Cout MMA per tap and 16 channels: 32+16 -> 16 channels at
// 128 x 256 x 128 voxels 1434 -> 176 us (990 TFLOP/s); the thirteen layers of
// the U-Net at 128 x 512 x 512 voxels 31.9 -> 4.6 ms, forward and
// backward-data at 128 x 256 x 128 8.1 -> 1.7 ms.
//
// Warp roles: warp 0 issues the TMA loads of the planes and of streamed
// weights; two or four warps issue the MMAs, each its sub-tiles in turn (an MMA
// takes ~45 cycles and a sub-tile's waits, commit and address set-up ~240, so
// one issuer cannot keep the tensor pipe fed; warp 1 owns the TMEM allocation);
// two or four sets of four warps drain the accumulators (each warp its 32 TMEM
// lanes = 32 voxels; the sets take the sub-tiles in turn), add the bias, apply
// ReLU or the caller's mask, convert to BF16 and
// store.  The CTA is persistent over its share of (column, plane) units.
// Every wait on an mbarrier is bounded: on timeout the thread records an
// error code, raises the CTA's abort flag and every role winds down, so a
// fault in the pipeline ends the kernel with a status instead of a hang.
#pragma once

#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>

#include "kv_tma.cuh"

namespace convtc {

// Warps by channel group: MMA issuers and sets of four warps that drain
// accumulators.  With 16 channels a sub-tile's nine MMAs take ~400 cycles and
// draining it ~1400, so four sets (16 -> 16 channels at 64 x 512 x 512 voxels:
// two sets and four sub-tiles 318 us, four sets and eight sub-tiles 278);
// streamed weights of 32 channels want an issuer a sub-tile (96 -> 32 at 64 x 256 x 256: two 1020, four 840
// us); with 64 channels the MMAs are long and registers are short.
__host__ __device__ constexpr int issuers(int cg) { return cg == 32 ? 4 : 2; }
__host__ __device__ constexpr int drain_sets(int cg) { return cg <= 16 ? 4 : 2; }
__host__ __device__ constexpr int threads(int cg) { return (1 + issuers(cg) + 4 * drain_sets(cg)) * 32; }
constexpr int kMaxIssuers = 4;
constexpr int kTileM = 128;
constexpr int kSeg = 16;          // channels per segment: one K step, one 32-byte row per voxel
constexpr int kRow = kSeg * 2;    // bytes of a row
constexpr int kMaxT = 10;         // sub-tiles per column (512 TMEM columns / 3 slots of 16)
constexpr int kMaxStages = 4;     // plane buffers
constexpr int kMaxChunks = 8;     // ring of streamed weights
constexpr int kChunkSegs = 4;     // segments in one piece of streamed weights
constexpr uint32_t kWaitLimit = 1u << 22;   // try_wait rounds before a wait is declared failed

// Output layer of the network on the 16 channels h (rounded to BF16) of a voxel: y = x + (b + sum w h).
struct Head {
    const float *w, *b, *x;
    float *y;
};

struct Params {
    int nseg, nseg1;              // input segments; the first nseg1 come from the first tensor
    int N, ncg;                   // output channels; groups of CG channels, one per CTA
    int D, H, W;                  // this level's volume
    int BW, BY, pitch;            // column extent in x and y; rows from one y to the next (BW + 2)
    int T, mstep;                 // sub-tiles; rows between their first rows
    uint32_t pitch_magic;         // ceil(2^20 / pitch): row / pitch by multiplication
    int tiles_x;                  // columns in x
    long long units;              // columns x planes, of one channel group
    int groups;                   // dz groups of the weights in shared memory (3 or 5)
    int resident;                 // the weights stay in shared memory
    uint32_t stages, a_bytes;     // plane buffers; bytes of one segment of a plane
    uint32_t a_tx;                // bytes the TMA load of one segment of a plane delivers
    uint32_t b_off;               // first byte of the weights
    uint32_t b_seg_bytes;         // weights of one segment (resident: nine taps, streamed: one)
    uint32_t chunks;              // ring of streamed weights, kChunkSegs segments each
    uint32_t tmem_cols;
    const __nv_bfloat16 *w;       // [N][27][16 nseg], for z_border
    const float *bias;            // nullptr: none
    int relu;
    const __nv_bfloat16 *mask;    // nullptr: none; else outputs where mask <= 0 become 0
    __nv_bfloat16 *out;           // [voxels][N]; nullptr: not stored
    int out32;                    // out is 32-byte aligned
    Head head;                    // y == nullptr: none (N = 16 only)
    int *status;                  // 0 ok; set on a failed wait
};

using kvtma::mbar_arrive;
using kvtma::mbar_arrive_expect_tx;
using kvtma::mbar_init;
using kvtma::mbar_try_wait;
using kvtma::smem_u32;
using kvtma::tma_load_3d;
using kvtma::tma_load_4d;

// Bounded wait for the phase of `bar` with parity `parity` to complete.
// Returns false (after recording `code`) on timeout or when another role
// has already aborted.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort, int *status,
                                          int code) {
    for (uint32_t i = 0; i < kWaitLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
        if (i >= 16) __nanosleep(128);
    }
    atomicCAS(status, 0, code);
    *abort = 1;
    return false;
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One thread of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(pred));
    return pred != 0;
}

// D += A B, issued by one thread; the descriptors' low words (start address) differ from MMA to MMA, the high word is
// the same for every operand.
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t hi, uint32_t idesc) {
    asm volatile(
            "{\n .reg .pred p;\n .reg .b64 a, b;\n setp.ne.b32 p, 1, 0;\n mov.b64 a, {%1, %3};\n mov.b64 b, {%2, %3};\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n}\n" ::"r"(tmem_d),
            "r"(alo), "r"(blo), "r"(hi), "r"(idesc)
            : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t *bar) {
    if (elect_one())
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// zeroes 16 columns of the warp's 32 lanes
__device__ __forceinline__ void tc_zero16(uint32_t taddr) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
        "r"(0u)
        : "memory");
}

// 32 bytes as one store (32-byte aligned): two 16-byte stores a lane write every sector in two parts
__device__ __forceinline__ void st32(void *p, const uint4 &a, const uint4 &b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z),
                 "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile of 32-byte rows
// stored with the 32-byte swizzle by TMA: start address >> 4 (bits 0-13),
// leading byte offset (unused for swizzled K-major tiles, 16 bytes) >> 4
// (16-29), stride byte offset = 8 rows >> 4 (32-45), descriptor version 1
// (46-47), swizzle mode (61-63: 6 = 32 B).  The swizzle follows the address
// (TMA wrote the tile from a 1024-byte boundary), so a start address at any
// row reads the rows from there on.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1u << 16) | ((uint64_t)((8u * kRow) >> 4) << 32) |
           (1ull << 46) | (6ull << 61);
}

// The MMAs of NT taps (nine, or the one that `a` and the weights start at) of NS segments for one sub-tile, tap by
// tap, one piece (n1 == 0) or two; called by a converged warp, issued by one thread.
template <int NT, int NS>
__device__ __forceinline__ void issue_taps(uint32_t t0, uint32_t t1, uint32_t a, uint32_t b0, uint32_t b1, uint32_t hi,
                                           uint32_t id0, uint32_t id1, int n1, uint32_t y_step, uint32_t tap_step,
                                           uint32_t a_seg, uint32_t b_seg) {
    if (elect_one()) {
        // unrolled over dx and the segments only: all 36 addresses at once spilled (230 us on the layer above, now 176)
#pragma unroll 1
        for (int dy = 0; dy < (NT + 2) / 3; ++dy) {
            if (n1 == 0) {
#pragma unroll
                for (int dx = 0; dx < (NT < 3 ? NT : 3); ++dx)
#pragma unroll
                    for (int s = 0; s < NS; ++s)
                        tc_mma(t0, a + dx * (kRow >> 4) + s * a_seg, b0 + dx * tap_step + s * b_seg, hi, id0);
            } else {
#pragma unroll
                for (int dx = 0; dx < (NT < 3 ? NT : 3); ++dx)
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        tc_mma(t0, a + dx * (kRow >> 4) + s * a_seg, b0 + dx * tap_step + s * b_seg, hi, id0);
                        tc_mma(t1, a + dx * (kRow >> 4) + s * a_seg, b1 + dx * tap_step + s * b_seg, hi, id1);
                    }
            }
            a += y_step;
            b0 += 3 * tap_step;
            b1 += 3 * tap_step;
        }
    }
    __syncwarp();
}

// What the taps that reach a plane of zeros below (dz = 0, needed where `below`) or above (dz = 2, `above`) the volume
// add to each of the channels n0 .. n0 + CG - 1: 0, or NaN where a weight is not finite.  Called by the WARPS warps that
// drain accumulators while the first plane's MMAs run; their barrier makes it visible to them.
template <int CG, int WARPS>
__device__ __forceinline__ void z_border(const __nv_bfloat16 *w, int n0, int K, float (*border)[CG], bool below, bool above,
                                         int warp, int lane) {
    const int units = 9 * K / 8;   // of 16 bytes; the nine taps of one dz are contiguous
    auto not_finite = [](uint4 q) {
        const uint32_t v[4] = {q.x, q.y, q.z, q.w};
        bool bad = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) bad |= (v[j] & 0x7f80u) == 0x7f80u || (v[j] & 0x7f800000u) == 0x7f800000u;
        return bad;
    };
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int n = warp; n < CG; n += WARPS) {
        const uint4 *lo = reinterpret_cast<const uint4 *>(w + (size_t)(n0 + n) * 27 * K), *hi = lo + 2 * units;
        bool bad_lo = false, bad_hi = false;
        for (int i0 = lane; i0 < units; i0 += 128) {   // eight loads in flight
            uint4 q[4], r[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                q[j] = below && i0 + 32 * j < units ? __ldg(lo + i0 + 32 * j) : zero;
                r[j] = above && i0 + 32 * j < units ? __ldg(hi + i0 + 32 * j) : zero;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bad_lo |= not_finite(q[j]);
                bad_hi |= not_finite(r[j]);
            }
        }
        const bool nan_lo = __any_sync(0xffffffffu, bad_lo), nan_hi = __any_sync(0xffffffffu, bad_hi);
        if (lane == 0) {
            border[0][n] = nan_lo ? __int_as_float(0x7fffffff) : 0.f;
            border[1][n] = nan_hi ? __int_as_float(0x7fffffff) : 0.f;
        }
    }
    asm volatile("bar.sync 1, %0;" ::"r"(32 * WARPS) : "memory");
}

// ANY_W: the weights may hold infinities and NaN.
template <int CG, bool ANY_W>
__global__ void __launch_bounds__(threads(CG), 1)
    conv3_march_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                       const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_b2,
                       const __grid_constant__ Params P) {
    constexpr int kIssuers = issuers(CG), kSets = drain_sets(CG);
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], acc_full[kMaxT], acc_empty[kMaxT],
        b_full[kMaxChunks], b_empty[kMaxChunks], drain_bar[kMaxIssuers];
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int abort_flag;
    __shared__ unsigned long long issued_sh, b_issued_sh;   // planes / pieces of weights loaded by TMA
    __shared__ float border[2][CG];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (uint32_t s = 0; s < P.stages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], kIssuers);
        }
        for (int t = 0; t < P.T; ++t) {
            mbar_init(&acc_full[t], 1);
            mbar_init(&acc_empty[t], 4);
        }
        for (int i = 0; i < kMaxChunks; ++i) {
            mbar_init(&b_full[i], 1);
            mbar_init(&b_empty[i], kIssuers);
        }
        for (int i = 0; i < kIssuers; ++i) mbar_init(&drain_bar[i], 1);
        issued_sh = 0;
        b_issued_sh = 0;
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
    if (warp > kIssuers && warp <= kIssuers + 4) {   // every accumulator starts at zero
        for (uint32_t c = 0; c < P.tmem_cols; c += 16) tc_zero16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + c);
        tc_wait_st();
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();

    // this CTA's channel group and its range of (column, plane) units
    const int cg = (int)blockIdx.x % P.ncg;
    const long long part = (long long)blockIdx.x / P.ncg, parts = (long long)gridDim.x / P.ncg;
    const long long u_begin = P.units * part / parts, u_end = P.units * (part + 1) / parts;

    if (warp == 0) {
        // ---------------------------------------------------------- TMA producer
        if (lane == 0) {
            if (P.resident) {
                mbar_arrive_expect_tx(&b_full[0], P.b_seg_bytes * (uint32_t)P.nseg);
                for (int s = 0; s < P.nseg; ++s) {
                    const uint32_t sb = base + P.b_off + (uint32_t)s * P.b_seg_bytes;
                    if (P.groups == 5) {
                        for (int tap = 0; tap < 9; ++tap) {
                            const uint32_t tb = sb + (uint32_t)(tap * 5 * CG * kRow);
                            tma_load_4d(tb, &map_b, &b_full[0], s * kSeg, cg * CG, 0, tap);
                            tma_load_4d(tb + 3u * CG * kRow, &map_b2, &b_full[0], s * kSeg, cg * CG, 0, tap);
                        }
                    } else {
                        tma_load_4d(sb, &map_b, &b_full[0], s * kSeg, cg * CG, 0, 0);
                    }
                }
                b_issued_sh = 1;
            }
            uint32_t stage = 0, phase = 0, chunk = 0, bphase = 0;
            bool ok = true;
            for (long long u = u_begin; u < u_end && ok;) {
                const int col = (int)(u / P.D), zs = (int)(u % P.D);
                const int ze = (int)(u_end - u < P.D - zs ? zs + (u_end - u) : P.D);
                const int x0 = (col % P.tiles_x) * P.BW, y0 = (col / P.tiles_x) * P.BY;
                for (int z = max(zs - 1, 0); z <= min(ze, P.D - 1) && ok; ++z) {
                    if (!mbar_wait(&empty_bar[stage], phase ^ 1u, &abort_flag, P.status, 1)) { ok = false; break; }
                    mbar_arrive_expect_tx(&full_bar[stage], P.a_tx * (uint32_t)P.nseg);
                    const uint32_t sb = base + stage * (uint32_t)P.nseg * P.a_bytes;
                    for (int s = 0; s < P.nseg; ++s)
                        tma_load_4d(sb + (uint32_t)s * P.a_bytes, s < P.nseg1 ? &map_a0 : &map_a1, &full_bar[stage],
                                    (s < P.nseg1 ? s : s - P.nseg1) * kSeg, x0 - 1, y0 - 1, z);
                    ++issued_sh;
                    if (++stage == P.stages) { stage = 0; phase ^= 1u; }
                    if (P.resident) continue;
                    for (int tap = 0; tap < 9 && ok; ++tap)
                        for (int s0 = 0; s0 < P.nseg; s0 += kChunkSegs) {
                            const int ns = min(kChunkSegs, P.nseg - s0);
                            if (!mbar_wait(&b_empty[chunk], bphase ^ 1u, &abort_flag, P.status, 7)) { ok = false; break; }
                            mbar_arrive_expect_tx(&b_full[chunk], P.b_seg_bytes * (uint32_t)ns);
                            const uint32_t cb = base + P.b_off + chunk * (uint32_t)kChunkSegs * P.b_seg_bytes;
                            for (int s = 0; s < ns; ++s)
                                tma_load_4d(cb + (uint32_t)s * P.b_seg_bytes, &map_b, &b_full[chunk],
                                            (s0 + s) * kSeg, cg * CG, 0, tap);
                            ++b_issued_sh;
                            if (++chunk == P.chunks) { chunk = 0; bphase ^= 1u; }
                        }
                }
                u += ze - zs;
            }
        }
    } else if (warp <= kIssuers) {
        // ---------------------------------------------------------- MMA issuers
        const int issuer = warp - 1;
        // The whole warp runs this role converged (every wait's outcome is agreed on by a vote) and one elected
        // thread issues: the operands of tcgen05.mma live in uniform registers, and values computed in a
        // one-thread branch would have to be moved there MMA by MMA.
        //
        // kind::f16 instruction descriptor: FP32 accumulator (bits 4-5 = 1), BF16 A
        // and B (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28
        constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTileM >> 4) << 24);
        constexpr uint32_t kIdescN = (uint32_t)(CG >> 3) << 17;   // per dz group
        constexpr uint32_t kGroup = (uint32_t)(CG * kRow) >> 4;
        constexpr uint32_t kRowStep = kRow >> 4;
        const uint32_t ubase = __shfl_sync(0xffffffffu, base, 0), utmem = __shfl_sync(0xffffffffu, tmem, 0);
        const uint32_t lo0 = (uint32_t)smem_desc(ubase), hi = (uint32_t)(smem_desc(0) >> 32);
        const uint32_t tap_step = (uint32_t)P.groups * kGroup, y_step = (uint32_t)P.pitch * kRowStep;
        const uint32_t a_seg = P.a_bytes >> 4, b_seg = P.b_seg_bytes >> 4;
        auto wait = [&](uint64_t *bar, uint32_t parity, int code) {
            return __all_sync(0xffffffffu, mbar_wait(bar, parity, &abort_flag, P.status, code));
        };
        uint32_t stage = 0, phase = 0, plane_phase = 0, chunk = 0, bphase = 0;
        bool ok = true;
        if (P.resident && u_begin < u_end) ok = wait(&b_full[0], 0, 8);
        for (long long u = u_begin; u < u_end && ok;) {
            const int zs = (int)(u % P.D);
            const int ze = (int)(u_end - u < P.D - zs ? zs + (u_end - u) : P.D);
            for (int z = max(zs - 1, 0); z <= min(ze, P.D - 1) && ok; ++z) {
                // dz groups of plane z that fall on output planes zs .. ze-1 (plane z + 1 - dz), and the
                // slot of dz = 0; one piece, or two where the slots wrap
                const int dlo = max(0, z + 2 - ze), dhi = min(2, z + 1 - zs);
                const int c = (2 * (z + 1)) % 3;          // (-(z + 1)) mod 3
                int n0, b0, d0, n1 = 0, b1 = 0, d1 = 0;   // pieces: groups, first weight group, first slot
                if (P.groups == 5 && dlo == 0 && dhi == 2) {
                    n0 = 3;
                    b0 = (3 - c) % 3;
                    d0 = 0;
                } else {
                    const int wrap = min(max(3 - c, dlo), dhi + 1);   // first dz past the wrap
                    n0 = wrap - dlo;
                    b0 = dlo;
                    d0 = dlo + c;
                    n1 = dhi + 1 - wrap;
                    b1 = wrap;
                    d1 = wrap + c - 3;
                    if (n0 == 0) {
                        n0 = n1;
                        b0 = b1;
                        d0 = d1;
                        n1 = 0;
                    }
                }
                const uint32_t id0 = kIdesc + (uint32_t)n0 * kIdescN, id1 = kIdesc + (uint32_t)n1 * kIdescN;
                const uint32_t bo0 = (uint32_t)b0 * kGroup, bo1 = (uint32_t)b1 * kGroup;
                if (!wait(&full_bar[stage], phase, 3)) { ok = false; break; }
                tc_fence_after();
                const uint32_t da0 = lo0 + ((stage * (uint32_t)P.nseg * P.a_bytes) >> 4), db0 = lo0 + (P.b_off >> 4);
                if (P.resident) {
                    for (int t = issuer; t < P.T; t += kIssuers) {
                        if (!wait(&acc_empty[t], plane_phase ^ 1u, 2)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t dt = utmem + (uint32_t)(t * 3 * CG);
                        const uint32_t t0 = dt + (uint32_t)(d0 * CG), t1 = dt + (uint32_t)(d1 * CG);
                        const uint32_t at = da0 + (uint32_t)(t * P.mstep) * kRowStep;
                        switch (P.nseg) {
                        case 1: issue_taps<9, 1>(t0, t1, at, db0 + bo0, db0 + bo1, hi, id0, id1, n1, y_step, tap_step, a_seg, b_seg); break;
                        case 2: issue_taps<9, 2>(t0, t1, at, db0 + bo0, db0 + bo1, hi, id0, id1, n1, y_step, tap_step, a_seg, b_seg); break;
                        case 3: issue_taps<9, 3>(t0, t1, at, db0 + bo0, db0 + bo1, hi, id0, id1, n1, y_step, tap_step, a_seg, b_seg); break;
                        default: issue_taps<9, 4>(t0, t1, at, db0 + bo0, db0 + bo1, hi, id0, id1, n1, y_step, tap_step, a_seg, b_seg); break;
                        }
                        tc_commit(&acc_full[t]);   // the plane's sums are in
                    }
                } else {
                    for (int tap = 0; tap < 9 && ok; ++tap) {
                        const uint32_t ay = da0 + (uint32_t)(tap / 3) * y_step + (uint32_t)(tap % 3) * kRowStep;
                        for (int s0 = 0; s0 < P.nseg; s0 += kChunkSegs) {
                            if (!wait(&b_full[chunk], bphase, 9)) { ok = false; break; }
                            tc_fence_after();
                            const uint32_t db = db0 + chunk * (uint32_t)kChunkSegs * b_seg;
                            for (int t = issuer; t < P.T; t += kIssuers) {
                                if (tap == 0 && s0 == 0) {
                                    if (!wait(&acc_empty[t], plane_phase ^ 1u, 2)) { ok = false; break; }
                                    tc_fence_after();
                                }
                                const uint32_t dt = utmem + (uint32_t)(t * 3 * CG);
                                const uint32_t t0 = dt + (uint32_t)(d0 * CG), t1 = dt + (uint32_t)(d1 * CG);
                                const uint32_t at = ay + (uint32_t)(t * P.mstep) * kRowStep + (uint32_t)s0 * a_seg;
                                switch (P.nseg - s0) {
                                case 1: issue_taps<1, 1>(t0, t1, at, db + bo0, db + bo1, hi, id0, id1, n1, 0u, 0u, a_seg, b_seg); break;
                                case 2: issue_taps<1, 2>(t0, t1, at, db + bo0, db + bo1, hi, id0, id1, n1, 0u, 0u, a_seg, b_seg); break;
                                case 3: issue_taps<1, 3>(t0, t1, at, db + bo0, db + bo1, hi, id0, id1, n1, 0u, 0u, a_seg, b_seg); break;
                                default: issue_taps<1, 4>(t0, t1, at, db + bo0, db + bo1, hi, id0, id1, n1, 0u, 0u, a_seg, b_seg); break;
                                }
                            }
                            if (!ok) break;
                            tc_commit(&b_empty[chunk]);
                            if (++chunk == P.chunks) { chunk = 0; bphase ^= 1u; }
                        }
                    }
                    if (ok)
                        for (int t = issuer; t < P.T; t += kIssuers) tc_commit(&acc_full[t]);
                }
                if (!ok) break;
                tc_commit(&empty_bar[stage]);      // frees the plane when these MMAs are done
                if (++stage == P.stages) { stage = 0; phase ^= 1u; }
                plane_phase ^= 1u;
            }
            u += ze - zs;
        }
        // every MMA has completed before TMEM is released (below)
        tc_commit(&drain_bar[issuer]);
        volatile int never = 0;
        mbar_wait(&drain_bar[issuer], 0, &never, P.status, 6);
    } else {
        // ---------------------------------------------------------- epilogue
        const int quarter = warp & 3;                  // TMEM lanes 32*quarter .. +31
        const int set = (warp - 1 - kIssuers) >> 2;
        float hw[CG == 16 ? 17 : 1];                   // the output layer's weights and bias
        if (CG == 16 && P.head.y != nullptr) {
#pragma unroll
            for (int j = 0; j < 17; ++j) hw[j] = __ldg(j < 16 ? P.head.w + j : P.head.b);
        }
        if (ANY_W && u_begin < u_end) {
            const long long first = u_begin % P.D, last = first + (u_end - u_begin) - 1;
            const bool below = first == 0 || last >= P.D, above = last >= P.D - 1;   // of the output planes of this share
            if (below || above)
                z_border<CG, 4 * kSets>(P.w, cg * CG, P.nseg * kSeg, border, below, above, warp - 1 - kIssuers, lane);
        }
        uint32_t plane_phase = 0;
        bool ok = true;
        for (long long u = u_begin; u < u_end && ok;) {
            const int col = (int)(u / P.D), zs = (int)(u % P.D);
            const int ze = (int)(u_end - u < P.D - zs ? zs + (u_end - u) : P.D);
            const int x0 = (col % P.tiles_x) * P.BW, y0 = (col / P.tiles_x) * P.BY;
            for (int z = max(zs - 1, 0); z <= min(ze, P.D - 1) && ok; ++z) {
                for (int t = set; t < P.T; t += kSets) {
                    const bool got = mbar_wait(&acc_full[t], plane_phase, &abort_flag, P.status, 4);
                    if (!__all_sync(0xffffffffu, got)) { ok = false; break; }   // warp-uniform: tcgen05.ld is .sync.aligned
                    tc_fence_after();
                    const uint32_t row = (uint32_t)(t * P.mstep + quarter * 32 + lane);
                    const uint32_t yy = (row * P.pitch_magic) >> 20, xx = row - yy * (uint32_t)P.pitch;
                    const int x = x0 + (int)xx, y = y0 + (int)yy;
                    const bool live = xx < (uint32_t)P.BW && yy < (uint32_t)P.BY && x < P.W && y < P.H;
                    // plane z finishes output plane z - 1, and itself where no plane follows
                    for (int zo = max(z - 1, zs); zo <= z; ++zo) {
                        if (zo == z && !(z == P.D - 1 && ze == P.D)) break;
                        const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) +
                                            (uint32_t)((t * 3 + (2 * zo) % 3) * CG);
                        uint32_t v[CG / 16][16];
#pragma unroll
                        for (int q = 0; q < CG / 16; ++q) tc_ld16(ta + (uint32_t)(16 * q), v[q]);
                        tc_wait_ld();
#pragma unroll
                        for (int q = 0; q < CG / 16; ++q) tc_zero16(ta + (uint32_t)(16 * q));
                        if (ANY_W && (zo == 0 || zo == P.D - 1)) {   // of its own: in the loop below it cost the network 7 %
                            const float *lo = border[0], *hi = border[1];
                            if (zo != 0) lo = hi;
                            if (zo != P.D - 1) hi = lo;
#pragma unroll
                            for (int q = 0; q < CG / 16; ++q)
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    v[q][j] = __float_as_uint(__uint_as_float(v[q][j]) + (lo[16 * q + j] + hi[16 * q + j]));
                        }
                        if (live) {
                            const size_t o = (((size_t)zo * P.H + y) * P.W + x) * P.N + cg * CG;
#pragma unroll
                            for (int q = 0; q < CG / 16; ++q) {
                                __align__(16) __nv_bfloat162 r[8];
                                __align__(16) __nv_bfloat162 m[8];
                                if (P.mask != nullptr) {
                                    const uint4 *ms = reinterpret_cast<const uint4 *>(P.mask + o + 16 * q);
                                    reinterpret_cast<uint4 *>(m)[0] = __ldg(ms);
                                    reinterpret_cast<uint4 *>(m)[1] = __ldg(ms + 1);
                                }
#pragma unroll
                                for (int j = 0; j < 8; ++j) {
                                    float a = __uint_as_float(v[q][2 * j]), b = __uint_as_float(v[q][2 * j + 1]);
                                    if (P.bias != nullptr) {
                                        a += __ldg(P.bias + cg * CG + 16 * q + 2 * j);
                                        b += __ldg(P.bias + cg * CG + 16 * q + 2 * j + 1);
                                    }
                                    if (P.relu) {
                                        a = fmaxf(a, 0.f);
                                        b = fmaxf(b, 0.f);
                                    }
                                    if (P.mask != nullptr) {
                                        const float2 mf = __bfloat1622float2(m[j]);
                                        if (!(mf.x > 0.f)) a = 0.f;
                                        if (!(mf.y > 0.f)) b = 0.f;
                                    }
                                    r[j] = __floats2bfloat162_rn(a, b);
                                }
                                if (P.out != nullptr) {
                                    uint4 *d4 = reinterpret_cast<uint4 *>(P.out + o + 16 * q);
                                    const uint4 *r4 = reinterpret_cast<const uint4 *>(r);
                                    if (P.out32) {
                                        st32(d4, r4[0], r4[1]);
                                    } else {
                                        d4[0] = r4[0];
                                        d4[1] = r4[1];
                                    }
                                }
                                if (CG == 16 && P.head.y != nullptr) {
                                    float h = hw[16];
#pragma unroll
                                    for (int j = 0; j < 8; ++j) {
                                        const float2 f = __bfloat1622float2(r[j]);
                                        h = fmaf(hw[2 * j], f.x, h);
                                        h = fmaf(hw[2 * j + 1], f.y, h);
                                    }
                                    const size_t vox = o / 16;
                                    P.head.y[vox] = __ldg(P.head.x + vox) + h;
                                }
                            }
                        }
                        __syncwarp();
                    }
                    tc_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[t]);
                }
                plane_phase ^= 1u;
            }
            u += ze - zs;
        }
    }

    // wind down: every role has left its loop (all waits are bounded)
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) {
        // loads still in flight after an abort: at most the last ones into each buffer (bounded waits; a load
        // that was waited for already passes at once)
        volatile int never = 0;
        if (abort_flag) {
            for (unsigned long long q = issued_sh > P.stages ? issued_sh - P.stages : 0; q < issued_sh; ++q)
                mbar_wait(&full_bar[q % P.stages], (uint32_t)((q / P.stages) & 1u), &never, P.status, 5);
            const unsigned long long nb = P.resident ? 1 : P.chunks;
            for (unsigned long long q = b_issued_sh > nb ? b_issued_sh - nb : 0; q < b_issued_sh; ++q)
                mbar_wait(&b_full[q % nb], (uint32_t)((q / nb) & 1u), &never, P.status, 5);
        }
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

// ------------------------------------------------------------------ host side

using kvtma::encoder;

// Activation map: [D][H][W][C] BF16, box {16, bx, by, 1}.
inline bool encode_act(CUtensorMap *m, const void *ptr, int C, int D, int H, int W, int bx, int by) {
    cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D};
    cuuint64_t strides[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
    cuuint32_t box[4] = {(cuuint32_t)kSeg, (cuuint32_t)bx, (cuuint32_t)by, 1};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Weight map: [N][27][K] BF16 seen as (K, N, 3 dz, 9 (dy, dx)), box {16, cg, dz, taps}.
inline bool encode_w(CUtensorMap *m, const void *ptr, int N, int K, int cg, int dz, int taps) {
    cuuint64_t dims[4] = {(cuuint64_t)K, (cuuint64_t)N, 3, 9};
    cuuint64_t strides[3] = {(cuuint64_t)27 * K * 2, (cuuint64_t)9 * K * 2, (cuuint64_t)K * 2};
    cuuint32_t box[4] = {(cuuint32_t)kSeg, (cuuint32_t)cg, (cuuint32_t)dz, (cuuint32_t)taps};
    cuuint32_t es[4] = {1, 1, 1, 1};
    return encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(ptr), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline uint32_t align1k(uint32_t x) { return (x + 1023u) & ~1023u; }

// Whether a D x H x W volume is a whole number of 128-voxel boxes (BW =
// min(W, 128), BH = min(H, 128 / BW), the rest in z): what the tensor-core
// entry of the single-layer convolution accepts.
inline bool tile_shape(int D, int H, int W) {
    const int BW = W < kTileM ? W : kTileM;
    if (BW <= 0 || kTileM % BW != 0 || W % BW != 0) return false;
    const int BH = H < kTileM / BW ? H : kTileM / BW;
    if (BH <= 0 || (kTileM / BW) % BH != 0 || H % BH != 0) return false;
    return D % (kTileM / (BW * BH)) == 0;
}

// The largest group of output channels, a multiple of 16 up to 64 that divides N.
inline int channel_group(int N) {
    for (int g = 64; g > 16; g -= 16)
        if (N % g == 0) return g;
    return 16;
}

// Shape of one launch: column extent, sub-tiles, plane buffers and weights in
// shared memory, chosen by the estimated time of the busiest CTA.  An MMA of n
// dz groups takes max(shared-memory reads of A and B at 128 B a cycle, n * CG /
// 2 cycles of arithmetic), measured 46 cycles at CG = 16, n = 3; loads come at
// about 32 B a cycle and SM out of L2; waits, commits and address set-up cost
// about 300 cycles a sub-tile (resident weights) or a piece of weights;
// draining a sub-tile takes about 1200 + 10 CG cycles from its last MMA to the
// next plane's first, so few sub-tiles leave the pipe idle (16 -> 16 channels
// at 64 x 512 x 512 voxels: four 318 us, eight 278).  A single plane buffer
// exposes its load.
inline bool plan_shape(Params &P, int CG, int sm_count, int *grid, size_t *smem) {
    const uint32_t budget = 224u * 1024u;
    const int max_t = std::min(kMaxT, 512 / (3 * CG));
    const int parts = sm_count / P.ncg > 0 ? sm_count / P.ncg : 1;
    auto mma = [&](int n) {
        const double rd = (kTileM * kRow + n * CG * kRow) / 128.0, ar = n * CG / 2.0;
        return rd > ar ? rd : ar;
    };
    const double whole = mma(3), split = (mma(3) + 2 * (mma(2) + mma(1))) / 3;
    double best = 1e300;
    for (int wide = 0; wide < 6; ++wide) {
        // one y row per sub-tile (wide == 0), or consecutive rows of a narrower column
        const int BW = wide == 0 ? kTileM : (wide == 1 ? P.W : 256 >> wide);   // W, 64, 32, 16, 8
        if (wide == 0 ? P.W < kTileM : (wide == 1 ? P.W > 254 : BW >= P.W)) continue;
        const int pitch = BW + 2;
        for (int T = 1; T <= max_t; ++T) {
            if (wide != 0 && T * kTileM < BW) continue;
            int BY = wide == 0 ? T : (T * kTileM - BW) / pitch + 1;
            if (BY > 254) continue;
            if (BY > P.H) {
                if (wide == 0 || (P.H - 1) * pitch + BW <= (T - 1) * kTileM) continue;   // fewer sub-tiles do
                BY = P.H;
            }
            const int mstep = wide == 0 ? pitch : kTileM;
            const int tx = (P.W + BW - 1) / BW, ty = (P.H + BY - 1) / BY;
            const long long units = (long long)tx * ty * P.D;
            const uint32_t rows = (uint32_t)std::max((BY + 2) * pitch, (T - 1) * mstep + kTileM + 2 * pitch + 2);
            const uint32_t a_bytes = align1k(rows * kRow), plane_bytes = a_bytes * (uint32_t)P.nseg;
            for (int mode = 0; mode < 3; ++mode) {   // resident x 5 groups, resident x 3, streamed x 3
                if (mode < 2 && P.nseg > kChunkSegs) continue;
                const int groups = mode == 0 ? 5 : 3;
                const uint32_t b_seg = (uint32_t)((mode < 2 ? 9 : 1) * groups * CG * kRow);
                const uint32_t piece = b_seg * (uint32_t)kChunkSegs;
                for (uint32_t bufs = 1; bufs <= (mode < 2 ? 4u : 2u); ++bufs) {
                    uint32_t chunks = 0, b_bytes;
                    if (mode < 2) {
                        b_bytes = align1k(b_seg * (uint32_t)P.nseg);
                    } else {
                        if (bufs * plane_bytes + 2 * piece > budget) continue;
                        chunks = std::min<uint32_t>(kMaxChunks, (budget - bufs * plane_bytes) / piece);
                        b_bytes = align1k(chunks * piece);
                    }
                    if (bufs * plane_bytes + b_bytes > budget) continue;
                    const int tiles = (T + issuers(CG) - 1) / issuers(CG);   // of one issuer
                    const int pieces = mode < 2 ? tiles : 9 * ((P.nseg + kChunkSegs - 1) / kChunkSegs);
                    const double compute = 9.0 * T * P.nseg * (mode == 0 ? whole : split) + 150.0 * pieces;
                    const double load_a = (double)P.nseg * (BY + 2) * pitch * kRow / 32.0;
                    const double load_b = mode < 2 ? 0.0 : 27.0 * P.nseg * CG * kRow / 32.0;
                    const double drain = 1200.0 + 10.0 * CG, drains = (T + drain_sets(CG) - 1) / drain_sets(CG) * 0.6 * drain;
                    // a sub-tile's next plane waits for its drain: its own MMAs (those of the issuers side by side),
                    // then the drain; streamed weights finish every sub-tile at the plane's end
                    const double chain = compute / T * (mode == 2 ? T : std::min(T, issuers(CG))) + drain;
                    double plane = bufs == 1 ? std::max(compute, load_b) + load_a + 1500.0
                                             : std::max(compute, load_a + load_b) + (bufs == 2 ? 200.0 : 0.0);
                    plane = std::max(plane, std::max(drains, chain));
                    const long long per = (units + parts - 1) / parts;
                    const double cols = 1.0 + (double)per / P.D;
                    const double total = plane * (per + 0.8 * 2 * cols) + (mode < 2 ? b_bytes / 32.0 : 0.0);
                    if (total >= best) continue;
                    best = total;
                    P.BW = BW;
                    P.BY = BY;
                    P.pitch = pitch;
                    P.T = T;
                    P.mstep = mstep;
                    P.pitch_magic = ((1u << 20) + pitch - 1) / pitch;
                    P.tiles_x = tx;
                    P.units = units;
                    P.groups = groups;
                    P.resident = mode < 2;
                    P.stages = bufs;
                    P.a_bytes = a_bytes;
                    P.a_tx = (uint32_t)((BY + 2) * pitch * kRow);
                    P.b_off = bufs * plane_bytes;
                    P.b_seg_bytes = b_seg;
                    P.chunks = chunks;
                    *grid = (int)std::min<long long>(parts, units) * P.ncg;
                    *smem = (size_t)bufs * plane_bytes + b_bytes + 1024;
                }
            }
        }
    }
    return best < 1e300;
}

// out[v][N] = conv3(in1 (c1 channels) ++ in2 (c2 channels), w [N][27][c1+c2]) + bias, ReLU optional, zero where
// `mask` (a tensor like out; nullptr: none) is not positive; out may be nullptr where `head` takes the result.
// any_w: the weights may hold infinities and NaN (which meet the zeros outside the volume).
// Returns a message on a configuration this kernel does not cover (nullptr: launched).
inline const char *launch(const __nv_bfloat16 *in1, int c1, const __nv_bfloat16 *in2, int c2,
                          const __nv_bfloat16 *w, const float *bias, bool relu, const __nv_bfloat16 *mask,
                          const Head *head, __nv_bfloat16 *out, int N, int D, int H, int W, bool any_w, int *status,
                          int sm_count, cudaStream_t stream) {
    if (encoder() == nullptr) return "cuTensorMapEncodeTiled is not available";
    const int K = c1 + c2;
    auto ok_c = [](int c) { return c == 16 || c == 32 || c == 64 || c == 128; };
    if (!ok_c(c1) || (c2 != 0 && !ok_c(c2))) return "input channels must be 16, 32, 64 or 128";
    if (N % 16 != 0 || N < 16 || N > 256) return "output channels must be a multiple of 16 up to 256";
    // The operator's limits: four segments of one width, and 128 + N rows of every segment twice in 200 KB.  This kernel
    // could take more (plan_shape); they are the interface's, tested, so that no caller comes to rely on others.
    const int kseg = std::min(std::min(c1, 64), c2 != 0 ? c2 : 64), segs = K / kseg;
    if (segs > 4) return "too many input channel segments";
    if (2 * (size_t)segs * (align1k(kTileM * kseg * 2) + align1k(N * kseg * 2)) > 200 * 1024)
        return "stage does not fit in shared memory";
    if ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(mask)) % 16 != 0)
        return "output or mask is not 16-byte aligned";
    if (head != nullptr && N != 16) return "the output layer takes 16 channels";
    const int CG = channel_group(N);
    Params P{};
    P.nseg = K / kSeg;
    P.nseg1 = c1 / kSeg;
    P.N = N;
    P.ncg = N / CG;
    P.D = D;
    P.H = H;
    P.W = W;
    int grid = 0;
    size_t smem = 0;
    if (!plan_shape(P, CG, sm_count, &grid, &smem)) return "no tile shape for this volume";
    P.tmem_cols = 32;
    while (P.tmem_cols < (uint32_t)(3 * CG * P.T)) P.tmem_cols <<= 1;
    P.w = w;
    P.bias = bias;
    P.relu = relu ? 1 : 0;
    P.mask = mask;
    P.out = out;
    P.out32 = reinterpret_cast<uintptr_t>(out) % 32 == 0;
    if (head != nullptr) P.head = *head;
    P.status = status;
    CUtensorMap ma0, ma1, mb, mb2;
    if (!encode_act(&ma0, in1, c1, D, H, W, P.pitch, P.BY + 2)) return "activation tensor map rejected";
    if (!encode_act(&ma1, c2 ? in2 : in1, c2 ? c2 : c1, D, H, W, P.pitch, P.BY + 2))
        return "activation tensor map rejected";
    const bool per_tap = P.resident && P.groups == 5;   // dz = 0 1 2 and dz = 0 1 of one (dy, dx) per load
    if (!encode_w(&mb, w, N, K, CG, 3, per_tap || !P.resident ? 1 : 9) || !encode_w(&mb2, w, N, K, CG, 2, 1))
        return "weight tensor map rejected";
    auto go = [&](auto kernel) -> const char * {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
            return "shared memory request rejected";
        kernel<<<(unsigned)grid, threads(CG), smem, stream>>>(ma0, ma1, mb, mb2, P);
        return nullptr;
    };
    switch (CG) {
    case 16: return any_w ? go(conv3_march_kernel<16, true>) : go(conv3_march_kernel<16, false>);
    case 32: return any_w ? go(conv3_march_kernel<32, true>) : go(conv3_march_kernel<32, false>);
    case 48: return any_w ? go(conv3_march_kernel<48, true>) : go(conv3_march_kernel<48, false>);
    default: return any_w ? go(conv3_march_kernel<64, true>) : go(conv3_march_kernel<64, false>);
    }
}

}  // namespace convtc
