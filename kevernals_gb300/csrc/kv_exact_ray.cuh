// kv_exact_ray.cuh -- one ray of the EXACT forward projector, walked voxel by
// voxel: the one-thread-per-ray kernel, and the rays that the slab kernel sums
// again.
#pragma once

#include "kv_exact_common.cuh"
#include "kv_internal.h"

namespace {

// Range [k0, k1] of slices in which the ray may be inside the volume laterally.
__device__ __forceinline__ void lateral_slices(float pos0, float slope, int n, int nz, float &klo,
                                               float &khi) {
    // pos(k) = pos0 + slope * k must stay in [0, n]
    if (fabsf(slope) < 1e-30f) {
        if (pos0 < 0.f || pos0 > (float)n) { klo = 1.f; khi = 0.f; }
        else { klo = 0.f; khi = (float)nz; }
        return;
    }
    float a = (0.f - pos0) / slope, b = ((float)n - pos0) / slope;
    klo = fminf(a, b);
    khi = fmaxf(a, b);
}

// Adds the ray's slice-local lengths times voxel values to acc (and, WSUM, the
// lengths to wsum).  Volume rows are `pitch` elements apart.
template <typename VolT, bool WSUM>
__device__ __forceinline__ void ray_walk(const ExGeom &G, const ExactTables &T, const VolT *vol, int pitch, int u, int v,
                                         int p, float &acc, float &wsum) {
    const float4 X = T.xt[(size_t)p * G.nu + u];
    const int ib = T.xi[(size_t)p * G.nu + u];
    const float4 Y = T.yt[(size_t)p * G.nv + v];
    const int jb = T.yi[(size_t)p * G.nv + v];
    const float4 VI = T.vinfo[p];
    const float *hr = T.hr + (size_t)p * (G.nz + 1);
    const int mvx = X.z > 0.f ? 1 : -1, mvy = Y.z > 0.f ? 1 : -1;
    const int ex = mvx > 0 ? 1 : 0, ey = mvy > 0 ? 1 : 0;

    // lateral clipping to the slices the ray can reach inside the volume
    const float hr0 = hr[0], dh = VI.y;
    float kxl, kxh, kyl, kyh;
    lateral_slices((float)ib + fmaf(X.y, hr0, X.x), X.y * dh, G.nx, G.nz, kxl, kxh);
    lateral_slices((float)jb + fmaf(Y.y, hr0, Y.x), Y.y * dh, G.ny, G.nz, kyl, kyh);
    // clamp in float first: converting a huge value saturates and the -1 / +1 would wrap
    const float klo = fmaxf(fmaxf(kxl, kyl), -2.f), khi = fminf(fminf(kxh, kyh), (float)G.nz + 2.f);
    int k0 = 0, k1 = -1;
    if (klo <= khi) {
        k0 = max(0, (int)floorf(klo) - 1);
        k1 = min(G.nz - 1, (int)ceilf(khi) + 1);
    }
    // interior slices: the whole path in the slice stays two voxels away
    // from the lateral faces, so no voxel it visits needs a bounds check
    float ixl, ixh, iyl, iyh;
    lateral_slices((float)ib + fmaf(X.y, hr0, X.x) - 2.f, X.y * dh, G.nx - 4, G.nz, ixl, ixh);
    lateral_slices((float)jb + fmaf(Y.y, hr0, Y.x) - 2.f, Y.y * dh, G.ny - 4, G.nz, iyl, iyh);
    const float kil = fmaxf(fmaxf(ixl, iyl), -2.f), kih = fminf(fminf(ixh, iyh), (float)G.nz + 2.f);
    int ki0 = (int)ceilf(kil), ki1 = (int)floorf(kih) - 1;   // slice k needs planes k, k+1 inside
    if (G.nx < 5 || G.ny < 5) {   // no interior: the margins above would invert
        ki0 = 1;
        ki1 = 0;
    }

    const size_t plane = (size_t)pitch * G.ny;
    const float fmvx = (float)mvx, fmvy = (float)mvy;
    const int step_y = mvy * pitch;
    for (int k = k1; k >= k0; --k) {
        const float htop = hr[k + 1];
        const float ftx = __fmaf_rn(X.y, htop, X.x);
        const float fty = __fmaf_rn(Y.y, htop, Y.x);
        const int i = mvx > 0 ? (int)floorf(ftx) : (int)ceilf(ftx) - 1;
        const int j = mvy > 0 ? (int)floorf(fty) : (int)ceilf(fty) - 1;
        // next x / y plane as floats (exact integers): cross_t without conversions
        float fxp = (float)(i + ex), fyp = (float)(j + ey);
        float tx = __fmul_rn(__fsub_rn(fxp, ftx), X.z);
        float ty = __fmul_rn(__fsub_rn(fyp, fty), Y.z);
        float t = 0.f;
        const VolT *slice = vol + (size_t)k * plane;
        if (k >= ki0 && k <= ki1) {
            // Row segments of the (warp-uniform) y walk; inside each, the
            // lane's x crossings.  Weights: same expressions as the
            // backprojector's min(1, tx_hi, ty_hi) - max(0, tx_lo, ty_lo).
            const VolT *ptr = slice + (size_t)(jb + j) * pitch + (ib + i);
            while (true) {
                const float tb = fminf(ty, 1.0f);
                const bool cross = tx < tb;
                const float te = fminf(tx, tb);
                const float w = __fsub_rn(te, t);
                acc = fmaf(w, Store<VolT>::ld(ptr), acc);
                if (WSUM) wsum += w;
                // the common case -- at most one column crossing in the
                // row segment -- without a divergent branch
                float vc = cross ? Store<VolT>::ld(ptr + mvx) : 0.f;
                ptr += cross ? mvx : 0;
                fxp += cross ? fmvx : 0.f;
                tx = __fmul_rn(__fsub_rn(fxp, ftx), X.z);
                float tc = te;
                while (tx < tb) {   // rarely: a second crossing in the same row
                    const float w2 = __fsub_rn(tx, tc);
                    acc = fmaf(w2, vc, acc);
                    if (WSUM) wsum += w2;
                    tc = tx;
                    ptr += mvx;
                    fxp += fmvx;
                    tx = __fmul_rn(__fsub_rn(fxp, ftx), X.z);
                    vc = Store<VolT>::ld(ptr);
                }
                const float w3 = __fsub_rn(tb, tc);
                acc = fmaf(w3, vc, acc);
                if (WSUM) wsum += w3;
                t = tb;
                if (tb >= 1.0f) break;
                ptr += step_y;
                fyp += fmvy;
                ty = __fmul_rn(__fsub_rn(fyp, fty), Y.z);
            }
        } else {
            int ai = ib + i, aj = jb + j;
            while (true) {
                const float tb = fminf(ty, 1.0f);
                const bool row_in = (unsigned)aj < (unsigned)G.ny;
                const VolT *row = slice + (size_t)(row_in ? aj : 0) * pitch;
                while (tx < tb) {
                    if (row_in && (unsigned)ai < (unsigned)G.nx) {
                        const float w = __fsub_rn(tx, t);
                        acc = fmaf(w, Store<VolT>::ld(row + ai), acc);
                        if (WSUM) wsum += w;
                    }
                    t = tx;
                    ai += mvx;
                    fxp += fmvx;
                    tx = __fmul_rn(__fsub_rn(fxp, ftx), X.z);
                }
                if (row_in && (unsigned)ai < (unsigned)G.nx) {
                    const float w = __fsub_rn(tb, t);
                    acc = fmaf(w, Store<VolT>::ld(row + ai), acc);
                    if (WSUM) wsum += w;
                }
                t = tb;
                if (tb >= 1.0f) break;
                aj += mvy;
                fyp += fmvy;
                ty = __fmul_rn(__fsub_rn(fyp, fty), Y.z);
            }
        }
    }
}

}  // namespace
